"""Inputs at the edges of what the calls accept.

Planes that break the input contract under FLAG_NO_VALIDATE give counts outside
0 .. N and scores that mean nothing; the call must still stay inside its tables
and buffers and leave the next search correct.
"""
import numpy as np
import pytest

from test_parity_gpu import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("score", ["k2", "mi"])
@pytest.mark.parametrize("engine,order", [("simt", 2), ("simt", 3), ("tensor", 2)])
def test_impossible_counts_stay_inside_the_score_tables(episdet, oracle, engine, order, score):
    """Both planes of a SNP full: derived cells are negative, down to -N."""
    M, nc, nn, k = 40, 700, 900, 64
    good = episdet.generate(0x1A7, M, nc, nn)
    bad = [p.copy() for p in good]
    for p, n in zip(bad, (nc, nn)):
        p[5:9, :, : n // 32] = 0xFFFFFFFF
    try:
        episdet.search(*bad, nc, nn, order=order, score=score, top_k=k, engine=engine, flags=episdet.FLAG_NO_VALIDATE)
    except episdet.EpisdetError as e:
        assert e.name == "EPISDET_ERR_INTERNAL"
    o = oracle.search(*good, nc, nn, order=order, score=score, top_k=k)
    assert_same(episdet.search(*good, nc, nn, order=order, score=score, top_k=k, engine=engine), o, k)
