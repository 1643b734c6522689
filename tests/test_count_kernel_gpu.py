"""The counting kernel at the edges of its tiles, against the oracle.

Tiles are 128 A SNPs x 112 (wide) or 56 (narrow) B SNPs; panels of up to 704
SNPs and 48,000 samples run narrow triplet tiles, pairs run narrow tiles when wide ones are fewer
than the CTA pairs.  Counts pass through a buffer of 16-bit values, or 32-bit
ones for a first SNP with a kept genotype of more than 65,535 samples.  K is
cut in blocks of 256 samples per segment.  Everything is exact, so the bar is
equality; FILTER_OFF scores every set exactly, without the score bound.
"""
import pytest

from test_parity_gpu import assert_same

pytestmark = pytest.mark.gpu


def check(episdet, oracle, order, M, nc, nn, score, k, maf=(0.05, 0.5), seed=0xC0DE, slab=(0, 0), flags=(0,), **planted):
    cases, controls = episdet.generate(seed + M, M, nc, nn, maf=maf, **planted)
    o = oracle.search(cases, controls, nc, nn, order=order, score=score, top_k=k, first_begin=slab[0], first_end=slab[1])
    for f in flags:
        r = episdet.search(cases, controls, nc, nn, order=order, score=score, top_k=k, engine="tensor",
                           first_begin=slab[0], first_end=slab[1], flags=f)
        assert_same(r, o, k)
        assert r.sets_evaluated == o["sets"]


@pytest.mark.parametrize("score", ["k2", "mi"])
@pytest.mark.parametrize("order,M", [(2, 2), (3, 3), (3, 56), (3, 57), (3, 113), (2, 127), (2, 129), (3, 129), (2, 1130)])
def test_tile_edges(episdet, oracle, order, M, score):
    k = 300
    check(episdet, oracle, order, M, 257, 511, score, k, flags=(0, episdet.FLAG_FILTER_OFF))


@pytest.mark.parametrize("score", ["k2", "mi"])
@pytest.mark.parametrize("M,slab", [(704, (696, 0)), (705, (0, 1)), (705, (126, 129)), (784, (330, 336))])
def test_triplet_tile_widths_and_list_edges(episdet, oracle, M, slab, score):
    check(episdet, oracle, 3, M, 1300, 900, score, 1536, slab=slab)


def test_narrow_tiles_with_counts_past_16_bits(tmp_path):
    """Reached by an autotuned choice only (here from a cache file)."""
    import os
    import subprocess
    import sys

    import episdet as e

    cache = tmp_path / "tune.txt"
    cache.write_text("3 0 17 0\n")
    code = f"""
import sys
sys.path.insert(0, {os.path.dirname(e.__file__)!r})
import numpy as np, episdet
n = (170000, 150000)
data = episdet.generate(11, 40, *n, maf=(0.3, 0.36))
wide, narrow = (episdet.search(*data, *n, order=3, top_k=64, engine="tensor", flags=f | episdet.FLAG_TIMING)
                for f in (0, episdet.FLAG_AUTOTUNE))
assert 1.9 < wide.executed_macs / narrow.executed_macs < 2.1
assert np.array_equal(wide.top_snps, narrow.top_snps) and np.array_equal(wide.top_fp64, narrow.top_fp64)
assert np.array_equal(wide.top_fp32.view(np.uint32), narrow.top_fp32.view(np.uint32))
"""
    p = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, EPISDET_TUNE_CACHE=str(cache)))
    assert p.returncode == 0, p.stderr


def test_tile_width_follows_the_samples_too(episdet, oracle):
    """40 SNPs are one tile of either width: a wide one issues twice the MACs."""
    M, k, macs = 40, 64, []
    for nn in (24000, 24001):
        cases, controls = episdet.generate(5, M, 24000, nn, maf=(0.3, 0.36))
        r = episdet.search(cases, controls, 24000, nn, order=3, top_k=k, engine="tensor", flags=episdet.FLAG_TIMING)
        assert_same(r, oracle.search(cases, controls, 24000, nn, order=3, score="k2", top_k=k), k)
        macs.append(r.executed_macs)
    assert 1.9 < macs[1] / macs[0] < 2.1


@pytest.mark.parametrize("order,M,slab", [(3, 24, (0, 0)), (3, 710, (3, 4)), (2, 40, (0, 0)), (2, 1500, (700, 703))])
def test_counts_past_16_bits(episdet, oracle, order, M, slab):
    check(episdet, oracle, order, M, 170000, 150000, "k2", 64, maf=(0.3, 0.36), slab=slab,
          flags=(0, episdet.FLAG_FILTER_OFF))


@pytest.mark.parametrize("order,M,slab", [(3, 30, (0, 0)), (2, 40, (0, 0)), (2, 1500, (700, 702))])
def test_counts_past_16_bits_mi(episdet, oracle, order, M, slab):
    check(episdet, oracle, order, M, 170000, 150000, "mi", 64, maf=(0.3, 0.36), slab=slab,
          flags=(0, episdet.FLAG_FILTER_OFF))


@pytest.mark.parametrize("score", ["k2", "mi"])
@pytest.mark.parametrize("nc", [20000, 80000])
def test_permutations_past_16_bits(episdet, oracle, score, nc):
    """Pair totals of 150,000 samples (32-bit counts, one class); 80,000 cases are
    counted in 32 bits too, 20,000 in 16."""
    n, M, k = 150000, 40, 50
    planes = episdet.generate_cohort(31, M, n, maf=(0.3, 0.5))
    labels = episdet.generate_labels(32, n, nc, 2)
    got = episdet.search_perm(planes, n, labels, order=2, score=score, top_k=k)
    for lab, r in zip(labels, got):
        a, b, na, nb = oracle.split_by_label(planes, n, lab)
        assert_same(r, oracle.search(a, b, na, nb, order=2, score=score, top_k=k), k)


@pytest.mark.parametrize("score", ["k2", "mi"])
def test_more_ties_than_the_merge_holds(episdet, oracle, score):
    """Every SNP the same: all scores equal, the smallest sets win."""
    import numpy as np

    cases, controls = episdet.generate(9, 1, 300, 260)
    M, k = 260, 500
    cases, controls = np.repeat(cases, M, 0), np.repeat(controls, M, 0)
    o = oracle.search(cases, controls, 300, 260, order=2, score=score, top_k=k)
    for flags in (0, episdet.FLAG_FILTER_OFF):
        assert_same(episdet.search(cases, controls, 300, 260, order=2, score=score, top_k=k, engine="tensor",
                                   flags=flags), o, k)


def test_autotune_keeps_the_answer(episdet, oracle):
    check(episdet, oracle, 3, 120, 2000, 2100, "k2", 200, flags=(episdet.FLAG_AUTOTUNE, 0))
    assert episdet.tuned_stage(3, "k2", 2000, 2100) in (0, 1)


def test_autotuned_choice_is_for_its_panel_size(episdet, oracle):
    check(episdet, oracle, 3, 100, 600, 500, "k2", 100, flags=(episdet.FLAG_AUTOTUNE,))
    assert episdet.tuned_tiles(3, "k2", 100, 600, 500) in (0, 1)
    assert episdet.tuned_tiles(3, "k2", 1500, 600, 500) == -1


def test_permutations_device_labels_and_unaligned_planes(episdet, oracle):
    """Label mode takes labels and planes of either memory; planes that are not
    16-byte aligned go through the per-label split.  Same answers."""
    import numpy as np
    import torch

    n, M, nc, nl = 2085, 150, 700, 3
    planes = episdet.generate_cohort(77, M, n)
    labels = episdet.generate_labels(78, n, nc, nl)
    want = []
    for lab in labels:
        a, b, na, nb = oracle.split_by_label(planes, n, lab)
        want.append(oracle.search(a, b, na, nb, order=2, score="k2", top_k=40))
    dev = torch.from_numpy(planes.view(np.int32)).cuda()
    shifted = torch.zeros(dev.numel() + 1, dtype=torch.int32, device="cuda")
    shifted[1:] = dev.flatten()
    off = shifted[1:].view(dev.shape)
    dl = torch.from_numpy(labels.view(np.int32)).cuda()
    torch.cuda.synchronize()
    assert off.data_ptr() % 16 == 4
    for p, q in ((planes, labels), (dev, dl), (off, dl)):
        for r, o in zip(episdet.search_perm(p, n, q, order=2, score="k2", top_k=40), want):
            assert_same(r, o, 40)


def test_permutations_reject_overlapping_planes(episdet):
    n, M = 1500, 20
    planes = episdet.generate_cohort(5, M, n)
    labels = episdet.generate_labels(6, n, 600, 2)
    bad = planes.copy()
    bad[3, 0, 1] |= 0x10
    bad[3, 1, 1] |= 0x10
    with pytest.raises(episdet.EpisdetError) as e:
        episdet.search_perm(bad, n, labels, top_k=8)
    assert e.value.name == "EPISDET_ERR_INVALID_INPUT"
    empty = labels.copy()
    empty[1] = 0
    with pytest.raises(episdet.EpisdetError) as e:
        episdet.search_perm(planes, n, empty, top_k=8)
    assert e.value.name == "EPISDET_ERR_INVALID_ARGUMENT" and "label 1" in str(e.value)


@pytest.mark.parametrize("M,n", [(1, 2), (7, 1025), (8, 33000), (17, 70001)])
def test_binarize_groups_and_chunks(episdet, oracle, M, n):
    import numpy as np

    rng = np.random.default_rng(M)
    g = rng.integers(0, 3, size=(M, n)).astype(np.uint8)
    flags = rng.random(n) < 0.3
    flags[0], flags[-1] = True, False
    cases, controls, nc, nn = episdet.binarize(g, flags)
    assert np.array_equal(cases, oracle.pack(g[:, flags])) and np.array_equal(controls, oracle.pack(g[:, ~flags]))


def test_binarize_unaligned_device_arrays(episdet, oracle):
    """Device arrays that start at odd bytes (genotypes) and words (planes)."""
    import numpy as np
    import torch

    M, n = 19, 1301
    rng = np.random.default_rng(3)
    g = rng.integers(0, 3, size=(M, n)).astype(np.uint8)
    flags = (rng.random(n) < 0.5).astype(np.uint8)
    nc = int(flags.sum())
    wc, wn = episdet.class_words(nc), episdet.class_words(n - nc)
    dg = torch.zeros(M * n + 1, dtype=torch.uint8, device="cuda")
    dg[1:] = torch.from_numpy(g.reshape(-1)).cuda()
    df = torch.from_numpy(flags).cuda()
    out = [torch.zeros(M * 2 * w + 1, dtype=torch.int32, device="cuda") for w in (wc, wn)]
    torch.cuda.synchronize()
    st = episdet.lib().episdet_binarize(dg.data_ptr() + 1, M, n, df.data_ptr(), out[0].data_ptr() + 4,
                                        out[1].data_ptr() + 4, episdet.DEVICE, 0)
    assert st == 0
    for o, cls in zip(out, (flags != 0, flags == 0)):
        got = o.cpu().numpy().view(np.uint32)
        assert got[0] == 0 and np.array_equal(got[1:], oracle.pack(g[:, cls]).reshape(-1))
