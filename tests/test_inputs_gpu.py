"""Inputs at the edges of what the calls accept.

Planes that break the input contract under FLAG_NO_VALIDATE give counts outside
0 .. N and scores that mean nothing; the call must still stay inside its tables
and buffers and leave the next search correct.  Device inputs may still be on
their way on the stream that the call is given, and a cohort's padding bits are
not read.
"""
import ctypes

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


@pytest.mark.parametrize("full", [0, 1], ids=["cases", "controls"])
def test_kept_samples_stay_inside_the_regrouped_rows(episdet, oracle, full):
    """Both planes full in one class, genotype 2 the most frequent over both: the
    two kept genotypes list that class's samples twice, more than a row holds."""
    M, k = 150, 64
    n = [3000, 3000]
    n[full] = 1024  # 4 blocks of 256 samples a genotype; the class's region has 6
    good = episdet.generate(0x1A8, M, *n)
    bad = [p.copy() for p in good]
    for c, p in enumerate(bad):
        p[:, :, : n[c] // 32] = 0xFFFFFFFF if c == full else 0
    with pytest.raises(episdet.EpisdetError) as e:
        episdet.search(*bad, *n, order=3, top_k=k, engine="tensor", flags=episdet.FLAG_NO_VALIDATE)
    assert e.value.name == "EPISDET_ERR_INVALID_INPUT"
    o = oracle.search(*good, *n, order=3, score="k2", top_k=k)
    assert_same(episdet.search(*good, *n, order=3, top_k=k, engine="tensor"), o, k)


@pytest.mark.parametrize("score", ["k2", "mi"])
def test_cohort_padding_bits_are_not_counted(episdet, oracle, score):
    """Set bits past the last sample, of the planes and of the labels: label mode
    and the per-label split give the answer of the clean cohort."""
    n, M, nc, k = 2085, 60, 900, 50
    planes = episdet.generate_cohort(17, M, n)
    labels = episdet.generate_labels(18, n, nc, 2)
    want = []
    for lab in labels:
        a, b, na, nb = oracle.split_by_label(planes, n, lab)
        want.append(oracle.search(a, b, na, nb, order=2, score=score, top_k=k))
    rng = np.random.default_rng(19)
    for words in (planes, labels):
        w = n // 32
        words[..., w] |= rng.integers(0, 1 << (32 - n % 32), words[..., w].shape, dtype=np.uint32)
        words[..., w + 1:] = rng.integers(0, 1 << 32, words[..., w + 1:].shape, dtype=np.uint32)
    for flags in (0, episdet.FLAG_PERM_SPLIT):
        for r, o in zip(episdet.search_perm(planes, n, labels, order=2, score=score, top_k=k, flags=flags), want):
            assert_same(r, o, k)


@pytest.mark.parametrize("order,engine", [(2, "tensor"), (3, "tensor"), (3, "simt")])
def test_device_planes_still_being_written_on_the_callers_stream(episdet, oracle, order, engine):
    import torch

    M, nc, nn, k = 70, 1500, 1300, 32
    planes = episdet.generate(93, M, nc, nn)
    new = [torch.from_numpy(p.view("int32")).cuda() for p in planes]
    late = [torch.zeros_like(p) for p in new]
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(400_000_000)
        for p, q in zip(late, new):
            p.copy_(q)
    assert not stream.query()
    r = episdet.search(*late, nc, nn, order=order, top_k=k, engine=engine, stream=stream.cuda_stream)
    assert_same(r, oracle.search(*planes, nc, nn, order=order, score="k2", top_k=k), k)


def test_device_labels_still_being_written_on_the_callers_stream(episdet, oracle):
    """The labels (all zero until then) arrive on the caller's stream behind a
    wait of some tenths of a second, and are not what the buffer held before."""
    import torch

    n, M, nc, nl, k = 3000, 90, 1100, 3, 32
    planes = episdet.generate_cohort(91, M, n)
    labels = episdet.generate_labels(92, n, nc, nl)
    dev = torch.from_numpy(planes.view("int32")).cuda()
    new = torch.from_numpy(labels.view("int32")).cuda()
    late = torch.zeros_like(new)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    c = episdet.Cohort(dev.data_ptr(), M, n, episdet.DEVICE)
    o = episdet.make_options(2, "k2", k, stream=stream.cuda_stream)
    rs, keep = (episdet.Result * nl)(), []
    for i in range(nl):
        rs[i], bufs = episdet._result_buffers(k)
        keep.append(bufs)
    with torch.cuda.stream(stream):
        torch.cuda._sleep(400_000_000)
        late.copy_(new)
    assert not stream.query()  # the labels are not there yet
    episdet._check(episdet.lib().episdet_search_perm(ctypes.byref(c), late.data_ptr(), nl, ctypes.byref(o), rs))
    for i, lab in enumerate(labels):
        a, b, na, nb = oracle.split_by_label(planes, n, lab)
        want = oracle.search(a, b, na, nb, order=2, score="k2", top_k=k)
        assert_same(episdet._to_result(2, rs[i], keep[i]), want, k)


def test_binarize_most_samples(episdet):
    """2^31 - 1 samples: sample i is a case if i is odd, and sample j of either
    class has genotype j % 3, so that the plane words repeat every three."""
    import torch

    n = 2**31 - 1
    try:
        i = torch.arange(n, dtype=torch.int32, device="cuda")
        flags = (i & 1).to(torch.uint8)
        i >>= 1
        i %= 3
        g = i.to(torch.uint8)[None]
        del i
        cases, controls, nc, nn = episdet.binarize(g, flags)
        assert (nc, nn) == (n // 2, n - n // 2)
        del g, flags
        for got, k in ((cases, nc), (controls, nn)):
            bits = (np.arange(96)[None] % 3 == np.arange(2)[:, None]).astype(np.uint32).reshape(2, 3, 32)
            table = torch.from_numpy((bits << np.arange(31, -1, -1, dtype=np.uint32)).sum(2, dtype=np.uint32).view(np.int32))
            w = episdet.class_words(k)
            want = table.cuda()[:, torch.arange(w, device="cuda") % 3]
            want[:, (k + 31) // 32:] = 0
            if k % 32:
                want[:, k // 32] &= -1 << (32 - k % 32)
            assert torch.equal(got.view(2, w), want)
    finally:
        episdet.release_workspace(0)
        torch.cuda.empty_cache()


def test_unaligned_cohort_planes_run_in_label_mode(episdet, oracle):
    """4-byte aligned planes are copied; without room for the copy every label is
    split, with the same answers."""
    import torch

    n, M, nc, nl, k = 2085, 150, 700, 2, 40
    planes = episdet.generate_cohort(77, M, n)
    labels = episdet.generate_labels(78, n, nc, nl)
    dev = torch.from_numpy(planes.view(np.int32)).cuda()
    shifted = torch.zeros(dev.numel() + 1, dtype=torch.int32, device="cuda")
    shifted[1:] = dev.flatten()
    off = shifted[1:].view(dev.shape)
    dl = torch.from_numpy(labels.view(np.int32)).cuda()
    torch.cuda.synchronize()
    assert off.data_ptr() % 16 == 4
    aligned = episdet.search_perm(dev, n, dl, top_k=k)
    split = episdet.search_perm(dev, n, dl, top_k=k, flags=episdet.FLAG_PERM_SPLIT)
    assert aligned[0].kernel_launches != split[0].kernel_launches
    for fail, same in ((0, aligned), (1, split)):
        episdet.release_workspace(0)
        episdet.test_fail_allocation(fail)
        for r, a, s in zip(episdet.search_perm(off, n, dl, top_k=k), aligned, same):
            assert r.kernel_launches == s.kernel_launches
            assert r.snps == a.snps and np.array_equal(r.top_snps, a.top_snps)
            assert np.array_equal(r.top_fp32, a.top_fp32) and np.array_equal(r.top_fp64, a.top_fp64)
