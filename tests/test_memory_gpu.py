"""3-way searches with little device memory.

A launch takes up to 64 first SNPs where their regrouped rows fit; with little
memory left it takes 4, and the search neither fails nor holds its pair table
in blocks for the sake of larger launches.
"""
import pytest

from test_parity_gpu import assert_same

pytestmark = pytest.mark.gpu


@pytest.fixture
def fresh(episdet):
    import torch

    torch.cuda.empty_cache()
    episdet.release_workspace(0)  # the next search allocates its buffers again
    yield
    episdet.test_fail_allocation(0)
    episdet.release_workspace(0)
    torch.cuda.empty_cache()


@pytest.mark.parametrize("after", range(11, 20))
def test_a_failed_buffer_of_a_search_means_smaller_launches(episdet, oracle, fresh, after):
    """Allocations 11 to 19 are the operand, regrouping and pair-table buffers
    (8 of the first 10 are the planes, counts and score tables)."""
    M, nc, nn, k = 50, 2000, 2200, 64
    cases, controls = episdet.generate(0xA10D, M, nc, nn)
    o = oracle.search(cases, controls, nc, nn, order=3, score="k2", top_k=k)
    episdet.test_fail_allocation(after)
    r = episdet.search(cases, controls, nc, nn, order=3, top_k=k, engine="tensor")
    assert_same(r, o, k)
    assert r.count_kernel_launches == 12  # 48 first SNPs, 4 a launch
    r = episdet.search(cases, controls, nc, nn, order=3, top_k=k, engine="tensor")
    assert_same(r, o, k)
    assert r.count_kernel_launches == 1


def test_little_free_memory(episdet, oracle, fresh):
    """1500 SNPs x 40000 samples with 8 GB free: launches of 34 first SNPs would
    take 4.3 GB; the whole pair table is 72 MB."""
    import torch

    M, nc, nn, k = 1500, 20000, 20000, 64
    cases, controls = episdet.generate(0x8B, M, nc, nn)
    o = oracle.search(cases, controls, nc, nn, order=3, score="k2", top_k=k, first_begin=0, first_end=8)
    episdet.search(cases, controls, nc, nn, order=2, top_k=k)  # the context and the kernels are loaded
    episdet.release_workspace(0)
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (8 << 30), dtype=torch.uint8, device="cuda")
    try:
        r = episdet.search(cases, controls, nc, nn, order=3, top_k=k, engine="tensor", first_begin=0, first_end=8)
    finally:
        del hold
    assert_same(r, o, k)
    assert r.count_kernel_launches == 2  # 4 first SNPs a launch, one pass over them


def test_limited_launches_stay_as_they_are(episdet, oracle, fresh):
    """With 12 GB free the launches take a few first SNPs more than the smallest;
    repeated searches take the same and no more memory, and a later one with room
    takes all."""
    import torch

    M, nc, nn, k = 1500, 20000, 20000, 64
    data = episdet.generate(0x8E, M, nc, nn)
    kw = dict(order=3, top_k=k, engine="tensor", first_begin=0, first_end=32)
    episdet.search(*data, nc, nn, order=2, top_k=k)
    episdet.release_workspace(0)
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (12 << 30), dtype=torch.uint8, device="cuda")
    try:
        seen = []
        for _ in range(3):
            r = episdet.search(*data, nc, nn, **kw)
            seen.append((r.count_kernel_launches, torch.cuda.mem_get_info()[0]))
    finally:
        del hold
    assert 1 < seen[0][0] < 8 and seen == seen[:1] * 3
    torch.cuda.empty_cache()
    for _ in range(70):
        r = episdet.search(*data, nc, nn, **dict(kw, first_end=8))
    assert r.count_kernel_launches == 1
    assert_same(r, oracle.search(*data, nc, nn, order=3, score="k2", top_k=k, first_begin=0, first_end=8), k)


def test_room_held_by_larger_launches_is_given_back(episdet, oracle, fresh):
    """After a search whose launches hold 4 GB, one whose pair table (2.9 GB) does
    not fit beside them: they go, not the whole table."""
    import torch

    first = episdet.generate(0x8C, 1500, 20000, 20000)
    M, nc, nn, k = 9500, 500, 500, 64
    cases, controls = episdet.generate(0x8D, M, nc, nn)
    o = oracle.search(cases, controls, nc, nn, order=3, score="k2", top_k=k, first_begin=0, first_end=2)
    episdet.search(*first, 20000, 20000, order=3, top_k=k, engine="tensor", first_begin=0, first_end=2)
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (6 << 30), dtype=torch.uint8, device="cuda")
    try:
        r = episdet.search(cases, controls, nc, nn, order=3, top_k=k, engine="tensor", first_begin=0, first_end=2)
    finally:
        del hold
    assert_same(r, o, k)
    assert r.count_kernel_launches == 1
