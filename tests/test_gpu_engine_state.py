"""The state an engine keeps between searches (row bounds and pacing slots,
zero before each): no search reads anything else there, whichever stream it
comes on and whatever memory the engine was given."""
import numpy as np
import pytest
import torch

import rotormap as rm

pytestmark = pytest.mark.gpu

E4M3_INT = np.array([0xC4, 0xC0, 0xB8, 0x00, 0x38, 0x40, 0x44], np.uint8)  # -3..3
VALUES = np.arange(-3, 4).astype(np.float32)


def integers(seed, rows, rdim=256):
    """Rows of small integers as e4m3 bytes on the GPU, and their values: every
    score is a whole number below 2^24, exact in any order of summation."""
    at = np.random.default_rng(seed).integers(0, 7, size=(rows, rdim))
    return torch.from_numpy(E4M3_INT[at]).cuda(), VALUES[at]


def top(a, b, k):
    """Top k columns (value descending, equal values by column), 1-based."""
    sc = a @ b.T
    loc = np.argsort(-sc, axis=1, kind="stable")[:, :k]
    return np.take_along_axis(sc, loc, 1), (loc + 1).astype(np.int32)


@pytest.mark.parametrize("nb,kernel", [(100, "1sm"), (300, "2sm")])
def test_new_engine_searches_at_once_on_any_stream(nb, kernel):
    """Engines made on recycled memory while the default stream is busy, each
    searched at once on a stream that does not wait for the default one."""
    A, a = integers(1, nb)
    B, b = integers(2, 9000)
    wv, wl = top(a, b, 20)
    v = torch.empty((nb, 20), device="cuda")
    l = torch.empty((nb, 20), dtype=torch.int32, device="cuda")
    side = torch.cuda.Stream()
    for byte in (0xFF, 0xC0, 0x00, 0x7F, 0x45, 0xC0):
        # bytes that read as row bounds (large values, NaN) in memory just given back
        junk = torch.full((256 << 20,), byte, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        del junk
        torch.cuda.empty_cache()
        torch.cuda._sleep(40_000_000)
        eng = rm.TopKEngine(B, k=20, rows_cap=nb, score="f32", kernel=kernel)
        eng.search(A, nb, None, v, l, side)
        side.synchronize()
        assert np.array_equal(v.cpu().numpy(), wv)
        assert np.array_equal(l.cpu().numpy(), wl)
        eng.close()


def captured(eng, A, v, l, ruin=False):
    """Node types of a search captured on a stream of its own (ruin: the
    capture is made invalid first, so the search's launch fails)."""
    from cuda.bindings import driver as drv

    st = torch.cuda.Stream()
    assert drv.cuStreamBeginCapture(st.cuda_stream, drv.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_RELAXED)[0] == 0
    if ruin:
        assert drv.cuStreamSynchronize(st.cuda_stream)[0] != 0  # refused, and it ends the capture
    try:
        eng.search(A, A.shape[0], None, v, l, st)
    finally:
        err, g = drv.cuStreamEndCapture(st.cuda_stream)
    assert err == 0
    n = drv.cuGraphGetNodes(g, 0)[2]
    kinds = [drv.cuGraphNodeGetType(x)[1].name.split("_TYPE_")[1] for x in drv.cuGraphGetNodes(g, n)[1][:n]]
    assert drv.cuGraphDestroy(g)[0] == 0
    return sorted(kinds)


@pytest.mark.parametrize("nb,kernel", [(100, "1sm"), (300, "2sm")])
def test_a_captured_clear_does_not_stand_for_one_that_ran(nb, kernel):
    """After a launch that failed, and could not be cleaned up after, every
    search clears the state until a clear has run: those that are captured as
    well, one after another, since none of them has run yet."""
    A, a = integers(3, nb)
    B, b = integers(4, 5000)
    wv, wl = top(a, b, 20)
    eng = rm.TopKEngine(B, k=20, rows_cap=nb, score="f32", kernel=kernel)
    v = torch.empty((nb, 20), device="cuda")
    l = torch.empty((nb, 20), dtype=torch.int32, device="cuda")

    def search():
        eng.search(A, nb, None, v, l)
        assert np.array_equal(v.cpu().numpy(), wv) and np.array_equal(l.cpu().numpy(), wl)

    search()
    assert captured(eng, A, v, l) == ["KERNEL", "KERNEL"]
    with pytest.raises(rm.R2MError):
        captured(eng, A, v, l, ruin=True)
    for _ in range(2):
        assert captured(eng, A, v, l) == ["KERNEL", "KERNEL", "MEMSET"]
    search()
    assert captured(eng, A, v, l) == ["KERNEL", "KERNEL"]
    search()
    eng.close()


@pytest.mark.parametrize("k,kt", [(5, 8), (20, 20), (64, 64)])
def test_workspace_bytes_are_all_that_the_engine_allocates(k, kt):
    """1,024 pacing slots of 8 bytes, and for each partial list a 4-byte row
    bound and kt values and columns; the allocator hands out whole 2 MiB pages."""
    B, _ = integers(5, 70_000)
    torch.cuda.synchronize()
    a8 = rm.TopKEngine(B, k=k, rows_cap=4000)  # torch's pool holds the staging buffer from here on
    a8.close()
    del a8
    free = torch.cuda.mem_get_info()[0]
    eng = rm.TopKEngine(B, k=k, rows_cap=4000)
    held = eng.workspace_bytes
    assert (held - 8192) % (8 * kt + 4) == 0
    assert held <= free - torch.cuda.mem_get_info()[0] <= held + (4 << 20)
    eng.set_tuning(splits=1)  # a schedule that needs less keeps what there is
    assert eng.workspace_bytes == held
    eng.set_tuning(splits=64)
    assert eng.workspace_bytes > held and (eng.workspace_bytes - 8192) % (8 * kt + 4) == 0
    eng.close()
