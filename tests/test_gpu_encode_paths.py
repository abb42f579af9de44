"""The encoder's dispatch: the register path of the FP32 rescoring and the bulk
e4m3 conversion give the bytes of the general path they stand in for, at the
edges of their tiles and on fragments whose windows crowd into few bins."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc

import rotormap as rm
from rotormap._lib import check, lib, ptr

pytestmark = pytest.mark.gpu

def fragments(rng, n, k):
    """Random fragments, homopolymers and short tandem repeats, as codes."""
    codes = rng.integers(0, 4, size=(n, k)).astype(np.uint8)
    codes[0] = 0
    codes[1] = 2
    for i, period in ((2, 2), (3, 7), (4, 33)):
        codes[i] = np.resize(codes[i, :period], k)
    codes[5, k // 2:] = 3
    return codes


def pack(codes):
    n, k = codes.shape
    full = np.zeros((n, (k + 15) // 16 * 16), np.uint32)
    full[:, :k] = codes
    return (full.reshape(n, -1, 16) << (2 * np.arange(16, dtype=np.uint32))).sum(2, dtype=np.uint32)


@pytest.mark.parametrize("k,s,m,c", [(150, 8, 4, 4), (100, 8, 4, 3), (250, 8, 2, 4), (160, 5, 1, 5), (37, 5, 1, 4)])
@pytest.mark.parametrize("nb,kc,topk", [(1, 64, 20), (7, 5, 5), (40, 33, 1)])
def test_rescoring_equals_the_general_kernel(k, s, m, c, nb, kc, topk, monkeypatch):
    rng = np.random.default_rng(k + nb)
    genome = fragments(rng, 6, 4000).reshape(-1)
    gw = np.concatenate([pack(genome[None])[0], np.zeros(4, np.uint32)])
    N = 500
    pos = rng.integers(0, genome.size - k + 1, N).astype(np.int64)
    strand = rng.integers(0, 2, N).astype(np.uint8)
    reads = fragments(rng, max(nb, 6), k)[-nb:]
    cand = rng.integers(-1, N + 2, size=(nb, kc)).astype(np.int32)  # ids outside 1..N score -inf
    cand[0, :2] = 3  # the same candidate twice
    d = [torch.from_numpy(x).cuda() for x in (pack(reads).view(np.int32), cand, gw.view(np.int32), pos, strand)]
    res = []
    for path in ("auto", "dense"):
        monkeypatch.setenv("R2M_ENCODER", path)
        sc = torch.empty((nb, kc), device="cuda")
        v, l = torch.empty((nb, topk), device="cuda"), torch.empty((nb, topk), dtype=torch.int32, device="cuda")
        check(lib().r2m_rescore_fp32(ptr(d[0]), nb, ptr(d[1]), kc, ptr(d[2]), ptr(d[3]), ptr(d[4]), N, k, s, m, c, 0,
                                     ptr(sc), ptr(v), ptr(l), topk, torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        res.append([t.cpu().numpy() for t in (sc, v, l)])
    for a, b in zip(*res):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("src0,dst0", [(0, 0), (8, 16), (1, 0), (0, 3), (5, 7)])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 4095, 4113, 70_001])
def test_bulk_e4m3_at_every_alignment(dtype, src0, dst0, n):
    rng = np.random.default_rng(n)
    x = (rng.standard_normal(n) * np.exp2(rng.integers(-12, 12, n))).astype(np.float32)
    x[rng.integers(0, n, n // 9)] = np.inf
    x[rng.integers(0, n, n // 9)] = -np.inf
    x[rng.integers(0, n, n // 9)] = np.nan
    src = torch.zeros(src0 + n + 1, dtype=dtype, device="cuda")
    src[src0:src0 + n] = torch.from_numpy(x).cuda().to(dtype)
    dst = torch.full((dst0 + n + 1,), 0x55, dtype=torch.uint8, device="cuda")
    (rm.f16_to_f8 if dtype == torch.float16 else rm.f32_to_f8)(dst[dst0:dst0 + n], src[src0:src0 + n])
    got = dst.cpu().numpy()
    vals = src[src0:src0 + n].float().cpu().numpy()
    assert np.array_equal(got[dst0:dst0 + n], orc.f32_to_e4m3(vals))
    assert np.all(got[:dst0] == 0x55) and got[-1] == 0x55
