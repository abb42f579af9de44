"""Encoders and rescoring beyond one wave: blocks and warps that take a second
fragment, in the launch forms that only large calls take.  Reference: the same
rows from the one-warp kernels, or from calls too small for the form."""
import numpy as np
import pytest
import torch

from rotormap._lib import check, lib, ptr

from test_gpu_encode_paths import fragments, pack

pytestmark = pytest.mark.gpu


def tensor(words):
    return torch.from_numpy(words.view(np.int32)).cuda()


def kernels(call):
    """Names of the kernels that a call launches."""
    from cuda.bindings import driver as drv

    st = torch.cuda.Stream()
    call(st.cuda_stream)
    st.synchronize()
    assert drv.cuStreamBeginCapture(st.cuda_stream, drv.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_RELAXED)[0] == 0
    call(st.cuda_stream)
    err, g = drv.cuStreamEndCapture(st.cuda_stream)
    assert err == 0
    names = []
    for node in drv.cuGraphGetNodes(g, drv.cuGraphGetNodes(g, 0)[2])[1]:
        if drv.cuGraphNodeGetType(node)[1] == drv.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            p = drv.cuGraphKernelNodeGetParams(node)[1]
            err, name = drv.cuFuncGetName(p.func) if int(p.func) else drv.cuKernelGetName(p.kern)
            assert err == 0
            names.append(name.decode())
    assert drv.cuGraphDestroy(g)[0] == 0
    return names


def mixed(seed, n, k):
    """Fragments of which every seventh is a homopolymer or a tandem repeat."""
    codes = np.random.default_rng(seed).integers(0, 4, (n, k)).astype(np.uint8)
    odd = codes[::7]
    odd[:] = fragments(np.random.default_rng(seed + 1), max(6, len(odd)), k)[np.arange(len(odd)) % 6]
    return codes


# tables formed once in the block, with every tile, and read from device memory;
# one block per SM and two (148 or 296 in all); up to 4^6 c-mers
LONG = [(2000, 5, 1, 5, 700), (5000, 5, 1, 5, 700), (6300, 5, 1, 5, 700), (9000, 5, 1, 5, 700), (1500, 8, 4, 4, 700),
        (2200, 8, 4, 4, 700), (3000, 8, 8, 3, 700), (3000, 5, 3, 2, 700), (2600, 7, 1, 6, 200)]
# per-copy norms, which keep more of a fragment to one warp: longer ones
LONG1 = [(5000, 5, 1, 5, 700), (6300, 5, 1, 5, 700), (9000, 5, 1, 5, 700), (3000, 8, 8, 3, 700), (3000, 5, 3, 2, 700)]


@pytest.mark.parametrize("k,s,m,c,n,kind,normalize,ref", [(*x, 3, 0, False) for x in LONG] + [(*x, 1, 0, True) for x in LONG]
                         + [(*x, 0, 1, False) for x in LONG1])
def test_long_blocks_take_several_fragments(k, s, m, c, n, kind, normalize, ref, monkeypatch):
    codes = mixed(k, n, k)
    words = tensor(pack(codes))
    genome = tensor(np.concatenate([pack(codes[:60].reshape(1, -1))[0], np.zeros(4, np.uint32)]))
    pos = torch.arange(n // 2, dtype=torch.int64, device="cuda") * (59 * k // (n // 2))
    dtype = {0: torch.float32, 1: torch.float16, 3: torch.uint8}[kind]
    out = torch.empty((n, 2 * m * 4 ** c), dtype=dtype, device="cuda")
    norms, scales = torch.zeros((n, m), device="cuda"), torch.zeros(n, device="cuda")

    def call(stream):
        sc = ptr(scales) if kind == 3 else None
        if ref:
            check(lib().r2m_encode_ref_windows(ptr(out), kind, ptr(norms), sc, ptr(genome), ptr(pos), n // 2, 100, k, s,
                                               m, c, normalize, stream))
        else:
            check(lib().r2m_encode_frag_real_batch(ptr(out), kind, ptr(norms), sc, ptr(words), n, k, s, m, c, normalize,
                                                   stream))

    res = []
    for path in ("auto", "dense"):
        monkeypatch.setenv("R2M_ENCODER", path)
        assert any("k_encode_long" in name for name in kernels(call)) == (path == "auto")
        res.append([t.clone() for t in (out, norms, scales)])
    for a, b in zip(*res):
        assert torch.equal(a, b)


@pytest.mark.parametrize("k,s,m,c", [(150, 8, 4, 4), (100, 8, 4, 3), (250, 8, 2, 4), (160, 5, 1, 5), (37, 5, 1, 4)])
@pytest.mark.parametrize("nb", [296, 297, 3001])
def test_rescoring_of_many_reads_equals_the_general_kernel(k, s, m, c, nb, monkeypatch):
    """Eight warps a read up to twice the SMs' number, four beyond; blocks that
    take several reads."""
    rng = np.random.default_rng(nb + k)
    kc, topk, N = 5, 3, 500
    genome = mixed(k, 6, 4000).reshape(-1)
    gw = tensor(np.concatenate([pack(genome[None])[0], np.zeros(4, np.uint32)]))
    pos = torch.from_numpy(rng.integers(0, genome.size - k + 1, N).astype(np.int64)).cuda()
    strand = torch.from_numpy(rng.integers(0, 2, N).astype(np.uint8)).cuda()
    reads = tensor(pack(mixed(nb, nb, k)))
    cand = torch.from_numpy(rng.integers(0, N + 1, (nb, kc)).astype(np.int32)).cuda()
    sc, v = torch.empty((nb, kc), device="cuda"), torch.empty((nb, topk), device="cuda")
    l = torch.empty((nb, topk), dtype=torch.int32, device="cuda")

    def call(stream):
        check(lib().r2m_rescore_fp32(ptr(reads), nb, ptr(cand), kc, ptr(gw), ptr(pos), ptr(strand), N, k, s, m, c, 0,
                                     ptr(sc), ptr(v), ptr(l), topk, stream))

    res = []
    for path in ("auto", "dense"):
        monkeypatch.setenv("R2M_ENCODER", path)
        assert any("k_rescore_dense" in name for name in kernels(call)) == (path == "auto")
        res.append([t.clone() for t in (sc, v, l)])
    for a, b in zip(*res):
        assert torch.equal(a, b)


@pytest.mark.parametrize("k,s,m,c", [(150, 8, 4, 4), (250, 8, 4, 4), (60, 8, 4, 3), (150, 5, 1, 5)])
@pytest.mark.parametrize("kind", [2, 3])
@pytest.mark.parametrize("ref", [False, True])
def test_reads_in_large_calls_equal_small_ones(k, s, m, c, kind, ref):
    """One-byte rows at m = 4 come from blocks of up to 18 warps, two per SM,
    each warp several fragments; calls of at most 8 a SM have blocks of 8."""
    n = 14_001
    codes = mixed(k, n, k)
    words = tensor(pack(codes))
    genome = tensor(np.concatenate([pack(codes[:2000].reshape(1, -1))[0], np.zeros(4, np.uint32)]))
    pos = torch.arange(n, dtype=torch.int64, device="cuda") * 7  # within 2,000 fragments
    rows, rdim = (2 if ref else 1) * n, 2 * m * 4 ** c
    st = torch.cuda.current_stream().cuda_stream

    def run(step):
        out = torch.empty((rows, rdim), dtype=torch.uint8, device="cuda")
        norms, scales = torch.zeros((rows, m), device="cuda"), torch.zeros(rows, device="cuda")
        for lo in range(0, n, step):
            nb, at = min(step, n - lo), (2 if ref else 1) * lo
            args = (ptr(out[at:]), kind, ptr(norms[at:]), ptr(scales[at:]) if kind == 3 else None)
            if ref:
                check(lib().r2m_encode_ref_windows(*args, ptr(genome), ptr(pos[lo:]), nb, 1000, k, s, m, c, 0, st))
            else:
                check(lib().r2m_encode_frag_real_batch(*args, ptr(words[lo:]), nb, k, s, m, c, 0, st))
        torch.cuda.synchronize()
        return out, norms, scales

    for a, b in zip(run(n), run(1000)):
        assert torch.equal(a, b)
