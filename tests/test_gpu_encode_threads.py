"""Encoders called from several threads with other sizes at a time: no call
changes what another one's launch may use."""
import threading

import numpy as np
import pytest
import torch

from rotormap._lib import check, lib, ptr

from test_gpu_encode_paths import fragments, pack

pytestmark = pytest.mark.gpu

# shared memory of a block from a few KiB to the most there is
SIZES = [(40, 4, 1, 1), (150, 8, 8, 4), (60, 4, 1, 1), (300, 8, 4, 4)]


def state(k, s, m, c, n=8):
    """An encode, an index encode and a rescoring of one size, and the bytes
    that each leaves when it runs alone."""
    rng = np.random.default_rng(k)
    codes = fragments(rng, n, k)
    words = torch.from_numpy(pack(codes).view(np.int32)).cuda()
    genome = torch.from_numpy(np.concatenate([pack(codes.reshape(1, -1))[0], np.zeros(4, np.uint32)]).view(np.int32)).cuda()
    pos = k * torch.arange(n, dtype=torch.int64, device="cuda")
    strand = torch.zeros(n, dtype=torch.uint8, device="cuda")
    cand = torch.from_numpy(rng.integers(1, n + 1, (n, 4)).astype(np.int32)).cuda()
    rows, cols = (torch.empty((i * n, 2 * m * 4 ** c), device="cuda") for i in (1, 2))
    norms, norms2 = torch.empty((n, m), device="cuda"), torch.empty((2 * n, m), device="cuda")
    sc, v = torch.empty((n, 4), device="cuda"), torch.empty((n, 4), device="cuda")
    l = torch.empty((n, 4), dtype=torch.int32, device="cuda")

    def run(stream):
        check(lib().r2m_encode_frag_real_batch(ptr(rows), 0, ptr(norms), None, ptr(words), n, k, s, m, c, 0, stream))
        check(lib().r2m_encode_ref_windows(ptr(cols), 0, ptr(norms2), None, ptr(genome), ptr(pos), n, n, k, s, m, c, 0,
                                           stream))
        check(lib().r2m_rescore_fp32(ptr(words), n, ptr(cand), 4, ptr(genome), ptr(pos), ptr(strand), n, k, s, m, c, 0,
                                     ptr(sc), ptr(v), ptr(l), 4, stream))

    run(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    outs = (rows, cols, norms, norms2, sc, v, l)
    return run, outs, [t.clone() for t in outs]


def test_sizes_in_other_threads_do_not_refuse_a_launch(monkeypatch):
    monkeypatch.setenv("R2M_ENCODER", "dense")  # the kernels whose shared memory grows with the fragment
    states = [state(*size) for size in SIZES]
    errors = []

    def work(run):
        stream = torch.cuda.Stream()
        try:
            for _ in range(1000):
                run(stream.cuda_stream)
        except Exception as e:  # noqa: BLE001
            errors.append(repr(e))
        stream.synchronize()

    threads = [threading.Thread(target=work, args=(run,)) for run, _, _ in states]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for _, outs, want in states:
        for a, b in zip(outs, want):
            assert torch.equal(a, b)
