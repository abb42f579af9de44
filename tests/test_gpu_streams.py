"""Streams that the library makes for itself wait for what was queued before:
an engine's buffers are filled on the stream that was current then."""
import numpy as np
import pytest
import torch

import rotormap as rm
from conftest import random_words
from rotormap import serving
from rotormap.batching import RaggedBatcher

pytestmark = pytest.mark.gpu

K = 60


def setup(score="scaled"):
    re = rm.RopeEncoder(k=K, s=8, m=4, c=3)
    rng = np.random.default_rng(6)
    B = rm.encode_frag_real_batch_alloc(torch.uint8, re, torch.from_numpy(
        random_words(rng, 5000, K).reshape(-1).view(np.int32)).cuda(), scaled=True)
    words = random_words(rng, 256, K)
    a8, _, sa = rm.encode_frag_real_batch_alloc(torch.uint8, re, torch.from_numpy(
        words.reshape(-1).view(np.int32)).cuda(), scaled=True)
    eng = rm.TopKEngine(B[0], k=20, rows_cap=256, score=score, scaleB=B[2])
    v, l = eng.search(a8, 256, sa)
    torch.cuda.synchronize()
    want = v.cpu().numpy(), l.cpu().numpy()
    eng.close()
    return re, B, words, want


def engine(B):
    torch.cuda._sleep(200_000_000)  # the default stream is busy for a tenth of a second
    return rm.TopKEngine(B[0], k=20, rows_cap=256, score="scaled", scaleB=B[2])


def waits(stream):
    idle = stream.query()
    return not (idle and not torch.cuda.current_stream().query())


def test_mapper():
    re, B, words, want = setup()
    m = rm.Mapper(engine(B), re)
    assert waits(m.stream)
    for a, b in zip(m.map_words(words), want):
        assert np.array_equal(a, b)


def test_ragged_batcher():
    re, B, words, want = setup()
    r = RaggedBatcher(engine(B), re, 256)
    assert waits(r.stream)
    got = r.run([words[:100], words[100:]])
    for i in (0, 1):
        assert np.array_equal(np.concatenate([g[i] for g in got]), want[i])


def test_plain_map():
    re, B, words, want = setup()
    (_, v, l), = serving.plain_map(engine(B), re, [(0.0, words)], batch=256)
    assert np.array_equal(v, want[0]) and np.array_equal(l, want[1])


def test_server():
    re, B, words, want = setup()
    eng = engine(B)
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)
    srv = serving.MappingServer(eng, re)
    for h in [srv.submit(words) for _ in range(4)]:
        for a, b in zip(h.result(timeout=60), want):
            assert np.array_equal(a, b)
    srv.close()
