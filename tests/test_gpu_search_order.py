"""The fused search's candidate buffers and reservoir at their edges: score
orders in which every column is a candidate (rising), only the first k are
(falling), ties fill the list (flat), or bursts of candidates overflow a
lane's buffer (saw), for rows that differ, at tile edges and every reservoir
size.  Scores are small integers times powers of two, exact in every score
form and summation order, so values and locations must equal a stable sort."""
import numpy as np
import pytest
import torch

import rotormap as rm

pytestmark = pytest.mark.gpu

RDIM = 256
ONE = 0x38  # e4m3 1.0


def levels(order, N):
    j = np.arange(N)
    return {"rising": 1 + j * (RDIM - 1) // N, "falling": RDIM - j * (RDIM - 1) // N, "flat": np.full(N, 7),
            "saw": 1 + (j * 37 % 113) + (j // 113) % 100}[order]


def check(order, nb, N, splits, k, score):
    lv = levels(order, N)
    B = (np.arange(RDIM)[None, :] < lv[:, None]).astype(np.uint8) * ONE
    # row r sees the first RDIM - r % 97 levels: equal scores beyond, other thresholds
    width = RDIM - np.arange(nb) % 97
    A = (np.arange(RDIM)[None, :] < width[:, None]).astype(np.uint8) * ONE
    want = np.minimum(lv[None, :], width[:, None]).astype(np.float32)
    sb = sa = None
    if score == "scaled":
        sb = np.exp2(np.arange(N) % 3).astype(np.float32)
        sa = np.exp2(-(np.arange(nb) % 4)).astype(np.float32)
        want = want * sb[None, :]
    loc = np.argsort(-want, axis=1, kind="stable")[:, :k]
    val = np.take_along_axis(want, loc, 1)
    if sa is not None:
        val = val * sa[:, None]
    d = lambda x: None if x is None else torch.from_numpy(x).cuda()  # noqa: E731
    for epilogue in ("auto", "4"):
        eng = rm.TopKEngine(d(B), k=k, rows_cap=nb, score=score, scaleB=d(sb), splits=splits, epilogue=epilogue)
        v, l = eng.search(d(A), nb, d(sa))
        torch.cuda.synchronize()
        assert np.array_equal(l.cpu().numpy(), loc + 1)
        assert np.array_equal(v.cpu().numpy(), val)
        eng.close()


@pytest.mark.parametrize("order", ["rising", "falling", "flat", "saw"])
@pytest.mark.parametrize("nb,N,splits", [(1, 64, 0), (37, 511, 1), (128, 2305, 0), (129, 2305, 2), (300, 4097, 3)])
@pytest.mark.parametrize("k,score", [(1, "f32"), (5, "f16"), (16, "scaled"), (20, "f16"), (32, "scaled"), (64, "f32")])
def test_every_candidate_order(order, nb, N, splits, k, score):
    check(order, nb, N, splits, k, score)


# sizes at which units are one or two tiles: 64, 128, 192 and 256 columns wide
@pytest.mark.parametrize("order", ["rising", "saw"])
@pytest.mark.parametrize("nb", [1, 16, 128, 129, 256, 1000])
@pytest.mark.parametrize("N", [65, 1000, 4736, 9473, 14209, 20000])
@pytest.mark.parametrize("k,score", [(20, "scaled"), (64, "f16")])
def test_few_columns_per_unit(order, nb, N, k, score):
    check(order, nb, N, 0, k, score)
