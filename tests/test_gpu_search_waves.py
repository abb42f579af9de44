"""Row bounds carried from one wave of units to the next, on the adversarial
score orders: few CTAs, so that every read tile runs several column splits one
after another, and splits that do not divide the CTAs."""
import numpy as np
import pytest
import torch

import rotormap as rm
from test_gpu_search_order import ONE, RDIM, levels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["rising", "falling", "flat", "saw"])
@pytest.mark.parametrize("nb,kernel", [(37, "1sm"), (300, "2sm")])
@pytest.mark.parametrize("ctas,splits", [(2, 7), (4, 7), (6, 12), (4, 12)])
@pytest.mark.parametrize("k,score", [(5, "f16"), (20, "scaled"), (64, "f32")])
def test_every_candidate_order_over_several_waves(order, nb, kernel, ctas, splits, k, score):
    N = 12 * 256 + 77
    lv = levels(order, N)
    width = RDIM - np.arange(nb) % 97
    B = (np.arange(RDIM)[None, :] < lv[:, None]).astype(np.uint8) * ONE
    A = (np.arange(RDIM)[None, :] < width[:, None]).astype(np.uint8) * ONE
    want = np.minimum(lv[None, :], width[:, None]).astype(np.float32)
    sb, sa = np.exp2(np.arange(N) % 3).astype(np.float32), np.exp2(-(np.arange(nb) % 4)).astype(np.float32)
    if score == "scaled":
        want = want * sb[None, :]
    loc = np.argsort(-want, axis=1, kind="stable")[:, :k]
    val = np.take_along_axis(want, loc, 1) * (sa[:, None] if score == "scaled" else 1)
    dA, dB, dsa, dsb = (torch.from_numpy(x).cuda() for x in (A, B, sa, sb))
    scaled = score == "scaled"
    for epilogue in ("auto", "4"):
        eng = rm.TopKEngine(dB, k=k, rows_cap=nb, score=score, scaleB=dsb if scaled else None, splits=splits, ctas=ctas,
                            kernel=kernel, epilogue=epilogue)
        for _ in range(2):  # the second search on the state that the first left
            v, l = eng.search(dA, nb, dsa if scaled else None)
            assert np.array_equal(l.cpu().numpy(), loc + 1)
            assert np.array_equal(v.cpu().numpy(), val)
        eng.close()
