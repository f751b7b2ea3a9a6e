"""TAA resolve at image sizes around the kernel's tiles (32 x 8) and its prefetch distance, with motion
past the image's edges and infinite motion: bit-exact against the CPU oracle, first frame, history
and in-place output."""
import numpy as np
import pytest

import oracle as O
import snkpt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (1, 300), (2, 2), (31, 7), (32, 8), (33, 9), (64, 16), (4000, 3), (320, 400),
                                 (1283, 721)])
def test_sizes_match_oracle(cuda, built_lib, w, h):
    import torch
    rng = np.random.default_rng(w * 10000 + h)
    t, ot = snkpt.TaaResolve(w, h), O.OracleTaa(w, h)
    for k in range(3):
        r = rng.lognormal(-0.5, 1.2, (h * w, 4)).astype(np.float32)
        r[rng.uniform(size=(h * w, 4)) < 0.05] *= -1.0
        r[:, 3] = 1.0
        mv = rng.normal(0.0, 0.01, (h * w, 2)).astype(np.float32)
        mv[rng.uniform(size=h * w) < 0.1] *= 200.0
        mv[:: max(1, h * w // 7)] = [np.inf, -np.inf]
        rt, mt = torch.from_numpy(r).cuda(), torch.from_numpy(mv).cuda()
        out = t.resolve(rt, mt, out=rt if k == 1 else None)
        torch.cuda.synchronize()
        ref = ot.resolve(r, mv)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), ref.view(np.uint32)), k
