"""The longest-first order at the sizes where its sort changes: every instance is taken once, whatever the order, in the
first sweep (ordered by horizon) and in later ones (by the previous sweep's counts, reused by the backward)."""
import numpy as np
import pytest
import torch

from vectorizedadjoint_gb300 import Solver

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.tensor(np.array(a, order="C"), dtype=torch.float64, device="cuda")


@pytest.mark.parametrize("precision", ["fp64", "mixed_dw"])
@pytest.mark.parametrize("B", [1, 31, 1023, 1025, 4095, 4096, 4097, 9000])
def test_every_instance_once(cuda, precision, B):
    rng = np.random.default_rng(B)
    y0, p, t1 = rng.uniform(-2, 2, (B, 2)), 10 ** rng.uniform(-1, 0.5, (B, 1)), rng.uniform(0.0, 3.0, B)
    if B > 1:
        t1[B // 2] = 0.0
    got = []
    for flip in (slice(None), slice(None, None, -1)):
        s = Solver("vdp", 2, 1, B, precision=precision)
        for _ in range(3):
            r = s.gradient("sumsq", dev(y0[flip]), dev(p[flip]), dev(np.zeros(B)), dev(t1[flip]))
            got.append({k: v.cpu().numpy()[flip].copy() for k, v in r.items()})
            for v in r.values():  # a result left from the call before would be seen
                v.zero_()
        s.close()
    assert (got[0]["status"] == 0).all() and (got[0]["n_acc"] > 0).sum() == B - (B > 1)
    for g in got[1:]:
        for k in ("yT", "dy0", "dp", "n_acc", "status"):
            np.testing.assert_array_equal(g[k], got[0][k], err_msg=k)
