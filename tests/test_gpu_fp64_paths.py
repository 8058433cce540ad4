"""The FP64 sweeps chosen by fp64_path against the oracle, bit for bit, where
they can go wrong: batches around the sizes at which the path changes, and
states and parameters that the integer products do not take (beyond
2^+-240, infinities) or take specially (zeros of both signs)."""
import numpy as np
import pytest
import torch

from vectorizedadjoint_gb300 import Solver

pytestmark = pytest.mark.gpu

NP = {"vdp": 1, "vdp_petsc": 1, "dho": 2, "decay": 1}


def dev(a):
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def draw(model, B, seed):
    rng = np.random.default_rng(seed)
    n = 1 if model == "decay" else 2
    p = {"vdp": 10 ** rng.uniform(-1, 1, (B, 1)), "vdp_petsc": 10 ** rng.uniform(-1, 0.5, (B, 1)),
         "dho": np.stack([rng.uniform(0.5, 5, B), rng.uniform(0, 0.5, B)], 1),
         "decay": rng.uniform(0.1, 3, (B, 1))}[model]
    return rng.uniform(-2, 2, (B, n)), p, rng.uniform(0.5, 3.0, B)


def check(oracle, model, tab, y0, p, t1, picks, stride=0, tol=1e-6):
    B, n = y0.shape
    s = Solver(model, n, NP[model], B, tableau=tab, precision="fp64", atol=tol, rtol=tol, ckpt_stride=stride)
    out = s.gradient("sumsq", dev(y0), dev(p), dev(np.zeros(B)), dev(t1))
    torch.cuda.synchronize()
    r = {k: v.cpu().numpy() for k, v in out.items()}
    s.close()
    pb = oracle.problem(model, tab, n, NP[model], tol, tol)
    for b in picks:
        g = oracle.gradient(pb, "sumsq", y0[b], p[b], 0.0, t1[b])
        assert int(r["status"][b]) == g["status"], b
        if g["status"] != 0:
            continue
        assert int(r["n_acc"][b]) == g["n_acc"], b
        for k in ("yT", "dy0", "dp"):
            np.testing.assert_array_equal(r[k][b], g[k], err_msg=f"{k} {b}")


@pytest.mark.parametrize("model", sorted(NP))
@pytest.mark.parametrize("tab", ["dopri5", "ck54", "rkf78"])
@pytest.mark.parametrize("B", [1, 33, 1217, 5000])
def test_paths_bit_exact(oracle, cuda, model, tab, B):
    y0, p, t1 = draw(model, B, B)
    check(oracle, model, tab, y0, p, t1, sorted({0, B // 2, B - 1, min(31, B - 1), min(1216, B - 1)}))


@pytest.mark.parametrize("tab,stride", [("dopri5", 0), ("ck54", 0), ("rkf78", 0), ("dopri5", 3)])
@pytest.mark.parametrize("B", [7, 6000])
def test_special_values_bit_exact(oracle, cuda, tab, stride, B):
    """Linear oscillators: zeros, both signs, no damping, no frequency, and magnitudes across and beyond the range of the
    integer products (the other instances of the same warp stay on it)."""
    y0, p, t1 = draw("dho", B, 5)
    special = [(0.0, 1.0), (-0.0, 1.0), (1.0, -0.0), (0.0, 0.0), (1e-70, 1e-75), (1e-90, 1.0), (1e74, -1e70),
               (3e150, 1.0), (1e-310, 1e-300), (np.inf, 1.0), (np.nan, 0.0)]
    for k, v in enumerate(special[:B]):
        y0[k] = v
    if B > 40:
        p[20] = (2.0, 0.0)
        p[21] = (0.0, 0.3)
        p[22] = (1e-80, 0.1)
        p[23], t1[23] = (1e3, 0.0), 0.05
    check(oracle, "dho", tab, y0, p, t1, range(min(B, 40)), stride)
