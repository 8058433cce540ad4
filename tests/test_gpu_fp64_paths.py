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
@pytest.mark.parametrize("B", [1, 33, 2007, 5000, 9800])
def test_paths_bit_exact(oracle, cuda, model, tab, B):
    y0, p, t1 = draw(model, B, B)
    check(oracle, model, tab, y0, p, t1, sorted({0, B // 2, B - 1, min(31, B - 1), min(1216, B - 1)}))


@pytest.mark.parametrize("tab,stride", [("dopri5", 0), ("ck54", 0), ("rkf78", 0), ("dopri5", 3)])
@pytest.mark.parametrize("B", [7, 1300, 3000, 6000, 10000])
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
    check(oracle, "dho", tab, y0, p, t1, range(min(B, 26)), stride)


@pytest.mark.parametrize("tab", ["dopri5", "rkf78"])
@pytest.mark.parametrize("stride", [0, 5])
@pytest.mark.parametrize("B", [3, 1300])
def test_team_seeds_history_and_refill(oracle, cuda, tab, stride, B):
    """Teams with several seeds, direct parameter gradients, the adjoint history, and fewer resident teams than instances
    (64-thread blocks, one per SM for a batch of more): the bits of single-seed calls on a batch that every lane path
    takes, and of the one-lane sweeps (a block size that teams do not take)."""
    y0, p, t1 = draw("vdp", B, 9)
    rng = np.random.default_rng(3)
    lam, mud = rng.standard_normal((B, 2, 2)), rng.standard_normal((B, 2, 1))
    res = []
    for block, bps in ((0, 0), (64, 1), (48, 0)):
        s = Solver("vdp", 2, 1, B, nout=2, tableau=tab, atol=1e-6, rtol=1e-6, ckpt_stride=stride, block_size=block,
                   blocks_per_sm=bps)
        s.set_adjoint_history(4)
        f = s.forward(dev(y0), dev(p), dev(np.zeros(B)), dev(t1))
        g = s.backward(dev(p), dev(lam), dev(mud))
        hist = s.adjoint_history(B - 1, times=False)[1]
        res.append([v.cpu().numpy() for v in (f["yT"], f["n_acc"], f["n_rej"], g["status"], g["dy0"], g["dp"])] + [hist])
        s.close()
    for r in res[:2]:
        for a, b in zip(r, res[2]):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("tab,stride", [("ck54", 0), ("rkf78", 0), ("dopri5", 7)])
@pytest.mark.parametrize("even", [True, False])
@pytest.mark.parametrize("B", [2100, 4100, 7200, 15000])
def test_choice_by_load(oracle, cuda, tab, stride, even, B):
    """Batches whose load, the sum of lengths over the longest, falls in the range of every team and of one lane (even
    lengths: near B; uneven: a few long instances), first by horizons, then by step counts: the one-lane bits."""
    y0, p, _ = draw("dho", B, B)
    t1 = np.full(B, 1.0)
    if even:
        p[:] = (2.0, 0.1)
    else:
        t1[::97] = 20.0
    res = []
    for block in (0, 48):
        s = Solver("dho", 2, 2, B, tableau=tab, atol=1e-6, rtol=1e-6, ckpt_stride=stride, block_size=block)
        for _ in range(2):
            out = s.gradient("sumsq", dev(y0), dev(p), dev(np.zeros(B)), dev(t1))
            torch.cuda.synchronize()
            res.append([out[k].cpu().numpy() for k in ("yT", "dy0", "dp", "n_acc", "status")])
        s.close()
    assert (res[0][4] == 0).all()
    for r in res[1:]:
        for a, b in zip(r, res[0]):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("N,B", [(5, 7), (5, 7400), (10, 7), (10, 300)])
@pytest.mark.parametrize("tab", ["dopri5", "ck54"])
def test_lotka_volterra_special_values_bit_exact(oracle, cuda, N, B, tab):
    """Lane groups with integer products (N = 10 forward always, N = 5 where the batch fills two warps per quadrant): zero
    and huge entries of A, r and x on some lanes only, beside ordinary groups of the same warp."""
    rng = np.random.default_rng(N + B)
    A = rng.normal(0, 0.1, (B, N, N))
    A[:, np.arange(N), np.arange(N)] = -1.0
    r, y0, t1 = rng.uniform(0.5, 1.5, (B, N)), rng.uniform(0.1, 1.0, (B, N)), np.full(B, 2.0)
    A[0][np.arange(N) != np.arange(N)[:, None]] = 0.0
    y0[1, 2], r[1, 0] = 0.0, -0.0
    y0[2, 1] = 1e-100
    A[3, 1, 2] = 1e-90
    y0[4] = 0.0
    A[5, 0, 3], y0[5, 3] = -1e80, 1e-79
    y0[6, 0] = np.inf
    p = np.concatenate([r, A.reshape(B, N * N)], 1)
    NP["glv"] = N + N * N
    check(oracle, "glv", tab, y0, p, t1, sorted({*range(7), B // 2, B - 1}))


@pytest.mark.parametrize("N", [5, 10])
@pytest.mark.parametrize("tab", ["dopri5", "ck54"])
@pytest.mark.parametrize("B", [1, 40, 900])
def test_lotka_volterra_warps(oracle, cuda, N, tab, B):
    """A warp per instance against lane groups (a block size that it does not take): several seeds, direct gradients, the
    adjoint history, fewer resident warps than instances, short chunks, failed instances."""
    rng = np.random.default_rng(N * 1000 + B)
    A = rng.normal(0, 0.1, (B, N, N))
    A[:, np.arange(N), np.arange(N)] = -1.0
    p = np.concatenate([rng.uniform(0.5, 1.5, (B, N)), A.reshape(B, N * N)], 1)
    y0, t1 = rng.uniform(0.1, 1.0, (B, N)), rng.uniform(0.0, 8.0, B)
    if B > 10:
        p[3, 0], t1[4], y0[5, 1] = np.nan, 0.0, np.inf
    lam, mud = rng.standard_normal((B, 2, N)), rng.standard_normal((B, 2, N + N * N))
    res = []
    for block, bps, chunk in ((0, 0, 0), (64, 1, 3), (96, 0, 0), (224, 0, 0)):
        s = Solver("glv", N, N + N * N, B, nout=2, tableau=tab, atol=1e-7, rtol=1e-7, block_size=block, blocks_per_sm=bps,
                   chunk_len=chunk, max_steps=45)
        s.set_adjoint_history(4)
        for _ in range(2):
            f = s.forward(dev(y0), dev(p), dev(np.zeros(B)), dev(t1))
            g = s.backward(dev(p), dev(lam), dev(mud))
        res.append([v.cpu().numpy() for v in (f["yT"], f["n_acc"], f["n_rej"], f["status"], g["status"], g["dy0"], g["dp"])])
        s.close()
    pb = oracle.problem("glv", tab, N, N + N * N, 1e-7, 1e-7)
    for b in {0, B - 1}:
        if res[0][3][b] == 0:
            fw = oracle.forward(pb, y0[b], p[b], 0.0, t1[b])
            assert fw["n_acc"] == res[0][1][b]
            np.testing.assert_array_equal(fw["states"][-1], res[0][0][b])
    for r in res[1:]:
        for a, b in zip(r, res[0]):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("model", sorted(NP))
@pytest.mark.parametrize("tab", ["dopri5", "ck54"])
@pytest.mark.parametrize("B,nout", [(1, 2), (33, 3), (700, 2), (2500, 5), (6000, 2)])
def test_two_seeds_at_once(cuda, model, tab, B, nout):
    """Seed rows two at a time against one call per seed row: gradients, status and lambda history, an odd last seed, direct
    gradients, failed instances, instances without a step, a seed that is not finite."""
    y0, p, t1 = draw(model, B, B + nout)
    n, P = y0.shape[1], p.shape[1]
    if B > 10:
        p[3, 0], t1[4], y0[5, 0] = np.nan, 0.0, np.inf
    rng = np.random.default_rng(nout)
    lam, mud = rng.standard_normal((B, nout, n)), rng.standard_normal((B, nout, P))
    if B > 10:
        lam[7, 0, 0], lam[8, nout - 1, 0] = np.inf, np.nan
    got = []
    for rows in [range(nout)] + [[k] for k in range(nout)]:
        s = Solver(model, n, P, B, nout=len(rows), tableau=tab, precision="fp64", atol=1e-6, rtol=1e-6)
        s.set_adjoint_history(6)
        s.forward(dev(y0), dev(p), dev(np.zeros(B)), dev(t1))
        g = s.backward(dev(p), dev(lam[:, rows]), dev(mud[:, rows]))
        hist = [s.adjoint_history(b)[1] for b in {0, B - 1}]
        got.append([g[k].cpu().numpy() for k in ("dy0", "dp", "status")] + [hist])
        s.close()
    for k in range(nout):
        for both, one in zip(got[0][:2], got[1 + k][:2]):
            np.testing.assert_array_equal(both[:, k], one[:, 0])
        for both, one in zip(got[0][3], got[1 + k][3]):
            np.testing.assert_array_equal(both[k], one[0])
    np.testing.assert_array_equal(got[0][2], got[nout][2])  # the last seed row's status


@pytest.mark.parametrize("B,nout", [(4097, 1), (12000, 1), (12000, 2), (40000, 1)])
@pytest.mark.parametrize("tab", ["dopri5", "ck54"])
def test_longest_instances_apart(cuda, tab, B, nout):
    """Uneven batches, whose longest instances run in teams beside the rest, against the same call in an explicit launch
    shape (one sweep for all): every instance's outputs, failed instances, short chunks, the lambda history, a stream of
    its own with graph replays."""
    rng = np.random.default_rng(B)
    y0, p, _ = draw("dho", B, B)
    t1 = np.exp(rng.uniform(np.log(0.2), np.log(30.0), B))
    p[3, 0], t1[4], y0[5, 0] = np.nan, 0.0, np.inf
    t1[6], p[6] = 80.0, (5.0, 0.0)  # out of steps
    lam, mud = rng.standard_normal((B, nout, 2)), rng.standard_normal((B, nout, 2))
    got, keys = [], ("yT", "n_acc", "n_rej", "status")
    for kw in (dict(block_size=64), dict(), dict(chunk_len=3)):
        s = Solver("dho", 2, 2, B, nout=nout, tableau=tab, precision="fp64", atol=1e-7, rtol=1e-7, max_steps=900, **kw)
        s.set_adjoint_history(3)
        for _ in range(2):  # ordered by horizon, then by counts
            f = s.forward(dev(y0), dev(p), dev(np.zeros(B)), dev(t1))
            g = s.backward(dev(p), dev(lam), dev(mud))
            got.append([f[k].cpu().numpy() for k in keys] + [g[k].cpu().numpy() for k in ("status", "dy0", "dp")] +
                       [s.adjoint_history(b)[1] for b in (0, int(np.argmax(t1 * (np.arange(B) != 6))))])
        s.close()
    assert got[0][3][6] != 0 and (got[0][3] == 0).sum() >= B - 4
    for r in got[1:]:
        for a, b in zip(r, got[0]):
            np.testing.assert_array_equal(a, b)
    if nout > 1:
        return
    s = Solver("dho", 2, 2, B, tableau=tab, precision="fp64", atol=1e-7, rtol=1e-7, max_steps=900)
    ins = [dev(v) for v in (y0, p, np.zeros(B), t1)]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(3):
            r = s.gradient("sumsq", *ins)
    side.synchronize()
    np.testing.assert_array_equal(r["yT"].cpu().numpy(), got[0][0])
    np.testing.assert_array_equal(r["n_acc"].cpu().numpy(), got[0][1])
    ref = Solver("dho", 2, 2, B, tableau=tab, precision="fp64", atol=1e-7, rtol=1e-7, max_steps=900, block_size=64)
    want = ref.gradient("sumsq", *ins)
    for k in ("dy0", "dp", "status"):
        np.testing.assert_array_equal(r[k].cpu().numpy(), want[k].cpu().numpy())


@pytest.mark.parametrize("model", ["vdp", "vdp_petsc", "dho"])
@pytest.mark.parametrize("tab", ["dopri5", "ck54"])
@pytest.mark.parametrize("B", [1, 45, 700])
def test_special_values_one_lane(oracle, cuda, model, tab, B):
    """One lane per instance with integer products, forward and backward, at any batch size (a block size that teams do not
    take): zeros of both signs, states and parameters across and beyond the products' range, infinities and NaN, where
    attempt64 and back_step64 refuse and the general step takes over, beside ordinary lanes of the same warp."""
    y0, p, t1 = draw(model, B, 11)
    t1 = np.minimum(t1, 1.0)
    special = [(0.0, 1.0), (-0.0, 1.0), (1.0, -0.0), (0.0, 0.0), (1e-70, 1e-75), (1e-90, 1.0), (1e-310, 1e-300),
               (0.5, 4e-320), (np.inf, 1.0), (1.0, -np.inf), (np.nan, 0.0)]
    if model == "dho":  # (a nonlinear model would be stiff there)
        special += [(1e-30, -1e74), (1e74, -1e70), (3e150, 1.0)]
    for k, v in enumerate(special):
        y0[k % B] = v
        if B == 1:
            break
    if B > 40:
        for k, v in enumerate([0.0, -0.0, 1e-80, 1e-310, 2.0 ** -241, 2.0 ** -239]):
            p[20 + k, 0] = v
            p[30 + k, -1] = v
        p[26], t1[26] = 1e3, 1e-3
        t1[27], t1[28] = 0.0, 1e-12
    n = y0.shape[1]
    s = Solver(model, n, NP[model], B, tableau=tab, precision="fp64", atol=1e-6, rtol=1e-6, block_size=48)
    out = s.gradient("sumsq", dev(y0), dev(p), dev(np.zeros(B)), dev(t1))
    torch.cuda.synchronize()
    r = {k: v.cpu().numpy() for k, v in out.items()}
    s.close()
    pb = oracle.problem(model, tab, n, NP[model], 1e-6, 1e-6)
    ran = 0
    for b in range(min(B, 45)):
        g = oracle.gradient(pb, "sumsq", y0[b], p[b], 0.0, t1[b])
        assert int(r["status"][b]) == g["status"], b
        if g["status"] != 0:
            continue
        ran += 1
        assert int(r["n_acc"][b]) == g["n_acc"], b
        for k in ("yT", "dy0", "dp"):
            np.testing.assert_array_equal(r[k][b], g[k], err_msg=f"{k} {b}")
    assert ran >= min(B, 30)


def parts(lengths, quads):
    """What the longest-first sort makes of a batch: its load and the size of the longest part (0: not split)."""
    top = lengths.max()
    load = lengths.sum() / top
    if not 1.5 * quads < load <= 40 * quads:
        return load, 0
    for share in (0.4, 0.5, 0.6, 0.75):
        part = lengths[lengths > share * top]
        if part.sum() / top <= 2 * quads:
            return load, len(part)
    return load, 0


@pytest.mark.parametrize("nout,stride", [(1, 0), (2, 0), (3, 0), (1, 5)])
@pytest.mark.parametrize("tab", ["dopri5", "ck54"])
def test_split_batch(cuda, tab, nout, stride):
    """Batches well inside the range in which the longest instances run apart, by horizons (first call) and by step counts
    (second), dozens of them and all successful: forward, backward with one and several seed rows, and the
    forward's split with the two-level backward, against one sweep for all in an explicit launch shape."""
    B = 40000
    quads = 4.0 * torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(3)
    y0, p, _ = draw("dho", B, 4)
    t1 = rng.uniform(0.2, 5.0, B)
    long = rng.choice(B, 1200, replace=False)
    t1[long] = rng.uniform(15.0, 30.0, len(long))
    lam, mud = rng.standard_normal((B, nout, 2)), rng.standard_normal((B, nout, 2))
    got = []
    for kw in (dict(block_size=64), dict()):
        s = Solver("dho", 2, 2, B, nout=nout, tableau=tab, precision="fp64", atol=1e-7, rtol=1e-7, ckpt_stride=stride, **kw)
        if not stride:
            s.set_adjoint_history(3)
        for _ in range(2):
            f = s.forward(dev(y0), dev(p), dev(np.zeros(B)), dev(t1))
            g = s.backward(dev(p), dev(lam), dev(mud))
            got.append([f[k].cpu().numpy() for k in ("yT", "n_acc", "n_rej", "status")] +
                       [g[k].cpu().numpy() for k in ("status", "dy0", "dp")] +
                       ([s.adjoint_history(int(b))[1] for b in (long[0], 0)] if not stride else []))
        s.close()
    assert (got[0][3] == 0).all() and (got[0][4] == 0).all()
    for lengths in (t1, (got[0][1] + got[0][2]).astype(float), got[0][1].astype(float)):
        load, part = parts(lengths, quads)
        assert 1.6 * quads < load < 30 * quads and 48 <= part <= 2000, (load, part)  # else this tests nothing
    for r in got[1:]:
        for a, b in zip(r, got[0]):
            np.testing.assert_array_equal(a, b)
