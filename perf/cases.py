"""Performance cases: the discrete-adjoint calls that a user of this package makes.

A case is one batch of one built-in model, taken through `Solver` as a program
takes it: one gradient call, or a forward and a backward sweep with seed rows,
or the gradient call on pinned host buffers.  Inputs follow the distributions
of `vectorizedadjoint_gb300.workloads` (Van der Pol, damped oscillator,
Lotka-Volterra with a matrix per instance or one shared by the batch), drawn
from the seed.  What a program keeps between calls (the handle with its
checkpoint pool, pinned buffers, the shared matrix) is made in `prepare`.
"""
import math

import numpy as np
import torch

from vectorizedadjoint_gb300 import Solver

# Every key a case has; `listed` and `draw` state the ones that differ.
DEFAULTS = dict(model="vdp", n=2, tableau="dopri5", precision="fp64", batch=1, tol=1e-6, horizon=20.0, spread=1.0,
                entry="gradient", nout=1, stride=0, dt0=1e-3)


def _case(**kw):
    return {**DEFAULTS, **kw}


def listed():
    return [
        # the reference's own use: one trajectory, one gradient, FP64 (an optimiser's inner call); latency only
        _case(name="vdp_one_fp64", batch=1, tol=1e-8, horizon=10.0, spread=0.3),
        # a small parameter study that wants the sensitivity matrix: two seed rows after one forward sweep, odd size
        _case(name="vdp_sensitivity_fp64", batch=1003, tableau="ck54", nout=2, entry="pair"),
        # oscillators with uneven horizons in the drop-in precision, Cash-Karp (the reference's 5(4) pair)
        _case(name="dho_batch_fp64", model="dho", tableau="ck54", batch=65536, tol=1e-8, horizon=50.0),
        # a large Van der Pol ensemble in the drop-in precision
        _case(name="vdp_batch_fp64", batch=65536),
        # Fehlberg 7(8) at a tight tolerance, a mid-sized ragged batch
        _case(name="vdp_rkf78_fp64", batch=5003, tableau="rkf78", tol=1e-9, horizon=10.0),
        # memory-bounded: every 16th step checkpointed, segments re-integrated
        _case(name="vdp_two_level_fp64", batch=9001, stride=16),
        # the full Van der Pol ensemble in double-word arithmetic
        _case(name="vdp_batch_dw", precision="mixed_dw", batch=262144),
        # oscillators in double-word arithmetic from pinned host buffers, results back on the host
        _case(name="dho_host_dw", model="dho", tableau="ck54", precision="mixed_dw", batch=65536, tol=1e-8,
              horizon=50.0, entry="host"),
        # a mid-sized ensemble with FP32 stages
        _case(name="vdp_mixed", precision="mixed", batch=20011),
        # per-instance Lotka-Volterra communities: FP64 at a small odd size, double-word at the full size
        _case(name="glv5_fp64", model="glv", n=5, batch=777, tol=1e-7),
        _case(name="glv10_dw", model="glv", n=10, precision="mixed_dw", batch=16384, tol=1e-7),
        # one interaction matrix shared by the batch, its gradient included
        _case(name="glv256_dw", model="glv_shared", n=256, precision="mixed_dw", batch=1024, tol=1e-7, horizon=10.0),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["vdp", "vdp", "vdp", "dho", "dho", "rkf78", "two_level", "mixed", "glv", "glv_shared"])
    spread = rng.choice([0.3, 1.0])
    entry = rng.choice(["gradient", "gradient", "pair", "host"])
    nout = rng.choice([1, 2, 3]) if entry == "pair" else 1
    tab = rng.choice(["dopri5", "ck54"])
    # horizons keep a drawn case within the listed ones' cost
    if kind == "vdp":
        prec = rng.choice(["fp64", "mixed_dw"])
        return _case(tableau=tab, precision=prec, batch=int(_log(rng, 1, 65536 if prec == "fp64" else 262144)),
                     tol=10.0 ** -rng.choice([6, 7, 8]), horizon=rng.uniform(5.0, 12.0), spread=spread, entry=entry,
                     nout=nout)
    if kind == "dho":
        return _case(model="dho", tableau=tab, precision=rng.choice(["fp64", "mixed_dw"]),
                     batch=int(_log(rng, 1, 65536)), tol=10.0 ** -rng.choice([6, 7, 8]),
                     horizon=rng.uniform(10.0, 50.0), entry=entry, nout=1 if nout == 1 else 2)
    if kind == "rkf78":
        return _case(tableau="rkf78", batch=int(_log(rng, 1, 8192)), tol=10.0 ** -rng.choice([7, 8, 9]),
                     horizon=rng.uniform(4.0, 12.0), spread=spread, entry=entry, nout=nout)
    if kind == "two_level":
        return _case(batch=int(_log(rng, 16, 20000)), tableau=tab, stride=rng.choice([4, 16, 50]),
                     horizon=rng.uniform(5.0, 20.0), spread=spread)
    if kind == "mixed":
        return _case(precision="mixed", batch=int(_log(rng, 16, 65536)), tableau=tab, horizon=rng.uniform(5.0, 20.0),
                     spread=spread)
    if kind == "glv":
        n = rng.choice([5, 10])
        prec = rng.choice(["fp64", "mixed_dw"])
        return _case(model="glv", n=n, precision=prec, batch=int(_log(rng, 1, 16384)), tableau=tab, tol=1e-7,
                     horizon=rng.uniform(5.0, 20.0), entry="gradient" if entry == "pair" else entry)
    n = rng.choice([64, 256])
    return _case(model="glv_shared", n=n, precision="mixed_dw", batch=int(_log(rng, 4, 1024)), tol=1e-7,
                 horizon=rng.uniform(4.0, 10.0))


def _npar(case):
    n = case["n"]
    return {"vdp": 1, "dho": 2, "glv": n + n * n, "glv_shared": n}[case["model"]]


def _inputs(case, seed):
    """Host arrays: y0 [B, n], params [B, P], t0 [B], t1 [B], the shared matrix or None, seeds [B, nout, n] or None."""
    rng = np.random.Generator(np.random.PCG64(seed))
    B, n, T = case["batch"], case["n"], case["horizon"]
    shared = lam = None
    t1 = np.full(B, T)
    if case["model"] == "vdp":
        # mu log-uniform in 10^[-spread, spread]: step counts vary up to 100x
        params = 10.0 ** rng.uniform(-case["spread"], case["spread"], (B, 1))
        y0 = rng.uniform(-2.0, 2.0, (B, 2))
    elif case["model"] == "dho":
        params = np.stack([rng.uniform(0.5, 5.0, B), rng.uniform(0.0, 0.5, B)], axis=1)
        y0 = rng.uniform(-1.0, 1.0, (B, 2))
        t1 = rng.uniform(0.1 * T, T, B)
    elif case["model"] == "glv":
        A = rng.normal(0.0, 0.1, (B, n, n))
        A[:, np.arange(n), np.arange(n)] = -1.0
        params = np.concatenate([rng.uniform(0.5, 1.5, (B, n)), A.reshape(B, n * n)], axis=1)
        y0 = rng.uniform(0.1, 1.0, (B, n))
    else:
        shared = rng.normal(0.0, 0.5 / np.sqrt(n), (n, n))
        shared[np.arange(n), np.arange(n)] = -1.0
        params = rng.uniform(0.5, 1.5, (B, n))
        y0 = rng.uniform(0.1, 1.0, (B, n))
    if case["entry"] == "pair":
        lam = rng.standard_normal((B, case["nout"], n))
    return y0, np.ascontiguousarray(params), np.zeros(B), t1, shared, lam


def _cost(case):
    return "sum" if case["model"].startswith("glv") else "sumsq"


def prepare(case, seed):
    y0, params, t0, t1, shared, lam = _inputs(case, seed)
    solver = Solver(case["model"], case["n"], _npar(case), case["batch"], nout=case["nout"], tableau=case["tableau"],
                    precision=case["precision"], atol=case["tol"], rtol=case["tol"], dt0=case["dt0"],
                    ckpt_stride=case["stride"])
    st = {"case": case, "solver": solver}

    def dev(a):
        return torch.tensor(a, dtype=torch.float64, device="cuda")

    if case["entry"] == "host":
        def pin(a):
            return torch.tensor(a).pin_memory()
        B, n, P = case["batch"], case["n"], _npar(case)
        st["in"] = [pin(a) for a in (y0, params, t0, t1)]
        st["out"] = dict(yT=pin(np.empty((B, n))), dy0=pin(np.empty((B, n))), dp=pin(np.empty((B, P))),
                         n_acc=pin(np.empty(B, np.int32)), status=pin(np.empty(B, np.int32)))
    else:
        st["in"] = [dev(a) for a in (y0, params, t0, t1)]
    if shared is not None:
        st["dA"] = torch.empty(case["n"], case["n"], dtype=torch.float64, device="cuda")
        solver.set_shared(dev(shared), st["dA"])
    if lam is not None:
        st["lam"] = dev(lam)
    return st


def run(state):
    case, solver = state["case"], state["solver"]
    if case["entry"] == "pair":
        fw = solver.forward(*state["in"])
        bw = solver.backward(state["in"][1], state["lam"])
        return {"yT": fw["yT"], "n_acc": fw["n_acc"], "n_rej": fw["n_rej"], "status": bw["status"],
                "dy0": bw["dy0"], "dp": bw["dp"]}
    if case["entry"] == "host":
        return dict(solver.gradient_host(_cost(case), *state["in"], out=state["out"]))
    out = dict(solver.gradient(_cost(case), *state["in"]))
    if "dA" in state:
        out["dA"] = state["dA"]
    return out


def work(case):
    """Bytes: each input read and each output written once.  Flops: the algorithm's FP64 operations, steps estimated
    from the horizon and the tolerance (a 5(4) pair at tol 1e-6 takes about 8 steps per unit of time on Van der Pol)."""
    B, n, P, Q = case["batch"], case["n"], _npar(case), case["nout"]
    order, stages = (8, 13) if case["tableau"] == "rkf78" else (5, 6)
    per_t = 8.0 if order == 5 else 5.0
    steps = per_t * case["horizon"] * (case["tol"] / 1e-6) ** (-1.0 / order) * {"vdp": 1.0, "dho": 0.3}.get(case["model"], 0.25)
    rhs = 2.0 * n * n if case["model"].startswith("glv") else 3.0 * n
    nnz = 0.5 * stages * (stages - 1) * (0.55 if order == 8 else 1.0)
    fwd = stages * rhs + 2.0 * n * (nnz + 2 * stages) + 30.0
    bwd = stages * rhs + 2.0 * n * nnz + Q * (2.0 * stages * rhs + 3.0 * n * nnz)
    byt = 8.0 * B * (n + P + 2 + n + Q * (n + P) + (Q * n if case["entry"] == "pair" else 0)) + 8.0 * B
    byt += 16.0 * n * n if case["model"] == "glv_shared" else 0.0
    return {"bytes": byt, "flops": B * steps * (fwd + bwd)}


# ---------------------------------------------------------------- 64-bit reference
#
# The controlled Runge-Kutta loop (odeint's controller) and its frozen-step discrete adjoint in torch FP64, the
# whole batch at a time.

def _tableau(name):
    if name == "dopri5":
        a = [[], [1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9],
             [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
             [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656]]
        b = [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]
        e = [b[0] - 5179 / 57600, 0, b[2] - 7571 / 16695, b[3] - 393 / 640, b[4] + 92097 / 339200, b[5] - 187 / 2100]
        return a, b, e, -1 / 40, 4, 5
    if name == "ck54":
        a = [[], [1 / 5], [3 / 40, 9 / 40], [3 / 10, -9 / 10, 6 / 5], [-11 / 54, 5 / 2, -70 / 27, 35 / 27],
             [1631 / 55296, 175 / 512, 575 / 13824, 44275 / 110592, 253 / 4096]]
        b = [37 / 378, 0, 250 / 621, 125 / 594, 0, 512 / 1771]
        e = [b[0] - 2825 / 27648, 0, b[2] - 18575 / 48384, b[3] - 13525 / 55296, -277 / 14336, b[5] - 1 / 4]
        return a, b, e, None, 4, 5
    a = [[], [2 / 27], [1 / 36, 1 / 12], [1 / 24, 0, 1 / 8], [5 / 12, 0, -25 / 16, 25 / 16], [1 / 20, 0, 0, 1 / 4, 1 / 5],
         [-25 / 108, 0, 0, 125 / 108, -65 / 27, 125 / 54], [31 / 300, 0, 0, 0, 61 / 225, -2 / 9, 13 / 900],
         [2, 0, 0, -53 / 6, 704 / 45, -107 / 9, 67 / 90, 3],
         [-91 / 108, 0, 0, 23 / 108, -976 / 135, 311 / 54, -19 / 60, 17 / 6, -1 / 12],
         [2383 / 4100, 0, 0, -341 / 164, 4496 / 1025, -301 / 82, 2133 / 4100, 45 / 82, 45 / 164, 18 / 41],
         [3 / 205, 0, 0, 0, 0, -6 / 41, -3 / 205, -3 / 41, 3 / 41, 6 / 41],
         [-1777 / 4100, 0, 0, -341 / 164, 4496 / 1025, -289 / 82, 2193 / 4100, 51 / 82, 33 / 164, 12 / 41, 0, 1]]
    b = [0, 0, 0, 0, 0, 34 / 105, 9 / 35, 9 / 35, 9 / 280, 9 / 280, 0, 41 / 840, 41 / 840]
    e = [-41 / 840, 0, 0, 0, 0, 0, 0, 0, 0, 0, -41 / 840, 41 / 840, 41 / 840]
    return a, b, e, None, 7, 8


def _model(case, par, shared):
    """rhs(x) and vjp(w, x) -> (J_x^T w, per-instance J_p^T w, contribution to the shared matrix's gradient)."""
    n = case["n"]
    if case["model"] == "vdp":
        mu = par[:, 0]

        def rhs(x):
            return torch.stack([x[:, 1], mu * (1 - x[:, 0] ** 2) * x[:, 1] - x[:, 0]], 1)

        def vjp(w, x):
            c = 1 - x[:, 0] ** 2
            gx = torch.stack([w[:, 1] * (-2 * mu * x[:, 0] * x[:, 1] - 1), w[:, 0] + w[:, 1] * mu * c], 1)
            return gx, (w[:, 1] * c * x[:, 1])[:, None], None
    elif case["model"] == "dho":
        om, ze = par[:, 0], par[:, 1]

        def rhs(x):
            return torch.stack([x[:, 1], -om * om * x[:, 0] - 2 * ze * om * x[:, 1]], 1)

        def vjp(w, x):
            gx = torch.stack([-w[:, 1] * om * om, w[:, 0] - 2 * ze * om * w[:, 1]], 1)
            gp = torch.stack([w[:, 1] * (-2 * om * x[:, 0] - 2 * ze * x[:, 1]), -2 * om * w[:, 1] * x[:, 1]], 1)
            return gx, gp, None
    else:
        r = par[:, :n]
        A = par[:, n:].reshape(-1, n, n) if shared is None else shared

        def mul(v, M, trans):
            if M.dim() == 2:
                return v @ (M if trans else M.T)
            return torch.einsum("bji,bj->bi" if trans else "bij,bj->bi", M, v)

        def rhs(x):
            return x * (r + mul(x, A, False))

        def vjp(w, x):
            wx = w * x
            gx = w * (r + mul(x, A, False)) + mul(wx, A, True)
            if shared is not None:
                return gx, wx, wx.T @ x
            return gx, torch.cat([wx, (wx[:, :, None] * x[:, None, :]).reshape(-1, n * n)], 1), None
    return rhs, vjp


def exact(case, seed):
    y0, params, t0, t1, shared, lam = _inputs(case, seed)
    a, b, e, e_new, err_order, order = _tableau(case["tableau"])
    d = "cuda" if torch.cuda.is_available() else "cpu"
    y, par, t, t1 = (torch.tensor(v, device=d) for v in (y0, params, t0, t1))
    A = None if shared is None else torch.tensor(shared, device=d)
    rhs, vjp = _model(case, par, A)
    B, n, tol, S = case["batch"], case["n"], case["tol"], len(a)
    eps = float(np.finfo(np.float64).eps)

    def stages(y, h):
        X, K = [], []
        for row in a:
            x = y
            for c, k in zip(row, K):
                if c:
                    x = x + (c * h)[:, None] * k
            X.append(x)
            K.append(rhs(x))
        return X, K

    def comb(w, K, h):
        return sum((c * h)[:, None] * k for c, k in zip(w, K) if c)

    dt = torch.full((B,), case["dt0"], dtype=torch.float64, device=d)
    cnt = torch.zeros(B, dtype=torch.int64, device=d)
    idx = torch.arange(B, device=d)
    cap = 256
    Y = torch.zeros(cap + 1, B, n, dtype=torch.float64, device=d)
    Ts = torch.zeros(cap + 1, B, dtype=torch.float64, device=d)
    for attempt in range(200000):
        if attempt % 32 == 0:
            if not bool((t1 - t > eps).any()):
                break
            if int(cnt.max()) + 33 > cap:
                Y, Ts = torch.cat([Y, torch.zeros_like(Y[:cap])]), torch.cat([Ts, torch.zeros_like(Ts[:cap])])
                cap *= 2
        top = t1 - t > eps
        Y[cnt, idx], Ts[cnt, idx] = y, t
        h = torch.where(t + dt - t1 > eps, t1 - t, dt)
        h = torch.where(top, h, torch.zeros_like(h))
        X, K = stages(y, h)
        yn = y + comb(b, K, h)
        ev = comb(e, K, h)
        if e_new is not None:
            ev = ev + (e_new * h)[:, None] * rhs(yn)
        err = (ev.abs() / (tol + tol * (y.abs() + h.abs()[:, None] * K[0].abs()))).amax(1)
        bad = top & (err > 1)
        ok = top & ~bad
        shrink = h * torch.clamp(0.9 * err.clamp(min=1e-300) ** (-1.0 / (err_order - 1)), min=0.2)
        grow = torch.where(err < 0.5, h * 0.9 * err.clamp(min=5.0 ** -order) ** (-1.0 / order), h)
        dt = torch.where(bad, shrink, torch.where(ok, grow, dt))
        t = torch.where(ok, t + h, t)
        y = torch.where(ok[:, None], yn, y)
        cnt = cnt + ok
    Y[cnt, idx], Ts[cnt, idx] = y, t
    Q = case["nout"]
    dA = torch.zeros(n, n, dtype=torch.float64, device=d)
    lams = ([torch.tensor(lam[:, q], device=d) for q in range(Q)] if lam is not None
            else [2 * y if _cost(case) == "sumsq" else torch.ones_like(y)])
    mus = [torch.zeros(B, par.shape[1], dtype=torch.float64, device=d) for _ in lams]
    for j in range(int(cnt.max()) - 1, -1, -1):
        on = cnt > j
        h = torch.where(on, Ts[j + 1] - Ts[j], torch.zeros_like(t))
        X, _ = stages(torch.where(on[:, None], Y[j], y), h)
        for q, l0 in enumerate(lams):
            bars = [(c * h)[:, None] * l0 for c in b]
            l1 = l0
            for m in range(S - 1, -1, -1):
                gx, gp, gA = vjp(bars[m], X[m])
                l1 = l1 + gx
                mus[q] = mus[q] + gp
                if gA is not None:
                    dA = dA + gA
                for k, c in enumerate(a[m]):
                    if c:
                        bars[k] = bars[k] + (c * h)[:, None] * gx
            lams[q] = l1
    outs_y, outs_p = torch.stack(lams, 1), torch.stack(mus, 1)
    if case["entry"] == "pair":
        return {"yT": y, "n_acc": None, "n_rej": None, "status": None, "dy0": outs_y, "dp": outs_p}
    out = {"yT": y, "dy0": outs_y[:, 0], "dp": outs_p[:, 0], "n_acc": None, "status": None}
    if shared is not None:
        out["dA"] = dA
    return out
