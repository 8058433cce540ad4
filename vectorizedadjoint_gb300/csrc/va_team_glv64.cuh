// FP64 sweeps of the per-instance Lotka-Volterra model for small batches: a
// warp per instance, its lanes in 30 / N groups of N, lane i of each group on
// component i.
//
// With a warp per quadrant an FP64 step costs its FP64 instruction count times
// 64 cycles (va_int64.cuh).  The lane groups of va_group.cuh issue ~170 per
// attempt and ~320 per back step at N = 5, most of them the same on every row
// of the tableau.  Here the groups share them out: forward, each group keeps
// the running sums of its own rows (as the teams of va_team64.cuh); backward,
// each group recomputes another step (stage points and rates, which do not
// depend on lambda), and in the chain through lambda it keeps its own K-bar
// rows, forms its own columns' products A_ki v_k and accumulates its own
// columns of dA.  ~95 and ~105 FP64 instructions.  Every sum takes its terms in
// the groups' order, so the bits are the same.
#pragma once

#include "va_team64.cuh"

namespace va {

template <int NN>
struct GlvWarp {
    static constexpr int NG = 30 / NN; // groups
    static constexpr unsigned mask = (1u << (NG * NN)) - 1u;
    static constexpr int CQ = NN / NG + 1; // columns per group, that of r included
    int lane, g, i;
    __device__ __forceinline__ GlvWarp() : lane(threadIdx.x & 31), g(lane / NN), i(lane % NN) {}
    __device__ __forceinline__ bool active() const { return lane < NG * NN; }
    __device__ __forceinline__ static double get(double v, int src) { return __shfl_sync(mask, v, src); }
    __device__ __forceinline__ int take(unsigned int *counter) const
    {
        int v = 0;
        if (lane == 0)
            v = (int)atomicAdd(counter, 1u);
        return __shfl_sync(mask, v, 0);
    }
};

// ------------------------------------------------------------ forward sweep

template <int NN, class Tab>
struct GlvForward {
    static constexpr int G = GlvWarp<NN>::NG * NN, NS = Tab::S;
    using Rows = TeamRows<Tab, NN, G>;
    static constexpr int Q = Rows::Q, J = NS + 1;
    GlvWarp<NN> wp;
    double c[J][Q];
    bool new_row[Q], err[Q], den[Q];

    __device__ __forceinline__ GlvForward()
    {
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const int rank = wp.g + GlvWarp<NN>::NG * q;
            new_row[q] = rank == Rows::rank_b;
            err[q] = rank == Rows::rank_e;
            den[q] = rank == Rows::rank_d;
#pragma unroll
            for (int j = 0; j < J; j++)
                c[j][q] = wp.active() ? kTeamForward<Tab, NN, G>.c[j][wp.lane + G * q] : 0.0;
        }
    }
    // component `comp` of a row
    __device__ __forceinline__ double row(const double (&acc)[Q], int rank, int comp) const
    {
        return wp.get(acc[rank / GlvWarp<NN>::NG], rank % GlvWarp<NN>::NG * NN + comp);
    }
    // f_i at the point that a row holds; x: its own component
    __device__ __forceinline__ double rhs(const double (&acc)[Q], int rank, const double (&p)[1 + NN], double &x) const
    {
        double s = 0.0;
#pragma unroll
        for (int j = 0; j < NN; j++)
            s = p[1 + j] * row(acc, rank, j) + s;
        x = row(acc, rank, wp.i);
        return x * (p[0] + s);
    }
    __device__ __forceinline__ void add(double (&acc)[Q], int j, double K, double dt, double atol, double rtol) const
    {
#pragma unroll
        for (int q = 0; q < Q; q++)
            if (Rows::any_used(q, j)) {
                double w = c[j][q] * dt, k = K, s = acc[q];
                const bool dq = Rows::has(q, Rows::rank_d);
                if (dq && j == 1) { // the denominator's atol + rtol (|y| + |dt K_0|)
                    w = den[q] ? rtol : w;
                    k = den[q] ? s : k;
                    s = den[q] ? atol : s;
                }
                double term = w * k;
                if (dq && j == 0)
                    term = den[q] ? fabs(term) : term;
                s = s + term;
                bool keep = false; // as TeamForward::add
                if (Rows::has(q, Rows::rank_b) && !Rows::used(Rows::rank_b, j))
                    keep = keep || new_row[q];
                if (Rows::has(q, Rows::rank_e) && !Rows::used(Rows::rank_e, j))
                    keep = keep || err[q];
                if (dq && !Rows::used(Rows::rank_d, j))
                    keep = keep || den[q];
                acc[q] = keep ? acc[q] : s;
            }
    }
    // the attempt on every lane's component; the error norm on all
    __device__ __forceinline__ double attempt(double y, double k0, const double (&p)[1 + NN], double dt, double atol,
                                              double rtol, double &ynew, double &knew) const
    {
        double acc[Q], x;
#pragma unroll
        for (int q = 0; q < Q; q++)
            acc[q] = err[q] ? -0.0 : den[q] ? fabs(y) : y;
        add(acc, 0, k0, dt, atol, rtol);
#pragma unroll
        for (int m = 1; m < NS; m++)
            add(acc, m, rhs(acc, Rows::rank_x(m), p, x), dt, atol, rtol);
        if constexpr (Tab::FSAL) {
            knew = rhs(acc, Rows::rank_b, p, ynew);
            add(acc, NS, knew, dt, atol, rtol);
        } else {
            ynew = row(acc, Rows::rank_b, wp.i);
        }
        const double r = quotient64(fabs(row(acc, Rows::rank_e, wp.i)), row(acc, Rows::rank_d, wp.i));
        double worst = 0.0;
        bool nan = false;
#pragma unroll
        for (int j = 0; j < NN; j++) {
            const double o = wp.get(r, j);
            nan = nan || is_nan64(o);
            worst = max_nonneg64(worst, o);
        }
        return nan ? __longlong_as_double(0x7ff8000000000000ll) : worst;
    }
};

template <int NN, class Tab>
__global__ void __launch_bounds__(256) forward_glv_warp_kernel(FwdParams a)
{
    constexpr int PT = NN + NN * NN, RS = record_doubles(NN);
    if (gated_off(a))
        return;
    const GlvForward<NN, Tab> gf;
    const GlvWarp<NN> &wp = gf.wp;
    if (!wp.active())
        return;
    const bool first = wp.lane == 0;
    const int i = wp.i, CH = a.pool.chunk_len;
    const unsigned mask = GlvWarp<NN>::mask;

    int b = -1;
    double y = 0.0, k0 = 0.0, p[1 + NN], t = 0.0, t1 = 0.0, dt = 0.0;
    int count = 0, rej = 0, fails = 0, status = ST_OK, chunk = -1, slot = 0;
    bool at_top = true;

    // f at y, which every group holds
    auto slope = [&]() -> double {
        double s = 0.0;
#pragma unroll
        for (int j = 0; j < NN; j++)
            s = p[1 + j] * wp.get(y, j) + s;
        return y * (p[0] + s);
    };
    auto fetch = [&]() -> bool {
        if (__shfl_sync(mask, first && gives_up(a, 32) ? 1 : 0, 0))
            return false;
        b = wp.take(&a.ctl->fwd_next);
        if (b >= a.B)
            return false;
        if (a.order)
            b = a.order[b];
        y = a.y0[(size_t)b * NN + i];
        const double *par = a.par + (size_t)b * PT;
        p[0] = par[i];
#pragma unroll
        for (int j = 0; j < NN; j++)
            p[1 + j] = par[NN + i * NN + j];
        t = a.t0[b];
        t1 = a.t1[b];
        dt = a.dt0;
        count = rej = fails = 0;
        status = ST_OK;
        at_top = true;
        slot = 0;
        chunk = wp.take(&a.ctl->pool_next);
        if (chunk >= a.pool.n_chunks) {
            status = ST_CKPT_BUDGET;
            chunk = -1;
            if (first)
                atomicOr(&a.ctl->pool_fail, 1u);
        } else if (first) {
            a.pool.chunk_prev[chunk] = -1;
        }
        k0 = slope();
        return true;
    };
    auto reserve = [&]() -> bool {
        if (chunk < 0)
            return false;
        if (slot == CH) {
            const int c = wp.take(&a.ctl->pool_next);
            if (c >= a.pool.n_chunks) {
                if (first)
                    atomicOr(&a.ctl->pool_fail, 1u);
                return false;
            }
            if (first)
                a.pool.chunk_prev[c] = chunk;
            chunk = c;
            slot = 0;
        }
        return true;
    };
    auto write = [&]() {
        double *r = record_ptr<RS>(a.pool, chunk, slot);
        if (first)
            *reinterpret_cast<double2 *>(r) = make_double2(t, dt);
        if (wp.g == 0)
            r[2 + i] = y;
        slot++;
    };
    auto finish = [&]() {
        if (status == ST_OK) {
            if (reserve())
                write();
            else
                status = ST_CKPT_BUDGET;
            if (__any_sync(mask, !is_finite64(y)))
                status = ST_NONFINITE;
        }
        if (a.yT && wp.g == 0)
            a.yT[(size_t)b * NN + i] = y;
        if (first) {
            a.inst_T[b] = count;
            a.inst_last[b] = chunk;
            a.inst_status[b] = status;
            if (a.inst_t1)
                a.inst_t1[b] = t1;
            note_work(a, b, count + rej);
            note_finished(a, b, count + rej);
            if (a.n_acc_out)
                a.n_acc_out[b] = count;
            if (a.n_rej_out)
                a.n_rej_out[b] = rej;
            if (a.status_out)
                a.status_out[b] = status;
        }
    };

    bool alive = fetch();
    while (alive) {
        if (status != ST_OK) {
            finish();
            alive = fetch();
            continue;
        }
        if (at_top) {
            if (!greater_pos64(t1 - t, kDblEps)) {
                finish();
                alive = fetch();
                continue;
            }
            if (count >= a.max_steps) {
                status = ST_MAX_STEPS;
                continue;
            }
            if (a.stride <= 1 || count % a.stride == 0) {
                if (!reserve()) {
                    status = ST_CKPT_BUDGET;
                    continue;
                }
                write();
            }
            if (greater_pos64((t + dt) - t1, kDblEps))
                dt = t1 - t;
            fails = 0;
            at_top = false;
        }
        double ynew, knew = 0.0;
        const double err = gf.attempt(y, k0, p, dt, a.atol, a.rtol, ynew, knew);
        bool ok;
        if (is_nan64(err)) {
            status = ST_NONFINITE;
            continue;
        }
        unsigned int *undecided = first ? &a.ctl->pow_undecided : nullptr;
        if (greater_nonneg64(err, 1.0)) {
            dt = decrease_step<Tab, double>(dt, err, a.step_pow, undecided);
            rej++;
            ok = false;
        } else {
            t += dt;
            dt = increase_step<Tab, double>(dt, err, a.step_pow, undecided);
            y = ynew;
            k0 = Tab::FSAL ? knew : slope();
            ok = true;
        }
        if (fails >= a.max_fail) {
            status = ST_MAX_REJECTS;
            continue;
        }
        fails++;
        if (ok) {
            count++;
            at_top = true;
        } else if (!positive_finite64(dt)) {
            status = ST_NONFINITE;
        }
    }
}

// ----------------------------------------------------------- backward sweep

template <int NN, class Tab>
__global__ void __launch_bounds__(256) backward_glv_warp_kernel(AdjParams a)
{
    using W = GlvWarp<NN>;
    constexpr int PT = NN + NN * NN, RS = record_doubles(NN), NS = Tab::S, NG = W::NG, CQ = W::CQ;
    constexpr int Q = (NS + NG - 1) / NG; // K-bar rows g, g + NG, .. of a group
    if (gated_off(a))
        return;
    const W wp;
    if (!wp.active())
        return;
    const bool first = wp.lane == 0;
    const int i = wp.i, g = wp.g, CH = a.pool.chunk_len;
    const unsigned mask = W::mask;

    double ca[NS][Q], cb[Q]; // a_mk and b_k of the group's rows
#pragma unroll
    for (int q = 0; q < Q; q++) {
        cb[q] = 0.0;
#pragma unroll
        for (int m = 0; m < NS; m++)
            ca[m][q] = 0.0;
#pragma unroll
        for (int k = q * NG; k < (q + 1) * NG && k < NS; k++)
            if (g + NG * q == k) {
                cb[q] = Tab::b(k);
#pragma unroll
                for (int m = k + 1; m < NS; m++)
                    ca[m][q] = Tab::a(m, k);
            }
    }

    int b = -1, s0 = 0, j = -1, chunk = -1, slot = 0, T = 0, last = -1, ready = 0, pos = 0;
    double lam = 0.0, mu[CQ], t_next = 0.0, h = 0.0, X[NS], rate[NS];
    double p[1 + NN]; // r_i and row i of A
    double col[CQ];   // A_ki of the group's columns k = g, g + NG, ..

    // stage points and rates of the steps j, j - 1, .., a group a step
    auto prepare = [&]() {
        ready = j + 1 < NG ? j + 1 : NG;
        pos = 0;
        int c = chunk, s = slot - 1 - (g < ready ? g : ready - 1);
        while (s < 0) {
            c = a.pool.chunk_prev[c];
            s += CH;
        }
        const double *r = record_ptr<RS>(a.pool, c, s);
        const double tn = r[0], y[1] = {r[2 + i]};
        const double above = __shfl_sync(mask, tn, g > 0 ? wp.lane - NN : wp.lane);
        h = (g == 0 ? t_next : above) - tn;
        t_next = __shfl_sync(mask, tn, (ready - 1) * NN);
        chunk = __shfl_sync(mask, c, (ready - 1) * NN);
        slot = __shfl_sync(mask, s, (ready - 1) * NN);
        double K[NS][1], Xm[1];
#pragma unroll
        for (int m = 0; m < NS; m++) {
            form_stage<Tab, 1, double>(m, y, y, K, h, h, Xm);
            double acc = 0.0;
#pragma unroll
            for (int k = 0; k < NN; k++)
                acc = p[1 + k] * W::get(Xm[0], g * NN + k) + acc;
            X[m] = Xm[0];
            rate[m] = p[0] + acc;
            K[m][0] = Xm[0] * rate[m];
        }
    };

    auto start_seed = [&]() {
        chunk = last;
        slot = T % CH;
        const double *r = record_ptr<RS>(a.pool, chunk, slot);
        t_next = r[0];
        const double yT = r[2 + i];
        const size_t o = ((size_t)b * a.nout + s0);
        lam = a.cost == 0 ? 2.0 * yT : a.cost == 1 ? 1.0 : a.lambdaT[o * NN + i];
#pragma unroll
        for (int c = 0; c < CQ; c++)
            mu[c] = 0.0;
        if (g == 0)
            note_lambda_lane(a, b, s0, T, NN, i, lam);
        j = T - 1;
        ready = pos = 0;
    };
    auto fetch = [&]() -> bool {
        for (;;) {
            const int w = wp.take(&a.ctl->adj_next);
            if (w >= a.B)
                return false;
            b = a.order ? a.order[w] : w;
            const int st = a.inst_status[b];
            if (st != ST_OK) {
                const double nan = __longlong_as_double(0x7ff8000000000000ll);
                for (int qq = 0; qq < a.nout; qq++) {
                    const size_t o = ((size_t)b * a.nout + qq);
                    if (g == 0)
                        a.dy0[o * NN + i] = nan;
                    for (int k = wp.lane; k < PT; k += NG * NN)
                        a.dpar[o * PT + k] = nan;
                }
                if (a.status_out && first)
                    a.status_out[b] = st;
                continue;
            }
            const double *par = a.par + (size_t)b * PT;
            p[0] = par[i];
#pragma unroll
            for (int k = 0; k < NN; k++)
                p[1 + k] = par[NN + i * NN + k];
#pragma unroll
            for (int c = 0; c < CQ; c++)
                col[c] = g + NG * c < NN ? par[NN + (g + NG * c) * NN + i] : 0.0;
            T = a.inst_T[b];
            last = a.inst_last[b];
            s0 = 0;
            start_seed();
            return true;
        }
    };
    auto finish_seed = [&]() {
        const size_t o = ((size_t)b * a.nout + s0);
        if (g == 0)
            a.dy0[o * NN + i] = lam;
        bool finite = is_finite64(lam);
#pragma unroll
        for (int c = 0; c < CQ; c++) {
            const int k = g + NG * c;
            if (k <= NN) { // column k of row i, or r_i
                const int at = k < NN ? NN + i * NN + k : i;
                a.dpar[o * PT + at] = (a.mu_direct ? a.mu_direct[o * PT + at] : 0.0) + mu[c];
                finite = finite && is_finite64(mu[c]);
            }
        }
        const bool all_finite = __all_sync(mask, finite);
        if (a.status_out && first && (s0 == a.nout - 1 || !all_finite))
            a.status_out[b] = all_finite ? ST_OK : ST_NONFINITE;
    };

    bool alive = fetch();
    while (alive) {
        if (j < 0) {
            finish_seed();
            if (s0 + 1 < a.nout) {
                s0++;
                start_seed();
            } else {
                alive = fetch();
            }
            continue;
        }
        if (pos == ready)
            prepare();
        // back_step with the points and rates of group pos
        const double hs = __shfl_sync(mask, h, pos * NN);
        double Kb[Q], ybar = lam;
#pragma unroll
        for (int q = 0; q < Q; q++)
            Kb[q] = (cb[q] * hs) * lam;
#pragma unroll
        for (int m = NS - 1; m >= 0; m--) {
            const double w = W::get(Kb[m / NG], m % NG * NN + i);
            const double x = W::get(X[m], pos * NN + i), rt = W::get(rate[m], pos * NN + i);
            const double v = w * x;
            double prod[CQ];
#pragma unroll
            for (int c = 0; c < CQ; c++) {
                const int k = g + NG * c;
                prod[c] = col[c] * W::get(v, k < NN ? k : 0);
                // dA_ik += v_i x_k, dr_i += v_i
                const double xk = W::get(X[m], pos * NN + (k < NN ? k : 0)), term = v * xk;
                mu[c] += k == NN ? v : term;
            }
            double gx = w * rt;
#pragma unroll
            for (int k = 0; k < NN; k++)
                gx = W::get(prod[k / NG], k % NG * NN + i) + gx;
            ybar += gx;
#pragma unroll
            for (int q = 0; q < Q; q++)
                if (q * NG < m)
                    Kb[q] += gx * ca[m][q] * hs;
        }
        lam = ybar;
        if (g == 0)
            note_lambda_lane(a, b, s0, j, NN, i, lam);
        pos++;
        j--;
    }
}

} // namespace va
