// FP64 sweeps for small batches: one instance is carried by a team of G lanes.
//
// An FP64 instruction takes its SM quadrant's FP64 unit for 64 cycles however
// many lanes are active and however independent its neighbours are
// (va_int64.cuh), so with one warp on a quadrant the time of a step is its
// FP64 instruction count: a lane that carries an instance alone issues ~230
// of them per attempt of a 5(4) pair (two components) while the other 31
// lanes, or the other quadrants, have nothing to do.  A team spreads what is
// independent: lane l keeps the running sums of one (row, component) pair,
// the rows being the stages X_1 .. X_{s-1}, the new state, the error estimate
// and the error's denominator; a stage's slope K_j, once known to every lane,
// is then added to all rows with one product and one sum.  The right-hand
// side and the controller run on every lane alike.  ~60 FP64 instructions per
// attempt (G = 16) instead of ~230, and the same bits: every (row, component)
// sum takes the terms of form_stage / attempt_pair in their order.
//
// The backward sweep is spread twice.  What a back step needs from the forward
// trajectory -- the stage values recomputed from y_n with h_n, and the VJP's
// weights at them -- does not depend on lambda, so a team forms it for G steps
// at once, a lane a step (~170 FP64 instructions for G steps of a 5(4) pair).
// The chain through lambda is then ~33 FP64 instructions per step, its rows
// (lambda, mu, K-bar_0 .. K-bar_{s-1}) spread over the lanes.
//
// Measured, forward + backward: one Van der Pol instance 4.4 ms (a lane, FP64
// products) -> 2.0 ms with the recompute spread over rows -> 1.5 ms over steps;
// 1,216 instances 6.2 -> 2.5 -> 1.96; Fehlberg 7(8), 600 instances 9.5 -> 2.5
// -> 1.9; two-level backward, 600 instances 11.2 -> 3.6 -> 2.9, and 0.8
// with a segment a lane.  What is left is the
// latency of a step's chain (right-hand side, one product and one sum per
// stage, the shuffles between them, the step factor): the FP64 unit is busy
// about half the time.
#pragma once

#include "va_group.cuh"
#include "va_registry.h"

namespace va {

// Rows of the forward sums.  Order (rank): y_new, error, X_{s-1} .. X_1,
// error denominator.  Slot rank * N + i is kept by lane slot % G as its
// accumulator slot / G.
template <class Tab, int N, int G>
struct TeamRows {
    static constexpr int NS = Tab::S;
    static constexpr int R = NS + 2;
    static constexpr int Q = (R * N + G - 1) / G;
    static constexpr int rank_b = 0, rank_e = 1, rank_d = R - 1;
    __host__ __device__ static constexpr int rank_x(int m) { return NS + 1 - m; }
    // weight of K_j in the row (the denominator's 1 |K_0|)
    __host__ __device__ static constexpr double coef(int rank, int j)
    {
        if (rank == rank_b)
            return j < NS ? Tab::b(j) : 0.0;
        if (rank == rank_e)
            return j < NS ? Tab::e(j) : Tab::E_NEW;
        if (rank == rank_d)
            return j == 0 ? 1.0 : 0.0;
        const int m = NS + 1 - rank;
        return j < m && j < NS ? Tab::a(m, j) : 0.0;
    }
    // whether the row takes a term at j: the stages take every j < m (their
    // zero coefficients included, as form_stage), y_new and the error the
    // non-zero ones, the denominator its two
    __host__ __device__ static constexpr bool used(int rank, int j)
    {
        if (rank == rank_b || rank == rank_e)
            return coef(rank, j) != 0.0;
        if (rank == rank_d)
            return j <= 1;
        return j < NS + 1 - rank;
    }
    __host__ __device__ static constexpr bool any_used(int q, int j)
    {
        for (int s = q * G; s < (q + 1) * G && s < R * N; s++)
            if (used(s / N, j))
                return true;
        return false;
    }
    __host__ __device__ static constexpr bool has(int q, int rank)
    {
        for (int i = 0; i < N; i++)
            if ((rank * N + i) / G == q)
                return true;
        return false;
    }
};

// The rows' weights by lane, read once per kernel.
template <class Tab, int N, int G>
struct TeamForwardTable {
    using Rows = TeamRows<Tab, N, G>;
    static constexpr int J = Tab::S + 1, W = Rows::Q * G;
    double c[J][W];
    unsigned use[W];
    __host__ __device__ constexpr TeamForwardTable() : c(), use()
    {
        for (int s = 0; s < Rows::R * N; s++)
            for (int j = 0; j < J; j++) {
                c[j][s] = Rows::coef(s / N, j);
                use[s] |= Rows::used(s / N, j) ? 1u << j : 0u;
            }
    }
};
template <class Tab, int N, int G>
__device__ constexpr TeamForwardTable<Tab, N, G> kTeamForward{};

// v[i] for a lane-dependent i without a local array
template <int N>
__device__ __forceinline__ double pick(const double (&v)[N], int i)
{
    double r = v[0];
#pragma unroll
    for (int k = 1; k < N; k++)
        r = i == k ? v[k] : r;
    return r;
}

// A lane's part of the forward sums: its rows' coefficients, and which of
// them it holds.
template <class M, class Tab, int G>
struct TeamForward {
    static constexpr int N = M::N, NS = Tab::S;
    using Rows = TeamRows<Tab, N, G>;
    static constexpr int Q = Rows::Q, J = NS + 1;
    double c[J][Q];
    int comp[Q];
    unsigned use[Q];      // bit j: the row takes a term at j
    bool err[Q], den[Q];  // the error row, its denominator
    LaneGroup<G> team;

    __device__ __forceinline__ TeamForward()
    {
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const int s = team.index + G * q;
            comp[q] = s % N;
            use[q] = kTeamForward<Tab, N, G>.use[s];
            err[q] = s / N == Rows::rank_e;
            den[q] = s / N == Rows::rank_d;
#pragma unroll
            for (int j = 0; j < J; j++)
                c[j][q] = kTeamForward<Tab, N, G>.c[j][s];
        }
    }

    // component i of a row, to every lane
    __device__ __forceinline__ double row(const double (&acc)[Q], int rank, int i) const
    {
        const int s = rank * N + i;
        return shfl(acc[s / G], team.base + s % G, team.mask);
    }

    // acc += (c_j dt) K_j for every row that takes the term
    __device__ __forceinline__ void add(double (&acc)[Q], int j, const double (&K)[N], double dt, double atol,
                                        double rtol) const
    {
#pragma unroll
        for (int q = 0; q < Q; q++)
            if (Rows::any_used(q, j)) {
                double w = c[j][q] * dt, k = pick<N>(K, comp[q]), s = acc[q];
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
                // rows that must not take the term: y_new and the error where
                // their weight is zero, the denominator; a finished stage is
                // not read again
                const bool keep = Rows::has(q, Rows::rank_b) || Rows::has(q, Rows::rank_e) || dq;
                acc[q] = !keep || (use[q] >> j & 1u) ? s : acc[q];
            }
    }

    // attempt_pair, the results on every lane
    __device__ __forceinline__ double attempt(const double (&y)[N], const double (&k0)[N], const double (&p)[M::P],
                                              double t, double dt, double atol, double rtol, double (&ynew)[N],
                                              double (&knew)[N]) const
    {
        double acc[Q];
#pragma unroll
        for (int q = 0; q < Q; q++) {
            acc[q] = pick<N>(y, comp[q]);
            if (Rows::has(q, Rows::rank_d))
                acc[q] = den[q] ? fabs(acc[q]) : acc[q];
            if (Rows::has(q, Rows::rank_e))
                acc[q] = err[q] ? -0.0 : acc[q]; // -0 + x = x: the first term
        }
        add(acc, 0, k0, dt, atol, rtol);
#pragma unroll
        for (int m = 1; m < NS; m++) {
            double X[N], K[N];
#pragma unroll
            for (int i = 0; i < N; i++)
                X[i] = row(acc, Rows::rank_x(m), i);
            M::template rhs<double>(X, p, t + Tab::c(m) * dt, K);
            add(acc, m, K, dt, atol, rtol);
        }
#pragma unroll
        for (int i = 0; i < N; i++)
            ynew[i] = row(acc, Rows::rank_b, i);
        if constexpr (Tab::FSAL) {
            M::template rhs<double>(ynew, p, t + dt, knew);
            add(acc, NS, knew, dt, atol, rtol);
        }
        double worst = 0.0;
        if constexpr (Q == 1) {
            // every lane forms the quotient of its own component, the
            // error rows' ones are those of the components
            const int from = team.base + (Rows::rank_e * N + comp[0]) % G;
            const int dfrom = team.base + (Rows::rank_d * N + comp[0]) % G;
            const double e = shfl(acc[0], from, team.mask), d = shfl(acc[0], dfrom, team.mask);
            const double r = quotient64(fabs(e), d);
#pragma unroll
            for (int i = 0; i < N; i++)
                worst = worse(worst, shfl(r, team.base + i, team.mask));
        } else {
#pragma unroll
            for (int i = 0; i < N; i++)
                worst = worse(worst, quotient64(fabs(row(acc, Rows::rank_e, i)), row(acc, Rows::rank_d, i)));
        }
        return worst;
    }
    // the larger, a NaN kept
    __device__ __forceinline__ static double worse(double a, double b)
    {
        return is_nan64(a) ? a : is_nan64(b) ? b : max_nonneg64(a, b);
    }
};

template <class Tab, int N, int P, int G>
struct TeamBackwardTable {
    static constexpr int NS = Tab::S, SLOTS = N + P + NS * N, W = (SLOTS + G - 1) / G * G;
    double ca[NS][W], cb[W];
    __host__ __device__ constexpr TeamBackwardTable() : ca(), cb()
    {
        for (int s = N + P; s < SLOTS; s++) {
            const int k = (s - N - P) / N;
            cb[s] = Tab::b(k);
            for (int m = k + 1; m < NS; m++)
                ca[m][s] = Tab::a(m, k);
        }
    }
};
template <class Tab, int N, int P, int G>
__device__ constexpr TeamBackwardTable<Tab, N, P, G> kTeamBackward{};

// Rows of the backward sums.  Slots: lambda (N), mu (P), then K-bar_k
// component i at N + P + k N + i.  The model gives its VJP outputs o (gx, then
// gp) as w[kVjpW] W_o(x), plus w[0] for o = kVjpAdd (vjp_weights).
// SEEDS seed rows at once: H = G / SEEDS lanes each hold a seed's rows, and
// the weights serve all of them.
template <class M, class Tab, int G, int SEEDS = 1>
struct TeamBackward {
    static constexpr int H = G / SEEDS;
    static constexpr int N = M::N, P = M::PG, NS = Tab::S;
    static constexpr int SLOTS = N + P + NS * N, Q = (SLOTS + H - 1) / H;
    using Weights = double[NS][N + P];
    double ca[NS][Q]; // a_mk of the lane's K-bar_k
    double cb[Q];     // b_k
    int kind[Q];      // 0 lambda, 1 mu, 2 K-bar
    int comp[Q];      // component (lambda, K-bar) or parameter (mu)
    LaneGroup<G> team;
    int seed, rows; // the lane's seed of the team's, and the first lane with that seed's rows

    __device__ __forceinline__ TeamBackward() : seed(team.index / H), rows(team.base + team.index / H * H)
    {
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const int s = team.index % H + H * q;
            kind[q] = s < N ? 0 : s < N + P ? 1 : 2;
            comp[q] = s < N ? s : s < N + P ? s - N : (s - N - P) % N;
            cb[q] = kTeamBackward<Tab, N, P, H>.cb[s];
#pragma unroll
            for (int m = 0; m < NS; m++)
                ca[m][q] = kTeamBackward<Tab, N, P, H>.ca[m][s];
        }
    }

    // Whether accumulator q holds a row that stage m adds to
    __host__ __device__ static constexpr bool live(int q, int m)
    {
        for (int s = q * H; s < (q + 1) * H && s < SLOTS; s++)
            if (s < N + P || (s - N - P) / N < m)
                return true;
        return false;
    }
    __host__ __device__ static constexpr bool only_kbar(int q) { return q * H >= N + P; }
    __host__ __device__ static constexpr bool only_sums(int q, int m)
    {
        for (int s = q * H; s < (q + 1) * H && s < SLOTS; s++)
            if (s >= N + P && (s - N - P) / N < m)
                return false;
        return true;
    }

    // mu into its lanes, at the start of a seed
    __device__ __forceinline__ void clear(double (&mu)[Q]) const
    {
#pragma unroll
        for (int q = 0; q < Q; q++)
            mu[q] = 0.0;
    }
    __device__ __forceinline__ double param(const double (&mu)[Q], int k) const
    {
        return shfl(mu[(N + k) / H], rows + (N + k) % H, team.mask);
    }

    // VJP weights of every stage of this lane's step (back_step's recompute)
    __device__ __forceinline__ static void weights(const double (&y)[N], double tn, double h, const double (&p)[M::P],
                                                   Weights &W)
    {
        double X[N], K[NS][N];
#pragma unroll
        for (int m = 0; m < NS; m++) {
            form_stage<Tab, N, double>(m, y, y, K, h, h, X);
            if (m < NS - 1)
                M::template rhs<double>(X, p, tn + Tab::c(m) * h, K[m]);
            M::vjp_weights(X, p, W[m]);
        }
    }

    // back_step with the weights that lane `from` of the team holds and its
    // step's h: lam on every lane of the seed, mu in its lanes
    __device__ __forceinline__ void step(const Weights &W, int from, double h, double (&lam)[N], double (&mu)[Q]) const
    {
        const int src = team.base + from;
        double acc[Q];
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const double l = pick<N>(lam, comp[q]);
            acc[q] = (cb[q] * h) * l; // seeds K-bar_k = (b_k h) lambda
            if (!only_kbar(q))
                acc[q] = kind[q] == 2 ? acc[q] : kind[q] == 0 ? l : mu[q];
        }
#pragma unroll
        for (int m = NS - 1; m >= 0; m--) {
            double w[N], Wm[N + P];
#pragma unroll
            for (int i = 0; i < N; i++) {
                const int s = N + P + m * N + i;
                w[i] = shfl(acc[s / H], rows + s % H, team.mask);
            }
#pragma unroll
            for (int o = 0; o < N + P; o++)
                Wm[o] = shfl(W[m][o], src, team.mask);
#pragma unroll
            for (int q = 0; q < Q; q++)
                if (live(q, m)) {
                    // the row's VJP output: gx of its component, or gp
                    const int o = kind[q] == 1 ? N + comp[q] : comp[q];
                    double g = w[M::kVjpW] * pick<N + P>(Wm, o);
                    if constexpr (M::kVjpAdd >= 0)
                        g = o == M::kVjpAdd ? w[0] + g : g;
                    // K-bar_k + (gx a_mk) h; a row k >= m is not read again
                    double term = only_sums(q, m) ? g : (g * ca[m][q]) * h;
                    if (!only_kbar(q))
                        term = kind[q] == 2 ? term : g;
                    acc[q] = acc[q] + term;
                }
        }
#pragma unroll
        for (int i = 0; i < N; i++)
            lam[i] = shfl(acc[i / H], rows + i % H, team.mask);
#pragma unroll
        for (int q = 0; q < Q; q++)
            mu[q] = acc[q];
    }
};

// ------------------------------------------------------------ forward sweep

// forward_kernel with the step spread over a team
template <class M, class Tab, int G>
__global__ void __launch_bounds__(256) forward_team_kernel(FwdParams a)
{
    constexpr int N = M::N, P = M::P;
    constexpr int RS = record_doubles(N);
    if (gated_off(a))
        return;
    const TeamForward<M, Tab, G> tf;
    const bool first = tf.team.index == 0;
    const int CH = a.pool.chunk_len;

    int b = -1;
    double y[N], k0[N], p[P], t = 0.0, t1 = 0.0, dt = 0.0;
    int count = 0, rej = 0, fails = 0, status = ST_OK, chunk = -1, slot = 0;
    bool at_top = true;

    auto take = [&](unsigned int *counter) -> int {
        int v = 0;
        if (first)
            v = (int)atomicAdd(counter, 1u);
        return shfl(v, tf.team.base, tf.team.mask);
    };

    const int limit = a.part == SPLIT_LONG ? split_of(a) : a.B;
    auto fetch = [&]() -> bool {
        if (__shfl_sync(tf.team.mask, first && gives_up(a, G) ? 1 : 0, tf.team.base))
            return false;
        b = take(a.part == SPLIT_LONG ? &a.ctl->fwd_long : &a.ctl->fwd_next);
        if (b >= limit)
            return false;
        if (a.order)
            b = a.order[b];
#pragma unroll
        for (int i = 0; i < N; i++)
            y[i] = a.y0[(size_t)b * N + i];
#pragma unroll
        for (int k = 0; k < P; k++)
            p[k] = a.par[(size_t)b * P + k];
        t = a.t0[b];
        t1 = a.t1[b];
        dt = a.dt0;
        count = rej = fails = 0;
        status = ST_OK;
        at_top = true;
        slot = 0;
        chunk = take(&a.ctl->pool_next);
        if (chunk >= a.pool.n_chunks) {
            status = ST_CKPT_BUDGET;
            chunk = -1;
            if (first)
                atomicOr(&a.ctl->pool_fail, 1u);
        } else if (first) {
            a.pool.chunk_prev[chunk] = -1;
        }
        M::template rhs<double>(y, p, t, k0);
        return true;
    };

    // Reserve the slot of the next stored record; false if the pool ran out.
    auto reserve = [&]() -> bool {
        if (chunk < 0)
            return false;
        if (slot == CH) {
            const int c = take(&a.ctl->pool_next);
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
        if (first)
            write_record<N>(record_ptr<RS>(a.pool, chunk, slot), t, dt, y);
        slot++;
    };

    auto finish = [&]() {
        if (status == ST_OK) {
            if (reserve())
                write();
            else
                status = ST_CKPT_BUDGET;
#pragma unroll
            for (int i = 0; i < N; i++)
                if (!is_finite64(y[i]))
                    status = ST_NONFINITE;
        }
        if (!first)
            return;
        if (a.yT) {
#pragma unroll
            for (int i = 0; i < N; i++)
                a.yT[(size_t)b * N + i] = y[i];
        }
        a.inst_T[b] = count;
        a.inst_last[b] = chunk;
        a.inst_status[b] = status;
        note_work(a, b, count + rej);
        note_finished(a, b, count + rej);
        if (a.inst_t1)
            a.inst_t1[b] = t1;
        if (a.n_acc_out)
            a.n_acc_out[b] = count;
        if (a.n_rej_out)
            a.n_rej_out[b] = rej;
        if (a.status_out)
            a.status_out[b] = status;
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
        double ynew[N], knew[N];
        const double err = tf.attempt(y, k0, p, t, dt, a.atol, a.rtol, ynew, knew);
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
            accept_state<M, Tab, double>(y, y, k0, ynew, ynew, knew, p, t);
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

// outputs of an instance without a trajectory
template <int N, int P>
__device__ __forceinline__ void team_fail(const AdjParams &a, int b, int st)
{
    for (int qq = 0; qq < a.nout; qq++) {
        const size_t o = ((size_t)b * a.nout + qq);
        for (int i = 0; i < N; i++)
            a.dy0[o * N + i] = __longlong_as_double(0x7ff8000000000000ll);
        for (int k = 0; k < P; k++)
            a.dpar[o * P + k] = __longlong_as_double(0x7ff8000000000000ll);
    }
    if (a.status_out)
        a.status_out[b] = st;
}

// lambda_0 and mu of a finished seed (one lane writes)
template <int N, int P>
__device__ __forceinline__ void team_store(const AdjParams &a, int b, int q, const double (&lam)[N],
                                           const double (&mu)[P])
{
    const size_t o = ((size_t)b * a.nout + q);
    bool finite = true;
#pragma unroll
    for (int i = 0; i < N; i++) {
        a.dy0[o * N + i] = lam[i];
        finite = finite && is_finite64(lam[i]);
    }
#pragma unroll
    for (int k = 0; k < P; k++) {
        const double d = a.mu_direct ? a.mu_direct[o * P + k] : 0.0;
        a.dpar[o * P + k] = d + mu[k];
        finite = finite && is_finite64(mu[k]);
    }
    if (a.status_out && q == a.nout - 1)
        a.status_out[b] = finite ? ST_OK : ST_NONFINITE;
}

// backward_kernel with the steps spread over a team, SEEDS seed rows at once.
// Two seed rows in the halves of a warp, where one half holds a seed's rows
// (the 5(4) pairs): the recompute serves both, and the chain through lambda is
// issued once for both.
template <class M, class Tab, int G, int SEEDS = 1>
__global__ void __launch_bounds__(256) backward_team_kernel(AdjParams a)
{
    constexpr int N = M::N, P = M::P;
    constexpr int RS = record_doubles(N);
    using TB = TeamBackward<M, Tab, G, SEEDS>;
    if (gated_off(a))
        return;
    const TB tb;
    const int me = tb.team.index;
    const bool first = me == 0, writes = me % TB::H == 0;
    const int CH = a.pool.chunk_len;

    int b = -1, q = 0 /* the team's first seed */, j = -1, chunk = -1, slot = 0, T = 0, last = -1;
    int ready = 0, pos = 0; // steps whose weights the lanes hold, and the next of them
    double lam[N], mu[TB::Q], t_next = 0.0, p[P], h = 0.0;
    typename TB::Weights W;

    // weights of the steps j, j - 1, .., a lane a step
    auto prepare = [&]() {
        ready = j + 1 < G ? j + 1 : G;
        pos = 0;
        int c = chunk, s = slot - 1 - (me < ready ? me : ready - 1);
        while (s < 0) {
            c = a.pool.chunk_prev[c];
            s += CH;
        }
        double y[N], tn;
        read_record<N>(record_ptr<RS>(a.pool, c, s), tn, y);
        const double above = __shfl_up_sync(tb.team.mask, tn, 1, G);
        h = (first ? t_next : above) - tn;
        // the walk and the time go on from the block's last record
        t_next = shfl(tn, tb.team.base + ready - 1, tb.team.mask);
        chunk = shfl(c, tb.team.base + ready - 1, tb.team.mask);
        slot = shfl(s, tb.team.base + ready - 1, tb.team.mask);
        TB::weights(y, tn, h, p, W);
    };

    auto start_seed = [&]() {
        chunk = last;
        slot = T % CH;
        double yTl[N];
        read_record<N>(record_ptr<RS>(a.pool, chunk, slot), t_next, yTl);
        // an odd last seed fills the lanes of its successor too
        const int mine = q + tb.seed < a.nout ? q + tb.seed : a.nout - 1;
        const size_t o = ((size_t)b * a.nout + mine);
#pragma unroll
        for (int i = 0; i < N; i++)
            lam[i] = a.cost == 0 ? 2.0 * yTl[i] : a.cost == 1 ? 1.0 : a.lambdaT[o * N + i];
        tb.clear(mu);
        if (writes && q + tb.seed < a.nout)
            note_lambda<N>(a, b, q + tb.seed, T, lam);
        j = T - 1;
        ready = pos = 0;
    };
    const int limit = a.part == SPLIT_LONG ? split_of(a) : a.B;
    auto fetch = [&]() -> bool {
        for (;;) {
            int w = 0;
            if (first)
                w = (int)atomicAdd(a.part == SPLIT_LONG ? &a.ctl->adj_long : &a.ctl->adj_next, 1u);
            w = shfl(w, tb.team.base, tb.team.mask);
            if (w >= limit)
                return false;
            b = a.order ? a.order[w] : w;
            const int st = a.inst_status[b];
            if (st != ST_OK) {
                if (first)
                    team_fail<N, P>(a, b, st);
                continue;
            }
#pragma unroll
            for (int k = 0; k < P; k++)
                p[k] = a.par[(size_t)b * P + k];
            T = a.inst_T[b];
            last = a.inst_last[b];
            q = 0;
            start_seed();
            return true;
        }
    };

    bool alive = fetch();
    while (alive) {
        if (j < 0) {
            double m[P];
#pragma unroll
            for (int k = 0; k < P; k++)
                m[k] = tb.param(mu, k);
            if (writes && q + tb.seed < a.nout)
                team_store<N, P>(a, b, q + tb.seed, lam, m);
            if (q + SEEDS < a.nout) {
                q += SEEDS;
                start_seed();
            } else {
                alive = fetch();
            }
            continue;
        }
        if (pos == ready)
            prepare();
        tb.step(W, pos, shfl(h, tb.team.base + pos, tb.team.mask), lam, mu);
        if (writes && q + tb.seed < a.nout)
            note_lambda<N>(a, b, q + tb.seed, j, lam);
        pos++;
        j--;
    }
}

// --------------------------------------------- backward sweep, two levels

// backward_kernel_2level with a team per instance.  The segments between
// checkpoints are re-integrated G at once, a lane a segment (each from its own
// checkpoint, one lane's attempt of forward_kernel: the same bits), into the
// lanes' scratch; the back steps then run through all of them, last first,
// their recompute G steps at once as in backward_team_kernel.  Spreading one
// segment's attempts over the team instead (forward_team_kernel's step) took
// ~60 FP64 instructions per step of one instance, a lane a segment ~260 / G.
template <class M, class Tab, int G>
__global__ void __launch_bounds__(256) backward_team_kernel_2level(AdjParams a)
{
    constexpr int N = M::N, P = M::P;
    constexpr int RS = record_doubles(N);
    using TB = TeamBackward<M, Tab, G>;
    if (gated_off(a))
        return;
    const TB tb;
    const unsigned mask = tb.team.mask;
    const int me = tb.team.index, base = tb.team.base;
    const bool first = me == 0;
    const int CH = a.pool.chunk_len, SK = a.stride;
    const int segs = team_segments(G, SK);
    const size_t seg_doubles = (size_t)(SK + 1) * RS;
    // lane l's segment: team_scr + l seg_doubles, l < segs
    double *team_scr = a.scratch + ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / G * segs * seg_doubles;

    int b = -1, q = 0, j = -1, T = 0, R = 0, last = -1, chunk = -1, slot = 0;
    int top = 0, low = 0;   // the lanes hold the segments top, top - 1, .. of steps low .. j
    int ready = 0, pos = 0; // as backward_team_kernel
    double lam[N], mu[TB::Q], t1 = 0.0, t_end = 0.0, y_end[N], p[P], h = 0.0;
    typename TB::Weights W;

    // Re-integrates the segments that end with step j; false: one of them did
    // not land on its next checkpoint.
    auto reintegrate = [&]() -> bool {
        top = j / SK;
        const int cnt = top + 1 < segs ? top + 1 : segs;
        low = (top - cnt + 1) * SK;
        bool run = me < cnt;
        const int at = run ? me : cnt - 1, first_step = (top - at) * SK;
        const int L = j + 1 - first_step < SK ? j + 1 - first_step : SK;
        int c = chunk, s = slot - 1 - at; // the walk is on checkpoint top + 1
        while (s < 0) {
            c = a.pool.chunk_prev[c];
            s += CH;
        }
        const double *r = record_ptr<RS>(a.pool, c, s);
        double t, y[N], dt = r[1], te, ye[N];
        read_record<N>(r, t, y);
        // the segment's end: the next checkpoint, which the lane above starts from
        te = __shfl_up_sync(mask, t, 1, G);
        te = first ? t_end : te;
#pragma unroll
        for (int i = 0; i < N; i++) {
            const double v = __shfl_up_sync(mask, y[i], 1, G);
            ye[i] = first ? y_end[i] : v;
        }
        t_end = shfl(t, base + cnt - 1, mask);
#pragma unroll
        for (int i = 0; i < N; i++)
            y_end[i] = shfl(y[i], base + cnt - 1, mask);
        chunk = shfl(c, base + cnt - 1, mask);
        slot = shfl(s, base + cnt - 1, mask);

        double *scr = team_scr + me * seg_doubles, k0[N];
        auto keep = [&](int n) {
            double *w = scr + (size_t)n * RS;
            w[0] = t;
#pragma unroll
            for (int i = 0; i < N; i++)
                w[2 + i] = y[i];
        };
        __syncwarp(mask); // the back steps have read the segments before
        if (run)
            keep(0);
        M::template rhs<double>(y, p, t, k0);
        int done = 0, fails = 0;
        bool at_top = true, ok = true;
        while (run) {
            if (at_top) {
                if (greater_pos64((t + dt) - t1, kDblEps))
                    dt = t1 - t;
                fails = 0;
                at_top = false;
            }
            double ynew[N], ys[N], knew[N];
            const double err = attempt<M, Tab, double>(y, y, k0, p, t, dt, a.atol, a.rtol, ynew, ys, knew);
            if (is_nan64(err) || fails >= a.max_fail) {
                ok = run = false;
                continue;
            }
            fails++;
            if (greater_nonneg64(err, 1.0)) {
                dt = decrease_step<Tab, double>(dt, err, a.step_pow, &a.ctl->pow_undecided);
                continue;
            }
            t += dt;
            dt = increase_step<Tab, double>(dt, err, a.step_pow, &a.ctl->pow_undecided);
            accept_state<M, Tab, double>(y, y, k0, ynew, ynew, knew, p, t);
            at_top = true;
            done++;
            keep(done);
            if (done == L) {
                run = false;
                ok = t == te;
#pragma unroll
                for (int i = 0; i < N; i++)
                    ok = ok && y[i] == ye[i];
            }
        }
        __syncwarp(mask); // the segments are in place
        return __all_sync(mask, ok);
    };
    // step n's record in the lanes' scratch, its successor behind it
    auto step_record = [&](int n) -> const double * {
        return team_scr + (top - n / SK) * seg_doubles + (size_t)(n % SK) * RS;
    };

    auto start_seed = [&]() {
        chunk = last;
        slot = (R - 1) % CH;
        read_record<N>(record_ptr<RS>(a.pool, chunk, slot), t_end, y_end);
        const size_t o = ((size_t)b * a.nout + q);
#pragma unroll
        for (int i = 0; i < N; i++)
            lam[i] = a.cost == 0 ? 2.0 * y_end[i] : a.cost == 1 ? 1.0 : a.lambdaT[o * N + i];
        tb.clear(mu);
        if (first)
            note_lambda<N>(a, b, q, T, lam);
        j = T - 1;
        low = T;
        ready = pos = 0;
    };
    auto fetch = [&]() -> bool {
        for (;;) {
            int w = 0;
            if (first)
                w = (int)atomicAdd(&a.ctl->adj_next, 1u);
            w = shfl(w, base, mask);
            if (w >= a.B)
                return false;
            b = a.order ? a.order[w] : w;
            const int st = a.inst_status[b];
            if (st != ST_OK) {
                if (first)
                    team_fail<N, P>(a, b, st);
                continue;
            }
#pragma unroll
            for (int kk = 0; kk < P; kk++)
                p[kk] = a.par[(size_t)b * P + kk];
            T = a.inst_T[b];
            R = (T + SK - 1) / SK + 1;
            last = a.inst_last[b];
            t1 = a.inst_t1[b];
            q = 0;
            start_seed();
            return true;
        }
    };

    bool alive = fetch();
    while (alive) {
        if (j < 0) {
            double m[P];
#pragma unroll
            for (int kk = 0; kk < P; kk++)
                m[kk] = tb.param(mu, kk);
            if (first)
                team_store<N, P>(a, b, q, lam, m);
            if (q + 1 < a.nout) {
                q++;
                start_seed();
            } else {
                alive = fetch();
            }
            continue;
        }
        if (j < low && !reintegrate()) {
            if (first)
                team_fail<N, P>(a, b, ST_RECOMPUTE_MISMATCH);
            alive = fetch();
            continue;
        }
        if (pos == ready) { // weights of the steps j, j - 1, .. that the lanes hold
            ready = j + 1 - low < G ? j + 1 - low : G;
            pos = 0;
            const double *r = step_record(j - (me < ready ? me : ready - 1));
            double yj[N];
#pragma unroll
            for (int i = 0; i < N; i++)
                yj[i] = r[2 + i];
            h = r[RS] - r[0];
            TB::weights(yj, r[0], h, p, W);
        }
        tb.step(W, pos, shfl(h, base + pos, mask), lam, mu);
        if (first)
            note_lambda<N>(a, b, q, j, lam);
        pos++;
        j--;
    }
}

} // namespace va
