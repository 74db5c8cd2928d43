// newton_batch.cuh -- the batch Newton solve of speciation.cu (up to five
// components, up to kEqDevSpecies species), in two kernels.
//
// newton_queue_kernel: one solve per thread, the threads fed from a queue.  A
// trip of a thread's loop is one evaluation (residual, weights and Jacobian
// at its trial point) followed by whatever that point asks for: accept it,
// test convergence, factor and set the next trial, or halve the step.  The
// lanes of a warp may be in different iterations and trials; a lane whose
// solve ends takes the next one, so a warp is never held by its slowest
// solve and no trial costs the warp more than one evaluation.  An accepted
// trial is evaluated once (the run-to-the-end loops of newton.cuh evaluate
// it twice).
//   What bounds it: issue slots (62 % issue at 19 warps an SM, the FP64 pipe
//   is active 36 % of the time; an evaluation of 14 species over 5 components
//   is about 1300 instructions a warp).  The species' products read powers a,
//   a^2, 1/a, 1/a^2 of each component from a column of shared memory by slots
//   set on the host, instead of testing every exponent, and a row of zero
//   coefficients is skipped whole.  2^20 cold solves: 12.6 -> 2.15 ms.
// newton_warp_kernel: one solve per warp, for the few solves that need many
// iterations and for small batches: a lane per species, then a lane per sum,
// so an evaluation costs the latency of one species and of one chain over
// the species.  The slow solves of those 2^20: 4.9 -> 2.4 ms
// (1.8 in other draws: the slowest solve sets it).
//
// Both take the iterates of the step's loops (eq_newton) bit for bit: every sum
// runs over the species in the same order with the same fused operations, and a
// power is the same repeated product.
#pragma once
#include "newton.cuh"

namespace cl {

// The tableau as the batch kernels read it: its active species in order, each
// with the power of every component its product takes (a slot of the power
// table: 0 holds 1, 1 + 4 j + {0: a_j, 1: a_j^2, 2: 1/a_j, 3: 1/a_j^2};
// multiplying by 1 changes nothing, so no exponent is tested), and the
// components it holds.
template <int NC>
struct EqProg {
    int ns, neg;                      // active species; components some species divides by
    struct Row {
        double s[NC], logk, k10;
        int slot[NC];
        int general;                  // 1: an exponent beyond +-2 (ip), 2: a fractional one
        int mask;                     // components with a nonzero coefficient
        int unit;                     // the component of a species that is one (coefficient 1 alone), else -1
        signed char ip[8];
    } row[kEqDevSpecies];
};
template <int NC> constexpr int kSlots = 4 * NC + 1;

template <int NC>
inline EqProg<NC> eq_prog(const EqDev& e) {
    EqProg<NC> p{};
    for (int j = 0; j < NC; ++j) if (e.neg[j]) p.neg |= 1 << j;
    for (int i = 0; i < e.ns; ++i) {
        if (!e.active[i]) continue;
        auto& r = p.row[p.ns++];
        r.logk = e.logk[i];
        r.k10 = e.k10[i];
        r.general = e.all_int ? 0 : 2;
        for (int j = 0; j < NC; ++j) {
            const int q = e.ipow[i][j];
            r.s[j] = e.stoich[i][j];
            r.ip[j] = (signed char)q;
            if (r.s[j] != 0.0) r.mask |= 1 << j;
            if (!e.all_int || q == 0) continue;
            if (q > 2 || q < -2) r.general = 1;
            else r.slot[j] = 1 + 4 * j + (q > 0 ? q - 1 : 1 - q);
        }
        r.unit = -1;
        for (int j = 0; j < NC; ++j) if (r.mask == 1 << j && r.s[j] == 1.0 && e.all_int) r.unit = j;
    }
    return p;
}

// a species whose product the slots do not hold: the repeated products of
// species_eval, or 10^lc where a coefficient is not an integer
template <int NC, class Pow>
__device__ __noinline__ double general_species(int general, double k10, double lc, const signed char* ip, Pow pw) {
    if (general == 2) return cl_exp10(lc);
    double c = k10;
    for (int j = 0; j < NC; ++j) {
        const int q = ip[j];
        if (q == 0) continue;
        const double b = pw(1 + 4 * j + (q > 0 ? 0 : 2));
        double v = b;
        for (int k = 1; k < (q > 0 ? q : -q); ++k) v *= b;
        c *= v;
    }
    return c;
}

// Residual F = S^T c - T (F holds -T), weights |S|^T c and the lower triangle
// of S^T diag(c) S at xt.  pw: this thread's column for the powers.  A
// coefficient that is zero adds nothing, so its terms are left out.
template <int NC, int BLOCK>
__device__ __forceinline__ void batch_eval(const EqProg<NC>& p, const double (&xt)[NC], double (*pw)[BLOCK], int t,
                                           double (&F)[NC], double (&sc)[NC], double (&J)[NC][NC]) {
#pragma unroll
    for (int j = 0; j < NC; ++j) {
        const double a = cl_exp10(xt[j]);
        pw[1 + 4 * j][t] = a;
        pw[2 + 4 * j][t] = a * a;
        if ((p.neg >> j) & 1) {
            const double ai = 1.0 / a;
            pw[3 + 4 * j][t] = ai;
            pw[4 + 4 * j][t] = ai * ai;
        }
    }
#pragma unroll 1
    for (int i = 0; i < p.ns; ++i) {
        const auto& r = p.row[i];
        const int u = r.unit;
        if (u >= 0) {
            double x = xt[0];
#pragma unroll
            for (int j = 1; j < NC; ++j) if (u == j) x = xt[j];
            const double lc = r.logk + x;
            double c = r.k10 * pw[1 + 4 * u][t], cj = c;
            if (lc > 1.0) { c = 10.0; cj = 0.0; }
            if (lc < -30.0) { c = 1e-30; cj = 0.0; }
#pragma unroll
            for (int a = 0; a < NC; ++a)
                if (u == a) { F[a] += c; sc[a] += c; J[a][a] += cj; }
            continue;
        }
        double s[NC], lc = r.logk;
#pragma unroll
        for (int j = 0; j < NC; ++j) { s[j] = r.s[j]; lc = fma(s[j], xt[j], lc); }
        double c = r.k10;
#pragma unroll
        for (int j = 0; j < NC; ++j) c *= pw[r.slot[j]][t];
        if (r.general) c = general_species<NC>(r.general, r.k10, lc, r.ip, [&](int q) { return pw[q][t]; });
        double cj = c;
        if (lc > 1.0) { c = 10.0; cj = 0.0; }
        if (lc < -30.0) { c = 1e-30; cj = 0.0; }
        const int m = r.mask;
#pragma unroll
        for (int a = 0; a < NC; ++a) {
            if (!((m >> a) & 1)) continue;
            F[a] = fma(s[a], c, F[a]);
            sc[a] = fma(fabs(s[a]), c, sc[a]);
            const double sac = s[a] * cj;
#pragma unroll
            for (int b = 0; b <= a; ++b) J[a][b] = fma(sac, s[b], J[a][b]);
        }
    }
}

// What a phase (the warm start, the cold start) solves and where its results
// go.  Systems come from in_list (all n where it is null), each from its
// logfree row, for at most `limit` iterations.  A solve that fails goes to
// fail_list when the phase has a fallback, else its status is 2.  A solve the
// queue kernel hands on goes to cont_list with its iterations so far above
// kEntryBits, and its point back to logfree.
struct NewtonJob {
    const double* totals;
    double* logfree;
    int32_t* iters;
    uint8_t* status;
    const int64_t* in_list;
    const unsigned long long* in_count;
    int64_t n;
    int64_t* fail_list;
    unsigned long long* fail_count;
    int64_t* cont_list;
    unsigned long long* cont_count;
    unsigned long long* queue;      // next entry to take (newton_queue_kernel)
    double tol;
    int limit, ok_status, fallback, add_iters;
};
constexpr int kEntryBits = 44;      // systems below 2^44, iterations above

// lists at most this long run one solve per warp throughout (8000 cold
// systems of the 5 x 14 tableau: 1.04 ms; 9000 through the queue: 1.35 ms; one
// to three components: the same on either side, 8192 and 8193 systems within
// 0.07 and 0.08 to 1.16 and 1.13 ms)
constexpr int64_t kWarpListMax = 8192;
// evaluations after which the queue kernel hands a solve on: all but 0.5 % of
// the cold solves of the 5 x 14 tableau need fewer (the median 15), and the
// few that search their line ten trials deep in every one of 200 iterations
// would hold the launch.  Where many pass it the warp kernel takes most of the
// time and the batch is still faster than before there were two kernels: 2^20
// solves of three components, 22 % of them without a root, 61 -> 44 ms; 5 x 14
// with half of the totals drawn at random, 76 -> 11.6 ms.
constexpr int kQueueEvals = 32;
constexpr int kQueueBlock = 128, kWarpBlock = 32;

__device__ __forceinline__ void newton_finish(const NewtonJob& jb, int64_t k, int it, bool conv) {
    if (jb.iters) jb.iters[k] = (jb.add_iters ? jb.iters[k] : 0) + it;
    if (conv) { if (jb.status) jb.status[k] = (uint8_t)jb.ok_status; }
    else if (jb.fallback) jb.fail_list[atomicAdd(jb.fail_count, 1ull)] = k;
    else if (jb.status) jb.status[k] = 2;
}

template <int NC>
__global__ void __launch_bounds__(kQueueBlock, 5)
newton_queue_kernel(const __grid_constant__ EqProg<NC> e, const __grid_constant__ NewtonJob jb) {
    // a column of shared memory per thread: the powers, then T, x, d, w
    __shared__ double sh[kSlots<NC> + 4 * NC][kQueueBlock];
    const int64_t cnt = jb.in_list ? (int64_t)*jb.in_count : jb.n;
    if (cnt <= kWarpListMax) return;
    const int t = threadIdx.x, lane = t & 31;
    double (*sT)[kQueueBlock] = sh + kSlots<NC>;
    double (*sx)[kQueueBlock] = sh + kSlots<NC> + NC;
    double (*sd)[kQueueBlock] = sh + kSlots<NC> + 2 * NC;
    double (*sw)[kQueueBlock] = sh + kSlots<NC> + 3 * NC;
    int64_t k = -1;                   // this lane's system, -1: none
    int it = 0, ls = -1, evals = 0;   // iterations done; trial of the line search, -1: a fresh start
    double fn = 0.0, alpha = 1.0, xt[NC];
#pragma unroll
    for (int j = 0; j < NC; ++j) { xt[j] = 0.0; sT[j][t] = 1.0; }
    sh[0][t] = 1.0;
    int64_t pos = 0, end = 0;         // entries this warp holds from the queue
    bool drained = false;
    for (;;) {
        // lanes without a solve take the next entries
        unsigned need = __ballot_sync(0xffffffffu, k < 0);
        while (need && !(drained && pos == end)) {
            if (pos == end) {
                unsigned long long p = 0;
                if (lane == 0) p = atomicAdd(jb.queue, 32ull);
                p = __shfl_sync(0xffffffffu, p, 0);
                if ((int64_t)p >= cnt) { drained = true; break; }
                pos = (int64_t)p;
                end = min(pos + 32, cnt);
            }
            const int64_t mine = pos + __popc(need & ((1u << lane) - 1u));
            if (((need >> lane) & 1u) && mine < end) {
                k = jb.in_list ? jb.in_list[mine] : mine;
#pragma unroll
                for (int j = 0; j < NC; ++j) { sT[j][t] = jb.totals[k * NC + j]; xt[j] = jb.logfree[k * NC + j]; }
                it = 0;
                ls = -1;
                evals = 0;
            }
            pos = min(pos + __popc(need), end);
            need = __ballot_sync(0xffffffffu, k < 0);
        }
        if (need == 0xffffffffu) return;
        double F[NC], sc[NC], J[NC][NC];
#pragma unroll
        for (int a = 0; a < NC; ++a) {
            F[a] = -sT[a][t]; sc[a] = 0.0;
#pragma unroll
            for (int b = 0; b < NC; ++b) J[a][b] = 0.0;
        }
        batch_eval<NC, kQueueBlock>(e, xt, sh, t, F, sc, J);
        if (k < 0) continue;
        ++evals;
        // the trial's verdict: move to it, or halve the step
        bool stuck = false;
        if (ls >= 0) {
            double fnt = 0.0;
#pragma unroll
            for (int a = 0; a < NC; ++a) { const double r = F[a] * sw[a][t]; fnt = fma(r, r, fnt); }
            const double q = fma(-1e-4, alpha, 1.0);
            if (!(fnt < fn * (q * q))) {
                if (ls == 39) stuck = true;          // the last trial: the solve stops there
                else {
                    alpha *= 0.5;
                    ++ls;
#pragma unroll
                    for (int a = 0; a < NC; ++a) xt[a] = fmin(fmax(fma(alpha, sd[a][t], sx[a][t]), -30.0), 1.0);
                    if (evals >= kQueueEvals) {      // from the last point accepted
#pragma unroll
                        for (int j = 0; j < NC; ++j) jb.logfree[k * NC + j] = sx[j][t];
                        jb.cont_list[atomicAdd(jb.cont_count, 1ull)] = k | ((int64_t)it << kEntryBits);
                        k = -1;
                    }
                    continue;
                }
            }
            ++it;
        }
        double rel = 0.0, w[NC];
        fn = 0.0;
#pragma unroll
        for (int a = 0; a < NC; ++a) {
            w[a] = 1.0 / fmax(sc[a], 1e-300);
            const double r = fabs(F[a]) * w[a];
            rel = (r > rel || r != r) ? r : rel;
            fn = fma(r, r, fn);
        }
        const bool conv = rel <= jb.tol;
        bool done = conv || !(rel < 1e300) || stuck || it >= jb.limit;
        if (!done) {
            double d[NC];
            if (!newton_direction<NC>(F, J, d)) { done = true; ++it; }
            else {
                alpha = 1.0;
                ls = 0;
#pragma unroll
                for (int a = 0; a < NC; ++a) {
                    sx[a][t] = xt[a];
                    sd[a][t] = d[a];
                    sw[a][t] = w[a];
                    xt[a] = fmin(fmax(d[a] + xt[a], -30.0), 1.0);
                }
            }
        }
        if (done) {
#pragma unroll
            for (int j = 0; j < NC; ++j) jb.logfree[k * NC + j] = xt[j];
            newton_finish(jb, k, it, conv);
            k = -1;
        }
    }
}

// One solve per warp.  A point's species go one to a lane, then its sums one
// to a lane (F, |S|^T c, the Jacobian's lower triangle), each over the
// species in order; every lane then takes all sums and does the rest alike.
// The line search runs 32 / NC trials at a time, NC lanes to a trial (a power
// each, the species dealt out, a residual each): where the full step fails,
// and from the full step on where the iteration before needed more than that.
// Runs the phase's systems when they are few, else the solves the queue
// kernel handed on.
//   What bounds it: latency.  A stalled solve is 200 iterations in a row, each
// a chain of dependent FP64 operations (exp10, products, 14 sums deep, the
// factorisation, two or three passes of trials), and the slowest solve is the
// launch; so independent species and trials are spread over lanes, no
// exponent is branched on, and an accepted trial's species are not evaluated
// again.
template <int NC>
__global__ void __launch_bounds__(kWarpBlock)
newton_warp_kernel(const __grid_constant__ EqProg<NC> e, const __grid_constant__ NewtonJob jb) {
    constexpr int kG = 32 / NC;       // trials at a time
    constexpr int kU = 3;             // species of a lane evaluated together
    __shared__ double sS[kEqDevSpecies][NC], sK[2][kEqDevSpecies];
    __shared__ int sSlot[kEqDevSpecies][NC], sGen[kEqDevSpecies];
    __shared__ signed char sIp[kEqDevSpecies][8];
    constexpr int kW = kWarpBlock / 32;
    __shared__ double sPow[kW][kG][kSlots<NC>], sC[kW][kG][kEqDevSpecies], sAcc[kW][32];
    const int64_t in = jb.in_list ? (int64_t)*jb.in_count : jb.n;
    const bool whole = in <= kWarpListMax;
    const int64_t* list = whole ? jb.in_list : jb.cont_list;
    const int64_t cnt = whole ? in : (int64_t)*jb.cont_count;
    for (int i = threadIdx.x; i < kEqDevSpecies; i += blockDim.x) {
        for (int j = 0; j < NC; ++j) { sS[i][j] = e.row[i].s[j]; sSlot[i][j] = e.row[i].slot[j]; }
        sK[0][i] = e.row[i].logk;
        sK[1][i] = e.row[i].k10;
        sGen[i] = e.row[i].general;
        for (int j = 0; j < 8; ++j) sIp[i][j] = e.row[i].ip[j];
    }
    for (int i = threadIdx.x; i < kW * kG; i += blockDim.x) sPow[i / kG][i % kG][0] = 1.0;
    __syncthreads();
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, ns = e.ns;
    // this lane's trial and component in the line search
    const int tg = lane / NC, tj = lane - tg * NC, t0 = tg < kG ? tg * NC : 0;
    // this lane's sum
    int qa = 0, qb = 0, kind = 3;
    if (lane < NC) { kind = 0; qa = lane; }
    else if (lane < 2 * NC) { kind = 1; qa = lane - NC; }
    else {
        int r = lane - 2 * NC;
#pragma unroll
        for (int a = 0; a < NC; ++a)
#pragma unroll
            for (int b = 0; b <= a; ++b) { if (r == 0) { kind = 2; qa = a; qb = b; } --r; }
    }
    const int64_t stride = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t q = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < cnt; q += stride) {
        const int64_t entry = list ? list[q] : q;
        const int64_t k = entry & ((1ll << kEntryBits) - 1);
        int it = (int)(entry >> kEntryBits);
        double T[NC], x[NC], xt[NC], d[NC], w[NC], F[NC], J[NC][NC];
#pragma unroll
        for (int j = 0; j < NC; ++j) { T[j] = jb.totals[k * NC + j]; xt[j] = jb.logfree[k * NC + j]; x[j] = xt[j]; d[j] = 0.0; w[j] = 0.0; }
        double fn = 0.0;
        double Tq = 0.0, Tj = T[0];
#pragma unroll
        for (int j = 0; j < NC; ++j) {
            if (kind == 0 && qa == j) Tq = -T[j];
            if (tj == j) Tj = T[j];
        }
        // the species of `step` lanes' stride from `first` at the point xs, whose
        // powers are in pw, into cs; a species at a clamp bound is stored negative
        auto species = [&](const double* xs, const double* pw, double* cs, int first, int step) {
            for (int i0 = first; i0 < ns; i0 += kU * step) {
                double lc[kU], c[kU];
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    const int i = min(i0 + u * step, kEqDevSpecies - 1);
                    lc[u] = sK[0][i];
                    c[u] = sK[1][i];
#pragma unroll
                    for (int j = 0; j < NC; ++j) {
                        lc[u] = fma(sS[i][j], xs[j], lc[u]);
                        c[u] *= pw[sSlot[i][j]];
                    }
                }
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    const int i = i0 + u * step;
                    if (i < ns) {
                        if (sGen[i]) c[u] = general_species<NC>(sGen[i], sK[1][i], lc[u], sIp[i], [&](int s) { return pw[s]; });
                        if (lc[u] > 1.0) c[u] = -10.0;
                        if (lc[u] < -30.0) c[u] = -1e-30;
                        cs[i] = c[u];
                    }
                }
            }
        };
        // the powers of component j at x into its slots
        auto powers = [&](double* pw, int j, double xj) {
            const double a = cl_exp10(xj), ai = 1.0 / a;
            pw += 1 + 4 * j;
            pw[0] = a; pw[1] = a * a; pw[2] = ai; pw[3] = ai * ai;
        };
        // F, |S|^T c (into sc) and J from a trial's species
        auto sums = [&](const double* cs, double (&sc)[NC]) {
            double acc = Tq;
#pragma unroll 7
            for (int i = 0; i < ns; ++i) {
                const double cv = cs[i], ci = fabs(cv), cj = cv < 0.0 ? 0.0 : cv;
                const double sa = sS[i][qa], sb = sS[i][qb];
                const double sac = sa * cj;
                acc = fma(kind == 2 ? sac : kind == 0 ? sa : fabs(sa), kind == 2 ? sb : ci, acc);
            }
            sAcc[wp][lane] = acc;
            __syncwarp();
#pragma unroll
            for (int a = 0; a < NC; ++a) { F[a] = sAcc[wp][a]; sc[a] = sAcc[wp][NC + a]; }
            int at = 2 * NC;
#pragma unroll
            for (int a = 0; a < NC; ++a)
#pragma unroll
                for (int b = 0; b <= a; ++b) J[a][b] = sAcc[wp][at++];
            __syncwarp();
        };
        bool conv = false, deep = false, accepted = true, fresh = true;
        for (;;) {
            double sc[NC];
            // the next point and its sums: the start, the full step, or the first
            // trial alpha = 2^-k, k = 0 .. 39, that passes (else the last one)
            bool known = fresh;
            if (fresh || !deep) {
                if (lane < NC) {
                    double xj = xt[0];
#pragma unroll
                    for (int j = 1; j < NC; ++j) if (lane == j) xj = xt[j];
                    powers(sPow[wp][0], lane, xj);
                }
                __syncwarp();
                species(xt, sPow[wp][0], sC[wp][0], lane, 32);
                __syncwarp();
                sums(sC[wp][0], sc);
                if (!fresh) {
                    double fnt = 0.0;
#pragma unroll
                    for (int a = 0; a < NC; ++a) { const double r = F[a] * w[a]; fnt = fma(r, r, fnt); }
                    const double q1 = 1.0 - 1e-4;
                    known = fnt < fn * (q1 * q1);
                }
            }
            if (!known) {
                double xj = x[0], dj = d[0], wj = w[0];
#pragma unroll
                for (int j = 1; j < NC; ++j) if (tj == j) { xj = x[j]; dj = d[j]; wj = w[j]; }
                int src = 0;
                accepted = false;
                for (int base = deep ? 0 : 1; base < 40 && !accepted; base += kG) {
                    const int kk = min(base + tg, 39);
                    const bool on = tg < kG && base + tg < 40;
                    // 2^-kk through the exponent field
                    const double alpha = __longlong_as_double((long long)(1023 - kk) << 52);
                    const double xkj = fmin(fmax(fma(alpha, dj, xj), -30.0), 1.0);
                    if (on) powers(sPow[wp][tg], tj, xkj);
                    double xk[NC];
#pragma unroll
                    for (int j = 0; j < NC; ++j) xk[j] = __shfl_sync(kAll, xkj, t0 + j);
                    __syncwarp();
                    if (on) species(xk, sPow[wp][tg], sC[wp][tg], tj, NC);
                    __syncwarp();
                    double Fj = -Tj;
                    if (on) {
#pragma unroll 7
                        for (int i = 0; i < ns; ++i) Fj = fma(sS[i][tj], fabs(sC[wp][tg][i]), Fj);
                    }
                    const double rj = Fj * wj;
                    double fk = 0.0;
#pragma unroll
                    for (int a = 0; a < NC; ++a) { const double r = __shfl_sync(kAll, rj, t0 + a); fk = fma(r, r, fk); }
                    const double qq = fma(-1e-4, alpha, 1.0);
                    const unsigned bal = __ballot_sync(kAll, on && fk < fn * (qq * qq));
                    accepted = bal != 0;
                    src = bal ? (__ffs(bal) - 1) / NC : min(39 - base, kG - 1);
#pragma unroll
                    for (int a = 0; a < NC; ++a) xt[a] = __shfl_sync(kAll, xk[a], src * NC);
                    deep = !accepted || base + src > 0;
                }
                sums(sC[wp][src], sc);
            }
            if (!fresh) ++it;
            fresh = false;
            bool bad = false;
            conv = true;
            fn = 0.0;
#pragma unroll
            for (int a = 0; a < NC; ++a) {
                x[a] = xt[a];
                w[a] = 1.0 / fmax(sc[a], 1e-300);
                const double r = fabs(F[a]) * w[a];
                conv = conv && r <= jb.tol;
                bad = bad || !(r < 1e300);
                fn = fma(r, r, fn);
            }
            // a point no trial of which was accepted ends the solve
            if (conv || bad || !accepted || it >= jb.limit) break;
            if (!newton_direction<NC>(F, J, d)) { ++it; break; }
#pragma unroll
            for (int a = 0; a < NC; ++a) xt[a] = fmin(fmax(d[a] + x[a], -30.0), 1.0);
        }
        __syncwarp();                    // every lane has read iters[k] and the list
        if (lane == 0) {
#pragma unroll
            for (int j = 0; j < NC; ++j) jb.logfree[k * NC + j] = x[j];
            newton_finish(jb, k, it, conv);
        }
        __syncwarp();
    }
}

// the reference's cold start of the listed systems into logfree
template <int NC>
__global__ void newton_cold_kernel(const __grid_constant__ EqDev e, const double* cold_species, double* logfree,
                                   const int64_t* in_list, const unsigned long long* in_count, int64_t n) {
    const int64_t cnt = in_list ? (int64_t)*in_count : n;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < cnt; q += (int64_t)gridDim.x * blockDim.x) {
        const int64_t k = in_list ? in_list[q] : q;
        double x[NC];
        eq_cold_start<NC>(e, cold_species + k * e.ns, x);
#pragma unroll
        for (int j = 0; j < NC; ++j) logfree[k * NC + j] = x[j];
    }
}

}  // namespace cl
