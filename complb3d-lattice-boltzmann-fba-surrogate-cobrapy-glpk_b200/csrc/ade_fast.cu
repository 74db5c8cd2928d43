// ade_fast.cu -- the transport step of a compiled chemistry: one launch, or
// three for a chemistry with networks on a large lattice (srg_step).
//
// For a configuration that matches a chemistry of chem.cuh every size is a
// compile-time constant, so the reaction chain of a voxel (run_kinetics +
// update_rxnLattices, abiotic + dissolution + update_abiotic_rxnLattices,
// run_equilibrium_biotic with Newton; src/complab.cpp:1252-1374) keeps its
// concentrations, increments and Newton state in registers, and the chain and
// the collide-stream of the voxel's populations run in the same thread:
//
//   per live site (one thread):
//     gather the populations of this step, sum each mobile solute's density
//     (the BGK collision keeps it, so it is the post-collision density the
//     processors read), run the chain, apply the immobile and biomass
//     increments;
//     gather again (the same slots, still in L1 / L2), collide, add t_i*dC,
//     scatter (AA pattern, in place).
//
// DRAM sees each population read once and written once.  The AA read and
// write sets of a site coincide and belong to no other site, so one thread
// owns its slots from the first gather to the scatter.
//
// The arithmetic is that of the run-time-table launches (ade_kernels.cuh)
// operation for operation, so both give the same fields.
#include "ade_kernels.cuh"
#include "chem.cuh"
#include "learned.cuh"

namespace cl {

// dissolution increments reaching voxel n (dissol_gather with the solute loop
// unrolled): the products of each phase-carrying face neighbour, and the
// voxel's own decrement at its phase substrate, in the reference's order
template <int S>
__device__ __forceinline__ void fast_dissol_gather(const AdeK& k, int64_t n, int x, int y, int z, uint8_t cls,
                                                   double (&D)[S]) {
    const AdeParams& p = k.p;
    const int64_t N = k.g.N, plane = k.g.plane, nz = k.g.nz;
    const int64_t q[7] = {n - plane, n - nz, n - 1, n, n + 1, n + nz, n + plane};
    const bool ok[7] = {x - 1 >= 1, y > 0, z > 0, (cls & F_PHASE_SELF) != 0,
                        z < k.g.nz - 1, y < k.g.ny - 1, x + 1 <= k.g.nx - 2};
#pragma unroll
    for (int j = 0; j < 7; ++j) {
        if (!ok[j]) continue;
        const int pid = k.phase[q[j]];
        if (pid == 0) continue;
        const int sM = p.phase[pid - 1].substrate;
        if (j == 3) {
            const double v = k.rel[(int64_t)sM * N + n];
#pragma unroll
            for (int s = 0; s < S; ++s) if (s == sM) D[s] += v;
            continue;
        }
#pragma unroll
        for (int s = 0; s < S; ++s)
            if (s != sM) D[s] += k.rel[(int64_t)s * N + q[j]];
    }
}

// The reaction chain of one voxel on register arrays (reaction_chain with
// the Newton solver).  C: densities, updated as each processor applies its
// increments; A: the total increment per solute.  Returns 1 if the
// equilibrium solve did not converge.
template <class Chem>
__device__ __forceinline__ int fast_chain(const AdeK& k, const typename Chem::Consts& kc, int64_t n, uint32_t sto,
                                          int x, int y, int z, uint8_t cls, double (&C)[Chem::S],
                                          double (&A)[Chem::S], const double* net_in, const double* net_out,
                                          int ncs) {
    constexpr int S = Chem::S, M = Chem::M, MW = Chem::MW, NC = Chem::NC;
    const AdeParams& p = k.p;
    const int64_t N = k.g.N;
    int nonconv = 0;
    double R[S];
    // kinetics and the surrogate networks deposit into the same increments,
    // applied together (kinetics_increments + the update of reaction_chain)
    if (p.do_kin || (Chem::kSrg && p.n_srg > 0)) {
        double B[MW], BR[MW];
#pragma unroll
        for (int m = 0; m < MW; ++m) {
            const double b = m < M ? k.bio[m * N + n] : 0.0;
            B[m] = b < THRD ? 0.0 : b;
        }
        if (p.do_kin) {
            Chem::kinetics(p, C, B, R, BR, k.mask[n]);
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const double d = R[s] * p.dt;
                R[s] = (d > THRD || d < -THRD) ? d : 0.0;
            }
#pragma unroll
            for (int m = 0; m < MW; ++m) {
                const double d = BR[m] * p.dt;
                BR[m] = (d > THRD || d < -THRD) ? d : 0.0;
            }
        } else {
#pragma unroll
            for (int s = 0; s < S; ++s) R[s] = 0.0;
#pragma unroll
            for (int m = 0; m < MW; ++m) BR[m] = 0.0;
        }
        if constexpr (Chem::kSrg) {
            if (p.n_srg > 0) Chem::combine(net_in, net_out, ncs, B, R, BR);
        }
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const double d = R[s];
            if (d > THRD || d < -THRD) { C[s] += d; A[s] += d; }
        }
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const double d = BR[m];
            if (d > THRD || d < -THRD) {
                k.bio[m * N + n] += d;
            }
        }
    }
    const bool abio = p.do_abio && (!p.surface_only || (cls & F_SURFACE));
    const bool dis = p.do_dissol && (cls & (F_PHASE_NBR | F_PHASE_SELF));
    if (abio || dis) {
        if (abio) {
            Chem::abiotic(p, C, R, k.mask[n]);
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const double d = R[s] * p.dt;
                R[s] = (d > THRD || d < -THRD) ? d : 0.0;
            }
        } else {
#pragma unroll
            for (int s = 0; s < S; ++s) R[s] = 0.0;
        }
        if (dis) fast_dissol_gather<S>(k, n, x, y, z, cls, R);
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const double d = R[s];
            if (d > THRD || d < -THRD) { C[s] += d; A[s] += d; }
        }
    }
    if constexpr (NC > 0) {
        if (!p.do_eq) return 0;
        const EqDev& e = k.e;
        const typename Chem::Tab tb{e};
        double x[NC], T[NC];
#pragma unroll
        for (int j = 0; j < NC; ++j) T[j] = 0.0;
#pragma unroll
        for (int i = 0; i < S; ++i) {
            if (!tb.active(i)) continue;
            const double c = fmin(fmax(C[i], 1e-30), 10.0);
#pragma unroll
            for (int j = 0; j < NC; ++j) {
                if constexpr (Chem::Tab::kFixed) { if (tb.ipow(i, j) == 0) continue; }
                T[j] = fma(tb.s(i, j), c, T[j]);
            }
        }
#pragma unroll
        for (int j = 0; j < NC; ++j) T[j] = fmax(T[j], 1e-30);
        int conv = 0, it = 0;
        bool warm = false;
        double xprev[NC];
        if (k.eq_x) {
            warm = true;
            bool two = true;
#pragma unroll
            for (int j = 0; j < NC; ++j) {
                xprev[j] = (double)k.eq_x[(int64_t)j * N + sto];
                warm = warm && (xprev[j] == xprev[j]);
                const double xq = (double)k.eq_xp[(int64_t)j * N + sto];
                two = two && (xq == xq);
                x[j] = xprev[j];
                if (two) x[j] = fmin(fmax(2.0 * xprev[j] - xq, -30.0), 1.0);
            }
            if (!two) {
#pragma unroll
                for (int j = 0; j < NC; ++j) x[j] = xprev[j];
            }
        }
        // the reference's cold start: log10 of each component's own species
        auto cold = [&](double* xs) {
#pragma unroll
            for (int j = 0; j < NC; ++j) {
                const int idx = e.comp_species[j];
                double c = 1e-7;
#pragma unroll
                for (int s = 0; s < S; ++s) if (s == idx) c = C[s];
                xs[j] = log10(fmin(fmax(c, 1e-30), 10.0));
            }
        };
        // no previous solution of its own: the network's guess, once trained,
        // where it is closer to equilibrium than the cold start by the relative
        // mass-balance residual (the cold start reads the voxel's own species,
        // which transport keeps near equilibrium)
        if (!warm && k.learn_w) {
            LearnVec<NC> tv;
#pragma unroll
            for (int j = 0; j < NC; ++j) tv.v[j] = T[j];
            const LearnVec<NC> xv = learn_start<NC>(k.learn_w, k.learn_norm, tv);
#pragma unroll
            for (int j = 0; j < NC; ++j) x[j] = xv.v[j];
            double xc[NC], F[NC];
            cold(xc);
            warm = eq_residual_t<NC, S>(tb, T, x, F) < eq_residual_t<NC, S>(tb, T, xc, F);
        }
        for (int phase = warm ? 0 : 1; phase < 2; ++phase) {
            if (phase == 1) cold(x);
            it += eq_newton_t<NC, S>(tb, T, x, phase == 0 ? p.eq.warm_iter : p.eq.max_iter, p.eq.tol, &conv, R, 1);
            if (conv) break;
        }
        if (k.eq_x && conv) {
#pragma unroll
            for (int j = 0; j < NC; ++j) {
                k.eq_xp[(int64_t)j * N + sto] = (float)xprev[j];
                k.eq_x[(int64_t)j * N + sto] = (float)x[j];
            }
        }
        if (k.eq_iters) k.eq_iters[n] = it;
        if (conv && k.pair_T && learn_sampled((uint32_t)n, k.pair_salt, k.pair_mask))
            learn_store<NC>(k.pair_T, k.pair_X, k.pair_count, k.pair_cap, T, x);
        if (!conv) nonconv = 1;
        else {
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const double conc = fmax(C[s], 1e-30);
                double eqc = !tb.active(s) ? fmin(conc, 10.0) : (NC <= 3 ? R[s] : species_c<NC>(e, s, x));
                eqc = fmin(fmax(eqc, 1e-30), 10.0);
                double d = eqc - conc;
                const double mx = fmax(1e-9, 0.1 * fabs(conc));
                if (fabs(d) > mx) d = d > 0 ? mx : -mx;
                if (conc + d < 1e-20) d = 1e-20 - conc;
                if (fabs(d) > THRD) { C[s] += d; A[s] += d; }
            }
        }
    }
    return nonconv;
}

// The networks of a block's voxels (chemistries with kSrg; every thread of
// the block calls it).  Biomass sits on a fraction of the voxels, so nearly
// every warp holds a few that need a network and, evaluated in place, would
// run both networks for them; the voxels of each organism are listed instead
// and the lists dealt out to the block's warps, 32 voxels of one organism at a
// time (each organism's weights stay operands of its code).  A full block so
// runs as many rounds as in place, whichever organisms fill it: with half of
// the warps to each organism, one organism everywhere held the other half
// idle (256^3, spheres of radius 4-10, porosity 0.4: 1.92 ms a step, 1.35 dealt
// out, 1.37 in place).  Both
// organisms on 13 % of the pore voxels: 2.18 ms in place, 1.42 from the lists;
// everywhere: 2.40 and 2.34.
template <class Chem, int B>
struct NetBlock {
    double in[Chem::S][B];                // thresholded densities
    double b[2][B];
    double out[2][Chem::S + 1][B];        // per organism: draws, growth
    int count[2];
    short list[2][B];
};
template <class Chem, int B>
__device__ __forceinline__ void block_networks(const AdeK& k, const typename Chem::Consts& kc, NetBlock<Chem, B>& nb,
                                               bool on, uint32_t n, const double (&C)[Chem::S]) {
    const int t = threadIdx.x;
    if (t < 2) nb.count[t] = 0;
    __syncthreads();
    if (on) {
        bool any = false;
#pragma unroll
        for (int o = 0; o < 2; ++o) {
            const double v = k.bio[o * k.g.N + n];
            const double b = v < THRD ? 0.0 : v;
            if (b > THRD) {
                nb.b[o][t] = b;
                nb.list[o][atomicAdd(&nb.count[o], 1)] = (short)t;
                any = true;
            }
        }
        if (any) {
#pragma unroll
            for (int s = 0; s < Chem::S; ++s) nb.in[s][t] = C[s] > THRD ? C[s] : 0.0;
        }
    }
    __syncthreads();
    const int chunks0 = (nb.count[0] + 31) / 32, chunks = chunks0 + (nb.count[1] + 31) / 32;
    for (int w = t >> 5; w < chunks; w += B / 32) {
        const int o = w < chunks0 ? 0 : 1;
        const int q = (w - o * chunks0) * 32 + (t & 31);
        if (q >= nb.count[o]) continue;
        const int v = nb.list[o][q];
        if (o == 0) Chem::template organism<0>(k.p, kc, &nb.in[0][v], nb.b[0][v], &nb.out[0][0][v], B);
        else Chem::template organism<1>(k.p, kc, &nb.in[0][v], nb.b[1][v], &nb.out[1][0][v], B);
    }
    __syncthreads();
}

// The same step in three launches, for large lattices.  Biomass
// sits on a fraction of the voxels and everywhere else the step is streaming
// alone: a launch that evaluates networks beside the streaming gives every
// site the registers of the networks and every warp a few lanes that need one.
// So the voxels whose chain can change anything are listed first, a second
// launch runs the chain for the list with one voxel per lane, and the
// streaming launch of the run-time table adds what that left in dc.
//   Both networks of 3-20-20-4, 256^3 (spheres of radius 5-10, porosity 0.4),
// each organism on 13 % of the pore voxels: one launch with the networks in
// place 2.12 ms a step, with a list per block of 128 voxels 1.43 ms, these
// three 1.05 ms (list 0.055, chain 0.435, streaming 0.545).  The chain waits on its gathers (isolated sectors,
// half of the copy rate) as much as on the networks; five and six blocks an
// SM were no faster (1.06, 1.10 ms: spills).
//
//   On a small lattice the launches' latencies are the step, and the list per
// block stays, up to two and a half waves of its blocks (kSplitSites).  Each organism on
// 13 %: 40x32x24 25 us a step, 64^3 (two waves) 50 against 50 with three
// launches, 96x64x64 (three) 64 against 57, 128x128x64 113 against
// 95; without biomass 64^3 27 against 45.
//
// Lists (entries of the live list): voxels with biomass of organism 0 only from
// the front of `list`, of organism 1 only from its back, all others from
// `list + cap`; so a warp of the chain runs one network, or both on voxels that
// hold both organisms.  Without biomass the chain changes nothing: every solute
// of the chemistry is mobile, so there is no dissolvable phase (a phase needs an
// immobile mineral), and its abiotic rates are zero.
constexpr int64_t kSplitSites = 5 * 148 * 4 * 128 / 2;
constexpr int kListBlock = 256, kListSites = 4;
__global__ void __launch_bounds__(kListBlock)
srg_list_kernel(const uint2* entry, uint8_t* lcls, const double* bio, int64_t N, int64_t count, uint32_t* list,
                int64_t cap, unsigned long long* total) {
    __shared__ int cnt[3];
    __shared__ unsigned long long base[3];
    const int t = threadIdx.x;
    const int64_t r0 = (int64_t)blockIdx.x * (kListBlock * kListSites) + t;
    if (t < 3) cnt[t] = 0;
    uint32_t n[kListSites];
    uint8_t cls[kListSites];
    double b[kListSites][2];
#pragma unroll
    for (int j = 0; j < kListSites; ++j) {
        const int64_t r = r0 + j * kListBlock;
        n[j] = r < count ? entry[r].x : 0u;
        cls[j] = r < count ? lcls[r] : (uint8_t)0;
    }
#pragma unroll
    for (int j = 0; j < kListSites; ++j)
#pragma unroll
        for (int o = 0; o < 2; ++o) b[j][o] = (cls[j] & F_REACTIVE) ? bio[o * N + n[j]] : 0.0;
    __syncthreads();
    int kind[kListSites], at[kListSites];
#pragma unroll
    for (int j = 0; j < kListSites; ++j) {
        // biomass below thrd reads as none: no network, no decay (b is 0 where
        // nothing reacts)
        kind[j] = -1;
        if (b[j][0] >= THRD || b[j][1] >= THRD) {
            kind[j] = b[j][0] > THRD ? (b[j][1] > THRD ? 2 : 0) : (b[j][1] > THRD ? 1 : 2);
            at[j] = atomicAdd(&cnt[kind[j]], 1);
        }
        const uint8_t want = kind[j] >= 0 ? (cls[j] | F_LISTED) : (cls[j] & ~F_LISTED);
        if (want != cls[j]) lcls[r0 + j * kListBlock] = want;
    }
    __syncthreads();
    if (t < 3) base[t] = cnt[t] ? atomicAdd(total + t, (unsigned long long)cnt[t]) : 0ull;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kListSites; ++j) {
        if (kind[j] < 0) continue;
        const int64_t q = (int64_t)base[kind[j]] + at[j];
        list[kind[j] == 0 ? q : kind[j] == 1 ? cap - 1 - q : cap + q] = (uint32_t)(r0 + j * kListBlock);
    }
}

template <class Chem, int PARITY>
__global__ void __launch_bounds__(128, 4)
srg_chain_kernel(const __grid_constant__ AdeK k, const __grid_constant__ typename Chem::Consts kc, const uint32_t* list,
                 int64_t cap, const unsigned long long* total, float* dc) {
    constexpr int S = Chem::S, NMOB = Chem::NMOB;
    static_assert(NMOB == S, "every solute of the chemistry is mobile");
    const int64_t N = k.g.N;
    const uint32_t N32 = (uint32_t)N;
    const int lane = threadIdx.x & 31;
    const int64_t c0 = total[0], c1 = total[1], c2 = total[2];
    const int64_t w0 = (c0 + 31) / 32, w1 = w0 + (c1 + 31) / 32, w2 = w1 + (c2 + 31) / 32;
    for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < w2;
         w += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        int64_t q, r;
        if (w < w0) { q = w * 32 + lane; if (q >= c0) continue; r = list[q]; }
        else if (w < w1) { q = (w - w0) * 32 + lane; if (q >= c1) continue; r = list[cap - 1 - q]; }
        else { q = (w - w1) * 32 + lane; if (q >= c2) continue; r = list[cap + q]; }
        const uint2 en = k.entry[r];
        const uint32_t n = en.x;
        const uint8_t cls = k.lcls[r];
        int x, y, z;
        decode(k.g, n, x, y, z);
        SSite st;
        if (!make_ssite<PARITY>(k.g, k.sidx, x, y, z, n, (int32_t)en.y, st)) atomicAdd(&k.counters[1], 1ull);
        double C[S], A[S], in[S], out[2 * (S + 1)];
        for_chunks<NMOB>([&](auto off, auto wd) {
            float f[wd][7];
            gather7<PARITY, wd>(k.pop + 7 * N * off, N32, st, f);
#pragma unroll
            for (int s = 0; s < S; ++s) {
                if (Chem::slot(s) < off || Chem::slot(s) >= off + wd) continue;
                float rr = 0.f;
#pragma unroll
                for (int i = 0; i < 7; ++i) rr += f[Chem::slot(s) - off][i];
                C[s] = (double)rr;
            }
        });
#pragma unroll
        for (int s = 0; s < S; ++s) {
            A[s] = 0.0;
            in[s] = C[s] > THRD ? C[s] : 0.0;
        }
        const double b0 = k.bio[n], b1 = k.bio[N + n];
        if (b0 > THRD) Chem::template organism<0>(k.p, kc, in, b0, out, 1);
        if (b1 > THRD) Chem::template organism<1>(k.p, kc, in, b1, out + S + 1, 1);
        fast_chain<Chem>(k, kc, n, st.s, x, y, z, cls, C, A, in, out, 1);
        for_chunks<NMOB>([&](auto off, auto wd) {
            using V = typename PopVec<wd>::T;
            V v;
            float* e = reinterpret_cast<float*>(&v);
#pragma unroll
            for (int s = 0; s < S; ++s)
                if (Chem::slot(s) >= off && Chem::slot(s) < off + wd) e[Chem::slot(s) - off] = (float)A[s];
            *(reinterpret_cast<V*>(dc + N * off) + st.s) = v;
        });
    }
}

// Whether a step lists its voxels: the lattice is large enough, and the last
// lists were short of 16 (c0 + c1) + 13 c2 = 12 live sites.  Above that the chain
// gathers most sites and the streaming gathers them all again.  256^3, both
// organisms on 13, 50, 75, 100 % of the pore voxels: three launches 1.12, 1.93,
// 2.49, 2.75 ms, one 1.42, 2.23, 2.39, 2.33 (the line is at 56 %); one
// organism on 13, 100 %: 0.84, 1.65 and 1.20, 1.35 (the line is at 75 %).
// With the networks in place of the lists, one launch took 2.18, 2.41, 2.40,
// 2.40 and 1.33, 1.37 ms: no share is slower than that.
//   The host learns the lists' lengths with the status words at the end of a
// call (srg_decide), and while the voxels are not listed, every kSrgRecount-th
// step lists them again.
constexpr int kSrgRecount = 32;
static bool srg_split(const Ctx* c) {
    return c->ap.n_srg > 0 && c->fast_variant == 0 && c->n_live >= kSplitSites &&
           (!c->srg_dense || c->step_index % kSrgRecount == 0);
}

template <class Chem>
int srg_step(Ctx* c, const AdeK& k, const AdeS& ks, const typename Chem::Consts& kc) {
    const int64_t cap = c->geo.N - 2 * c->geo.plane;
    unsigned long long* total = c->d_counters + 4;
    uint32_t* list = reinterpret_cast<uint32_t*>(c->d_scratch);      // 2 cap entries: 8 bytes of the scratch's 8 N
    CL_CUDA(cudaMemsetAsync(total, 0, 3 * sizeof(unsigned long long), c->stream));
    srg_list_kernel<<<grid_for(c->n_live, kListBlock * kListSites, 1 << 30), kListBlock, 0, c->stream>>>(
        c->d_lentry, c->d_lcls, c->d_bio, c->geo.N, c->n_live, list, cap, total);
    CL_LAUNCH_CHECK("srg_list_kernel");
    const int blocks = grid_for(c->n_live, 128, 148 * 8);
    if (c->ade_parity == 0) srg_chain_kernel<Chem, 0><<<blocks, 128, 0, c->stream>>>(k, kc, list, cap, total, c->d_dc);
    else srg_chain_kernel<Chem, 1><<<blocks, 128, 0, c->stream>>>(k, kc, list, cap, total, c->d_dc);
    CL_LAUNCH_CHECK("srg_chain_kernel");
    c->launches += 2;
    c->srg_listed = true;
    return launch_stream<Chem::NMOB>(c, ks, c->stream, 0, c->n_live, F_LISTED, 148 * 8);
}

template <class Chem, int PARITY, int kFastBlock, int kMinBlocks>
__global__ void __launch_bounds__(kFastBlock, kMinBlocks)
ade_fast_kernel(const __grid_constant__ AdeK k, const __grid_constant__ typename Chem::Consts kc,
                int64_t count, int any_rxn) {
    constexpr int S = Chem::S, NMOB = Chem::NMOB;
    const AdeParams& p = k.p;
    const int64_t N = k.g.N, plane = k.g.plane;
    const uint32_t N32 = (uint32_t)N;
    unsigned long long nonconv = 0;
    for (int64_t r = (int64_t)blockIdx.x * kFastBlock + threadIdx.x; r < (Chem::kSrg ? count + threadIdx.x : count);
         r += (int64_t)gridDim.x * kFastBlock) {
        // (a block with networks stays together past the end of the list)
        const bool valid = !Chem::kSrg || r < count;
        const uint2 en = k.entry[valid ? r : 0];
        const uint32_t n = en.x;
        const uint8_t cls = k.lcls[valid ? r : 0];
        const uint8_t dyn = cls & 3;
        int x, y, z;
        decode(k.g, n, x, y, z);
        SSite st;
        if (!make_ssite<PARITY>(k.g, k.sidx, x, y, z, n, (int32_t)en.y, st)) atomicAdd(&k.counters[1], 1ull);
        float dcv[NMOB];
#pragma unroll
        for (int m = 0; m < NMOB; ++m) dcv[m] = 0.f;
        const bool react = any_rxn && valid && (cls & F_REACTIVE);
        double C[S], A[S];
        if (react) {
            for_chunks<NMOB>([&](auto off, auto w) {
                float f[w][7];
                gather7<PARITY, w>(k.pop + 7 * N * off, N32, st, f);
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    if (!Chem::mobile(s) || Chem::slot(s) < off || Chem::slot(s) >= off + w) continue;
                    float rr = 0.f;
#pragma unroll
                    for (int i = 0; i < 7; ++i) rr += f[Chem::slot(s) - off][i];
                    C[s] = (double)rr;
                }
            });
#pragma unroll
            for (int s = 0; s < S; ++s) {
                if (!Chem::mobile(s)) C[s] = k.imm[(int64_t)s * N + n];
                A[s] = 0.0;
            }
        }
        const double* net_in = nullptr;
        const double* net_out = nullptr;
        if constexpr (Chem::kSrg) {
            __shared__ NetBlock<Chem, kFastBlock> nb;
            if (p.n_srg > 0) block_networks<Chem, kFastBlock>(k, kc, nb, react, n, C);
            net_in = &nb.in[0][threadIdx.x];
            net_out = &nb.out[0][0][threadIdx.x];
        }
        if (!valid) continue;
        if (react) {
            nonconv += fast_chain<Chem>(k, kc, n, st.s, x, y, z, cls, C, A, net_in, net_out, kFastBlock);
#pragma unroll
            for (int s = 0; s < S; ++s) {
                if (Chem::mobile(s)) dcv[Chem::slot(s)] = (float)A[s];
                else if (A[s] != 0.0) k.imm[(int64_t)s * N + n] += A[s];
            }
        }
        const float ux = k.u[n], uy = k.u[N + n], uz = k.u[2 * N + n];
        const bool adj = (x == 1 || x == k.g.nx - 2);
        for_chunks<NMOB>([&](auto off, auto w) {
            float f[w][7];
            gather7<PARITY, w>(k.pop + 7 * N * off, N32, st, f);
#pragma unroll
            for (int g = 0; g < w; ++g) {
                const int m = off + g;
                float rho = 0.f;
                if (dyn == BB) {
#pragma unroll
                    for (int i = 1; i < 4; ++i) { const float tmp = f[g][i]; f[g][i] = f[g][i + 3]; f[g][i + 3] = tmp; }
                } else if (dyn != NODYN) {
                    const float om = (dyn == BIO) ? p.omega_bio[m] : p.omega_pore[m];
                    collide7(f[g], om, ux, uy, uz, rho);
                } else if (adj) {
#pragma unroll
                    for (int i = 0; i < 7; ++i) rho += f[g][i];
                }
                const float d = dcv[m];
                if (d != 0.f) {
#pragma unroll
                    for (int i = 0; i < 7; ++i) f[g][i] += t7(i) * d;
                }
                if (adj && dyn != BB) {
                    const int side = (x == 1) ? 0 : 1;
                    k.rho_adj[((int64_t)m * 2 + side) * plane + (n - (int64_t)x * plane)] = rho;
                }
            }
            scatter7<PARITY, w>(k.pop + 7 * N * off, N32, st, f);
        });
    }
    for (int o = 16; o > 0; o >>= 1) nonconv += __shfl_down_sync(0xffffffffu, nonconv, o);
    if ((threadIdx.x & 31) == 0 && nonconv) atomicAdd(&k.counters[0], nonconv);
}

template <class Chem, int B, int MB>
int fast_launch(Ctx* c, const AdeK& k, const typename Chem::Consts& kc, int any_rxn) {
    // one thread per live site: the block scheduler balances the reactive
    // sites' long chains against the cheap streaming-only sites (at
    // 512x256x256, with one array per solute: 2.76 ms, against 2.83 ms with a grid of 16 waves of
    // 148 x MB blocks striding over the list and 2.90 ms with one wave)
    const int blocks = grid_for(c->n_live, B, 1 << 30);
    if (c->ade_parity == 0)
        ade_fast_kernel<Chem, 0, B, MB><<<blocks, B, 0, c->stream>>>(k, kc, c->n_live, any_rxn);
    else
        ade_fast_kernel<Chem, 1, B, MB><<<blocks, B, 0, c->stream>>>(k, kc, c->n_live, any_rxn);
    CL_LAUNCH_CHECK("ade_fast_kernel");
    return CL_OK;
}

template <class Chem>
int fast_step(Ctx* c) {
    const bool any_rxn = c->ap.do_kin || c->ap.do_abio || c->ap.do_dissol || (Chem::NC > 0 && c->ap.do_eq) ||
                         (Chem::kSrg && c->ap.n_srg > 0);
    typename Chem::Consts kc{};
    if constexpr (Chem::kSrg) {
        for (int o = 0; o < 2; ++o) {
            if (c->h_srg_params[o].size() != (size_t)Chem::kP) { set_error("surrogate network not set"); return CL_ERR_STATE; }
            for (int i = 0; i < Chem::kP; ++i) kc.w[o][i] = c->h_srg_params[o][i];
        }
    }
    int r = CL_OK;
    if (c->store_dirty && (r = store_update(c, 0))) return r;
    if (c->live_dirty && (r = build_live_list(c))) return r;
    const AdeK k = make_adek(c);
    const AdeS ks = make_ades(k);
    if (any_rxn && c->ap.do_dissol && (r = dissol_release(c, k))) return r;
    if (c->n_live > 0) {
        if ((r = timing_begin(c, CL_KERNEL_ADE_MAIN))) return r;
        const int ar = any_rxn ? 1 : 0;
        bool split = false;
        if constexpr (Chem::kSrg) {
            split = srg_split(c);
            if (split) r = srg_step<Chem>(c, k, ks, kc);
        }
        if (!split) {
            // launch shapes (threads per block x blocks per SM, which sets the
            // register cap): 128x4 measured fastest on the coupled workload
            switch (c->fast_variant) {
                case 1: r = fast_launch<Chem, 128, 3>(c, k, kc, ar); break;
                case 2: r = fast_launch<Chem, 64, 6>(c, k, kc, ar); break;
                case 3: r = fast_launch<Chem, 64, 5>(c, k, kc, ar); break;
                default: r = fast_launch<Chem, 128, 4>(c, k, kc, ar); break;
            }
            c->launches += 1;
        }
        if (r) return r;
        if ((r = timing_end(c, CL_KERNEL_ADE_MAIN))) return r;
    }
    const int bblocks = grid_for(2 * c->geo.plane, 256, 148 * 4);
    if (c->ade_parity == 0) ade_boundary_kernel<Chem::NMOB, 0><<<bblocks, 256, 0, c->stream>>>(ks);
    else ade_boundary_kernel<Chem::NMOB, 1><<<bblocks, 256, 0, c->stream>>>(ks);
    CL_LAUNCH_CHECK("ade_boundary_kernel");
    c->launches += 1;
    c->ade_parity ^= 1;
    return CL_OK;
}

int chem_match(const cl_config& cfg) {
    // microbes solved by LBM run the rate table's launches
    for (int m = 0; m < CL_MAX_MICROBES; ++m) if (cfg.microbe_carrier[m]) return 0;
    if (ChemCoupled::matches(cfg)) return ChemCoupled::kId;
    if (ChemBiotic4::matches(cfg)) return ChemBiotic4::kId;
    if (ChemZhao24::matches(cfg)) return ChemZhao24::kId;
    if (ChemSurrogate2::matches(cfg)) return ChemSurrogate2::kId;
    return 0;
}

const char* chem_name(int id) {
    switch (id) {
        case ChemCoupled::kId: return ChemCoupled::kName;
        case ChemBiotic4::kId: return ChemBiotic4::kName;
        case ChemZhao24::kId: return ChemZhao24::kName;
        case ChemSurrogate2::kId: return ChemSurrogate2::kName;
        default: return "run-time rate table";
    }
}

// whether the context holds what its compiled chemistry's step needs (a
// surrogate chemistry: both networks set, of the compiled shape); otherwise
// the step runs the run-time-table launches
bool chem_ready(const Ctx* c) {
    if (c->chem == ChemSurrogate2::kId) return ChemSurrogate2::ready(c->ap);
    return true;
}

int ade_step_fast(Ctx* c) {
    switch (c->chem) {
        case ChemCoupled::kId: return fast_step<ChemCoupled>(c);
        case ChemBiotic4::kId: return fast_step<ChemBiotic4>(c);
        case ChemZhao24::kId: return fast_step<ChemZhao24>(c);
        case ChemSurrogate2::kId: return fast_step<ChemSurrogate2>(c);
        default: set_error("no compiled chemistry selected"); return CL_ERR_STATE;
    }
}

}  // namespace cl
