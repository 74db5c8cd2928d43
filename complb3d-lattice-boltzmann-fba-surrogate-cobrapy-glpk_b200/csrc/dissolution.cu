// dissolution.cu -- mineral release of the dissolvable phases
// (surfaceDissolutionKinetics3D, src/dissolutionVOP.hh:265-435).
//
// Eight lanes per phase voxel in x = 1..nx-2, taken from a list: one to a face,
// one to the voxel itself.  Its open faces are the face
// neighbours inside x = 1..nx-2 and inside y, z (no wrap) whose mask is not
// solid or bounce-back; the water it sees is the mean solute density over them
// after this step's kinetics, which the reference applies before dissolution
// runs (complab.cpp:1252-1318), so its lane recomputes the kinetics
// increments of each open neighbour from the same pre-step state the fused
// kernel starts from.  The rate law is the table of cl_phase; at most half the
// mineral goes per step and the products scale with it.  The result is stored
// per phase voxel in rel[S][N]: the products per open face (zero where
// |released| <= thrd) and, at the phase substrate, the voxel's own decrement.
// The fused kernel gathers those records; a decrement on a solid or
// bounce-back voxel is dropped as update_abiotic_rxnLattices drops it, or with
// dissol_apply_at_walls applied here (the voxel's inventory is read by no
// other thread of this launch).
#include "ade_kernels.cuh"

namespace cl {

template <int NMOB, int PARITY>
__device__ __forceinline__ void voxel_densities(const AdeK& k, int x, int y, int z, uint32_t n, double* C) {
    const AdeParams& p = k.p;
    SSite st;
    if (!make_ssite<PARITY>(k.g, k.sidx, x, y, z, n, st)) atomicAdd(&k.counters[1], 1ull);
    const uint32_t N32 = (uint32_t)k.g.N;
    for_chunks<NMOB>([&](auto off, auto w) {
        float f[w][7];
        gather7<PARITY, w>(k.pop + 7 * k.g.N * off, N32, st, f);
#pragma unroll
        for (int g = 0; g < w; ++g) {
            float r = 0.f;
#pragma unroll
            for (int i = 0; i < 7; ++i) r += f[g][i];
            C[p.mob_index[off + g]] = (double)r;
        }
    });
    for (int s = 0; s < p.S; ++s)
        if (p.mob_slot[s] < 0) C[s] = k.imm[(int64_t)s * k.g.N + n];
}

// densities after the kinetics increments of this step (update_rxnLattices)
template <int NMOB, int PARITY>
__device__ __forceinline__ void post_kinetics(const AdeK& k, int x, int y, int z, uint32_t n, double* C) {
    const AdeParams& p = k.p;
    voxel_densities<NMOB, PARITY>(k, x, y, z, n, C);
    if (p.do_kin || p.n_srg > 0) {
        double R[CL_MAX_SOLUTES], B[CL_MAX_MICROBES], BR[CL_MAX_MICROBES];
        kinetics_increments(p, k.bio, k.g.N, n, C, 1, R, B, BR, 1);
        for (int s = 0; s < p.S; ++s) {
            const double d = R[s];
            if (d > THRD || d < -THRD) C[s] += d;
        }
    }
}

// the phase voxels of x = 1..nx-2, in any order (each releases by itself)
__global__ void dissol_list_kernel(Geo g, const uint8_t* phase, uint32_t* list, unsigned long long* count) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    for (int64_t n0 = g.plane + (int64_t)blockIdx.x * blockDim.x; n0 < g.N - g.plane; n0 += stride) {
        const int64_t n = n0 + threadIdx.x;
        const bool hit = n < g.N - g.plane && phase[n] != 0;
        const unsigned ball = __ballot_sync(0xffffffffu, hit);
        if (!ball) continue;
        unsigned long long at = 0;
        if (lane == 0) at = atomicAdd(count, (unsigned long long)__popc(ball));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (hit) list[at + __popc(ball & ((1u << lane) - 1u))] = (uint32_t)n;
    }
}

//   What bounds it: latency.  A thread that scanned every site and took a
// phase voxel's six neighbours and itself one after another held the launch
// for seven gathers and kinetics in a row, and for the read of the phase field
// (eight mobile solutes, 256x128x128: 67 -> 16 us; 512x256x256: 228 -> 16 us).
template <int NMOB, int PARITY>
__global__ void __launch_bounds__(128) dissol_release_kernel(const __grid_constant__ AdeK k, const uint32_t* list,
                                                             const unsigned long long* count) {
    const AdeParams& p = k.p;
    const int64_t N = k.g.N;
    const int nx = k.g.nx, ny = k.g.ny, nz = k.g.nz;
    const int64_t cnt = (int64_t)*count;
    const int lane = threadIdx.x & 31, f = lane & 7, g0 = lane & ~7;
    const unsigned group = 0xffu << g0;
    for (int64_t q = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3; q < cnt;
         q += ((int64_t)gridDim.x * blockDim.x) >> 3) {
        const int64_t n = list[q];
        const int pid = k.phase[n];
        if (pid == 0) continue;
        const cl_phase& ph = p.phase[pid - 1];
        const int sM = ph.substrate;
        for (int s = f; s < p.S; s += 8) k.rel[(int64_t)s * N + n] = 0.0;
        int x, y, z;
        decode(k.g, n, x, y, z);
        const bool reactive = (k.cls[n] & F_REACTIVE) != 0;
        double C[CL_MAX_SOLUTES];
        // lane f < 6: the neighbour across face f, in the reference's direction
        // order +x -x +y -y +z -z; lane 6: the voxel itself
        const int dx = f == 0 ? 1 : f == 1 ? -1 : 0, dy = f == 2 ? 1 : f == 3 ? -1 : 0, dz = f == 4 ? 1 : f == 5 ? -1 : 0;
        const int ax = x + dx, ay = y + dy, az = z + dz;
        bool open = false;
        double mineral = 0.0;
        if (f == 6) {
            if (reactive && (p.do_kin || p.n_srg > 0)) {
                post_kinetics<NMOB, PARITY>(k, x, y, z, (uint32_t)n, C);
                mineral = C[sM];
            } else {
                mineral = k.imm[(int64_t)sM * N + n];
            }
        } else if (f < 6 && ax >= 1 && ax <= nx - 2 && ay >= 0 && ay < ny && az >= 0 && az < nz) {
            const uint32_t nb = (uint32_t)(((int64_t)ax * ny + ay) * nz + az);
            const int m = k.mask[nb];
            if (m != p.solid_code && m != p.bb_code) {
                open = true;
                post_kinetics<NMOB, PARITY>(k, ax, ay, az, nb, C);
            }
        }
        __syncwarp(group);               // the zeros above come before the releases below
        mineral = __shfl_sync(group, mineral, g0 + 6);
        const unsigned opens = (__ballot_sync(group, open) >> g0) & 0x3fu;
        const int n_open = __popc(opens);
        if (!(mineral > THRD) || (n_open == 0 && p.dissol_surface_only)) continue;
        // the rate law of the phase (defineDissolutionRate as a table) on the
        // mean water of the open faces, summed in face order
        auto water = [&](int s) {
            double w = 0.0;
            for (int d = 0; d < 6; ++d) {
                const double v = __shfl_sync(group, C[s], g0 + d);
                if ((opens >> d) & 1u) w += v;
            }
            if (n_open > 0) w /= (double)n_open;
            return w < 0.0 ? 0.0 : w;
        };
        double rate = ph.k * fmax(mineral, 0.0);
        for (int j = 0; j < ph.n_mass; ++j) rate *= water(ph.mass_s[j]);
        const double mineral_r = isfinite(rate) ? -rate : 0.0;
        if (!(mineral_r < 0.0)) continue;
        double dm = mineral_r * p.dt;
        double scale = 1.0;
        const double max_remove = 0.5 * mineral;
        if (-dm > max_remove) scale = max_remove / (-dm);
        dm *= scale;
        if (!(-dm > THRD)) continue;
        if (f == 6) {
            if (reactive) k.rel[(int64_t)sM * N + n] = dm;
            else if (p.dissol_walls) k.imm[(int64_t)sM * N + n] += dm;
        }
        if (n_open == 0) continue;
        for (int s = f; s < p.S; s += 8) {
            if (s == sM) continue;
            double sr = ph.nu[s] * rate;
            if (!isfinite(sr)) sr = 0.0;
            const double released = sr * p.dt * scale;
            if (fabs(released) <= THRD) continue;
            k.rel[(int64_t)s * N + n] = released / (double)n_open;
        }
    }
}

template <int NMOB>
static int launch_release(Ctx* c, const AdeK& k) {
    const unsigned long long* count = c->d_counters + 3;
    if (c->ade_parity == 0) dissol_release_kernel<NMOB, 0><<<148 * 8, 128, 0, c->stream>>>(k, c->d_phase_list, count);
    else dissol_release_kernel<NMOB, 1><<<148 * 8, 128, 0, c->stream>>>(k, c->d_phase_list, count);
    CL_LAUNCH_CHECK("dissol_release_kernel");
    c->launches += 1;
    return CL_OK;
}

// the list of phase voxels, after anything that may have written a phase id
static int phase_list(Ctx* c) {
    if (!c->phase_dirty) return CL_OK;
    CL_CUDA(cudaMemsetAsync(c->d_counters + 3, 0, sizeof(unsigned long long), c->stream));
    dissol_list_kernel<<<grid_for(c->geo.N, 256, 148 * 8), 256, 0, c->stream>>>(c->geo, c->d_phase, c->d_phase_list,
                                                                               c->d_counters + 3);
    CL_LAUNCH_CHECK("dissol_list_kernel");
    c->phase_dirty = false;
    return CL_OK;
}

int dissol_release(Ctx* c, const AdeK& k) {
    const int r = phase_list(c);
    if (r) return r;
    switch (c->ap.n_mob) {
        case 1: return launch_release<1>(c, k);
        case 2: return launch_release<2>(c, k);
        case 3: return launch_release<3>(c, k);
        case 4: return launch_release<4>(c, k);
        case 5: return launch_release<5>(c, k);
        case 6: return launch_release<6>(c, k);
        case 7: return launch_release<7>(c, k);
        case 8: return launch_release<8>(c, k);
        default: set_error("the fused transport step supports 1..8 mobile solutes");
                 return CL_ERR_ARG;
    }
}

}  // namespace cl
