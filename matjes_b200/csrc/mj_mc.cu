// Metropolis Monte Carlo on the device (Metropolis-MC/MCstep.f90).
//
// The reference makes single-spin moves at random sites (choose_spin.f90).
// Here a sweep moves every site once, colour by colour with a colouring in
// which no coupling joins two sites of one colour, so the moves of a colour are
// independent and run in parallel: the same single-spin moves and acceptance
// rule (mj_mc.cuh) in another site order.  Two families of colourings are
// searched and the one with fewer colours kept: linear, colour (x + b y + c z)
// mod q (2 colours for square and cubic nearest neighbours, 3 for triangular),
// and product, colour (x mod cx, y mod cy, z mod cz); a periodic size must keep
// the colour of its wrapped images.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "mj_device.cuh"
#include "mj_internal.hpp"
#include "mj_mc.cuh"

namespace mj {
namespace {

// The chain's state on the device during a call: accepted moves, the running
// totals (E, summed spins), the cone and its cosine (updated after every sweep).
struct McChain {
    unsigned long long acc;
    unsigned int counter[2];
    double run[4];
    double cone, cos_cone;
};

struct McCoef {
    double kT;          // eV
    double inv_kT;      // 1/kT (0 at T = 0)
    McChain* chain;
    const double* tab;  // sin/cos tables (the plan's thermal-draw tables)
    double* track;      // tracked totals: per-block partials [4][track_n] of (dE, dm) of accepted moves, or null
    int track_n;        // partials per component (colours x blocks of a sweep)
    int track_off;      // the first partial of this colour's blocks
    int proposal;       // MJ_MC_*
    uint32_t keys[20];  // Philox round keys of the seed
    uint32_t sweep;
    uint32_t stream;
};

// S: the plan's compile-time stencil shape, void for runtime offsets
template <class S>
__global__ void __launch_bounds__(32 * kMcBY, 8) k_mc_color(const __grid_constant__ StencilParams P, const double* __restrict__ bmap,
                                                  double* m, const McCoef C, const McClass K) {
    const int y = K.ry + K.sy * static_cast<int>(blockIdx.y * kMcBY + threadIdx.y);
    const int z = K.rz + K.sz * static_cast<int>(blockIdx.z);
    const int x = mc_class_x(K, y, z, static_cast<int>(blockIdx.x * 32 + threadIdx.x));
    bool acc = false;
    double dE = 0.0;
    double3 dm = make_double3(0.0, 0.0, 0.0);
    if (x < P.L[0] && y < P.L[1] && z < P.L[2]) {
        const int64_t N = static_cast<int64_t>(P.L[0]) * P.L[1] * P.L[2];
        const int64_t i = x + static_cast<int64_t>(P.L[0]) * (y + static_cast<int64_t>(P.L[1]) * z);
        const double3 s = ld3(m, i, N);
        const double3 Pf = pair_field<S>(P, m, N, P.L[0], P.L[1], P.L[2], x, y, z);
        double3 sn;
        acc = mc_move(P, C.keys, C.tab, C.proposal, C.kT, C.inv_kT, __ldg(&C.chain->cos_cone), static_cast<uint32_t>(i), C.sweep,
                      C.stream, s, Pf, zeeman(P, bmap, i, N), sn, dE);
        if (acc) {
            st3(m, i, N, sn);
            dm = make_double3(sn.x - s.x, sn.y - s.y, sn.z - s.z);
        }
    }
    if (C.track) {  // the block's share of the change of the totals (track_val, MCstep.f90:60-68)
        double v[4] = {acc ? dE : 0.0, dm.x, dm.y, dm.z};
        const int bid = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
        block_partials<4>(v, C.track, C.track_n, C.track_off + bid);
    }
    // accepted moves of the block, added once per block (an integer sum: any order gives the same count)
    const int n = __syncthreads_count(acc);
    if (threadIdx.x == 0 && threadIdx.y == 0 && n) atomicAdd(&C.chain->acc, static_cast<unsigned long long>(n));
}

// Sum of the spins (per-block partials summed in block order by the last block).
// Four blocks per SM walk the lattice: with one partial per 256 sites the last
// block's ordered sum was most of the launch (1024^2: 16.4 us, now 9.7).
constexpr int kMagBlocksPerSm = 4;
__global__ void __launch_bounds__(256) k_mc_magnetisation(const double* __restrict__ m, int64_t N, double* partials,
                                                          unsigned int* counter, double* out, int nblocks) {
    double v[3] = {0.0, 0.0, 0.0};
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
#pragma unroll 4
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < N; i += stride) {
        v[0] += m[i];
        v[1] += m[N + i];
        v[2] += m[2 * N + i];
    }
    grid_reduce<3>(v, partials, counter, out, nblocks);
}

// The end of a sweep, one launch instead of a one-block sum and a host round
// trip: block q < 4 (with partials) adds component q of the sweep's partials, in
// a fixed order, to the running total and copies it to E_out / M_out when given;
// the last block applies the cone rule of sample_sphere (track_value.f90
// cone_update: +-1e-4 per move toward an acceptance rate of 0.5, cone in
// [0.01, pi]) to the sweep's number of moves and the running rate.  1024^2, cone
// adapted and totals recorded after every sweep: 2.6 us, where the one-block sum
// took 15 and the round trip for the host's cone rule about 20; a sweep 82 -> 51 us.
constexpr int kMcEndThreads = 1024;
__global__ void __launch_bounds__(kMcEndThreads) k_mc_sweep_end(const double* __restrict__ partials, int n, McChain* chain,
                                                                double* E_out, double* M_out, int adapt,
                                                                long long accepted0, long long proposed, double step) {
    if (blockIdx.x + 1 == gridDim.x) {
        if (threadIdx.x == 0 && adapt) {
            const double rate = static_cast<double>(accepted0 + static_cast<long long>(chain->acc)) / static_cast<double>(proposed);
            double c = chain->cone;
            if (rate > 0.5 && c < kPi) c = fmin(kPi, __dadd_rn(c, step));
            else if (rate < 0.5 && c > 0.01) c = fmax(0.01, __dsub_rn(c, step));
            chain->cone = c;
            chain->cos_cone = cos(c);
        }
        return;
    }
    const int q = blockIdx.x, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __shared__ double wsum[kMcEndThreads / 32];
    double s = 0.0;
    for (int b = threadIdx.x; b < n; b += kMcEndThreads) s += __ldcg(partials + static_cast<int64_t>(q) * n + b);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) wsum[wid] = s;
    __syncthreads();
    if (wid != 0) return;
    s = wsum[lane];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) {
        const double t = chain->run[q] + s;
        chain->run[q] = t;
        if (q == 0 && E_out) *E_out = t;
        if (q > 0 && M_out) M_out[q - 1] = t;
    }
}

}  // namespace
}  // namespace mj

using namespace mj;

extern "C" {

mj_status mj_mc_sweeps(mj_plan* plan, double* m, mj_mc_params* p, int32_t nsweeps, double* E_dev, double* M_dev,
                       int64_t* accepted, int32_t* colors, void* stream) {
    if (!plan || !m || !p || nsweeps < 0) return set_error(MJ_ERR_ARG, "bad Monte Carlo arguments");
    if (!plan->is_stencil || plan->dip_on)
        return set_error(MJ_ERR_UNSUPPORTED, "Monte Carlo sweeps need a single-atom stencil plan, no dipolar term");
    if (p->proposal < MJ_MC_CONE || p->proposal > MJ_MC_OVERRELAX) return set_error(MJ_ERR_ARG, "unknown proposal");
    if (!(p->temperature >= 0.0) || !(p->cone > 0.0)) return set_error(MJ_ERR_ARG, "temperature >= 0 and cone > 0");
    int col[4] = {0, 0, 0, 0};
    if (!mc_colouring(plan->sp, plan->sp.L, 1, col))
        return set_error(MJ_ERR_UNSUPPORTED, "no linear or product colouring fits the stencil and the periodic "
                                             "sizes");
    if (colors)
        for (int d = 0; d < 4; ++d) colors[d] = col[d];
    const std::vector<McClass> classes = mc_classes(col);
    cudaSetDevice(plan->device);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int64_t N = plan->N;
    const int nbm = static_cast<int>(std::min<int64_t>((N + 255) / 256, kMagBlocksPerSm * static_cast<int64_t>(plan->num_sms)));
    const McClass& K0 = classes[0];
    const int sub[3] = {(plan->sp.L[0] + K0.qx - 1) / K0.qx, (plan->sp.L[1] + K0.sy - 1) / K0.sy,
                        (plan->sp.L[2] + K0.sz - 1) / K0.sz};
    const dim3 grid((sub[0] + 31) / 32, (sub[1] + kMcBY - 1) / kMcBY, sub[2]), blk(32, kMcBY);
    const int nbc = static_cast<int>(grid.x * grid.y * grid.z);  // blocks of one colour pass
    const int ncol = static_cast<int>(classes.size());
    const bool track = p->track_totals && (E_dev || M_dev);
    // the call's scratch: the chain's state; magnetisation partials; the tracked
    // totals' per-block partials
    McChain* d_scr = nullptr;
    double* d_part = nullptr;
    double* d_track = nullptr;
    mj_status st = cuda_status(cudaMalloc(&d_scr, sizeof(McChain)), "MC scratch");
    if (st == MJ_OK && (M_dev || track)) st = cuda_status(cudaMalloc(&d_part, sizeof(double) * 3 * nbm), "MC scratch");
    if (st == MJ_OK && track)
        st = cuda_status(cudaMalloc(&d_track, sizeof(double) * 4 * static_cast<size_t>(ncol) * nbc), "MC scratch");
    if (st != MJ_OK) {
        cudaFree(d_part);
        cudaFree(d_scr);
        return st;
    }
    McChain chain;
    std::memset(&chain, 0, sizeof(chain));
    chain.cone = p->cone;
    chain.cos_cone = std::cos(p->cone);
    cudaMemcpyAsync(d_scr, &chain, sizeof(chain), cudaMemcpyHostToDevice, s);
    if (track) {  // the totals at the start of the call
        if ((st = launch_energy(plan, m, &d_scr->run[0], s)) == MJ_OK) {
            k_mc_magnetisation<<<nbm, 256, 0, s>>>(m, N, d_part, d_scr->counter, &d_scr->run[1], nbm);
            st = cuda_status(cudaGetLastError(), "k_mc_magnetisation");
        }
        if (st != MJ_OK) {
            cudaFree(d_track);
            cudaFree(d_part);
            cudaFree(d_scr);
            return st;
        }
    }
    McCoef C;
    std::memset(&C, 0, sizeof(C));
    C.kT = p->temperature * kKB;
    C.inv_kT = C.kT > 0.0 ? 1.0 / C.kT : 0.0;
    C.tab = plan->d_noise_tab;
    C.proposal = p->proposal;
    C.stream = p->stream_id;
    mc_keys(p->seed, C.keys);
    C.chain = d_scr;
    C.track = d_track;
    C.track_n = ncol * nbc;
    // the adaptive cone's step per sweep; its rule runs on the device (k_mc_sweep_end)
    const bool adapt = p->adapt_cone && p->proposal == MJ_MC_CONE;
    const double cone_step = 1e-4 * static_cast<double>(N);
    const int64_t proposed0 = p->proposed_total;
    for (int32_t k = 0; k < nsweeps && st == MJ_OK; ++k) {
        C.sweep = p->sweep0 + static_cast<uint32_t>(k);
        for (int ci = 0; ci < ncol; ++ci) {
            const McClass& K = classes[ci];
            C.track_off = ci * nbc;
            switch (plan->sp.shape) {
                case kShapeSquareNN:
                    k_mc_color<ShapeSquareNN><<<grid, blk, 0, s>>>(plan->sp, plan->d_bmap, m, C, K);
                    break;
                case kShapeSquare2:
                    k_mc_color<ShapeSquare2><<<grid, blk, 0, s>>>(plan->sp, plan->d_bmap, m, C, K);
                    break;
                case kShapeTriNN:
                    k_mc_color<ShapeTriNN><<<grid, blk, 0, s>>>(plan->sp, plan->d_bmap, m, C, K);
                    break;
                case kShapeTri3:
                    k_mc_color<ShapeTri3><<<grid, blk, 0, s>>>(plan->sp, plan->d_bmap, m, C, K);
                    break;
                default:
                    k_mc_color<void><<<grid, blk, 0, s>>>(plan->sp, plan->d_bmap, m, C, K);
            }
        }
        if ((st = cuda_status(cudaGetLastError(), "k_mc_color")) != MJ_OK) break;
        if (track || adapt) {
            k_mc_sweep_end<<<track ? 5 : 1, kMcEndThreads, 0, s>>>(
                d_track, ncol * nbc, d_scr, E_dev ? E_dev + k : nullptr, M_dev ? M_dev + 3 * k : nullptr, adapt ? 1 : 0,
                static_cast<long long>(p->accepted_total), static_cast<long long>(proposed0 + N * (k + 1)), cone_step);
            if ((st = cuda_status(cudaGetLastError(), "k_mc_sweep_end")) != MJ_OK) break;
        }
        if (!track && E_dev && (st = launch_energy(plan, m, E_dev + k, s)) != MJ_OK) break;
        if (M_dev && !track) {
            k_mc_magnetisation<<<nbm, 256, 0, s>>>(m, N, d_part, d_scr->counter, M_dev + 3 * k, nbm);
            if ((st = cuda_status(cudaGetLastError(), "k_mc_magnetisation")) != MJ_OK) break;
        }
    }
    // the counts and the cone back (the call returns after its sweeps)
    if (st == MJ_OK) {
        st = cuda_status(cudaMemcpyAsync(&chain, d_scr, sizeof(chain), cudaMemcpyDeviceToHost, s), "MC counters");
        const mj_status sy = cuda_status(cudaStreamSynchronize(s), "MC sweeps");
        if (st == MJ_OK) st = sy;
    }
    if (st == MJ_OK) {
        p->accepted_total += static_cast<int64_t>(chain.acc);
        p->proposed_total += N * nsweeps;
        if (adapt) p->cone = chain.cone;
        p->sweep0 += static_cast<uint32_t>(nsweeps);
        if (accepted) *accepted = static_cast<int64_t>(chain.acc);
    }
    cudaFree(d_track);
    cudaFree(d_part);
    cudaFree(d_scr);
    return st;
}

}  // extern "C"
