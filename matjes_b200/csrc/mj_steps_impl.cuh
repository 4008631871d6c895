// Many time steps in one launch, for lattices whose tiles are all resident at
// once (mj_shapes.hpp lattices, no dipolar term).
//
// A small lattice's step is bound by its two dependent launches, not by its
// arithmetic: 64^2 sites are 16 tiles on 148 SMs, and a launch with its ramp,
// halo staging and last block takes 5 us of which the tile's own work is a
// fraction.  Here every block keeps one 32 x 8 tile for the whole call, its spins
// in registers and shared memory, and a pass needs only the halo from outside.
//
// Exchange (TileRing): a tile posts its edge spins in a box of its own in global
// memory, every 64-bit word half of a double and the pass number that wrote it; a
// reader polls the words it needs until all carry the pass it waits for.  A word
// is written and read whole, so data and flag arrive together: no fence, no
// counter, one trip through the L2 (posting with a release, polling a counter
// and then loading took three).  Boxes alternate between two halves by the
// pass's parity: a tile posts pass p + 2 after it has read its neighbours' p + 1,
// which they posted after reading p, so nothing is overwritten unread (whom a
// tile reads also reads it).  The thermal draw of a step is made before the wait,
// and neither it nor m_n goes through memory between the passes.  The launch is
// cooperative, so all blocks run at once and every wait ends; the waits are
// bounded all the same.  A tile whose wait gives up sets kStatusTimeout and returns;
// the others, which by then wait for it or for its neighbours, follow at about the
// same time.  The energies of such a launch become NaN (k_steps_energy,
// k_batch_energy), and so do the adjoint's gradients; the spins stay as they are, to
// be asked for with the status word.  (NaN spins from here, a limit in a register or a
// look at the status word in the wait's loop cost 2 to 10 % of a step.)
//
// The arithmetic is the tiled passes' (mj_tiled_impl.cuh): the spins are the
// same bit for bit.  us per SIB step at 10 K, this against two launches: square
// 16^2 3.1 / 10.6, 64^2 3.2 / 10.3, 256^2 4.0 / 11.6, 512^2 10.3 / 15.5;
// triangular, three shells, 64^2 3.7 / 12.6, 256^2 4.9 / 13.4, 512^2 12.2 / 18.3
// (with a release, a counter and a load per exchange 4.9 at 64^2, 6.6 at 256^2).
// What bounds it: the chain post - poll - pass, 1.6 to 2 us a pass up to 256^2.  At
// 512^2 (39 ps per site and step) still half of it: the schedulers issue in 0.51 of
// their cycles (0.33 at 256^2), per instruction a warp waits 4.4 cycles for memory
// (polls and halo) and 2.7 at the barriers.
#pragma once

#include "mj_tiled_impl.cuh"

namespace mj {
namespace {

struct StepsArgs {
    const double* m_in;  // spins entering step 0
    double* m;           // spins entering step k > 0 stored at m + k m_stride, unless null
    int64_t m_stride;
    double* mid;         // midpoint of step k stored at mid + k mid_stride, unless null
    int64_t mid_stride;
    double* m_out;       // spins after the last step
    const double* bmap;
    double* partials;    // energy partials, one per warp: [slot][warps of the launch]
    int e_slot0;         // slot of the energy of the spins entering step 0 (-1: not recorded), step k's at + k
    int e_on;
    int e_final;         // also the energy of the spins after the last step
    int half;            // the last step makes its predictor only
    int nsteps;
    uint32_t step0;
    unsigned long long* box;  // the tiles' boxes, zero at the launch
    int mute;                 // 1: nothing is posted, so that every wait runs out (a test)
    int* status;
};

// looks after which a wait gives up, about a second
constexpr uint32_t kStepsWaitPolls = 1u << 20;

// The halo of a block's tile (TileGeom layout) and the boxes its cells come from.  A tile's box: [parity][word][kN]
// over the sites within R of the tile's edge (box_index), word 2 c and 2 c + 1
// the low and high half of component c.
template <class S, int BYT, int RY>
struct TileRing {
    using G = TileGeom<S, BYT, RY>;
    static constexpr int R = G::R, NT = 32 * BYT;
    static constexpr int KH = ((G::TX + 2 * R) * (G::TY + 2 * R) - G::TX * G::TY + NT - 1) / NT;  // cells per thread
    static constexpr int kN = steps_box_sites(R);
    static_assert(G::TX == 32 && G::TY == kStepsTY, "box_index");
    int hpos[KH], hsrc[KH];  // a halo cell's place in the tile, its site in the layer (-1: none, or past an open edge)
    int hbox[KH];            // its place in the boxes
    int obox[RY];            // the thread's sites' places in the tile's box (-1: not posted)
    unsigned long long* box;

    // place of site (lx, ly) of a w x h tile in its box: the first R rows, the last R, then the sides; -1 inside
    static __device__ __forceinline__ int box_index(int lx, int ly, int w, int h) {
        if (ly < R) return ly * 32 + lx;
        if (ly >= h - R) return (R + ly - (h - R)) * 32 + lx;
        if (lx < R) return 64 * R + (ly - R) * 2 * R + lx;
        if (lx >= w - R) return 64 * R + (ly - R) * 2 * R + R + lx - (w - R);
        return -1;
    }
    // tile (bx, by) of the nx tiles a row of an Lx x Ly layer whose first box is number tile0
    __device__ __forceinline__ void init(const int* periodic, int Lx, int Ly, int bx, int by, int nx, int tile0,
                                         unsigned long long* boxes, int mute) {
        const int tid = threadIdx.x + 32 * threadIdx.y;
        const int x0 = bx * G::TX, y0 = by * G::TY;
        const int w = min(G::TX, Lx - x0), h = min(G::TY, Ly - y0);
        auto base_of = [&](int tx, int ty) { return 12 * kN * (tile0 + tx + nx * ty); };
        box = boxes;
        // the ring of width R about the tile's w x h sites: rows below and above, then the sides
        const int full = w + 2 * R;
#pragma unroll
        for (int q = 0; q < KH; ++q) {
            const int c = tid + q * NT;
            int lx = 0, ly = -1;  // relative to the tile's first site
            if (c < R * full) {
                lx = c % full - R;
                ly = c / full - R;
            } else if (c < 2 * R * full) {
                lx = (c - R * full) % full - R;
                ly = h + (c - R * full) / full;
            } else if (c < 2 * R * (full + h)) {
                const int d = c - 2 * R * full;
                ly = d / (2 * R);
                lx = d % (2 * R);
                lx = lx < R ? lx - R : w + lx - R;
            }
            hsrc[q] = -1;
            hbox[q] = 0;
            hpos[q] = (ly + R) * G::PX + lx + G::RX;
            if (c < 2 * R * (full + h)) {
                int gx = x0 + lx, gy = y0 + ly;
                const bool outx = gx < 0 || gx >= Lx, outy = gy < 0 || gy >= Ly;
                if (!((outx && !periodic[0]) || (outy && !periodic[1]))) {
                    if (outx) gx = ((gx % Lx) + Lx) % Lx;
                    if (outy) gy = ((gy % Ly) + Ly) % Ly;
                    hsrc[q] = gx + Lx * gy;
                    const int tx = gx / G::TX, ty = gy / G::TY;
                    hbox[q] = base_of(tx, ty) + box_index(gx - tx * G::TX, gy - ty * G::TY, min(G::TX, Lx - tx * G::TX),
                                                          min(G::TY, Ly - ty * G::TY));
                }
            }
        }
#pragma unroll
        for (int r = 0; r < RY; ++r) {
            const int lx = threadIdx.x, ly = threadIdx.y * RY + r;
            const int b = lx < w && ly < h ? box_index(lx, ly, w, h) : -1;
            obox[r] = b < 0 || mute ? -1 : base_of(bx, by) + b;
        }
    }
    // the halo cells of a layer of `src` (component stride N) into the tile
    __device__ __forceinline__ void load(const double* src, int64_t N, double* sm) const {
#pragma unroll
        for (int q = 0; q < KH; ++q)
            if (hsrc[q] >= 0)
                set(sm, hpos[q], make_double3(__ldcg(src + hsrc[q]), __ldcg(src + N + hsrc[q]), __ldcg(src + 2 * N + hsrc[q])));
    }
    // the vector v of the thread's site r as pass `pass` into the box
    __device__ __forceinline__ void post(int r, double3 v, unsigned int pass) const {
        if (obox[r] < 0) return;
        unsigned long long* b = box + obox[r] + (pass & 1u) * (6 * kN);
        const unsigned long long tag = static_cast<unsigned long long>(pass) << 32;
        const double c[3] = {v.x, v.y, v.z};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            put_word(b + (2 * k) * kN, tag | static_cast<unsigned int>(__double2loint(c[k])));
            put_word(b + (2 * k + 1) * kN, tag | static_cast<unsigned int>(__double2hiint(c[k])));
        }
    }
    // the halo cells as the neighbours posted them in pass `pass` into the tile;
    // false (all threads of the block, after a barrier) when a wait gave up
    __device__ __forceinline__ bool fetch(unsigned int pass, double* sm, int* status) const {
        bool bad = false;
#pragma unroll
        for (int q = 0; q < KH; ++q) {
            if (hsrc[q] < 0) continue;
            const unsigned long long* b = box + hbox[q] + (pass & 1u) * (6 * kN);
            unsigned long long u[6];
            for (uint32_t it = 0;; ++it) {
                bool ok = true;
#pragma unroll
                for (int k = 0; k < 6; ++k) u[k] = get_word(b + k * kN);
#pragma unroll
                for (int k = 0; k < 6; ++k) ok = ok && static_cast<unsigned int>(u[k] >> 32) == pass;
                if (ok) break;
                if (it > kStepsWaitPolls) {
                    bad = true;
                    break;
                }
                if (it > 4096) __nanosleep(64);
            }
            auto half = [&](int k) { return static_cast<int>(static_cast<unsigned int>(u[k])); };
            set(sm, hpos[q], make_double3(__hiloint2double(half(1), half(0)), __hiloint2double(half(3), half(2)),
                                          __hiloint2double(half(5), half(4))));
        }
        if (__syncthreads_or(bad)) {
            if (threadIdx.x == 0 && threadIdx.y == 0) atomicOr(status, kStatusTimeout);
            return false;
        }
        return true;
    }
    static __device__ __forceinline__ void set(double* sm, int c, double3 v) {
        sm[c] = v.x;
        sm[G::NS + c] = v.y;
        sm[2 * G::NS + c] = v.z;
    }
    static __device__ __forceinline__ void put_word(unsigned long long* p, unsigned long long v) {
        asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
    }
    static __device__ __forceinline__ unsigned long long get_word(const unsigned long long* p) {
        unsigned long long v;
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
        return v;
    }
};

template <class S, int BYT, int RY, int MINB, int SP, int INTEG>
__global__ void __launch_bounds__(32 * BYT, MINB) k_steps(const __grid_constant__ StencilParams P,
                                                          const __grid_constant__ DynCoef C,
                                                          const __grid_constant__ StepsArgs A) {
    using G = TileGeom<S, BYT, RY>;
    constexpr int R = G::R, NT = 32 * BYT;
    constexpr bool kTwo = INTEG != MJ_EULER;  // passes per step
    extern __shared__ __align__(128) double sm[];
    const int Lx = P.L[0], Ly = P.L[1];
    const int64_t layer = static_cast<int64_t>(Lx) * Ly, N = layer * P.L[2];
    const int z = blockIdx.z;
    const int x0 = blockIdx.x * G::TX, y0 = blockIdx.y * G::TY;
    const int tid = threadIdx.x + 32 * threadIdx.y;
    const int bid = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
    // cells across an open edge stay zero
    for (int q = tid; q < 3 * G::NS; q += NT) sm[q] = 0.0;
    TileRing<S, BYT, RY> ring;
    ring.init(P.periodic, Lx, Ly, blockIdx.x, blockIdx.y, gridDim.x, gridDim.x * gridDim.y * z, A.box, A.mute);
    const int x = x0 + static_cast<int>(threadIdx.x), yt = y0 + static_cast<int>(threadIdx.y) * RY;
    const int64_t i0 = layer * z + x + static_cast<int64_t>(Lx) * yt;
    const int base = static_cast<int>(threadIdx.y) * RY * G::PX + static_cast<int>(threadIdx.x);
    const int own = base + G::R * G::PX + G::RX;  // the first own site's cell
    double3 mn[RY];
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RY; ++r) {
        mn[r] = make_double3(0.0, 0.0, 0.0);
        if (x < Lx && yt + r < Ly) {
            const int64_t i = i0 + static_cast<int64_t>(Lx) * r;
            mn[r] = make_double3(__ldcg(A.m_in + i), __ldcg(A.m_in + N + i), __ldcg(A.m_in + 2 * N + i));
            const int c = own + r * G::PX;
            sm[c] = mn[r].x;
            sm[G::NS + c] = mn[r].y;
            sm[2 * G::NS + c] = mn[r].z;
        }
    }
    // field of the thread's sites from the staged tile, m0[r] their own spins: real-space
    // field into B, the sites' energy returned when wanted
    auto field = [&](const double3 (&m0)[RY], double3 (&B)[RY], bool want_e) -> double {
        double bx[RY], by[RY], bz[RY];
#pragma unroll
        for (int r = 0; r < RY; ++r) bx[r] = by[r] = bz[r] = 0.0;
        all_columns<S, BYT, RY, SP>(P, sm, base, bx, by, bz, std::make_integer_sequence<int, 2 * S::R + 1>{});
        double e = 0.0;
#pragma unroll
        for (int r = 0; r < RY; ++r) {
            double b0 = bx[r], b1 = by[r], b2 = bz[r];
            if (P.has_onsite) {
                const double* W = P.W0;
                if constexpr (SP == SP_AXIAL) {
                    b2 = fma(W[8], m0[r].z, b2);
                } else {
                    b0 = fma(W[0], m0[r].x, fma(W[1], m0[r].y, fma(W[2], m0[r].z, b0)));
                    b1 = fma(W[3], m0[r].x, fma(W[4], m0[r].y, fma(W[5], m0[r].z, b1)));
                    b2 = fma(W[6], m0[r].x, fma(W[7], m0[r].y, fma(W[8], m0[r].z, b2)));
                }
            }
            const bool in = x < Lx && yt + r < Ly;
            double3 zee = make_double3(0.0, 0.0, 0.0);
            if (P.zee_on) {
                if (A.bmap) {
                    const int64_t i = in ? i0 + static_cast<int64_t>(Lx) * r : 0;
                    zee = make_double3(P.zc * __ldg(A.bmap + i), P.zc * __ldg(A.bmap + N + i),
                                       P.zc * __ldg(A.bmap + 2 * N + i));
                } else if constexpr (SP == SP_AXIAL) {
                    zee.z = P.zc * P.bext[2];
                } else {
                    zee = make_double3(P.zc * P.bext[0], P.zc * P.bext[1], P.zc * P.bext[2]);
                }
            }
            // the axial form adds no x, y Zeeman field without a map, as the tiled passes
            const bool zax = SP == SP_AXIAL && !A.bmap;
            B[r] = zax ? make_double3(b0, b1, b2 + zee.z) : make_double3(b0 + zee.x, b1 + zee.y, b2 + zee.z);
            if (want_e && in) {
                const double mz = zax ? m0[r].z * zee.z : dot(m0[r], zee);
                e += -0.5 * (dot(m0[r], B[r]) + mz);
            }
        }
        return e;
    };
    const int nwarps = static_cast<int>(gridDim.x * gridDim.y * gridDim.z) * BYT;
    auto record = [&](double e, int slot) {
        for (int o = 16; o > 0; o >>= 1) e += __shfl_down_sync(0xffffffffu, e, o);
        if (threadIdx.x == 0) A.partials[static_cast<int64_t>(slot) * nwarps + bid * BYT + threadIdx.y] = e;
    };
    // new spins v of the thread's sites: posted as pass `pass` (0: not) as soon as
    // they are known, into the tile once every thread has read it, and into dst
    auto store = [&](const double3 (&v)[RY], unsigned int pass, double* dst) {
        if (pass)
#pragma unroll
            for (int r = 0; r < RY; ++r) ring.post(r, v[r], pass);
        __syncthreads();
#pragma unroll
        for (int r = 0; r < RY; ++r)
            if (x < Lx && yt + r < Ly) {
                ring.set(sm, own + r * G::PX, v[r]);
                if (dst) st3(dst, i0 + static_cast<int64_t>(Lx) * r, N, v[r]);
            }
    };
    TiledArgs TA = {};
    for (int k = 0; k < A.nsteps; ++k) {
        const bool last = k + 1 == A.nsteps;
        Pre pre[RY];
        TA.step = A.step0 + static_cast<uint32_t>(k);
        if (C.thermal) prefetch_sites<S, BYT, RY, PASS_SIB1>(P, C, TA, x0, y0, z, pre);
        if (k == 0) {
            ring.load(A.m_in + layer * z, N, sm);
            __syncthreads();
        } else if (!ring.fetch(static_cast<unsigned int>(kTwo ? 2 * k : k), sm, A.status)) {
            return;
        }
        double3 B[RY], v[RY];
        const int slot = A.e_slot0 + k;
        const bool want_e = A.e_on && slot >= 0;
        const double e = field(mn, B, want_e);
        if (want_e) record(e, slot);
        if constexpr (!kTwo) {
#pragma unroll
            for (int r = 0; r < RY; ++r) {
                const double3 D = llg_rhs(B[r], mn[r], C.alpha, C.inv_den);
                const double c = C.h_over_hbar;
                double3 t = advance(mn[r], D, c);
                if (C.thermal) {
                    const double3 DT = llg_rhs(pre[r].b, mn[r], C.alpha, C.inv_den);
                    t = advance(t, DT, c);
                }
                v[r] = project(t, mn[r]);
                if (x < Lx && yt + r < Ly) flag_nonfinite(A.status, v[r]);
            }
#pragma unroll
            for (int r = 0; r < RY; ++r) mn[r] = v[r];
            const unsigned int pass = static_cast<unsigned int>(k + 1);
            if (last && A.nsteps == 1) {
                // the neighbours may still read the spins that m_out replaces: their
                // first pass says that they have
                store(v, pass, nullptr);
                if (!ring.fetch(pass, sm, A.status)) return;
                store(v, 0u, A.m_out);
            } else {
                store(v, last && !A.e_final ? 0u : pass, last ? A.m_out : nullptr);
            }
            continue;
        }
        double3 kept[RY];  // Heun: what the corrector needs of the predictor's slopes
#pragma unroll
        for (int r = 0; r < RY; ++r) {
            if constexpr (INTEG == MJ_SIB) {
                double3 H = B[r];
                if (C.thermal) H = make_double3(H.x + pre[r].b.x, H.y + pre[r].b.y, H.z + pre[r].b.z);
                v[r] = sib_solve<true>(mn[r], mn[r], H, C.alpha, C.sib_hc);
            } else {
                const double3 D = llg_rhs(B[r], mn[r], C.alpha, C.inv_den);
                v[r] = project(advance(mn[r], D, C.h_over_hbar), mn[r]);
                kept[r] = heun_kept(D, C.thermal, C.thermal ? llg_rhs(pre[r].b, mn[r], C.alpha, C.inv_den) : D);
            }
        }
        const bool end = last && A.half;
        store(v, end ? 0u : static_cast<unsigned int>(2 * k + 1), A.mid ? A.mid + k * A.mid_stride : nullptr);
        if (end) return;
        if (!ring.fetch(static_cast<unsigned int>(2 * k + 1), sm, A.status)) return;
        field(v, B, false);
#pragma unroll
        for (int r = 0; r < RY; ++r) {
            if constexpr (INTEG == MJ_SIB) {
                double3 H = B[r];
                if (C.thermal) H = make_double3(H.x + pre[r].b.x, H.y + pre[r].b.y, H.z + pre[r].b.z);
                mn[r] = sib_solve(mn[r], v[r], H, C.alpha, C.sib_hc);
            } else {
                const double3 D2 = llg_rhs(B[r], v[r], C.alpha, C.inv_den);
                const double3 t = advance(v[r], heun_slope(kept[r], D2), C.h_over_hbar);
                mn[r] = project(t, v[r]);
            }
            if (x < Lx && yt + r < Ly) flag_nonfinite(A.status, mn[r]);
        }
        store(mn, last && !A.e_final ? 0u : static_cast<unsigned int>(2 * k + 2),
              last ? A.m_out : (A.m ? A.m + (k + 1) * A.m_stride : nullptr));
    }
    if (A.e_final) {
        if (!ring.fetch(static_cast<unsigned int>(kTwo ? 2 * A.nsteps : A.nsteps), sm, A.status)) return;
        double3 B[RY];
        const double e = field(mn, B, true);
        record(e, A.e_slot0 + A.nsteps);
    }
}

template <class S, int BYT, int RY, int MINB, int SP, int INTEG>
mj_status launch_steps_cfg(mj_plan* p, const DynCoef& C, const StepsArgs& A, dim3 grid, cudaStream_t s) {
    auto kern = k_steps<S, BYT, RY, MINB, SP, INTEG>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(32, BYT);
    cfg.dynamicSmemBytes = TileGeom<S, BYT, RY>::buf_bytes;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cuda_status(cudaLaunchKernelEx(&cfg, kern, p->sp, C, A), "k_steps");
}

// A halo reaches the next tile alone, unless a last tile is thinner than the
// reach: the one before it is then in reach of the periodic images too.
template <class S>
bool thin_last_tile(const int* periodic, int Lx, int Ly) {
    auto thin = [](bool per, int L, int t) { return per && L > t && L % t != 0 && L % t < S::R; };
    return thin(periodic[0] != 0, Lx, 32) || thin(periodic[1] != 0, Ly, kStepsTY);
}

// Resident tiles of a configuration on the plan's device.
template <class S, int BYT, int RY, int MINB, int SP, int INTEG>
int steps_capacity(const mj_plan* p) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_steps<S, BYT, RY, MINB, SP, INTEG>, 32 * BYT,
                                                      TileGeom<S, BYT, RY>::buf_bytes) != cudaSuccess)
        return 0;
    return per_sm * p->num_sms;
}

template <class S, int SP, int INTEG>
mj_status steps_run(mj_plan* p, const StepsJob* job, const DynCoef& C, int* warps, bool& fits, cudaStream_t s) {
    using G = TileGeom<S, 8, 1>;
    static_assert(G::TY == kStepsTY && TileGeom<S, 4, 2>::TY == kStepsTY, "one tile height");
    const dim3 grid((p->sp.L[0] + 31) / 32, (p->sp.L[1] + kStepsTY - 1) / kStepsTY, p->sp.L[2]);
    const int64_t tiles = static_cast<int64_t>(grid.x) * grid.y * grid.z;
    fits = false;
    if (thin_last_tile<S>(p->sp.periodic, p->sp.L[0], p->sp.L[1])) return MJ_OK;
    // one site per thread while the blocks of eight warps that are resident hold
    // the lattice (the shortest chain per pass): at two blocks per SM, then three
    // (80 registers) and four (64).  Two sites per thread above: at six blocks per
    // SM, then at eight with the registers that leaves (64; 512^2 10.3 us a step
    // where the two launches take 15.5).  us per SIB step at 10 K, one site at
    // three or four blocks against two sites at six: square 288^2 4.7 / 5.4, 352 x
    // 320 4.9 / 5.7, 384^2 5.7 / 6.1 (T = 0 5.4 / 6.2).  A longer reach (three
    // triangular shells) keeps more in registers: three blocks gain where the
    // draw gives the eight warps work (352 x 320 6.3 / 6.8, T = 0 5.7 / 5.7 and
    // 288^2 5.7 / 5.5), four spill (384^2 T = 0 7.1 / 6.4).
    const bool one2 = tiles <= steps_capacity<S, 8, 1, 2, SP, INTEG>(p);
    const bool one3 = !one2 && (S::R == 1 || C.thermal) && tiles <= steps_capacity<S, 8, 1, 3, SP, INTEG>(p);
    bool one4 = false;
    if constexpr (S::R == 1) one4 = !one2 && !one3 && tiles <= steps_capacity<S, 8, 1, 4, SP, INTEG>(p);
    const bool one = one2 || one3 || one4;
    const bool six = tiles <= steps_capacity<S, 4, 2, 6, SP, INTEG>(p);
    if (!one && !six && tiles > steps_capacity<S, 4, 2, 8, SP, INTEG>(p)) return MJ_OK;
    fits = true;
    if (!job) return MJ_OK;
    *warps = static_cast<int>(tiles) * (one ? 8 : 4);
    StepsArgs A;
    std::memset(&A, 0, sizeof(A));
    A.m_in = job->m_in;
    A.m = job->m;
    A.m_stride = job->m_stride;
    A.mid = job->mid;
    A.mid_stride = job->mid_stride;
    A.m_out = job->m_out;
    A.bmap = p->d_bmap;
    A.partials = job->partials;
    A.e_on = job->partials != nullptr;
    A.e_slot0 = job->e_slot0;
    A.e_final = job->e_final;
    A.half = job->half;
    A.nsteps = job->nsteps;
    A.step0 = job->step0;
    A.box = job->box;
    A.mute = p->mute_tiles ? 1 : 0;
    A.status = p->d_status;
    mj_status st = cuda_status(cudaMemsetAsync(job->box, 0, sizeof(unsigned long long) * 12 * steps_box_sites(S::R) * tiles, s),
                               "step boxes");
    if (st != MJ_OK) return st;
    if (one2) return launch_steps_cfg<S, 8, 1, 2, SP, INTEG>(p, C, A, grid, s);
    if (one3) return launch_steps_cfg<S, 8, 1, 3, SP, INTEG>(p, C, A, grid, s);
    if constexpr (S::R == 1)
        if (one4) return launch_steps_cfg<S, 8, 1, 4, SP, INTEG>(p, C, A, grid, s);
    if (six) return launch_steps_cfg<S, 4, 2, 6, SP, INTEG>(p, C, A, grid, s);
    return launch_steps_cfg<S, 4, 2, 8, SP, INTEG>(p, C, A, grid, s);
}

// job = null: only whether the plan's lattice fits (`fits`)
template <class S>
mj_status launch_steps_shape(mj_plan* p, const StepsJob* job, const DynCoef& C, int* warps, bool& fits, cudaStream_t s) {
    const bool axial = stencil_axial<S>(p->sp, p->d_bmap != nullptr);
    switch (C.integrator) {
        case MJ_EULER:
            return axial ? steps_run<S, SP_AXIAL, MJ_EULER>(p, job, C, warps, fits, s)
                         : steps_run<S, SP_FULL, MJ_EULER>(p, job, C, warps, fits, s);
        case MJ_HEUN_MATJES:
            return axial ? steps_run<S, SP_AXIAL, MJ_HEUN_MATJES>(p, job, C, warps, fits, s)
                         : steps_run<S, SP_FULL, MJ_HEUN_MATJES>(p, job, C, warps, fits, s);
        default:
            return axial ? steps_run<S, SP_AXIAL, MJ_SIB>(p, job, C, warps, fits, s)
                         : steps_run<S, SP_FULL, MJ_SIB>(p, job, C, warps, fits, s);
    }
}

}  // namespace
}  // namespace mj
