// Dipolar field as a zero-padded FFT convolution (one magnetic atom per cell).
//
// Reference route (paths relative to Matjes src/): the K tensor of
// Energy/dipolar_magnetic.f90:58-177 on the N_rep grid of
// Hamiltonian_type/fft_ham_base.f90:191-220 (open axes doubled, periodic axes
// with images), K_F = FFT(K)/prod(N_rep) once (fft_ham_fftw.f90:134-178,
// cuda_fft.cpp:96-143), and per call pad -> D2Z -> H_F = K_F M_F -> Z2D ->
// unpack (fft_ham_fftw.f90:239-262, cuda_fft.cu:38-70, fft_ham_internal.f90).
//
// Here the 3D transform of the padded spins is split by axis so that the zero
// planes of an open z axis cost nothing: 2D real transforms over (y, x) of the
// Lz lattice planes only, then complex transforms of length N_rep,z along z
// (the planes z >= Lz of that buffer are zero once and never written).  The
// inverse runs the z transforms and then 2D inverse transforms of the Lz
// planes the consumers read.  Layouts are z-major, [z][component][y][x], so
// that one batched plan covers every (plane, component).  When K is even on
// the N_rep grid (K(-r) = K(r), e.g. open axes without images) K_F is real and
// the pointwise product reads 6 real instead of 6 complex values per wave
// vector; with periodic axes the reference's truncated image sums leave K
// slightly uneven (imaginary parts of K_F ~1e-7 of its scale), and the complex
// product is kept whenever they exceed 1e-13.  The unpack is fused into the consumers: the field and
// step kernels read H on the padded (y, x) grid of the lattice planes.
//
// With few lattice planes (zdirect_pays) the z part is not transformed at all: k_zdirect
// sums H_z = sum_z' K(ky, kx, z - z') M_z' over the planes for every (ky, kx)
// column, with K transformed along y and x only.  It serves every N_rep,z, reads
// and writes the Lz planes alone, and for an open z axis uses the mirror symmetry
// of K (K_xz and K_yz odd in z, the others even) to read half of K.
//
// Otherwise, when N_rep,z is a power of two from 2 to 32, the z transforms and the
// pointwise product are one kernel (k_zconv): one warp per (ky, kx) column, lane = z,
// a radix-2 FFT across the lanes by shuffles (forward in decimation in
// frequency, which leaves the spectrum in bit-reversed order, K_F stored per
// column in that order, inverse in decimation in time back to natural order).
// It reads only the Lz lattice planes of the 2D spectra (the others are the
// zero padding) and writes only the Lz planes the inverse 2D transform reads.
#include <cufft.h>

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "mj_internal.hpp"

namespace mj {
namespace {

struct DipolarPlan {
    int nrep[3];        // padded grid (x, y, z)
    int lz = 1;         // lattice planes
    int64_t pr = 0;     // real plane: nrep_y * nrep_x
    int64_t pc = 0;     // complex plane: nrep_y * (nrep_x/2 + 1)
    bool real_kf = true;
    double* d_pad = nullptr;               // [lz][3][y][x] real, zero outside the lattice
    double* d_h = nullptr;                 // [lz][3][y][x] real, H of the lattice planes
    cufftDoubleComplex* d_cx = nullptr;    // [nrz][3][y][kx]: 2D spectra, planes >= lz stay zero
    cufftDoubleComplex* d_cz = nullptr;    // [nrz][3][y][kx]: full spectrum, then H's z transform
    double* d_kfr = nullptr;               // [6][nrz][y][kx] real K_F (xx xy xz yy yz zz)
    cufftDoubleComplex* d_kfc = nullptr;   // complex K_F when it is not real
    cufftHandle f2d = 0, fz = 0, b2d = 0;
    bool have_f2d = false, have_fz = false, have_b2d = false;
    // the direct z sum: K transformed along y and x, [6][nkd][y][kx] (the lz distances of one sign
    // when the mirror gives the others, else all nz).  K_F above is then made only when the
    // cuFFT z transforms are asked for (dipolar_transforms)
    int zdir = 0;                          // 0: not used, else 1 + its mode (ZdirMode)
    int nkd = 0;
    cufftDoubleComplex* d_kd = nullptr;
    // the fused z convolution: K_F per column [pc][nz][6] (kz in bit-reversed
    // order), real or complex, and the twiddles exp(-2 pi i m / nz), m < nz / 2
    bool zconv = false;
    double* d_kzr = nullptr;
    cufftDoubleComplex* d_kzc = nullptr;
    double tw[32] = {};
};

__global__ void k_pad(const double* __restrict__ m, double* __restrict__ pad, int Lx, int Ly, int Lz, int px,
                      int64_t pr) {
    const int64_t N = static_cast<int64_t>(Lx) * Ly * Lz;
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i >= N) return;
    const int x = static_cast<int>(i % Lx);
    const int64_t r = i / Lx;
    const int y = static_cast<int>(r % Ly);
    const int z = static_cast<int>(r / Ly);
    const int64_t q = x + static_cast<int64_t>(px) * y + 3 * pr * z;
    pad[q] = __ldg(m + i);
    pad[pr + q] = __ldg(m + N + i);
    pad[2 * pr + q] = __ldg(m + 2 * N + i);
}

__device__ __forceinline__ cufftDoubleComplex cmul(cufftDoubleComplex a, cufftDoubleComplex b) {
    return make_cuDoubleComplex(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ cufftDoubleComplex cfma(cufftDoubleComplex a, cufftDoubleComplex b, cufftDoubleComplex c) {
    return make_cuDoubleComplex(fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y)));
}
__device__ __forceinline__ cufftDoubleComplex rfma(double a, cufftDoubleComplex b, cufftDoubleComplex c) {
    return make_cuDoubleComplex(fma(a, b.x, c.x), fma(a, b.y, c.y));
}

// H_F = K_F M_F over the spectrum [kz][c][ky][kx] (in place), K_F real [6][kz][ky][kx]
__global__ void k_pointwise_real(cufftDoubleComplex* __restrict__ spec, const double* __restrict__ kf, int64_t pc,
                                 int64_t nkc) {
    const int64_t k = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (k >= nkc) return;
    const int64_t kz = k / pc, w = k - kz * pc;
    cufftDoubleComplex* s = spec + kz * 3 * pc + w;
    const cufftDoubleComplex mx = s[0], my = s[pc], mz = s[2 * pc];
    const double kxx = __ldg(kf + k), kxy = __ldg(kf + nkc + k), kxz = __ldg(kf + 2 * nkc + k);
    const double kyy = __ldg(kf + 3 * nkc + k), kyz = __ldg(kf + 4 * nkc + k), kzz = __ldg(kf + 5 * nkc + k);
    const cufftDoubleComplex z0 = make_cuDoubleComplex(0.0, 0.0);
    s[0] = rfma(kxx, mx, rfma(kxy, my, rfma(kxz, mz, z0)));
    s[pc] = rfma(kxy, mx, rfma(kyy, my, rfma(kyz, mz, z0)));
    s[2 * pc] = rfma(kxz, mx, rfma(kyz, my, rfma(kzz, mz, z0)));
}

__global__ void k_pointwise_cplx(cufftDoubleComplex* __restrict__ spec, const cufftDoubleComplex* __restrict__ kf,
                                 int64_t pc, int64_t nkc) {
    const int64_t k = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (k >= nkc) return;
    const int64_t kz = k / pc, w = k - kz * pc;
    cufftDoubleComplex* s = spec + kz * 3 * pc + w;
    const cufftDoubleComplex mx = s[0], my = s[pc], mz = s[2 * pc];
    const cufftDoubleComplex kxx = kf[k], kxy = kf[nkc + k], kxz = kf[2 * nkc + k];
    const cufftDoubleComplex kyy = kf[3 * nkc + k], kyz = kf[4 * nkc + k], kzz = kf[5 * nkc + k];
    s[0] = cfma(kxx, mx, cfma(kxy, my, cmul(kxz, mz)));
    s[pc] = cfma(kxy, mx, cfma(kyy, my, cmul(kyz, mz)));
    s[2 * pc] = cfma(kxz, mx, cfma(kyz, my, cmul(kzz, mz)));
}

__global__ void k_scale(cufftDoubleComplex* __restrict__ a, int64_t n, double s) {
    const int64_t k = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (k >= n) return;
    a[k].x *= s;
    a[k].y *= s;
}

// Twiddles of a length-NZ transform: (cos, sin) of -2 pi m / NZ, m < NZ/2
struct ZTwiddle {
    double c[16], s[16];
};

__device__ __forceinline__ double2 shfl_xor_c(double2 v, int h) {
    return make_double2(__shfl_xor_sync(0xffffffffu, v.x, h), __shfl_xor_sync(0xffffffffu, v.y, h));
}
__device__ __forceinline__ double2 cmul_d(double2 a, double c, double s) {  // a (c + i s)
    return make_double2(fma(a.x, c, -(a.y * s)), fma(a.x, s, a.y * c));
}

// The forward transform of the lanes' values (lane l of a group of NZ holds
// element l): decimation in frequency, lane l ends with X(bitrev(l)).
template <int NZ>
__device__ __forceinline__ double2 zfft_forward(double2 x, int l, const double2* __restrict__ tw) {
#pragma unroll
    for (int h = NZ / 2; h >= 1; h >>= 1) {
        const double2 p = shfl_xor_c(x, h);
        if (l & h) {
            const double2 w = tw[(l & (h - 1)) * (NZ / (2 * h))];
            x = cmul_d(make_double2(p.x - x.x, p.y - x.y), w.x, w.y);
        } else {
            x = make_double2(x.x + p.x, x.y + p.y);
        }
    }
    return x;
}

// The inverse (exp(+2 pi i ...), unscaled) of bit-reversed lanes: decimation
// in time, lane l ends with y(l).
template <int NZ>
__device__ __forceinline__ double2 zfft_inverse(double2 x, int l, const double2* __restrict__ tw) {
#pragma unroll
    for (int h = 1; h < NZ; h <<= 1) {
        const double2 w = tw[(l & (h - 1)) * (NZ / (2 * h))];
        const double2 t = (l & h) ? cmul_d(x, w.x, -w.y) : x;
        const double2 p = shfl_xor_c(t, h);
        x = (l & h) ? make_double2(p.x - t.x, p.y - t.y) : make_double2(t.x + p.x, t.y + p.y);
    }
    return x;
}

// z transforms and the product H_F = K_F M_F in one pass: spec_in [z][c][col]
// (planes z < lz), out [z][c][col] (planes z < lz), K_F [col][6][l] with l the
// lane (bit-reversed kz); REAL: K_F real.  A block of 8 warps takes C = 256/NZ
// consecutive columns, one column per NZ lanes (every lane one z): the rows
// (z, c) of its columns are read and written whole through shared memory,
// [z][c * C + column] with rows of 3 C + 1 16-byte slots, so that the lanes of
// one column hit distinct banks.
template <int NZ>
struct ZcGeom {
    static constexpr int C = 256 / NZ;   // columns per block
    static constexpr int ROW = 3 * C + 1;
    static constexpr size_t smem = sizeof(double2) * NZ * ROW;
};

template <int NZ, bool REAL>
__global__ void __launch_bounds__(256) k_zconv(const double2* __restrict__ in, double2* __restrict__ out,
                                               const double* __restrict__ kr, const double2* __restrict__ kc,
                                               int64_t pc, int lz, const ZTwiddle W) {
    using Z = ZcGeom<NZ>;
    extern __shared__ double2 zs[];  // [NZ][ROW]
    // the twiddles in shared memory (the lanes index them differently)
    __shared__ double2 tw[16];
    if (threadIdx.x < NZ / 2) tw[threadIdx.x] = make_double2(W.c[threadIdx.x], W.s[threadIdx.x]);
    const int64_t col0 = static_cast<int64_t>(blockIdx.x) * Z::C;
    const int ncol = pc - col0 < Z::C ? static_cast<int>(pc - col0) : Z::C;
    // rows (z, c), z < lz: consecutive threads on consecutive columns of a row
    for (int idx = threadIdx.x; idx < 3 * lz * Z::C; idx += blockDim.x) {
        const int row = idx / Z::C, q = idx - row * Z::C;
        const int z = row / 3, c = row - 3 * z;
        zs[z * Z::ROW + c * Z::C + q] =
            q < ncol ? in[(static_cast<int64_t>(z) * 3 + c) * pc + col0 + q] : make_double2(0.0, 0.0);
    }
    __syncthreads();
    const int l = threadIdx.x % NZ, q = threadIdx.x / NZ;  // this lane's z and column
    const int64_t col = col0 + (q < ncol ? q : 0);
    double2 v[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        v[c] = l < lz ? zs[l * Z::ROW + c * Z::C + q] : make_double2(0.0, 0.0);
        v[c] = zfft_forward<NZ>(v[c], l, tw);
    }
    double2 h[3];
    if constexpr (REAL) {
        const double* k = kr + col * 6 * NZ + l;
        const double kxx = __ldg(k), kxy = __ldg(k + NZ), kxz = __ldg(k + 2 * NZ), kyy = __ldg(k + 3 * NZ),
                     kyz = __ldg(k + 4 * NZ), kzz = __ldg(k + 5 * NZ);
        h[0] = make_double2(fma(kxx, v[0].x, fma(kxy, v[1].x, kxz * v[2].x)),
                            fma(kxx, v[0].y, fma(kxy, v[1].y, kxz * v[2].y)));
        h[1] = make_double2(fma(kxy, v[0].x, fma(kyy, v[1].x, kyz * v[2].x)),
                            fma(kxy, v[0].y, fma(kyy, v[1].y, kyz * v[2].y)));
        h[2] = make_double2(fma(kxz, v[0].x, fma(kyz, v[1].x, kzz * v[2].x)),
                            fma(kxz, v[0].y, fma(kyz, v[1].y, kzz * v[2].y)));
    } else {
        const double2* k = kc + col * 6 * NZ + l;
        const double2 kxx = k[0], kxy = k[NZ], kxz = k[2 * NZ], kyy = k[3 * NZ], kyz = k[4 * NZ], kzz = k[5 * NZ];
        auto mac = [](double2 a, double2 b, double2 acc) {
            return make_double2(fma(a.x, b.x, fma(-a.y, b.y, acc.x)), fma(a.x, b.y, fma(a.y, b.x, acc.y)));
        };
        const double2 z0 = make_double2(0.0, 0.0);
        h[0] = mac(kxx, v[0], mac(kxy, v[1], mac(kxz, v[2], z0)));
        h[1] = mac(kxy, v[0], mac(kyy, v[1], mac(kyz, v[2], z0)));
        h[2] = mac(kxz, v[0], mac(kyz, v[1], mac(kzz, v[2], z0)));
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const double2 y = zfft_inverse<NZ>(h[c], l, tw);
        if (l < lz) zs[l * Z::ROW + c * Z::C + q] = y;  // this lane's own slot, read above by it alone
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < 3 * lz * Z::C; idx += blockDim.x) {
        const int row = idx / Z::C, q2 = idx - row * Z::C;
        const int z = row / 3, c = row - 3 * z;
        if (q2 < ncol) out[(static_cast<int64_t>(z) * 3 + c) * pc + col0 + q2] = zs[z * Z::ROW + c * Z::C + q2];
    }
}

// H of the lattice planes by the sum over z (see the header).  A block takes 32
// consecutive columns, one per lane; its NW warps share the planes' spectra in
// shared memory, and warp w makes the planes z = w, w + NW, ... (ZPT of them): per
// distance dz one load of K's six components serves the pairs (z, z - dz) and
// (z, z + dz) of all of them, the next distance's K in flight meanwhile (holding
// a block's K in shared memory instead measured slower, 16.7 against 14.9 us at
// 16 planes of 128 x 65 columns).  Bound by the latency of K's loads behind few warps
// (13 planes of 128 x 65 columns: 0.34 of the issue slots, FP64 pipe 0.24, 22 % of the
// warps, 4.3 cycles waiting for memory per instruction; 36 fma a pair, Lz^2 pairs a
// column), on large planes by the bytes of K.
enum ZdirMode { kZdirMirror = 0, kZdirOpen = 1, kZdirCircular = 2 };
constexpr int kZdirMax = 16;  // planes: two per warp, the spectra in 24 KB of shared memory
// Whether the direct sum is taken for lz planes of pc columns; `even`: K(-r) = K(r)
// on the grid, `pow2`: k_zconv serves N_rep,z.  On small planes every route waits for
// its launches and the one with fewer wins.  On large ones the bytes of K decide:
// k_zdirect reads complex K, per column and component Lz values with the mirror
// symmetry, 2 Lz (open) or Lz (circular) without; the transforms read N_rep,z values,
// real ones when K is even (with images a truncated sum leaves K uneven: complex).
// us of a field call, direct / k_zconv or cuFFT z and product, n^2 cells (x and y open
// except where noted; open axes double the columns):
//   mirror, pow2: 2 planes 192^2 58.8 / 58.9, 256^2 68.6 / 66.3; 4 planes 128^2 41.5 /
//     43.6, 192^2 89.3 / 87.1; 8 planes 96^2 48.5 / 48.8, 128^2 76.4 / 66.2; uneven
//     (periodic x, y) 4 planes 512^2 127 / 132, 8 planes 192^2 52.8 / 55.5, 256^2 88.7 / 78.6
//   mirror, else: 3 planes 384^2 266 / 305; 5 planes 192^2 128 / 131, 256^2 172 / 170;
//     15 planes 96^2 80 / 83, 128^2 128 / 121; 7 planes 256^2 224 / 257 (cuFFT is slow at
//     lengths with a factor of 7 or more); uneven 6 planes 512^2 222 / 224, 15 256^2 140 / 149
//   open (third vector not normal), pow2: 2 planes 96^2 in x, y periodic 33 / 35, 256^2 40.4 /
//     39.3, 4 planes 64^2 32.2 / 31.5; else: 3 planes 256^2 104 / 107, 5 planes 128^2 55 / 60,
//     192^2 137 / 131, 7 planes 192^2 180 / 190, 9 planes 96^2 68 / 64; uneven 6 planes 256^2
//     75 / 79, 384^2 170 / 165, 11 planes 128^2 53 / 61, 192^2 84 / 92, 9 planes 192^2 74 / 72
//   circular, pow2: 4 planes 192^2 41.6 / 41.6, 384^2 100 / 95, 8 planes 128^2 41.5 / 39.5;
//     else: 3 planes 384^2 84 / 86, 512^2 97.7 / 96.0, 9 planes 192^2 60.6 / 61.1,
//     5 planes 256^2 56.8 / 54.9, 12 planes 192^2 75.5 / 71.6, 14 192^2 87 / 91, 256^2 132 / 124
// One plane has no z part to transform: the real product is never slower (1024^2 open
// 348 us, 473 by the direct sum's complex K).
bool zdirect_pays(int mode, int lz, int64_t pc, bool even, bool pow2) {
    if (lz < 2 || lz > kZdirMax) return false;
    const int64_t w = lz * pc;
    if (mode == kZdirMirror) {
        if (pow2) return lz <= 4 ? !even || pc <= 40000 : lz <= 8 && pc <= 20000;
        return !even || lz <= 3 || w <= 400000 || lz % 7 == 0 || lz % 11 == 0 || lz % 13 == 0;
    }
    if (mode == kZdirOpen) {
        if (pow2) return lz <= 2 && pc <= 20000;
        return lz == 3 || lz == 7 || (lz <= 7 && w <= (even ? 170000 : 400000)) || (lz <= 11 && pc <= 10000) ||
               ((lz == 11 || lz == 13) && pc > 4000 && pc <= (even ? 20000 : 40000));
    }
    if (pow2) return lz <= 4 && pc <= 20000;
    return lz <= 3 ? pc <= 100000 : w <= 160000 || (lz == 14 && pc <= 20000);
}

struct KSix {
    double2 xx, xy, xz, yy, yz, zz;
};
__device__ __forceinline__ KSix load_k6(const double2* __restrict__ k, int64_t stride) {
    return KSix{__ldg(k),              __ldg(k + stride),     __ldg(k + 2 * stride),
                __ldg(k + 3 * stride), __ldg(k + 4 * stride), __ldg(k + 5 * stride)};
}
__device__ __forceinline__ void cmac(double2& acc, double2 a, double2 b) {
    acc.x = fma(a.x, b.x, fma(-a.y, b.y, acc.x));
    acc.y = fma(a.x, b.y, fma(a.y, b.x, acc.y));
}
__device__ __forceinline__ void k6_mac(double2 (&h)[3], const KSix& K, double2 mx, double2 my, double2 mz) {
    cmac(h[0], K.xx, mx);
    cmac(h[1], K.xy, mx);
    cmac(h[2], K.xz, mx);
    cmac(h[0], K.xy, my);
    cmac(h[1], K.yy, my);
    cmac(h[2], K.yz, my);
    cmac(h[0], K.xz, mz);
    cmac(h[1], K.yz, mz);
    cmac(h[2], K.zz, mz);
}

template <int NW, int ZPT, int MODE>
__global__ void __launch_bounds__(32 * NW, 2) k_zdirect(const double2* __restrict__ in, double2* __restrict__ out,
                                                        const double2* __restrict__ kd, int64_t pc, int lz, int nz,
                                                        int nk) {
    extern __shared__ double2 zs[];  // [lz][3][32]
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t col = static_cast<int64_t>(blockIdx.x) * 32 + lane;
    const bool act = col < pc;
    for (int row = w; row < 3 * lz; row += NW)
        zs[row * 32 + lane] = act ? in[static_cast<int64_t>(row) * pc + col] : make_double2(0.0, 0.0);
    __syncthreads();
    double2 h[ZPT][3];
#pragma unroll
    for (int q = 0; q < ZPT; ++q) h[q][0] = h[q][1] = h[q][2] = make_double2(0.0, 0.0);
    const int64_t ks = static_cast<int64_t>(nk) * pc;  // component stride (nk planes of K kept)
    const double2* k = kd + (act ? col : 0);
    const int nd = MODE == kZdirCircular ? nz : lz;
    KSix kp = load_k6(k, ks), km = kp;
    auto pair = [&](double2 (&acc)[3], const KSix& K, int zp) {
        const double2* m = zs + zp * 96 + lane;
        k6_mac(acc, K, m[0], m[32], m[64]);
    };
    for (int dz = 0; dz < nd; ++dz) {
        KSix np = kp, nm = km;
        if (dz + 1 < nd) {
            np = load_k6(k + static_cast<int64_t>(dz + 1) * pc, ks);
            if constexpr (MODE == kZdirOpen) nm = load_k6(k + static_cast<int64_t>(nz - dz - 1) * pc, ks);
        }
        if constexpr (MODE == kZdirMirror) {
            km = kp;
            km.xz = make_double2(-kp.xz.x, -kp.xz.y);
            km.yz = make_double2(-kp.yz.x, -kp.yz.y);
        }
#pragma unroll
        for (int q = 0; q < ZPT; ++q) {
            const int z = w + NW * q;
            if (z >= lz) continue;
            if constexpr (MODE == kZdirCircular) {
                const int zp = z - dz;
                pair(h[q], kp, zp < 0 ? zp + nz : zp);
            } else {
                if (z - dz >= 0) pair(h[q], kp, z - dz);
                if (dz > 0 && z + dz < lz) pair(h[q], km, z + dz);
            }
        }
        kp = np;
        if constexpr (MODE == kZdirOpen) km = nm;
    }
    if (!act) return;
#pragma unroll
    for (int q = 0; q < ZPT; ++q) {
        const int z = w + NW * q;
        if (z >= lz) continue;
#pragma unroll
        for (int c = 0; c < 3; ++c) out[(static_cast<int64_t>(z) * 3 + c) * pc + col] = h[q][c];
    }
}

mj_status cufft_status(cufftResult r, const char* where) {
    if (r == CUFFT_SUCCESS) return MJ_OK;
    return set_error(MJ_ERR_CUDA, std::string("cuFFT error ") + std::to_string(static_cast<int>(r)) + " in " + where);
}

void free_plan(DipolarPlan* d) {
    if (!d) return;
    if (d->have_f2d) cufftDestroy(d->f2d);
    if (d->have_fz) cufftDestroy(d->fz);
    if (d->have_b2d) cufftDestroy(d->b2d);
    cudaFree(d->d_pad);
    cudaFree(d->d_h);
    cudaFree(d->d_cx);
    cudaFree(d->d_cz);
    cudaFree(d->d_kfr);
    cudaFree(d->d_kfc);
    cudaFree(d->d_kd);
    cudaFree(d->d_kzr);
    cudaFree(d->d_kzc);
    delete d;
}

// K_F (device, complex, taken over) kept as 6 real values per wave vector when its imaginary
// parts are rounding, else as it is; with `columns` also in k_zconv's layout.
mj_status keep_kf(DipolarPlan* d, cufftDoubleComplex* kf, bool columns) {
    const int nz = d->nrep[2];
    const int64_t nkc = d->pc * nz;
    mj_status st = MJ_OK;
    auto al = [&](auto** ptr, size_t bytes, const char* what) {
        return cuda_status(cudaMalloc(reinterpret_cast<void**>(ptr), bytes), what);
    };
    std::vector<cufftDoubleComplex> h(static_cast<size_t>(6) * nkc);
    if ((st = cuda_status(cudaMemcpy(h.data(), kf, sizeof(cufftDoubleComplex) * h.size(), cudaMemcpyDeviceToHost),
                          "K_F download")) != MJ_OK) {
        cudaFree(kf);
        return st;
    }
    double re = 0.0, im = 0.0;
    for (const cufftDoubleComplex& c : h) {
        re = std::max(re, std::fabs(c.x));
        im = std::max(im, std::fabs(c.y));
    }
    d->real_kf = im <= 1e-13 * re;
    // the fused z convolution's K_F: per column, kz in the lanes' bit-reversed order
    if (columns) {
        int bits = 0;
        while ((1 << bits) < nz) ++bits;
        auto bitrev = [&](int l) {
            int r = 0;
            for (int b = 0; b < bits; ++b) r |= ((l >> b) & 1) << (bits - 1 - b);
            return r;
        };
        const size_t ncol = static_cast<size_t>(d->pc);
        if (d->real_kf) {
            std::vector<double> kz(ncol * nz * 6);
            for (size_t col = 0; col < ncol; ++col)
                for (int c = 0; c < 6; ++c)
                    for (int l = 0; l < nz; ++l)
                        kz[(col * 6 + c) * nz + l] =
                            h[static_cast<size_t>(c) * nkc + static_cast<size_t>(bitrev(l)) * ncol + col].x;
            st = al(&d->d_kzr, sizeof(double) * kz.size(), "dipolar K_F columns");
            if (st == MJ_OK)
                st = cuda_status(cudaMemcpy(d->d_kzr, kz.data(), sizeof(double) * kz.size(), cudaMemcpyHostToDevice),
                                 "K_F columns upload");
        } else {
            std::vector<cufftDoubleComplex> kz(ncol * nz * 6);
            for (size_t col = 0; col < ncol; ++col)
                for (int c = 0; c < 6; ++c)
                    for (int l = 0; l < nz; ++l)
                        kz[(col * 6 + c) * nz + l] =
                            h[static_cast<size_t>(c) * nkc + static_cast<size_t>(bitrev(l)) * ncol + col];
            st = al(&d->d_kzc, sizeof(cufftDoubleComplex) * kz.size(), "dipolar K_F columns");
            if (st == MJ_OK)
                st = cuda_status(cudaMemcpy(d->d_kzc, kz.data(), sizeof(cufftDoubleComplex) * kz.size(),
                                            cudaMemcpyHostToDevice),
                                 "K_F columns upload");
        }
        if (st != MJ_OK) {
            cudaFree(kf);
            return st;
        }
        // exp(-2 pi i m / nz), m < nz / 2, rounded once from long double
        const long double pi = 3.141592653589793238462643383279502884L;
        for (int m = 0; m < nz / 2; ++m) {
            const long double a = 2.0L * pi * static_cast<long double>(m) / static_cast<long double>(nz);
            d->tw[m] = static_cast<double>(std::cos(a));
            d->tw[16 + m] = static_cast<double>(-std::sin(a));
        }
        d->zconv = true;
    }
    if (d->real_kf) {
        std::vector<double> r(h.size());
        for (size_t q = 0; q < h.size(); ++q) r[q] = h[q].x;
        if ((st = al(&d->d_kfr, sizeof(double) * r.size(), "dipolar K_F")) != MJ_OK ||
            (st = cuda_status(cudaMemcpy(d->d_kfr, r.data(), sizeof(double) * r.size(), cudaMemcpyHostToDevice),
                              "K_F upload")) != MJ_OK) {
            cudaFree(kf);
            cudaFree(d->d_kfr);
            d->d_kfr = nullptr;
            return st;
        }
        cudaFree(kf);
    } else {
        d->d_kfc = kf;
    }
    return MJ_OK;
}

// K_F's z transform input from the planes that the direct sum keeps: plane z, or with the
// mirror plane nz - z with xz and yz negated (no pair of sites is lz planes apart: zero).
__global__ void k_unfold(const cufftDoubleComplex* __restrict__ kd, cufftDoubleComplex* __restrict__ kf, int64_t pc, int nz,
                         int nkd, double f) {
    const int64_t q = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (q >= 6 * pc * nz) return;
    const int c = static_cast<int>(q / (pc * nz)), z = static_cast<int>(q / pc % nz);
    const int zs = z < nkd ? z : nz - z;
    if (zs >= nkd) {
        kf[q] = make_cuDoubleComplex(0.0, 0.0);
        return;
    }
    const double g = z >= nkd && (c == 2 || c == 4) ? -f : f;
    const cufftDoubleComplex v = kd[(static_cast<int64_t>(c) * nkd + zs) * pc + q % pc];
    kf[q] = make_cuDoubleComplex(g * v.x, g * v.y);
}

}  // namespace

mj_status dipolar_create(mj_plan* p, const std::vector<double>& K, cudaStream_t s) {
    DipolarPlan* d = new DipolarPlan();
    for (int k = 0; k < 3; ++k) d->nrep[k] = p->nrep[k];
    d->lz = p->sp.L[2];
    const int nx = d->nrep[0], ny = d->nrep[1], nz = d->nrep[2];
    const int nkx = nx / 2 + 1;
    const bool pow2 = nz >= 2 && nz <= 32 && (nz & (nz - 1)) == 0;  // k_zconv serves it
    d->pr = static_cast<int64_t>(ny) * nx;
    d->pc = static_cast<int64_t>(ny) * nkx;
    const int64_t nk = d->pr * nz, nkc = d->pc * nz;
    mj_status st = MJ_OK;
    auto fail = [&](mj_status e) {
        free_plan(d);
        return e;
    };
    if (d->lz > nz) return fail(set_error(MJ_ERR_ARG, "dipolar grid smaller than the lattice"));
    auto al = [&](auto** ptr, size_t bytes, const char* what) {
        return cuda_status(cudaMalloc(reinterpret_cast<void**>(ptr), bytes), what);
    };
    if ((st = al(&d->d_pad, sizeof(double) * 3 * d->pr * d->lz, "dipolar pad")) != MJ_OK ||
        (st = al(&d->d_h, sizeof(double) * 3 * d->pr * d->lz, "dipolar H")) != MJ_OK ||
        (st = al(&d->d_cx, sizeof(cufftDoubleComplex) * 3 * nkc, "dipolar spectra")) != MJ_OK ||
        (st = al(&d->d_cz, sizeof(cufftDoubleComplex) * 3 * nkc, "dipolar spectra")) != MJ_OK)
        return fail(st);
    // zero once: the pad outside the lattice rows/columns and the spectra planes z >= Lz
    if ((st = cuda_status(cudaMemsetAsync(d->d_pad, 0, sizeof(double) * 3 * d->pr * d->lz, s), "dipolar memset")) != MJ_OK ||
        (st = cuda_status(cudaMemsetAsync(d->d_cx, 0, sizeof(cufftDoubleComplex) * 3 * nkc, s), "dipolar memset")) != MJ_OK)
        return fail(st);

    // K of the six unique components: its transform along y and x (direct z sum), or K_F on
    // the full grid (3D transform), each scaled by one over the points transformed, once
    std::vector<double> k6(static_cast<size_t>(6) * nk);
    const int sel[6] = {0, 1, 2, 4, 5, 8};
    for (int c = 0; c < 6; ++c)
        for (int64_t q = 0; q < nk; ++q) k6[static_cast<size_t>(c) * nk + q] = K[static_cast<size_t>(q) * 9 + sel[c]];
    // K's symmetries where the choice depends on them: the mirror in z (open axis), value by
    // value, and K(-r) = K(r)
    auto pays = [&](int mode, bool even) { return zdirect_pays(mode, d->lz, d->pc, even, pow2); };
    auto mirrored = [&]() {
        for (int c = 0; c < 6; ++c) {
            const double sg = (c == 2 || c == 4) ? -1.0 : 1.0;
            for (int z = 1; z < d->lz; ++z) {
                const double* a = &k6[static_cast<size_t>(c) * nk + static_cast<size_t>(z) * d->pr];
                const double* b = &k6[static_cast<size_t>(c) * nk + static_cast<size_t>(nz - z) * d->pr];
                for (int64_t q = 0; q < d->pr; ++q)
                    if (a[q] != sg * b[q]) return false;
            }
        }
        return true;
    };
    auto is_even = [&]() {  // (from two planes: it decides the route's speed alone)
        double top = 0.0, odd = 0.0;
        for (int c = 0; c < 6; ++c)
            for (int z = 0; z < std::min(nz, 2); ++z)
                for (int y = 0; y < ny; ++y) {
                    const double* a = &k6[static_cast<size_t>(c) * nk + static_cast<size_t>(z) * d->pr + static_cast<size_t>(y) * nx];
                    const double* b = &k6[static_cast<size_t>(c) * nk + static_cast<size_t>((nz - z) % nz) * d->pr +
                                          static_cast<size_t>((ny - y) % ny) * nx];
                    for (int x = 0; x < nx; ++x) {
                        top = std::max(top, std::fabs(a[x]));
                        odd = std::max(odd, std::fabs(a[x] - b[x == 0 ? 0 : nx - x]));
                    }
                }
        return odd <= 1e-12 * top;
    };
    int zmode = kZdirCircular;
    if (nz >= 2 * d->lz) {
        const bool either = pays(kZdirMirror, true) || pays(kZdirMirror, false) || pays(kZdirOpen, true) || pays(kZdirOpen, false);
        zmode = either && mirrored() ? kZdirMirror : kZdirOpen;
    }
    const bool direct = pays(zmode, true) == pays(zmode, false) ? pays(zmode, true) : pays(zmode, is_even());
    const int planes = direct && zmode == kZdirMirror ? d->lz : nz;  // of K that are transformed
    {
        double* d_k6 = nullptr;
        cufftDoubleComplex* kf = nullptr;
        if ((st = al(&d_k6, sizeof(double) * 6 * planes * d->pr, "dipolar K")) != MJ_OK) return fail(st);
        if ((st = al(&kf, sizeof(cufftDoubleComplex) * 6 * planes * d->pc, "dipolar K_F")) != MJ_OK) {
            cudaFree(d_k6);
            return fail(st);
        }
        const size_t part = sizeof(double) * static_cast<size_t>(planes) * d->pr;  // a component's planes
        cudaError_t up = cudaSuccess;
        for (int c = 0; c < 6 && up == cudaSuccess; ++c)
            up = cudaMemcpyAsync(d_k6 + static_cast<int64_t>(c) * planes * d->pr, &k6[static_cast<size_t>(c) * nk], part,
                                 cudaMemcpyHostToDevice, s);
        int dims[3] = {nz, ny, nx}, inembed[3] = {nz, ny, nx}, onembed[3] = {nz, ny, nkx};
        const int rank = direct ? 2 : 3, batch = direct ? 6 * planes : 6, o = 3 - rank;
        const int64_t npc = static_cast<int64_t>(planes) * d->pc;
        cufftHandle pk;
        cufftResult r = up == cudaSuccess
                            ? cufftPlanMany(&pk, rank, dims + o, inembed + o, 1, static_cast<int>(direct ? d->pr : nk),
                                            onembed + o, 1, static_cast<int>(direct ? d->pc : nkc), CUFFT_D2Z, batch)
                            : CUFFT_EXEC_FAILED;
        if (r == CUFFT_SUCCESS) {
            cufftSetStream(pk, s);
            r = cufftExecD2Z(pk, d_k6, kf);
            if (r == CUFFT_SUCCESS)
                k_scale<<<static_cast<unsigned>((6 * npc + 255) / 256), 256, 0, s>>>(
                    kf, 6 * npc, 1.0 / static_cast<double>(direct ? d->pr : nk));
            cudaStreamSynchronize(s);
            cufftDestroy(pk);
        }
        cudaFree(d_k6);
        if (r != CUFFT_SUCCESS) {
            cudaFree(kf);
            return fail(cufft_status(r, "K transform"));
        }
        if (direct) {
            d->zdir = 1 + zmode;
            d->nkd = planes;
            d->d_kd = kf;
        } else if ((st = keep_kf(d, kf, pow2)) != MJ_OK) {
            return fail(st);
        }
    }
    // 2D real transforms over (y, x) of the lattice planes, batched over (z < Lz, component)
    {
        int n2[2] = {ny, nx}, in2[2] = {ny, nx}, on2[2] = {ny, nkx};
        cufftResult r = cufftPlanMany(&d->f2d, 2, n2, in2, 1, static_cast<int>(d->pr), on2, 1, static_cast<int>(d->pc),
                                      CUFFT_D2Z, 3 * d->lz);
        if (r != CUFFT_SUCCESS) return fail(cufft_status(r, "2D forward plan"));
        d->have_f2d = true;
        r = cufftPlanMany(&d->b2d, 2, n2, on2, 1, static_cast<int>(d->pc), in2, 1, static_cast<int>(d->pr), CUFFT_Z2D,
                          3 * d->lz);
        if (r != CUFFT_SUCCESS) return fail(cufft_status(r, "2D backward plan"));
        d->have_b2d = true;
    }
    // complex transforms along z: one line per (component, ky, kx), stride 3 pc
    if (nz > 1) {
        int nz1[1] = {nz}, emb[1] = {nz};
        const int stride = static_cast<int>(3 * d->pc);
        cufftResult r = cufftPlanMany(&d->fz, 1, nz1, emb, stride, 1, emb, stride, 1, CUFFT_Z2Z, stride);
        if (r != CUFFT_SUCCESS) return fail(cufft_status(r, "z plan"));
        d->have_fz = true;
    }
    p->dip = d;
    return MJ_OK;
}

mj_status dipolar_transforms(mj_plan* p) {
    DipolarPlan* d = static_cast<DipolarPlan*>(p->dip);
    if (!d || !d->zdir || d->d_kfr || d->d_kfc) return MJ_OK;
    const int nz = d->nrep[2];
    const int64_t nkc = d->pc * nz;
    cufftDoubleComplex* kf = nullptr;
    mj_status st = cuda_status(cudaMalloc(&kf, sizeof(cufftDoubleComplex) * 6 * nkc), "dipolar K_F");
    if (st != MJ_OK) return st;
    k_unfold<<<static_cast<unsigned>((6 * nkc + 255) / 256), 256>>>(d->d_kd, kf, d->pc, nz, d->nkd,
                                                                    1.0 / static_cast<double>(nz));
    st = cuda_status(cudaGetLastError(), "k_unfold");
    if (st == MJ_OK && nz > 1) {  // along z, a line per column
        int n1[1] = {nz}, emb[1] = {nz};
        const int stride = static_cast<int>(d->pc);
        cufftHandle pz;
        cufftResult r = cufftPlanMany(&pz, 1, n1, emb, stride, 1, emb, stride, 1, CUFFT_Z2Z, stride);
        if (r == CUFFT_SUCCESS) {
            for (int c = 0; c < 6 && r == CUFFT_SUCCESS; ++c) r = cufftExecZ2Z(pz, kf + c * nkc, kf + c * nkc, CUFFT_FORWARD);
            cudaStreamSynchronize(0);
            cufftDestroy(pz);
        }
        if (r != CUFFT_SUCCESS) st = cufft_status(r, "K z transform");
    }
    if (st != MJ_OK) {
        cudaFree(kf);
        return st;
    }
    return keep_kf(d, kf, false);
}

void dipolar_destroy(mj_plan* p) {
    free_plan(static_cast<DipolarPlan*>(p->dip));
    p->dip = nullptr;
}

mj_status dipolar_apply(mj_plan* p, const double* m, double* /*H unused: consumers read the padded grid*/,
                        cudaStream_t s) {
    DipolarPlan* d = static_cast<DipolarPlan*>(p->dip);
    if (!d) return set_error(MJ_ERR_ARG, "dipolar plan missing");
    const int64_t N = p->N;
    const int64_t nkc = d->pc * d->nrep[2];
    mj_status st = MJ_OK;
    // the pass that wrote m may have written the padded grid as well
    if (p->dip_pad_holds != m) {
        k_pad<<<static_cast<unsigned>((N + 255) / 256), 256, 0, s>>>(m, d->d_pad, p->sp.L[0], p->sp.L[1], p->sp.L[2],
                                                                      d->nrep[0], d->pr);
        if ((st = cuda_status(cudaGetLastError(), "k_pad")) != MJ_OK) return st;
    }
    p->dip_pad_holds = nullptr;
    cufftSetStream(d->f2d, s);
    cufftSetStream(d->b2d, s);
    if (d->have_fz) cufftSetStream(d->fz, s);
    // planes z < Lz of d_cx; the rest of it stays zero
    if ((st = cufft_status(cufftExecD2Z(d->f2d, d->d_pad, d->d_cx), "2D D2Z")) != MJ_OK) return st;
    if (d->zdir && p->dip_zconv) {
        const double2* in = reinterpret_cast<const double2*>(d->d_cx);
        double2* out = reinterpret_cast<double2*>(d->d_cz);
        const double2* kd = reinterpret_cast<const double2*>(d->d_kd);
        const unsigned nb = static_cast<unsigned>((d->pc + 31) / 32);
        const size_t smem = sizeof(double2) * 96 * d->lz;
        const int nz = d->nrep[2];
        auto go = [&](auto nw, auto zpt) {
            constexpr int W = decltype(nw)::value, Z = decltype(zpt)::value;
            auto run = [&](auto mode) {
                k_zdirect<W, Z, decltype(mode)::value><<<nb, 32 * W, smem, s>>>(in, out, kd, d->pc, d->lz, nz, d->nkd);
            };
            switch (d->zdir - 1) {
                case kZdirMirror: run(std::integral_constant<int, kZdirMirror>{}); break;
                case kZdirOpen: run(std::integral_constant<int, kZdirOpen>{}); break;
                default: run(std::integral_constant<int, kZdirCircular>{}); break;
            }
        };
        using std::integral_constant;
        if (d->lz <= 4) go(integral_constant<int, 4>{}, integral_constant<int, 1>{});
        else if (d->lz <= 8) go(integral_constant<int, 8>{}, integral_constant<int, 1>{});
        else go(integral_constant<int, 8>{}, integral_constant<int, 2>{});
        st = cuda_status(cudaGetLastError(), "k_zdirect");
        if (st != MJ_OK) return st;
        return cufft_status(cufftExecZ2D(d->b2d, d->d_cz, d->d_h), "2D Z2D");
    }
    if (d->zconv && p->dip_zconv) {
        // z transforms and product in one pass, into the planes z < Lz of d_cz
        ZTwiddle W;
        for (int m = 0; m < 16; ++m) {
            W.c[m] = d->tw[m];
            W.s[m] = d->tw[16 + m];
        }
        const int nz = d->nrep[2];
        const double2* in = reinterpret_cast<const double2*>(d->d_cx);
        double2* out = reinterpret_cast<double2*>(d->d_cz);
        const double2* kc = reinterpret_cast<const double2*>(d->d_kzc);
        auto go = [&](auto nzc) {
            constexpr int NZ = decltype(nzc)::value;
            using Z = ZcGeom<NZ>;
            const unsigned nb = static_cast<unsigned>((d->pc + Z::C - 1) / Z::C);
            if (d->real_kf) k_zconv<NZ, true><<<nb, 256, Z::smem, s>>>(in, out, d->d_kzr, kc, d->pc, d->lz, W);
            else k_zconv<NZ, false><<<nb, 256, Z::smem, s>>>(in, out, d->d_kzr, kc, d->pc, d->lz, W);
        };
        switch (nz) {
            case 2: go(std::integral_constant<int, 2>{}); break;
            case 4: go(std::integral_constant<int, 4>{}); break;
            case 8: go(std::integral_constant<int, 8>{}); break;
            case 16: go(std::integral_constant<int, 16>{}); break;
            default: go(std::integral_constant<int, 32>{}); break;
        }
        if ((st = cuda_status(cudaGetLastError(), "k_zconv")) != MJ_OK) return st;
        return cufft_status(cufftExecZ2D(d->b2d, d->d_cz, d->d_h), "2D Z2D");
    }
    cufftDoubleComplex* spec = d->d_cx;
    if (d->have_fz) {
        if ((st = cufft_status(cufftExecZ2Z(d->fz, d->d_cx, d->d_cz, CUFFT_FORWARD), "z forward")) != MJ_OK) return st;
        spec = d->d_cz;
    }
    if (d->real_kf)
        k_pointwise_real<<<static_cast<unsigned>((nkc + 255) / 256), 256, 0, s>>>(spec, d->d_kfr, d->pc, nkc);
    else
        k_pointwise_cplx<<<static_cast<unsigned>((nkc + 255) / 256), 256, 0, s>>>(spec, d->d_kfc, d->pc, nkc);
    if ((st = cuda_status(cudaGetLastError(), "k_pointwise")) != MJ_OK) return st;
    if (d->have_fz && (st = cufft_status(cufftExecZ2Z(d->fz, d->d_cz, d->d_cz, CUFFT_INVERSE), "z inverse")) != MJ_OK)
        return st;
    // H of the lattice planes: the first 3 Lz complex planes of the spectrum
    return cufft_status(cufftExecZ2D(d->b2d, spec, d->d_h), "2D Z2D");
}

DipPad dipolar_pad(const mj_plan* p) {
    const DipolarPlan* d = static_cast<const DipolarPlan*>(p->dip);
    if (!p->dip_on || !d) return DipPad{nullptr, 0, 0, 0};
    return DipPad{d->d_pad, d->pr, 3 * d->pr, d->nrep[0]};
}

DipView dipolar_view(const mj_plan* p) {
    DipView v;
    const DipolarPlan* d = static_cast<const DipolarPlan*>(p->dip);
    if (!p->dip_on || !d) {
        v.h = nullptr;
        v.cs = v.zs = 0;
        v.px = 0;
        return v;
    }
    v.h = d->d_h;
    v.cs = d->pr;
    v.zs = 3 * d->pr;
    v.px = d->nrep[0];
    return v;
}

}  // namespace mj
