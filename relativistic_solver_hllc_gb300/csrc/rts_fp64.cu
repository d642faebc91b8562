// rts_fp64.cu -- FP64 CUDA-core kernels of the scattering path:
//   * the plain FP64 scattering integral (replaces d_GetS / d_GetS_MPI /
//     d_GetS_MPI_Stream, cuda/cuda_kernel.cu:23-111), with the source update
//     and the FP64 residual fused into its epilogue;
//   * the direction-pair weights W (Gamma of cuda/cuda_utils.cu:7-16 times
//     area_j / full_area, or renormalised Henyey-Greenstein);
//   * FP64 energy and flux moments (cuda/cuda_utils.cu:18-67,
//     cuda/cuda_kernel.cu:113-134) in one pass over Illum;
//   * standalone source update / residual and the FP64 relaxation step;
//   * the synthetic lognormal Illum generator.
//
// The reference kernel gives each thread one (cell, out-direction) pair and
// loops over all in-directions, re-reading the 4 faces and recomputing Gamma
// for every pair and accumulating straight into global memory.  Here a CTA
// owns a 128-cell x 64-out-direction tile (the out-directions left over
// past a multiple of 64 take one narrower tile): the face mean is taken once per
// (in-direction, cell) while the tile of Ibar is staged in shared memory, W
// (FP64, precomputed once) is staged beside it, and each thread keeps an
// 8-cell x 4-direction block of accumulators in registers.  GB300 FP64 runs
// at a small fraction of its FP32 rate, so this kernel is FP64-pipe bound by
// design; memory traffic is ~40 B per cell-direction pair over M in-directions.
#include <cstdint>
#include <mutex>
#include <type_traits>

#include "rts_internal.h"

namespace {

constexpr int F64_TC = 128;  // cells per CTA
constexpr int F64_TK = 64;   // out-directions per CTA
constexpr int F64_KC = 16;   // in-directions per shared-memory chunk
constexpr int F64_THREADS = 256;

__device__ __forceinline__ double warp_max(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Residual bits: non-negative doubles order the same as their bit patterns.
__device__ __forceinline__ void residual_max(unsigned long long* dst, double v)
{
    v = warp_max(v);
    if ((threadIdx.x & 31) == 0 && v > 0.0)
        atomicMax(dst, (unsigned long long)__double_as_longlong(v));
}

// One tile of 128 cells x 16*NB out-directions [k0, k0 + 16*NB): each
// thread keeps 8 cells x NB directions of accumulators.  Every output is the
// same FMA chain over the in-directions in order whatever NB, so a tile's
// width changes no result.  GB300's FP64 pipe retires about two FMAs per SM
// per cycle, far below the shared-memory loads that feed them, so a narrow
// tile costs about NB/4 of a full one.
//
// kList: the tile's cells are entries [c0, n) of fx.list instead of
// consecutive ones, and only the outputs marked in fx.mask are written.
struct ListArgs {
    const unsigned int* list;  // null: the identity (every cell)
    const unsigned int* mask;  // [quarter tile][ld], a bit per column; null: every output
    int64_t ld;
    int bn, k_base;
    __device__ bool marked(int64_t c, int k) const
    {
        if (!mask) return true;
        const int kk = k - k_base, group = kk / (bn / 4);  // a word per quarter tile
        return (mask[(int64_t)group * ld + c] >> (kk - group * (bn / 4))) & 1u;
    }
};

template <bool kUpdate, bool kResidual, int NB, bool kList = false>
__device__ __forceinline__ void scatter_tile(double (*sI)[F64_TC], double (*sW)[F64_TK],
                                             const double* __restrict__ illum, const double* __restrict__ W,
                                             int64_t c0, int64_t n, int64_t N, int M, int ldw, int k0, int k_end,
                                             double* __restrict__ S, const double* __restrict__ B, double lambda,
                                             unsigned long long* __restrict__ resid, const ListArgs& fx = ListArgs())
{
    constexpr int TK = 16 * NB;
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    // cell of list position p < n
    auto cell = [&](int64_t p) { return kList && fx.list ? (int64_t)fx.list[p] : p; };

    double acc[NB][8];
#pragma unroll
    for (int m = 0; m < NB; ++m)
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[m][i] = 0.0;

    for (int j0 = 0; j0 < M; j0 += F64_KC) {
        // Ibar chunk: F64_KC x 128 (in-direction, cell) pairs, 8 per thread;
        // consecutive threads read consecutive cells' 32-byte face groups.
#pragma unroll
        for (int q = 0; q < (F64_KC * F64_TC) / F64_THREADS; ++q) {
            const int p = tid + F64_THREADS * q;
            const int jj = p / F64_TC, cc = p % F64_TC;
            const int j = j0 + jj;
            const int64_t c = c0 + cc;
            double v = 0.0;
            if (j < M && c < n) {
                const double2* src = reinterpret_cast<const double2*>(illum + ((int64_t)j * N + cell(c)) * 4);
                const double2 a = __ldg(src), b = __ldg(src + 1);
                double I = 0.0;  // faces 0..3 in order, then /4 (GET_FACE_TO_CELL)
                I += a.x;
                I += a.y;
                I += b.x;
                I += b.y;
                v = I / 4;
            }
            sI[jj][cc] = v;
        }
        // W chunk: F64_KC x TK, NB per thread
#pragma unroll
        for (int q = 0; q < (F64_KC * TK) / F64_THREADS; ++q) {
            const int p = tid + F64_THREADS * q;
            const int jj = p / TK, kk = p % TK;
            const int j = j0 + jj, k = k0 + kk;
            sW[jj][kk] = (j < M && k < k_end) ? __ldg(W + (int64_t)j * ldw + k) : 0.0;
        }
        __syncthreads();
#pragma unroll
        for (int jj = 0; jj < F64_KC; ++jj) {
            double iv[8], wv[NB];
#pragma unroll
            for (int i = 0; i < 8; ++i) iv[i] = sI[jj][tx + 16 * i];
#pragma unroll
            for (int m = 0; m < NB; ++m) wv[m] = sW[jj][ty + 16 * m];
#pragma unroll
            for (int m = 0; m < NB; ++m)
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[m][i] = fma(wv[m], iv[i], acc[m][i]);
        }
        __syncthreads();
    }

    double rmax = 0.0;
#pragma unroll
    for (int m = 0; m < NB; ++m) {
        const int k = k0 + ty + 16 * m;
        if (k >= k_end) continue;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (c0 + tx + 16 * i >= n) continue;
            const int64_t c = cell(c0 + tx + 16 * i);
            if (kList && !fx.marked(c, k)) continue;
            double v = acc[m][i];
            if (kUpdate) v = (1.0 - lambda) * B[c] + lambda * v;
            double* dst = S + (int64_t)k * N + c;
            if (kResidual) rmax = fmax(rmax, fabs(v - *dst));
            *dst = v;
        }
    }
    if (kResidual) residual_max(resid, rmax);
}

// Grid: x over 128-cell tiles; y over the out-directions [k_begin, k_end),
// n_full tiles of 64 and then, when the range is not a multiple of 64, one
// tile of 16*nb_last (nb_last 1..4) for the rest.  The narrow tiles are last
// in launch order, so they fill the final wave.
template <bool kUpdate, bool kResidual>
__global__ void __launch_bounds__(F64_THREADS, 2)
scatter_fp64_kernel(const double* __restrict__ illum, const double* __restrict__ W, int64_t n, int64_t N,
                    int M, int ldw, int k_begin, int k_end, int n_full, int nb_last, double* __restrict__ S,
                    const double* __restrict__ B, double lambda,
                    unsigned long long* __restrict__ resid)
{
    __shared__ double sI[F64_KC][F64_TC];
    __shared__ double sW[F64_KC][F64_TK];
    const int64_t c0 = (int64_t)blockIdx.x * F64_TC;
    const int k0 = k_begin + (int)blockIdx.y * F64_TK;
    const int nb = (int)blockIdx.y < n_full ? 4 : nb_last;
    switch (nb) {
    case 1:
        scatter_tile<kUpdate, kResidual, 1>(sI, sW, illum, W, c0, n, N, M, ldw, k0, k_end, S, B, lambda, resid);
        break;
    case 2:
        scatter_tile<kUpdate, kResidual, 2>(sI, sW, illum, W, c0, n, N, M, ldw, k0, k_end, S, B, lambda, resid);
        break;
    case 3:
        scatter_tile<kUpdate, kResidual, 3>(sI, sW, illum, W, c0, n, N, M, ldw, k0, k_end, S, B, lambda, resid);
        break;
    default:
        scatter_tile<kUpdate, kResidual, 4>(sI, sW, illum, W, c0, n, N, M, ldw, k0, k_end, S, B, lambda, resid);
        break;
    }
}

// Tiles of 32 cells x 32 out-directions for problems whose 128 x 64 tiles would
// leave SMs idle: 2,000 x 64 makes 16 of those, each a serial loop of loads,
// barriers and FMAs (152 us), and 126 of these (23 us).  A chunk's operands are
// loaded while the previous one is multiplied, one barrier a chunk.  Every output
// is the same FMA chain as in the larger tiles.  kList as in scatter_tile.
constexpr int S64_T = 32, S64_KC = 16, S64_THREADS = 256;
template <bool kUpdate, bool kList = false>
__device__ __forceinline__ void scatter_small_tile(double (*sI)[S64_KC][S64_T], double (*sW)[S64_KC][S64_T],
                                                   const double* __restrict__ illum, const double* __restrict__ W,
                                                   int64_t c0, int64_t n, int64_t N, int M, int ldw, int k0, int k_end,
                                                   double* __restrict__ S, const double* __restrict__ B, double lambda,
                                                   unsigned long long* __restrict__ resid,
                                                   const ListArgs& fx = ListArgs())
{
    constexpr int PER = S64_KC * S64_T / S64_THREADS;  // pairs of a chunk per thread: 2
    const int tx = threadIdx.x & (S64_T - 1), ty = threadIdx.x / S64_T;
    const bool in = c0 + tx < n;
    const int64_t c = kList && in && fx.list ? (int64_t)fx.list[c0 + tx] : c0 + tx;
    double2 p[PER], q[PER];
    double w[PER];
    auto load = [&](int j0) {
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int j = j0 + ty + (S64_THREADS / S64_T) * i;
            p[i] = q[i] = make_double2(0.0, 0.0);
            if (j < M && in) {
                const double2* src = reinterpret_cast<const double2*>(illum + ((int64_t)j * N + c) * 4);
                p[i] = __ldg(src);
                q[i] = __ldg(src + 1);
            }
            w[i] = (j < M && k0 + tx < k_end) ? __ldg(W + (int64_t)j * ldw + k0 + tx) : 0.0;
        }
    };
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    load(0);
    int b = 0;
    for (int j0 = 0; j0 < M; j0 += S64_KC, b ^= 1) {
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int jj = ty + (S64_THREADS / S64_T) * i;
            double I = 0.0;  // faces 0..3 in order, then /4 (GET_FACE_TO_CELL)
            I += p[i].x;
            I += p[i].y;
            I += q[i].x;
            I += q[i].y;
            sI[b][jj][tx] = I / 4;
            sW[b][jj][tx] = w[i];
        }
        __syncthreads();
        if (j0 + S64_KC < M) load(j0 + S64_KC);
        const int nj = min(S64_KC, M - j0);
        if (nj == S64_KC) {
#pragma unroll
            for (int jj = 0; jj < S64_KC; ++jj)
#pragma unroll
                for (int m = 0; m < 4; ++m) acc[m] = fma(sW[b][jj][ty + 8 * m], sI[b][jj][tx], acc[m]);
        } else {
            for (int jj = 0; jj < nj; ++jj)
#pragma unroll
                for (int m = 0; m < 4; ++m) acc[m] = fma(sW[b][jj][ty + 8 * m], sI[b][jj][tx], acc[m]);
        }
    }
    double rmax = 0.0;
    if (in) {
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const int k = k0 + ty + 8 * m;
            if (k >= k_end || (kList && !fx.marked(c, k))) continue;
            double v = acc[m];
            if (kUpdate) v = (1.0 - lambda) * B[c] + lambda * v;
            double* dst = S + (int64_t)k * N + c;
            if (resid) rmax = fmax(rmax, fabs(v - *dst));
            *dst = v;
        }
    }
    if (resid) residual_max(resid, rmax);
}

template <bool kUpdate>
__global__ void __launch_bounds__(S64_THREADS)
scatter_fp64_small_kernel(const double* __restrict__ illum, const double* __restrict__ W, int64_t n, int64_t N, int M,
                          int ldw, int k_begin, int k_end, double* __restrict__ S, const double* __restrict__ B,
                          double lambda, unsigned long long* __restrict__ resid)
{
    __shared__ double sI[2][S64_KC][S64_T], sW[2][S64_KC][S64_T];
    scatter_small_tile<kUpdate>(sI, sW, illum, W, (int64_t)blockIdx.x * S64_T, n, N, M, ldw,
                                k_begin + (int)blockIdx.y * S64_T, k_end, S, B, lambda, resid);
}

// The y extent of scatter_fp64_kernel's grid over `width` out-directions.
struct DirTiles {
    int n_full, nb_last, gy;
};
inline DirTiles dir_tiles(int64_t width)
{
    DirTiles t;
    t.n_full = (int)(width / F64_TK);
    const int rem = (int)(width % F64_TK);
    t.nb_last = rem ? (rem + 15) / 16 : 4;
    t.gy = t.n_full + (rem ? 1 : 0);
    return t;
}

// The outputs that the tensor-core route left (rts_launch_scatter_list): CTAs
// walk the tiles of the listed cells; count and list are the device's, so nothing
// waits on the host.  Usually there are none and the launch costs its latency.
// Rows that fill waves of the large tiles (two a SM) take those, the rest and
// shorter lists the 32 x 32 tiles, whose serial loop is an eighth as long (0.31
// us M against 2.2): a step of 40 x 1000 with one listed row 2,355 -> 478 us, of
// 20,000 x 400 with every row listed 7.70 -> 6.32 ms.  `taken` (zero before the
// launch) hands out the tiles, large, narrow, small, so that no SM is left with
// a large one at the end; small ones alone go round the CTAs, so that no SM takes
// two of the last (865 rows of 20,000 x 400: 0.79 ms a step, 0.90 handed out).
// stats: counts of listed rows and of contractions that gave up; residual_flag:
// set where one of a step with a residual did.
template <bool kUpdate, bool kResidual>
__global__ void __launch_bounds__(F64_THREADS, 2)
scatter_list_kernel(const double* __restrict__ illum, const double* __restrict__ W, int64_t n, int64_t N, int M,
                    int ldw, int k_begin, int k_end, DirTiles dt, int num_sms, double* __restrict__ S,
                    const double* __restrict__ B, double lambda, unsigned long long* __restrict__ resid, ListArgs fx,
                    const unsigned int* __restrict__ count, unsigned int* taken, unsigned long long* stats,
                    int* residual_flag)
{
    static_assert(F64_THREADS == S64_THREADS, "one launch for both tiles");
    __shared__ double mem[F64_KC * (F64_TC + F64_TK)];
    __shared__ unsigned int next;
    static_assert(sizeof(mem) >= sizeof(double) * 4 * S64_KC * S64_T, "both tiles' operands");
    const bool whole = count[1] != 0;  // the contraction gave up: every output of the range
    const int64_t cells = whole ? n : (int64_t)count[0];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (whole) {
            atomicAdd(stats + 1, 1ull);
            if (kResidual) atomicOr(residual_flag, (int)count[1]);
        } else if (count[0]) {
            atomicAdd(stats, (unsigned long long)count[0]);
        }
    }
    if (cells == 0) return;
    if (whole) fx.list = fx.mask = nullptr;
    // whole waves of large tiles, in quarter tiles (16 out-directions); the rest in small ones
    const int per_row = 4 * dt.n_full + (dt.gy > dt.n_full ? dt.nb_last : 0), wave = 8 * num_sms;
    const int64_t rows = cells / F64_TC * per_row / wave * wave / per_row;
    const int64_t full = rows * dt.n_full, large = rows * dt.gy, c_small = rows * F64_TC;
    const int gs = (k_end - k_begin + S64_T - 1) / S64_T;
    const int64_t work = large + (cells - c_small + S64_T - 1) / S64_T * gs;
    auto tile = [&](auto nb, int64_t row, int col) {
        auto* sI = reinterpret_cast<double(*)[F64_TC]>(mem);
        auto* sW = reinterpret_cast<double(*)[F64_TK]>(mem + F64_KC * F64_TC);
        scatter_tile<kUpdate, kResidual, decltype(nb)::value, true>(sI, sW, illum, W, row * F64_TC, cells, N, M, ldw,
                                                                    k_begin + col * F64_TK, k_end, S, B, lambda, resid,
                                                                    fx);
    };
    int64_t w = blockIdx.x;
    while (w < work) {
        if (w < full) {
            tile(std::integral_constant<int, 4>{}, w / dt.n_full, (int)(w % dt.n_full));
        } else if (w < large) {
            switch (dt.nb_last) {
            case 1: tile(std::integral_constant<int, 1>{}, w - full, dt.n_full); break;
            case 2: tile(std::integral_constant<int, 2>{}, w - full, dt.n_full); break;
            case 3: tile(std::integral_constant<int, 3>{}, w - full, dt.n_full); break;
            default: tile(std::integral_constant<int, 4>{}, w - full, dt.n_full); break;
            }
        } else {
            auto* sI = reinterpret_cast<double(*)[S64_KC][S64_T]>(mem);
            scatter_small_tile<kUpdate, true>(sI, sI + 2, illum, W, c_small + (w - large) / gs * S64_T, cells, N, M, ldw,
                                              k_begin + (int)((w - large) % gs) * S64_T, k_end, S, B, lambda,
                                              kResidual ? resid : nullptr, fx);
        }
        __syncthreads();  // the operands and the last number are read
        if (large == 0) {
            w += gridDim.x;
            continue;
        }
        if (threadIdx.x == 0) next = atomicAdd(taken, 1u);
        __syncthreads();
        w = (int64_t)gridDim.x + next;
    }
}

// Which of the two kernels: the larger tiles need four a SM (two resident at a
// time, two waves) to keep the FP64 pipe busy to the end.
inline bool small_tiles(int64_t gx, const DirTiles& dt, int num_sms) { return gx * dt.gy < 4 * num_sms; }
inline dim3 small_grid(int64_t n, int64_t width)
{
    return dim3((unsigned)((n + S64_T - 1) / S64_T), (unsigned)((width + S64_T - 1) / S64_T));
}

__device__ __forceinline__ double gamma_thomson(double ax, double ay, double az, double bx,
                                                double by, double bz)
{
    double dot = 0.0;  // x, y, z order as cuda/cuda_utils.cu:7-16
    dot += ax * bx;
    dot += ay * by;
    dot += az * bz;
    return (3. * (1 + dot * dot)) / 4;
}

// W [M][loc], a thread per element: Thomson's final, Henyey-Greenstein's before
// its columns are normalised.  Every element is a few dozen FP64 operations
// (the divisions and the square root among them) and the FP64 pipe retires two
// per SM per cycle, so the elements are spread over the whole device; a thread
// per column (the former layout) kept one to ten SMs busy with a serial loop:
// 38.7 -> 3.6 us at M = 64, 617 -> 31 us at M = 1000 (Thomson).
constexpr int WE_K = 32, WE_J = 8;  // block: 32 out-directions x 8 in-directions
__global__ void __launch_bounds__(WE_K * WE_J)
weights_kernel(const double* __restrict__ xyz, const double* __restrict__ area, int M, int k_off, int loc,
               double full_area, int phase, double g, double* __restrict__ W)
{
    const int kl = blockIdx.x * WE_K + (threadIdx.x & (WE_K - 1));
    if (kl >= loc) return;
    const int k = k_off + kl;
    const double bx = xyz[3 * k], by = xyz[3 * k + 1], bz = xyz[3 * k + 2];
    for (int j = blockIdx.y * WE_J + threadIdx.x / WE_K; j < M; j += gridDim.y * WE_J) {
        if (phase == RTS_PHASE_THOMSON) {
            W[(int64_t)j * loc + kl] =
                gamma_thomson(xyz[3 * j], xyz[3 * j + 1], xyz[3 * j + 2], bx, by, bz) * area[j] / full_area;
        } else {
            const double pi = 3.14159265358979323846264338327950288;
            const double mu = xyz[3 * j] * bx + xyz[3 * j + 1] * by + xyz[3 * j + 2] * bz;
            const double den = 1.0 + g * g - 2.0 * g * mu;
            const double kv = (1.0 - g * g) / (4.0 * pi * den * sqrt(den));
            W[(int64_t)j * loc + kl] = area[j] * kv;
        }
    }
}

// Normalises the columns of W: each divided by its sum.  A cluster of 8 CTAs
// owns 32 columns; a warp adds every 64th row of them (lane = column), the
// partial sums meet in the warps' and CTAs' order through shared and cluster
// memory, and each CTA divides its own rows -- FP64-pipe bound, like the sums
// spread over 8 SMs (a serial chain per column took 127 us at M = 1202 and 61 at
// M = 590, this 40 and 17).
constexpr int WN_CTAS = 8, WN_THREADS = 256, WN_ROWS = WN_CTAS * WN_THREADS / 32;
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}
__global__ void __cluster_dims__(1, WN_CTAS, 1) __launch_bounds__(WN_THREADS)
weights_normalise_kernel(double* __restrict__ W, int M, int loc)
{
    __shared__ double part[WN_THREADS / 32][32], ctasum[32], colsum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int kl = blockIdx.x * 32 + lane, j0 = blockIdx.y * (WN_THREADS / 32) + warp;
    double sum = 0.0;
    if (kl < loc)
#pragma unroll 4
        for (int j = j0; j < M; j += WN_ROWS) sum += W[(int64_t)j * loc + kl];
    part[warp][lane] = sum;
    __syncthreads();
    if (warp == 0) {
        for (int w = 1; w < WN_THREADS / 32; ++w) sum += part[w][lane];
        ctasum[lane] = sum;
    }
    cluster_sync();
    if (warp == 0) {
        const uint32_t mine = (uint32_t)__cvta_generic_to_shared(&ctasum[lane]);
        sum = 0.0;
        for (uint32_t r = 0; r < (uint32_t)WN_CTAS; ++r) {
            uint32_t addr;
            double x;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(mine), "r"(r));
            asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(x) : "r"(addr) : "memory");
            sum += x;
        }
        colsum[lane] = sum;
    }
    cluster_sync();  // no CTA leaves while another reads its sums; colsum is visible
    if (kl >= loc) return;
    sum = colsum[lane];
    for (int j = j0; j < M; j += WN_ROWS) W[(int64_t)j * loc + kl] /= sum;
}

// Cells (threads) per block of the moment kernels.  Every block walks all
// directions, so a launch takes as long as the SM with the most cells: 82,944 in
// blocks of 128 are 648, five on some SMs and 4.26 on average; 64 where that
// leaves the fullest SM fewer (82,944 x 400: moments_kernel 510 -> 452 us,
// illum_params_kernel 2,135 -> 2,018).  Below three blocks of 128 a SM a call is
// bound by one block's walk and keeps 128.
inline int cell_threads(int64_t N, int num_sms)
{
    auto fullest = [&](int t) { return ((N + t - 1) / t + num_sms - 1) / num_sms * t; };
    return N > (int64_t)3 * 128 * num_sms && fullest(64) < fullest(128) ? 64 : 128;
}

constexpr int MOM_DCHUNK = 256;

// Energy and flux of every cell in one pass over Illum (FP64).  Per
// direction the shared table holds area_j / 4 and w_j area_j / 4, so a
// (cell, direction) costs the face sum (3 adds) and four FMAs -- the
// reference's sum_j (sum_f I_f / 4) area_j w_j regrouped, the FP64 pipe
// being the bound.
template <int kThreads>
__global__ void __launch_bounds__(kThreads)
moments_kernel(const double* __restrict__ illum, const double* __restrict__ xyz,
               const double* __restrict__ area, int64_t N, int M, double full_area,
               double* __restrict__ energy, double* __restrict__ flux)
{
    __shared__ double sd[MOM_DCHUNK][4];
    const int64_t c = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    double e = 0.0, fx = 0.0, fy = 0.0, fz = 0.0;
    for (int j0 = 0; j0 < M; j0 += MOM_DCHUNK) {
        const int nj = min(MOM_DCHUNK, M - j0);
        for (int t = threadIdx.x; t < nj; t += kThreads) {
            const double a4 = area[j0 + t] * 0.25;  // exact
            sd[t][0] = a4;
            sd[t][1] = xyz[3 * (j0 + t)] * a4;
            sd[t][2] = xyz[3 * (j0 + t) + 1] * a4;
            sd[t][3] = xyz[3 * (j0 + t) + 2] * a4;
        }
        __syncthreads();
        if (c < N) {
            for (int jj = 0; jj < nj; ++jj) {
                const double2* src =
                    reinterpret_cast<const double2*>(illum + ((int64_t)(j0 + jj) * N + c) * 4);
                const double2 a = __ldg(src), b = __ldg(src + 1);
                const double sum = ((a.x + a.y) + b.x) + b.y;
                e = fma(sum, sd[jj][0], e);
                fx = fma(sum, sd[jj][1], fx);
                fy = fma(sum, sd[jj][2], fy);
                fz = fma(sum, sd[jj][3], fz);
            }
        }
        __syncthreads();
    }
    if (c < N) {
        energy[c] = e / full_area;
        flux[3 * c] = fx / full_area;
        flux[3 * c + 1] = fy / full_area;
        flux[3 * c + 2] = fz / full_area;
    }
}

// Energy, flux, impulse tensor and the divergences of flux and impulse of
// every cell in one pass over Illum (FP64).  The reference computes them in
// d_MakeIllumParam (cuda/cuda_kernel.cu:218-223: d_MakeEnergy :113-121,
// d_MakeDivStream :149-175, d_MakeDivImpuls :177-216) with per-face sums
// (cuda/cuda_utils.cu:86-167).  Here the per-face sums are never formed: with
// ia_f = I[j][c][f] * area_j and the face vectors nS_f = n_f * S_f,
//   flux      = sum_j w_j * (sum_f ia_f) / (4 full_area)
//   impuls    = sum_j w_j w_j^T * (sum_f ia_f) / (4 full_area)
//   divstream = sum_j (w_j . u_j) / (full_area V),   u_j = sum_f ia_f nS_f
//   divimpuls = sum_j w_j (w_j . u_j) / (full_area V)
// which are the reference's sums regrouped (the same terms, other order).
// The direction's area rides in the shared table (area_j, area_j w_j and
// area_j w_j w_j^T), so the face intensities are summed once and scaled by
// no per-cell multiply: 32 FP64 operations per (cell, direction) instead of
// the reference's 80.
constexpr int PAR_DCHUNK = 128;

template <int kThreads>
__global__ void __launch_bounds__(kThreads)
illum_params_kernel(const double* __restrict__ illum, const double* __restrict__ xyz,
                    const double* __restrict__ area, int64_t N, int M, double full_area,
                    const double* __restrict__ normals, const double* __restrict__ face_areas,
                    const double* __restrict__ volume, double* __restrict__ out)
{
    // per direction: area, area w (3), area w w^T (xx, xy, xz, yy, yz, zz), w (3)
    __shared__ double sd[PAR_DCHUNK][13];
    const int64_t c = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    const bool geo = normals != nullptr;
    double nS[4][3];
#pragma unroll
    for (int f = 0; f < 4; ++f)
#pragma unroll
        for (int d = 0; d < 3; ++d)
            nS[f][d] = (geo && c < N) ? normals[c * 12 + 3 * f + d] * face_areas[c * 4 + f] : 0.0;
    double e = 0.0, fl[3] = {0.0, 0.0, 0.0}, im[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    double ds = 0.0, di[3] = {0.0, 0.0, 0.0};
    for (int j0 = 0; j0 < M; j0 += PAR_DCHUNK) {
        const int nj = min(PAR_DCHUNK, M - j0);
        for (int t = threadIdx.x; t < nj; t += kThreads) {
            const double x = xyz[3 * (j0 + t)], y = xyz[3 * (j0 + t) + 1], z = xyz[3 * (j0 + t) + 2];
            const double a = area[j0 + t];
            sd[t][0] = a;
            sd[t][1] = a * x, sd[t][2] = a * y, sd[t][3] = a * z;
            sd[t][4] = a * (x * x), sd[t][5] = a * (x * y), sd[t][6] = a * (x * z);
            sd[t][7] = a * (y * y), sd[t][8] = a * (y * z), sd[t][9] = a * (z * z);
            sd[t][10] = x, sd[t][11] = y, sd[t][12] = z;
        }
        __syncthreads();
        if (c < N) {
            for (int jj = 0; jj < nj; ++jj) {
                const double2* src =
                    reinterpret_cast<const double2*>(illum + ((int64_t)(j0 + jj) * N + c) * 4);
                const double2 p = __ldg(src), q = __ldg(src + 1);
                const double sum = ((p.x + p.y) + q.x) + q.y;
                e = fma(sd[jj][0], sum, e);
#pragma unroll
                for (int d = 0; d < 3; ++d) fl[d] = fma(sd[jj][1 + d], sum, fl[d]);
#pragma unroll
                for (int d = 0; d < 6; ++d) im[d] = fma(sd[jj][4 + d], sum, im[d]);
                if (geo) {
                    // u = sum_f I_f nS_f; area_j w_j . u, and w_j times it
                    double u[3];
#pragma unroll
                    for (int d = 0; d < 3; ++d)
                        u[d] = fma(q.y, nS[3][d], fma(q.x, nS[2][d], fma(p.y, nS[1][d], p.x * nS[0][d])));
                    const double s = fma(sd[jj][3], u[2], fma(sd[jj][2], u[1], sd[jj][1] * u[0]));
                    ds += s;
#pragma unroll
                    for (int d = 0; d < 3; ++d) di[d] = fma(sd[jj][10 + d], s, di[d]);
                }
            }
        }
        __syncthreads();
    }
    if (c >= N) return;
    const double q4 = 1.0 / (4.0 * full_area);
    double* o = out;  // [energy N][flux 3N][impuls 9N][divstream N][divimpuls 3N]
    o[c] = e * q4;
    o += N;
#pragma unroll
    for (int d = 0; d < 3; ++d) o[3 * c + d] = fl[d] * q4;
    o += 3 * N;
    const double t[9] = {im[0], im[1], im[2], im[1], im[3], im[4], im[2], im[4], im[5]};
#pragma unroll
    for (int d = 0; d < 9; ++d) o[9 * c + d] = t[d] * q4;
    o += 9 * N;
    if (geo) {
        const double qv = 1.0 / (full_area * volume[c]);
        o[c] = ds * qv;
        o += N;
#pragma unroll
        for (int d = 0; d < 3; ++d) o[3 * c + d] = di[d] * qv;
    }
}

template <bool kResidual>
__global__ void update_kernel(double* __restrict__ S, const double* __restrict__ B, int64_t N,
                              int64_t rows, double lambda, unsigned long long* __restrict__ resid)
{
    double rmax = 0.0;
    const int64_t total = rows * N;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        const double old = S[i];
        const double v = (1.0 - lambda) * B[i % N] + lambda * old;
        if (kResidual) rmax = fmax(rmax, fabs(v - old));
        S[i] = v;
    }
    if (kResidual) residual_max(resid, rmax);
}

// Illum[j][c][f] <- 0.5 Illum[j][c][f] + 0.5 S[j][c], a thread per (j, c).  72
// bytes and five FP64 operations a pair (0.5 Illum is exact, so one fused
// multiply-add is the sum's only rounding): memory bound, 30,011 x 302 in 95 us
// (96 at the copy rate; 145 with nine FP64 operations and a grid-stride loop).
__global__ void __launch_bounds__(256) relax_fp64_kernel(double* __restrict__ illum, const double* __restrict__ S,
                                                         int64_t pairs)
{
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= pairs) return;
    const double h = 0.5 * S[i];
    double2* p = reinterpret_cast<double2*>(illum + i * 4);
    const double2 a = p[0], b = p[1];
    p[0] = make_double2(fma(0.5, a.x, h), fma(0.5, a.y, h));
    p[1] = make_double2(fma(0.5, b.x, h), fma(0.5, b.y, h));
}

// Counter hash shared with the CPU generator (splitmix64 finaliser).
__device__ __forceinline__ uint64_t mix64(uint64_t z)
{
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__device__ __forceinline__ double uniform01(uint64_t key, uint64_t idx)
{
    const uint64_t r = mix64(key ^ mix64(idx));
    return ((double)(r >> 11) + 0.5) * (1.0 / 9007199254740992.0);
}

__global__ void synth_illum_kernel(double* __restrict__ illum, int64_t pairs, uint64_t key,
                                   double mu, double sigma, int independent_faces)
{
    const double two_pi = 6.283185307179586476925286766559;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < pairs;
         i += (int64_t)gridDim.x * blockDim.x) {
        double v[4];
        if (independent_faces) {
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                const uint64_t idx = (uint64_t)i * 4 + f;
                const double u1 = uniform01(key, 2 * idx), u2 = uniform01(key, 2 * idx + 1);
                v[f] = exp(mu + sigma * (sqrt(-2.0 * log(u1)) * cos(two_pi * u2)));
            }
        } else {
            const uint64_t idx = (uint64_t)i;
            const double u1 = uniform01(key, 2 * idx), u2 = uniform01(key, 2 * idx + 1);
            v[0] = v[1] = v[2] = v[3] = exp(mu + sigma * (sqrt(-2.0 * log(u1)) * cos(two_pi * u2)));
        }
        double2* p = reinterpret_cast<double2*>(illum + i * 4);
        p[0] = make_double2(v[0], v[1]);
        p[1] = make_double2(v[2], v[3]);
    }
}

uint64_t host_mix64(uint64_t z)
{
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

dim3 weights_grid(int M, int loc)
{
    const int gy = (M + WE_J - 1) / WE_J;
    return dim3((unsigned)((loc + WE_K - 1) / WE_K), (unsigned)(gy < 65535 ? gy : 65535));
}

int grid_stride_blocks(rts_ctx* ctx, int64_t n, int threads)
{
    int64_t b = (n + threads - 1) / threads;
    const int64_t cap = (int64_t)ctx->num_sms * 16;
    if (b > cap) b = cap;
    return (int)(b < 1 ? 1 : b);
}

}  // namespace

int rts_launch_scatter_fp64(rts_ctx* ctx, int64_t k_begin, int64_t k_end, cudaStream_t st,
                            const double* B, double lambda, bool update, bool residual)
{
    return rts_launch_scatter_fp64_cells(ctx, 0, ctx->N, k_begin, k_end, st, B, lambda, update, residual);
}

int rts_launch_scatter_fp64_cells(rts_ctx* ctx, int64_t c_begin, int64_t c_end, int64_t k_begin, int64_t k_end,
                                  cudaStream_t st, const double* B, double lambda, bool update, bool residual)
{
    if (k_end <= k_begin || c_end <= c_begin) return RTS_OK;
    bool taken = false;
    const int rc = rts_sliced_scatter(ctx, c_begin, c_end, k_begin, k_end, st, B, lambda, update, residual, &taken);
    if (rc != RTS_OK || taken) return rc;
    const int64_t n = c_end - c_begin, gx = (n + F64_TC - 1) / F64_TC;
    const DirTiles dt = dir_tiles(k_end - k_begin);
    RTS_REQUIRE(ctx, gx < (1ll << 31) && dt.gy < 65536, RTS_ERR_UNSUPPORTED, "FP64 grid too large");
    dim3 grid((unsigned)gx, (unsigned)dt.gy);
    if (small_tiles(gx, dt, ctx->num_sms)) {
        auto* kernel = update ? scatter_fp64_small_kernel<true> : scatter_fp64_small_kernel<false>;
        rts_timing_begin(ctx, st);
        kernel<<<small_grid(n, k_end - k_begin), S64_THREADS, 0, st>>>(
            ctx->d_illum + 4 * c_begin, ctx->d_W, n, ctx->N, (int)ctx->M, (int)ctx->local(), (int)k_begin, (int)k_end,
            ctx->d_S + c_begin, update ? B + c_begin : nullptr, lambda, residual ? ctx->resid_target : nullptr);
        rts_timing_end(ctx, st);
        RTS_CHECK_LAUNCH(ctx, "scatter_fp64_small_kernel");
        ctx->launches++;
        return RTS_OK;
    }
    auto* kernel = update && residual ? scatter_fp64_kernel<true, true>
                   : update           ? scatter_fp64_kernel<true, false>
                                      : scatter_fp64_kernel<false, false>;
    rts_timing_begin(ctx, st);
    kernel<<<grid, F64_THREADS, 0, st>>>(ctx->d_illum + 4 * c_begin, ctx->d_W, n, ctx->N, (int)ctx->M,
                                         (int)ctx->local(), (int)k_begin, (int)k_end, dt.n_full, dt.nb_last,
                                         ctx->d_S + c_begin, update ? B + c_begin : nullptr, lambda,
                                         ctx->resid_target);
    rts_timing_end(ctx, st);
    RTS_CHECK_LAUNCH(ctx, "scatter_fp64_kernel");
    ctx->launches++;
    return RTS_OK;
}

int rts_launch_scatter_list(rts_ctx* ctx, int64_t c0, int64_t n, int64_t k_begin, int64_t k_end, int bn,
                            int64_t mask_ld, const unsigned int* mask, const unsigned int* list,
                            unsigned int* count, cudaStream_t st, const double* B, double lambda, bool update,
                            bool residual)
{
    const ListArgs fx{list, mask, mask_ld, bn, (int)k_begin};
    const dim3 most = small_grid(n, k_end - k_begin);
    const int64_t tiles = (int64_t)most.x * most.y;
    const unsigned grid = (unsigned)(tiles < 2 * ctx->num_sms ? tiles : 2 * ctx->num_sms);
    auto* kernel = update && residual ? scatter_list_kernel<true, true>
                   : update           ? scatter_list_kernel<true, false>
                                      : scatter_list_kernel<false, false>;
    kernel<<<grid, F64_THREADS, 0, st>>>(ctx->d_illum + 4 * c0, ctx->d_W, n, ctx->N, (int)ctx->M, (int)ctx->local(),
                                         (int)k_begin, (int)k_end, dir_tiles(k_end - k_begin), ctx->num_sms,
                                         ctx->d_S + c0, update ? B + c0 : nullptr, lambda, ctx->resid_target, fx, count,
                                         count + 2, ctx->d_fp64, ctx->d_flag + 1);
    RTS_CHECK_LAUNCH(ctx, "scatter_list_kernel");
    ctx->launches++;
    return RTS_OK;
}

int rts_launch_weights(rts_ctx* ctx)
{
    int rc = rts_launch_weights_raw(ctx, ctx->d_xyz, ctx->d_area, (int)ctx->M, (int)ctx->out_start, (int)ctx->local(),
                                    ctx->full_area, ctx->phase, ctx->phase_g, ctx->d_W,
                                    ctx->streams[RTS_STREAM_SCATTERING_1]);
    if (rc != RTS_OK) return rc;
    RTS_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->streams[RTS_STREAM_SCATTERING_1]));
    return RTS_OK;
}

int rts_launch_moments(rts_ctx* ctx, cudaStream_t st)
{
    const int threads = cell_threads(ctx->N, ctx->num_sms);
    const int64_t blocks = (ctx->N + threads - 1) / threads;
    rts_timing_begin(ctx, st);
    (threads == 64 ? moments_kernel<64> : moments_kernel<128>)<<<(unsigned)blocks, threads, 0, st>>>(ctx->d_illum, ctx->d_xyz, ctx->d_area,
                                                             ctx->N, (int)ctx->M, ctx->full_area,
                                                             ctx->d_energy, ctx->d_flux);
    rts_timing_end(ctx, st);
    RTS_CHECK_LAUNCH(ctx, "moments_kernel");
    ctx->launches++;
    return RTS_OK;
}

int rts_launch_illum_params(rts_ctx* ctx, cudaStream_t st)
{
    const int threads = cell_threads(ctx->N, ctx->num_sms);
    const int64_t blocks = (ctx->N + threads - 1) / threads;
    const double* geo = ctx->d_geo;
    const int64_t N = ctx->N;
    rts_timing_begin(ctx, st);
    (threads == 64 ? illum_params_kernel<64> : illum_params_kernel<128>)<<<(unsigned)blocks, threads, 0, st>>>(
        ctx->d_illum, ctx->d_xyz, ctx->d_area, N, (int)ctx->M, ctx->full_area, geo, geo ? geo + 12 * N : nullptr,
        geo ? geo + 16 * N : nullptr, ctx->d_params);
    rts_timing_end(ctx, st);
    RTS_CHECK_LAUNCH(ctx, "illum_params_kernel");
    ctx->launches++;
    return RTS_OK;
}

int rts_launch_update(rts_ctx* ctx, int64_t k_begin, int64_t k_end, cudaStream_t st,
                      const double* B, double lambda, bool residual)
{
    const int64_t rows = k_end - k_begin;
    if (rows <= 0) return RTS_OK;
    const int blocks = grid_stride_blocks(ctx, rows * ctx->N, 256);
    double* S = ctx->d_S + k_begin * ctx->N;
    if (residual)
        update_kernel<true><<<blocks, 256, 0, st>>>(S, B, ctx->N, rows, lambda, ctx->resid_target);
    else
        update_kernel<false><<<blocks, 256, 0, st>>>(S, B, ctx->N, rows, lambda, ctx->resid_target);
    RTS_CHECK_LAUNCH(ctx, "update_kernel");
    ctx->launches++;
    return RTS_OK;
}

int rts_launch_relax_fp64(rts_ctx* ctx, cudaStream_t st)
{
    const int64_t pairs = ctx->M * ctx->N;
    if (pairs <= 0) return RTS_OK;
    relax_fp64_kernel<<<(unsigned)((pairs + 255) / 256), 256, 0, st>>>(ctx->d_illum, ctx->d_S, pairs);
    RTS_CHECK_LAUNCH(ctx, "relax_fp64_kernel");
    ctx->launches++;
    return RTS_OK;
}

int rts_launch_synth(rts_ctx* ctx, uint64_t seed, double mu, double sigma, int independent_faces)
{
    const int64_t pairs = ctx->M * ctx->N;
    const uint64_t key = host_mix64(seed * 0x632BE59BD9B4E019ull + 1);
    synth_illum_kernel<<<grid_stride_blocks(ctx, pairs, 256), 256, 0,
                         ctx->streams[RTS_STREAM_SCATTERING_1]>>>(ctx->d_illum, pairs, key, mu, sigma,
                                                                  independent_faces);
    RTS_CHECK_LAUNCH(ctx, "synth_illum_kernel");
    ctx->launches++;
    RTS_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->streams[RTS_STREAM_SCATTERING_1]));
    return RTS_OK;
}

// ---------------------------------------------------------------------------
// Allocation-free FP64 scattering integral.
//
// For callers that cannot allocate device memory themselves or through us:
// code running under a caller-owned memory pool or arena that forbids
// allocations outside it, and hosts that account every device byte up
// front.  The caller passes device inputs and outputs; the only scratch --
// the M x M FP64 direction-pair matrix W -- lives in the file-scope array
// below, which every GPU that loads this library holds until the process
// exits.
// ---------------------------------------------------------------------------
namespace {

static __device__ __align__(256) double g_noalloc_w[RTS_NOALLOC_MAX_DIRS * RTS_NOALLOC_MAX_DIRS];

constexpr int NOALLOC_MAX_DEVICES = 64;
double* g_noalloc_w_addr[NOALLOC_MAX_DEVICES] = {};
std::mutex g_noalloc_mutex;

// Device address of the scratch array for `device` (current).  Host code
// cannot use the symbol itself as a pointer, so the address is looked up with
// cudaGetSymbolAddress.  Outside a stream capture it is looked up on every
// call, so a module reloaded after a device reset is seen at its new address;
// the last address found is kept for calls made while `st` is being captured,
// which must therefore follow an uncaptured call on the same device.
double* noalloc_scratch(int device, cudaStream_t st)
{
    if (device < 0 || device >= NOALLOC_MAX_DEVICES) return nullptr;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (cap != cudaStreamCaptureStatusNone) return g_noalloc_w_addr[device];
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_w) != cudaSuccess) {
        cudaGetLastError();  // our own lookup's error; none was pending on entry
        return nullptr;
    }
    g_noalloc_w_addr[device] = static_cast<double*>(p);
    return g_noalloc_w_addr[device];
}

bool aligned(const void* p, uintptr_t bytes) { return (reinterpret_cast<uintptr_t>(p) & (bytes - 1)) == 0; }

}  // namespace

extern "C" int rts_scattering_noalloc(const double* d_illum, const double* d_xyz, const double* d_area,
                                      int64_t N, int64_t M, double full_area, double* d_scattering,
                                      void* stream)
{
    if (!d_illum || !d_xyz || !d_area || !d_scattering) return RTS_ERR_INVALID_ARGUMENT;
    if (N <= 0 || M <= 0 || !(full_area > 0.0)) return RTS_ERR_INVALID_ARGUMENT;
    if (M > RTS_NOALLOC_MAX_DIRS) return RTS_ERR_INVALID_ARGUMENT;  // the scratch holds M <= 512
    // Illum is read as pairs of doubles (16-byte loads); the rest as doubles
    if (!aligned(d_illum, 16) || !aligned(d_xyz, 8) || !aligned(d_area, 8) || !aligned(d_scattering, 8))
        return RTS_ERR_INVALID_ARGUMENT;
    const int64_t gx = (N + F64_TC - 1) / F64_TC;
    if (gx >= (1ll << 31)) return RTS_ERR_INVALID_ARGUMENT;
    // An error left pending by the caller's own earlier work is theirs: report
    // it without launching and without clearing it.
    if (cudaPeekAtLastError() != cudaSuccess) return RTS_ERR_CUDA;
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) {
        cudaGetLastError();
        return RTS_ERR_CUDA;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    double* W = noalloc_scratch(device, st);
    if (!W) return RTS_ERR_CUDA;
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
        cudaGetLastError();
        return RTS_ERR_CUDA;
    }
    // W is rewritten in full (all M x M entries) by every call: nothing in the
    // scratch has to start at zero, and calls that overlap on the GPU race.
    weights_kernel<<<weights_grid((int)M, (int)M), WE_K * WE_J, 0, st>>>(d_xyz, d_area, (int)M, 0, (int)M, full_area,
                                                                         RTS_PHASE_THOMSON, 0.0, W);
    if (cudaGetLastError() != cudaSuccess) return RTS_ERR_CUDA;  // nothing was pending: this launch's error
    const DirTiles dt = dir_tiles(M);
    if (small_tiles(gx, dt, sms)) {
        scatter_fp64_small_kernel<false><<<small_grid(N, M), S64_THREADS, 0, st>>>(
            d_illum, W, N, N, (int)M, (int)M, 0, (int)M, d_scattering, nullptr, 0.0, nullptr);
        return cudaGetLastError() != cudaSuccess ? RTS_ERR_CUDA : RTS_OK;
    }
    dim3 grid((unsigned)gx, (unsigned)dt.gy);
    scatter_fp64_kernel<false, false><<<grid, F64_THREADS, 0, st>>>(d_illum, W, N, N, (int)M, (int)M, 0, (int)M,
                                                                     dt.n_full, dt.nb_last, d_scattering, nullptr,
                                                                     0.0, nullptr);
    if (cudaGetLastError() != cudaSuccess) return RTS_ERR_CUDA;
    return RTS_OK;
}

// W [M][loc] of an arbitrary direction set on `st`.
int rts_launch_weights_raw(rts_ctx* ctx, const double* d_xyz, const double* d_area, int M, int k_off, int loc,
                           double full_area, int phase, double g, double* W, cudaStream_t st)
{
    weights_kernel<<<weights_grid(M, loc), WE_K * WE_J, 0, st>>>(d_xyz, d_area, M, k_off, loc, full_area, phase, g, W);
    RTS_CHECK_LAUNCH(ctx, "weights_kernel");
    ctx->launches++;
    if (phase == RTS_PHASE_THOMSON) return RTS_OK;
    weights_normalise_kernel<<<dim3((unsigned)((loc + 31) / 32), WN_CTAS), WN_THREADS, 0, st>>>(W, M, loc);
    RTS_CHECK_LAUNCH(ctx, "weights_normalise_kernel");
    ctx->launches++;
    return RTS_OK;
}
