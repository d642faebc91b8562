// rts_sliced.cu -- the FP64 scattering integral on the tensor cores: both
// operands as sums of FP16 digits, products accumulated exactly in FP32, the
// sums combined in 64-bit integers (K. Ozaki, T. Ogita, S. Oishi, S. M. Rump,
// "Error-free transformations of matrix multiplication by using fast routines
// of matrix multiplication and its applications", Numerical Algorithms 59,
// 2012; D. Mukunoki et al., "DGEMM using tensor cores, and its accurate and
// reproducible versions", ISC 2020).
//
// Why: GB300's FP64 pipe runs 1.26 TFLOP/s, its FP16 tensor cores 1,900; the
// integral needs 21 digit products per FP64 product, so the tensor cores have
// about 70 times the FP64 pipe's rate for it.
//
//   Ibar_c,j = 2^(e_c - 54) sum_i a_i 2^(9 (5 - i)),   W_j,k likewise with e_k
//   (0 <= digit 0 <= 512, the others at most 256 in magnitude; rts_rows.cuh)
//   S_c,k    = 2^(e_c + e_k - 54) sum_{d = 0..5} 2^(9 (4 - d)) D_d,
//   D_d      = sum_j sum_{i = 0..d} a_i w_{d-i}
// The tensor core forms the D_d of 32 in-directions at a time: at most
// 32 (2 2^17 + 4 2^16) = 2^24, so every FP32 partial sum is an integer that
// FP32 holds exactly.  They are added as integers into one 64-bit total per
// output (D_5 rounded to the total's unit), which the column exponents keep
// below 2^64: sum_j W_jk <= 1022 2^e_k.
//
// Error.  In units of 2^-54 of 2^(e_c + e_k): at most 1.26 a direction from the
// products d >= 6 that are left out (five of 2^-2 at d = 6), half of Ibar / 2^e_c +
// W / 2^e_k a direction from the operands' last digits, 0.75 per 32 directions from
// D_5, and the rounding of S.  In ordinary rows the signs mix: measured against
// 113-bit sums with lognormal intensities, rms 1.0e-16 against 8.6e-16 for the
// FP64 FMA chain of scatter_fp64_kernel at M = 1000, 7.5e-17 against 3.8e-16 at
// M = 200, 7.6e-17 against 2.1e-16 at M = 64.  That is on average: single outputs,
// 7 to 15 % of those, are further off than the chain's, and rows of a few directions
// (where the chain rounds a few times only) can be too, by the bound above.
// An output below half of 2^(e_c + e_k) (a row dominated by a few directions far
// above the rest), where that bound is large against the output, is left to the
// chain, as are rows with negative values, infinities, NaN or exponents out of
// range -- the outputs are marked here and rts_launch_scatter_list computes them
// from the Illum.
//
// Kernel: persistent CTAs (one per SM) on tiles of 128 cells x up to 128
// out-directions.  Warp 0 brings the digits of 32 in-directions of both
// operands (96 KB) into a two-stage ring by TMA, in three parts of two digits;
// warps 1 and 2 issue the MMAs of the even and odd D_d into four TMEM
// accumulators in turn; warps 4..19 read each finished accumulator and add it
// into their 64-bit totals, up to 32 a thread.
//
// Bound: the drain, a conversion and a 64-bit multiply-add per accumulator value.
// A chunk of 32 in-directions takes 7.9k cycles at 162,000 x 1000; in copies of
// the kernel whose drain only releases the accumulators 4.3k (42 MMAs at 103
// cycles, fed from shared memory; 64 with resident operands), without the MMAs
// 6.8k.  With update and residual 162,000 x 1000 takes 9.1 ms, 35 TFLOP/s of FP64
// products (scatter_fp64_kernel 291 ms; 8.2 without them), 30,011 x 302 0.27 (5.27
// ms), 10,368 x 200 0.083 (0.94 ms).
#include <cuda.h>

#include <algorithm>

#include "rts_group.h"
#include "rts_internal.h"
#include "rts_ptx.cuh"
#include "rts_rows.cuh"

using namespace rts_ptx;
using rts_rows::ROW_BAD;
using rts_rows::ROW_ZERO;
using rts_rows::SLICES;

namespace {

constexpr int S_BM = 128;
constexpr int S_BN = 128;
constexpr int S_KC = 32;       // in-directions per chunk
constexpr int S_PARTS = 3;     // two digits (one 128-byte swizzle atom per row) each
constexpr int S_STAGES = 2;
constexpr int S_BOX = S_BM * 128;
constexpr int S_STAGE_BYTES = 2 * S_PARTS * S_BOX;
constexpr int S_ACCS = 4;      // TMEM accumulators of S_BN columns
constexpr int S_DRAIN_WARPS = 16, S_DRAIN_WARP0 = 4;  // whole warpgroups, for the register split
constexpr int S_THREADS = (S_DRAIN_WARP0 + S_DRAIN_WARPS) * 32;
constexpr size_t S_SMEM = (size_t)S_STAGES * S_STAGE_BYTES + 1024 + 256;
static_assert(S_SMEM <= 227 * 1024, "shared memory per CTA");
// Registers: 96 a thread at launch; the issuing warpgroup gives up 64 of them,
// so that the drain warps hold their 32 totals (64 registers) and the values
// in flight (26 bytes spilled outside their loop; at 96 the spills tripled the
// kernel's time).
constexpr int S_REGS = 96, S_REGS_ISSUE = 32, S_REGS_DRAIN = 112;
static_assert(S_DRAIN_WARP0 * S_REGS_ISSUE + S_DRAIN_WARPS * S_REGS_DRAIN <=
                  (S_DRAIN_WARP0 + S_DRAIN_WARPS) * S_REGS,
              "the register split within the launch's registers");
struct SlicedArgs {
    int64_t n;               // cells
    int64_t ld;              // row pitch of S in cells
    int64_t mask_ld;         // words per column group of the mask
    int m_tiles, n_tiles, chunks, cols;
    int k0;                  // first out-direction
    const int* rowexp;       // [n]
    const int* colexp;       // [out-directions]
    unsigned int* mask;      // [n_tiles * 4][mask_ld] outputs left to the FP64 kernel
    rts_rows::RowList rows;
    double* S;               // row 0 = out-direction k0
    const double* B;
    double lambda;
    unsigned long long* resid;
    int* flag;
};

// The total's unit is 2^-UNIT_BITS of 2^(e_c + e_k): that of D_4.
constexpr int UNIT_BITS = 2 * (rts_rows::SLICE_BITS - 45) + 36;
constexpr unsigned long long LIMIT = 1ull << (UNIT_BITS - 1);  // half of 2^(e_c + e_k)

// Adds v = D_d and w = D_{d+1} (d = 0, 2 or 4) of a chunk to the total, T +=
// D_0 2^36 + D_1 2^27 + D_2 2^18 + D_3 2^9 + D_4 + round(D_5 / 512), modulo 2^64
// (the D_d of d >= 1 may be negative).  A value takes a conversion and a 32 x
// 32 + 64 multiply-add, 2.2 cycles a warp on its quarter of the SM.
__device__ __forceinline__ void mad_wide(unsigned long long& T, int x, int scale)
{
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(T) : "r"(x), "r"(scale));
}
__device__ __forceinline__ void add_pair(int d, float v, float w, unsigned long long& T)
{
    if (d == 0) {
        asm("{\n\t.reg .b32 l, h;\n\tmov.b64 {l, h}, %0;\n\tmad.lo.s32 h, %1, 16, h;\n\tmov.b64 %0, {l, h};\n\t}"
            : "+l"(T)
            : "r"(__float2int_rn(v)));
        mad_wide(T, __float2int_rn(w), 1 << 27);
    } else if (d == 2) {
        mad_wide(T, __float2int_rn(v), 1 << 18);
        mad_wide(T, __float2int_rn(w), 1 << 9);
    } else {
        mad_wide(T, __float2int_rn(fmaf(w, 1.0f / 512.0f, v)), 1);
    }
}

// T * 2^e rounded to the nearest double (ties to even), in integer arithmetic
// (a conversion and a multiply would run on the FP64 pipe).  T > 0 and the
// result is in the normal range.
__device__ __forceinline__ double scaled_total(unsigned long long T, int e)
{
    const int lz = __clzll((long long)T);
    const unsigned long long m = T << lz;
    unsigned long long r = m >> 11;
    const unsigned int rem = (unsigned int)m & 0x7FFu;
    r += (rem > 0x400u || (rem == 0x400u && (r & 1ull))) ? 1ull : 0ull;
    // r (bit 52 set, or 2^53 after a carry) adds its leading bit to the exponent field
    return __longlong_as_double((long long)(r + ((unsigned long long)(1023 + 63 - lz + e - 1) << 52)));
}

// 32 lanes x 8 (or 4) columns of two accumulators; the registers hold the
// values after tmem_wait_ld, which names them so that no use moves above it.
__device__ __forceinline__ void tmem_ld8x2(uint32_t ta, uint32_t tb, uint32_t (&r)[16])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%16];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%17];"
                 : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]),
                   "=&r"(r[7]), "=&r"(r[8]), "=&r"(r[9]), "=&r"(r[10]), "=&r"(r[11]), "=&r"(r[12]), "=&r"(r[13]),
                   "=&r"(r[14]), "=&r"(r[15])
                 : "r"(ta), "r"(tb)
                 : "memory");
}
__device__ __forceinline__ void tmem_ld4x2(uint32_t ta, uint32_t tb, uint32_t (&r)[16])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%8];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%4,%5,%6,%7}, [%9];"
                 : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[8]), "=&r"(r[9]), "=&r"(r[10]),
                   "=&r"(r[11])
                 : "r"(ta), "r"(tb)
                 : "memory");
#pragma unroll
    for (int i = 0; i < 4; ++i) r[4 + i] = r[12 + i] = 0;
}
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&r)[16])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                   "+r"(r[15])
                 :
                 : "memory");
}

// kCols: columns per drain warp, a quarter of the tile's width.
template <int kCols, bool kUpdate, bool kResidual>
__global__ void __launch_bounds__(S_THREADS, 1)
sliced_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapW, const SlicedArgs p)
{
    constexpr int kBn = 4 * kCols;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S_STAGES * S_STAGE_BYTES);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 24);
    const uint32_t smem_base = smem_u32(smem), bar_base = smem_u32(bars);
    auto full_bar = [&](uint32_t s, int part) { return bar_base + 8u * (s * S_PARTS + (uint32_t)part); };
    auto empty_bar = [&](uint32_t s) { return bar_base + 8u * (S_STAGES * S_PARTS + s); };
    auto acc_full = [&](uint32_t a) { return bar_base + 8u * (S_STAGES * (S_PARTS + 1) + a); };
    auto acc_empty = [&](uint32_t a) { return bar_base + 8u * (S_STAGES * (S_PARTS + 1) + S_ACCS + a); };

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < S_STAGES; ++s) {
            for (int q = 0; q < S_PARTS; ++q) mbar_init(full_bar(s, q), 1);
            mbar_init(empty_bar(s), 2);  // both issuers
        }
        for (int a = 0; a < S_ACCS; ++a) {
            mbar_init(acc_full(a), 1);
            mbar_init(acc_empty(a), S_DRAIN_WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_proxy_async_smem();
    }
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const bool live = *(volatile int*)p.flag == 0;
    const int64_t tiles = (int64_t)p.m_tiles * p.n_tiles;

    if (warp < S_DRAIN_WARP0) reg_dec<S_REGS_ISSUE>();
    if (warp == 0) {
        // ------------------------------------------------------------ producer
        if (lane == 0 && live) {
            uint32_t it = 0;  // chunks of this CTA so far
            bool ok = true;
            const uint32_t tx = (uint32_t)(S_BOX + kBn * 128);
            for (int64_t t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
                const int m0 = (int)(t / p.n_tiles) * S_BM, n0 = p.k0 + (int)(t % p.n_tiles) * kBn;
                for (int c = 0; c < p.chunks; ++c, ++it) {
                    const uint32_t s = it % S_STAGES;
                    if (it >= (uint32_t)S_STAGES &&
                        !mbar_wait(empty_bar(s), ((it / S_STAGES) - 1) & 1, p.flag, FLAG_WAIT_PRODUCER)) {
                        ok = false;
                        break;
                    }
                    const uint32_t base = smem_base + s * S_STAGE_BYTES;
                    for (int q = 0; q < S_PARTS; ++q) {
                        const int x = (c * S_PARTS + q) * 64;
                        mbar_expect_tx(full_bar(s, q), tx);
                        tma_load_2d(base + q * S_BOX, &mapA, x, m0, full_bar(s, q));
                        tma_load_2d(base + (S_PARTS + q) * S_BOX, &mapW, x, n0, full_bar(s, q));
                    }
                }
            }
            // no copy may still be in flight when the CTA exits
            for (uint32_t i = (it > (uint32_t)S_STAGES ? it - S_STAGES : 0); i < it; ++i)
                for (int q = 0; q < S_PARTS; ++q)
                    mbar_wait(full_bar(i % S_STAGES, q), (i / S_STAGES) & 1, p.flag, FLAG_WAIT_PRODUCER);
            // nor a commit: the issuers' last arrivals on the ring
            for (uint32_t i = (it > (uint32_t)S_STAGES ? it - S_STAGES : 0); ok && i < it; ++i)
                mbar_wait(empty_bar(i % S_STAGES), (i / S_STAGES) & 1, p.flag, FLAG_WAIT_PRODUCER);
        }
    } else if (warp < S_DRAIN_WARP0) {
        // ------------------------------------------------------------ MMA issuers
        const int me = warp - 1;
        if (lane == 0 && me < 2 && live) {
            const uint32_t idesc = idesc_f16(true, S_BM, kBn);
            uint32_t it = 0;
            bool ok = true;
            for (int64_t t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
                for (int c = 0; c < p.chunks && ok; ++c, ++it) {
                    const uint32_t s = it % S_STAGES;
                    // descriptors' low words: digit i's K-step h starts
                    // (i / 2) S_BOX + (i % 2) 64 + 32 h bytes into its operand
                    const uint32_t A = (uint32_t)smem_desc_sw128(smem_base + s * S_STAGE_BYTES);
                    const uint32_t W = A + ((S_PARTS * S_BOX) >> 4);
#pragma unroll 1
                    for (int d = me; d < SLICES; d += 2) {  // D_d needs the digits 0..d: parts 0..d/2
                        const uint32_t g = it * SLICES + (uint32_t)d, slot = g % S_ACCS;
                        if (!mbar_wait(full_bar(s, d >> 1), (it / S_STAGES) & 1, p.flag, FLAG_WAIT_MMA) ||
                            (g >= (uint32_t)S_ACCS &&
                             !mbar_wait(acc_empty(slot), ((g / S_ACCS) - 1) & 1, p.flag, FLAG_WAIT_MMA))) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        const uint32_t acc = tmem + slot * S_BN;
#pragma unroll 1
                        for (int i = 0; i <= d; ++i) {
                            const uint32_t a = A + (uint32_t)((i >> 1) * (S_BOX >> 4) + (i & 1) * 4);
                            const uint32_t w = W + (uint32_t)(((d - i) >> 1) * (S_BOX >> 4) + ((d - i) & 1) * 4);
                            umma_lo<false>(acc, a, w, idesc, i != 0 ? 1u : 0u);
                            umma_lo<false>(acc, a + 2, w + 2, idesc, 1u);
                        }
                        if (d + 2 >= SLICES) umma_commit(empty_bar(s));  // the chunk's last MMAs of this issuer
                        umma_commit(acc_full(slot));
                    }
                }
            }
        }
    } else {
        // ------------------------------------------------------------ drain + epilogue warps
        reg_inc<S_REGS_DRAIN>();
        const int q = warp & 3, cs = (warp - S_DRAIN_WARP0) >> 2;
        const uint32_t lane_off = ((uint32_t)(q * 32) << 16) + (uint32_t)(cs * kCols);
        auto release = [&](uint32_t s0, uint32_t s1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(acc_empty(s0));
                mbar_arrive(acc_empty(s1));
            }
        };
        uint32_t it = 0;
        bool ok = live;
        for (int64_t t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
            unsigned long long T[kCols];
#pragma unroll
            for (int j = 0; j < kCols; ++j) T[j] = 0;
            for (int c = 0; c < p.chunks && ok; ++c, ++it) {
#pragma unroll
                for (int d = 0; d < SLICES; d += 2) {  // D_d and D_{d+1}
                    const uint32_t g = it * SLICES + (uint32_t)d, s0 = g % S_ACCS, s1 = (g + 1) % S_ACCS;
                    bool got = true;
                    if (lane == 0)
                        got = mbar_wait(acc_full(s0), (g / S_ACCS) & 1, p.flag, FLAG_WAIT_EPILOGUE) &&
                              mbar_wait(acc_full(s1), ((g + 1) / S_ACCS) & 1, p.flag, FLAG_WAIT_EPILOGUE);
                    if (!__shfl_sync(0xffffffffu, got ? 1 : 0, 0)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t ta = tmem + s0 * S_BN + lane_off, tb = tmem + s1 * S_BN + lane_off;
                    // 8 columns at a time (4 at the end), the next on their way while these are added
                    uint32_t cur[16], nxt[16];
                    tmem_ld8x2(ta, tb, cur);
                    tmem_wait_ld(cur);
#pragma unroll
                    for (int h = 0; h < kCols; h += 8) {
                        const bool more = h + 8 < kCols, half = h + 12 == kCols;
                        if (more && !half) tmem_ld8x2(ta + (uint32_t)(h + 8), tb + (uint32_t)(h + 8), nxt);
                        if (more && half) tmem_ld4x2(ta + (uint32_t)(h + 8), tb + (uint32_t)(h + 8), nxt);
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            if (h + j < kCols)
                                add_pair(d, __uint_as_float(cur[j]), __uint_as_float(cur[8 + j]), T[h + j]);
                        if (more) {
                            tmem_wait_ld(nxt);
                            if (h + 16 >= kCols) release(s0, s1);  // the last reads of these accumulators
#pragma unroll
                            for (int j = 0; j < 16; ++j) cur[j] = nxt[j];
                        }
                    }
                }
            }
            if (!ok) break;
            const int64_t r = (t / p.n_tiles) * S_BM + q * 32 + lane;
            const int n_tile = (int)(t % p.n_tiles);
            const int kb = n_tile * kBn + cs * kCols;  // first column, relative to k0
            unsigned long long rmax = 0;  // bits of a non-negative double, times two: they order as integers
            if (r < p.n) {
                const int er = p.rowexp[r];
                const double bterm = kUpdate ? (1.0 - p.lambda) * p.B[r] : 0.0;
                unsigned int left = 0;
                double* dst = p.S + (int64_t)kb * p.ld + r;
#pragma unroll
                for (int h = 0; h < kCols; h += 4) {
                    // the previous values of 4 columns at once: their latency is that of one
                    double old[4];
                    if (kResidual) {
#pragma unroll
                        for (int j = 0; j < 4; ++j) old[j] = kb + h + j < p.cols ? dst[(int64_t)(h + j) * p.ld] : 0.0;
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (kb + h + j >= p.cols) continue;
                        const int ec = __ldg(p.colexp + p.k0 + kb + h + j);
                        if (er == ROW_BAD || ec >= ROW_BAD || (er != ROW_ZERO && T[h + j] < LIMIT)) {
                            left |= 1u << (h + j);
                            continue;
                        }
                        // the row exponent is that of the face sum, 4 Ibar
                        double v = er == ROW_ZERO ? 0.0 : scaled_total(T[h + j], er + ec - 2 - UNIT_BITS);
                        if (kUpdate) v = fma(p.lambda, v, bterm);
                        dst[(int64_t)(h + j) * p.ld] = v;
                        if (kResidual) {
                            const unsigned long long ub = (unsigned long long)__double_as_longlong(v - old[j]) << 1;
                            if (ub > rmax && ub <= 0xFFE0000000000000ull) rmax = ub;  // NaN drops out, as in fmax
                        }
                    }
                }
                p.mask[(int64_t)(n_tile * 4 + cs) * p.mask_ld + r] = left;
                if (left && atomicExch(p.rows.flags + r, 1u) == 0u)
                    p.rows.list[atomicAdd(p.rows.count, 1u)] = (unsigned int)r;
            }
            if (kResidual) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const unsigned long long x = __shfl_xor_sync(0xffffffffu, rmax, o);
                    rmax = x > rmax ? x : rmax;
                }
                if (lane == 0 && rmax > 0) atomicMax(p.resid, rmax >> 1);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

using Kernel = void (*)(const CUtensorMap, const CUtensorMap, const SlicedArgs);
template <int kCols>
Kernel kernel_of(bool update, bool residual)
{
    return update && residual ? sliced_kernel<kCols, true, true>
           : update           ? sliced_kernel<kCols, true, false>
                              : sliced_kernel<kCols, false, false>;
}
Kernel kernel_for(int bn, bool update, bool residual)
{
    switch (bn) {
    case 64: return kernel_of<16>(update, residual);
    case 80: return kernel_of<20>(update, residual);
    case 96: return kernel_of<24>(update, residual);
    case 112: return kernel_of<28>(update, residual);
    default: return kernel_of<32>(update, residual);
    }
}

// Digit rows of W^T: out-direction k's column of W [M][ldw] as row k.  A block
// takes 32 out-directions: column maxima and sums of W first (lane =
// out-direction), then tiles of 64 in-directions through shared memory, a warp
// writing 64 directions of a row at a time.
constexpr int WS_THREADS = 256;
__global__ void __launch_bounds__(WS_THREADS)
slice_w_kernel(const double* __restrict__ W, int M, int loc, int ldw, int kpad, uint16_t* __restrict__ Ws,
               int* __restrict__ colexp)
{
    __shared__ double smax[WS_THREADS / 32][32], ssum[WS_THREADS / 32][32];
    __shared__ int sexp[32];
    __shared__ __align__(16) double tile[32][66];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int k = blockIdx.x * 32 + lane;
    double m = 0.0, sum = 0.0;
    bool nan = false;  // or negative
    if (k < loc)
        for (int j = warp; j < M; j += WS_THREADS / 32) {
            const double w = W[(int64_t)j * ldw + k];
            nan |= !(w >= 0.0);
            m = fmax(m, w);
            sum += w;
        }
    if (nan) m = __longlong_as_double(0x7FF0000000000000ll);
    smax[warp][lane] = m;
    ssum[warp][lane] = sum;
    __syncthreads();
    if (warp == 0) {
        for (int w = 1; w < WS_THREADS / 32; ++w) {
            m = fmax(m, smax[w][lane]);
            sum += ssum[w][lane];
        }
        int e = ROW_BAD;
        const int ex = (int)((unsigned long long)__double_as_longlong(m) >> 52);
        if (ex != 0 && ex != 0x7FF && ex > 1022 - 100 && ex < 1022 + 100) {
            e = ex - 1022;  // |W| < 2^e
            while (sum > 1022.0 * exp2((double)e)) ++e;  // and the 64-bit totals stay below 2^64
        }
        sexp[lane] = e;
        if (k < loc) colexp[k] = e;
    }
    __syncthreads();
    for (int j0 = 0; j0 < kpad; j0 += 64) {
        for (int jj = warp; jj < 64; jj += WS_THREADS / 32) {
            const int j = j0 + jj;
            tile[lane][jj] = (k < loc && j < M) ? W[(int64_t)j * ldw + k] : 0.0;
        }
        __syncthreads();
        for (int kk = warp; kk < 32; kk += WS_THREADS / 32) {
            const int kr = blockIdx.x * 32 + kk, j = j0 + 2 * lane;
            if (kr < loc && j < kpad) {
                const double2 x = *reinterpret_cast<const double2*>(&tile[kk][2 * lane]);
                const int e = sexp[kk];
                uint32_t d[SLICES];
                rts_rows::slice_digits(e >= ROW_BAD ? 0 : rts_rows::slice_int(x.x, e),
                                       e >= ROW_BAD ? 0 : rts_rows::slice_int(x.y, e), d);
                uint16_t* row = Ws + (int64_t)kr * SLICES * kpad + rts_rows::ilv_slice(j);
#pragma unroll
                for (int i = 0; i < SLICES; ++i) *reinterpret_cast<uint32_t*>(row + 32 * i) = d[i];
            }
        }
        __syncthreads();
    }
}

int slot_of(const rts_ctx* ctx, cudaStream_t st)
{
    for (int i = 0; i < RTS_STREAM_COUNT; ++i)
        if (ctx->streams[i] == st) return i;
    return -1;
}

int64_t kpad_of(const rts_ctx* ctx) { return (ctx->M + 31) / 32 * 32; }

// The digit rows of W for the current weights, on `st` (built by the first
// call after a change of W, the other streams' calls wait for that build).
int ensure_w(rts_ctx* ctx, cudaStream_t st)
{
    rts_sliced_state& s = ctx->sliced;
    const int64_t M = ctx->M, loc = ctx->local(), kpad = kpad_of(ctx);
    if (!s.w) {
        const size_t wb = (size_t)(loc * SLICES * kpad * 2), eb = (size_t)(loc * 4);
        void *w = nullptr, *e = nullptr;
        int rc = rts_dmalloc(ctx, &w, wb, "FP64 digits of W");
        if (rc == RTS_OK) rc = rts_dmalloc(ctx, &e, eb, "FP64 digit exponents of W");
        if (rc != RTS_OK) {
            rts_dfree(ctx, w, w ? wb : 0);
            return rc;
        }
        s.w = (uint16_t*)w;
        s.colexp = (int*)e;
        s.w_bytes = wb;
        s.e_bytes = eb;
        s.w_version = -1;
    }
    if (!s.ev_w) RTS_CUDA_TRY(ctx, cudaEventCreateWithFlags(&s.ev_w, cudaEventDisableTiming));
    if (s.w_version == ctx->w_version) {
        RTS_CUDA_TRY(ctx, cudaStreamWaitEvent(st, s.ev_w, 0));
        return RTS_OK;
    }
    for (cudaEvent_t ev : s.ev_use)  // contractions on other streams may still read the old rows
        if (ev) RTS_CUDA_TRY(ctx, cudaStreamWaitEvent(st, ev, 0));
    slice_w_kernel<<<(unsigned)((loc + 31) / 32), WS_THREADS, 0, st>>>(ctx->d_W, (int)M, (int)loc, (int)loc, (int)kpad,
                                                                       s.w, s.colexp);
    RTS_CHECK_LAUNCH(ctx, "slice_w_kernel");
    ctx->launches++;
    RTS_CUDA_TRY(ctx, cudaEventRecord(s.ev_w, st));
    s.w_version = ctx->w_version;
    return RTS_OK;
}

// Device bytes of the digit rows of one pass over a range of cells, at most.
constexpr int64_t S_ROWS_BYTES = (int64_t)1 << 31;

}  // namespace

// Whether the context's FP64 integrals take the digits: a weight kernel
// without a sharp peak (Thomson, or Henyey-Greenstein, whose largest weight
// over the column mean is at most M / 16), and enough work.  Depends on the whole grid and the weights only, so that every
// range of cells and out-directions, and every shard of the out-directions,
// takes the same route and outputs covered twice agree bit for bit.  A call
// without room for its scratch, or on a capturing stream, takes the FP64 cores
// all the same, and differs in the last bits.
//
// The limit of the peak.  How many rows have outputs below the accuracy limit
// depends on the Illum: few with Thomson's kernel, up to all of them near M / 16
// where the intensities of a row spread widely (lognormal with sigma 1.5), and
// then the call pays for the digits and the FP64 cores.  ms a step of 20,000
// cells, sigma 1 / 1.5, the FP64 cores alone in brackets: M = 100, g = 0.5 0.14 /
// 0.37 (0.70); 200, 0.6 0.31 / 1.33 (1.87); 400, 0.7 1.18 / 5.98 (6.23); 1000,
// 0.7 - / 20.7 and 0.8 10.4 / 38.1 (37.1).  With every row listed, whatever the
// kernel, the digits add 1 to 3 %.
//
// The size limit.  The digit rows, the contraction and the list pass take about
// 22 us + 0.14 us M at the smallest sizes, whatever the cells; the 32 x 32 tiles
// of scatter_fp64_small_kernel 0.31 us M in one wave of tiles, then by the
// products.  Digits against tiles: 2,000 x 64 31 and 27 us, 1,000 x 100 44 and
// 39, 1,200 x 128 49 and 47; 3,000 x 64 33 and 47, 2,000 x 100 45 and 70; and
// where M is large even for few cells: 300 x 200 55 and 70, 100 x 302 64 and
// 100, 40 x 1,000 156 and 313.
static bool sliced_fits(const rts_ctx* ctx)
{
    if (ctx->cc_major != 10 || !ctx->fp64_digits) return false;
    const int64_t N = ctx->N, M = ctx->M;
    size_t smem = 0;
    if (M < 48 || N >= ((int64_t)1 << 31) || rts_rows::cells_log2((int)kpad_of(ctx), &smem) == 0) return false;
    if (M < 160 && (double)N * (double)M * (double)M < 1.0e7) return false;  // M, not the shard's share of it
    double peak;
    if (ctx->phase == RTS_PHASE_THOMSON)
        peak = 1.5;
    else if (ctx->phase == RTS_PHASE_HG) {
        const double g = ctx->phase_g < 0 ? -ctx->phase_g : ctx->phase_g;
        peak = (1.0 + g) / ((1.0 - g) * (1.0 - g));
    } else
        return false;
    double amax = 0.0, asum = 0.0;
    for (double a : ctx->h_area) {
        if (!(a >= 0.0)) return false;
        amax = std::max(amax, a);
        asum += a;
    }
    return amax > 0.0 && peak * amax * (double)M * 16.0 <= asum * (double)M;
}

int rts_sliced_scatter(rts_ctx* ctx, int64_t c_begin, int64_t c_end, int64_t k_begin, int64_t k_end, cudaStream_t st,
                       const double* B, double lambda, bool update, bool residual, bool* taken)
{
    *taken = false;
    if (!sliced_fits(ctx)) return RTS_OK;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return RTS_OK;  // a captured call allocates nothing
    }
    const rts_spare spare(ctx);
    const std::string keep = ctx->last_error;
    auto no_room = [&](int rc) {
        if (rc != RTS_ERR_OVER_BUDGET && rc != RTS_ERR_OUT_OF_MEMORY) return rc;
        ctx->last_error = keep;  // not an error: the FP64 kernel needs no scratch
        return (int)RTS_OK;
    };
    const int64_t M = ctx->M, N = ctx->N, kpad = kpad_of(ctx), cols = k_end - k_begin;
    int rc = ensure_w(ctx, st);
    if (rc != RTS_OK) return no_room(rc);
    const int n_tiles = (int)((cols + S_BN - 1) / S_BN);
    // tile width: the out-directions balanced over the tiles, in steps of 16 and at least 64
    const int bn = (int)std::max<int64_t>(64, ((cols + n_tiles - 1) / n_tiles + 15) / 16 * 16);
    // cells per pass: whole 128-cell tiles within the scratch limit, and half as many as long as there is no room for
    // them and they make a tile for every SM (the passes change no output)
    const int64_t row_bytes = SLICES * kpad * 2, wave = (ctx->num_sms + n_tiles - 1) / n_tiles * S_BM;
    int64_t per = std::max<int64_t>(1, S_ROWS_BYTES / (S_BM * row_bytes)) * S_BM, step;
    size_t a_bytes, m_bytes, bytes;
    void* scratch = nullptr;
    for (;; per = step / 2) {
        const int64_t passes = (c_end - c_begin + per - 1) / per;
        step = ((c_end - c_begin + passes - 1) / passes + S_BM - 1) / S_BM * S_BM;
        a_bytes = (size_t)(step * row_bytes), m_bytes = (size_t)(n_tiles * 4 * step * 4);
        bytes = a_bytes + m_bytes + (size_t)(step * 12 + 16);  // and the row list
        rc = rts_pmalloc(ctx, &scratch, bytes, "FP64 digit rows", st);
        if (rc == RTS_OK) break;
        if ((rc != RTS_ERR_OVER_BUDGET && rc != RTS_ERR_OUT_OF_MEMORY) || step / 2 < wave) return no_room(rc);
    }
    ctx->last_error = keep;
    uint16_t* A = (uint16_t*)scratch;
    unsigned int* mask = (unsigned int*)((char*)scratch + a_bytes);
    int* exps = (int*)((char*)scratch + a_bytes + m_bytes);
    rts_rows::RowList rows{exps, (unsigned int*)exps + step, (unsigned int*)exps + 2 * step,
                           (unsigned int*)exps + 3 * step};
    auto run = [&]() -> int {
        alignas(64) CUtensorMap mapA, mapW;
        int rc2 = rts_group_make_map(ctx, &mapW, ctx->sliced.w, ctx->local(), SLICES * kpad, bn);
        if (rc2 != RTS_OK) return rc2;
        auto* kernel = kernel_for(bn, update, residual);
        RTS_CUDA_TRY(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S_SMEM));
        for (int64_t c0 = c_begin; c0 < c_end; c0 += step) {
            const int64_t n = std::min(step, c_end - c0);
            const double* illum = ctx->d_illum + 4 * c0;
            RTS_CUDA_TRY(ctx, cudaMemsetAsync(rows.count, 0, 16, st));
            if (ctx->fp64_digits == 2) RTS_CUDA_TRY(ctx, cudaMemsetAsync(rows.count + 1, 1, 4, st));
            if ((rc2 = rts_pp_slice_rows(ctx, illum, n, N, (int)M, (int)kpad, A, rows.exps, rows.flags, rows.list,
                                         rows.count, st)) != RTS_OK)
                return rc2;
            if ((rc2 = rts_group_make_map(ctx, &mapA, A, n, SLICES * kpad, S_BM)) != RTS_OK) return rc2;
            SlicedArgs p;
            p.n = n;
            p.ld = N;
            p.mask_ld = step;
            p.m_tiles = (int)((n + S_BM - 1) / S_BM);
            p.n_tiles = n_tiles;
            p.chunks = (int)(kpad / S_KC);
            p.cols = (int)cols;
            p.k0 = (int)k_begin;
            p.rowexp = rows.exps;
            p.colexp = ctx->sliced.colexp;
            p.mask = mask;
            p.rows = rows;
            p.S = ctx->d_S + k_begin * N + c0;
            p.B = update ? B + c0 : nullptr;
            p.lambda = lambda;
            p.resid = ctx->resid_target;
            p.flag = (int*)rows.count + 1;  // of this pass: a wait that gives up leaves it all to the list kernel
            const int64_t grid = std::min<int64_t>(ctx->num_sms, (int64_t)p.m_tiles * n_tiles);
            rts_timing_begin(ctx, st);
            kernel<<<(unsigned)grid, S_THREADS, S_SMEM, st>>>(mapA, mapW, p);
            RTS_CHECK_LAUNCH(ctx, "sliced_kernel");
            ctx->launches++;
            ctx->fp64_passes++;
            rc2 = rts_launch_scatter_list(ctx, c0, n, k_begin, k_end, bn, step, mask, rows.list, rows.count, st, B, lambda,
                                          update, residual);
            rts_timing_end(ctx, st);  // the rows it left are part of the integral's time
            if (rc2 != RTS_OK) return rc2;
        }
        const int slot = slot_of(ctx, st);
        if (slot >= 0) {
            cudaEvent_t& ev = ctx->sliced.ev_use[slot];
            if (!ev) RTS_CUDA_TRY(ctx, cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
            RTS_CUDA_TRY(ctx, cudaEventRecord(ev, st));
        }
        return RTS_OK;
    };
    rc = run();
    rts_pfree(ctx, scratch, bytes, st);
    *taken = rc == RTS_OK;
    return rc;
}

void rts_sliced_free(rts_ctx* ctx)
{
    rts_sliced_state& s = ctx->sliced;
    rts_dfree(ctx, s.w, s.w_bytes);
    rts_dfree(ctx, s.colexp, s.e_bytes);
    if (s.ev_w) cudaEventDestroy(s.ev_w);
    for (cudaEvent_t ev : s.ev_use)
        if (ev) cudaEventDestroy(ev);
    s = rts_sliced_state();
}
