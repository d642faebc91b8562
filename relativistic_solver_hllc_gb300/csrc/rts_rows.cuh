// rts_rows.cuh -- operand rows from the reference's face-layout Illum in one
// pass: every (cell, direction) is read once (32 bytes), its FP64 face sum
// kept in shared memory until the cell's largest sum -- and with it the row's
// scale -- is known, and the row written (4 bytes per direction as split
// FP16 / BF16, 8 as split TF32).
//
// Bound: HBM, 36 bytes per cell-direction for the 16-bit splits.  The FP64
// pipe does only the 3 adds of each face sum (2 per SM per cycle: 0.6 of the
// HBM time); the maximum and the scaled conversion run on the integer pipe.
// A block owns 8 cells (256 contiguous bytes of each direction) and all
// directions; at 1000 directions its sums take 66 KB, so three blocks share an
// SM and one's loads run under another's conversion.  162,000 x 1000 in FP16:
// 1.30 ms (4.5 TB/s), against 4.28 ms for a pass for the scales and a pass for
// the rows that did their arithmetic on the FP64 pipe; 82,944 x 400: 0.27 ms
// (0.33 with the sign masked off a sum's bits, which the compiler makes an FP64
// absolute value: a fourth of the pipe's work).
#pragma once

#include <cstdint>

#include "rts_internal.h"
#include "rts_ptx.cuh"

namespace rts_rows {

constexpr int THREADS = 256;

// 2^(13 - ilogb(m)), within FP32's normal range (rows or columns whose
// largest value is below 2^-113 or above 2^139 keep the nearest scale).
__device__ __forceinline__ float pow2_scale(double m)
{
    if (!(m > 0.0) || !isfinite(m)) return 1.0f;
    return ldexpf(1.0f, max(-126, min(127, 13 - ilogb(m))));
}

// x * 2^k rounded to the nearest FP32 (ties to even), from the bit pattern
// on the integer pipe: GB300's FP64 pipe issues about two instructions per SM
// per cycle against 128 for FP32 / integer, and would bound a pass that
// scaled and converted every value there.  Where x * 2^k is in FP32's normal
// range the 52-bit mantissa keeps its top 23 bits, rounded on the 29 below
// (a carry into the exponent is the correctly rounded result, up to
// infinity); zeros, FP64 subnormals, FP32 subnormal or overflowing results
// and NaN take ldexp and the hardware conversion.  Either way one rounding
// of the exact product.
__device__ __forceinline__ float pow2_scaled_to_f32(double x, int k)
{
    const unsigned long long u = (unsigned long long)__double_as_longlong(x);
    const int e = (int)((u >> 52) & 0x7FF);
    const int ef = e + k - 1023 + 127;  // biased FP32 exponent of x * 2^k
    if (e == 0 || e == 0x7FF || ef < 1 || ef > 254) return __double2float_rn(ldexp(x, k));
    const unsigned long long m = u & 0xFFFFFFFFFFFFFull;
    unsigned int f = ((unsigned int)ef << 23) | (unsigned int)(m >> 29);
    const unsigned int rem = (unsigned int)m & 0x1FFFFFFFu;
    if (rem > 0x10000000u || (rem == 0x10000000u && (f & 1u))) ++f;
    return __uint_as_float(f | ((unsigned int)(u >> 32) & 0x80000000u));
}

// log2 of a power-of-two FP32 scale (normal)
__device__ __forceinline__ int scale_log2(float s) { return (int)((__float_as_uint(s) >> 23) & 0xFF) - 127; }

// Shared-memory row pitch (doubles) of a block's sums: 32 bytes past a
// multiple of 256, so that the 8 cells x 4 directions of a warp's stores and
// the 64 directions of a warp's loads fall into distinct banks.
inline int pitch_of(int kpad) { return kpad + 4; }

// Cells per block for a row length: 8 where three blocks fit an SM, else 4
// (one 128-byte line per direction) or 2; 0 when not even 2 rows fit.
inline int cells_log2(int kpad, size_t* smem)
{
    for (int lg = 3; lg >= 1; --lg) {
        *smem = ((size_t)pitch_of(kpad) << lg) * sizeof(double);
        if (*smem <= (lg == 3 ? 74u * 1024 : 226u * 1024)) return lg;
    }
    return 0;
}

// ---- FP64 rows as sums of FP16 digits (mode 3, rts_sliced.cu) ----
//
// x = m * 2^(e - 54), 0 <= m <= 2^54 an integer, is held as six digits,
//   m = sum_i d_i 2^(9 (5 - i)),  d_0 in [0, 512], d_1..d_5 in [-256, 255],
// each exact in FP16.  Adding 256 to every digit but the first makes them plain
// bit fields, and 0x6400 + n is the FP16 number 1024 + n, so a digit costs a
// shift, a mask and half of a packed subtraction.
constexpr int SLICES = 6;
constexpr int SLICE_BITS = 54;                 // x < 2^e is rounded to a multiple of 2^(e - 54)
constexpr int ROW_BAD = 1 << 20;               // row exponents: a value negative or not finite, or e out of range
constexpr int ROW_ZERO = (1 << 20) + 1;        // every value of the row is zero
constexpr int ROW_EXP_MAX = 900;               // |e| of a row that takes the digits

// m of x >= 0 at the row exponent e (x < 2^e), rounded half up.
__device__ __forceinline__ unsigned long long slice_int(double x, int e)
{
    const unsigned long long u = (unsigned long long)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFull;
    const int ex = (int)(u >> 52);
    const unsigned long long f = u & 0xFFFFFFFFFFFFFull;
    const unsigned long long t = (ex ? (f | 0x10000000000000ull) : f) << 1;
    const int sh = min(1022 + e - (ex ? ex : 1), 63);  // x / 2^(e - 54) = t / 2^sh, sh >= 0
    return (t + ((1ull << sh) >> 1)) >> sh;
}

// The six digits of two values, packed as FP16 pairs (first in the low half).
__device__ __forceinline__ void slice_digits(unsigned long long m0, unsigned long long m1, uint32_t (&d)[SLICES])
{
    // 256 for the digits 1..5
    constexpr unsigned long long OFF = (1ull << 8) + (1ull << 17) + (1ull << 26) + (1ull << 35) + (1ull << 44);
    const unsigned long long a = m0 + OFF, b = m1 + OFF;
    const uint32_t al = (uint32_t)a, ah = (uint32_t)(a >> 32), bl = (uint32_t)b, bh = (uint32_t)(b >> 32);
    auto field = [](uint32_t x, uint32_t y, uint32_t sub) {
        const uint32_t w = (x | (y << 16)) + 0x64006400u;
        const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&w), *reinterpret_cast<const __half2*>(&sub));
        return *reinterpret_cast<const uint32_t*>(&h);
    };
    constexpr uint32_t S0 = 0x64006400u, S256 = 0x65006500u;  // FP16 1024 and 1280 = 1024 + 256, twice
    d[5] = field(al & 511u, bl & 511u, S256);
    d[4] = field((al >> 9) & 511u, (bl >> 9) & 511u, S256);
    d[3] = field((al >> 18) & 511u, (bl >> 18) & 511u, S256);
    d[2] = field(__funnelshift_r(al, ah, 27) & 511u, __funnelshift_r(bl, bh, 27) & 511u, S256);
    d[1] = field((ah >> 4) & 511u, (bh >> 4) & 511u, S256);
    d[0] = field(ah >> 13, bh >> 13, S0);
}

// offset (in halves) of digit 0 of in-direction j in a sliced row: per 32
// in-directions, the 32 values of each digit in turn (6 x 64 bytes)
__host__ __device__ __forceinline__ int64_t ilv_slice(int64_t j) { return (j >> 5) * (32 * SLICES) + (j & 31); }

// Rows that the digits cannot carry are collected for the FP64 kernel.
struct RowList {
    int* exps;            // [N] row exponents, ROW_BAD or ROW_ZERO
    unsigned int* flags;  // [N] the row is on the list
    unsigned int* list;   // [N]
    unsigned int* count;
};

struct Args {
    const double* illum;  // cell 0 of the range; a direction's row holds ld cells
    int64_t N, ld;        // cells of the range
    int M, kpad, pitch, lg;
    const double* B;      // [N] source (or null): joins the row's maximum
    float* rs;            // [2*npad] row scales and their inverses (or null)
    int64_t npad;
    uint16_t* A;          // rows
    RowList rows;         // kMode 3
};

// kMode: 0 BF16, 1 FP16 (scaled), 2 TF32, 3 FP64 as six FP16 digits (12 bytes
// per cell-direction written).
template <int kMode>
__global__ void __launch_bounds__(THREADS, 3) rows_from_faces_kernel(const Args a)
{
    extern __shared__ double sums[];  // [1 << lg][pitch]
    __shared__ unsigned long long cmax[8];
    __shared__ int klog[8];           // power of two that turns a sum into the scaled mean
    const int lg = a.lg, cells = 1 << lg;
    const int t = threadIdx.x, cell = t & (cells - 1);
    const int64_t c0 = (int64_t)blockIdx.x << lg;
    const int64_t c = c0 + cell;
    if (t < 8) cmax[t] = 0;
    __syncthreads();
    {
        const int jstep = THREADS >> lg;
        const bool in = c < a.N;
        double* row = sums + cell * a.pitch;
        const double* src = a.illum + 4 * c;
        const int64_t dir = 4 * a.ld;
        // NaN is skipped, as fmax does (kMode 3 keeps it and negative values:
        // larger than any other); non-negative doubles order as their bits
        unsigned long long mx = 0;
        constexpr int U = 4;
        for (int j0 = t >> lg; j0 < a.kpad; j0 += U * jstep) {
            double2 p[U], q[U];
#pragma unroll
            for (int i = 0; i < U; ++i) {
                const int j = j0 + i * jstep;
                if (in && j < a.M) {
                    const double2* f = reinterpret_cast<const double2*>(src + j * dir);
                    p[i] = __ldg(f);
                    q[i] = __ldg(f + 1);
                } else {
                    p[i] = q[i] = make_double2(0.0, 0.0);
                }
            }
#pragma unroll
            for (int i = 0; i < U; ++i) {
                const int j = j0 + i * jstep;
                if (j >= a.kpad) break;
                double I = p[i].x;  // faces 0..3 in order (GET_FACE_TO_CELL)
                I += p[i].y;
                I += q[i].x;
                I += q[i].y;
                row[j] = I;
                unsigned long long ub = (unsigned long long)__double_as_longlong(I);
                if (kMode == 3) {
                    if (ub == 0x8000000000000000ull) ub = 0;  // -0; negative values lie above every other pattern
                } else {
                    ub <<= 1;  // |I| times two as an integer (a mask would become an FP64 absolute value)
                }
                if ((kMode == 3 || ub <= 0xFFE0000000000000ull) && ub > mx) mx = ub;
            }
        }
        for (int o = 16; o >= cells; o >>= 1) {
            const unsigned long long v = __shfl_xor_sync(0xffffffffu, mx, o);
            mx = v > mx ? v : mx;
        }
        if ((t & 31) < cells) atomicMax(&cmax[cell], kMode == 3 ? mx : mx >> 1);
    }
    __syncthreads();
    if (kMode == 3 && t < cells) {
        // the exponent of the largest sum: every sum of the row < 2^e
        const unsigned long long mx = cmax[t];
        const int ex = (int)(mx >> 52), e = ex - 1022;
        const bool bad = mx != 0 && (ex == 0 || ex >= 0x7FF || e < -ROW_EXP_MAX || e > ROW_EXP_MAX);
        klog[t] = mx == 0 ? ROW_ZERO : bad ? ROW_BAD : e;
        if (c < a.N) {
            a.rows.exps[c] = klog[t];
            a.rows.flags[c] = bad ? 1u : 0u;
            if (bad) a.rows.list[atomicAdd(a.rows.count, 1u)] = (unsigned int)c;
        }
    }
    if (kMode != 3 && t < cells) {
        // the scale of 2 max(|mean|, |B|): max_j |sum / 4| = max_j |sum| / 4 exactly
        float s = 1.0f;
        if (a.rs && c < a.N) {
            const double m = a.B ? fabs(a.B[c]) : 0.0;
            s = pow2_scale(2.0 * fmax(m, __longlong_as_double((long long)cmax[t]) / 4));
        }
        klog[t] = (kMode == 1 ? scale_log2(s) : 0) - 2;
        if (a.rs && c < a.npad) {
            a.rs[c] = s;
            a.rs[a.npad + c] = 1.0f / s;
        }
    }
    __syncthreads();
    // a warp converts 64 directions of a cell at a time, a lane two of them
    const int lane = t & 31;
    const int groups = (a.kpad + 63) >> 6;
    for (int u = t >> 5; u < groups << lg; u += THREADS / 32) {
        const int uc = u & (cells - 1);
        const int j = ((u >> lg) << 6) + 2 * lane;
        if (c0 + uc >= a.N || j >= a.kpad) continue;
        const double2 x = *reinterpret_cast<const double2*>(sums + uc * a.pitch + j);
        const int k = klog[uc];
        if (kMode == 3) {
            uint32_t d[SLICES];
            const bool none = k >= ROW_BAD;  // zero digits
            slice_digits(none ? 0 : slice_int(x.x, k), none ? 0 : slice_int(x.y, k), d);
            uint16_t* row = a.A + (c0 + uc) * SLICES * (int64_t)a.kpad + ilv_slice(j);
#pragma unroll
            for (int i = 0; i < SLICES; ++i) *reinterpret_cast<uint32_t*>(row + 32 * i) = d[i];
            continue;
        }
        const float f0 = pow2_scaled_to_f32(x.x, k), f1 = pow2_scaled_to_f32(x.y, k);
        if (kMode == 2) {
            float* row = reinterpret_cast<float*>(a.A + (c0 + uc) * 4 * (int64_t)a.kpad) + rts_ptx::ilv_hi_tf32(j);
            float2 hi, lo;
            rts_ptx::split_tf32(f0, hi.x, lo.x);
            rts_ptx::split_tf32(f1, hi.y, lo.y);
            *reinterpret_cast<float2*>(row) = hi;
            *reinterpret_cast<float2*>(row + 16) = lo;
        } else {
            uint16_t* row = a.A + (c0 + uc) * 2 * (int64_t)a.kpad + rts_ptx::ilv_hi(j);
            uint32_t hi, lo;
            rts_ptx::split2_any(kMode == 1, f0, f1, hi, lo);
            *reinterpret_cast<uint32_t*>(row) = hi;
            *reinterpret_cast<uint32_t*>(row + 32) = lo;
        }
    }
}

}  // namespace rts_rows
