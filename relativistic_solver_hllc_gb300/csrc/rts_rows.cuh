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
// 1.50 ms (3.9 TB/s), against 4.28 ms for a pass for the scales and a pass for
// the rows that did their arithmetic on the FP64 pipe.
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

struct Args {
    const double* illum;  // cell 0 of the range; a direction's row holds ld cells
    int64_t N, ld;        // cells of the range
    int M, kpad, pitch, lg;
    const double* B;      // [N] source (or null): joins the row's maximum
    float* rs;            // [2*npad] row scales and their inverses (or null)
    int64_t npad;
    uint16_t* A;          // rows
};

// kMode: 0 BF16, 1 FP16 (scaled), 2 TF32.
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
        // NaN is skipped, as fmax does; non-negative doubles order as their bits
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
                const unsigned long long ub = (unsigned long long)__double_as_longlong(I) & 0x7FFFFFFFFFFFFFFFull;
                if (ub <= 0x7FF0000000000000ull && ub > mx) mx = ub;
            }
        }
        for (int o = 16; o >= cells; o >>= 1) {
            const unsigned long long v = __shfl_xor_sync(0xffffffffu, mx, o);
            mx = v > mx ? v : mx;
        }
        if ((t & 31) < cells) atomicMax(&cmax[cell], mx);
    }
    __syncthreads();
    if (t < cells) {
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
