// rts_sweep.cu -- the transport sweep that produces Illum, on the device.
//
// For every direction the reference walks the cells in dependency order
// (Illum_async.cpp:726-784): at each out-face node it takes the mean of the
// in-face the characteristic comes from, integrates GetCurIllum over the
// distance s to it, and stores the three node values of the face for the
// face and its neighbour's copy; ReCalcIllum then writes the face means into
// Illum and measures the change.  Here:
//   - the dependency order is cut into steps (build_graph's steps: cells
//     whose in-faces are all known), computed on the host, and one CTA per
//     direction walks the steps with a barrier between them;
//   - the unit of work within a step is an out-face (always 3 nodes, so the
//     lanes of a warp stay busy; a thread per cell would idle half its lanes
//     on the faces that are in-faces of its cell), and its 3 node distances
//     are the LocX0 records in the order the reference writes them;
//   - the in-face value a node needs is exactly the face mean its upstream
//     cell wrote, so only face means are kept, straight in the device Illum
//     [dir][cell][face] (the reference's node triples are never stored), and
//     ReCalcIllum's norm is taken as each face is written;
//   - the geometry (in-face and distance of every node) is built once per
//     mesh and direction set by a device kernel.
// Reference paths are relative to solver_hllc_illum_cuda/.
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <thread>
#include <vector>

#include "rts_internal.h"

void rts_face_normals_host(int64_t N, const double* vert, double* normals);
void rts_sweep_nodes_host(int64_t N, const double* vert, double* nodes);

namespace {

constexpr double SWEEP_EPS = 1e-10;  // `eps`, global_value.h:13
constexpr int kExpTable = 256;       // entries of the sweep's exponential (exp_fixed)

__host__ __device__ inline void face_verts(int f, int& a, int& b, int& c)
{
    // VTK's tetra faces {0,1,3}, {1,2,3}, {2,0,3}, {0,2,1}
    a = f == 1 ? 1 : f == 2 ? 2 : 0;
    b = f == 0 ? 1 : f == 1 ? 2 : f == 2 ? 0 : 2;
    c = f == 3 ? 1 : 3;
}

// ---------------------------------------------------------------- geometry

// Everything about an in-face that the characteristic test needs and that
// does not depend on the direction or the node, computed once per face:
//   [0..3]   the plane a x + b y + c z + d = 0 through A, B, C with the
//            coefficients IntersectionWithPlane forms
//            (utils/grid_geometry/geometry_solve.cpp:109-128);
//   [4..9]   the plane frame v1, v2 of SetBasis (:8-43) for the cell's
//            outward face normal n;
//   [10..13] B and C in that frame (Make2dPoint, :45-56, relative to A; A
//            itself maps to (0, 0)).
constexpr int kFrame = 16;  // doubles per face (14 used)

__device__ inline void face_frame(const double* A, const double* B, const double* C, const double* n, double* F)
{
    F[0] = A[1] * (B[2] - C[2]) + B[1] * (C[2] - A[2]) + C[1] * (A[2] - B[2]);
    F[1] = A[0] * (C[2] - B[2]) + B[0] * (A[2] - C[2]) + C[0] * (B[2] - A[2]);
    F[2] = A[0] * (B[1] - C[1]) + B[0] * (C[1] - A[1]) + C[0] * (A[1] - B[1]);
    F[3] = A[0] * (C[1] * B[2] - B[1] * C[2]) + B[0] * (A[1] * C[2] - C[1] * A[2]) +
           C[0] * (B[1] * A[2] - A[1] * B[2]);
    double v1[3], v2[3];
    if (fabs(n[1]) < 1e-20) {
        v1[0] = 0, v1[1] = 1, v1[2] = 0;
    } else {
        v1[0] = 1, v1[2] = 0;
        v1[1] = -(n[0] * v1[0] + n[2] * v1[2]) / n[1];
    }
    if (n[1] < 0)
        for (int i = 0; i < 3; ++i) v1[i] = -v1[i];
    v2[0] = -(n[1] * v1[2] - n[2] * v1[1]);
    v2[1] = -(n[2] * v1[0] - n[0] * v1[2]);
    v2[2] = -(n[0] * v1[1] - n[1] * v1[0]);
    const double z1 = sqrt(v1[0] * v1[0] + v1[1] * v1[1] + v1[2] * v1[2]);
    const double z2 = sqrt(v2[0] * v2[0] + v2[1] * v2[1] + v2[2] * v2[2]);
    for (int i = 0; i < 3; ++i) v1[i] /= z1, v2[i] /= z2;
    const double* P[2] = {B, C};
    for (int p = 0; p < 2; ++p) {
        double u = 0, w = 0;
        for (int k = 0; k < 3; ++k) {
            u += (P[p][k] - A[k]) * v1[k];
            w += (P[p][k] - A[k]) * v2[k];
        }
        F[10 + 2 * p] = u, F[11 + 2 * p] = w;
    }
    for (int i = 0; i < 3; ++i) F[4 + i] = v1[i], F[7 + i] = v2[i];
}

__global__ void __launch_bounds__(256) sweep_frames_kernel(const double* __restrict__ vert,
                                                           const double* __restrict__ normals, int64_t N,
                                                           double* __restrict__ frames)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < 4 * N; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t c = i >> 2;
        const int g = (int)(i & 3);
        int ia, ib, ic;
        face_verts(g, ia, ib, ic);
        const double* v = vert + 12 * c;
        face_frame(v + 3 * ia, v + 3 * ib, v + 3 * ic, normals + 3 * i, frames + kFrame * i);
    }
}

// The characteristic from node x back along dir meets the plane of in-face F
// at X (IntersectionWithPlane); InTriangle (geometry_solve.cpp:129-159):
// X strictly inside the triangle, in the face's 2-D frame.
__device__ inline bool hits_face(const double* __restrict__ F, const double* A, const double* x, const double* dir,
                                 double* X)
{
    const double t = -(F[0] * x[0] + F[1] * x[1] + F[2] * x[2] + F[3]) / (F[0] * dir[0] + F[1] * dir[1] + F[2] * dir[2]);
    for (int i = 0; i < 3; ++i) X[i] = dir[i] * t + x[i];
    double u = 0, w = 0;
    for (int k = 0; k < 3; ++k) {
        u += (X[k] - A[k]) * F[4 + k];
        w += (X[k] - A[k]) * F[7 + k];
    }
    const double bu = F[10], bw = F[11], cu = F[12], cw = F[13];
    const double r1 = (0.0 - u) * (bw - 0.0) - (bu - 0.0) * (0.0 - w);
    const double r2 = (bu - u) * (cw - bw) - (cu - bu) * (bw - w);
    const double r3 = (cu - u) * (0.0 - cw) - (0.0 - cu) * (cw - w);
    return (r1 < 0 && r2 < 0 && r3 < 0) || (r1 > 0 && r2 > 0 && r3 > 0);
}

// The word beside an item: the neighbour's copy of its face (its index in a
// direction's Illum, below 2^26), and in the top bits
//   kNoCopy     a boundary face, nothing to copy to;
//   kBoundCell  the cell has a boundary face;
//   kSharedOut  the face is an out-face of the neighbour too (the direction lies
//               in its plane), so another item writes the same two values.
constexpr uint32_t kNoCopy = 0x80000000u, kBoundCell = 0x40000000u, kSharedOut = 0x20000000u;
constexpr uint32_t kCopyIndex = 0x03FFFFFFu;

// pairs: all cells'; states: the direction's in-face flags (null: every face
// counts as shared, which is slower and always right).
__host__ __device__ inline uint32_t copy_word(const int32_t* pairs, const uint8_t* states, uint32_t w)
{
    const int32_t* p = pairs + 4 * (int64_t)(w >> 8);
    const int32_t nb = p[(w >> 6) & 3u];
    uint32_t x = (p[0] | p[1] | p[2] | p[3]) < 0 ? kBoundCell : 0u;
    if (nb < 0) return x | kNoCopy;
    if (!states || !((states[nb >> 2] >> (nb & 3)) & 1)) x |= kSharedOut;
    return x | (uint32_t)nb;
}

struct X0Args {
    const double* vert;      // [N][4][3]
    const double* frames;    // [N][4][kFrame]
    const double* nodes;     // [N][4][3][3]
    const int32_t* pairs;    // [N][4]
    const double* dirs;      // [D][3]
    const uint8_t* states;   // [D][N] in-face flags
    uint32_t* const* items;  // [D]
    double* const* recs;     // [D]
    int32_t* const* steps;   // [D]
    const int32_t* nsteps;   // [D]
    int64_t N;
    int64_t d0;              // first direction of this launch (grid y covers at most 65535)
    uint32_t* const* words;  // [D] the items' copy words (null: none)
    int* flag;               // set when a node finds no in-face
};

// CalculateNodeValue (make_illum_struct/struct_short_characteristics_logic_function.cpp:
// 222-254) for the 3 nodes of every item: the first in-face, in face order,
// whose triangle contains the back-traced point, and the distance to it.
// Grid: x over the items of a direction, y over the directions.
__global__ void __launch_bounds__(256) sweep_x0_kernel(X0Args a)
{
    const int64_t d = a.d0 + blockIdx.y;
    const int64_t n = a.steps[d][a.nsteps[d]];
    uint32_t* items = a.items[d];
    double* recs = a.recs[d];
    const double* dir = a.dirs + 3 * d;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        uint32_t w = items[i];
        const int64_t c = w >> 8;
        const int f = (int)((w >> 6) & 3u);
        const int st = a.states[d * a.N + c];
        const double* v = a.vert + 12 * c;
        for (int m = 0; m < 3; ++m) {
            const double* x = a.nodes + 36 * c + 9 * f + 3 * m;
            int found = -1, first_in = -1;
            double sv = 0.0;
            for (int g = 0; g < 4 && found < 0; ++g) {
                if (!((st >> g) & 1)) continue;
                if (first_in < 0) first_in = g;
                int ia, ib, ic;
                face_verts(g, ia, ib, ic);
                double x0[3];
                if (hits_face(a.frames + kFrame * (4 * c + g), v + 3 * ia, x, dir, x0)) {
                    const double d0 = x[0] - x0[0], d1 = x[1] - x0[1], d2 = x[2] - x0[2];
                    sv = sqrt(d0 * d0 + d1 * d1 + d2 * d2);
                    found = g;
                }
            }
            if (found < 0) {
                atomicOr(a.flag, 1);
                found = first_in < 0 ? 0 : first_in;
            }
            recs[3 * i + m] = sv;
            w |= (uint32_t)found << (2 * m);
        }
        items[i] = w;
        if (a.words) a.words[d][i] = copy_word(a.pairs, a.states + d * a.N, w);
    }
}

// ---------------------------------------------------------------- sweep

struct SweepArgs {
    uint32_t* const* items;  // [D]
    double* const* recs;     // [D]
    double* const* att;      // [D] factors per item (stored or read by the cached forms): e_0, e_1, e_2 and, up to
                             // five CTAs per SM, q
    int32_t* const* steps;   // [D]
    uint32_t* const* bnd;    // [D]
    const int32_t* nsteps;   // [D]
    const int32_t* nbnd;     // [D]
    const int32_t* pairs;    // [N][4]
    const double* nodes;     // [N][4][3][3] (read only with a ball)
    const double* med;       // [N][4] beta, Q, k, 1/k
    const double* S;         // [D][N]
    double* illum;           // [D][N][4], rows of the local directions
    int64_t N;
    uint32_t* const* words;  // [D] the items' copy words (null: formed here)
    rts_medium md;
    double bc[4];
    uint64_t exptab[kExpTable];  // 2^(-j/256) / 3, times 2^65
    double ball[4];          // medium table entry of the ball's coefficients
    unsigned long long* norm;
};

// exp(-x) for x in [1e-3, 700] in 64-bit fixed point.  GB300 retires two FP64
// operations per SM and cycle against 64 or more 32-bit integer ones, so the
// dozen 32 x 32 multiplies and the shifts and adds below cost a fraction of
// Tang's FP64 form (P. T. P. Tang, "Table-driven implementation of the
// exponential function in IEEE floating-point arithmetic", ACM TOMS 15(2),
// 1989), whose reduction they keep: x = (256 k + j) ln2/256 + u with |u| <=
// ln2/512, exp(-x) = 2^-k 2^(-j/256) exp(-u), 2^(-j/256) from a 256-entry table
// and exp(-u) = 1 - u + u^2/2 - u^3/6 + u^4/24 - u^5/120 (the next term is below
// 2^-60), each power with as many bits as its size asks for.  Within 0.65 units
// in the last place of the exact value over the range (0.5 is the rounding's).
//
// `tab` holds 2^(-j/256) times a factor, times 2^65 as integers in [2^62, 2^64);
// the result carries the factor.
constexpr uint64_t kExpC = 0xB8AA3B295C17F0BBull;  // 256 / ln 2 = (kExpC + kExpC2 / 2^32) / 2^55
constexpr uint32_t kExpC2 = 0xBE87FED0u;
constexpr uint64_t kLn2 = 0xB17217F7D1CF79ACull;   // ln 2 * 2^64

__device__ __forceinline__ double exp_fixed(double x, const uint64_t* __restrict__ tab)
{
    const uint64_t bits = (uint64_t)__double_as_longlong(x);
    const int E = (int)(bits >> 52) - 1023;  // -10..9
    const uint64_t m = ((bits & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull) << 11;  // x = m 2^(E - 63)
    // x 256 / ln 2 = (hi + lo / 2^64) 2^(E - 54)
    uint64_t hi = __umul64hi(m, kExpC), lo = m * kExpC;
    const uint64_t corr = (uint64_t)(uint32_t)(m >> 32) * kExpC2;
    lo += corr;
    hi += lo < corr ? 1 : 0;
    const int a = 10 + E;  // 0..19 bits of hi above the fraction
    const uint64_t frac = a ? (hi << a) | (lo >> (64 - a)) : hi;
    const int n = (a ? (int)(hi >> (64 - a)) : 0) + (int)(frac >> 63);  // rounded to nearest
    const int64_t F = (int64_t)frac;                                     // the signed rest, times 2^64
    // u = F / 2^64 * ln2 / 256, times 2^72
    const int64_t A = (int64_t)(__umul64hi((uint64_t)F, kLn2) - (F < 0 ? kLn2 : 0));
    const int ah = (int)(A >> 32);
    const int64_t B = (int64_t)ah * ah + (((int64_t)ah * (int64_t)(uint32_t)A) >> 31);  // u^2 2^80
    const int b32 = (int)(B >> 32);                                                      // u^2 2^48
    const int d3 = __mulhi(__mulhi(ah, b32), 715827882);   // u^3 / 6, times 2^56
    const int q4 = __mulhi(__mulhi(b32, b32), 178956970);  // u^4 / 24, times 2^64
    const int f5 = __mulhi(d3, b32) / 20;                  // u^5 / 120, times 2^72
    const int64_t V = (B >> 9) - A - ((int64_t)d3 << 16) + ((int64_t)q4 << 8) - f5;  // exp(-u) - 1, times 2^72
    const uint64_t G = tab[n & (kExpTable - 1)];
    const int64_t GV = (int64_t)(__umul64hi(G, (uint64_t)V) - (V < 0 ? G : 0));
    const uint64_t R = G + (uint64_t)(GV >> 8);
    const int lz = (int)(R >> 63) ^ 1;  // 2^62 < R < 2^64
    const uint64_t r = ((R << lz) + 0x400ull) >> 11;
    // r 2^(11 - lz) 2^-65 2^-(n / 256); r's leading bit adds to the exponent field
    return __longlong_as_double((int64_t)(r + ((uint64_t)(1023 + 52 + 11 - lz - 65 - (n >> 8) - 1) << 52)));
}

// Per-cell terms of GetCurIllum (solve_module/illum/Illum_async.cpp:259-470):
// scattering form k = alpha + beta, R = Q + S' beta; absorption form
// k = alpha, R = Q; ks = k * s_scale, Rk = R / k.  The medium table keeps beta
// (0 in the absorption form), Q, k and 1 / k per cell, so that neither an item
// nor a node adds or divides for them.
struct CellTerms {
    double k, ks, R, Rk;
};

__device__ inline double cell_source(const rts_medium& md, bool unit_i, double betta, double Q, double S)
{
    return Q + (unit_i ? S : S * md.i_scale) * betta;
}
// the table entry (beta, Q, k, 1/k) of coefficients alpha, beta, Q
__host__ __device__ inline void medium_entry(int mode, double alpha, double betta, double Q, double* e)
{
    const double k = mode == RTS_MEDIUM_ABSORPTION ? alpha : alpha + betta;
    e[0] = mode == RTS_MEDIUM_ABSORPTION ? 0.0 : betta;
    e[1] = Q;
    e[2] = k;
    e[3] = k != 0.0 ? 1.0 / k : 0.0;  // k = 0: those nodes take the reference's expression
}

// The reference's own expressions, for the nodes outside the fast path
// (kept out of line: they are rare and their exponentials cost registers).
__device__ __noinline__ double node_illum_ref(int mode, double k, double ss, double I0, double R)
{
    if (mode == RTS_MEDIUM_ABSORPTION) {
        if (k > 1e-15) return I0 * exp(-k * ss) + R * (1 - exp(-k * ss)) / k;
        return I0 * (1 - k * ss) + R * ss;
    }
    if (k > 1e-10) return (exp(-k * ss) * (I0 * k + (exp(k * ss) - 1) * R)) / k;
    return (1 - ss * k) * (I0 + ss * R);
}

// The fast range 1e-3 <= x <= 700 as bounds on the high word of x (x >= 0,
// and non-negative doubles order as their bit patterns): integer compares,
// off the FP64 pipe.  The bounds are 1e-3 - 8e-10 and 700 + 1e-13.
constexpr int kFastXLo = 0x3F50624D;  // high word of 1e-3
constexpr int kFastXHi = 0x4085E000;  // high word of 700

// GetCurIllum for one node at distance s from the in-face value I_0.  The
// reference evaluates exp(-x) (I0 k + (exp(x) - 1) R) / k, x = k s (the
// scattering form) or I0 exp(-x) + R (1 - exp(-x)) / k (the absorption
// form); where 1e-3 <= x <= 700 both are evaluated as e I0 + (1 - e) R / k
// with e = exp(-x) -- the same number up to a few ulp (the reference and this
// form both lose ~eps / x to the cancellation in exp(x) - 1, resp. 1 - e) for
// one exponential and no division per node, the dominant FP64 cost.  Outside
// that range the reference's own expression runs (including its overflow
// past x = 709).
//
// The node's attenuation factor e depends on the medium and the node's
// distance only, not on I_0 or the source S: node_att gives e / 3 (the face
// mean takes a third of each node), or kAttRef (negative; e never is) where
// the reference's expression has to run.  Within a source iteration the
// medium stays, so the factors can be stored by one sweep and read by the
// next ones.
constexpr double kAttRef = -1.0;

__device__ inline double node_att(double ks, double s, const uint64_t* __restrict__ tab)
{
    const double x = ks * s;
    const int hx = __double2hiint(x);
    return (hx >= kFastXLo && hx <= kFastXHi) ? exp_fixed(x, tab) : kAttRef;
}

// A third of the node value from its factor e3 = e / 3 (s is read only on
// the reference's path; sr: the node's distance record), clamped at 0.
__device__ inline double node_third(const rts_medium& md, bool unit_i, const CellTerms& t, double e3,
                                    const double* sr, double I_0)
{
    const double I0 = unit_i ? I_0 : I_0 * md.i_scale;
    double I;
    if (__double2hiint(e3) >= 0) {
        // (e I0 + (1 - e) R/k) / 3, as R/3k + e/3 (I0 - R/k)
        I = fma(e3, I0 - t.Rk, t.Rk * (1.0 / 3.0));
    } else {
        const double s = *sr;
        I = node_illum_ref(md.mode, t.k, md.s_scale == 1.0 ? s : s * md.s_scale, I0, t.R) * (1.0 / 3.0);
    }
    if (__double2hiint(I) < 0) I = 0.0;  // I < 0 (the sign bit, tested as an integer)
    return unit_i ? I : I / md.i_scale;
}

// ReCalcIllum's max of |old - cur| / cur over the faces (Illum_async.cpp:
// 488-493); NaN terms (0 / 0) drop out as in the reference.  A face whose term
// cannot raise the max is told from the high words alone.  As integers these
// step by 2^-20 of their octave's base 2^e: for cur = m 2^e and high words dh
// < 2^20 apart |old - cur| is below (dh + 1) 2^(e-20), or twice that where old
// lies in the next octave, so the term is below the max while dh + 1 <= max m 2^20; and
// for 0 <= old < cur it is at most 1.  The FP64 operations run only where a lane
// needs them.
struct NormMax {
    double loc = -1.0;
    unsigned int skip = 0;  // floor(loc 2^20), at most 2^21
    __device__ __forceinline__ bool below(double old, double cur) const
    {
        const int ho = __double2hiint(old), hc = __double2hiint(cur);
        const unsigned int lo = (unsigned int)min(ho, hc), dh = (unsigned int)max(ho, hc) - lo;
        const unsigned int m = ((unsigned int)hc & 0xFFFFFu) | 0x100000u;  // m 2^20
        const unsigned int lim = __umulhi(skip << 6, m << 6);              // max m 2^20, rounded down
        const unsigned int d = (ho >> 20) > (hc >> 20) ? 2 * dh + 1 : dh;
        return hc >= 0x00100000 &&
               ((dh < 1u << 20 && d < lim) || ((unsigned int)ho < (unsigned int)hc && skip >= 1u << 20));
    }
    // the terms of a face's own value and of the neighbour's copy
    __device__ __forceinline__ void term(double old, double cur, bool copy, double old_n)
    {
        if (below(old, cur) && (!copy || below(old_n, cur))) return;
#pragma unroll 1
        for (int j = copy ? 0 : 1; j < 2; ++j) {
            const double d = fabs((j ? old : old_n) - cur);
            if (d > loc * cur) {
                const double b = d / cur;
                if (b > loc) {
                    loc = b;
                    skip = b >= 2.0 ? 1u << 21 : (unsigned int)(b * 1048576.0);
                }
            }
        }
    }
};

// L2 eviction priorities of the sweep's loads.  Every direction reads the
// cells' medium entries (beta, Q: 16 B of 32 B per cell, 21 MB at 663,552 cells:
// they fit in L2), while the items, copy words and attenuation factors (4, 4 and
// 32 B per item) are read once per sweep.  Loads of the shared tables are
// marked evict-last and the streams evict-first, so the streams do not push
// the tables out of L2 (cache hints only: the values are the same).
__device__ __forceinline__ uint64_t l2_policy_last()
{
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint64_t l2_policy_first()
{
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ int4 ld_hint(const int4* q, uint64_t pol)
{
    int4 v;
    asm volatile("ld.global.nc.L2::cache_hint.v4.s32 {%0, %1, %2, %3}, [%4], %5;"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(q), "l"(pol));
    return v;
}
__device__ __forceinline__ double2 ld_hint(const double2* q, uint64_t pol)
{
    double2 v;
    asm volatile("ld.global.nc.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;" : "=d"(v.x), "=d"(v.y) : "l"(q), "l"(pol));
    return v;
}
__device__ __forceinline__ uint32_t ld_hint(const uint32_t* q, uint64_t pol)
{
    uint32_t v;
    asm volatile("ld.global.nc.L2::cache_hint.u32 %0, [%1], %2;" : "=r"(v) : "l"(q), "l"(pol));
    return v;
}


// What an item reads that nothing it depends on writes during a sweep (what its
// face and the neighbour's copy hold is changed by the item itself).
struct ItemData {
    uint32_t w, cp; // item and copy word
    double2 bq;     // beta, Q
    double2 ki;     // k, 1 / k (unless q is stored)
    double S;
    double2 fa, fb; // kAtt 2: the factors e_0, e_1, e_2 (thirds) and, where it is stored, q; else the node distances
    double old, old_n;
};

// Position in a direction's items: item idx of step lev, which ends at end.
struct ItemIter {
    int idx, lev, end;
    // a thread takes every T-th item of a step, and goes on to the next step that has one for it
    __device__ __forceinline__ void settle(const int32_t* steps, int ns)
    {
        while (idx >= end && lev + 1 < ns) {
            idx = end + (int)threadIdx.x;
            ++lev;
            end = steps[lev + 1];
        }
    }
    __device__ __forceinline__ bool valid() const { return idx < end; }
};

constexpr int kStepCache = 1024;  // step offsets kept in shared memory

// The face mean node by node, for the items whose nodes may clamp or take the
// reference's expression, and for media with a ball or a scale (out of line:
// rare, or bound by its divisions anyway).  e3: the factors, negative where the
// reference's expression applies.
__device__ __noinline__ double mean_by_nodes(const SweepArgs& a, uint32_t w, bool unit_i, double betta, double Q,
                                             double Sc, const double* sr, double e0, double e1, double e2, double v0,
                                             double v1, double v2, bool in0, bool in1, bool in2)
{
    const bool unit_s = a.md.s_scale == 1.0;
    const double* me = a.med + 4 * (int64_t)(w >> 8);
    const double k = me[2], ik = me[3];
    double mean = 0.0;
    for (int m = 0; m < 3; ++m) {
        const bool in = m == 0 ? in0 : m == 1 ? in1 : in2;
        CellTerms t;
        t.k = in ? a.ball[2] : k;
        t.R = cell_source(a.md, unit_i, in ? a.ball[0] : betta, in ? a.ball[1] : Q, Sc);
        t.ks = unit_s ? t.k : t.k * a.md.s_scale;
        t.Rk = t.R * (in ? a.ball[3] : ik);
        mean += node_third(a.md, unit_i, t, m == 0 ? e0 : m == 1 ? e1 : e2, sr + m, m == 0 ? v0 : m == 1 ? v1 : v2);
    }
    return mean;
}

// One CTA per local direction.  First the boundary in-faces take their
// boundary value (BoundaryConditions: the node triple (I0, I0, I0)); then the
// steps of the dependency order in turn, a thread per out-face of the step:
// its cell's in-face means were written by upstream cells in earlier steps
// (visible after the barrier); it writes its mean to the face and to the
// neighbour's copy.  Every face is written once per sweep, so each writer
// takes ReCalcIllum's term against the old value.
//
// A step is a chain: barrier, in-face means, five dependent FP64 operations,
// store.  Everything else an item needs is known before the step starts, so it
// is loaded one item ahead, across steps (the item words two); seven CTAs per SM
// hide the latency themselves and load an item's data when they come to it.
// What bounds it: latency (half of the stalls wait for the in-face means, a
// third of the issue slots are used), then the FP64 pipe, two operations per SM
// and cycle, of which an item takes five (the norm and the exponential are
// integer work), and with many directions the memory system (their steps' cells
// do not fit L2).  T threads, kCtas of them per SM with their registers.
// Reading the factors, 82,944 cells x 400 directions (192 threads, 3 CTAs per
// SM): 1.77 ms, 4.49 with node-by-node means, 24-byte factors, FP64 norm and
// loads where they are used; storing them 3.0, from 8.22 with FP64 exponentials;
// 6,000 x 48 (256 threads, one CTA per SM): 0.16 from 0.39 and 0.20 from 0.61.
// Seven CTAs per SM wait for memory and keep 24 bytes of factors an item, q
// formed again: 24,576 x 1000 1.43 ms reading and 2.13 storing, from 1.80 and
// 5.21.  663,552 x 1000, where every sweep evaluates (att_mode): 53.2 ms, from
// 133 storing and 53.2 reading.
// kAtt: 0 evaluates every node's attenuation factor, 1 also stores it,
// 2 reads the stored factors (no exponential).  kPlain: i_scale == 1 and no
// ball (the one-step face mean).
template <int kAtt, bool kPlain, int T, int kCtas>
__global__ void __launch_bounds__(T, kCtas) sweep_kernel(const __grid_constant__ SweepArgs a)
{
    const int64_t d = blockIdx.x;
    const int64_t N = a.N;
    const uint32_t* __restrict__ items = a.items[d];
    const double* __restrict__ recs = a.recs[d];
    const int ns = a.nsteps[d];
    const double* __restrict__ Sd = a.S + d * N;
    double* Il = a.illum + d * N * 4;
    const bool unit_i = kPlain || a.md.i_scale == 1.0;
    const bool ball = !kPlain && a.md.radius > 0;
    double2* att = kAtt ? reinterpret_cast<double2*>(a.att[d]) : nullptr;
    __shared__ uint64_t tab[kAtt == 2 ? 1 : kExpTable];
    __shared__ int32_t sstep[kStepCache];
    const int32_t* steps = a.steps[d];
    if (kAtt != 2)
        for (int i = threadIdx.x; i < kExpTable; i += T) tab[i] = a.exptab[i];
    if (ns < kStepCache) {
        for (int i = threadIdx.x; i <= ns; i += T) sstep[i] = steps[i];
        steps = sstep;
    }
    NormMax norm;
    {
        const uint32_t* bnd = a.bnd[d];
        const int nb = a.nbnd[d];
        for (int i = threadIdx.x; i < nb; i += T) {
            const uint32_t id = bnd[i];
            const double I0 = a.bc[-a.pairs[id] - 1];
            const double mean = (I0 + I0 + I0) * (1.0 / 3.0);
            norm.term(Il[id], mean, false, 0.0);
            Il[id] = mean;
        }
    }
    __syncthreads();
    constexpr bool kAhead = kCtas < 7;   // an item's data loaded while the one before is computed
    constexpr bool kWhole = kCtas < 7;   // q stored beside the three factors
    const uint64_t keep = l2_policy_last(), stream = l2_policy_first();
    const uint32_t* __restrict__ words = kAhead && a.words ? a.words[d] : nullptr;
    // cells are below 2^24 and items below 2^26, so 32-bit indexes reach everything
    auto load = [&](uint32_t w, uint32_t cp, uint32_t i, ItemData& x) {
        const uint32_t c = w >> 8;
        x.w = w;
        x.cp = cp;
        x.bq = ld_hint(reinterpret_cast<const double2*>(a.med) + 2 * c, keep);
        x.S = Sd[c];
        x.old = Il[4 * c + ((w >> 6) & 3u)];
        x.old_n = (int)cp >= 0 ? Il[cp & kCopyIndex] : 0.0;
        if (kAtt == 2 && kWhole) {
            x.fa = ld_hint(att + 2 * i, stream);
            x.fb = ld_hint(att + 2 * i + 1, stream);
        } else if (kAtt == 2) {
            const double* f = reinterpret_cast<const double*>(att) + 3 * (size_t)i;
            x.ki = ld_hint(reinterpret_cast<const double2*>(a.med) + 2 * c + 1, keep);
            x.fa.x = f[0], x.fa.y = f[1], x.fb.x = f[2];
        } else {
            x.ki = ld_hint(reinterpret_cast<const double2*>(a.med) + 2 * c + 1, keep);
            x.fa.x = recs[3 * (size_t)i];
            x.fa.y = recs[3 * (size_t)i + 1];
            x.fb.x = recs[3 * (size_t)i + 2];
        }
    };
    ItemIter it;  // the item whose words are fetched next
    it.lev = 0;
    it.idx = ns > 0 ? steps[0] + (int)threadIdx.x : 0;
    it.end = ns > 0 ? steps[1] : 0;
    it.settle(steps, ns);
    // the current item (i, lev; data in cur) and the next one's words
    int i = it.idx, lev = it.lev;
    bool have = it.valid();
    ItemData cur;
    uint32_t w1 = 0, cp1 = 0;
    auto load_words = [&](int idx, uint32_t& w, uint32_t& cp) {
        w = ld_hint(items + idx, stream);
        cp = !kAhead ? 0 : words ? ld_hint(words + idx, stream) : copy_word(a.pairs, nullptr, w);
    };
    if (have) {
        load_words(i, w1, cp1);
        if (kAhead) load(w1, cp1, (uint32_t)i, cur);
        it.idx += T;
        it.settle(steps, ns);
        if (kAhead && it.valid()) load_words(it.idx, w1, cp1);
    }
    for (int L = 0; L < ns; ++L) {
        while (have && lev == L) {
            if (!kAhead) load(w1, copy_word(a.pairs, nullptr, w1), (uint32_t)i, cur);
            const double* row = Il + 4 * (cur.w >> 8);
            double v0 = row[cur.w & 3u], v1 = row[(cur.w >> 2) & 3u], v2 = row[(cur.w >> 4) & 3u];
            // the next item's data and the words of the one after it
            ItemData nxt;
            const bool more = it.valid();
            const int i1 = it.idx, lev1 = it.lev;
            if (more) {
                if (kAhead)
                    load(w1, cp1, (uint32_t)i1, nxt);
                else
                    load_words(i1, w1, cp1);
                it.idx += T;
                it.settle(steps, ns);
                if (kAhead && it.valid()) load_words(it.idx, w1, cp1);
            }
            const double R = cell_source(a.md, unit_i, cur.bq.x, cur.bq.y, cur.S);
            double e0, e1, e2, q;
            bool in0 = false, in1 = false, in2 = false;
            if (ball) {  // class 0: other coefficients inside the ball
                const double* x = a.nodes + 36 * (int64_t)(cur.w >> 8) + 9 * ((cur.w >> 6) & 3u);
                auto inside = [&](const double* y) {
                    const double d0 = y[0] - a.md.ball[0], d1 = y[1] - a.md.ball[1], d2 = y[2] - a.md.ball[2];
                    return sqrt(d0 * d0 + d1 * d1 + d2 * d2) < a.md.radius;
                };
                in0 = inside(x), in1 = inside(x + 3), in2 = inside(x + 6);
            }
            if (kAtt == 2) {
                e0 = cur.fa.x, e1 = cur.fa.y, e2 = cur.fb.x;
                q = kWhole ? cur.fb.y : (1.0 - ((e0 + e1) + e2)) * cur.ki.y;
            } else {
                const double ks = a.md.s_scale == 1.0 ? cur.ki.x : cur.ki.x * a.md.s_scale;
                const double kb = a.md.s_scale == 1.0 ? a.ball[2] : a.ball[2] * a.md.s_scale;
                e0 = node_att(in0 ? kb : ks, cur.fa.x, tab);
                e1 = node_att(in1 ? kb : ks, cur.fa.y, tab);
                e2 = node_att(in2 ? kb : ks, cur.fb.x, tab);
                // the source's weight in the face mean, (1 - sum_m e_m / 3) / k
                q = (1.0 - ((e0 + e1) + e2)) * cur.ki.y;
                if (kAtt == 1 && kWhole) {
                    att[2 * (uint32_t)i] = make_double2(e0, e1);
                    att[2 * (uint32_t)i + 1] = make_double2(e2, q);
                } else if (kAtt == 1) {
                    double* f = reinterpret_cast<double*>(att) + 3 * (size_t)i;
                    f[0] = e0, f[1] = e1, f[2] = e2;
                }
            }
            if (kAhead && (cur.cp & kSharedOut)) {
                // what an earlier step's item may have written
                cur.old = row[(cur.w >> 6) & 3u];
                cur.old_n = Il[cur.cp & kCopyIndex];
            }
            if (cur.cp & kBoundCell) {
                // boundary in-faces give their value itself (CalculateIllumeOnInnerFace,
                // Illum_async.cpp:172-199)
                const int32_t* pr = a.pairs + 4 * (cur.w >> 8);
                auto bound = [&](uint32_t g, double v) {
                    const int nbg = pr[g & 3u];
                    return nbg < 0 ? a.bc[-nbg - 1] : v;
                };
                v0 = bound(cur.w, v0), v1 = bound(cur.w >> 2, v1), v2 = bound(cur.w >> 4, v2);
            }
            // The face mean (I_0 + I_1 + I_2) / 3.  Where no node can clamp
            // (R >= 0, every I0 >= 0 and every factor on the fast form: each node
            // value R/k + e (I0 - R/k) is then >= 0, all sign bits tested at
            // once) it is q R + sum_m e_m/3 I0_m with q = (1 - sum_m e_m/3) / k:
            // 4 operations and one for R, against 3 subtractions, 3 FMAs and 2 for
            // R/k without the stored q, and 11 node by node.
            double mean;
            if (kPlain && (__double2hiint(e0) | __double2hiint(e1) | __double2hiint(e2) | __double2hiint(v0) |
                           __double2hiint(v1) | __double2hiint(v2) | __double2hiint(R)) >= 0)
                mean = fma(e0, v0, fma(e1, v1, fma(e2, v2, q * R)));
            else
                mean = mean_by_nodes(a, cur.w, unit_i, cur.bq.x, cur.bq.y, cur.S, recs + 3 * (size_t)i, e0, e1, e2, v0,
                                     v1, v2, in0, in1, in2);
            // the neighbour's copy usually holds the value this face held (both
            // were written together by the last sweep): the same term again
            const bool copy = (int)cur.cp >= 0;
            norm.term(cur.old, mean, copy && __double_as_longlong(cur.old_n) != __double_as_longlong(cur.old),
                      cur.old_n);
            Il[4 * (cur.w >> 8) + ((cur.w >> 6) & 3u)] = mean;
            if (copy) Il[cur.cp & kCopyIndex] = mean;
            if (kAhead) cur = nxt;
            i = i1;
            lev = lev1;
            have = more;
        }
        __syncthreads();
        // any thread's max serves the warp: fewer terms need the FP64 operations
        norm.skip = __reduce_max_sync(0xffffffffu, norm.skip);
    }
    // max over the block, then over directions (non-negative doubles order
    // as their bit patterns; +1 keeps 0 for "no term")
    double loc = norm.loc;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) loc = fmax(loc, __shfl_xor_sync(0xffffffffu, loc, o));
    __shared__ double red[T / 32];
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = loc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double m = red[0];
        for (int j = 1; j < T / 32; ++j) m = fmax(m, red[j]);
        if (m >= 0) atomicMax(a.norm, (unsigned long long)__double_as_longlong(m) + 1ull);
    }
}

// ---------------------------------------------------------------- host side

// (a b) >> 128
unsigned __int128 mul_hi128(unsigned __int128 a, unsigned __int128 b)
{
    const uint64_t a1 = (uint64_t)(a >> 64), a0 = (uint64_t)a, b1 = (uint64_t)(b >> 64), b0 = (uint64_t)b;
    const unsigned __int128 lo = (unsigned __int128)a0 * b0, m1 = (unsigned __int128)a1 * b0,
                            m2 = (unsigned __int128)a0 * b1;
    const unsigned __int128 mid = (lo >> 64) + (uint64_t)m1 + (uint64_t)m2;
    return (unsigned __int128)a1 * b1 + (m1 >> 64) + (m2 >> 64) + (mid >> 64);
}

// v 2^(-j/256) for j < 256, rounded to 64 bits from a 128-bit first entry v
// (the table of exp_fixed: the factor times 2^129).
void exp2_table(unsigned __int128 v, uint64_t* tab)
{
    // 2^(-1/256) * 2^128
    const unsigned __int128 step = ((unsigned __int128)0xFF4ECB59511EC8A5ull << 64) | 0x301BA217EF18DD7Cull;
    for (int j = 0; j < kExpTable; ++j) {
        tab[j] = (uint64_t)((v + ((unsigned __int128)1 << 63)) >> 64);
        v = mul_hi128(v, step);
    }
}
constexpr unsigned __int128 kExpThird = ((unsigned __int128)0xAAAAAAAAAAAAAAAAull << 64) | 0xAAAAAAAAAAAAAAAAull;  // 1/3
constexpr unsigned __int128 kExpQuarter = (unsigned __int128)1 << 127;                                              // 1/4

// exp_fixed against CUDA's exp at n points spread over [-700, 0] (and the 1e-3
// end): the largest difference in units in the last place of CUDA's value.
__global__ void exp_check_kernel(int64_t n, const uint64_t* __restrict__ tab_in, double* out)
{
    __shared__ uint64_t tab[kExpTable];
    for (int i = threadIdx.x; i < kExpTable; i += blockDim.x) tab[i] = tab_in[i];
    __syncthreads();
    double worst = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double u = (double)i / (double)(n - 1);
        // the whole range from the fast form's lower end, and densely near it
        const double x = i & 1 ? fmin(-700.0 * u, -1e-3) : -1e-3 - u * u;
        const double a = 4.0 * exp_fixed(-x, tab), b = exp(x);
        const double ulp = fabs(__longlong_as_double(__double_as_longlong(b) + 1) - b);
        worst = fmax(worst, fabs(a - b) / ulp);
    }
    for (int o = 16; o > 0; o >>= 1) worst = fmax(worst, __shfl_xor_sync(0xffffffffu, worst, o));
    if ((threadIdx.x & 31) == 0) atomicMax((unsigned long long*)out, (unsigned long long)__double_as_longlong(worst));
}

int popcount4(int x) { return (x & 1) + ((x >> 1) & 1) + ((x >> 2) & 1) + ((x >> 3) & 1); }

// Dependency order of one direction: steps of cells whose in-faces all have
// known values (boundary faces are known from the start), each step in
// ascending cell id -- the order build_graph writes (build_graph/
// build_graph_calculation.cpp:347-391,482-510, driven by build_graph_main.cpp:
// 165-300).  A cell enters the step after the last of its upstream cells.
// lev receives the cell offset of every step and the end.  Returns false on
// a dependency cycle.
bool order_direction(int64_t N, const int32_t* pairs, const uint8_t* states, int32_t* order, std::vector<int32_t>& lev,
                     std::vector<int32_t>& indeg, std::vector<int32_t>& next)
{
    indeg.assign(N, 0);
    for (int64_t c = 0; c < N; ++c)
        for (int f = 0; f < 4; ++f)
            if (((states[c] >> f) & 1) && pairs[4 * c + f] >= 0) indeg[c]++;
    int64_t done = 0;
    lev.clear();
    for (int64_t c = 0; c < N; ++c)
        if (indeg[c] == 0) order[done++] = (int32_t)c;
    int64_t begin = 0;
    while (done > begin) {
        lev.push_back((int32_t)begin);
        const int64_t end = done;
        next.clear();
        for (int64_t i = begin; i < end; ++i) {
            const int64_t c = order[i];
            for (int f = 0; f < 4; ++f) {
                const int32_t nb = pairs[4 * c + f];
                if (nb < 0) continue;
                const int32_t nc = nb >> 2, nf = nb & 3;
                if (((states[nc] >> nf) & 1) && --indeg[nc] == 0) next.push_back(nc);
            }
        }
        std::sort(next.begin(), next.end());
        for (int32_t c : next) order[done++] = c;
        begin = end;
    }
    lev.push_back((int32_t)done);
    return done == N;
}

// Items, step offsets (in items) and boundary in-faces of one direction from
// its cell order, cell steps and face states.
void items_of(int64_t N, const int32_t* pairs, const uint8_t* states, const int32_t* order,
              const std::vector<int32_t>& lev, std::vector<uint32_t>& items, std::vector<int32_t>& steps,
              std::vector<uint32_t>& bnd)
{
    items.clear();
    steps.clear();
    bnd.clear();
    for (size_t L = 0; L + 1 < lev.size(); ++L) {
        steps.push_back((int32_t)items.size());
        for (int32_t p = lev[L]; p < lev[L + 1]; ++p) {
            const uint32_t c = (uint32_t)order[p];
            for (int f = 0; f < 4; ++f)
                if (!((states[c] >> f) & 1)) items.push_back(c << 8 | (uint32_t)f << 6);
        }
    }
    steps.push_back((int32_t)items.size());
    for (int64_t c = 0; c < N; ++c)
        for (int f = 0; f < 4; ++f)
            if (((states[c] >> f) & 1) && pairs[4 * c + f] < 0) bnd.push_back((uint32_t)(4 * c + f));
}

int alloc_tables(rts_ctx* ctx, rts_sweep_state& sw)
{
    const int64_t D = sw.D;
    void* p = nullptr;
    int rc;
    if ((rc = rts_dmalloc(ctx, &p, sizeof(uint32_t*) * D, "sweep item table")) != RTS_OK) return rc;
    sw.d_items = (uint32_t**)p;
    if ((rc = rts_dmalloc(ctx, &p, sizeof(double*) * D, "sweep record table")) != RTS_OK) return rc;
    sw.d_recs = (double**)p;
    if ((rc = rts_dmalloc(ctx, &p, sizeof(double*) * D, "sweep attenuation table")) != RTS_OK) return rc;
    sw.d_att = (double**)p;
    if ((rc = rts_dmalloc(ctx, &p, sizeof(int32_t*) * D, "sweep step table")) != RTS_OK) return rc;
    sw.d_steps = (int32_t**)p;
    if ((rc = rts_dmalloc(ctx, &p, sizeof(uint32_t*) * D, "sweep boundary table")) != RTS_OK) return rc;
    sw.d_bnd = (uint32_t**)p;
    if ((rc = rts_dmalloc(ctx, &p, rts_bytes<int32_t>(D), "sweep step counts")) != RTS_OK) return rc;
    sw.d_nsteps = (int32_t*)p;
    if ((rc = rts_dmalloc(ctx, &p, rts_bytes<int32_t>(D), "sweep boundary counts")) != RTS_OK) return rc;
    sw.d_nbnd = (int32_t*)p;
    sw.h_items.assign(D, nullptr);
    sw.h_words.assign(D, nullptr);
    sw.h_recs.assign(D, nullptr);
    sw.h_att.assign(D, nullptr);
    sw.h_steps.assign(D, nullptr);
    sw.h_bnd.assign(D, nullptr);
    sw.h_nsteps.assign(D, 0);
    sw.h_nbnd.assign(D, 0);
    sw.h_nitems.assign(D, 0);
    sw.have.assign(D, 0);
    return RTS_OK;
}

// the copy words given back, and no more made for these structures
void drop_words(rts_ctx* ctx, rts_sweep_state& sw)
{
    for (auto& b : sw.word_blocks) rts_dfree(ctx, b.first, b.second);
    sw.word_blocks.clear();
    rts_dfree(ctx, sw.d_words, sizeof(uint32_t*) * sw.D);
    sw.d_words = nullptr;
    std::fill(sw.h_words.begin(), sw.h_words.end(), nullptr);
    sw.copy_words = false;
}

void drop_att(rts_ctx* ctx, rts_sweep_state& sw)
{
    rts_dfree(ctx, sw.att_blk, sw.att_bytes);
    sw.att_blk = nullptr;
    sw.att_bytes = 0;
    sw.att_valid = false;
}

void free_blocks(rts_ctx* ctx, rts_sweep_state& sw)
{
    for (auto& b : sw.blocks) rts_dfree(ctx, b.first, b.second);
    sw.blocks.clear();
    drop_words(ctx, sw);
    sw.copy_words = true;
    drop_att(ctx, sw);
    std::fill(sw.h_items.begin(), sw.h_items.end(), nullptr);
    std::fill(sw.h_recs.begin(), sw.h_recs.end(), nullptr);
    std::fill(sw.h_steps.begin(), sw.h_steps.end(), nullptr);
    std::fill(sw.h_bnd.begin(), sw.h_bnd.end(), nullptr);
    std::fill(sw.h_nsteps.begin(), sw.h_nsteps.end(), 0);
    std::fill(sw.h_nbnd.begin(), sw.h_nbnd.end(), 0);
    std::fill(sw.h_nitems.begin(), sw.h_nitems.end(), 0);
    std::fill(sw.have.begin(), sw.have.end(), 0);
    sw.records = sw.max_levels = 0;
}

int alloc_block(rts_ctx* ctx, rts_sweep_state& sw, void** p, size_t bytes, const char* what)
{
    bytes = std::max<size_t>(bytes, 16);
    int rc = rts_dmalloc(ctx, p, bytes, what);
    if (rc == RTS_OK) sw.blocks.push_back({*p, bytes});
    return rc;
}

// Room for the copy words of n items and for their table, after everything that
// the structures need; null without it (no direction has words then).
uint32_t* alloc_words(rts_ctx* ctx, rts_sweep_state& sw, int64_t n)
{
    if (sw.D > 5 * ctx->num_sms) sw.copy_words = false;  // the form for so many directions does not read them
    if (!sw.copy_words) return nullptr;
    const rts_spare spare(ctx);
    const std::string keep = ctx->last_error;
    const size_t bytes = std::max<size_t>(rts_bytes<uint32_t>(n), 16);
    void *table = sw.d_words, *p = nullptr;
    if (!table) rts_dmalloc(ctx, &table, sizeof(uint32_t*) * sw.D, "sweep copy word table");
    sw.d_words = (uint32_t**)table;
    if (table) rts_dmalloc(ctx, &p, bytes, "sweep copy words");
    if (p) {
        sw.word_blocks.push_back({p, bytes});
    } else {
        ctx->last_error = keep;
        drop_words(ctx, sw);
    }
    return (uint32_t*)p;
}

int upload_words(rts_ctx* ctx, rts_sweep_state& sw, cudaStream_t st)
{
    if (!sw.copy_words) return RTS_OK;
    RTS_CUDA_TRY(ctx, cudaMemcpyAsync(sw.d_words, sw.h_words.data(), sizeof(uint32_t*) * sw.D, cudaMemcpyHostToDevice, st));
    RTS_CUDA_TRY(ctx, cudaStreamSynchronize(st));  // pageable source
    return RTS_OK;
}

int upload_tables(rts_ctx* ctx, rts_sweep_state& sw, cudaStream_t st)
{
    const int64_t D = sw.D;
    RTS_CUDA_TRY(ctx, cudaMemcpyAsync(sw.d_items, sw.h_items.data(), sizeof(uint32_t*) * D, cudaMemcpyHostToDevice, st));
    RTS_CUDA_TRY(ctx, cudaMemcpyAsync(sw.d_recs, sw.h_recs.data(), sizeof(double*) * D, cudaMemcpyHostToDevice, st));
    RTS_CUDA_TRY(ctx, cudaMemcpyAsync(sw.d_steps, sw.h_steps.data(), sizeof(int32_t*) * D, cudaMemcpyHostToDevice, st));
    RTS_CUDA_TRY(ctx, cudaMemcpyAsync(sw.d_bnd, sw.h_bnd.data(), sizeof(uint32_t*) * D, cudaMemcpyHostToDevice, st));
    RTS_CUDA_TRY(ctx, cudaMemcpyAsync(sw.d_nsteps, sw.h_nsteps.data(), sizeof(int32_t) * D, cudaMemcpyHostToDevice, st));
    RTS_CUDA_TRY(ctx, cudaMemcpyAsync(sw.d_nbnd, sw.h_nbnd.data(), sizeof(int32_t) * D, cudaMemcpyHostToDevice, st));
    RTS_CUDA_TRY(ctx, cudaStreamSynchronize(st));  // pageable sources
    return RTS_OK;
}

int check_flag(rts_ctx* ctx, const char* what)
{
    int flag = 0;
    RTS_CUDA_TRY(ctx, cudaMemcpy(&flag, ctx->d_flag + 2, sizeof(int), cudaMemcpyDeviceToHost));
    if (flag) {
        cudaMemset(ctx->d_flag + 2, 0, sizeof(int));
        return rts_fail(ctx, RTS_ERR_UNSUPPORTED, "%s: an out-face node found no in-face (a direction parallel to a face)",
                        what);
    }
    return RTS_OK;
}

}  // namespace

bool rts_sweep_give_way(rts_ctx* ctx)
{
    rts_sweep_state* sw = ctx->sweep;
    if (!sw || (!sw->att_blk && !sw->d_words)) return false;
    drop_att(ctx, *sw);
    drop_words(ctx, *sw);
    return true;
}

void rts_sweep_free(rts_ctx* ctx)
{
    rts_sweep_state* sw = ctx->sweep;
    if (!sw) return;
    free_blocks(ctx, *sw);
    const int64_t N = sw->N, D = sw->D;
    rts_dfree(ctx, sw->d_vert, rts_bytes<double>(N * 12));
    rts_dfree(ctx, sw->d_pairs, rts_bytes<int32_t>(N * 4));
    rts_dfree(ctx, sw->d_normals, rts_bytes<double>(N * 12));
    rts_dfree(ctx, sw->d_nodes, rts_bytes<double>(N * 36));
    rts_dfree(ctx, sw->d_med, rts_bytes<double>(N * 4));
    rts_dfree(ctx, sw->d_norm, sizeof(unsigned long long));
    rts_dfree(ctx, sw->d_items, sizeof(uint32_t*) * D);
    rts_dfree(ctx, sw->d_recs, sizeof(double*) * D);
    rts_dfree(ctx, sw->d_att, sizeof(double*) * D);
    rts_dfree(ctx, sw->d_steps, sizeof(int32_t*) * D);
    rts_dfree(ctx, sw->d_bnd, sizeof(uint32_t*) * D);
    rts_dfree(ctx, sw->d_nsteps, rts_bytes<int32_t>(D));
    rts_dfree(ctx, sw->d_nbnd, rts_bytes<int32_t>(D));
    delete sw;
    ctx->sweep = nullptr;
}

extern "C" int rts_sweep_set_mesh(rts_ctx* ctx, const double* vert, const int32_t* pairs, const double* normals)
{
    if (!ctx) return RTS_ERR_INVALID_ARGUMENT;
    RTS_REQUIRE(ctx, ctx->d_illum, RTS_ERR_BAD_STATE, "rts_sweep_set_mesh before rts_init");
    RTS_REQUIRE(ctx, vert && pairs && normals, RTS_ERR_INVALID_ARGUMENT, "rts_sweep_set_mesh: null array");
    const int64_t N = ctx->N;
    RTS_REQUIRE(ctx, N < (int64_t)1 << 24, RTS_ERR_INVALID_ARGUMENT,
                "rts_sweep_set_mesh: %lld cells; the sweep packs cell ids in 24 bits", (long long)N);
    for (int64_t i = 0; i < 4 * N; ++i)
        RTS_REQUIRE(ctx, pairs[i] < 4 * N && pairs[i] >= RTS_BOUND_INNER, RTS_ERR_INVALID_ARGUMENT,
                    "rts_sweep_set_mesh: pairs[%lld] = %d is neither a face nor a boundary code", (long long)i,
                    (int)pairs[i]);
    rts_sweep_free(ctx);
    rts_sweep_state* sw = new rts_sweep_state();
    ctx->sweep = sw;
    sw->N = N;
    sw->D = ctx->local();
    sw->h_vert.assign(vert, vert + 12 * N);
    sw->h_pairs.assign(pairs, pairs + 4 * N);
    sw->h_normals.assign(normals, normals + 12 * N);
    std::vector<double> nodes(36 * N);
    rts_sweep_nodes_host(N, vert, nodes.data());
    void* p = nullptr;
    int rc;
    if ((rc = rts_dmalloc(ctx, &p, rts_bytes<double>(N * 12), "sweep vertices")) != RTS_OK) return rc;
    sw->d_vert = (double*)p;
    if ((rc = rts_dmalloc(ctx, &p, rts_bytes<int32_t>(N * 4), "sweep pairs")) != RTS_OK) return rc;
    sw->d_pairs = (int32_t*)p;
    if ((rc = rts_dmalloc(ctx, &p, rts_bytes<double>(N * 12), "sweep normals")) != RTS_OK) return rc;
    sw->d_normals = (double*)p;
    if ((rc = rts_dmalloc(ctx, &p, rts_bytes<double>(N * 36), "sweep nodes")) != RTS_OK) return rc;
    sw->d_nodes = (double*)p;
    if ((rc = rts_dmalloc(ctx, &p, rts_bytes<double>(N * 4), "sweep medium")) != RTS_OK) return rc;
    sw->d_med = (double*)p;
    if ((rc = rts_dmalloc(ctx, &p, sizeof(unsigned long long), "sweep norm")) != RTS_OK) return rc;
    sw->d_norm = (unsigned long long*)p;
    RTS_CUDA_TRY(ctx, cudaMemcpy(sw->d_vert, vert, rts_bytes<double>(N * 12), cudaMemcpyHostToDevice));
    RTS_CUDA_TRY(ctx, cudaMemcpy(sw->d_pairs, pairs, rts_bytes<int32_t>(N * 4), cudaMemcpyHostToDevice));
    RTS_CUDA_TRY(ctx, cudaMemcpy(sw->d_normals, normals, rts_bytes<double>(N * 12), cudaMemcpyHostToDevice));
    RTS_CUDA_TRY(ctx, cudaMemcpy(sw->d_nodes, nodes.data(), rts_bytes<double>(N * 36), cudaMemcpyHostToDevice));
    RTS_CUDA_TRY(ctx, cudaMemset(sw->d_med, 0, rts_bytes<double>(N * 4)));
    return alloc_tables(ctx, *sw);
}

extern "C" int rts_sweep_build(rts_ctx* ctx, int64_t* records, int64_t* levels)
{
    if (!ctx) return RTS_ERR_INVALID_ARGUMENT;
    RTS_REQUIRE(ctx, ctx->sweep, RTS_ERR_BAD_STATE, "rts_sweep_build before rts_sweep_set_mesh");
    rts_sweep_state& sw = *ctx->sweep;
    const int64_t N = sw.N, D = sw.D;
    free_blocks(ctx, sw);
    // host: face states, dependency order, items of every direction
    std::vector<uint8_t> states((size_t)(D * N));
    std::vector<std::vector<uint32_t>> items((size_t)D), bnd((size_t)D);
    std::vector<std::vector<int32_t>> steps((size_t)D);
    std::vector<char> bad((size_t)D, 0);
    const int nthr = (int)std::max<int64_t>(1, std::min<int64_t>(D, std::max(1u, std::thread::hardware_concurrency())));
    auto work = [&](int w) {
        std::vector<int32_t> order((size_t)N), lev, indeg, next;
        for (int64_t d = w; d < D; d += nthr) {
            const double* dir = ctx->h_xyz.data() + 3 * (ctx->out_start + d);
            uint8_t* st = states.data() + d * N;
            for (int64_t c = 0; c < N; ++c) {
                int s = 0;
                const double* n = sw.h_normals.data() + 12 * c;
                for (int f = 0; f < 4; ++f)
                    if (n[3 * f] * dir[0] + n[3 * f + 1] * dir[1] + n[3 * f + 2] * dir[2] < -SWEEP_EPS) s |= 1 << f;
                st[c] = (uint8_t)s;
            }
            if (!order_direction(N, sw.h_pairs.data(), st, order.data(), lev, indeg, next)) {
                bad[d] = 1;
                continue;
            }
            items_of(N, sw.h_pairs.data(), st, order.data(), lev, items[d], steps[d], bnd[d]);
        }
    };
    std::vector<std::thread> pool;
    for (int w = 1; w < nthr; ++w) pool.emplace_back(work, w);
    work(0);
    for (auto& t : pool) t.join();
    for (int64_t d = 0; d < D; ++d)
        RTS_REQUIRE(ctx, !bad[d], RTS_ERR_UNSUPPORTED, "rts_sweep_build: direction %lld has a dependency cycle",
                    (long long)(ctx->out_start + d));
    // device: one block each of items, node records, steps and boundary faces
    int64_t ni = 0, nl = 0, nbd = 0, maxl = 0;
    for (int64_t d = 0; d < D; ++d) {
        ni += (int64_t)items[d].size();
        nl += (int64_t)steps[d].size();
        nbd += (int64_t)bnd[d].size();
        maxl = std::max<int64_t>(maxl, (int64_t)steps[d].size() - 1);
    }
    void *iblk = nullptr, *rblk = nullptr, *lblk = nullptr, *bblk = nullptr, *sblk = nullptr;
    int rc;
    if ((rc = alloc_block(ctx, sw, &iblk, rts_bytes<uint32_t>(ni), "sweep items")) != RTS_OK) return rc;
    if ((rc = alloc_block(ctx, sw, &rblk, rts_bytes<double>(3 * ni), "sweep node records")) != RTS_OK) return rc;
    if ((rc = alloc_block(ctx, sw, &lblk, rts_bytes<int32_t>(nl), "sweep steps")) != RTS_OK) return rc;
    if ((rc = alloc_block(ctx, sw, &bblk, rts_bytes<uint32_t>(nbd), "sweep boundary faces")) != RTS_OK) return rc;
    cudaStream_t st = ctx->streams[RTS_STREAM_SCATTERING_1];
    int64_t io = 0, lo = 0, bo = 0;
    for (int64_t d = 0; d < D; ++d) {
        sw.h_items[d] = (uint32_t*)iblk + io;
        sw.h_recs[d] = (double*)rblk + 3 * io;
        sw.h_steps[d] = (int32_t*)lblk + lo;
        sw.h_bnd[d] = (uint32_t*)bblk + bo;
        sw.h_nsteps[d] = (int32_t)steps[d].size() - 1;
        sw.h_nbnd[d] = (int32_t)bnd[d].size();
        sw.h_nitems[d] = (int64_t)items[d].size();
        RTS_CUDA_TRY(ctx, cudaMemcpyAsync(sw.h_items[d], items[d].data(), rts_bytes<uint32_t>(items[d].size()),
                                          cudaMemcpyHostToDevice, st));
        RTS_CUDA_TRY(ctx, cudaMemcpyAsync(sw.h_steps[d], steps[d].data(), rts_bytes<int32_t>(steps[d].size()),
                                          cudaMemcpyHostToDevice, st));
        if (!bnd[d].empty())
            RTS_CUDA_TRY(ctx, cudaMemcpyAsync(sw.h_bnd[d], bnd[d].data(), rts_bytes<uint32_t>(bnd[d].size()),
                                              cudaMemcpyHostToDevice, st));
        io += (int64_t)items[d].size();
        lo += (int64_t)steps[d].size();
        bo += (int64_t)bnd[d].size();
    }
    // the face states, for the builder kernel only
    if ((rc = rts_dmalloc(ctx, &sblk, rts_bytes<uint8_t>(std::max<int64_t>(D * N, 16)), "sweep face states")) !=
        RTS_OK)
        return rc;
    RTS_CUDA_TRY(ctx, cudaMemcpyAsync(sblk, states.data(), rts_bytes<uint8_t>(D * N), cudaMemcpyHostToDevice, st));
    if ((rc = upload_tables(ctx, sw, st)) != RTS_OK) {
        rts_dfree(ctx, sblk, rts_bytes<uint8_t>(std::max<int64_t>(D * N, 16)));
        return rc;
    }
    // device: the in-face frames, then the in-face and distance of every node
    void* fblk = nullptr;
    if ((rc = rts_dmalloc(ctx, &fblk, rts_bytes<double>(kFrame * 4 * N), "sweep face frames")) != RTS_OK) {
        rts_dfree(ctx, sblk, rts_bytes<uint8_t>(std::max<int64_t>(D * N, 16)));
        return rc;
    }
    uint32_t* words = alloc_words(ctx, sw, ni);
    for (int64_t d = 0; words && d < D; words += sw.h_nitems[d++]) sw.h_words[d] = words;
    if ((rc = upload_words(ctx, sw, st)) != RTS_OK) {
        rts_dfree(ctx, sblk, rts_bytes<uint8_t>(std::max<int64_t>(D * N, 16)));
        rts_dfree(ctx, fblk, rts_bytes<double>(kFrame * 4 * N));
        return rc;
    }
    if (N > 0) {
        sweep_frames_kernel<<<(unsigned)std::min<int64_t>((4 * N + 255) / 256, 8192), 256, 0, st>>>(
            sw.d_vert, sw.d_normals, N, (double*)fblk);
        ctx->launches++;
    }
    X0Args a;
    a.vert = sw.d_vert;
    a.frames = (const double*)fblk;
    a.nodes = sw.d_nodes;
    a.pairs = sw.d_pairs;
    a.dirs = ctx->d_xyz + 3 * ctx->out_start;
    a.states = (const uint8_t*)sblk;
    a.items = sw.d_items;
    a.recs = sw.d_recs;
    a.steps = sw.d_steps;
    a.nsteps = sw.d_nsteps;
    a.N = N;
    a.words = sw.d_words;
    a.flag = ctx->d_flag + 2;
    if (D > 0) {
        const int64_t per = std::max<int64_t>(1, std::min<int64_t>((2 * N + 255) / 256, 64));
        cudaError_t e = cudaSuccess;
        for (int64_t d0 = 0; d0 < D && e == cudaSuccess; d0 += 65535) {
            a.d0 = d0;
            sweep_x0_kernel<<<dim3((unsigned)per, (unsigned)std::min<int64_t>(D - d0, 65535)), 256, 0, st>>>(a);
            e = cudaGetLastError();
            ctx->launches++;
        }
        cudaStreamSynchronize(st);
        rts_dfree(ctx, sblk, rts_bytes<uint8_t>(std::max<int64_t>(D * N, 16)));
        rts_dfree(ctx, fblk, rts_bytes<double>(kFrame * 4 * N));
        if (e != cudaSuccess)
            return rts_fail(ctx, RTS_ERR_CUDA, "launch of sweep_x0_kernel failed: %s", cudaGetErrorString(e));
    } else {
        rts_dfree(ctx, sblk, rts_bytes<uint8_t>(16));
        rts_dfree(ctx, fblk, rts_bytes<double>(kFrame * 4 * N));
    }
    RTS_CUDA_TRY(ctx, cudaStreamSynchronize(st));
    if ((rc = check_flag(ctx, "rts_sweep_build")) != RTS_OK) return rc;
    std::fill(sw.have.begin(), sw.have.end(), 1);
    sw.records = 3 * ni;
    sw.max_levels = maxl;
    if (records) *records = 3 * ni;
    if (levels) *levels = maxl;
    return RTS_OK;
}

extern "C" int rts_sweep_import_direction(rts_ctx* ctx, int64_t d, const int32_t* order, const int32_t* states,
                                          const void* locx0, int64_t count)
{
    if (!ctx) return RTS_ERR_INVALID_ARGUMENT;
    RTS_REQUIRE(ctx, ctx->sweep, RTS_ERR_BAD_STATE, "rts_sweep_import_direction before rts_sweep_set_mesh");
    rts_sweep_state& sw = *ctx->sweep;
    const int64_t N = sw.N;
    RTS_REQUIRE(ctx, 0 <= d && d < sw.D, RTS_ERR_INVALID_ARGUMENT, "rts_sweep_import_direction: direction %lld outside "
                "the %lld local directions", (long long)d, (long long)sw.D);
    RTS_REQUIRE(ctx, order && states && (locx0 || count == 0), RTS_ERR_INVALID_ARGUMENT,
                "rts_sweep_import_direction: null array");
    const int32_t* pairs = sw.h_pairs.data();
    // steps from the file's order: a cell goes one step after its latest
    // upstream cell (the file's order must list upstream cells first)
    std::vector<int32_t> step((size_t)N, -1), start_rec((size_t)N, 0);
    std::vector<uint8_t> st8((size_t)N);
    int64_t rec = 0;
    int32_t nsteps = 0;
    for (int64_t h = 0; h < N; ++h) {
        const int32_t c = order[h];
        RTS_REQUIRE(ctx, 0 <= c && c < N && step[c] < 0, RTS_ERR_INVALID_ARGUMENT,
                    "rts_sweep_import_direction: order[%lld] = %d is not a new cell", (long long)h, (int)c);
        const int st = states[c] & 15;
        st8[c] = (uint8_t)st;
        int32_t lv = 0;
        for (int f = 0; f < 4; ++f) {
            if (!((st >> f) & 1) || pairs[4 * c + f] < 0) continue;
            const int32_t u = pairs[4 * c + f] >> 2;
            RTS_REQUIRE(ctx, step[u] >= 0, RTS_ERR_INVALID_ARGUMENT,
                        "rts_sweep_import_direction: cell %d comes before its upstream cell %d", (int)c, (int)u);
            lv = std::max(lv, step[u] + 1);
        }
        step[c] = lv;
        nsteps = std::max(nsteps, lv + 1);
        start_rec[c] = (int32_t)rec;
        rec += 3 * (4 - popcount4(st));
    }
    RTS_REQUIRE(ctx, rec == count, RTS_ERR_INVALID_ARGUMENT,
                "rts_sweep_import_direction: %lld records given, the states need %lld", (long long)count,
                (long long)rec);
    // cells grouped by step, the file's order kept within a step
    std::vector<int32_t> lev((size_t)nsteps + 1, 0), pos_order((size_t)N);
    for (int64_t c = 0; c < N; ++c) lev[step[c] + 1]++;
    for (int32_t L = 0; L < nsteps; ++L) lev[L + 1] += lev[L];
    {
        std::vector<int32_t> fill(lev.begin(), lev.end() - 1);
        for (int64_t h = 0; h < N; ++h) pos_order[fill[step[order[h]]]++] = order[h];
    }
    std::vector<uint32_t> items, bnd;
    std::vector<int32_t> steps;
    items_of(N, pairs, st8.data(), pos_order.data(), lev, items, steps, bnd);
    // node records of every item, in item order
    std::vector<double> recs(std::max<size_t>(3 * items.size(), 1));
    const unsigned char* in = (const unsigned char*)locx0;
    for (size_t i = 0; i < items.size(); ++i) {
        const uint32_t c = items[i] >> 8;
        const int f = (int)((items[i] >> 6) & 3u);
        const int st = st8[c];
        int slot = 0;  // rank of f among the cell's out-faces
        for (int g = 0; g < f; ++g)
            if (!((st >> g) & 1)) ++slot;
        for (int m = 0; m < 3; ++m) {
            const unsigned char* r = in + 32 * (int64_t)(start_rec[c] + 3 * slot + m);
            double sv;
            memcpy(&sv, r, sizeof(double));
            const int g = r[24];
            RTS_REQUIRE(ctx, g < 4 && ((st >> g) & 1), RTS_ERR_INVALID_ARGUMENT,
                        "rts_sweep_import_direction: record %lld names face %d, not an in-face of cell %u",
                        (long long)(start_rec[c] + 3 * slot + m), g, c);
            recs[3 * i + m] = sv;
            items[i] |= (uint32_t)g << (2 * m);
        }
    }
    // this direction's own blocks
    int rc;
    void *iblk = nullptr, *rblk = nullptr, *lblk = nullptr, *bblk = nullptr;
    if ((rc = alloc_block(ctx, sw, &iblk, rts_bytes<uint32_t>(items.size()), "sweep items")) != RTS_OK) return rc;
    if ((rc = alloc_block(ctx, sw, &rblk, rts_bytes<double>(3 * items.size()), "sweep node records")) != RTS_OK)
        return rc;
    if ((rc = alloc_block(ctx, sw, &lblk, rts_bytes<int32_t>(steps.size()), "sweep steps")) != RTS_OK) return rc;
    if ((rc = alloc_block(ctx, sw, &bblk, rts_bytes<uint32_t>(bnd.size()), "sweep boundary faces")) != RTS_OK)
        return rc;
    RTS_CUDA_TRY(ctx, cudaMemcpy(iblk, items.data(), rts_bytes<uint32_t>(items.size()), cudaMemcpyHostToDevice));
    uint32_t* const wblk = alloc_words(ctx, sw, (int64_t)items.size());
    if (wblk) {
        std::vector<uint32_t> words(items.size());
        for (size_t i = 0; i < items.size(); ++i) words[i] = copy_word(pairs, st8.data(), items[i]);
        RTS_CUDA_TRY(ctx, cudaMemcpy(wblk, words.data(), rts_bytes<uint32_t>(words.size()), cudaMemcpyHostToDevice));
    }
    RTS_CUDA_TRY(ctx, cudaMemcpy(rblk, recs.data(), rts_bytes<double>(3 * items.size()), cudaMemcpyHostToDevice));
    RTS_CUDA_TRY(ctx, cudaMemcpy(lblk, steps.data(), rts_bytes<int32_t>(steps.size()), cudaMemcpyHostToDevice));
    if (!bnd.empty())
        RTS_CUDA_TRY(ctx, cudaMemcpy(bblk, bnd.data(), rts_bytes<uint32_t>(bnd.size()), cudaMemcpyHostToDevice));
    sw.att_valid = false;
    if (sw.have[d]) sw.records -= 3 * sw.h_nitems[d];
    sw.records += 3 * (int64_t)items.size();
    sw.h_items[d] = (uint32_t*)iblk;
    sw.h_words[d] = wblk;
    sw.h_recs[d] = (double*)rblk;
    sw.h_steps[d] = (int32_t*)lblk;
    sw.h_bnd[d] = (uint32_t*)bblk;
    sw.h_nsteps[d] = nsteps;
    sw.h_nbnd[d] = (int32_t)bnd.size();
    sw.h_nitems[d] = (int64_t)items.size();
    sw.have[d] = 1;
    sw.max_levels = std::max<int64_t>(sw.max_levels, nsteps);
    if ((rc = upload_words(ctx, sw, ctx->streams[RTS_STREAM_SCATTERING_1])) != RTS_OK) return rc;
    return upload_tables(ctx, sw, ctx->streams[RTS_STREAM_SCATTERING_1]);
}

extern "C" int rts_sweep_export_direction(rts_ctx* ctx, int64_t d, int32_t* order, int32_t* states, void* locx0,
                                          int64_t capacity, int64_t* count)
{
    if (!ctx) return RTS_ERR_INVALID_ARGUMENT;
    RTS_REQUIRE(ctx, ctx->sweep, RTS_ERR_BAD_STATE, "rts_sweep_export_direction before rts_sweep_set_mesh");
    rts_sweep_state& sw = *ctx->sweep;
    const int64_t N = sw.N;
    RTS_REQUIRE(ctx, 0 <= d && d < sw.D && sw.have[d], RTS_ERR_INVALID_ARGUMENT,
                "rts_sweep_export_direction: direction %lld has no structures", (long long)d);
    const int64_t ni = sw.h_nitems[d];
    if (count) *count = 3 * ni;
    std::vector<uint32_t> items((size_t)std::max<int64_t>(ni, 1));
    if (ni)
        RTS_CUDA_TRY(ctx, cudaMemcpy(items.data(), sw.h_items[d], rts_bytes<uint32_t>(ni), cudaMemcpyDeviceToHost));
    // cells in order of their first item; a cell's faces that are not items are in-faces
    std::vector<int32_t> od;
    std::vector<uint8_t> outs((size_t)N, 0);
    od.reserve((size_t)N);
    for (int64_t i = 0; i < ni; ++i) {
        const uint32_t c = items[i] >> 8;
        if (!outs[c]) od.push_back((int32_t)c);
        outs[c] |= (uint8_t)(1u << ((items[i] >> 6) & 3u));
    }
    RTS_REQUIRE(ctx, (int64_t)od.size() == N, RTS_ERR_BAD_STATE,
                "rts_sweep_export_direction: %lld of %lld cells have out-faces", (long long)od.size(), (long long)N);
    if (order) memcpy(order, od.data(), rts_bytes<int32_t>(N));
    if (states)
        for (int64_t c = 0; c < N; ++c) states[c] = (int32_t)(~outs[c] & 15u);
    if (!locx0 || capacity < 3 * ni) return RTS_OK;
    std::vector<double> recs((size_t)std::max<int64_t>(3 * ni, 1));
    if (ni)
        RTS_CUDA_TRY(ctx, cudaMemcpy(recs.data(), sw.h_recs[d], rts_bytes<double>(3 * ni), cudaMemcpyDeviceToHost));
    unsigned char* out = (unsigned char*)locx0;
    memset(out, 0, (size_t)(32 * 3 * ni));
    for (int64_t i = 0; i < 3 * ni; ++i) {
        memcpy(out + 32 * i, &recs[i], sizeof(double));
        out[32 * i + 24] = (unsigned char)((items[i / 3] >> (2 * (i % 3))) & 3u);
    }
    return RTS_OK;
}

extern "C" int rts_sweep_set_medium(rts_ctx* ctx, const rts_medium* md, const double* alpha, const double* beta,
                                    const double* Q, const double* bc)
{
    if (!ctx) return RTS_ERR_INVALID_ARGUMENT;
    RTS_REQUIRE(ctx, ctx->sweep, RTS_ERR_BAD_STATE, "rts_sweep_set_medium before rts_sweep_set_mesh");
    RTS_REQUIRE(ctx, md && alpha && beta && Q, RTS_ERR_INVALID_ARGUMENT, "rts_sweep_set_medium: null argument");
    RTS_REQUIRE(ctx, md->mode == RTS_MEDIUM_SCATTERING || md->mode == RTS_MEDIUM_ABSORPTION, RTS_ERR_INVALID_ARGUMENT,
                "rts_sweep_set_medium: unknown mode %d", md->mode);
    RTS_REQUIRE(ctx, md->i_scale != 0.0, RTS_ERR_INVALID_ARGUMENT, "rts_sweep_set_medium: i_scale must not be 0");
    rts_sweep_state& sw = *ctx->sweep;
    const int64_t N = sw.N;
    std::vector<double> m((size_t)(4 * N));
    for (int64_t c = 0; c < N; ++c) medium_entry(md->mode, alpha[c], beta[c], Q[c], &m[4 * c]);
    RTS_CUDA_TRY(ctx, cudaMemcpy(sw.d_med, m.data(), rts_bytes<double>(4 * N), cudaMemcpyHostToDevice));
    sw.md = *md;
    if (bc)
        for (int i = 0; i < 4; ++i) sw.bc[i] = bc[i];
    else
        sw.bc[0] = 0.0, sw.bc[1] = 0.0, sw.bc[2] = 1.0, sw.bc[3] = 0.0;
    sw.has_medium = true;
    sw.att_valid = false;
    return RTS_OK;
}

// Threads per direction, up to the mean size of a step, and as many as leave
// every resident CTA its registers.  Reading form, 82,944 x 400, three CTAs per
// SM: 192 threads 1.83 ms, 160 1.94, 256 (80 registers, spills) 2.30.  With more
// directions 128 threads, 5 CTAs per SM while those hold them all (24,576 x 700,
// five sweeps with their integrals 7.5 ms against 9.6 with 7), then 7 with at
// most 72 registers: one wave of 152 x 7 CTAs holds 1,000 directions.
enum class SweepForm { t512, t256, t192, t128, t128x7 };
static SweepForm sweep_form(const rts_ctx* ctx, const rts_sweep_state& sw)
{
    const int64_t items = sw.records / 3, per_step = items / std::max<int64_t>(1, sw.D * sw.max_levels);
    if (sw.D > 5 * ctx->num_sms) return SweepForm::t128x7;
    if (sw.D > 3 * ctx->num_sms || per_step <= 128) return SweepForm::t128;
    if (sw.D > 2 * ctx->num_sms) return SweepForm::t192;
    return sw.D > ctx->num_sms || per_step <= 256 ? SweepForm::t256 : SweepForm::t512;
}

// The form of the next sweep: 2 reads the stored attenuation factors, 1
// stores them (laying out, and where needed allocating, their block), 0
// evaluates them (the cache switched off, no room for the factors, or so many
// cells of so many directions that the reads take longer than the arithmetic:
// with seven CTAs per SM and 1,000 directions reading takes 1.43 ms and
// evaluating 1.94 at 24,576 cells, 17.4 and 18.2 at 235,824, 54.8 and 53.4 at
// 663,552).
constexpr int64_t kReadCells = (int64_t)1 << 19;
static int att_mode(rts_ctx* ctx, rts_sweep_state& sw, cudaStream_t st, int* mode)
{
    *mode = 0;
    const bool many = sweep_form(ctx, sw) == SweepForm::t128x7;
    if (!ctx->sweep_cache || (many && sw.N > kReadCells)) return RTS_OK;
    if (sw.att_valid) {
        *mode = 2;
        return RTS_OK;
    }
    int64_t nfac = 0;
    const int64_t per = many ? 3 : 4;  // factors per item
    for (int64_t d = 0; d < sw.D; ++d) nfac += per * sw.h_nitems[d];
    const size_t need = rts_bytes<double>(std::max<int64_t>(nfac, 2));
    if (sw.att_bytes != need) {
        rts_dfree(ctx, sw.att_blk, sw.att_bytes);
        sw.att_blk = nullptr;
        sw.att_bytes = 0;
        const std::string keep = ctx->last_error;
        void* p = nullptr;
        const rts_spare spare(ctx);
        if (rts_dmalloc(ctx, &p, need, "sweep attenuation factors") != RTS_OK) {
            ctx->last_error = keep;  // not an error: this sweep evaluates the factors
            return RTS_OK;
        }
        sw.att_blk = (double*)p;
        sw.att_bytes = need;
    }
    int64_t o = 0;
    for (int64_t d = 0; d < sw.D; ++d) {
        sw.h_att[d] = sw.att_blk + o;
        o += per * sw.h_nitems[d];
    }
    RTS_CUDA_TRY(ctx, cudaMemcpyAsync(sw.d_att, sw.h_att.data(), sizeof(double*) * sw.D, cudaMemcpyHostToDevice, st));
    *mode = 1;
    return RTS_OK;
}

template <int T, int kCtas>
static void launch_sweep(const SweepArgs& a, unsigned grid, int mode, cudaStream_t st)
{
    const bool plain = a.md.i_scale == 1.0 && !(a.md.radius > 0);
    auto* kernel = plain ? (mode == 2   ? sweep_kernel<2, true, T, kCtas>
                            : mode == 1 ? sweep_kernel<1, true, T, kCtas>
                                        : sweep_kernel<0, true, T, kCtas>)
                         : (mode == 2   ? sweep_kernel<2, false, T, kCtas>
                            : mode == 1 ? sweep_kernel<1, false, T, kCtas>
                                        : sweep_kernel<0, false, T, kCtas>);
    kernel<<<grid, T, 0, st>>>(a);
}

static int enqueue_sweep(rts_ctx* ctx, cudaStream_t st)
{
    rts_sweep_state& sw = *ctx->sweep;
    int mode = 0;
    int rc = att_mode(ctx, sw, st, &mode);
    if (rc != RTS_OK) return rc;
    RTS_CUDA_TRY(ctx, cudaMemsetAsync(sw.d_norm, 0, sizeof(unsigned long long), st));
    SweepArgs a;
    a.items = sw.d_items;
    a.recs = sw.d_recs;
    a.att = sw.d_att;
    a.steps = sw.d_steps;
    a.bnd = sw.d_bnd;
    a.nsteps = sw.d_nsteps;
    a.nbnd = sw.d_nbnd;
    a.pairs = sw.d_pairs;
    a.nodes = sw.d_nodes;
    a.med = sw.d_med;
    a.S = ctx->d_S;
    a.illum = ctx->d_illum + ctx->out_start * sw.N * 4;
    a.N = sw.N;
    a.words = sw.d_words;
    a.md = sw.md;
    for (int i = 0; i < 4; ++i) a.bc[i] = sw.bc[i];
    exp2_table(kExpThird, a.exptab);
    medium_entry(sw.md.mode, sw.md.ball_alpha, sw.md.ball_beta, sw.md.ball_q, a.ball);
    a.norm = sw.d_norm;
    if (sw.D > 0) {
        rts_timing_begin(ctx, st);
        const unsigned grid = (unsigned)sw.D;
        switch (sweep_form(ctx, sw)) {
        case SweepForm::t512: launch_sweep<512, 1>(a, grid, mode, st); break;
        case SweepForm::t256: launch_sweep<256, 2>(a, grid, mode, st); break;
        case SweepForm::t192: launch_sweep<192, 3>(a, grid, mode, st); break;
        case SweepForm::t128: launch_sweep<128, 5>(a, grid, mode, st); break;
        case SweepForm::t128x7: launch_sweep<128, 7>(a, grid, mode, st); break;
        }
        rts_timing_end(ctx, st);
        RTS_CHECK_LAUNCH(ctx, "sweep_kernel");
        ctx->launches++;
        if (mode == 1) sw.att_valid = true;
    }
    return RTS_OK;
}

static int read_norm(rts_ctx* ctx, cudaStream_t st, double* norm)
{
    unsigned long long bits = 0;
    RTS_CUDA_TRY(ctx, cudaMemcpyAsync(&bits, ctx->sweep->d_norm, sizeof(bits), cudaMemcpyDeviceToHost, st));
    RTS_CUDA_TRY(ctx, cudaStreamSynchronize(st));
    if (bits == 0) {
        *norm = -1.0;
    } else {
        const unsigned long long b = bits - 1;
        memcpy(norm, &b, sizeof(double));
    }
    return RTS_OK;
}

static int sweep_ready(rts_ctx* ctx)
{
    RTS_REQUIRE(ctx, ctx->sweep, RTS_ERR_BAD_STATE, "sweep before rts_sweep_set_mesh");
    rts_sweep_state& sw = *ctx->sweep;
    RTS_REQUIRE(ctx, sw.has_medium, RTS_ERR_BAD_STATE, "sweep before rts_sweep_set_medium");
    for (int64_t d = 0; d < sw.D; ++d)
        RTS_REQUIRE(ctx, sw.have[d], RTS_ERR_BAD_STATE,
                    "sweep: direction %lld has no structures (rts_sweep_build or rts_sweep_import_direction)",
                    (long long)d);
    return RTS_OK;
}

extern "C" int rts_sweep(rts_ctx* ctx, int stream, double* norm)
{
    if (!ctx) return RTS_ERR_INVALID_ARGUMENT;
    RTS_REQUIRE(ctx, stream >= 0 && stream < RTS_STREAM_COUNT, RTS_ERR_INVALID_ARGUMENT, "bad stream id %d", stream);
    int rc = sweep_ready(ctx);
    if (rc != RTS_OK) return rc;
    cudaStream_t st = ctx->streams[stream];
    rts_inputs_changed(ctx);  // the device Illum changes under a resident tensor-core iteration
    if ((rc = enqueue_sweep(ctx, st)) != RTS_OK) return rc;
    if (norm) return read_norm(ctx, st, norm);
    return RTS_OK;
}

extern "C" int rts_illum_solve(rts_ctx* ctx, int precision, int max_iter, double accuracy, int64_t* iters,
                               double* norms)
{
    if (!ctx) return RTS_ERR_INVALID_ARGUMENT;
    RTS_REQUIRE(ctx, max_iter >= 1, RTS_ERR_INVALID_ARGUMENT, "rts_illum_solve: max_iter %d < 1", max_iter);
    const bool tensor =
        precision == RTS_PREC_BF16X3 || precision == RTS_PREC_FP16X3 || precision == RTS_PREC_TF32X3;
    RTS_REQUIRE(ctx, tensor || precision == RTS_PREC_FP64, RTS_ERR_INVALID_ARGUMENT, "unknown precision %d",
                precision);
    int rc = sweep_ready(ctx);
    if (rc != RTS_OK) return rc;
    cudaStream_t st = ctx->streams[RTS_STREAM_SCATTERING_1];
    rts_inputs_changed(ctx);
    int64_t count = 0;
    double norm = -1.0;
    do {
        if ((rc = enqueue_sweep(ctx, st)) != RTS_OK) return rc;
        if (max_iter > 1) {
            rc = tensor ? rts_split_device_call(ctx, precision, st)
                        : rts_launch_scatter_fp64(ctx, 0, ctx->local(), st, nullptr, 0.0, false, false);
            if (rc != RTS_OK) return rc;
        }
        if ((rc = read_norm(ctx, st, &norm)) != RTS_OK) return rc;
        if (norms) norms[count] = norm;
        ++count;
    } while (norm > accuracy && count < max_iter);
    if (iters) *iters = count;
    if (tensor) {
        int flag = 0;
        RTS_CUDA_TRY(ctx, cudaMemcpy(&flag, ctx->d_flag, sizeof(int), cudaMemcpyDeviceToHost));
        if (flag) return rts_fail(ctx, RTS_ERR_DEVICE_WAIT, "tensor-path kernel reported device flag %d", flag);
    }
    return RTS_OK;
}

extern "C" int rts_sweep_exp_check(rts_ctx* ctx, int64_t n, double* max_ulp)
{
    if (!ctx) return RTS_ERR_INVALID_ARGUMENT;
    RTS_REQUIRE(ctx, n >= 2 && max_ulp, RTS_ERR_INVALID_ARGUMENT, "rts_sweep_exp_check: n >= 2 and an output");
    uint64_t tab[kExpTable];
    exp2_table(kExpQuarter, tab);
    void* p = nullptr;
    int rc = rts_dmalloc(ctx, &p, (kExpTable + 1) * sizeof(double), "exp check");
    if (rc != RTS_OK) return rc;
    double* d = (double*)p;
    cudaStream_t st = ctx->streams[RTS_STREAM_SCATTERING_1];
    cudaError_t e = cudaMemcpyAsync(d, tab, sizeof(tab), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(d + kExpTable, 0, sizeof(double), st);
    if (e == cudaSuccess) {
        exp_check_kernel<<<(unsigned)std::min<int64_t>((n + 255) / 256, 1024), 256, 0, st>>>(n, (const uint64_t*)d,
                                                                                             d + kExpTable);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(max_ulp, d + kExpTable, sizeof(double), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    rts_dfree(ctx, d, (kExpTable + 1) * sizeof(double));
    if (e != cudaSuccess) return rts_fail(ctx, RTS_ERR_CUDA, "rts_sweep_exp_check: %s", cudaGetErrorString(e));
    ctx->launches++;
    return RTS_OK;
}

// The reference's unit system and constants (global_value.h:32-52): code units
// of length, density, pressure and radiation, and SI physical constants.
namespace gas {
constexpr double kPi = 3.14159265358979323846;
constexpr double kCLight = 299792458.0;
constexpr double kDist = 1e6;
constexpr double kVelocity = 3 * 1e8;
constexpr double kDensity = 3.34 * 10e-14;
constexpr double kPressure = kDensity * kVelocity * kVelocity;
constexpr double kRadiation = kDensity * kVelocity * kVelocity * kVelocity;
constexpr double kRGas = 8.314;
constexpr double kHPlank = 6.62 * 1e-34;
constexpr double kBoltzmann = 1.38 * 1e-23;
constexpr double kSigmaThomson = 6.652 * 1e-29;
constexpr double kMHydrogen = 1.6735575 * 1e-27;
}  // namespace gas

extern "C" int rts_sweep_medium_gas(int64_t N, const double* density, const double* pressure, double* alpha,
                                    double* beta, double* Q, rts_medium* md)
{
    if (N < 0 || (N > 0 && (!density || !pressure || !alpha || !beta || !Q)) || !md) return RTS_ERR_INVALID_ARGUMENT;
    using namespace gas;
    for (int64_t c = 0; c < N; ++c) {
        const double d = density[c] * kDensity;
        const double p = pressure[c] * kPressure;
        const double T = std::min(1e-6 * p / (d * kRGas), 5000.);
        const double T1 = kBoltzmann * kPi * T;
        const double T2 = T1 * T1;
        const double T4 = T2 * T2;
        const double Ie = T4 * 2 / (15 * kHPlank * kHPlank * kHPlank * kCLight * kCLight);
        const double betta = d * (kSigmaThomson / kMHydrogen);
        alpha[c] = betta;
        beta[c] = betta;
        Q[c] = betta * Ie;
    }
    *md = rts_medium{};
    md->mode = RTS_MEDIUM_SCATTERING;
    md->s_scale = kDist;
    md->i_scale = kRadiation;
    return RTS_OK;
}

