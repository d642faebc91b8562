// rts_group_kernel.cuh -- persistent, grouped tcgen05 contraction of the
// split-precision scattering integral (included by rts_group.cu).
//
// One launch runs one source-iteration step of every problem of a batch: the
// tiles of all problems (128 cells x up to 160 out-directions each; problems
// of different cell and direction counts, phase kernels and precisions) form
// one list that persistent CTAs (one per SM) walk with a fixed stride.
//
// A tile's epilogue moves 16 bytes of HBM per output (the previous S read, S,
// Ibar and the next Ibar), about as long as its contraction takes, so the two
// overlap: 512 TMEM columns hold two accumulators of up to 160 columns and the
// finished sums of the tile before, which warps of their own work on.  (With
// 256-column tiles there was no room: the warps that drained also ran the
// epilogue while the tensor cores waited, 1.29 ms a step of 162,000 x 1,000 in
// FP16; now 0.82.  Tensor-core time 0.5 ms, HBM 0.4 ms.  The contraction alone
// takes 0.62 ms: an accumulator is used again after its chunk's MMAs, the
// drain and the hand-overs between the warps; the epilogue warps' instruction
// fetch and latency are the rest.  Three accumulators of 128 columns instead:
// the copies from L2 take as long as the MMAs, 0.81; with the pair of an SM's
// neighbours on one MMA (cta_group::2) as well, 0.77, but 0.3 more for a queue
// of small problems.)
//
// Warp roles (20 warps, 640 threads, one CTA per SM):
//   warp 0       TMA producer: A (split Ibar rows) and B (split W rows)
//                K-slices into a 5-stage shared-memory ring;
//   warps 1, 2   MMA issuers (one thread each) on alternate chunks of the
//                in-direction range of a tile, an accumulator each, so that
//                one is drained while the other fills; warp 1 also owns TMEM.
//                A stage goes back to the producer as soon as the last MMA
//                that reads it is done;
//   warps 4..11  drain: warp w reads TMEM lanes 32*(w%4).. and half of the
//                tile's columns (rounded up to 16).  After every chunk of
//                `flush` K-slices they add the chunk's accumulator into FP32
//                registers (round-to-nearest adds: the tensor core truncates
//                each accumulate) and release it; a finished tile's sums go
//                to their own TMEM columns;
//   warps 12..19 epilogue (unscaling, source update, residual, S store,
//                relaxation of Ibar in split form) of those sums, 8 columns
//                at a time.
// The drain warps hold 80 sums a thread: the first warpgroup gives them its
// registers.
// Within a chunk the cross products hi*lo and lo*hi (2^-11 or 2^-8 of the
// result) are issued first, while the accumulator is still small, and the two
// hi*hi products last: the truncation then costs about one FP32 ulp of the
// chunk sum per hi*hi MMA.
//
// Relaxed source iterations correct the truncation of the FP32 accumulate
// (each tcgen05.mma rounds toward zero, so the sums come out low by ~1e-7,
// by an amount that depends on how the partial sums grow inside an MMA) with
// a conserved quantity instead of a measured constant: for any W,
//     sum_k (W^T I)_k = sum_j v_j I_j,    v_j = sum_k W[j][k]  (FP64, once).
// E_exact of a step's input needs no pass over it: the relaxation makes the
// next input x' = x/2 + rs S/2, so E_exact' = E_exact/2 + rs (sum_j v_j S_j)/2,
// and the first input's E_exact is computed once at set-up
// (group_energy_init_kernel).  Every relaxed step writes, per cell and per
// epilogue warp, the partial sums of its raw integrals and of v_j S_j into
// per-slot arrays; group_energy_kernel adds the slots, stores each cell's
// delta = E_exact / E_tensor - 1 and advances E_exact, and the next step
// scales that cell's integrals by (1 + delta).  This removes the cell's isotropic bias, the part
// that a relaxed iteration would otherwise compound step after step.  The
// partial sums are exact fixed-point numbers: each block of 8 columns is
// summed in FP32 in column order and rounded to a multiple of a per-row
// power-of-two quantum (2^-43 of a bound on the row's totals), so neither the
// order of the additions nor the tiling of the out-directions changes delta,
// and results stay bit-identical across tile widths and runs.  The kernel is
// compiled with and without this bookkeeping (kEnergy); launches without a
// relaxed problem that uses it run the lighter instantiation.
//
// Every mbarrier wait is bounded (rts_ptx::mbar_wait); a wait that gives up
// sets the device flag, every role stops at its next wait, and the kernel
// drains and exits.

#include <type_traits>

constexpr int G_BM = 128;
constexpr int G_BN = 160;    // at most: the accumulators and the finished sums in 512 TMEM columns
constexpr int G_ACCS = 2;    // accumulators
constexpr int G_STAGES = 5;
constexpr int G_A_BYTES = G_BM * 128;
constexpr int G_B_BYTES = G_BN * 128;
constexpr int G_STAGE_BYTES = G_A_BYTES + G_B_BYTES;
constexpr int G_SLICES = 2;  // column slices of a tile: a warpgroup drains each, another runs its epilogue
constexpr int G_DRAIN_WARP0 = 4, G_DRAIN_WARPS = 4 * G_SLICES;
constexpr int G_EPI_WARP0 = G_DRAIN_WARP0 + G_DRAIN_WARPS, G_EPI_WARPS = 4 * G_SLICES;
constexpr int G_COLS = G_BN / G_SLICES;  // columns of a slice, at most (a multiple of 16)
constexpr int G_THREADS = (G_EPI_WARP0 + G_EPI_WARPS) * 32;
// registers a thread: G_REGS at launch; the first warpgroup gives most of its
// own to the two that drain.  Fewer than 40 for it spill in the issuing loop.
constexpr int G_REGS = 96, G_REGS_ISSUE = 40, G_REGS_DRAIN = 120;
static_assert(G_REGS_ISSUE + 2 * G_REGS_DRAIN + 2 * G_REGS <= 5 * G_REGS, "registers of the block");
constexpr int G_CTAS_PER_SM = 1;
constexpr uint32_t G_TMEM_COLS = 512;
constexpr uint32_t G_FIN = G_ACCS * G_BN;  // TMEM column of the finished sums
constexpr int G_MAX_FLUSH = 2;             // K-slices per chunk
constexpr int G_REL_NB = 2;           // relaxation row buffers per epilogue warp
constexpr int G_REL_BYTES = 2048;     // 32 rows x 32 B hi, then 32 rows x 32 B lo
// ring, accumulator and hand-over barriers (the relaxation's from index
// G_REL_BAR), then the TMEM address
constexpr int G_REL_BAR = 2 * G_STAGES + 2 * G_ACCS + 2;
constexpr int G_BAR_BYTES = (8 * (G_REL_BAR + 1 + G_REL_NB * G_EPI_WARPS) + 127) / 128 * 128;
constexpr int G_REL_BUF = G_REL_NB * G_REL_BYTES;
constexpr size_t G_REL_OFF = (size_t)G_STAGES * G_STAGE_BYTES + G_BAR_BYTES;
constexpr size_t G_SMEM = G_REL_OFF + (size_t)G_EPI_WARPS * G_REL_BUF + 1024;
static_assert(G_SMEM <= 227 * 1024, "shared memory per CTA");

struct GroupProblem {  // aligned as its CUtensorMap members
    CUtensorMap mapA[2];  // split Ibar, ping-pong buffers
    CUtensorMap mapW;     // split W^T
    CUtensorMap mapR[2];  // split Ibar in relaxation boxes (32 + 32 bytes x 32 rows), ping-pong buffers
    int64_t N;            // cells per group
    int64_t ldS;          // row pitch of S32 / S64 in cells (>= N; N unless the output is a cell range of a wider S)
    int64_t rows;         // groups * N
    int64_t tile_begin;   // first global tile index of this problem in the launch
    int64_t tile_off;     // the problem's own first tile in this launch (a step may span launches)
    int m_tiles, n_tiles;
    int Mout, kpad, kblocks, bn, flush, groups;
    int order;            // tile order: 0 the column tiles of a row tile in turn, 1 the row tiles of a column tile
    uint32_t idesc;
    float bias;           // relative correction of the truncation bias of the sums
    int fp16;
    int tf32;             // split TF32 operands (kind::tf32, 16 in-directions per K-slice)
    int sw;               // columns per column slice: half of bn rounded up to 16
    int cur;              // buffer holding the current Ibar
    int relax, residual;
    int flip;             // the step ends in this launch: flip the ping-pong Ibar buffer after it
    const float* rs;      // [rows_pad] row scales (FP16 mode) or null
    const float* rs_inv;
    const float* cs_inv;  // [mpad] column unscale (FP16 mode) or null
    const float* B;       // [rows] source (null: no update)
    const float* lam;     // [groups] albedo
    float* S32;           // [groups][Mout][N], FP32 (the source iteration)
    double* S64;          // [groups][Mout][N], FP64 (host-buffer calls); used instead of S32 when set
    uint16_t* a[2];       // [rows_pad][2*kpad] interleaved split rows
    unsigned long long* resid;  // residual bits of this problem's step
    // energy-conservation correction of relaxed steps (null: none)
    const float* vrow;    // [kpad + 4] v_j = sum_k W[j][k], 0 past M; vrow[kpad] = q0 (below), then c, D, 1/c:
                          // c the mean of the v_j, D = sum_j (v_j - c); output column Mout holds
                          // sum_j (v_j - c) raw_j
    int2* part;           // [n_tiles * G_SLICES][rows_pad] sum_k raw_k in quanta (high, low part) per slot
    float* extra;         // [rows_pad] the raw value of column Mout
    double* ex;           // [rows_pad] sum_j v_j x_j of the current input, in quanta
    float* delta;         // [rows_pad] per-cell correction of the next step (0: none yet)
    const float* rsb;     // [rows_pad] power of two with rsb * 2 max(|Ibar|, |B|) < 2^14 (all modes)
};

// Scale of a row's partial sums: q0 * (the row's scale for the unscaled
// formats), a power of two with (scale * bound of the row's totals) <= 2^21.
// q0 = 2^(7 - ceil(log2 sum_jk |W_jk|)) comes with vrow; values in the units
// the epilogue sees are below 2^14 (FP16, scaled) or 2^14 / rsb (BF16,
// TF32).  0 when out of FP32 range (no correction for the row).
__device__ __forceinline__ float energy_scale(float q0, float rsb)  // rsb: 1 in FP16 mode
{
    const float q = q0 * rsb;
    return (q > 0.0f && q < 3.0e38f) ? q : 0.0f;
}

// Adds y (|y| <= 2^21) to an exact fixed-point sum kept as integer high and
// low parts, hi + lo * 2^-22 (units of 1 and 2^-22): adding 1.5 * 2^23 rounds
// to an integer in FP32, and the remainder, scaled by 2^22 (exact), is
// rounded the same way.  No conversion instructions; the sum of such parts is
// exact in any order.
__device__ __forceinline__ void fixed_add(float y, int& hi, int& lo)
{
    constexpr float MAGIC = 12582912.0f;  // 1.5 * 2^23
    const float t = y + MAGIC;
    const float r = y - (t - MAGIC);
    const float t2 = fmaf(r, 4194304.0f, MAGIC);
    hi += __float_as_int(t) - __float_as_int(MAGIC);
    lo += __float_as_int(t2) - __float_as_int(MAGIC);
}

__device__ __forceinline__ int find_problem(const GroupProblem* probs, int nprob, int64_t t)
{
    int lo = 0, hi = nprob - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (probs[mid].tile_begin <= t)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// a / b of non-negative values, in 32 bits where they fit (a 64-bit division
// is some 200 instructions on the tiles' serial path)
__device__ __forceinline__ int64_t divide(int64_t a, int64_t b)
{
    return ((a | b) >> 32) == 0 ? (int64_t)((uint32_t)a / (uint32_t)b) : a / b;
}

// Row and column tile of a problem's tile lt (0 <= lt < m_tiles * n_tiles).
__device__ __forceinline__ void tile_coords(const GroupProblem& P, int64_t lt, int& m_tile, int& n_tile)
{
    const int per = P.order ? P.m_tiles : P.n_tiles, hi = (int)divide(lt, per), lo = (int)(lt - (int64_t)hi * per);
    m_tile = P.order ? lo : hi;
    n_tile = P.order ? hi : lo;
}

// Relaxation of 8 columns of one split row in place (shared memory):
// Ibar' = 0.5 Ibar + 0.5 * (rs * S), split again into hi + lo; columns at or
// past `nk` become zero (the padding of the split rows).  Returns true when
// an FP16 value leaves the range the row scale allows.
template <bool kFp16>
__device__ __forceinline__ bool relax8(uint4* hp, uint4* lp, const float* snew, float hrsc, int nk)
{
    const uint4 rh = *hp, rl = *lp;
    const uint32_t hw[4] = {rh.x, rh.y, rh.z, rh.w};
    const uint32_t lw[4] = {rl.x, rl.y, rl.z, rl.w};
    uint32_t nh[4], nl[4];
    float amax = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
        const float2 i2 = rts_ptx::join2_any(kFp16, hw[j >> 1], lw[j >> 1]);
        const float x0 = (j < nk) ? fmaf(snew[j], hrsc, 0.5f * i2.x) : 0.0f;
        const float x1 = (j + 1 < nk) ? fmaf(snew[j + 1], hrsc, 0.5f * i2.y) : 0.0f;
        if (kFp16) amax = fmaxf(amax, fmaxf(fabsf(x0), fabsf(x1)));
        rts_ptx::split2_any(kFp16, x0, x1, nh[j >> 1], nl[j >> 1]);
    }
    *hp = make_uint4(nh[0], nh[1], nh[2], nh[3]);
    *lp = make_uint4(nl[0], nl[1], nl[2], nl[3]);
    return amax > 60000.0f;
}

// The same for 4 columns of a split TF32 row (hi and lo as FP32, no scale).
__device__ __forceinline__ void relax4_tf32(float4* hp, float4* lp, const float* snew, float hrsc, int nk)
{
    const float4 h = *hp, l = *lp;
    const float hv[4] = {h.x, h.y, h.z, h.w}, lv[4] = {l.x, l.y, l.z, l.w};
    float nh[4], nl[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float x = (j < nk) ? fmaf(snew[j], hrsc, 0.5f * (hv[j] + lv[j])) : 0.0f;
        rts_ptx::split_tf32(x, nh[j], nl[j]);
    }
    *hp = make_float4(nh[0], nh[1], nh[2], nh[3]);
    *lp = make_float4(nl[0], nl[1], nl[2], nl[3]);
}

template <bool kEnergy>
__global__ void __launch_bounds__(G_THREADS, 1)
group_kernel(const GroupProblem* __restrict__ probs, int nprob, int64_t total_tiles, int* flag)
{
    using namespace rts_ptx;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + G_STAGES * G_STAGE_BYTES);  // G_BAR_BYTES
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + G_REL_BAR + G_REL_NB * G_EPI_WARPS);
    const uint32_t smem_base = smem_u32(smem);
    const uint32_t bar_base = smem_u32(bars);
    auto full_bar = [&](uint32_t s) { return bar_base + 8u * s; };
    auto empty_bar = [&](uint32_t s) { return bar_base + 8u * (G_STAGES + s); };
    auto acc_full_bar = [&](uint32_t a) { return bar_base + 8u * (2 * G_STAGES + a); };
    auto acc_empty_bar = [&](uint32_t a) { return bar_base + 8u * (2 * G_STAGES + G_ACCS + a); };
    const uint32_t fin_full = bar_base + 8u * (2 * G_STAGES + 2 * G_ACCS), fin_empty = fin_full + 8u;
    // relaxation row buffers: barrier of buffer b of epilogue warp w
    auto rel_bar = [&](int w, uint32_t b) { return bar_base + 8u * (G_REL_BAR + G_REL_NB * w + (int)b); };

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < G_STAGES; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (uint32_t a = 0; a < G_ACCS; ++a) {
            mbar_init(acc_full_bar(a), 1);
            mbar_init(acc_empty_bar(a), G_DRAIN_WARPS);
        }
        mbar_init(fin_full, G_DRAIN_WARPS);
        mbar_init(fin_empty, G_EPI_WARPS);
        for (int w = 0; w < G_EPI_WARPS; ++w)
            for (int b = 0; b < G_REL_NB; ++b) mbar_init(rel_bar(w, (uint32_t)b), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), G_TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const bool live = *(volatile int*)flag == 0;

    if (warp < G_DRAIN_WARP0) {
        reg_dec<G_REGS_ISSUE>();
        if (warp == 0) {
            // -------------------------------------------------------- producer
            if (lane == 0 && live) {
                uint32_t it = 0;
                bool ok = true;
                for (int64_t t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
                    const GroupProblem& P = probs[find_problem(probs, nprob, t)];
                    const int64_t lt = t - P.tile_begin + P.tile_off;
                    const int nkb = P.kblocks, bn = P.bn;
                    int m_tile, n_tile;
                    tile_coords(P, lt, m_tile, n_tile);
                    const int m0 = m_tile * G_BM, n0 = n_tile * bn;
                    const void* mapA = &P.mapA[P.cur];
                    const void* mapW = &P.mapW;
                    const uint32_t tx = (uint32_t)(G_A_BYTES + bn * 128);
                    for (int kb = 0; kb < nkb; ++kb, ++it) {
                        const uint32_t s = it % G_STAGES;
                        if (it >= (uint32_t)G_STAGES &&
                            !mbar_wait(empty_bar(s), ((it / G_STAGES) - 1) & 1, flag, FLAG_WAIT_PRODUCER)) {
                            ok = false;
                            break;
                        }
                        mbar_expect_tx(full_bar(s), tx);
                        const uint32_t sa = smem_base + s * G_STAGE_BYTES;
                        tma_load_2d(sa, mapA, kb * 64, m0, full_bar(s));
                        tma_load_2d(sa + G_A_BYTES, mapW, kb * 64, n0, full_bar(s));
                    }
                }
                // no copy may still be in flight when the CTA exits
                for (uint32_t i = (it > (uint32_t)G_STAGES ? it - G_STAGES : 0); i < it; ++i)
                    mbar_wait(full_bar(i % G_STAGES), (i / G_STAGES) & 1, flag, FLAG_WAIT_PRODUCER);
                // nor a commit: the issuers' last arrivals on the ring (those on the accumulators' barriers,
                // committed after them, are waited for by the drain warps, which orders the MMAs, not the arrivals)
                for (uint32_t i = (it > (uint32_t)G_STAGES ? it - G_STAGES : 0); ok && i < it; ++i)
                    mbar_wait(empty_bar(i % G_STAGES), (i / G_STAGES) & 1, flag, FLAG_WAIT_PRODUCER);
            }
        } else if (warp < 3) {
            // -------------------------------------------------------- MMA issuers
            const uint32_t me = (uint32_t)(warp - 1);
            if (lane == 0 && live) {
                const uint32_t desc0 = (uint32_t)smem_desc_sw128(smem_base);  // low word, stage 0
                uint32_t gsl = 0, gch = 0;  // K-slice and chunk counters of this CTA (across tiles)
                bool ok = true;
                for (int64_t t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
                    const GroupProblem& P = probs[find_problem(probs, nprob, t)];
                    const uint32_t idesc = P.idesc, nkb = (uint32_t)P.kblocks, flush = (uint32_t)P.flush;
                    const uint32_t nchunks = (nkb + flush - 1) / flush;
                    // the chunk loop, compiled once per MMA kind
                    auto chunks = [&](auto tf32c) {
                        constexpr bool tf32 = decltype(tf32c)::value;
                        uint32_t acc = 0;
                        // a K-slice's cross products (32 bytes high, 32 bytes low parts, twice), its hi*hi
                        auto cross = [&](uint32_t a, uint32_t accumulate) {
                            const uint32_t b = a + (G_A_BYTES >> 4);
                            umma_lo<tf32>(acc, a, b + 4, idesc, accumulate);
                            umma_lo<tf32>(acc, a + 4, b, idesc, 1u);
                            umma_lo<tf32>(acc, a + 2, b + 6, idesc, 1u);
                            umma_lo<tf32>(acc, a + 6, b + 2, idesc, 1u);
                        };
                        auto high = [&](uint32_t a) {
                            const uint32_t b = a + (G_A_BYTES >> 4);
                            umma_lo<tf32>(acc, a, b, idesc, 1u);
                            umma_lo<tf32>(acc, a + 2, b + 2, idesc, 1u);
                        };
#pragma unroll 1
                        for (uint32_t c = (gch ^ me) & 1u; c < nchunks; c += 2) {
                            const uint32_t g = gch + c, a = g % G_ACCS, i0 = gsl + c * flush, i1 = i0 + 1;
                            const bool two = flush > 1 && c * flush + 1 < nkb;
                            const uint32_t s0 = i0 % G_STAGES, s1 = i1 % G_STAGES;
                            if ((g >= G_ACCS &&
                                 !mbar_wait(acc_empty_bar(a), (g / G_ACCS - 1) & 1, flag, FLAG_WAIT_MMA)) ||
                                !mbar_wait(full_bar(s0), (i0 / G_STAGES) & 1, flag, FLAG_WAIT_MMA) ||
                                (two && !mbar_wait(full_bar(s1), (i1 / G_STAGES) & 1, flag, FLAG_WAIT_MMA))) {
                                ok = false;
                                break;
                            }
                            tc_fence_after();
                            acc = tmem + G_BN * a;
                            const uint32_t a0 = desc0 + s0 * (G_STAGE_BYTES >> 4);
                            const uint32_t a1 = desc0 + s1 * (G_STAGE_BYTES >> 4);
                            // cross products first (the accumulator starts from zero), hi*hi last
                            cross(a0, 0u);
                            if (two) cross(a1, 1u);
                            high(a0);
                            umma_commit(empty_bar(s0));
                            if (two) {
                                high(a1);
                                umma_commit(empty_bar(s1));
                            }
                            umma_commit(acc_full_bar(a));
                        }
                    };
                    if (P.tf32)
                        chunks(std::true_type{});
                    else
                        chunks(std::false_type{});
                    gch += nchunks;
                    gsl += nkb;
                }
            }
        }
    } else if (warp < G_EPI_WARP0) {
        // ------------------------------------------------------------ drain warps
        reg_inc<G_REGS_DRAIN>();
        const int q = warp & 3;                      // TMEM lane quarter
        const int cs = (warp - G_DRAIN_WARP0) >> 2;  // column slice of the tile
        const uint32_t lane_off = (uint32_t)(q * 32) << 16;
        uint32_t gch = 0, tiles = 0;
        bool ok = live;
        // one lane's wait, for the warp
        auto wait = [&](uint32_t bar, uint32_t parity) {
            bool got = true;
            if (lane == 0) got = mbar_wait(bar, parity, flag, FLAG_WAIT_EPILOGUE);
            return __shfl_sync(0xffffffffu, got ? 1 : 0, 0) != 0;
        };
        for (int64_t t = blockIdx.x; t < total_tiles && ok; t += gridDim.x, ++tiles) {
            const GroupProblem& P = probs[find_problem(probs, nprob, t)];
            const int nchunks = (P.kblocks + P.flush - 1) / P.flush;
            const int sw = P.sw;                          // columns per slice (multiple of 16)
            const int ncols = min(sw, P.bn - sw * cs);    // columns of this warp (multiple of 16; <= 0: none)
            const uint32_t col = lane_off + (uint32_t)(sw * cs);
            float run[G_COLS];
#pragma unroll
            for (int j = 0; j < G_COLS; ++j) run[j] = 0.0f;
#pragma unroll 1
            for (int c = 0; c < nchunks; ++c) {
                const uint32_t g = gch + (uint32_t)c, a = g % G_ACCS;
                if (!wait(acc_full_bar(a), (g / G_ACCS) & 1)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t acc = tmem + G_BN * a + col;
#pragma unroll
                for (int j0 = 0; j0 < G_COLS; j0 += 16) {
                    if (j0 < ncols) {
                        float v[16];
                        tmem_ld16(acc + (uint32_t)j0, v);
#pragma unroll
                        for (int j = 0; j < 16; ++j) run[j0 + j] += v[j];
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty_bar(a));
            }
            gch += (uint32_t)nchunks;
            if (!ok) break;
            // hand the sums over, once the epilogue has read the previous tile's
            if (tiles > 0 && !wait(fin_empty, (tiles - 1) & 1)) break;
            tc_fence_after();
#pragma unroll
            for (int j0 = 0; j0 < G_COLS; j0 += 16) {
                if (j0 < ncols) {
                    float v[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = run[j0 + j];
                    tmem_st16(tmem + G_FIN + col + (uint32_t)j0, v);
                }
            }
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(fin_full);
        }
    } else {
        // ------------------------------------------------------------ epilogue warps
        const int q = warp & 3;
        const int cs = (warp - G_EPI_WARP0) >> 2;
        const uint32_t lane_off = (uint32_t)(q * 32) << 16;
        const int ew = warp - G_EPI_WARP0;
        uint8_t* rbuf = smem + G_REL_OFF + (size_t)ew * G_REL_BUF;
        const uint32_t rbuf_s = smem_u32(rbuf);
        uint32_t rel_issued = 0, rel_used = 0;  // relaxation row blocks fetched / consumed by this warp
        uint32_t tiles = 0;
        bool ok = live;
        // the largest change over this warp's tiles of a problem
        float rmax = 0.0f;
        unsigned long long* resid = nullptr;
        auto flush_residual = [&]() {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) rmax = fmaxf(rmax, __shfl_xor_sync(0xffffffffu, rmax, o));
            if (lane == 0 && rmax > 0.0f)
                atomicMax(resid, (unsigned long long)__double_as_longlong((double)rmax));
            rmax = 0.0f;
        };
        for (int64_t t = blockIdx.x; t < total_tiles && ok; t += gridDim.x, ++tiles) {
            const GroupProblem& P = probs[find_problem(probs, nprob, t)];
            if (P.resid != resid) {
                flush_residual();
                resid = P.resid;
            }
            const int sw = P.sw;
            const int ncols = min(sw, P.bn - sw * cs);
            const int64_t lt = t - P.tile_begin + P.tile_off;
            int m_tile, n_tile;
            tile_coords(P, lt, m_tile, n_tile);
            const uint32_t fin = tmem + G_FIN + lane_off + (uint32_t)(sw * cs);
            auto wait_sums = [&]() {
                bool got = true;
                if (lane == 0) got = mbar_wait(fin_full, tiles & 1, flag, FLAG_WAIT_EPILOGUE);
                ok = __shfl_sync(0xffffffffu, got ? 1 : 0, 0) != 0;
                tc_fence_after();
                return ok;
            };
            auto release_sums = [&]() {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(fin_empty);
            };
            if (ncols <= 0) {
                if (wait_sums()) release_sums();
                continue;
            }

            // ---- fused epilogue, reading the sums 8 columns at a time:
            //   S = (1 - lam) B + lam * rs_inv[row] * cs_inv[k] * acc
            //   Ibar' = 0.5 Ibar + 0.5 rs[row] * S   (relaxation, split again)
            const int64_t r = (int64_t)m_tile * G_BM + q * 32 + lane;
            const int64_t Nc = P.N, ld = P.ldS;
            const int Mout = P.Mout;
            const bool in_row = r < P.rows;
            const int64_t grp = in_row ? divide(r, Nc) : 0;
            const int64_t cc = in_row ? r - grp * Nc : 0;
            const bool fp16 = P.fp16 != 0;
            // the energy instantiation runs relaxed source-iteration steps only
            const bool relax = kEnergy || P.relax != 0, residual = kEnergy || P.residual != 0;
            const bool has_B = kEnergy || P.B != nullptr;
            const bool want_rel = kEnergy || (relax && P.S64 == nullptr);  // relax implies Mout == M <= kpad
            // the row's parameters: loads only, used once the sums are there
            const float r_lam = (in_row && has_B) ? P.lam[grp] : 1.0f;
            const float r_inv = (fp16 && in_row) ? P.rs_inv[r] : 1.0f;
            const float r_B = (in_row && has_B) ? P.B[r] : 0.0f;
            const float r_rs = (fp16 && in_row) ? P.rs[r] : 1.0f;
            // energy-conservation correction (relaxed steps): this cell's delta
            // from the previous step; the partial sums of this one.
            const bool ewarp = kEnergy && want_rel && P.part != nullptr;
            const float r_q0 = ewarp ? P.vrow[P.kpad] : 0.0f, r_rsb = (ewarp && in_row && !fp16) ? P.rsb[r] : 1.0f;
            const float r_delta = (ewarp && in_row) ? P.delta[r] : 0.0f, r_bias = P.bias;
            float qrow = 0.0f;
            // the partial sums: sum_k raw_k in fixed point, and the raw value
            // of the extra column Mout (sum_j (v_j - c) raw_j) where this warp
            // holds it; group_energy_kernel derives sum_j v_j S_j from them
            int th = 0, tl = 0;
            float raw_e = 0.0f;
            const int kbase = n_tile * P.bn + sw * cs;
            float* __restrict__ S = P.S32 ? P.S32 + grp * (int64_t)Mout * ld + cc : nullptr;
            // (the energy instantiation runs relaxed source iterations, whose output is S32)
            double* __restrict__ S64 = (!kEnergy && P.S64) ? P.S64 + grp * (int64_t)Mout * ld + cc : nullptr;
            // the column unscales of this warp's columns, a column per lane
            float cs_lane[(G_COLS + 31) / 32];
#pragma unroll
            for (int j = 0; j < (G_COLS + 31) / 32; ++j)
                cs_lane[j] = fp16 && 32 * j + lane < ncols ? __ldg(P.cs_inv + kbase + 32 * j + lane) : 1.0f;
            // The relaxation's split rows move by TMA in units of 32 B hi and
            // 32 B lo of each of the warp's 32 rows (16 columns of a 16-bit
            // split, 8 of a TF32 split): a box load into one of two shared-memory
            // buffers per warp, one unit ahead, and after the update a box store
            // back into the other ping-pong buffer (rows 4*kpad bytes apart would
            // otherwise cost a line per lane on every access).
            bool overflow = false;
            // the steps, compiled once per split format (columns per relaxation unit)
            auto run_steps = [&](auto tf32c) {
                constexpr bool tf32 = decltype(tf32c)::value;
                constexpr int ucols = tf32 ? 8 : 16, ublock = tf32 ? 4 : 5;  // columns per unit, log2 of a block's
                const int row0 = m_tile * G_BM + q * 32;
                const void* map_in = &P.mapR[P.cur];
                const void* map_out = &P.mapR[P.cur ^ 1];
                // units of this warp's columns that hold outputs
                const int u_real = want_rel ? max(0, min(ncols, Mout - kbase) + ucols - 1) / ucols : 0;
                auto unit_x = [&](int k0) { return (k0 & ((1 << ublock) - 1)) * (tf32 ? 2 : 1); };
                auto unit_z = [&](int k0) { return (k0 >> ublock) * 2; };
                int u_next = 0;  // next unit to fetch
                // fetches up to unit u_max, once the store that last read its buffer has done so
                auto pump = [&](int u_max) {
                    for (; u_next < u_real && u_next <= u_max; ++u_next, ++rel_issued) {
                        if (lane == 0) {
                            const uint32_t b = rel_issued % G_REL_NB;
                            const int k0 = kbase + u_next * ucols;
                            bulk_wait_read0();
                            mbar_expect_tx(rel_bar(ew, b), G_REL_BYTES);
                            tma_load_3d(rbuf_s + b * G_REL_BYTES, map_in, unit_x(k0), row0, unit_z(k0), rel_bar(ew, b));
                        }
                    }
                };
                // previous S of a block of 8 columns, loaded one block ahead
                float old[8];
                auto load_old = [&](int e0) {
                    const int k0 = kbase + e0;
                    const int nk = e0 < ncols ? min(8, Mout - k0) : 0;
                    const bool on = in_row && residual && S;
                    const float* sp = S + (int64_t)k0 * ld;
#pragma unroll
                    for (int j = 0; j < 8; ++j, sp += ld) old[j] = on && j < nk ? *sp : 0.0f;
                };
                pump(0);
                load_old(0);
                if (!wait_sums()) return;
                const float lr = r_lam * r_inv, bterm = (1.0f - r_lam) * r_B, hrsc = 0.5f * r_rs;
                qrow = in_row ? energy_scale(r_q0, r_rsb) : 0.0f;
                const bool cons = qrow > 0.0f;
                const float bias = r_bias + (cons ? r_delta : 0.0f);
#pragma unroll 1
                for (int e0 = 0; e0 < ncols; e0 += 8) {
                    const int k0 = kbase + e0;
                    const int nk = min(8, Mout - k0);  // valid columns of this block (same for all lanes)
                    const bool live_k = in_row && nk > 0;
                    float v[8];
                    tmem_ld8(fin + (uint32_t)e0, v);
                    if (e0 + 8 >= ncols) release_sums();
                    float eb = 0.0f;  // raw integrals, in column order
                    const float cl = e0 < 32 ? cs_lane[0] : e0 < 64 ? cs_lane[1] : cs_lane[(G_COLS - 1) / 32];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        // the unscale is a power of two: exact
                        const float raw = v[j] * __shfl_sync(0xffffffffu, cl, (e0 & 31) + j);
                        v[j] = fmaf(fmaf(raw, bias, raw), lr, bterm);
                        if (kEnergy && j < nk) eb += raw;
                        if (kEnergy && j == nk) raw_e = raw;  // column Mout (one block of one warp)
                    }
                    // blocks of 8 columns start at multiples of 8 of the out-directions
                    if (kEnergy && cons && live_k) fixed_add(eb * qrow, th, tl);
                    if (live_k) {
                        if (S64) {
                            double* dp = S64 + (int64_t)k0 * ld;
#pragma unroll
                            for (int j = 0; j < 8; ++j, dp += ld)
                                if (j < nk) *dp = (double)v[j];
                        } else {
                            float* sp = S + (int64_t)k0 * ld;
#pragma unroll
                            for (int j = 0; j < 8; ++j, sp += ld)
                                if (j < nk) {
                                    *sp = v[j];
                                    if (residual) rmax = fmaxf(rmax, fabsf(v[j] - old[j]));
                                }
                        }
                    }
                    load_old(e0 + 8);
                    // this block's unit: wait for the load, relax this lane's row in
                    // place (rows outside the problem stay unchanged), store the box
                    // into the other ping-pong buffer
                    const int u = e0 / ucols, ku = kbase + u * ucols;
                    if (u >= u_real) continue;
                    const uint32_t b = rel_used % G_REL_NB;
                    if (tf32 || !(e0 & 8)) {
                        // the buffer fetched into was read by the previous unit's store, issued
                        // before the TMEM read and the S stores above
                        pump(u + 1);
                        const bool got =
                            mbar_wait(rel_bar(ew, b), (rel_used / G_REL_NB) & 1u, flag, FLAG_WAIT_EPILOGUE);
                        if (!__all_sync(0xffffffffu, got)) {
                            ok = false;
                            break;
                        }
                    }
                    uint8_t* hi = rbuf + b * G_REL_BYTES + 32 * lane;
                    uint8_t* lo = hi + G_REL_BYTES / 2;
                    if (in_row) {
                        if (tf32) {
#pragma unroll
                            for (int h = 0; h < 2; ++h)  // 16 bytes of each part
                                relax4_tf32(reinterpret_cast<float4*>(hi) + h, reinterpret_cast<float4*>(lo) + h,
                                            v + 4 * h, hrsc, nk - 4 * h);
                        } else {
                            uint4* hp = reinterpret_cast<uint4*>(hi + 2 * (e0 & 8));
                            uint4* lp = reinterpret_cast<uint4*>(lo + 2 * (e0 & 8));
                            if (fp16)
                                overflow |= relax8<true>(hp, lp, v, hrsc, nk);
                            else
                                relax8<false>(hp, lp, v, hrsc, nk);
                        }
                    }
                    if (tf32 || (e0 & 8)) {
                        ++rel_used;
                        fence_proxy_async_smem();
                        __syncwarp();
                        if (lane == 0) {
                            tma_store_3d(map_out, unit_x(ku), row0, unit_z(ku), rbuf_s + b * G_REL_BYTES);
                            bulk_commit();
                        }
                    }
                }
            };
            if (P.tf32)
                run_steps(std::true_type{});
            else
                run_steps(std::false_type{});
            if (!ok) break;
            if (kEnergy && ewarp && in_row) {  // this slot's partial sums (zero: no correction)
                P.part[((int64_t)n_tile * G_SLICES + cs) * (P.m_tiles * (int64_t)G_BM) + r] = make_int2(th, tl);
                if (kbase <= Mout && Mout < kbase + ncols) P.extra[r] = qrow > 0.0f ? raw_e : 0.0f;
            }
            if (overflow) atomicOr(flag, FLAG_SCALE_OVERFLOW);
        }
        flush_residual();
        // no copy may still be in flight when the CTA exits (loads are left only by a wait that gave up)
        for (; rel_used < rel_issued; ++rel_used)
            mbar_wait(rel_bar(ew, rel_used % G_REL_NB), (rel_used / G_REL_NB) & 1u, flag, FLAG_WAIT_EPILOGUE);
        if (lane == 0) bulk_wait0();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, G_TMEM_COLS);
    }
}

// After a relaxed step: each cell's correction for the next step, from the
// per-slot partial sums of the step (added in a fixed slot order):
// delta = sum_j v_j I_j / sum_k raw_k - 1, or 0 when either sum is not
// positive or the ratio is far from 1 (a W with cancelling signs).
// blockIdx.y: problem; only problems whose step ended in this launch.
__global__ void group_energy_kernel(const GroupProblem* __restrict__ probs, int nprob)
{
    const GroupProblem& P = probs[blockIdx.y];
    if (!(P.relax && P.flip && P.part && P.S64 == nullptr)) return;
    const int64_t ld = P.m_tiles * (int64_t)G_BM;
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < P.rows;
         r += (int64_t)gridDim.x * blockDim.x) {
        long long et = 0;  // exact: in units of 2^-22 of the row's quantum
        const float raw_e = P.extra[r];
        for (int nt = 0; nt < P.n_tiles; ++nt)
            for (int cs = 0; cs < G_SLICES; ++cs) {
                if (P.sw * cs >= P.bn) continue;  // a column slice without columns
                const int2 v = P.part[((int64_t)nt * G_SLICES + cs) * ld + r];
                et += ((long long)v.x << 22) + v.y;
            }
        const double q22 = 1.0 / 4194304.0;  // the slots' units, in quanta
        const double ex = P.ex[r];           // sum_j v_j x_j of this step's input, in quanta
        const bool fp16 = P.fp16 != 0;
        const float qrow = energy_scale(P.vrow[P.kpad], fp16 ? 1.0f : P.rsb[r]);
        // the step's S_j = (1 + b) lr raw_j + bterm (lr = lam / rs, rs = 1
        // for the unscaled formats), so with v_j = c + d_j
        //   rs sum_j v_j S_j = (1 + b) lam (c sum_j raw_j + sum_j d_j raw_j) + rs bterm sum_j v_j,
        // the raw sums in the units the epilogue sees (scaled by rs)
        const float d_old = P.delta[r];
        const double b1 = 1.0 + (double)(P.bias + (qrow > 0.0f ? d_old : 0.0f));
        const int64_t grp = r / P.N;
        const double lam = (double)P.lam[grp];
        const double bterm = P.B ? (1.0 - lam) * (double)P.B[r] : 0.0;
        const double rs = fp16 ? (double)P.rs[r] : 1.0;
        const double c = (double)P.vrow[P.kpad + 1], V = c * P.Mout + (double)P.vrow[P.kpad + 2];
        const double ev = b1 * lam * (c * ((double)et * q22) + (double)raw_e * qrow) + rs * bterm * V * qrow;
        float d = 0.0f;
        if (ex > 0.0 && et > 0) {
            const double g = ex / ((double)et * q22) - 1.0;
            if (fabs(g) < 1e-4) d = (float)g;
        }
        P.delta[r] = d;
        // the next input is x / 2 + rs S / 2
        P.ex[r] = qrow > 0.0f ? 0.5 * ex + 0.5 * ev : 0.0;
    }
}

// x as FP64, from the bits on the integer pipe (the conversion instruction
// runs on the FP64 pipe, at two per SM per cycle); zeros, subnormals and
// non-finite values take the instruction, out of line: predicated into the
// loop it would hold the FP64 pipe without doing anything.
__device__ __noinline__ double f32_to_f64_cvt(float x) { return (double)x; }
__device__ __forceinline__ double f32_to_f64_bits(float x)
{
    const uint32_t u = __float_as_uint(x);
    const uint32_t e = u & 0x7F800000u;
    if (e == 0u || e == 0x7F800000u) return f32_to_f64_cvt(x);
    return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7FFFFFFFu) >> 3) + (896u << 20))), (int)(u << 29));
}

// sum_j v_j x_j of every row of the current split input, in the quanta of
// energy_scale (FP64, once per set-up of an iteration): the split values
// joined as the tensor core multiplies them (hi + lo).  A warp per row, its
// lanes on consecutive columns (coalesced), FP64 lane sums reduced in a fixed
// shuffle order.  The conversions of both factors are integer operations:
// 1,151 us with conversion instructions, 416 this way (162,000 x 1000).
__global__ void group_energy_init_kernel(const uint16_t* __restrict__ A, int64_t rows, int kpad, int M, int mode,
                                         const float* __restrict__ vrow, const float* __restrict__ rs, double* ex)
{
    const int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (r >= rows) return;  // r is uniform over the warp
    float q = vrow[kpad] * (mode == 1 ? 1.0f : rs[r]);
    if (!(q > 0.0f && q < 3.0e38f)) q = 0.0f;
    double s = 0.0;
    if (mode == 2) {
        const float* row = reinterpret_cast<const float*>(A + r * 4 * (int64_t)kpad);
#pragma unroll 4
        for (int j = lane; j < M; j += 32) {
            const int h = (j >> 4) * 32 + (j & 15);
            s += f32_to_f64_bits(vrow[j]) * f32_to_f64_bits(row[h] + row[h + 16]);
        }
    } else {
        const uint16_t* row = A + r * 2 * (int64_t)kpad;
#pragma unroll 4
        for (int j = lane; j < M; j += 32) {
            const int64_t h = rts_ptx::ilv_hi(j);
            s += f32_to_f64_bits(vrow[j]) * f32_to_f64_bits(rts_ptx::join_any(mode == 1, row[h], row[h + 32]));
        }
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) ex[r] = s * (double)q;
}

// Flip the ping-pong Ibar buffer of every problem whose relaxed step ended in
// this launch (launched after it, so that a captured graph replays step after
// step on the device).
__global__ void group_flip_kernel(GroupProblem* probs, int nprob)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < nprob && probs[p].flip) probs[p].cur ^= 1;
}
