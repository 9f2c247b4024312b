// oz_gemm.cuh -- stage (c) + (d): slice-pair GEMMs on tcgen05 with exact
// accumulation, fused with the FP64 reconstruction.
//
// Reference semantics (atlarge-research/ozAIE):
//   bins[p+q] += A_p . B_q over the pair set      src/aie_kernels/aie2p/mm_ozaki.cc:255-308
//   bins accumulate over all of K per C tile       whole_array_iron_ozaki.py:494-548
//   bin-weighted sum + exponent scale-back         src/aie_kernels/generic/ozaki_base.cc:143-340
//   int128 -> double reconstruction                include/oz_aie.h:92-150
//
// GB300 design (persistent CTAs, one per SM, each looping over 128 x BN tiles of
// C; 640 threads: a producer warp, up to three MMA-issuing warps on three schedulers
// and 16 drain/epilogue warps):
//   * Carrier: tcgen05.mma kind::f16 with bf16 slices (|v| <= 127 is exact in
//     bf16) and fp32 accumulators in TMEM.  (kind::i8 is not accepted by ptxas
//     for sm_103a.)  Slices of b <= 4 bits may instead be e4m3 (kind::f8f6f4,
//     template F8): a 64-deep e4m3 chunk has the byte layout of a 32-deep bf16
//     one, so only the instruction and its operand formats change.  Every
//     partial sum is an integer of magnitude <= 2^24 as
//     long as bin j accumulates at most KB_j K-values between drains,
//     pairs_in_bin(j) * KB_j * (2^b-1)^2 <= 2^24, so the fp32 accumulation is exact.
//   * TMEM holds one fp32 accumulator of BN columns per bin j (column j*BN), and
//     a second range for each double-buffered block where the columns allow it.
//     Bins are partitioned into up to 8 blocks of at most 256 columns.  A UMMA
//     takes A slice p against the B slices q = j - p of the bins j of one block,
//     which are consecutive in shared memory, and covers exactly the bins that
//     hold a pair.  On GB300 a M=128, K=16 UMMA of N columns takes
//     max(N/2, 32 + N/4) cycles (the tensor pipe, or its operands from shared
//     memory at 128 bytes a cycle).
//   * Each block belongs to one issuing warp, which issues its UMMAs in order, and the
//     first one after a drain overwrites the accumulator.  Issuers do not wait for
//     one another beyond the stage ring.  (Assumed: the tensor pipe executes the UMMAs of
//     one thread on overlapping accumulator columns in the order of issue, also where N and
//     the first column change.  The PTX text promises that order for equal accumulator and
//     shape; for the rest it rests on the bit-exact tests against the oracle, in which a
//     UMMA that overtook the overwriting one would lose its products.)  e4m3 plans of two
//     blocks deal their UMMAs over all three issuers where one would have most of them
//     (oz_plan.cpp); those only accumulate, in any order.
//   * Each block is a drain group with its own period: its tightest bin's, or longer
//     where the norms of the tile's slices allow it (DrainSchedule).  A block
//     whose accumulator is being read out holds up its own issuer only; a
//     double-buffered block switches ranges at each drain instead.
//   * Drain (warps 4..19): TMEM -> registers, fp32 -> int32 (exact), then one
//     32 x 32 -> 64-bit multiply-add by 2^rel into the 64-bit accumulator of the
//     bin's group (consecutive bins whose weights relative to the group's first
//     bin stay <= 2^30).  The buffer is released as soon as its last bin is in
//     registers.
//   * The last partial wave of a launch may be split along K (split_parts): the
//     parts add their 64-bit group sums into global scratch with atomics and
//     the part that completes a tile's count rounds and stores it.
//   * Epilogue: the exact sum is rounded once to FP64 with the scale
//     2^{Er+Ec-2044-b(J+1)} (round-to-nearest, or the reference's truncating
//     decode, or written raw for parity dumps).
//   * Every mbarrier wait is bounded (globaltimer); on expiry the kernel records
//     an error code, waits for its own copies and MMAs, frees TMEM and returns.
//
// At 4096^3 (s = 8, p + q <= 8, 2752 tiles of 128 x 48) the launch takes 3.35 ms (1764
// TFLOP/s of slice-pair products; 3.27 ms with the autotuner's plan): 1440 cycles per K step
// of a tile, of which the UMMAs need 1104.  Without drains it takes 1270; the rest is the
// issuers and drain warps sharing the schedulers.  (1769 cycles before: UMMAs over whole
// blocks, 1224 cycles a K step with their zero slices, and drains by the worst case.)
#pragma once
#include <cuda_runtime.h>

#include <atomic>

#include "oz_internal.h"
#include "oz_ptx.cuh"

namespace ozgb {

// ------------------------------------------------------------ drain adds
// d = a * m + c with a 64-bit result: one multiply-add per drained value.
__device__ __forceinline__ long long mad_wide(int32_t a, int32_t m, long long c) {
    long long d;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(m), "l"(c));
    return d;
}

// acc[i][A] += v[i] * 2^rel modulo 2^64 for NV fp32 values holding exact
// integers (|v| <= 2^24).  Exact-mode plans keep rel <= 30; the paired output of the
// reference (sums modulo 2^64) may need up to 63.  (An FP32 add of 1.5 2^23 instead of
// F2I, for values below 2^22, measured 1 % slower: the check costs what it saves.)
template <int NA, int A, int NV>
__device__ __forceinline__ void acc_add(long long (*acc)[NA], const uint32_t *v, int rel) {
    if (rel <= 30) {
        const int32_t m = 1 << rel;
#pragma unroll
        for (int i = 0; i < NV; ++i) acc[i][A] = mad_wide(__float2int_rz(__uint_as_float(v[i])), m, acc[i][A]);
    } else {
#pragma unroll
        for (int i = 0; i < NV; ++i)
            acc[i][A] += static_cast<long long>(
                static_cast<unsigned long long>(static_cast<long long>(__float2int_rz(__uint_as_float(v[i])))) << rel);
    }
}

// The accumulator index is a template argument: a runtime index into acc would
// place the whole array in local memory.
template <int NA, int NV>
__device__ __forceinline__ void acc_add_group(long long (*acc)[NA], const uint32_t *v, int a, int rel) {
    switch (a) {
        case 0: acc_add<NA, 0, NV>(acc, v, rel); break;
        case 1: if constexpr (NA > 1) acc_add<NA, 1, NV>(acc, v, rel); break;
        case 2: if constexpr (NA > 2) acc_add<NA, 2, NV>(acc, v, rel); break;
        case 3: if constexpr (NA > 3) acc_add<NA, 3, NV>(acc, v, rel); break;
        default: break;
    }
}

// ------------------------------------------------------------ q -> double
// The exact sum of an element's accumulator groups, sum_x acc[x] 2^B[x] (B[0] = 0),
// as a 128-bit window S = (hi, lo), two's complement, and what lies below it: value =
// (S + f) 2^low with 0 <= f < 1 and sticky = (f != 0).  The bits of a group above the
// next group's weight are first carried into that group (the groups are at most 37
// bits apart and stay below 2^62); then the window takes the groups from the top.  A
// group that no longer fits (|S| is then past 2^64, well over the 53 bits of a result)
// only sets sticky.  64-bit words throughout: the compiler's 128-bit shifts by a
// variable made this and the rounding 390 instructions, now about 80.
struct Window {
    long long hi;
    unsigned long long lo;
    bool sticky;
    int low;
};
template <int NA>
OZ_HD inline Window acc_window(const long long (&acc)[NA], int n_acc, const int (&B)[kMaxAcc]) {
    long long top = acc[0];
    unsigned long long dig[NA];  // dig[x]: group x's bits below group x + 1's weight
#pragma unroll
    for (int x = 1; x < NA; ++x)
        if (x < n_acc) {
            const int d = B[x] - B[x - 1];
            dig[x - 1] = static_cast<unsigned long long>(top) & ((1ull << d) - 1ull);
            top = acc[x] + (top >> d);
        }
    Window w;
    w.hi = top >> 63;
    w.lo = static_cast<unsigned long long>(top);
    w.sticky = false;
    w.low = B[n_acc - 1];
    bool full = false;
#pragma unroll
    for (int x = NA - 1; x >= 1; --x)
        if (x < n_acc) {
            const int d = B[x] - B[x - 1];
            // the first of these fits: |top| < 2^63; else |S| < 2^(126 - d)
            if (x == n_acc - 1 || (!full && ((w.hi ^ (w.hi >> 63)) >> (62 - d)) == 0)) {
                w.hi = static_cast<long long>((static_cast<unsigned long long>(w.hi) << d) | (w.lo >> (64 - d)));
                w.lo = (w.lo << d) | dig[x - 1];
                w.low = B[x - 1];
            } else {
                full = true;
                w.sticky = w.sticky || dig[x - 1] != 0;
            }
        }
    return w;
}

OZ_HD inline int clz64(unsigned long long x) {
#if defined(__CUDA_ARCH__)
    return __clzll(static_cast<long long>(x));
#else
    return __builtin_clzll(x);
#endif
}

// Bits of the double nearest to h 2^(biased - 1086) (h normalised, its lowest bit
// sticky) when the biased exponent is outside [1, 2046]: subnormal, zero or infinite.
OZ_HD inline unsigned long long round_out_of_range(unsigned long long h, int biased) {
    if (biased >= 2047) return 0x7FF0000000000000ull;
    const int sh = 12 - biased;  // >= 12
    if (sh > 64) return 0ull;
    if (sh == 64) return h > 0x8000000000000000ull ? 1ull : 0ull;
    unsigned long long mm = h >> sh;
    const bool rb = ((h >> (sh - 1)) & 1ull) != 0, st = (h & ((1ull << (sh - 1)) - 1ull)) != 0;
    if (rb && (st || (mm & 1ull))) ++mm;
    return mm;
}

// Bits of (S + f) 2^(e2 + low) as a double: rounded to nearest even (OUT_RN) or the
// reference's truncating decode (OUT_RZ_REF, include/oz_aie.h:129-146: 53 truncated
// bits and the exponent added modulo 2^64).
OZ_HD inline unsigned long long window_bits(const Window &w, int e2, int mode) {
    // the magnitude's floor: -(S + f) = ~S + (1 - f) when f != 0
    const unsigned long long neg = static_cast<unsigned long long>(w.hi >> 63);
    unsigned long long lo = w.lo ^ neg, hi = static_cast<unsigned long long>(w.hi) ^ neg;
    if (neg != 0 && !w.sticky) hi += ++lo == 0 ? 1u : 0u;
    if ((hi | lo) == 0) return 0ull;
    // normalise: the top bit to bit 63 of hi, what falls below into its lowest bit
    int L = 128;
    if (hi == 0) {
        hi = lo;
        lo = 0;
        L = 64;
    }
    const int n = clz64(hi);
    L -= n;
    hi = (hi << n) | ((lo >> 1) >> (63 - n));
    if ((lo << n) != 0 || w.sticky) hi |= 1ull;
    const unsigned long long sign = neg << 63;
    const int biased = L + e2 + w.low + 1022;
    if (mode == OUT_RZ_REF)
        return (hi >> 11) - 0x0010000000000000ull + sign +
               (static_cast<unsigned long long>(static_cast<long long>(biased)) << 52);
    if (biased < 1 || biased > 2046) return sign | round_out_of_range(hi, biased);
    const uint32_t w0 = static_cast<uint32_t>(hi);
    const uint32_t up = ((w0 & 0x7FFu) + 0x3FFu + ((w0 >> 11) & 1u)) >> 11;
    return sign + (static_cast<unsigned long long>(biased - 1) << 52) + (hi >> 11) + up;
}

// ------------------------------------------------------------------ kernel
// The operands and output of one tile and its position.  Grouped rasterisation:
// 8 M-tiles share the same stream of B tiles.
struct TileRef {
    const uint8_t *a_src;
    const uint8_t *b_src;
    const int32_t *er;
    const int32_t *ec;
    double *c;
    long ldc;
    const float *na, *nb;  // the tile's slice norms (null: static drain periods)
    int M, N, n_kc, mt, nt;
    int c0, c1;  // chunks of K this work unit covers
    int split;   // index of the split tile (-1: the unit is a whole tile)
};

// Tile t of a problem whose tiles are rasterised in groups of 8 row tiles that
// share the same stream of B tiles.
OZ_HD inline void raster(int t, int tiles_m, int tiles_n, int *mt, int *nt) {
    const int GM = 8;
    const int per_group = GM * tiles_n;
    const int grp = t / per_group;
    const int first_m = grp * GM;
    const int gm = (tiles_m - first_m) < GM ? (tiles_m - first_m) : GM;
    const int rr = t - grp * per_group;
    *mt = first_m + rr % gm;
    *nt = rr / gm;
}

// Work unit u of a grouped launch: problem tile_prob[u], its tile u - tile0.
// Shared by the kernel and the host-side check of grouped launches.
OZ_HD inline void group_tile_ref(const GroupProblem *probs, const int *tile_prob, int u, uint32_t a_block_bytes,
                                 uint32_t b_block_bytes, TileRef *r) {
    const GroupProblem &P = probs[tile_prob[u]];
    r->split = -1;
    r->c0 = 0;
    r->c1 = P.n_kc;
    r->er = P.er;
    r->ec = P.ec;
    r->c = P.c;
    r->ldc = P.ldc;
    r->M = P.M;
    r->N = P.N;
    r->n_kc = P.n_kc;
    raster(u - P.tile0, P.tiles_m, P.tiles_n, &r->mt, &r->nt);
    r->a_src = P.a_tiles + static_cast<size_t>(r->mt) * P.n_kc * a_block_bytes;
    r->b_src = P.b_tiles + static_cast<size_t>(r->nt) * P.n_kc * b_block_bytes;
    r->na = r->nb = nullptr;
}

__device__ __forceinline__ void tile_ref(const GemmArgs &g, int u, TileRef *r) {
    if (g.probs) {
        group_tile_ref(g.probs, g.tile_prob, u, g.a_block_bytes, g.b_block_bytes, r);
        return;
    }
    int t = u, kpart = 0;
    r->split = -1;
    if (g.split_parts > 1 && u >= g.split_start) {
        const int v = u - g.split_start;
        r->split = v / g.split_parts;
        kpart = v - r->split * g.split_parts;
        t = g.split_start + r->split;
    }
    r->c0 = r->split < 0 ? 0 : (kpart * g.n_kc) / g.split_parts;
    r->c1 = r->split < 0 ? g.n_kc : ((kpart + 1) * g.n_kc) / g.split_parts;
    r->er = g.er;
    r->ec = g.ec;
    r->c = g.c;
    r->ldc = g.ldc;
    r->M = g.M;
    r->N = g.N;
    r->n_kc = g.n_kc;
    raster(t, g.tiles_m, g.tiles_n, &r->mt, &r->nt);
    r->a_src = reinterpret_cast<const uint8_t *>(g.a_tiles) + static_cast<size_t>(r->mt) * g.n_kc * g.a_block_bytes;
    r->b_src = reinterpret_cast<const uint8_t *>(g.b_tiles) + static_cast<size_t>(r->nt) * g.n_kc * g.b_block_bytes;
    r->na = g.na ? g.na + static_cast<size_t>(r->mt) * g.s : nullptr;
    r->nb = g.na ? g.nb + static_cast<size_t>(r->nt) * g.s : nullptr;
}

// ------------------------------------------------------------ drain schedule
// Block g is drained after chunk c when (c + 1 + off) % period == 0, and every block
// after the last chunk.  One warp steps it, lane i for block i; every issuing warp and
// the first drain warp step identical copies.  With norms (GemmArgs::na) a tile's
// periods follow from its operands: about 600 cycles per tile, for 1.8 to 3 times
// fewer drains on operands whose digits are spread over their range.
struct DrainSchedule {
    int period, until;  // of block `lane`: chunks between drains, chunks to the next one
    __device__ __forceinline__ void init(const GemmArgs &g, const TileRef &tr, int lane) {
        period = 1 << 29;
        if (lane < g.G) period = g.blk_period[lane];
        if (tr.na) {
            // rounded up throughout; a bound of 0 (no such digits) leaves the period long
            const float a = lane < g.s ? __fsqrt_ru(ld_after_wait(tr.na + lane)) : 0.0f;
            const float b = lane < g.s ? __fsqrt_ru(ld_after_wait(tr.nb + lane)) : 0.0f;
            float bound = 0.0f;  // of bin `lane`, per chunk
            for (int p = 0; p < g.s; ++p) {
                const float ap = __shfl_sync(0xffffffffu, a, p);
                const float bq = __shfl_sync(0xffffffffu, b, (lane - p) & 31);
                if (lane >= p && lane - p < g.s) bound = __fmaf_ru(ap, bq, bound);
            }
            const int chunks =
                bound > 16.0f ? static_cast<int>(__fdiv_rd(16777216.0f, bound)) : 1 << 20;
            const int lo = lane < g.G ? g.blk_lo[lane] : 0, hi = lane < g.G ? lo + g.blk_nb[lane] - 1 : -1;
            int mine = 1 << 20;
            for (int j = 0; j < g.J; ++j) {
                const int cj = __shfl_sync(0xffffffffu, chunks, j);
                if (j >= lo && j <= hi) mine = min(mine, cj);
            }
            if (lane < g.G) period = max(period, mine);
        }
        until = lane < g.G ? period - static_cast<int>((static_cast<long long>(lane) * period) / g.G) : 1 << 29;
    }
    // Chunks to the next drain, at most left.
    __device__ __forceinline__ int next(int left) const {
        return min(static_cast<int>(__reduce_min_sync(0xffffffffu, static_cast<unsigned>(until))), left);
    }
    // Mask of the blocks drained `step` chunks on (next's result), without the tile's end.
    __device__ __forceinline__ uint32_t advance(int step, int lane, int G) {
        until -= step;
        const uint32_t m = __ballot_sync(0xffffffffu, until == 0 && lane < G);
        if (until == 0) until = period;
        return m;
    }
};

// Persistent: CTA b processes tiles b, b + gridDim.x, ...  The stage ring, the
// bin-block barriers and TMEM persist across tiles, so the producer prefetches
// the next tile's first chunks and the UMMAs of the next tile start as soon as
// each block's final drain of the previous tile has read it out, while the
// drain warps round and store the previous tile.
template <int BN, int W, int KC, bool F8>
__global__ void __launch_bounds__(kThreads, 1) oz_gemm_kernel(const __grid_constant__ GemmArgs g) {
    constexpr int PARTS = kEpiWarps / 4;          // drain warps sharing one TMEM lane quadrant
    constexpr int COLS = BN / PARTS;              // columns per drain thread
    constexpr int NA = W > 2 ? W - 1 : 1;         // 64-bit accumulator groups per column
    static_assert(NA <= kMaxAcc, "accumulator groups");
    static_assert(COLS % 4 == 0, "BN must split into 4-column parts");

    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    // A in parts (e4m3 plans whose slices fill shared memory, GemmArgs::parts): a ring of
    // A parts and one of two B blocks; otherwise a ring of stages that hold both
    const int parts = F8 ? g.parts : 1;
    const uint32_t a_stride = parts > 1 ? g.part_bytes : g.stage_bytes;
    const uint32_t b_base = parts > 1 ? static_cast<uint32_t>(g.stages) * g.part_bytes : g.a_block_bytes;
    const uint32_t b_stride = parts > 1 ? g.b_block_bytes : g.stage_bytes;
    uint64_t *full = reinterpret_cast<uint64_t *>(
        smem + (parts > 1 ? b_base + kPartStagesB * g.b_block_bytes : static_cast<uint32_t>(g.stages) * g.stage_bytes));
    uint64_t *empty = full + g.stages;
    uint64_t *fullb = empty + g.stages;  // parts > 1: the B ring
    uint64_t *emptyb = fullb + kPartStagesB;
    uint64_t *gfull = emptyb + kPartStagesB;
    uint64_t *gempty = gfull + 2 * kMaxGroups;  // [block][buffer]: index 2 * blk + buf
    uint64_t *mma_done = gempty + 2 * kMaxGroups;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(mma_done + 1);
    int *abort_flag = reinterpret_cast<int *>(tmem_slot + 1);
    volatile int *vabort = abort_flag;
    // accumulator group of bin j and the log2 of its weight in it: a | rel << 8 at [j]
    int *bin_tab = abort_flag + 1;
    int *split_flag = bin_tab + 32;  // this CTA's part completed a split tile
    // the drain warps' last two commands
    int2 *drain_cmd = reinterpret_cast<int2 *>((reinterpret_cast<uintptr_t>(split_flag + 1) + 7) & ~uintptr_t(7));
    // the issuers' UMMA lists, decoded: x = accumulator column | the block's other
    // buffer's << 16, y = A offset | the block's first << 14 and last << 15 entries of the
    // chunk | block << 16 | entries left in the block (and part) << 24,
    // z = B offset (descriptor units), w = instruction descriptor
    uint4 *recs = reinterpret_cast<uint4 *>((reinterpret_cast<uintptr_t>(drain_cmd + 2) + 15) & ~uintptr_t(15));

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    const int n_iss = g.n_iss < 1 ? 1 : (g.n_iss > kMaxIssuers ? kMaxIssuers : g.n_iss);  // MMA-issuing warps
    for (int i = threadIdx.x; i < g.op_end[n_iss - 1]; i += kThreads) {
        const uint32_t op = g.ops[i];
        const int p = op_p(op), lo = op_lo(op), nb = op_nb(op), blk = op_blk(op);
        const uint32_t d0 = static_cast<uint32_t>(lo * BN);
        const uint32_t d1 = ((g.dbl_mask >> blk) & 1u)
                                ? static_cast<uint32_t>(g.blk_col1[blk] + (lo - g.blk_lo[blk]) * BN)
                                : d0;
        const uint32_t idesc = (F8 ? idesc_e4m3_f32(BM, 16) : idesc_bf16_f32(BM, 16)) & ~(0x3Fu << 17);
        recs[i] = make_uint4(d0 | (d1 << 16),
                             static_cast<uint32_t>(p % g.part_slices) * ((BM * KC * 2) >> 4) |
                                 (op_first(op) ? 0x4000u : 0u) | (op_last(op) ? 0x8000u : 0u) | (static_cast<uint32_t>(blk) << 16) |
                                 (static_cast<uint32_t>(op_left(op)) << 24),
                             static_cast<uint32_t>(lo - p) * ((BN * KC * 2) >> 4),
                             idesc | (static_cast<uint32_t>((nb * BN) >> 3) << 17));
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < g.stages; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], n_iss);
        }
        for (int i = 0; i < kPartStagesB; ++i) {
            mbar_init(&fullb[i], 1);
            mbar_init(&emptyb[i], n_iss);
        }
        for (int i = 0; i < g.G; ++i) {
            for (int b = 0; b < 2; ++b) {
                mbar_init(&gfull[2 * i + b], g.blk_commits[i]);
                mbar_init(&gempty[2 * i + b], kEpiWarps);
            }
        }
        mbar_init(mma_done, n_iss);
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == 1 && lane < g.J) {
        const int tb = g.J - 1 - lane;
        int a = 0, t0 = 0;
        for (int y = 1; y < g.n_acc; ++y)
            if (tb >= g.acc_t0[y]) {
                a = y;
                t0 = g.acc_t0[y];
            }
        bin_tab[lane] = a | (g.b * (tb - t0)) << 8;
    }
    if (warp == 0) {
        tmem_alloc(tmem_slot, g.tmem_cols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const uint64_t TO = g.timeout_ns;
    if (g.zero_mask && warp >= kCtrlWarps) {
        // blocks whose UMMAs always accumulate start zeroed
        const uint32_t quarter = g.tmem_cols >> 2;
        const uint32_t base =
            tmem + (static_cast<uint32_t>(32 * (warp & 3)) << 16) + ((warp - kCtrlWarps) >> 2) * quarter;
        for (uint32_t col = 0; col < quarter; col += 8) tmem_st8_zero(base + col);
        tmem_st_wait();
    }
    if (g.zero_mask) {
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
    }

    // everything above overlaps the end of the kernel before this one in the stream.  That
    // kernel writes the exponents, the norms and the slices: they are read below this line
    // only, by coherent loads, which the wait orders (a non-coherent load asks for data that
    // nothing writes while the kernel runs, and the wait need not order it)
    grid_wait_predecessor();
    if (threadIdx.x == 0 && *reinterpret_cast<volatile int *>(g.err) != 0) *vabort = 1;

    if (warp < kCtrlWarps) {
      regs_dec<kCtrlRegs>();
      if (warp == 0) {
        // ------------------------------------------------------ producer
        if (lane == 0) {
            // uses of the ring's entries (and of the B ring's) by this CTA over all of its tiles
            long long issued = 0, issued_b = 0;
            bool ok = true;
            // waits until the next entry of a ring may be refilled: its use r (>= 1) waits for
            // the entry's release r - 1
            auto acquire = [&](uint64_t *released, long long uses, int n) -> int {
                const long long r = uses / n;
                const int e = static_cast<int>(uses - r * n);
                const bool got = (r == 0) || mbar_wait(&released[e], static_cast<uint32_t>((r - 1) & 1), vabort, TO);
                if (!got && !*vabort) {
                    atomicCAS(g.err, 0, DEVERR_TIMEOUT_PRODUCER);
                    *vabort = 1;
                }
                return got ? e : -1;
            };
            for (int t = g.tile_begin + static_cast<int>(blockIdx.x); ok && t < g.total_tiles; t += gridDim.x) {
                TileRef tr;
                tile_ref(g, t, &tr);
                for (int c = tr.c0; ok && c < tr.c1; ++c) {
                    const uint8_t *a_src = tr.a_src + static_cast<size_t>(c) * g.a_block_bytes;
                    const uint8_t *b_src = tr.b_src + static_cast<size_t>(c) * g.b_block_bytes;
                    if (parts > 1) {
                        const int sb = *vabort ? -1 : acquire(emptyb, issued_b, kPartStagesB);
                        if (sb < 0) {
                            ok = false;
                            break;
                        }
                        mbar_arrive_expect_tx(&fullb[sb], g.b_block_bytes);
                        bulk_g2s(smem + b_base + static_cast<uint32_t>(sb) * b_stride, b_src, g.b_block_bytes, &fullb[sb]);
                        ++issued_b;
                    }
                    uint32_t left = g.a_block_bytes;
                    for (int i = 0; i < parts; ++i) {
                        const int st = *vabort ? -1 : acquire(empty, issued, g.stages);
                        if (st < 0) {
                            ok = false;
                            break;
                        }
                        uint8_t *dst = smem + static_cast<size_t>(st) * a_stride;
                        const uint32_t bytes = parts > 1 ? min(left, g.part_bytes) : left;
                        mbar_arrive_expect_tx(&full[st], bytes + (parts > 1 ? 0u : g.b_block_bytes));
                        bulk_g2s(dst, a_src, bytes, &full[st]);
                        if (parts == 1) bulk_g2s(dst + g.a_block_bytes, b_src, g.b_block_bytes, &full[st]);
                        a_src += bytes;
                        left -= bytes;
                        ++issued;
                    }
                }
            }
            // every copy issued must land before the CTA may exit
            const int zero = 0;
            for (long long u = issued > g.stages ? issued - g.stages : 0; u < issued; ++u)
                mbar_wait(&full[u % g.stages], static_cast<uint32_t>((u / g.stages) & 1), &zero, TO);
            for (long long u = issued_b > kPartStagesB ? issued_b - kPartStagesB : 0; u < issued_b; ++u)
                mbar_wait(&fullb[u % kPartStagesB], static_cast<uint32_t>((u / kPartStagesB) & 1), &zero, TO);
        }
      } else {
        // ---------------------------------------------------- MMA issuers
        // Up to three issuing warps (on different SM sub-partitions).  Each owns some of
        // the bin blocks and issues all of their UMMAs in order (blocks of zero_mask may be
        // shared, GemmArgs::blk_commits): the first after a drain overwrites the accumulator,
        // and a block that waits for its drain holds up its issuer alone, while the others go
        // on to the chunks that the stage ring holds.  What the warp executes per UMMA decides its rate
        // (it shares its scheduler with four drain warps): four entries at a time, so
        // that their loads and descriptor arithmetic overlap, run warp-wide with one
        // elected lane issuing (55 cycles a UMMA with nothing else on the SM, 77 in a
        // branch of lane 0; one entry at a time 190 to 230 in this kernel).
        const int iss = warp - 1;
        if (iss < n_iss) {
            constexpr int ksteps = KC >> 4;
            constexpr uint32_t sbo = KC * 16;
            // descriptors of stage 0's A and B; the address is in the low word, and
            // adding offsets never carries out of its 14 bits
            const uint32_t a0 = smem_u32(smem);
            const uint64_t ad0 = smem_desc(a0, 128, sbo), bd0 = smem_desc(a0 + b_base, 128, sbo);
            const uint32_t a_lo = static_cast<uint32_t>(ad0), b_lo = static_cast<uint32_t>(bd0);
            const uint64_t d_hi = ad0 & 0xFFFFFFFF00000000ull;
            const int list0 = iss ? g.op_end[iss - 1] : 0;
            int stb = 0;             // B ring
            uint32_t bparity = 0;
            uint32_t ephase = 0;   // parity of the gempty waits, bit 2 blk + buf
            uint32_t pend = 0;     // drains committed and not yet waited for, bit 2 blk + buf
            uint32_t bufm = 0;     // accumulator buffer each block writes now
            uint32_t fresh = ~0u;  // blocks whose next UMMA is the first after a drain
            int st = 0;
            uint32_t fparity = 0;
            bool ok = true;
            for (int t = g.tile_begin + static_cast<int>(blockIdx.x); ok && t < g.total_tiles; t += gridDim.x) {
                TileRef tr;
                tile_ref(g, t, &tr);
                DrainSchedule ds;
                ds.init(g, tr, lane);
                int step = ds.next(tr.c1 - tr.c0), till = step;  // chunks to the next drain
                for (int c = tr.c0; c < tr.c1; ++c) {
                    uint32_t cur = 0;
                    if (--till == 0) {
                        cur = ds.advance(step, lane, g.G);
                        if (c == tr.c1 - 1) cur = (1u << g.G) - 1u;
                        else till = step = ds.next(tr.c1 - 1 - c);
                    }
                    if (parts > 1 && !__all_sync(0xffffffffu, mbar_wait(&fullb[stb], bparity, vabort, TO))) {
                        ok = false;
                        break;
                    }
                    int r0 = list0;
                    for (int part = 0; part < parts; ++part) {
                    const int r1 = parts > 1 ? g.part_end[iss * kMaxParts + part] : g.op_end[iss];
                    if (!__all_sync(0xffffffffu, mbar_wait(&full[st], fparity, vabort, TO))) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t soff = (static_cast<uint32_t>(st) * a_stride) >> 4;
                    const uint32_t boff = (static_cast<uint32_t>(parts > 1 ? stb : st) * b_stride) >> 4;
                    for (int i = r0; i < r1;) {
                        // one block (of this part): its list ends where the first entry's count says
                        uint4 rc[4];
#pragma unroll
                        for (int x = 0; x < 4; ++x) rc[x] = recs[min(i + x, r1 - 1)];
                        const uint32_t blk = (rc[0].y >> 16) & 0xFu;
                        const int end = i + static_cast<int>(rc[0].y >> 24);
                        const uint32_t buf = (bufm >> blk) & 1u, ix = 2 * blk + buf;
                        // with parts, the block's first and last entries of the chunk are marked
                        const bool first = parts == 1 || (rc[0].y & 0x4000u), last = parts == 1 || (rc[0].y & 0x8000u);
                        if (first && ((pend >> ix) & 1u)) {
                            // the buffer's previous drain must have read it out
                            if (!__all_sync(0xffffffffu, mbar_wait(&gempty[ix], (ephase >> ix) & 1u, vabort, TO))) {
                                ok = false;
                                break;
                            }
                            ephase ^= 1u << ix;
                            pend &= ~(1u << ix);
                            tc_fence_after();
                        }
                        // a drained block's first UMMA spans the block and overwrites it
                        uint32_t acc0 = first ? ((fresh & ~g.zero_mask) >> blk & 1u) ^ 1u : 1u;
                        fresh &= ~(1u << blk);
                        while (true) {
                            if (elect_one()) {
#pragma unroll
                                for (int x = 0; x < 4; ++x) {
                                    const uint32_t d = tmem + (buf ? rc[x].x >> 16 : rc[x].x & 0xFFFFu);
                                    const uint64_t ad = d_hi | (a_lo + soff + (rc[x].y & 0x3FFFu));
                                    const uint64_t bd = d_hi | (b_lo + boff + rc[x].z);
                                    if (x == 0 || i + x < end) {
#pragma unroll
                                        for (int kk = 0; kk < ksteps; ++kk) {
                                            // one UMMA covers 32 bytes of K per row: 16 bf16 or 32 e4m3 values
                                            const uint32_t acc = x == 0 && kk == 0 ? acc0 : 1u;
                                            if constexpr (F8)
                                                umma_e4m3(d, ad + kk * 16, bd + kk * 16, rc[x].w, acc);
                                            else
                                                umma_bf16(d, ad + kk * 16, bd + kk * 16, rc[x].w, acc);
                                        }
                                    }
                                }
                            }
                            __syncwarp();
                            acc0 = 1u;
                            i = min(i + 4, end);
                            if (i == end) break;
#pragma unroll
                            for (int x = 0; x < 4; ++x) rc[x] = recs[min(i + x, r1 - 1)];
                        }
                        if (last && ((cur >> blk) & 1u)) {
                            if (elect_one()) umma_commit(&gfull[ix]);
                            __syncwarp();
                            pend |= 1u << ix;
                            bufm ^= g.dbl_mask & (1u << blk);
                            fresh |= 1u << blk;
                        }
                    }
                    if (!ok) break;
                    if (elect_one()) umma_commit(&empty[st]);
                    __syncwarp();
                    if (++st == g.stages) {
                        st = 0;
                        fparity ^= 1u;
                    }
                    r0 = r1;
                    }
                    if (!ok) break;
                    if (parts > 1) {
                        if (elect_one()) umma_commit(&emptyb[stb]);
                        __syncwarp();
                        if (++stb == kPartStagesB) {
                            stb = 0;
                            bparity ^= 1u;
                        }
                    }
                }
            }
            if (!ok && lane == 0 && !*vabort) {
                atomicCAS(g.err, 0, DEVERR_TIMEOUT_MMA);
                *vabort = 1;
            }
            // all MMAs issued by this warp complete before TMEM is released
            if (elect_one()) umma_commit(mma_done);
            __syncwarp();
            const int zero = 0;
            mbar_wait(mma_done, 0, &zero, TO);
        }
      }
      __syncwarp();
    } else {
        // ------------------------------------------ drain + epilogue warps
        regs_inc<kDrainRegs>();
        const int ew = warp - kCtrlWarps;
        const int qd = warp & 3;  // TMEM lane quadrant accessible to this warp
        const int part = ew >> 2;  // which COLS-wide column slice of the tile
        const uint32_t trow = tmem + (static_cast<uint32_t>(32 * qd) << 16) + static_cast<uint32_t>(part * COLS);

        long long acc[COLS][NA];
        // The first drain warp steps the drain schedule, waits for each drain's UMMAs (a
        // bounded wait) and passes the others a command through shared memory: x the
        // TMEM column of the buffer less lo BN, y = lo | hi << 8 | zero it << 16 | end of the
        // tile << 17 | gempty index << 20, or -1 when the wait gave up.  They wait at
        // a hardware barrier.  (Sixteen warps stepping the schedule and waiting on the
        // mbarrier took issue slots that the MMA-issuing warps of their schedulers
        // needed.)  One command slot per parity: a slot is written again only after
        // every warp has passed the barrier in between, so all of them leave at the
        // same command.
        uint32_t fphase = 0;  // parity of the gfull waits, bit 2 blk + buf
        uint32_t dbuf = 0;    // accumulator buffer each block's next drain reads
        uint32_t n_cmd = 0;
        bool ok = true;
        for (int t = g.tile_begin + static_cast<int>(blockIdx.x); ok && t < g.total_tiles; t += gridDim.x) {
#pragma unroll
            for (int i = 0; i < COLS; ++i)
#pragma unroll
                for (int a = 0; a < NA; ++a) acc[i][a] = 0;
            DrainSchedule ds;
            int left = 0;    // the first warp: chunks of the tile still to go
            uint32_t m = 0;  // and blocks still to drain at this point
            if (ew == 0) {
                TileRef tr;
                tile_ref(g, t, &tr);
                left = tr.c1 - tr.c0;
                ds.init(g, tr, lane);
            }
            for (bool end = false; !end;) {
                if (ew == 0) {
                    if (m == 0) {
                        const int step = ds.next(left);
                        left -= step;
                        m = ds.advance(step, lane, g.G);
                        if (left == 0) m = (1u << g.G) - 1u;
                    }
                    const int blk = __ffs(m) - 1;
                    m &= m - 1;
                    const int ix = 2 * blk + static_cast<int>((dbuf >> blk) & 1u);
                    const int blo = g.blk_lo[blk];
                    const int2 cmd = make_int2(
                        (ix & 1) ? g.blk_col1[blk] - blo * BN : 0,
                        blo | (blo + g.blk_nb[blk] - 1) << 8 | static_cast<int>((g.zero_mask >> blk) & 1u) << 16 |
                            (m == 0 && left == 0 ? 1 << 17 : 0) | ix << 20);
                    const bool got = mbar_wait(&gfull[ix], (fphase >> ix) & 1u, vabort, TO);
                    fphase ^= 1u << ix;
                    dbuf ^= g.dbl_mask & (1u << blk);
                    if (lane == 0) drain_cmd[n_cmd & 1] = got ? cmd : make_int2(0, -1);
                    tc_fence_before();
                }
                named_barrier<1, 32 * kEpiWarps>();
                tc_fence_after();
                const int2 cmd = drain_cmd[n_cmd++ & 1];
                if (cmd.y < 0) {
                    ok = false;
                    break;
                }
                end = ((cmd.y >> 17) & 1) != 0;
                const int lo = cmd.y & 0xFF, hi = (cmd.y >> 8) & 0xFF;
                const uint32_t bbase = trow + static_cast<uint32_t>(cmd.x);  // bin j at bbase + j BN
                // One bin at a time (several at once, for overlapped loads, cost more in
                // registers and code: 3.86 against 3.67 ms at 4096^3, s = 8, p + q <= 8); after
                // the last bin's load the buffer is free, so that its conversion overlaps the
                // block's next UMMAs.
#pragma unroll 1
                for (int j = lo; j <= hi; ++j) {
                    uint32_t v[COLS];
                    const uint32_t taddr = bbase + static_cast<uint32_t>(j * BN);
                    tmem_ld_cols<COLS>(taddr, v);
                    const int bt = bin_tab[j];
                    tmem_ld_wait();
                    if ((cmd.y >> 16) & 1) {
                        tmem_zero_cols<COLS>(taddr);
                        tmem_st_wait();
                    }
                    if (j == hi) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&gempty[cmd.y >> 20]);
                    }
#pragma unroll
                    for (int i = 0; i < COLS; ++i) reg_fence(v[i]);
                    acc_add_group<NA, COLS>(acc, v, bt & 0xFF, bt >> 8);
                }
            }
            if (!ok) break;

            TileRef tr;
            tile_ref(g, t, &tr);
            if (tr.split >= 0) {
                // a part of a split tile: add the exact group sums into the tile's
                // scratch (integer adds, exact in any order); the part that completes
                // the tile's count reads the totals and runs the epilogue
                unsigned long long *sa = g.split_acc + static_cast<size_t>(tr.split) * (NA * BN * BM);
                const int rl = 32 * qd + lane;
#pragma unroll
                for (int i = 0; i < COLS; ++i)
#pragma unroll
                    for (int a = 0; a < NA; ++a)
                        if (a < g.n_acc)
                            atomicAdd(sa + (static_cast<size_t>(a) * BN + part * COLS + i) * BM + rl,
                                      static_cast<unsigned long long>(acc[i][a]));
                __threadfence();
                named_barrier<1, 32 * kEpiWarps>();
                if (ew == 0 && lane == 0)
                    *split_flag = (atomicAdd(g.split_cnt + tr.split, 1) == g.split_parts - 1) ? 1 : 0;
                named_barrier<1, 32 * kEpiWarps>();
                if (!*reinterpret_cast<volatile int *>(split_flag)) continue;
                __threadfence();
                // the totals, leaving the scratch zero for the next launch
#pragma unroll
                for (int i = 0; i < COLS; ++i)
#pragma unroll
                    for (int a = 0; a < NA; ++a) {
                        acc[i][a] = 0;
                        if (a < g.n_acc) {
                            unsigned long long *ptr = sa + (static_cast<size_t>(a) * BN + part * COLS + i) * BM + rl;
                            acc[i][a] = static_cast<long long>(__ldcg(ptr));
                            __stcg(ptr, 0ull);
                        }
                    }
                if (ew == 0 && lane == 0) g.split_cnt[tr.split] = 0;
            }

            // --------------------------------------------------- epilogue
            // A rolled loop over pairs of columns: after each, the accumulators move down by
            // two registers' worth.  (Unrolled over the columns it is 30 to 40 KB of code that
            // a small product runs once, from a cold instruction cache: 22000 of the 46000
            // cycles of a 64^3 product.)
            const int row = tr.mt * BM + 32 * qd + lane;
            const bool row_ok = row < tr.M;
            const int col0 = tr.nt * BN + part * COLS;
            const int er = row_ok ? ld_after_wait(tr.er + row) : 0;
            const int e_base = er - 2044 - g.b * (g.J + 1);
            double *crow = tr.c + static_cast<size_t>(row) * tr.ldc;
            const bool plain = g.alpha == 1.0 && g.beta == 0.0;
            int B[kMaxAcc];
#pragma unroll
            for (int x = 0; x < kMaxAcc; ++x) B[x] = g.b * g.acc_t0[x];
            // the next pair's scale exponents are loaded a step ahead
            auto col_exp = [&](int col) { return col < tr.N ? ld_after_wait(tr.ec + col) : 0; };
            int e_next[2] = {col_exp(col0), col_exp(col0 + 1)};
#pragma unroll 1
            for (int i = 0; i < COLS; i += 2) {
                const int col = col0 + i;
                const int ec[2] = {e_next[0], e_next[1]};
                if (i + 2 < COLS) {
                    e_next[0] = col_exp(col + 2);
                    e_next[1] = col_exp(col + 3);
                }
                if (row_ok && col < tr.N) {
                    const bool two = col + 1 < tr.N;
                    if (g.out_mode == OUT_PAIRS || g.out_mode == OUT_RAW) {
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            if (u && !two) break;
                            const size_t at = static_cast<size_t>(row) * tr.N + col + u;
                            if (g.out_mode == OUT_PAIRS) {
                                // the reference's device output: lo, then hi with bits 51..62 = Er + Ec
                                long long *dst = reinterpret_cast<long long *>(g.raw) + at * 2;
                                unsigned long long hi = 0;
                                if constexpr (NA > 1)
                                    hi = g.n_acc > 1 ? static_cast<unsigned long long>(acc[u][1]) : 0ull;
                                const unsigned long long scale =
                                    static_cast<unsigned long long>(static_cast<uint32_t>(er + ec[u]));
                                dst[0] = acc[u][0];
                                dst[1] = static_cast<long long>((hi & 0x8007FFFFFFFFFFFFull) | ((scale & 0xFFFull) << 51));
                            } else {
                                // the exact sum modulo 2^128
                                unsigned __int128 q = 0;
#pragma unroll
                                for (int x = 0; x < NA; ++x)
                                    if (x < g.n_acc && B[x] < 128)
                                        q += static_cast<unsigned __int128>(static_cast<__int128>(acc[u][x])) << B[x];
                                int32_t *dst = g.raw + at * 4;
#pragma unroll
                                for (int w = 0; w < 4; ++w) dst[w] = static_cast<int32_t>(q >> (32 * w));
                            }
                        }
                    } else {
                        double v[2];
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            v[u] = __longlong_as_double(static_cast<long long>(
                                window_bits(acc_window<NA>(acc[u], g.n_acc, B), ec[u] + e_base, g.out_mode)));
                            // BLAS semantics: C is not read when beta == 0
                            if (!plain && (u == 0 || two))
                                v[u] = g.beta == 0.0 ? g.alpha * v[u] : fma(g.beta, crow[col + u], g.alpha * v[u]);
                        }
                        // one 16-byte store where aligned
                        if (two && (reinterpret_cast<uintptr_t>(crow + col) & 15) == 0) {
                            *reinterpret_cast<double2 *>(crow + col) = make_double2(v[0], v[1]);
                        } else {
                            crow[col] = v[0];
                            if (two) crow[col + 1] = v[1];
                        }
                    }
                }
#pragma unroll
                for (int k = 0; k + 2 < COLS; ++k)
#pragma unroll
                    for (int a = 0; a < NA; ++a) acc[k][a] = acc[k + 2][a];
            }
        }
        if (!ok && !*vabort) {
            atomicCAS(g.err, 0, DEVERR_TIMEOUT_EPI);
            *vabort = 1;
        }
    }

    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, g.tmem_cols);
    }
}

// Number of SMs of the current device (one persistent CTA each).
inline int device_sm_count() {
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (!cached[dev]) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        cached[dev] = n;
    }
    return cached[dev];
}

// F8: e4m3 slices (kind::f8f6f4); KC is then the bf16-equivalent chunk (bytes / 2
// per row and slice), i.e. half the K values the chunk holds.
template <int BN, int W, int KC, bool F8 = false>
void launch_gemm_variant(const GemmArgs &args, int tiles, size_t smem, void *stream) {
    auto kern = oz_gemm_kernel<BN, W, KC, F8>;
    // the shared-memory limit is raised once per device to the opt-in maximum (a
    // per-launch attribute call costs more than the launch itself; every caller
    // sets the same value, so two host threads that both make the first call only
    // repeat the same attribute call)
    static std::atomic<bool> raised[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    int threads = kThreads;
    if (dev < 0 || dev >= 64 || !raised[dev].load(std::memory_order_acquire)) {
        // a kernel built with fewer registers than its split hands out would wait for
        // them forever: refused here as an invalid launch
        cudaFuncAttributes fa{};
        if (cudaFuncGetAttributes(&fa, kern) != cudaSuccess || fa.numRegs < kLaunchRegs) threads = 0;
        int opt = 0;
        cudaDeviceGetAttribute(&opt, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             opt > static_cast<int>(smem) ? opt : static_cast<int>(smem));
        if (threads && dev >= 0 && dev < 64) raised[dev].store(true, std::memory_order_release);
    }
    const int range = args.total_tiles - args.tile_begin;
    const int grid = range < device_sm_count() ? range : device_sm_count();
    (void)tiles;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = args.pdl ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kern, args);
}

}  // namespace ozgb
