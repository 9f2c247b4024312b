// oz_split.cu -- stages (a) and (b): per-row / per-column maximum exponent and the
// error-free split of FP64 values into signed b-bit slices.
//
// Reference semantics (atlarge-research/ozAIE, src/aie_kernels/generic/ozaki_base.cc):
//   (a) ozaki_get_max_exponent_inner_tiled_wise_half_half  :342-440  (max of bits 52..62, start 0)
//   (b) extract_splits_acc64_half_half                     :449-639  (see split_value below)
// All work on the FP64 bit patterns is integer; FP64 arithmetic appears only in
// the optional sum of squares that the precision knob reads.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>

#include "oz_internal.h"
#include "oz_plan.h"
#include "oz_ptx.cuh"

namespace ozgb {

__device__ __forceinline__ int exp_field(double x) {
    return static_cast<int>((static_cast<unsigned long long>(__double_as_longlong(x)) >> 52) & 0x7FF);
}

// ------------------------------------------------------------- stage (a)
// One warp per row of A: max exponent field (and sum of squares when ss != null).
__device__ __forceinline__ void rowmax_body(const double *__restrict__ A, long lda, int M, int K, int32_t *__restrict__ er,
                         double *__restrict__ ss, int bx, int by) {
    const int warp = (bx * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= M) return;
    const double *row = A + static_cast<size_t>(warp) * lda;
    int e = 0;
    double s2 = 0.0;
#pragma unroll 8  // loads in flight: the loop is their latency
    for (int k = lane; k < K; k += 32) {
        const double x = __ldg(row + k);
        e = max(e, exp_field(x));
        if (ss) s2 = fma(x, x, s2);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
        if (ss) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    }
    if (lane == 0) {
        if (er) er[warp] = e;
        if (ss) ss[warp] = s2;
    }
}
__global__ void k_rowmax(const double *__restrict__ A, long lda, int M, int K, int32_t *__restrict__ er,
                         double *__restrict__ ss) {
    rowmax_body(A, lda, M, K, er, ss, blockIdx.x, blockIdx.y);
}

// One thread per column of B over a slab of rows; combined with atomicMax
// (ec must be zeroed first) and, when ss != null, atomicAdd of squares.
__device__ __forceinline__ void colmax_body(const double *__restrict__ B, long ldb, int K, int N, int rows_per_slab,
                         int32_t *__restrict__ ec, double *__restrict__ ss, int bx, int by) {
    const int n = bx * blockDim.x + threadIdx.x;
    if (n >= N) return;
    const int k0 = by * rows_per_slab;
    const int k1 = min(K, k0 + rows_per_slab);
    int e = 0;
    double s2 = 0.0;
#pragma unroll 8
    for (int k = k0; k < k1; ++k) {
        const double x = __ldg(B + static_cast<size_t>(k) * ldb + n);
        e = max(e, exp_field(x));
        if (ss) s2 = fma(x, x, s2);
    }
    if (ec) atomicMax(ec + n, e);
    if (ss) atomicAdd(ss + n, s2);
}
__global__ void k_colmax(const double *__restrict__ B, long ldb, int K, int N, int rows_per_slab,
                         int32_t *__restrict__ ec, double *__restrict__ ss) {
    colmax_body(B, ldb, K, N, rows_per_slab, ec, ss, blockIdx.x, blockIdx.y);
}

// ------------------------------------------------------------- stage (b)
// The reference's split of one double (ozaki_base.cc:497-628), restated:
//   bias = E - e (uint32), mantissa with implicit one for normal numbers only,
//   m64 = mant << 11 (MSB at bit 63), words w0..w3 selected by bias >= 32/64/96
//   (w3 not cleared for bias >= 128 when two 64-bit windows are used),
//   X = (w0:w1:w2:w3) >> (bias mod 32),
//   slice_i = sign * ((X >> (128 - b(i+1))) & (2^b - 1)).
struct SplitState {
    unsigned __int128 X;
    bool neg;
};

__device__ __forceinline__ SplitState split_value(double x, int E, bool two_windows) {
    const unsigned long long u = static_cast<unsigned long long>(__double_as_longlong(x));
    const uint32_t e = static_cast<uint32_t>((u >> 52) & 0x7FF);
    const unsigned long long mant = (u & ((1ull << 52) - 1)) | (e ? (1ull << 52) : 0ull);
    const uint32_t bias = static_cast<uint32_t>(E) - e;
    const unsigned long long m64 = mant << 11;
    const uint32_t vhi = static_cast<uint32_t>(m64 >> 32), vlo = static_cast<uint32_t>(m64);
    const uint32_t w0 = bias >= 32u ? 0u : vhi;
    const uint32_t w1 = bias >= 64u ? 0u : (bias >= 32u ? vhi : vlo);
    uint32_t w2 = 0, w3 = 0;
    if (two_windows) {
        w2 = bias >= 96u ? 0u : (bias >= 64u ? vhi : (bias >= 32u ? vlo : 0u));
        w3 = bias >= 96u ? vhi : (bias >= 64u ? vlo : 0u);
    }
    const unsigned __int128 W = (static_cast<unsigned __int128>((static_cast<unsigned long long>(w0) << 32) | w1)
                                 << 64) |
                                static_cast<unsigned __int128>((static_cast<unsigned long long>(w2) << 32) | w3);
    SplitState st;
    st.X = W >> (bias & 31u);
    st.neg = (u >> 63) != 0;
    return st;
}

// The split window as four 32-bit words, most significant first (w[4] = 0 so that
// a slice straddling two words is one funnel shift), and the bf16 sign bit.
__device__ __forceinline__ void split_words(const SplitState &st, uint32_t (&w)[5], uint32_t &sign) {
    w[0] = static_cast<uint32_t>(st.X >> 96);
    w[1] = static_cast<uint32_t>(st.X >> 64);
    w[2] = static_cast<uint32_t>(st.X >> 32);
    w[3] = static_cast<uint32_t>(st.X);
    w[4] = 0u;
    sign = st.neg ? 0x8000u : 0u;
}

// Slice p of an element as a signed float.
template <int B>
__device__ __forceinline__ uint32_t slice_digit(const uint32_t (&w)[5], int p) {
    const int pos = B * p;
    const int idx = pos >> 5, off = pos & 31;
    return __funnelshift_l(w[idx + 1], w[idx], off) >> (32 - B);
}
template <int B>
__device__ __forceinline__ float slice_float(const uint32_t (&w)[5], uint32_t sign, int p) {
    const float f = __uint_as_float(0x4B000000u | slice_digit<B>(w, p)) - 8388608.0f;
    return sign ? -f : f;
}
// Slice p of four elements as e4m3 bytes (element 0 in the lowest byte): every
// magnitude is < 16, so the conversion is exact.  Digits of up to 3 bits select their
// code from the eight of 0..7 by one byte permute; signs holds 0x80 in the bytes of
// negative elements.
template <int B>
__device__ __forceinline__ uint32_t slices_e4m3x4(const uint32_t (*w)[5], const uint32_t *sg, uint32_t signs, int p) {
    if constexpr (B <= 3) {
        const uint32_t sel = slice_digit<B>(w[0], p) | slice_digit<B>(w[1], p) << 4 | slice_digit<B>(w[2], p) << 8 |
                             slice_digit<B>(w[3], p) << 12;
        return __byte_perm(0x44403800u, 0x4E4C4A48u, sel) | signs;  // e4m3 of 0 1 2 3, 4 5 6 7
    }
    uint16_t lo, hi;
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;"
        : "=h"(lo)
        : "f"(slice_float<B>(w[1], sg[1], p)), "f"(slice_float<B>(w[0], sg[0], p)));
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;"
        : "=h"(hi)
        : "f"(slice_float<B>(w[3], sg[3], p)), "f"(slice_float<B>(w[2], sg[2], p)));
    return static_cast<uint32_t>(lo) | (static_cast<uint32_t>(hi) << 16);
}

// One-window split (s b within the first window, see split_two_windows): the
// slices are then the top s b bits of V = (mantissa << 11) >> bias (0 for
// bias >= 64), the same bits as split_value's 128-bit window, whose low 64 bits
// hold no slice.  V is kept as two words plus the element's sign in the two
// forms the bf16 conversion below uses.
struct FastElem {
    uint32_t hi, lo;  // V
    uint32_t sgnc;    // 0x4B000000 with the sign bit of x
    float cadd;       // -2^23 for x >= 0, +2^23 for x < 0
};
__device__ __forceinline__ FastElem fast_elem(double x, int E) {
    const unsigned long long u = static_cast<unsigned long long>(__double_as_longlong(x));
    const uint32_t e = static_cast<uint32_t>((u >> 52) & 0x7FF);
    const unsigned long long mant = (u & ((1ull << 52) - 1)) | (e ? (1ull << 52) : 0ull);
    const uint32_t bias = static_cast<uint32_t>(E) - e;
    const unsigned long long v = bias < 64u ? (mant << 11) >> bias : 0ull;
    const uint32_t neg = static_cast<uint32_t>(u >> 63);
    FastElem r;
    r.hi = static_cast<uint32_t>(v >> 32);
    r.lo = static_cast<uint32_t>(v);
    r.sgnc = 0x4B000000u | (neg << 31);
    r.cadd = neg ? 8388608.0f : -8388608.0f;
    return r;
}
// Slice p (B bits at bit B*p from the top of V) as a signed float: the FP32
// bits of +-(2^23 + v) plus -+2^23 give +-v exactly (and +0 for v = 0): one
// shift, one three-input logic operation and one add.
template <int B>
__device__ __forceinline__ float fast_slice(const FastElem &x, int p) {
    const int sh = 64 - B * (p + 1);  // V >> sh puts the slice in the low bits
    const uint32_t f = sh >= 32 ? (x.hi >> (sh - 32)) : __funnelshift_r(x.lo, x.hi, sh);
    return __uint_as_float((f & ((1u << B) - 1u)) | x.sgnc) + x.cadd;
}
// Two floats holding integers of magnitude < 256 as bf16 (exact): lo in bits 0..15.
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    uint32_t d;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}
// 16 bytes of bf16: 8 consecutive K values of one unit's slice.
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
    return make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]),
                      pack_bf16x2(f[6], f[7]));
}
__device__ __forceinline__ float sum_sq8(const float (&f)[8]) {
    float n = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) n = fmaf(f[i], f[i], n);
    return n;
}

__host__ __device__ inline bool split_two_windows(int b, int s) {
    const int avoid = 1 + (b == 3 ? 3 : 0);
    const int nv0 = 64 - avoid - ((64 - avoid) % b);
    return s * b > nv0;
}

// Slices of 8 consecutive K values x of one unit (row of A or column of B) with
// exponent E: one 16-byte piece per bf16 slice (8 bytes per e4m3 slice) at dst + p
// slice_elems.  one_window: !split_two_windows(B, s).  NORM: nrm[p] += the squares of
// slice p's values (exact: integers below 2^24).
template <int B, bool F8, bool NORM>
__device__ __forceinline__ void emit8(const double (&x)[8], int E, bool one_window, int s, size_t slice_elems,
                                      uint8_t *__restrict__ dst, float *nrm) {
    if (!F8 && one_window) {
        FastElem fe[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) fe[i] = fast_elem(x[i], E);
#pragma unroll
        for (int p = 0; p < 64 / B; ++p)
            if (p < s) {
                float f[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) f[i] = fast_slice<B>(fe[i], p);
                if constexpr (NORM) nrm[p] += sum_sq8(f);
                *reinterpret_cast<uint4 *>(dst + p * slice_elems * 2) = pack8(f);
            }
        return;
    }
    uint32_t w[8][5], sg[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) split_words(split_value(x[i], E, !one_window), w[i], sg[i]);
    uint32_t signs[2] = {0, 0};
#pragma unroll
    for (int i = 0; i < 8; ++i) signs[i >> 2] |= (sg[i] ? 0x80u : 0u) << (8 * (i & 3));
#pragma unroll
    for (int p = 0; p < (NORM ? kMaxNormSlices : 128 / B); ++p) {
        if (p < s) {
            if constexpr (F8) {
                uint2 v;
                v.x = slices_e4m3x4<B>(w, sg, signs[0], p);
                v.y = slices_e4m3x4<B>(w + 4, sg + 4, signs[1], p);
                *reinterpret_cast<uint2 *>(dst + p * slice_elems) = v;
            } else {
                uint32_t v[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float f0 = slice_float<B>(w[2 * i], sg[2 * i], p), f1 = slice_float<B>(w[2 * i + 1], sg[2 * i + 1], p);
                    if constexpr (NORM) nrm[p] = fmaf(f1, f1, fmaf(f0, f0, nrm[p]));
                    v[i] = pack_bf16x2(f0, f1);
                }
                *reinterpret_cast<uint4 *>(dst + p * slice_elems * 2) = make_uint4(v[0], v[1], v[2], v[3]);
            }
        }
    }
}

// The largest of the warp's chunk sums of squares per slice into the tile's maxima (bit
// patterns of non-negative floats order like integers): tiles t0 and, for lanes whose
// unit lies in the next tile, t0 + 1.  (By shuffles: with __reduce_max_sync here nvcc 13.0
// built a k_split_a, whose maxima pass through a loop, that lost those of two or three
// slices and left other registers' contents in their place.)
__device__ __forceinline__ void norm_max(const float *nrm, int s, float *__restrict__ out, int t0, int t) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int d = 0; d < 2; ++d) {
        if (!__any_sync(0xffffffffu, t == t0 + d)) continue;
        uint32_t mine = 0;
#pragma unroll
        for (int p = 0; p < kMaxNormSlices; ++p)
            if (p < s) {
                uint32_t v = t == t0 + d ? __float_as_uint(nrm[p]) : 0u;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
                if (lane == p) mine = v;
            }
        if (lane < s) {
            uint32_t *at = reinterpret_cast<uint32_t *>(out) + static_cast<size_t>(t0 + d) * s + lane;
            if (mine > __ldcg(at)) atomicMax(at, mine);
        }
    }
}

// Where the slices of unit u at K values k0 .. k0 + 7 go: blocks [u / TB][k0 / KC][p][TB x KC].
template <bool F8>
__device__ __forceinline__ uint8_t *slice_dst(uint16_t *tiles, int u, int k0, int TB, int KC, int n_kc, int s) {
    const int t = u / TB, r = u % TB, c = k0 / KC, kk = k0 % KC;
    const size_t at = (static_cast<size_t>(t) * n_kc + c) * s * (static_cast<size_t>(TB) * KC);
    return reinterpret_cast<uint8_t *>(tiles) +
           (F8 ? at + canon_offset8(r, kk, KC) : 2 * (at + canon_offset(r, kk, KC)));
}

// 8 consecutive doubles of a row, 0 from position n on; 128-bit loads where all are in
// range and aligned.
__device__ __forceinline__ void load8(const double *__restrict__ src, int n, double (&x)[8]) {
    if (n >= 8 && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const double2 d = __ldg(reinterpret_cast<const double2 *>(src) + i);
            x[2 * i] = d.x;
            x[2 * i + 1] = d.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = i < n ? __ldg(src + i) : 0.0;
    }
}

// A [M][K] row-major -> A slice blocks [mt][c][p][128 x KC].  One thread takes 8
// consecutive K values of one row and writes one 16-byte piece per slice; a warp
// covers 8 rows x 32 K (4 core matrices of each slice, 512 contiguous bytes).  NORM:
// the chunk's sums of squares are the sums over the lanes of a row (KC = 16 or 32); a
// block takes kNormSteps times as much of K, so that it merges its maxima once.
// WIN: windows of the split (split_two_windows), 0 for one or two by (B, s) at run time.
constexpr int kNormSteps = 4;
template <int B, bool F8 = false, bool NORM = false, int WIN = 0>
__device__ __forceinline__ void split_a_body(const double *__restrict__ A, long lda, int M, int K,
                                             const int32_t *__restrict__ er, int s, int KC, int n_kc, int Mp,
                                             uint16_t *__restrict__ tiles, int bx, int by, bool trans,
                                             float *__restrict__ norm = nullptr) {
    const int r8 = threadIdx.x & 7;
    const int kgl = threadIdx.x >> 3;  // 0..31
    const int m = by * 8 + r8;
    const int Kp = n_kc * KC;
    float top[NORM ? kMaxNormSlices : 1];
    if constexpr (NORM) {
#pragma unroll
        for (int p = 0; p < kMaxNormSlices; ++p) top[p] = 0.0f;
    }
    const int E = m < M ? er[m] : 0;
#pragma unroll 1
    for (int it = 0; it < (NORM ? kNormSteps : 1); ++it) {
        const int k0 = ((bx * (NORM ? kNormSteps : 1) + it) * 32 + kgl) * 8;
        float nrm[NORM ? kMaxNormSlices : 1];
        if constexpr (NORM) {
#pragma unroll
            for (int p = 0; p < kMaxNormSlices; ++p) nrm[p] = 0.0f;
        }
        if (m < Mp && k0 < Kp) {
            double x[8];
            if (!trans) {
                load8(A + static_cast<size_t>(m) * lda + k0, m < M ? K - k0 : 0, x);
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    x[i] = (m < M && k0 + i < K) ? __ldg(A + static_cast<size_t>(k0 + i) * lda + m) : 0.0;
            }
            emit8<B, F8, NORM>(x, E, WIN ? WIN == 1 : !split_two_windows(B, s), s, static_cast<size_t>(BM) * KC,
                               slice_dst<F8>(tiles, m, k0, BM, KC, n_kc, s), nrm);
        }
        if constexpr (NORM) {
            __syncwarp();
#pragma unroll
            for (int p = 0; p < kMaxNormSlices; ++p)
                if (p < s) {
                    nrm[p] += __shfl_xor_sync(0xffffffffu, nrm[p], 8);
                    if (KC == 32) nrm[p] += __shfl_xor_sync(0xffffffffu, nrm[p], 16);
                    top[p] = fmaxf(top[p], nrm[p]);
                }
        }
    }
    if constexpr (NORM) {
        if (by * 8 < Mp) norm_max(top, s, norm, (by * 8) / BM, (by * 8) / BM);
    }
}
template <int B, bool F8, bool NORM = false>
__global__ void k_split_a(const double *__restrict__ A, long lda, int M, int K, const int32_t *__restrict__ er,
                          int s, int KC, int n_kc, int Mp, uint16_t *__restrict__ tiles, int trans,
                          float *__restrict__ norm) {
    split_a_body<B, F8, NORM>(A, lda, M, K, er, s, KC, n_kc, Mp, tiles, blockIdx.x, blockIdx.y, trans != 0, norm);
}

// B [K][N] row-major -> slice blocks of B^T [nt][c][q][BN x KC].  One thread
// takes one column n and 8 consecutive K; a warp reads 32 consecutive columns
// per row (coalesced) and writes four 128-byte core matrices per slice.  NORM: one
// thread takes all KC (16 or 32) values of its column's chunk, 8 at a time, so that the
// chunk's sums of squares are its own.
template <int B, bool F8 = false, bool NORM = false, int WIN = 0>
__device__ __forceinline__ void split_b_body(const double *__restrict__ Bm, long ldb, int K, int N,
                                             const int32_t *__restrict__ ec, int s, int KC, int n_kc, int BN, int Np,
                                             uint16_t *__restrict__ tiles, int bx, int by, bool trans,
                                             float *__restrict__ norm = nullptr) {
    const int n = bx * 32 + (threadIdx.x & 31);
    const int groups = NORM ? KC >> 3 : 1;
    const int kw = (by * 8 + (threadIdx.x >> 5)) * 8 * groups;
    const int Kp = n_kc * KC;
    if (kw >= Kp) return;  // whole warps
    float nrm[NORM ? kMaxNormSlices : 1];
    if constexpr (NORM) {
#pragma unroll
        for (int p = 0; p < kMaxNormSlices; ++p) nrm[p] = 0.0f;
    }
    if (n < Np) {
        const int E = n < N ? ec[n] : 0;
#pragma unroll 1
        for (int k0 = kw; k0 < kw + 8 * groups; k0 += 8) {
            double x[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int k = k0 + i;
                x[i] = (n < N && k < K)
                           ? __ldg(trans ? Bm + static_cast<size_t>(n) * ldb + k : Bm + static_cast<size_t>(k) * ldb + n)
                           : 0.0;
            }
            emit8<B, F8, NORM>(x, E, WIN ? WIN == 1 : !split_two_windows(B, s), s, static_cast<size_t>(BN) * KC,
                               slice_dst<F8>(tiles, n, k0, BN, KC, n_kc, s), nrm);
        }
    }
    if constexpr (NORM) {
        __syncwarp();
        // 32 columns from a multiple of 32 on span at most two tiles
        const int t0 = (bx * 32) / BN;
        norm_max(nrm, s, norm, t0, n < Np ? n / BN : -1);
    }
}
template <int B, bool F8, bool NORM = false>
__global__ void k_split_b(const double *__restrict__ Bm, long ldb, int K, int N, const int32_t *__restrict__ ec,
                          int s, int KC, int n_kc, int BN, int Np, uint16_t *__restrict__ tiles, int trans,
                          float *__restrict__ norm) {
    grid_launch_dependents();
    split_b_body<B, F8, NORM>(Bm, ldb, K, N, ec, s, KC, n_kc, BN, Np, tiles, blockIdx.x, blockIdx.y, trans != 0, norm);
}

// ------------------------------------------- stages (a) and (b) in one launch
// For small operands without the precision knob: a block takes all of K of a few
// units, finds their exponents and splits them in a second pass over the same data
// (from L1 / L2).  One launch and no exponents to zero, instead of a memset and two
// launches.  Units that are rows of the stored operand (contiguous in K): 8 per block,
// a warp each for the exponent; columns of it: 16 per block, 128 contiguous bytes of a
// row per load.
struct ExpSplitJob {
    const double *X;
    long ld;
    int units, padded, K;  // padded: units rounded up to whole tiles
    int TB;                // units per tile
    int rows;              // units are rows of X (1) or columns (0)
    int32_t *e_out;
    uint16_t *tiles;
    float *norm;
};
template <int B, bool F8, bool NORM>
__device__ __forceinline__ void exp_split_body(const ExpSplitJob &j, int s, int KC, int n_kc, int bx) {
    const int Kp = n_kc * KC;
    const bool one = !split_two_windows(B, s);
    const size_t slice_elems = static_cast<size_t>(j.TB) * KC;
    if (j.rows) {
        __shared__ int sh_e[8];
        const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const int uw = bx * 8 + wid;
        int e = 0;
        if (uw < j.units) {
            const double *row = j.X + static_cast<size_t>(uw) * j.ld;
#pragma unroll 8
            for (int k = lane; k < j.K; k += 32) e = max(e, exp_field(__ldg(row + k)));
        }
        e = __reduce_max_sync(0xffffffffu, e);
        if (lane == 0) {
            sh_e[wid] = e;
            if (uw < j.units) j.e_out[uw] = e;
        }
        __syncthreads();
        const int r8 = threadIdx.x & 7, u = bx * 8 + r8;
        const int E = sh_e[r8];
        float top[NORM ? kMaxNormSlices : 1];
        if constexpr (NORM) {
#pragma unroll
            for (int p = 0; p < kMaxNormSlices; ++p) top[p] = 0.0f;
        }
        for (int kb = 0; kb < Kp; kb += 256) {
            const int k0 = kb + (threadIdx.x >> 3) * 8;
            float nrm[NORM ? kMaxNormSlices : 1];
            if constexpr (NORM) {
#pragma unroll
                for (int p = 0; p < kMaxNormSlices; ++p) nrm[p] = 0.0f;
            }
            if (k0 < Kp) {
                double x[8];
                load8(j.X + static_cast<size_t>(u) * j.ld + k0, u < j.units ? j.K - k0 : 0, x);
                emit8<B, F8, NORM>(x, E, one, s, slice_elems, slice_dst<F8>(j.tiles, u, k0, j.TB, KC, n_kc, s), nrm);
            }
            if constexpr (NORM) {
                __syncwarp();
#pragma unroll
                for (int p = 0; p < kMaxNormSlices; ++p)
                    if (p < s) {
                        nrm[p] += __shfl_xor_sync(0xffffffffu, nrm[p], 8);
                        if (KC == 32) nrm[p] += __shfl_xor_sync(0xffffffffu, nrm[p], 16);
                        top[p] = fmaxf(top[p], nrm[p]);
                    }
            }
        }
        if constexpr (NORM) norm_max(top, s, j.norm, bx * 8 / j.TB, bx * 8 / j.TB);
    } else {
        __shared__ int sh_c[16][17];
        const int c = threadIdx.x & 15, kl = threadIdx.x >> 4;
        const int u = bx * 16 + c;
        int e = 0;
        if (u < j.units) {
#pragma unroll 8
            for (int k = kl; k < j.K; k += 16) e = max(e, exp_field(__ldg(j.X + static_cast<size_t>(k) * j.ld + u)));
        }
        sh_c[kl][c] = e;
        __syncthreads();
        int E = 0;
#pragma unroll
        for (int r = 0; r < 16; ++r) E = max(E, sh_c[r][c]);
        if (kl == 0 && u < j.units) j.e_out[u] = E;
        // NORM: a warp holds 16 K values of each column at a time; a chunk of 32 is bounded
        // by twice the largest 16
        float top[NORM ? kMaxNormSlices : 1];
        if constexpr (NORM) {
#pragma unroll
            for (int p = 0; p < kMaxNormSlices; ++p) top[p] = 0.0f;
        }
        for (int kb = 0; kb < Kp; kb += 128) {
            const int k0 = kb + kl * 8;
            float nrm[NORM ? kMaxNormSlices : 1];
            if constexpr (NORM) {
#pragma unroll
                for (int p = 0; p < kMaxNormSlices; ++p) nrm[p] = 0.0f;
            }
            if (k0 < Kp) {
                double x[8];
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    x[i] = (u < j.units && k0 + i < j.K) ? __ldg(j.X + static_cast<size_t>(k0 + i) * j.ld + u) : 0.0;
                emit8<B, F8, NORM>(x, E, one, s, slice_elems, slice_dst<F8>(j.tiles, u, k0, j.TB, KC, n_kc, s), nrm);
            }
            if constexpr (NORM) {
                __syncwarp();
#pragma unroll
                for (int p = 0; p < kMaxNormSlices; ++p)
                    if (p < s) {
                        nrm[p] += __shfl_xor_sync(0xffffffffu, nrm[p], 16);
                        top[p] = fmaxf(top[p], KC == 32 ? 2.0f * nrm[p] : nrm[p]);
                    }
            }
        }
        if constexpr (NORM) norm_max(top, s, j.norm, bx * 16 / j.TB, bx * 16 / j.TB);
    }
}
// NORM: two blocks per SM (128 registers, 40 bytes spilled; 146 without the bound, whose
// one block per SM left the pass short of loads in flight: us a call, s = 8, 24000 x 64 x
// 1500 with p + q <= 8 557 -> 435, 128 x 24000 x 400 with B transposed 264 -> 202, 2304 x
// 2000 x 2000 516 -> 504).
template <int B, bool F8, bool NORM = false>
__global__ void __launch_bounds__(256, NORM ? 2 : 0) k_exp_split(const __grid_constant__ ExpSplitJob a,
                                                   const __grid_constant__ ExpSplitJob b, int n0, int s, int KC,
                                                   int n_kc) {
    grid_launch_dependents();
    const int bid = blockIdx.x;
    if (bid < n0) exp_split_body<B, F8, NORM>(a, s, KC, n_kc, bid);
    else exp_split_body<B, F8, NORM>(b, s, KC, n_kc, bid - n0);
}

// b (1..7) as a template argument: the slice positions become constants.
#define OZ_SPLIT_DISPATCH(b, CALL) \
    switch (b) {                   \
        case 1: CALL(1); break;    \
        case 2: CALL(2); break;    \
        case 3: CALL(3); break;    \
        case 4: CALL(4); break;    \
        case 5: CALL(5); break;    \
        case 6: CALL(6); break;    \
        default: CALL(7); break;   \
    }
// b <= 4 (the e4m3 carrier holds |v| <= 15 exactly)
#define OZ_SPLIT_DISPATCH_F8(b, CALL) \
    switch (b) {                      \
        case 1: CALL(1); break;       \
        case 2: CALL(2); break;       \
        case 3: CALL(3); break;       \
        default: CALL(4); break;      \
    }

// A kernel whose only wait is on an mbarrier that nothing arrives on: exercises
// the bounded-wait path (records DEVERR_TIMEOUT_SELFTEST and returns).
__global__ void k_selftest_timeout(int *err, unsigned long long timeout_ns) {
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const int zero = 0;
        if (!mbar_wait(&bar, 0, &zero, timeout_ns)) atomicCAS(err, 0, DEVERR_TIMEOUT_SELFTEST);
    }
}

// Block-wide reductions over blockDim.x threads (a multiple of 32, at most 1024).
__device__ int block_max_int(int v, int *sh) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    int m = sh[0];
    for (int w = 1; w < nw; ++w) m = max(m, sh[w]);
    return m;
}

__device__ double block_max_nonneg(double v, double *sh) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    double m = sh[0];
    for (int w = 1; w < nw; ++w) m = fmax(m, sh[w]);
    return m;
}

__device__ double block_sum(double v, double *sh) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    double s = 0.0;
    for (int w = 0; w < nw; ++w) s += sh[w];
    return s;
}

// Precision-knob statistics, all scaled by the largest row exponent ea of A and
// the largest column exponent eb of B so that they stay in range:
//   out[0] = sum_i 4^{Er_i-ea}           out[1] = sum_i |a_i|^2 4^{1022-ea}
//   out[2] = sum_j 4^{Ec_j-eb}           out[3] = sum_j |b_j|^2 4^{1022-eb}
//   out[4] = sum_k |A(:,k)|^2 |B(k,:)|^2 4^{2044-ea-eb}
// Block 0 makes the A terms, block 1 the B terms, block 2 the K-direction term.
// 2^e as an exact double for e in [-1022, 1023] (0 below: those terms are
// negligible in the knob's sums).
__device__ __forceinline__ double pow2i(int e) {
    if (e < -1022) return 0.0;
    return __longlong_as_double(static_cast<long long>(min(e, 1023) + 1023) << 52);
}
// x * 2^e for e in [-2046, 2046], as two exact power-of-two products.
__device__ __forceinline__ double scale2(double x, int e) {
    const int h = e / 2;
    return x * pow2i(h) * pow2i(e - h);
}

// ------------------------------------------------ FP32 scaled sums of squares
// 4^d as a float for d <= 0 (0 below the normal range).
__device__ __forceinline__ float pow4f(int d) { return d < -63 ? 0.0f : __int_as_float((127 + 2 * d) << 23); }

// (E, s) += the square of x: s is in units of 4^(E-1023), E the largest exponent
// field seen; x's own mantissa m in [1, 2) squared is added at 4^(e-E).
__device__ __forceinline__ void sq_add(int &E, float &s, double x) {
    const unsigned long long u = static_cast<unsigned long long>(__double_as_longlong(x));
    const int e = static_cast<int>((u >> 52) & 0x7FF);
    if (e == 0 || e == 0x7FF) return;  // zeros and subnormals (negligible); no infinities
    const float m = __uint_as_float(0x3F800000u | static_cast<uint32_t>((u >> 29) & 0x7FFFFF));
    if (e > E) {
        s *= pow4f(E - e);
        E = e;
    }
    s = fmaf(m * m, pow4f(e - E), s);
}
__device__ __forceinline__ void sq_merge(int &E, float &s, int E2, float s2) {
    const int Em = max(E, E2);
    s = s * pow4f(E - Em) + s2 * pow4f(E2 - Em);
    E = Em;
}
__device__ __forceinline__ unsigned long long sq_pack(int E, float s) {
    return (static_cast<unsigned long long>(static_cast<uint32_t>(E)) << 32) | __float_as_uint(s);
}

// (E, s) += m2 * 4^(e - 1023) for an element with exponent field e and squared
// mantissa m2 (0 for zeros, subnormals and non-finite values).
__device__ __forceinline__ void sq_add_em(int &E, float &s, int e, float m2) {
    if (e > E) {
        s *= pow4f(E - e);
        E = e;
    }
    s = fmaf(m2, pow4f(e - E), s);
}

// One 64-row x 256-column tile.  Lane l of each warp owns the 8 columns
// bx*256 + l + 32k (each load instruction of a warp reads 256 contiguous bytes)
// and warp w the rows w, w+8, ..., so a row is reduced by the
// warp's shuffles alone (no block barrier in the row loop); the 8 warps' column
// partials are merged once through shared memory at the end.
__device__ __forceinline__ void stats2d_body(const double *__restrict__ X, long ld, int rows, int cols,
                                             int32_t *__restrict__ row_e, int32_t *__restrict__ col_e,
                                             unsigned long long *__restrict__ row_part,
                                             unsigned long long *__restrict__ col_part, int bx, int by) {
    constexpr int NW = kStageThreads / 32;           // warps per block
    constexpr int CPL = kStatsCols / 32;             // columns per lane (8)
    static_assert(CPL == 8 && kStatsRows % NW == 0, "stats tile");
    __shared__ int shE[NW][kStatsCols];
    __shared__ float shS[NW][kStatsCols];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int c0 = bx * kStatsCols + lane;            // this lane's first column; then every 32nd
    const int r0 = by * kStatsRows;
    const bool rows_wanted = row_e || row_part;
    const int nbx = (cols + kStatsCols - 1) / kStatsCols;
    int Ec[CPL];
    float sc[CPL];
#pragma unroll
    for (int k = 0; k < CPL; ++k) {
        Ec[k] = 0;
        sc[k] = 0.0f;
    }
    auto load_row = [&](int r, double (&x)[CPL]) {
#pragma unroll
        for (int k = 0; k < CPL; ++k)
            x[k] = (r < rows && c0 + 32 * k < cols) ? __ldg(X + static_cast<size_t>(r) * ld + c0 + 32 * k) : 0.0;
    };
    // the next row's loads are issued before this row is reduced
    double x[CPL], xn[CPL];
    if (wid < kStatsRows) load_row(r0 + wid, xn);
    for (int i = wid; i < kStatsRows; i += NW) {
        const int r = r0 + i;
#pragma unroll
        for (int k = 0; k < CPL; ++k) x[k] = xn[k];
        if (i + NW < kStatsRows) load_row(r + NW, xn);
        int ex[CPL];
        uint32_t mb[CPL];  // FP32 mantissa bits of each element; 0 for zeros, subnormals, non-finite
        int Er = 0;
#pragma unroll
        for (int k = 0; k < CPL; ++k) {
            const unsigned long long bits = static_cast<unsigned long long>(__double_as_longlong(x[k]));
            ex[k] = static_cast<int>((bits >> 52) & 0x7FF);
            mb[k] = (ex[k] != 0 && ex[k] != 0x7FF) ? (0x800000u | static_cast<uint32_t>((bits >> 29) & 0x7FFFFF)) : 0u;
            Er = max(Er, ex[k]);
        }
        // columns: running exponent per column, rescaled only when a larger one
        // appears (rare after the first rows); x scaled by 2^(-Ec) squared by one FMA
#pragma unroll
        for (int k = 0; k < CPL; ++k) {
            if (ex[k] > Ec[k]) {
                sc[k] *= pow4f(Ec[k] - ex[k]);
                Ec[k] = ex[k];
            }
            const int d = ex[k] - Ec[k];
            const float xs = (mb[k] && d >= -63) ? __uint_as_float((static_cast<uint32_t>(d + 127) << 23) |
                                                                   (mb[k] & 0x7FFFFFu))
                                                 : 0.0f;
            sc[k] = fmaf(xs, xs, sc[k]);
        }
        if (rows_wanted) {
            // rows: one exponent for the whole row (the warp's maximum), then plain sums
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) Er = max(Er, __shfl_xor_sync(0xffffffffu, Er, o));
            float sr = 0.0f;
#pragma unroll
            for (int k = 0; k < CPL; ++k) {
                const int d = ex[k] - Er;
                const float xs = (mb[k] && d >= -63) ? __uint_as_float((static_cast<uint32_t>(d + 127) << 23) |
                                                                       (mb[k] & 0x7FFFFFu))
                                                     : 0.0f;
                sr = fmaf(xs, xs, sr);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sr += __shfl_xor_sync(0xffffffffu, sr, o);
            if (lane == 0 && r < rows) {
                if (row_part) row_part[static_cast<size_t>(r) * nbx + bx] = sq_pack(Er, sr);
                if (row_e) atomicMax(row_e + r, Er);
            }
        }
    }
    // columns: merge the warps' partials
#pragma unroll
    for (int k = 0; k < CPL; ++k) {
        shE[wid][lane + 32 * k] = Ec[k];
        shS[wid][lane + 32 * k] = sc[k];
    }
    __syncthreads();
    const int c = bx * kStatsCols + static_cast<int>(threadIdx.x);
    if (c < cols) {
        int E = 0;
        float sv = 0.0f;
#pragma unroll
        for (int w = 0; w < NW; ++w) sq_merge(E, sv, shE[w][threadIdx.x], shS[w][threadIdx.x]);
        if (col_part) col_part[static_cast<size_t>(by) * cols + c] = sq_pack(E, sv);
        if (col_e) atomicMax(col_e + c, E);
    }
}


// Combined (E, s) of unit u, by one warp: lanes load the unit's partials in
// parallel and merge them; every lane returns the result.
__device__ __forceinline__ void unit_sq_warp(const StatParts &sp, int u, int lane, int *E, float *s) {
    int e = 0;
    float v = 0.0f;
    const unsigned long long *p = sp.p + u * sp.unit_stride;
    for (int i = lane; i < sp.nparts; i += 32) {
        const unsigned long long w = __ldg(p + i * sp.part_stride);
        sq_merge(e, v, static_cast<int>(w >> 32), __uint_as_float(static_cast<uint32_t>(w)));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const int e2 = __shfl_xor_sync(0xffffffffu, e, o);
        const float v2 = __shfl_xor_sync(0xffffffffu, v, o);
        sq_merge(e, v, e2, v2);
    }
    *E = e;
    *s = v;
}

// Combined (E, s) of unit u by one thread, for units with few partials: the
// loads of many units are in flight at once instead of one unit per warp.
__device__ __forceinline__ void unit_sq_thread(const StatParts &sp, int u, int *E, float *s) {
    int e = 0;
    float v = 0.0f;
    const unsigned long long *p = sp.p + u * sp.unit_stride;
#pragma unroll 4
    for (int i = 0; i < sp.nparts; ++i) {
        const unsigned long long w = __ldg(p + i * sp.part_stride);
        sq_merge(e, v, static_cast<int>(w >> 32), __uint_as_float(static_cast<uint32_t>(w)));
    }
    *E = e;
    *s = v;
}

// Part `chunk` of `chunks` of one of the three knob sums (role 0: A terms, 1: B
// terms, 2: the k-direction term), added atomically into j.out (zeroed before);
// one warp per unit.  With ea, eb the largest row / column exponents of op(A) /
// op(B):
//   sa = sum_r 4^(Er - ea), na = sum_r |a_r|^2 4^(1022 - ea), likewise for B,
//   t  = sum_k |op(A)(:,k)|^2 |op(B)(k,:)|^2 4^(2044 - ea - eb),
// and for the elementwise criterion ia = max_r 1 / (|a_r|^2 4^(1022 - Er)) over
// the non-zero rows (ib likewise over the columns of op(B)), combined by an
// integer max of the bit patterns (order-preserving for non-negative doubles).
__device__ __forceinline__ void knob_stats_body(const KnobJob &j, const int role, const int chunk, const int chunks) {
    __shared__ int sh_i[32];
    __shared__ double sh_d[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    // every block finds the largest exponents for itself, eight loads in flight per thread
    auto largest = [&](const int32_t *e, int n) {
        int m = 0;
#pragma unroll 8
        for (int i = threadIdx.x; i < n; i += blockDim.x) m = max(m, __ldg(e + i));
        return block_max_int(m, sh_i);
    };
    const int ea = role != 1 ? largest(j.er, j.M) : 0;
    const int eb = role != 0 ? largest(j.ec, j.N) : 0;
    const int n = role == 0 ? j.M : (role == 1 ? j.N : j.K);
    const int per = (n + chunks - 1) / chunks;
    const int i0 = chunk * per, i1 = min(n, i0 + per);
    double num = 0.0, den = 0.0, t = 0.0, inv = 0.0;
    // 1 / (|x_u|^2 4^(1022 - E_u)) of a unit whose squares sum to sq 4^(E - 1023)
    auto flat_inv = [](float sq, int E, int Eu) {
        return sq > 0.0f ? scale2(1.0 / static_cast<double>(sq), 2 * (Eu + 1 - E)) : 0.0;
    };
    const int nparts = role == 0 ? j.ra.nparts : (role == 1 ? j.cb.nparts : max(j.ka.nparts, j.kb.nparts));
    if (nparts <= 32) {
        // one thread per unit
        for (int u = i0 + static_cast<int>(threadIdx.x); u < i1; u += blockDim.x) {
            if (role < 2) {
                const StatParts &sp = role == 0 ? j.ra : j.cb;
                const int emax = role == 0 ? ea : eb;
                int E;
                float sq;
                unit_sq_thread(sp, u, &E, &sq);
                const int Eu = role == 0 ? j.er[u] : j.ec[u];
                num += pow2i(2 * (Eu - emax));
                den += scale2(static_cast<double>(sq), 2 * (E - emax) - 2);
                inv = fmax(inv, flat_inv(sq, E, Eu));
            } else {
                int E1, E2;
                float s1, s2;
                unit_sq_thread(j.ka, u, &E1, &s1);
                unit_sq_thread(j.kb, u, &E2, &s2);
                t += scale2(static_cast<double>(s1) * s2, 2 * (E1 + E2 - ea - eb - 2));
            }
        }
    } else {
        // one warp per unit
        for (int u = i0 + wid; u < i1; u += nw) {
            if (role < 2) {
                const StatParts &sp = role == 0 ? j.ra : j.cb;
                const int emax = role == 0 ? ea : eb;
                int E;
                float sq;
                unit_sq_warp(sp, u, lane, &E, &sq);
                if (lane == 0) {
                    const int Eu = role == 0 ? j.er[u] : j.ec[u];
                    num += pow2i(2 * (Eu - emax));
                    den += scale2(static_cast<double>(sq), 2 * (E - emax) - 2);
                    inv = fmax(inv, flat_inv(sq, E, Eu));
                }
            } else {
                int E1, E2;
                float s1, s2;
                unit_sq_warp(j.ka, u, lane, &E1, &s1);
                unit_sq_warp(j.kb, u, lane, &E2, &s2);
                if (lane == 0) t += scale2(static_cast<double>(s1) * s2, 2 * (E1 + E2 - ea - eb - 2));
            }
        }
    }
    if (role < 2) {
        num = block_sum(num, sh_d);
        den = block_sum(den, sh_d);
        inv = block_max_nonneg(inv, sh_d);
        if (threadIdx.x == 0) {
            atomicAdd(j.out + 2 * role, num);
            atomicAdd(j.out + 2 * role + 1, den);
            if (inv > 0.0)
                atomicMax(reinterpret_cast<unsigned long long *>(j.out + 5 + role),
                          static_cast<unsigned long long>(__double_as_longlong(inv)));
        }
    } else {
        t = block_sum(t, sh_d);
        if (threadIdx.x == 0) atomicAdd(j.out + 4, t);
    }
}

__global__ void k_knob_stats(const KnobJob j) { knob_stats_body(j, blockIdx.x % 3, blockIdx.x / 3, gridDim.x / 3); }

// Grouped knob reduction: blocks 3p, 3p+1, 3p+2 reduce problem p.
__global__ void k_knob_grouped(const KnobJob *__restrict__ jobs) {
    const KnobJob j = jobs[blockIdx.x / 3];
    knob_stats_body(j, blockIdx.x % 3, 0, 1);
}

// One stage job on its local block index (the per-problem kernels' bodies).
// TRANS: the kernel also serves transposed splits; STAGE: 1 the jobs of stage (a), 2
// those of stage (b); WIN: 1 splits of one window (bf16), 2 the others, 0 all of them.  (A
// kernel of fewer bodies keeps its registers down and its blocks per SM up.)
template <bool TRANS, int STAGE, int WIN = 0>
__device__ __forceinline__ void run_stage_job(const StageJob &j, int local) {
    const int bx = local % j.gx, by = local / j.gx;
    const bool tr = TRANS && j.trans != 0;
    if constexpr (STAGE == 1) {
        if (j.kind == JOB_ROWMAX) rowmax_body(j.X, j.ld, j.rows, j.cols, j.e_out, j.ss_out, bx, by);
        else if (j.kind == JOB_COLMAX) colmax_body(j.X, j.ld, j.rows, j.cols, 64, j.e_out, j.ss_out, bx, by);
        else stats2d_body(j.X, j.ld, j.rows, j.cols, j.e_out, j.e_out2, j.prow, j.pcol, bx, by);
        return;
    }
    switch (j.kind) {
        // the transpose flag as a constant at each call site: a runtime flag would
        // compile both load paths into every split (measured 20 % slower)
        case JOB_SPLIT_A: {
#define OZ_JOB_A(BB, T) \
    split_a_body<BB, false, false, WIN>(j.X, j.ld, j.rows, j.cols, j.e_in, j.s, j.KC, j.n_kc, j.padded, j.tiles, bx, by, T)
#define OZ_JOB_A8(BB, T) \
    split_a_body<BB, true, false, WIN>(j.X, j.ld, j.rows, j.cols, j.e_in, j.s, j.KC, j.n_kc, j.padded, j.tiles, bx, by, T)
#define OZ_JOB_AN(BB) OZ_JOB_A(BB, false)
#define OZ_JOB_AT(BB) OZ_JOB_A(BB, true)
#define OZ_JOB_A8N(BB) OZ_JOB_A8(BB, false)
#define OZ_JOB_A8T(BB) OZ_JOB_A8(BB, true)
            if (WIN != 1 && j.f8) {
                if (tr) {
                    OZ_SPLIT_DISPATCH_F8(j.b, OZ_JOB_A8T)
                } else {
                    OZ_SPLIT_DISPATCH_F8(j.b, OZ_JOB_A8N)
                }
            } else {
                if (tr) {
                    OZ_SPLIT_DISPATCH(j.b, OZ_JOB_AT)
                } else {
                    OZ_SPLIT_DISPATCH(j.b, OZ_JOB_AN)
                }
            }
#undef OZ_JOB_A
#undef OZ_JOB_A8
#undef OZ_JOB_AN
#undef OZ_JOB_AT
#undef OZ_JOB_A8N
#undef OZ_JOB_A8T
            break;
        }
        default: {
#define OZ_JOB_B(BB, T) \
    split_b_body<BB, false, false, WIN>(j.X, j.ld, j.rows, j.cols, j.e_in, j.s, j.KC, j.n_kc, j.BN, j.padded, j.tiles, bx, by, T)
#define OZ_JOB_B8(BB, T) \
    split_b_body<BB, true, false, WIN>(j.X, j.ld, j.rows, j.cols, j.e_in, j.s, j.KC, j.n_kc, j.BN, j.padded, j.tiles, bx, by, T)
#define OZ_JOB_BN(BB) OZ_JOB_B(BB, false)
#define OZ_JOB_BT(BB) OZ_JOB_B(BB, true)
#define OZ_JOB_B8N(BB) OZ_JOB_B8(BB, false)
#define OZ_JOB_B8T(BB) OZ_JOB_B8(BB, true)
            if (WIN != 1 && j.f8) {
                if (tr) {
                    OZ_SPLIT_DISPATCH_F8(j.b, OZ_JOB_B8T)
                } else {
                    OZ_SPLIT_DISPATCH_F8(j.b, OZ_JOB_B8N)
                }
            } else {
                if (tr) {
                    OZ_SPLIT_DISPATCH(j.b, OZ_JOB_BT)
                } else {
                    OZ_SPLIT_DISPATCH(j.b, OZ_JOB_BN)
                }
            }
#undef OZ_JOB_B
#undef OZ_JOB_B8
#undef OZ_JOB_BN
#undef OZ_JOB_BT
#undef OZ_JOB_B8N
#undef OZ_JOB_B8T
            break;
        }
    }
}

// Persistent: block b runs work blocks b, b + gridDim.x, ... of the job list; the
// job of a work block is found by a forward scan from the previous one (work
// blocks only increase), so no block pays a search over all jobs, and a grouped
// call of many small problems does not launch one block per 2048 elements.
template <int STAGE>
__global__ void __launch_bounds__(kStageThreads, 3)
    k_stage_jobs(const StageJob *__restrict__ jobs, const int *__restrict__ block0, int n_jobs) {
    const int total = __ldg(block0 + n_jobs);
    int j = 0;
    for (int bid = blockIdx.x; bid < total; bid += gridDim.x) {
        while (j + 1 < n_jobs && __ldg(block0 + j + 1) <= bid) ++j;
        run_stage_job<false, STAGE>(jobs[j], bid - __ldg(block0 + j));
        // the statistics job's shared memory is written again by the next work block
        __syncthreads();
    }
}

// Two jobs of one problem and stage (A and B) in one launch: blocks [0, n0) run j0.  A
// kernel for each stage and, of stage (b), for splits of one window and the others, three
// blocks per SM each (one kernel of all bodies took 88 registers and two blocks).
template <int STAGE, int WIN>
__global__ void __launch_bounds__(kStageThreads, 3)
    k_stage_pair(const __grid_constant__ StageJob j0, const __grid_constant__ StageJob j1, int n0) {
    grid_launch_dependents();
    const int bid = blockIdx.x;
    if (bid < n0) run_stage_job<true, STAGE, WIN>(j0, bid);
    else run_stage_job<true, STAGE, WIN>(j1, bid - n0);
}

// Pseudo-random doubles in [-1, 1) (splitmix64 of the index): inputs for the
// autotuner's timing runs, whose speed does not depend on the values.
__global__ void k_fill_random(double *__restrict__ x, size_t n, unsigned long long seed) {
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (i + 1);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        x[i] = static_cast<double>(z >> 11) * 0x1.0p-52 - 1.0;
    }
}

void launch_fill_random(double *x, size_t n, unsigned long long seed, void *stream) {
    if (n) k_fill_random<<<4 * 152, 256, 0, static_cast<cudaStream_t>(stream)>>>(x, n, seed);
}

// C = beta * C over an M x N block with leading dimension ldc (beta == 0 writes
// zeros without reading C, as BLAS does).
__global__ void k_scale(double *__restrict__ C, long ldc, int M, int N, double beta) {
    const size_t total = static_cast<size_t>(M) * N;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        double *c = C + (i / N) * ldc + (i % N);
        *c = beta == 0.0 ? 0.0 : beta * *c;
    }
}

void launch_scale(double *C, long ldc, int M, int N, double beta, void *stream) {
    k_scale<<<4 * 152, 256, 0, static_cast<cudaStream_t>(stream)>>>(C, ldc, M, N, beta);
}

void stage_grid(const StageJob &j, int *gx, int *gy) {
    switch (j.kind) {
        case JOB_ROWMAX:
            *gx = (j.rows * 32 + kStageThreads - 1) / kStageThreads;
            *gy = 1;
            break;
        case JOB_COLMAX:
            *gx = (j.cols + kStageThreads - 1) / kStageThreads;
            *gy = (j.rows + 63) / 64;
            break;
        case JOB_STATS:
            *gx = (j.cols + kStatsCols - 1) / kStatsCols;
            *gy = (j.rows + kStatsRows - 1) / kStatsRows;
            break;
        case JOB_SPLIT_A:
            *gx = (j.n_kc * j.KC / 8 + 31) / 32;
            *gy = j.padded / 8;
            break;
        default:
            *gx = (j.padded + 31) / 32;
            *gy = (j.n_kc * j.KC / 8 + 7) / 8;
            break;
    }
}

void launch_stage_pair(StageJob j0, StageJob j1, void *stream) {
    stage_grid(j0, &j0.gx, &j0.gy);
    stage_grid(j1, &j1.gx, &j1.gy);
    const int n0 = j0.gx * j0.gy, n1 = j1.gx * j1.gy;
    if (n0 + n1 <= 0) return;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (j0.kind != JOB_SPLIT_A && j0.kind != JOB_SPLIT_B)
        k_stage_pair<1, 0><<<n0 + n1, kStageThreads, 0, st>>>(j0, j1, n0);
    else if (!j0.f8 && !split_two_windows(j0.b, j0.s))
        k_stage_pair<2, 1><<<n0 + n1, kStageThreads, 0, st>>>(j0, j1, n0);
    else
        k_stage_pair<2, 2><<<n0 + n1, kStageThreads, 0, st>>>(j0, j1, n0);
}

template <int STAGE>
void launch_stage_jobs_of(const StageJob *jobs, const int *block0, int n_jobs, int total_blocks, void *stream) {
    // resident blocks of the kernel on the current device, found once per device
    static std::atomic<int> resident[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    int grid = 0;
    if (dev >= 0 && dev < 64) grid = resident[dev].load(std::memory_order_relaxed);
    if (grid <= 0) {
        int sms = 0, per_sm = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_stage_jobs<STAGE>, kStageThreads, 0) != cudaSuccess ||
            per_sm <= 0)
            per_sm = 2;
        cudaGetLastError();
        grid = sms * per_sm;
        if (dev >= 0 && dev < 64) resident[dev].store(grid, std::memory_order_relaxed);
    }
    k_stage_jobs<STAGE><<<std::min(grid, total_blocks), kStageThreads, 0, static_cast<cudaStream_t>(stream)>>>(
        jobs, block0, n_jobs);
}

void launch_stage_jobs(int stage, const StageJob *jobs, const int *block0, int n_jobs, int total_blocks,
                       void *stream) {
    if (total_blocks <= 0) return;
    if (stage == 1) launch_stage_jobs_of<1>(jobs, block0, n_jobs, total_blocks, stream);
    else launch_stage_jobs_of<2>(jobs, block0, n_jobs, total_blocks, stream);
}

void launch_knob_grouped(const KnobJob *jobs, int n, void *stream) {
    if (n > 0) k_knob_grouped<<<3 * n, 256, 0, static_cast<cudaStream_t>(stream)>>>(jobs);
}

void launch_knob_stats(const KnobJob &j, void *stream) {
    // each of the three sums split over blocks of 8 warps, about 64 units per block (8 to
    // 32 units measured no faster: 113 to 115 us per 1024^3 call, 2.71 to 2.73 ms at 4096^3)
    const int chunks = std::max(1, std::min(1024, std::max(j.M, std::max(j.N, j.K)) / 64));
    cudaMemsetAsync(j.out, 0, sizeof(KnobStats), static_cast<cudaStream_t>(stream));
    k_knob_stats<<<3 * chunks, 256, 0, static_cast<cudaStream_t>(stream)>>>(j);
}

void launch_rowmax(const double *A, long lda, int M, int K, int32_t *er, double *ss, void *stream) {
    const int threads = 256;
    const int blocks = (M * 32 + threads - 1) / threads;
    k_rowmax<<<blocks, threads, 0, static_cast<cudaStream_t>(stream)>>>(A, lda, M, K, er, ss);
}

void launch_colmax(const double *B, long ldb, int K, int N, int32_t *ec, double *ss, void *stream) {
    const int threads = 256;
    const int rows = 64;
    dim3 grid((N + threads - 1) / threads, (K + rows - 1) / rows);
    k_colmax<<<grid, threads, 0, static_cast<cudaStream_t>(stream)>>>(B, ldb, K, N, rows, ec, ss);
}

void launch_exp_split(const double *A, long lda, bool ta, int M, int Mp, int32_t *er, uint16_t *at, const double *B,
                      long ldb, bool tb, int N, int Np, int BN, int32_t *ec, uint16_t *bt, int K, int b, int s, int KC,
                      int n_kc, bool f8, void *stream, float *norm_a, float *norm_b) {
    const ExpSplitJob ja{A, lda, M, Mp, K, BM, ta ? 0 : 1, er, at, norm_a};
    const ExpSplitJob jb{B, ldb, N, Np, K, BN, tb ? 1 : 0, ec, bt, norm_b};
    const int n0 = Mp / (ja.rows ? 8 : 16), n1 = Np / (jb.rows ? 8 : 16);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
#define OZ_CALL_ES(BB) k_exp_split<BB, false><<<n0 + n1, 256, 0, st>>>(ja, jb, n0, s, KC, n_kc)
#define OZ_CALL_ES8(BB) k_exp_split<BB, true><<<n0 + n1, 256, 0, st>>>(ja, jb, n0, s, KC, n_kc)
    if (norm_a) {
        k_exp_split<7, false, true><<<n0 + n1, 256, 0, st>>>(ja, jb, n0, s, KC, n_kc);
    } else if (f8) {
        OZ_SPLIT_DISPATCH_F8(b, OZ_CALL_ES8)
    } else {
        OZ_SPLIT_DISPATCH(b, OZ_CALL_ES)
    }
#undef OZ_CALL_ES
#undef OZ_CALL_ES8
}

void launch_split_a(const double *A, long lda, int M, int K, const int32_t *er, int b, int s, int KC, int n_kc,
                    int Mp, uint16_t *tiles, void *stream, bool trans, bool f8, float *norm) {
    const int Kp = n_kc * KC;
    dim3 grid((Kp / 8 + 31) / 32, Mp / 8);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
#define OZ_CALL_A(BB) k_split_a<BB, false><<<grid, 256, 0, st>>>(A, lda, M, K, er, s, KC, n_kc, Mp, tiles, trans ? 1 : 0, nullptr)
#define OZ_CALL_A8(BB) k_split_a<BB, true><<<grid, 256, 0, st>>>(A, lda, M, K, er, s, KC, n_kc, Mp, tiles, trans ? 1 : 0, nullptr)
    if (norm) {
        grid.x = (grid.x + kNormSteps - 1) / kNormSteps;
        k_split_a<7, false, true><<<grid, 256, 0, st>>>(A, lda, M, K, er, s, KC, n_kc, Mp, tiles, trans ? 1 : 0, norm);
    } else if (f8) {
        OZ_SPLIT_DISPATCH_F8(b, OZ_CALL_A8)
    } else {
        OZ_SPLIT_DISPATCH(b, OZ_CALL_A)
    }
#undef OZ_CALL_A
#undef OZ_CALL_A8
}

void launch_split_b(const double *B, long ldb, int K, int N, const int32_t *ec, int b, int s, int KC, int n_kc,
                    int BN, int Np, uint16_t *tiles, void *stream, bool trans, bool f8, float *norm) {
    const int Kp = n_kc * KC;
    dim3 grid((Np + 31) / 32, norm ? (n_kc + 7) / 8 : (Kp / 8 + 7) / 8);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
#define OZ_CALL_B(BB) \
    k_split_b<BB, false><<<grid, 256, 0, st>>>(B, ldb, K, N, ec, s, KC, n_kc, BN, Np, tiles, trans ? 1 : 0, nullptr)
#define OZ_CALL_B8(BB) \
    k_split_b<BB, true><<<grid, 256, 0, st>>>(B, ldb, K, N, ec, s, KC, n_kc, BN, Np, tiles, trans ? 1 : 0, nullptr)
    if (norm) {
        k_split_b<7, false, true><<<grid, 256, 0, st>>>(B, ldb, K, N, ec, s, KC, n_kc, BN, Np, tiles, trans ? 1 : 0, norm);
    } else if (f8) {
        OZ_SPLIT_DISPATCH_F8(b, OZ_CALL_B8)
    } else {
        OZ_SPLIT_DISPATCH(b, OZ_CALL_B)
    }
#undef OZ_CALL_B
#undef OZ_CALL_B8
}

int launch_selftest_timeout(int *err, unsigned long long timeout_ns, void *stream) {
    k_selftest_timeout<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(err, timeout_ns);
    return 0;
}

}  // namespace ozgb
