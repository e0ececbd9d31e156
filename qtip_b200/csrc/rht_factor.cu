// Hadamard transforms of n = kfac * 2^p values on the tensor cores.
//
// The +-1 factor multiply is the only part with real arithmetic (kfac values per output), and it is a matrix product:
// (kfac x kfac) +-1 times the (kfac, 2^p) view of the row.  The factor is exact in fp16; the row is too when it is an fp16
// activation times signs (found out at run time, per row), else it is scaled by a power of two and split into an fp16 head
// and an fp16 remainder (22 bits); fp32 accumulation either way.  The remainders are accumulated before the heads, because the tensor
// cores' additions truncate.  Error against 64 bits, fp32 rows: 0.9e-7 to 1.2e-7 of the norm at all widths (heads and remainders in turn
// 1.3e-7 to 3.0e-7; kfac fp32 additions per value 1.0e-7 to 1.6e-7).  The factor runs before the Walsh-Hadamard stages (they commute),
// on the exact values.
// A warp's task is 16 result rows x up to 64 columns of the view: the accumulator holds all of it, so the lowest stages are
// register adds and two shuffles; higher stages and the output sit behind one exchange through shared memory.
//
//   rht_row_kernel      a CTA makes the result rows m0 .. m0 + 16*mt_here of the view: few rows are spread over the chip by
//                       these parts, many rows take whole-row CTAs that read their input once and walk over the rows.
//   rht_cluster_kernel  a thread-block cluster per row, for few long rows.
//
// Measured, microseconds per launch (fp16 -> fp16, general path; before: 4 to 8 result rows per CTA, each CTA re-reading the row, fp32
// multiply-adds):  11008 x 1000 rows 1021 -> 62, x 120 124 -> 13, x 8 13.6 -> 5.9, x 1 6.6 -> 5.6;  28672 x 1000 454 -> 99,
// x 27 18.7 -> 7.3, x 1 9.3 -> 5.4;  53248 x 8 15.6 -> 8.4.  Many rows are bound by the operand reads from shared memory
// (two wavefronts per mma) and the mma.sync rate together; few rows by the chain load, barrier, product, exchange, store.
// fp16 rows without statistics and conversions (HALVES): 11008 x 1000 rows 55 -> 45, x 120 10.3 -> 9.3, x 1 6.4 -> 4.6;
// 28672 x 1000 with signs 98 -> 67; 14336 x 1000 43 -> 30.
// Nothing is full there: a CTA's rows are strictly serial (load, barrier, product, exchange, store) at 16 resident warps, so the time is the
// chain's, in which instructions count (20 000 per row of 11008, a quarter of them in the last pass at two values per thread; now 15 900,
// issued in 36 % of the slots).  Up to eight values per thread there, and a multiply-add instead of two predicated adds per shuffle: fp16 rows,
// signs after the transform, 11008 x 1000 39.8 -> 33.6, x 120 8.4 -> 7.2, x 1 4.5 -> 3.2; 14336 x 1000 40.2 -> 27.9; 28672 x 1000
// 88.6 -> 59.7, x 120 12.4 -> 8.6; 53248 x 1000 270 -> 224.  (A variant of 64 registers with more resident warps spilled: slower.)
#include <algorithm>

#include "rht.cuh"

namespace qtip {
namespace {

__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

constexpr int kRowMaxThreads = 512;
constexpr int kClusterThreads = 256;

// words per row of the packed operand and of the exchanged result: 8 more than the columns puts the eight rows (four
// row pairs) a fragment access touches into different banks
__host__ __device__ __forceinline__ int mma_stride(int len) { return len + (len == 8 ? 16 : 8); }

struct RowShape {
    int mt, kt, kq;      // 16-row tiles of the result, 16-deep steps of the product, groups of four such steps
    int mt_cta;          // result tiles per CTA
    int parts;           // CTAs per row
};
struct ClusterShape {
    int mt, kt;
    int csize_log;       // CTAs per cluster
};

// Walsh-Hadamard stages over the columns a warp's accumulator holds: bit 0 is the register pair, bits 1-2 the lane's
// position in its group of four, the others the n-tile.
template <int NTL, bool FMA>
__device__ __forceinline__ void fwht_fragment(float (&acc)[NTL][4], int lane) {
#pragma unroll
    for (int nt = 0; nt < NTL; nt++)
#pragma unroll
        for (int h = 0; h < 4; h += 2) {
            const float x = acc[nt][h], y = acc[nt][h + 1];
            acc[nt][h] = x + y;
            acc[nt][h + 1] = x - y;
        }
#pragma unroll
    for (int bit = 1; bit < 4; bit <<= 1) {
        const float mine = (lane & bit) ? -1.f : 1.f;        // FMA: o +- x as one multiply-add (the product is exact), for a register
#pragma unroll
        for (int nt = 0; nt < NTL; nt++)
#pragma unroll
            for (int h = 0; h < 4; h++) {
                const float o = __shfl_xor_sync(kFullMask, acc[nt][h], bit);
                if constexpr (FMA) acc[nt][h] = fmaf(acc[nt][h], mine, o);
                else acc[nt][h] = (lane & bit) ? o - acc[nt][h] : acc[nt][h] + o;
            }
    }
#pragma unroll
    for (int s = 1; s < NTL; s <<= 1)
#pragma unroll
        for (int nt = 0; nt < NTL; nt++)
            if (!(nt & s))
#pragma unroll
                for (int h = 0; h < 4; h++) {
                    const float x = acc[nt][h], y = acc[nt | s][h];
                    acc[nt][h] = x + y;
                    acc[nt | s][h] = x - y;
                }
}

// butterflies over the register index of E groups of W columns
template <int E, int W>
__device__ __forceinline__ void butterflies(float (&v)[E][W]) {
#pragma unroll
    for (int s = 1; s < E; s <<= 1)
#pragma unroll
        for (int k = 0; k < E; k++)
            if (!(k & s))
#pragma unroll
                for (int h = 0; h < W; h++) {
                    const float x = v[k][h], y = v[k | s][h];
                    v[k][h] = x + y;
                    v[k | s][h] = x - y;
                }
}
// W = 2, 4 or 8 consecutive values, W values aligned
template <int W>
__device__ __forceinline__ void load_row(const float *p, float (&v)[W]) {
    if constexpr (W == 2) {
        const float2 q = __ldg(reinterpret_cast<const float2 *>(p));
        v[0] = q.x; v[1] = q.y;
    } else {
#pragma unroll
        for (int c = 0; c < W; c += 4) {
            const float4 q = __ldg(reinterpret_cast<const float4 *>(p + c));
            v[c] = q.x; v[c + 1] = q.y; v[c + 2] = q.z; v[c + 3] = q.w;
        }
    }
}
template <int W>
__device__ __forceinline__ void store_row(const RhtArgs &a, size_t e, const float (&v)[W]) {
    if (a.out_dtype == QTIP_F16) {
        uint32_t h[W / 2];
#pragma unroll
        for (int c = 0; c < W; c += 2) {
            const __half2 q = __floats2half2_rn(v[c], v[c + 1]);
            h[c / 2] = *reinterpret_cast<const uint32_t *>(&q);
        }
        __half *o = static_cast<__half *>(a.out) + e;
        if constexpr (W == 8) *reinterpret_cast<uint4 *>(o) = make_uint4(h[0], h[1], h[2], h[3]);
        else if constexpr (W == 4) *reinterpret_cast<uint2 *>(o) = make_uint2(h[0], h[1]);
        else *reinterpret_cast<uint32_t *>(o) = h[0];
    } else {
        float *o = static_cast<float *>(a.out) + e;
        if constexpr (W == 2) *reinterpret_cast<float2 *>(o) = make_float2(v[0], v[1]);
        else
#pragma unroll
            for (int c = 0; c < W; c += 4) *reinterpret_cast<float4 *>(o + c) = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
    }
}
__device__ __forceinline__ void store_pair(const RhtArgs &a, size_t e, float y0, float y1) {
    if (a.out_dtype == QTIP_F16) *reinterpret_cast<__half2 *>(static_cast<__half *>(a.out) + e) = __floats2half2_rn(y0, y1);
    else *reinterpret_cast<float2 *>(static_cast<float *>(a.out) + e) = make_float2(y0, y1);
}

// Factor fragments as sign bits: word (tile, q, lane) holds the product steps 4q..4q+3 of result rows m0 + 16*tile ..; register
// r of step 4q + kk has its two sign bits at 15 - (4kk + r) and 31 - (4kk + r).  `bits` holds the packed factor afterwards.
__device__ __forceinline__ void build_fragments(const RhtArgs &a, uint32_t *afrag, uint32_t *bits, int m0, int mt_here, int kq) {
    const int kfac = a.kfac, wpr = (kfac + 31) >> 5;
    for (int i = threadIdx.x; i < kfac * wpr; i += blockDim.x) bits[i] = a.hadk_bits[i];
    __syncthreads();
    for (int idx = threadIdx.x; idx < mt_here * kq * 32; idx += blockDim.x) {
        const int g = (idx >> 2) & 7, t = idx & 3, q = (idx >> 5) % kq, row = m0 + 16 * ((idx >> 5) / kq) + g;
        uint32_t w = 0;
        if (!a.transpose) {
#pragma unroll
            for (int half = 0; half < 2; half++) {               // rows g and g + 8 of the fragment
                const int rr = min(row + 8 * half, kfac - 1);
#pragma unroll
                for (int hw = 0; hw < 2; hw++) {                 // two words = 64 factor columns
                    const uint32_t neg = ~bits[rr * wpr + min(2 * q + hw, wpr - 1)] >> (2 * t);
#pragma unroll
                    for (int c = 0; c < 4; c++) {                // columns 16*(c >> 1) + 8*(c & 1) + 2t, +1 of the word
                        const int at = 4 * (2 * hw + (c >> 1)) + 2 * (c & 1) + half;
                        w |= (((neg >> (8 * c)) & 1u) << (15 - at)) | (((neg >> (8 * c + 1)) & 1u) << (31 - at));
                    }
                }
            }
        } else {
            const int word = min(row >> 5, wpr - 1), sh = row & 31;      // columns g and g + 8 of the factor share a word
#pragma unroll
            for (int c = 0; c < 8; c++)                                  // factor rows 64q + 8c + 2t, +1
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const uint32_t neg = ~bits[min(64 * q + 8 * c + 2 * t + e, kfac - 1) * wpr + word] >> sh;
                    const int at = 2 * c;                                // register 2*(c & 1) (+ 1 for g + 8) of step c >> 1
                    w |= ((neg & 1u) << (15 + 16 * e - at)) | (((neg >> 8) & 1u) << (14 + 16 * e - at));
                }
        }
        afrag[idx] = w;
    }
    __syncthreads();
}

// Largest magnitude (as bits) and whether a value is not an fp16 number, over the CTA; scratch: 64 words.  Two barriers, the
// first of which also ends every earlier use of scratch.
struct RowStats {
    uint32_t mx = 0, inexact = 0;
    __device__ __forceinline__ void add(const float (&x)[8]) {
#pragma unroll
        for (int c = 0; c < 8; c++) {
            mx = max(mx, __float_as_uint(x[c]) & 0x7FFFFFFFu);
            inexact |= __float_as_uint(__half2float(__float2half_rn(x[c])) - x[c]);
        }
    }
    __device__ __forceinline__ void over_cta(uint32_t *scratch) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
        mx = __reduce_max_sync(kFullMask, mx);
        const bool any = __any_sync(kFullMask, inexact != 0u);
        __syncthreads();
        if (lane == 0) { scratch[warp] = mx; scratch[32 + warp] = any ? 1u : 0u; }
        __syncthreads();
        mx = 0; inexact = 0;
        for (int w = 0; w < nwarps; w++) { mx = max(mx, scratch[w]); inexact |= scratch[32 + w]; }
    }
    // exponent of the power of two that brings the largest magnitude into [2^14, 2^15); 0 for fp16 values
    __device__ __forceinline__ int scale_exponent() const {
        return inexact && mx < 0x7F800000u ? min(max(14 - ((int)(mx >> 23) - 127), -112), 126) : 0;
    }
};

// Columns c .. c+7 of rows 2k2 and 2k2 + 1 as packed pairs: fp16 heads at dst, remainders one plane further
__device__ __forceinline__ void put_pairs(uint32_t *dst, int plane, bool remainder, float up, const float (&x0)[8], const float (&x1)[8]) {
    uint32_t w[8], r[8];
#pragma unroll
    for (int c = 0; c < 8; c++) {
        const float s0 = x0[c] * up, s1 = x1[c] * up;
        const __half2 hi = __floats2half2_rn(s0, s1);
        const __half2 lo = __floats2half2_rn(s0 - __low2float(hi), s1 - __high2float(hi));
        w[c] = *reinterpret_cast<const uint32_t *>(&hi);
        r[c] = *reinterpret_cast<const uint32_t *>(&lo);
    }
    reinterpret_cast<uint4 *>(dst)[0] = make_uint4(w[0], w[1], w[2], w[3]);
    reinterpret_cast<uint4 *>(dst)[1] = make_uint4(w[4], w[5], w[6], w[7]);
    if (remainder) {
        reinterpret_cast<uint4 *>(dst + plane)[0] = make_uint4(r[0], r[1], r[2], r[3]);
        reinterpret_cast<uint4 *>(dst + plane)[1] = make_uint4(r[4], r[5], r[6], r[7]);
    }
}

// one step of the product: acc += A * (operand rows at ra, rb)
template <int NTL>
__device__ __forceinline__ void product_step(float (&acc)[NTL][4], const uint32_t (&A)[4], const uint32_t *ra, const uint32_t *rb) {
#pragma unroll
    for (int nt = 0; nt < NTL; nt++) mma_f16(acc[nt], A, ra[nt * 8], rb[nt * 8]);
}

// acc (16 rows x 8*NTL columns) += factor tile * operand columns; `frag` = this lane's word of the tile's first group, `col` =
// the operand at this lane's column.  Operand rows beyond k2n read the zero row k2n.  A row's remainders, if it has them, go first: the
// tensor cores' additions truncate, and while the accumulator holds only remainders that costs nothing.
template <int NTL>
__device__ __forceinline__ void factor_product(float (&acc)[NTL][4], const uint32_t *frag, const uint32_t *col, int kt, int k2n, int stride,
                                               int plane, bool remainder) {
    const int t = threadIdx.x & 3;
    if (remainder) col += plane;
    for (int pass = remainder ? 0 : 1; pass < 2; pass++, col -= plane) {
        uint32_t w = 0;
        for (int k = 0; k < kt; k++) {
            if ((k & 3) == 0) w = frag[(k >> 2) * 32];
            uint32_t A[4];
#pragma unroll
            for (int r = 0; r < 4; r++) { A[r] = (w & 0x80008000u) | 0x3C003C00u; w <<= 1; }
            product_step<NTL>(acc, A, col + min(k * 8 + t, k2n) * stride, col + min(k * 8 + t + 4, k2n) * stride);
        }
    }
}

// The same with the fragments taken from the packed factor itself (shared memory, row-major): a few more instructions per
// step, but no table to build - for CTAs that make one row.
template <int NTL>
__device__ __forceinline__ void factor_product_bits(float (&acc)[NTL][4], const uint32_t *bits, int wpr, int kfac, bool transpose, int m0,
                                                    const uint32_t *col, int kt, int k2n, int stride, int plane, bool remainder) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    if (remainder) col += plane;
    for (int pass = remainder ? 0 : 1; pass < 2; pass++, col -= plane)
#pragma unroll 4
    for (int k = 0; k < kt; k++) {
        uint32_t A[4];
        if (!transpose) {
#pragma unroll
            for (int half = 0; half < 2; half++) {           // rows g, g + 8; entries 16k + 2t, +1 and + 8, + 9
                const int row = min(m0 + g + 8 * half, kfac - 1);
                const uint32_t w = bits[row * wpr + (k >> 1)] >> (16 * (k & 1) + 2 * t);
                A[half] = (w << 15 & 0x8000u) | (w << 30 & 0x80000000u);
                A[2 + half] = (w << 7 & 0x8000u) | (w << 22 & 0x80000000u);
            }
        } else {
            const int c = m0 + g, word = min(c >> 5, wpr - 1), sh = c & 31;      // columns g, g + 8 share a word (m0 % 16 == 0)
            uint32_t r[4];
#pragma unroll
            for (int e = 0; e < 4; e++) r[e] = bits[min(16 * k + 2 * t + (e & 1) + 8 * (e >> 1), kfac - 1) * wpr + word] >> sh;
#pragma unroll
            for (int half = 0; half < 2; half++)
#pragma unroll
                for (int hh = 0; hh < 2; hh++)
                    A[2 * hh + half] = ((r[2 * hh] >> (8 * half)) << 15 & 0x8000u) | ((r[2 * hh + 1] >> (8 * half)) << 31);
        }
#pragma unroll
        for (int r = 0; r < 4; r++) A[r] = (A[r] ^ 0x80008000u) | 0x3C003C00u;      // a set bit is +1
        product_step<NTL>(acc, A, col + min(k * 8 + t, k2n) * stride, col + min(k * 8 + t + 4, k2n) * stride);
    }
}

// The stages above the fragment's, scale, sign and store: a thread owns columns lo .. lo + W - 1 and their 2^R partners.  WIDE: up to
// eight columns with partners too (14336 x 1000 rows 40 -> 28 us); the general variant's registers are full (wider there: 2 to 4 % slower).
template <int R, bool WIDE>
__device__ __forceinline__ void row_finish(const RhtArgs &a, const float *obuf, int ostride, int cw_log, int rows_here, size_t sign_at,
                                           size_t out_at, float inv) {
    constexpr int E = 1 << R, W_log = R <= 1 ? 3 : WIDE && R <= 3 ? 2 : 1, W = 1 << W_log;
    const int items_log = cw_log - W_log;
    for (int it = threadIdx.x; it < (rows_here << items_log); it += blockDim.x) {
        const int i = it >> items_log, lo = (it & ((1 << items_log) - 1)) * W;
        const float *src = obuf + i * ostride + lo;
        const size_t e0 = ((size_t)i << a.p) + lo;
        float v[E][W];
#pragma unroll
        for (int k = 0; k < E; k++)
#pragma unroll
            for (int c = 0; c < W; c += 4) {
                if constexpr (W == 2) {
                    const float2 q = *reinterpret_cast<const float2 *>(src + (k << cw_log));
                    v[k][0] = q.x; v[k][1] = q.y;
                } else {
                    const float4 q = *reinterpret_cast<const float4 *>(src + (k << cw_log) + c);
                    v[k][c] = q.x; v[k][c + 1] = q.y; v[k][c + 2] = q.z; v[k][c + 3] = q.w;
                }
            }
        butterflies<E, W>(v);
#pragma unroll
        for (int k = 0; k < E; k++) {
            const size_t e = e0 + ((size_t)k << cw_log);
#pragma unroll
            for (int c = 0; c < W; c++) v[k][c] = v[k][c] * inv * a.scale;
            if (a.sign_out) {
                float s[W];
                load_row<W>(a.sign_out + sign_at + e, s);
#pragma unroll
                for (int c = 0; c < W; c++) v[k][c] *= s[c];
            }
            store_row<W>(a, out_at + e, v[k]);
        }
    }
}

// NTL: n-tiles (8 columns) of a warp task, at most min(2^p, 64) / 8;  TPW: tasks per warp;  HOLD: row-vector pairs a thread
// keeps in registers between the statistics and the conversion; 0: rows too long for that are read again.  HALVES: fp16 rows with at
// most fp16 signs before the transform.
template <int NTL, int TPW, int HOLD, bool HALVES>
__global__ void __launch_bounds__(kRowMaxThreads) rht_row_kernel(const RhtArgs a, const RowShape S, const long rows) {
    extern __shared__ __align__(16) float sm[];
    const int len = 1 << a.p, kfac = a.kfac, n = a.n;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int stride = mma_stride(len), k2n = kfac >> 1, plane = (k2n + 1) * stride;
    const int tile0 = blockIdx.x * S.mt_cta, mt_here = min(S.mt_cta, S.mt - tile0), m0 = tile0 * 16;
    const int rows_here = min(mt_here * 16, kfac - m0);
    // shared memory: per-warp scratch | factor fragments | operand planes (heads, remainders), overlaid by the result
    float *scratch = sm;
    uint32_t *afrag = reinterpret_cast<uint32_t *>(sm + 64);
    uint32_t *b0p = afrag + S.mt_cta * S.kq * 32;
    float *obuf = reinterpret_cast<float *>(b0p);
    build_fragments(a, afrag, b0p, m0, mt_here, S.kq);
    rht_wait(a);

    const int j8_log = a.p - 3, npairs = k2n << j8_log;
    constexpr int cw_log = NTL == 8 ? 6 : NTL == 4 ? 5 : NTL == 2 ? 4 : 3;
    const int chunks_log = a.p - cw_log;
    auto at = [&](int q, int h) { return (size_t)((((q >> j8_log) * 2 + h) << a.p) + 8 * (q & ((1 << j8_log) - 1))); };
    for (long row = blockIdx.y; row < rows; row += gridDim.y) {
        const size_t sign_off = (size_t)(row % a.sign_rep) * n, in_off = (size_t)row * a.in_row_stride;
        const bool write_res = a.residual_out && blockIdx.x == 0 && (a.in_row_stride != 0 || row == 0);
        auto dst = [&](int q) { return b0p + (q >> j8_log) * stride + 8 * (q & ((1 << j8_log) - 1)); };
        float inv = 1.f;
        bool remainder = false, packed = false;
        if constexpr (HALVES) {
            // an fp16 row, its signs applied to the sign bits, is the operand as it is: no statistics, no conversions.  Decided by the
            // row's signs; one that is not +-1 sends the row through the general path.
            uint4 w[HOLD][2];
            bool other = false;
#pragma unroll
            for (int u = 0; u < HOLD; u++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int q = threadIdx.x + u * blockDim.x;
                    if (q < npairs) w[u][h] = *reinterpret_cast<const uint4 *>(static_cast<const __half *>(a.in) + in_off + at(q, h));
                }
            if (a.sign_in) {
#pragma unroll
                for (int u = 0; u < HOLD; u++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int q = threadIdx.x + u * blockDim.x;
                        if (q < npairs) {
                            const uint4 s = *reinterpret_cast<const uint4 *>(static_cast<const __half *>(a.sign_in) + sign_off + at(q, h));
                            other |= (((s.x ^ 0x3C003C00u) | (s.y ^ 0x3C003C00u) | (s.z ^ 0x3C003C00u) | (s.w ^ 0x3C003C00u)) & 0x7FFF7FFFu) != 0u;
                            w[u][h].x ^= s.x & 0x80008000u; w[u][h].y ^= s.y & 0x80008000u;
                            w[u][h].z ^= s.z & 0x80008000u; w[u][h].w ^= s.w & 0x80008000u;
                        }
                    }
            }
            packed = !__syncthreads_or(other);                   // also frees the result buffer of the row before
            if (packed) {
#pragma unroll
                for (int u = 0; u < HOLD; u++) {
                    const int q = threadIdx.x + u * blockDim.x;
                    if (q < npairs) {
                        const uint4 x = w[u][0], y = w[u][1];
                        reinterpret_cast<uint4 *>(dst(q))[0] = make_uint4(__byte_perm(x.x, y.x, 0x5410), __byte_perm(x.x, y.x, 0x7632),
                                                                          __byte_perm(x.y, y.y, 0x5410), __byte_perm(x.y, y.y, 0x7632));
                        reinterpret_cast<uint4 *>(dst(q))[1] = make_uint4(__byte_perm(x.z, y.z, 0x5410), __byte_perm(x.z, y.z, 0x7632),
                                                                          __byte_perm(x.w, y.w, 0x5410), __byte_perm(x.w, y.w, 0x7632));
                    }
                }
            }
        }
        if (!packed) {
            float rnorm = 0.f, ss = 0.f;
            float v[HOLD > 0 ? HOLD : 1][2][8];
            RowStats st;
            auto sum_squares = [&](size_t e, const float (&x)[8]) {
                if (write_res) store8_f16(a.residual_out, in_off + e, x);
#pragma unroll
                for (int c = 0; c < 8; c++) ss += x[c] * x[c];
            };
            if constexpr (HOLD > 0) {
                // every load of the row is requested before the first value is used
#pragma unroll
                for (int u = 0; u < HOLD; u++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int q = threadIdx.x + u * blockDim.x;
                        if (q < npairs) load_row_vec(a, in_off, at(q, h), v[u][h]);
                        else
#pragma unroll
                            for (int c = 0; c < 8; c++) v[u][h][c] = 0.f;
                    }
                if (a.norm_weight || write_res) {
#pragma unroll
                    for (int u = 0; u < HOLD; u++)
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            const int q = threadIdx.x + u * blockDim.x;
                            if (q < npairs) sum_squares(at(q, h), v[u][h]);
                        }
                }
                if (a.norm_weight) rnorm = rsqrtf(block_sum(ss, scratch) / (float)n + a.eps);
#pragma unroll
                for (int u = 0; u < HOLD; u++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int q = threadIdx.x + u * blockDim.x;
                        if (q < npairs) finish_row_vec(a, in_off, sign_off, at(q, h), rnorm, v[u][h]);
                        st.add(v[u][h]);
                    }
            } else {
                if (a.norm_weight || write_res) {
                    for (int q = threadIdx.x; q < npairs; q += blockDim.x)
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            load_row_vec(a, in_off, at(q, h), v[0][h]);
                            sum_squares(at(q, h), v[0][h]);
                        }
                }
                if (a.norm_weight) rnorm = rsqrtf(block_sum(ss, scratch) / (float)n + a.eps);
                for (int q = threadIdx.x; q < npairs; q += blockDim.x)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        load_row_vec(a, in_off, at(q, h), v[0][h]);
                        finish_row_vec(a, in_off, sign_off, at(q, h), rnorm, v[0][h]);
                        st.add(v[0][h]);
                    }
            }
            st.over_cta(reinterpret_cast<uint32_t *>(scratch));      // its first barrier also frees the result buffer of the row before
            const int ex = st.scale_exponent();
            const float up = __uint_as_float((uint32_t)(127 + ex) << 23);
            inv = __uint_as_float((uint32_t)(127 - ex) << 23);
            remainder = st.inexact != 0u;
            if constexpr (HOLD > 0) {
#pragma unroll
                for (int u = 0; u < HOLD; u++) {
                    const int q = threadIdx.x + u * blockDim.x;
                    if (q < npairs) put_pairs(dst(q), plane, remainder, up, v[u][0], v[u][1]);
                }
            } else {
                for (int q = threadIdx.x; q < npairs; q += blockDim.x) {
                    float x[2][8];
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        load_row_vec(a, in_off, at(q, h), x[h]);
                        finish_row_vec(a, in_off, sign_off, at(q, h), rnorm, x[h]);
                    }
                    put_pairs(dst(q), plane, remainder, up, x[0], x[1]);
                }
            }
        }
        for (int i = threadIdx.x; i < stride; i += blockDim.x) { b0p[k2n * stride + i] = 0u; b0p[plane + k2n * stride + i] = 0u; }
        __syncthreads();

        float acc[TPW][NTL][4] = {};
#pragma unroll
        for (int q = 0; q < TPW; q++) {
            const int task = warp + q * nwarps, tile = task >> chunks_log, c0 = (task & ((1 << chunks_log) - 1)) << cw_log;
            if (tile < mt_here) factor_product<NTL>(acc[q], afrag + tile * S.kq * 32 + lane, b0p + c0 + g, S.kt, k2n, stride, plane, remainder);
        }
        __syncthreads();                       // the operand planes are read: the result overlays them
#pragma unroll
        for (int q = 0; q < TPW; q++) {
            const int task = warp + q * nwarps, tile = task >> chunks_log, c0 = (task & ((1 << chunks_log) - 1)) << cw_log;
            if (tile >= mt_here) continue;     // uniform over the warp
            fwht_fragment<NTL, HALVES>(acc[q], lane);
            float *o = obuf + (tile * 16 + g) * stride + c0 + 2 * t;
#pragma unroll
            for (int nt = 0; nt < NTL; nt++) {
                *reinterpret_cast<float2 *>(o + nt * 8) = make_float2(acc[q][nt][0], acc[q][nt][1]);
                *reinterpret_cast<float2 *>(o + nt * 8 + 8 * stride) = make_float2(acc[q][nt][2], acc[q][nt][3]);
            }
        }
        __syncthreads();
        const size_t first = (size_t)m0 << a.p, s_at = sign_off + first, o_at = (size_t)row * n + first;
        switch (chunks_log) {
            case 0: row_finish<0, HALVES>(a, obuf, stride, cw_log, rows_here, s_at, o_at, inv); break;
            case 1: row_finish<1, HALVES>(a, obuf, stride, cw_log, rows_here, s_at, o_at, inv); break;
            case 2: row_finish<2, HALVES>(a, obuf, stride, cw_log, rows_here, s_at, o_at, inv); break;
            case 3: row_finish<3, HALVES>(a, obuf, stride, cw_log, rows_here, s_at, o_at, inv); break;
            case 4: row_finish<4, HALVES>(a, obuf, stride, cw_log, rows_here, s_at, o_at, inv); break;
            default: row_finish<5, HALVES>(a, obuf, stride, cw_log, rows_here, s_at, o_at, inv); break;
        }
    }
}

// ---- few long rows: one thread-block cluster per row ---------------------------------------------------------------------
// A row is a chain of latencies, not of bandwidth: CTAs that each read the whole row spent most of their time on it.  Here
// CTA r of a cluster owns a range of COLUMNS of the view - the factor acts on columns independently - so the row is read
// once, and only the stages over the cluster's column bits need the other CTAs: every CTA leaves its part in its shared
// memory, one cluster barrier, and each makes its share of the outputs from all parts.

// The stages over column bits above a fragment's: partner k of column lo sits in CTA k >> lb, local column lo + (k mod
// 2^lb) * width.  Contains the barrier after which the other CTAs' parts can be read; the signs of a thread's first item are
// requested before it.
template <int R>
__device__ __forceinline__ void cluster_finish(const RhtArgs &a, uint32_t obuf, int ostride, int cw_log, int lb, int csize_log, size_t sign_at,
                                               size_t out_at) {
    constexpr int E = 1 << R;
    const int pairs_log = cw_log - 1, items = a.kfac << pairs_log, first = (int)cluster_rank() * kClusterThreads + (int)threadIdx.x;
    float2 sg[E];
    auto signs = [&](int it) {
        const size_t e0 = ((size_t)(it >> pairs_log) << a.p) + (it & ((1 << pairs_log) - 1)) * 2;
#pragma unroll
        for (int k = 0; k < E; k++) sg[k] = __ldg(reinterpret_cast<const float2 *>(a.sign_out + sign_at + e0 + ((size_t)k << cw_log)));
    };
    if (a.sign_out && first < items) signs(first);
    cluster_sync();
    for (int it = first; it < items; it += kClusterThreads << csize_log) {
        const int i = it >> pairs_log, lo = (it & ((1 << pairs_log) - 1)) * 2;
        const size_t e0 = ((size_t)i << a.p) + lo;
        float v[E][2];
#pragma unroll
        for (int k = 0; k < E; k++) {
            const float2 q = peer_load2(peer_smem(obuf + (uint32_t)(i * ostride + lo + ((k & ((1 << lb) - 1)) << cw_log)) * 4u, k >> lb));
            v[k][0] = q.x; v[k][1] = q.y;
        }
        butterflies<E, 2>(v);
        if (a.sign_out && it != first) signs(it);
#pragma unroll
        for (int k = 0; k < E; k++) {
            float y0 = v[k][0] * a.scale, y1 = v[k][1] * a.scale;
            if (a.sign_out) { y0 *= sg[k].x; y1 *= sg[k].y; }
            store_pair(a, out_at + e0 + ((size_t)k << cw_log), y0, y1);
        }
    }
}

template <int NTL, int TPW, int HOLD>
__global__ void __launch_bounds__(kClusterThreads, 2) rht_cluster_kernel(const RhtArgs a, const ClusterShape S) {
    extern __shared__ __align__(16) float sm[];
    constexpr int nwarps = kClusterThreads / 32;
    const int kfac = a.kfac, n = a.n;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int wlog = a.p - S.csize_log, width = 1 << wlog;         // columns of this CTA
    const int stride = mma_stride(width), k2n = kfac >> 1, plane = (k2n + 1) * stride;
    // shared memory: scratch | packed factor | operand planes | result (read by the whole cluster)
    const int wpr = (kfac + 31) >> 5, nbits = (kfac * wpr + 3) & ~3;
    float *scratch = sm;
    uint32_t *bits = reinterpret_cast<uint32_t *>(sm + 64);
    uint32_t *b0p = bits + nbits;
    float *obuf = reinterpret_cast<float *>(b0p + 2 * plane);
    for (int i = threadIdx.x; i < kfac * wpr; i += kClusterThreads) bits[i] = __ldg(a.hadk_bits + i);
    rht_wait(a);

    const long row = blockIdx.y;
    const size_t sign_off = (size_t)(row % a.sign_rep) * n, in_off = (size_t)row * a.in_row_stride;
    const size_t col0 = (size_t)cluster_rank() << wlog;
    const bool write_res = a.residual_out && (a.in_row_stride != 0 || row == 0);
    const int j8_log = wlog - 3, npairs = k2n << j8_log;
    auto at = [&](int q, int h) { return ((size_t)((q >> j8_log) * 2 + h) << a.p) + col0 + 8 * (q & ((1 << j8_log) - 1)); };
    float v[HOLD][2][8], rnorm = 0.f;
    RowStats st;
#pragma unroll
    for (int u = 0; u < HOLD; u++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int q = threadIdx.x + u * kClusterThreads;
            if (q < npairs) load_row_vec(a, in_off, at(q, h), v[u][h]);
            else
#pragma unroll
                for (int c = 0; c < 8; c++) v[u][h][c] = 0.f;
        }
    if (a.norm_weight || write_res) {
        float ss = 0.f;
#pragma unroll
        for (int u = 0; u < HOLD; u++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int q = threadIdx.x + u * kClusterThreads;
                if (q >= npairs) continue;
                if (write_res) store8_f16(a.residual_out, in_off + at(q, h), v[u][h]);
#pragma unroll
                for (int c = 0; c < 8; c++) ss += v[u][h][c] * v[u][h][c];
            }
        if (a.norm_weight) {
            rnorm = rsqrtf(cluster_sum(ss, scratch, 1 << S.csize_log) / (float)n + a.eps);
            cluster_sync();                    // every CTA has read the partial sums before scratch is used again
        }
    }
#pragma unroll
    for (int u = 0; u < HOLD; u++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int q = threadIdx.x + u * kClusterThreads;
            if (q < npairs) finish_row_vec(a, in_off, sign_off, at(q, h), rnorm, v[u][h]);
            st.add(v[u][h]);
        }
    // head, remainder and scale are this CTA's own choice: its result is scaled back before the cluster adds
    st.over_cta(reinterpret_cast<uint32_t *>(scratch));
    const int ex = st.scale_exponent();
    const float up = __uint_as_float((uint32_t)(127 + ex) << 23), inv = __uint_as_float((uint32_t)(127 - ex) << 23);
    const bool remainder = st.inexact != 0u;
#pragma unroll
    for (int u = 0; u < HOLD; u++) {
        const int q = threadIdx.x + u * kClusterThreads;
        if (q < npairs) put_pairs(b0p + (q >> j8_log) * stride + 8 * (q & ((1 << j8_log) - 1)), plane, remainder, up, v[u][0], v[u][1]);
    }
    for (int i = threadIdx.x; i < stride; i += kClusterThreads) { b0p[k2n * stride + i] = 0u; b0p[plane + k2n * stride + i] = 0u; }
    __syncthreads();

    constexpr int cw_log = NTL == 8 ? 6 : NTL == 4 ? 5 : NTL == 2 ? 4 : 3;
    const int chunks_log = wlog - cw_log;
#pragma unroll
    for (int q = 0; q < TPW; q++) {
        const int task = warp + q * nwarps, tile = task >> chunks_log, c0 = (task & ((1 << chunks_log) - 1)) << cw_log;
        if (tile >= S.mt) continue;              // uniform over the warp
        float acc[NTL][4] = {};
        factor_product_bits<NTL>(acc, bits, wpr, kfac, a.transpose, tile * 16, b0p + c0 + g, S.kt, k2n, stride, plane, remainder);
        fwht_fragment<NTL, false>(acc, lane);
        float *o = obuf + (tile * 16 + g) * stride + c0 + 2 * t;
#pragma unroll
        for (int nt = 0; nt < NTL; nt++) {
            *reinterpret_cast<float2 *>(o + nt * 8) = make_float2(acc[nt][0] * inv, acc[nt][1] * inv);
            *reinterpret_cast<float2 *>(o + nt * 8 + 8 * stride) = make_float2(acc[nt][2] * inv, acc[nt][3] * inv);
        }
    }
    const uint32_t ob = (uint32_t)__cvta_generic_to_shared(obuf);
    const size_t o_at = (size_t)row * n;
    switch (a.p - cw_log) {
        case 0: cluster_finish<0>(a, ob, stride, cw_log, chunks_log, S.csize_log, sign_off, o_at); break;
        case 1: cluster_finish<1>(a, ob, stride, cw_log, chunks_log, S.csize_log, sign_off, o_at); break;
        case 2: cluster_finish<2>(a, ob, stride, cw_log, chunks_log, S.csize_log, sign_off, o_at); break;
        case 3: cluster_finish<3>(a, ob, stride, cw_log, chunks_log, S.csize_log, sign_off, o_at); break;
        case 4: cluster_finish<4>(a, ob, stride, cw_log, chunks_log, S.csize_log, sign_off, o_at); break;
        default: cluster_finish<5>(a, ob, stride, cw_log, chunks_log, S.csize_log, sign_off, o_at); break;
    }
    cluster_sync();                              // no CTA leaves while others read its part
}

// ---- launch ------------------------------------------------------------------------------------------------------------
// kernel(args...) with programmatic stream serialization and, cluster > 1, that cluster size; dynamic shared memory is opted
// in once per kernel and device
template <class... Params, class... Args>
int launch_opted_in(void (*kernel)(Params...), bool (&attr_set)[64], dim3 grid, int threads, size_t smem, int cluster, cudaStream_t s,
                    const Args &...args) {
    int dev = 0;
    QTIP_CUDA_TRY(cudaGetDevice(&dev));
    if (dev >= 64 || !attr_set[dev]) {
        QTIP_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
        if (dev < 64) attr_set[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    QTIP_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, args...));
    return check_launch();
}

template <int NTL, int TPW, int HOLD>
int launch_rows_variant(const RhtArgs &a, const RowShape &S, long rows, int threads, int grid_y, size_t smem, cudaStream_t s) {
    static bool attr_set[64] = {}, attr_set_halves[64] = {};
    // an own variant: the general path alone is 2 to 5 % faster than beside the packed one
    const bool halves = a.in_dtype == QTIP_F16 && !a.residual && !a.residual_out && !a.norm_weight && !a.gate &&
                        (!a.sign_in || a.sign_in_dtype == QTIP_F16);
    if constexpr (HOLD > 0)
        if (halves)
            return launch_opted_in(rht_row_kernel<NTL, TPW, HOLD, true>, attr_set_halves, dim3(S.parts, grid_y), threads, smem, 1, s, a, S, rows);
    return launch_opted_in(rht_row_kernel<NTL, TPW, HOLD, false>, attr_set, dim3(S.parts, grid_y), threads, smem, 1, s, a, S, rows);
}
// The variants that the supported widths reach, at any number of rows and SMs (by enumeration of the rules in launch_rht_rows): with
// eight n-tiles one or two tasks per warp and rows of up to 27648 values in registers, longer ones read again; with fewer n-tiles
// short rows and more tasks, or (4 and 2) rows of 17920 to 27648 values and one task.  Anything else: kNoVariant.
constexpr int kNoVariant = -1;
template <int NTL>
int launch_rows_ntl(const RhtArgs &a, const RowShape &S, long rows, int threads, int grid_y, int tpw, int hold, size_t smem, cudaStream_t s) {
    if constexpr (NTL == 8) {
        if (hold == 0) return tpw <= 1 ? launch_rows_variant<8, 1, 0>(a, S, rows, threads, grid_y, smem, s)
                                       : launch_rows_variant<8, 2, 0>(a, S, rows, threads, grid_y, smem, s);
        if (tpw == 2) return launch_rows_variant<8, 2, 4>(a, S, rows, threads, grid_y, smem, s);
    }
    if (hold <= 2) {
        if constexpr (NTL <= 2)
            if (tpw > 2) return launch_rows_variant<NTL, 4, 2>(a, S, rows, threads, grid_y, smem, s);
        if constexpr (NTL <= 4)
            if (tpw == 2) return launch_rows_variant<NTL, 2, 2>(a, S, rows, threads, grid_y, smem, s);
        if (tpw <= 1) return launch_rows_variant<NTL, 1, 2>(a, S, rows, threads, grid_y, smem, s);
    } else if constexpr (NTL >= 2)
        if (tpw <= 1) return launch_rows_variant<NTL, 1, 4>(a, S, rows, threads, grid_y, smem, s);
    return kNoVariant;
}

template <int NTL, int TPW, int HOLD>
int launch_cluster_variant(const RhtArgs &a, const ClusterShape &S, long rows, size_t smem, cudaStream_t s) {
    static bool attr_set[64] = {};
    return launch_opted_in(rht_cluster_kernel<NTL, TPW, HOLD>, attr_set, dim3(1u << S.csize_log, (unsigned)rows), kClusterThreads, smem,
                           1 << S.csize_log, s, a, S);
}
// Reached by the supported widths: one task per warp, except in rows of 17920 to 22016 values (two n-tiles) and 35840 to 44032 (four).
template <int NTL>
int launch_cluster_ntl(const RhtArgs &a, const ClusterShape &S, long rows, int tpw, int hold, size_t smem, cudaStream_t s) {
    if (tpw == 1 && hold == 1) return launch_cluster_variant<NTL, 1, 1>(a, S, rows, smem, s);
    if constexpr (NTL == 8)
        if (tpw == 1) return launch_cluster_variant<8, 1, 2>(a, S, rows, smem, s);
    if constexpr (NTL == 4) return launch_cluster_variant<4, 2, 2>(a, S, rows, smem, s);
    if constexpr (NTL == 2)
        if (hold == 1) return launch_cluster_variant<2, 2, 1>(a, S, rows, smem, s);
    return kNoVariant;
}

}  // namespace

// Rows of the view of 8 to 2048 columns whose operand fits shared memory (up to 53248 = 52 * 1024 values), any row count.
bool launch_rht_rows(const RhtArgs &a, long rows, cudaStream_t s, int &status) {
    const int len = 1 << a.p;
    if (a.kfac == 1 || !a.vec_ok || len < 8 || len > 2048) return false;
    RowShape S;
    S.mt = S.kt = (a.kfac + 15) / 16;
    S.kq = (S.kt + 3) / 4;
    // Threads: a row's vector pairs spread so that a thread holds at most four of them in registers.  Few rows: more
    // threads, to have more of the row in flight at once.
    const long want_parts = sm_count() / rows;
    const bool few = want_parts >= 1;
    const int threads = a.n > 16384 || (few && a.n > 4096) ? 512 : (a.n > 4096 || few ? 256 : 128), warps = threads / 32;
    const int npairs = a.n / 16, hold = (npairs + threads - 1) / threads;
    // Columns of a warp's task: the whole row of the view or 64 of it; fewer when the CTA would have idle warps otherwise.
    int ntl = len >= 64 ? 8 : len / 8;
    const int max_tpw = ntl >= 4 ? 2 : 4;
    auto chunks = [&]() { return len / (8 * ntl); };
    const int full = std::min(S.mt, max_tpw * warps / chunks());      // most tiles a CTA can hold (>= 1: chunks <= 32)
    const int parts_min = (S.mt + full - 1) / full, parts = std::max(parts_min, (int)std::min((long)S.mt, want_parts));
    S.mt_cta = (S.mt + parts - 1) / parts;
    S.parts = (S.mt + S.mt_cta - 1) / S.mt_cta;
    while (ntl > 1 && hold <= 4 && S.mt_cta * chunks() * 2 <= warps && chunks() < 32) ntl >>= 1;
    const int tpw = (S.mt_cta * chunks() + warps - 1) / warps;
    const int stride = mma_stride(len), wpr = (a.kfac + 31) / 32;
    const size_t body = std::max(std::max(2 * (size_t)(a.kfac / 2 + 1) * stride, (size_t)16 * S.mt_cta * stride), (size_t)a.kfac * wpr);
    const size_t smem = (64 + (size_t)S.mt_cta * S.kq * 32 + body) * sizeof(float);
    if (smem > 227 * 1024) return false;
    // Many rows: as many CTAs as are resident (128 registers a thread), each walking over an equal share of the rows.
    const long per_sm = std::max(1L, std::min((long)(65536 / (128 * threads)), (long)(227 * 1024 / (smem + 1024))));
    const long cap = std::max(1L, per_sm * sm_count() / S.parts), trips = (rows + cap - 1) / cap;
    const int grid_y = (int)((rows + trips - 1) / trips);
    const int h = hold > 4 ? 0 : hold;
    if (h == 0 && ntl != 8) return false;
    switch (ntl) {
        case 8: status = launch_rows_ntl<8>(a, S, rows, threads, grid_y, tpw, h, smem, s); break;
        case 4: status = launch_rows_ntl<4>(a, S, rows, threads, grid_y, tpw, h, smem, s); break;
        case 2: status = launch_rows_ntl<2>(a, S, rows, threads, grid_y, tpw, h, smem, s); break;
        default: status = launch_rows_ntl<1>(a, S, rows, threads, grid_y, tpw, h, smem, s); break;
    }
    return status != kNoVariant;
}

// Few long rows: a cluster of eight CTAs per row.  Below 128 columns a CTA would have too little of a row (the parts of
// launch_rht_rows are faster: 11008 = 172 * 64, 27 rows: 6.6 against 8.8 us).
bool launch_rht_cluster(const RhtArgs &a, long rows, cudaStream_t s, int &status) {
    const int len = 1 << a.p;
    if (a.kfac == 1 || !a.vec_ok || len < 128) return false;
    ClusterShape S;
    S.mt = S.kt = (a.kfac + 15) / 16;
    S.csize_log = 3;                                       // the portable cluster size
    // two CTAs fit an SM, but clusters of eight do not pack: 27 rows run at once (7.3 us at 28672 columns), 36 take twice that
    if (rows > (3 * sm_count() / 2) >> S.csize_log) return false;
    const int width = len >> S.csize_log, warps = kClusterThreads / 32;
    const int hold = ((a.kfac / 2) * (width / 8) + kClusterThreads - 1) / kClusterThreads;
    if (hold > 2) return false;
    // whole fragments: the more columns a warp transforms in registers, the fewer partners the last stage gathers
    const int ntl = std::min(8, width / 8), tpw = (S.mt * (width / (8 * ntl)) + warps - 1) / warps;
    if (tpw > 2 || len / (8 * ntl) > 32) return false;
    const int stride = mma_stride(width), wpr = (a.kfac + 31) / 32;
    const size_t smem = (64 + ((a.kfac * wpr + 3) & ~3) + 2 * (size_t)(a.kfac / 2 + 1) * stride + (size_t)16 * S.mt * stride) * sizeof(float);
    if (smem > 160 * 1024) return false;
    switch (ntl) {
        case 8: status = launch_cluster_ntl<8>(a, S, rows, tpw, hold, smem, s); break;
        case 4: status = launch_cluster_ntl<4>(a, S, rows, tpw, hold, smem, s); break;
        default: status = launch_cluster_ntl<2>(a, S, rows, tpw, hold, smem, s); break;
    }
    return status != kNoVariant;
}

}  // namespace qtip
