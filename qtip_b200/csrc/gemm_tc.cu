// Decompress-GEMM for batches 9..128 on the 5th-generation tensor cores (tcgen05 + TMEM).
//
//   out (bs, m) fp32 = X (bs, n) fp16 @ decode(codes)^T        HYB code, kernel layout
//
// One CTA owns 128 output rows (four 32-row blocks) and a contiguous range of input columns.  The
// weights are the A operand: D[128 x N] += A[128 x 16] * B[16 x N] with D AND A in tensor memory, B in
// shared memory, K-major, 128-byte swizzle; N = batch rounded up to 16.
//   * 24 decode warps turn packed codes into fp16 and store them with tcgen05.st into a stage of weights (128 rows x 128
//     columns = 16 tile blocks, two per warp; three stages are filled concurrently).  A kernel-layout tile block in its lanes IS
//     the 16x128b store shape, so the weights never pass through shared memory, whose wavefronts the table lookups need.
//   * one thread copies the slices of X with tiled TMA loads (no multicast; rows beyond the batch are filled with zeros) into a ring
//     of its own, as deep as the memory beside the table allows;
//   * one thread issues eight tcgen05.mma (K = 16 each) per step and commits them to the stages'
//     "empty" barriers; a last commit signals the epilogue.
//   * warps 0-3 read the accumulator with tcgen05.ld (warp w owns TMEM lanes 32w..32w+31 = rows) and
//     write out (coalesced along rows); when the row ranges leave SMs idle the columns are split over the
//     2, 4 or 8 CTAs of a cluster, which leave their parts in shared memory and add them in order.
// The compute codes (3INST / 1MAD, V = 1, plain layout) use the same kernel with another producer: a lane decodes one row of a
// tile (its own 2K bytes and the start of the next row), lanes 2r and 2r + 1 row r of two tiles, and stores a row per
// tensor-memory lane; the accumulator's lanes are mapped back to rows when they are read.
// Bound: instruction issue of the decode warps up to about 64 rows (8192 x 28672, 27 rows: leaving out three of four MMAs 45.6 -> 43.0 us,
// the lookups 35.4), the MMAs above (120 rows: 58.3 -> 48.9 and 54.4 us).  Hence two blocks per warp and step between the barriers, x
// through TMA instead of copies by the decode warps, scalar control (the warp index through a shuffle), control threads that sleep
// between polls, and codes requested two steps ahead.  Warp instructions per block of weights, HYB 27 rows 190 -> 145, 3INST 295 -> 217
// (of which the mask of mask_3inst 32).
// Measured, one block per warp and step with x copied by the decode warps -> now (microseconds, K = 2 unless stated): HYB 8192 x 8192
// 27 rows 20.5 -> 17.2; 8192 x 28672 120 rows 73 -> 58.5; 14336 x 4096 K = 3 27 rows 19.7 -> 15.8; 28672 x 8192 K = 4 64 rows 70 -> 57;
// 3INST 8192 x 8192 16 rows 30.5 -> 21.6, 8192 x 28672 120 rows 107 -> 69.5; 1MAD 8192 x 8192 K = 3 32 rows 33.0 -> 29.2.  A second
// accumulator for every other MMA changes nothing.
// This replaces decode-to-HBM + dense GEMM of BitshiftLinearKernelAG upstream
// (lib/codebook/bitshift.py:476-489), which writes and re-reads 16x the packed bytes at 2 bits.
//
// Every mbarrier wait is bounded: after kSpinLimit polls the waiter records an error code in
// `status`, raises a CTA-wide abort flag that makes every later wait fall through, and the kernel
// still runs to its end, frees its tensor memory and returns (with meaningless results).
#include <cuda.h>

#include <algorithm>
#include <mutex>

#include "common.cuh"

namespace qtip {
namespace {

constexpr int kGroups = 3;                               // groups of 8 decode warps; a group fills one stage
constexpr int kDecodeWarps = 8 * kGroups;
constexpr int kMmaWarp = kDecodeWarps, kCopyWarp = kDecodeWarps + 1;      // TMEM allocation and MMA issue; copies of x
constexpr int kGemmThreads = (kDecodeWarps + 2) * 32;
constexpr int kStages = 2 * kGroups;                    // stages of weights: every group may be one step ahead of the MMA
constexpr int kRows = 128;                               // output rows per CTA
constexpr int kStageCols = 128;                          // input columns per step: two blocks per decode warp, two tiles of x
constexpr int kTileCols = 64;                            // 128 bytes of fp16: the swizzle span
constexpr int kAStageCols = kStageCols / 2;              // 32-bit tensor-memory columns of a stage of weights: two weights each
constexpr int kLut512Bytes = 1024 * 32 * 4;              // (512 entries + sign-flipped twins) x 32 lane-private copies
constexpr int kMaxN = 128;
constexpr int kXRingBytes = 96 * 1024;                   // at most, beside the table
constexpr unsigned kSpinLimit = 1u << 22;
// A warp that polls takes issue slots from the decode warps of its sub-partition, so the two control threads sleep between polls; both
// are one or more stages ahead of what they wait for.
constexpr unsigned kMmaSleepNs = 40, kCopySleepNs = 200;

// stages of x: a step's tiles are npad x 128 columns
__host__ __device__ __forceinline__ int x_stages(int npad) {
    const int fit = kXRingBytes / (npad * kStageCols * 2);
    return fit < kStages ? fit : kStages;
}

struct GemmCtrl {
    unsigned long long full[kStages], empty[kStages];        // weights
    unsigned long long xfull[kStages], xempty[kStages];      // x
    unsigned long long done;
    uint32_t tmem_base;
    int abort_flag;
};

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// false: the wait gave up (its own limit, or another waiter raised the abort flag)
template <unsigned kSleepNs = 0>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag, unsigned *status,
                                          unsigned code) {
    if (mbar_try_wait(bar, parity)) return true;
    for (unsigned spin = 0; spin < kSpinLimit; spin++) {
        if (kSleepNs > 0) __nanosleep(kSleepNs);
        if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
    }
    *abort_flag = 1;
    atomicCAS(status, 0u, code);
    return false;
}
// bounded wait that does not look at the abort flag (used before tensor memory is released)
__device__ __forceinline__ void mbar_wait_bounded(uint32_t bar, uint32_t parity) {
    for (unsigned spin = 0; spin < kSpinLimit; spin++)
        if (mbar_try_wait(bar, parity)) return;
}

__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Box of x at column c (a multiple of 64) and row r: rows beyond the tensor are filled with zeros
__device__ __forceinline__ void copy_x_tile(uint32_t dst, const CUtensorMap *map, int c, int r, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(c), "r"(r), "r"(bar) : "memory");
}

// Shared-memory matrix descriptor: K-major, 128-byte swizzle, rows of 128 bytes, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);          // start address
    d |= (uint64_t)1 << 16;                            // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;                  // stride byte offset between 8-row groups
    d |= (uint64_t)1 << 46;                            // descriptor version of sm_100
    d |= (uint64_t)2 << 61;                            // SWIZZLE_128B
    return d;
}

__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// 16 rows x 16 words of tensor memory; lane (a, b) holds words 4j + b of rows a (v[2j]) and a + 8 (v[2j + 1])
__device__ __forceinline__ void tmem_st_16x128b_x4(uint32_t addr, const uint32_t *v) {
    asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(addr), "r"(v[0]), "r"(v[1]),
                 "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
// 32 rows x 16 words, a row per lane
__device__ __forceinline__ void tmem_st_32x32b_x16(uint32_t addr, const uint32_t *v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(addr),
                 "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
                 "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
                 : "memory");
}
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// Plain layout (V = 1 codes): a 16x16 tile is 16K 16-bit words, first stream bit = top bit of word 0, circular.  Row r of a tile is
// K words; its 16 states' windows start K bits apart at word K*r and end 12..15 bits into the next row.
// a: the row's first two words, b: the words after them, first in the top half
template <int K>
struct PlainRow {
    uint32_t a, b;
};
template <int K>
__device__ __forceinline__ PlainRow<K> load_plain_row(const uint16_t *__restrict__ row) {
    PlainRow<K> r = {};
    if constexpr (K == 2) r.a = __byte_perm(__ldg(reinterpret_cast<const uint32_t *>(row)), 0, 0x1032);
    else if constexpr (K == 3) {
        r.a = (uint32_t)__ldg(row) << 16 | __ldg(row + 1);
        r.b = (uint32_t)__ldg(row + 2) << 16;
    } else {
        const uint2 v = __ldg(reinterpret_cast<const uint2 *>(row));
        r.a = __byte_perm(v.x, 0, 0x1032);
        r.b = __byte_perm(v.y, 0, 0x1032);
    }
    return r;
}
// state i of a row; next: the following row's first two words
template <int K>
__device__ __forceinline__ uint32_t plain_state(const PlainRow<K> &r, uint32_t next, int i) {
    uint32_t hi = r.a, lo = r.b;
    if constexpr (K == 2) lo = next;
    if constexpr (K == 3) lo = r.b | next >> 16;
    if (K * i >= 32) {          // i is a compile-time constant after unrolling
        hi = lo;
        lo = next;
    }
    // a window that starts in one of the upper three bytes is two bytes of the stream shifted by less than one: a permute, and the
    // shift is shared by the states of the same residue (K = 2, 4: 23 and 18 instructions a row instead of 32)
    const int bit = K * i & 31, byte = bit >> 3, rest = bit & 7;
    if (K != 3 && byte < 3) {
        const uint32_t shifted = rest ? __funnelshift_l(lo, hi, rest) : hi;
        return __byte_perm(shifted, 0, byte == 0 ? 0x4432 : byte == 1 ? 0x4421 : 0x4410);
    }
    return __funnelshift_l(lo, hi, bit) >> 16;
}

constexpr int kMaxSplit = 8;
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}
__device__ __forceinline__ float cluster_load(uint32_t addr, int rank) {
    uint32_t p;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(p) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(p) : "memory");
    return v;
}

// Two weights of the compute codes, packed.  3INST: each state's two fp16 terms are added by a half2 instruction that takes them
// from one register (the multiply pipe has room; gathering both states' terms for one addition costs a permute more, 31.3 against
// 29.4 us at 8192 x 8192, 27 rows).  1MAD: byte sums of the LCG values by dot product, weights from the lane's copy of the table.
// `mask` is 0x8FFF8FFF as a run-time value: a three-input logic instruction takes one literal, so with two it becomes two
// instructions (8192 x 8192, 16 rows, 26.0 -> 21.6; 8192 x 28672, 120 rows, 83 -> 69.5 us).
__device__ __forceinline__ uint32_t mask_3inst(int npad) { return 0x8FFF8FFFu | (uint32_t)npad >> 16; }
__device__ __forceinline__ uint32_t pair_3inst(uint32_t s0, uint32_t s1, uint32_t mask) {
    const uint32_t r0 = ((s0 * 89226354u + 64248484u) & mask) ^ 0x3B603B60u, r1 = ((s1 * 89226354u + 64248484u) & mask) ^ 0x3B603B60u;
    const __half2 h0 = *reinterpret_cast<const __half2 *>(&r0), h1 = *reinterpret_cast<const __half2 *>(&r1);
    const __half2 w0 = __hadd2(__low2half2(h0), __high2half2(h0)), w1 = __hadd2(__low2half2(h1), __high2half2(h1));
    return __byte_perm(*reinterpret_cast<const uint32_t *>(&w0), *reinterpret_cast<const uint32_t *>(&w1), 0x5410);
}
__device__ __forceinline__ uint32_t pair_1mad(uint32_t s0, uint32_t s1, uint32_t lut_lane) {
    uint32_t w0, w1;
    asm("ld.shared.u32 %0, [%1];" : "=r"(w0) : "r"(__dp4a(s0 * 34038481u + 76625530u, 0x01010101u, 0u) * 128u + lut_lane));
    asm("ld.shared.u32 %0, [%1];" : "=r"(w1) : "r"(__dp4a(s1 * 34038481u + 76625530u, 0x01010101u, 0u) * 128u + lut_lane));
    return __byte_perm(w0, w1, 0x5410);
}

// A decode warp's codes of a step: two blocks (HYB), or rows of 2 x 2 tiles each (V = 1).
template <int K>
struct StepCodes {
    LaneCodes<K> blk[2];
    PlainRow<K> rows[2][2];
};
template <int K, int CODE>
__device__ __forceinline__ void load_step(StepCodes<K> &c, const uint8_t *src, const uint16_t *prow) {
    if constexpr (CODE == QTIP_CODE_HYB) {
#pragma unroll
        for (int h = 0; h < 2; h++) c.blk[h] = load_lane_codes<K>(src + h * (128 * K));
    } else {
#pragma unroll
        for (int h = 0; h < 4; h++) c.rows[h >> 1][h & 1] = load_plain_row<K>(prow + h * (16 * K));
    }
}
// Block h as the words that its tensor-memory stores take (HYB: 8 per 16 rows; V = 1: a row per lane).  lut_lane: the lane's copy of the
// table; 3INST, which has none: the mask
template <int K, int CODE>
__device__ __forceinline__ void decode_half(const StepCodes<K> &c, int h, uint32_t lut_lane, int lane, uint32_t (&wv)[16]) {
    if constexpr (CODE == QTIP_CODE_HYB) {
        LaneCodes<K> nxt = {};
#pragma unroll
        for (int i = 0; i < K; i++) nxt.w[i] = __shfl_sync(kFullMask, c.blk[h].w[i], lane + 1);
#pragma unroll
        for (int tt = 0; tt < 4; tt++) {
            const int ks = tt >> 1, ms = tt & 1;
            uint32_t st[4];
            tile_states<K>(c.blk[h], nxt, tt, st);
#pragma unroll
            for (int q = 0; q < 4; q++)       // q = 2c + d: column half, row half of the 16x16 tile
                wv[8 * ms + 4 * ks + q] = hyb_lookup(st[q], lut_lane);
        }
    } else {
#pragma unroll
        for (int ks = 0; ks < 2; ks++) {
            const uint32_t next = __shfl_sync(kFullMask, c.rows[h][ks].a, lane + 2);      // row 15 -> row 0: tail-biting
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const uint32_t s0 = plain_state<K>(c.rows[h][ks], next, 2 * j), s1 = plain_state<K>(c.rows[h][ks], next, 2 * j + 1);
                wv[8 * ks + j] = CODE == QTIP_CODE_3INST ? pair_3inst(s0, s1, lut_lane) : pair_1mad(s0, s1, lut_lane);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 16; i++) asm volatile("" : "+r"(wv[i]));
}
// lane-private copies of the table: entry e = sign << 9 | index, copy l at byte e*128 + l*4; the sign bit of
// the hash flips the first weight of the pair, so it is folded into the table (no per-state sign op)
// 1MAD: the weight of every byte sum (decode_1mad's own arithmetic) in the same form, 1021 entries used
template <int CODE>
__device__ __forceinline__ void build_table(uint32_t *lut, const uint32_t *__restrict__ tlut) {
    for (int i = threadIdx.x; CODE != QTIP_CODE_3INST && i < 1024 * 8; i += blockDim.x) {
        const uint32_t e = CODE == QTIP_CODE_1MAD ? (uint32_t)__half_as_ushort(__float2half_rn(__fdiv_rn((float)((i >> 3) - 510), 147.800537109375f)))
                                                  : __ldg(tlut + ((i >> 3) & 511)) ^ ((uint32_t)(i >> 12) << 15);
        reinterpret_cast<uint4 *>(lut)[i] = make_uint4(e, e, e, e);
    }
}

template <int K, int CODE>
__global__ void __launch_bounds__(kGemmThreads, 1)
    decompress_gemm_kernel(float *__restrict__ out, const uint8_t *__restrict__ codes, const __grid_constant__ CUtensorMap xmap,
                           const uint32_t *__restrict__ tlut, int m, int n, int bs, int npad, int splitk,
                           unsigned *__restrict__ status) {
    constexpr int kBlockBytes = 128 * K;
    constexpr bool kHyb = CODE == QTIP_CODE_HYB;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_addr(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;                 // swizzled tiles need 1024-byte alignment
    uint8_t *smem = smem_raw + (base - raw);
    const int xstages = x_stages(npad), tile_bytes = npad * kTileCols * 2, x_stage_bytes = 2 * tile_bytes;
    // layout: stages of x | LUT | control
    const uint32_t b_base = base;
    uint32_t *lut = reinterpret_cast<uint32_t *>(smem + xstages * x_stage_bytes);
    GemmCtrl *ctl = reinterpret_cast<GemmCtrl *>(smem + xstages * x_stage_bytes + kLut512Bytes);
    volatile int *abort_flag = &ctl->abort_flag;

    // through a shuffle: known to be the same in all lanes, so that the control of a warp's steps is scalar
    const int warp = __shfl_sync(kFullMask, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    // tensor memory: kStages stages of weights, then the accumulator's npad columns
    constexpr int kTmemD = kStages * kAStageCols, kTmemCols = 512;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; s++) {
            mbar_init(smem_addr(&ctl->full[s]), 8);     // eight decode warps fill a stage
            mbar_init(smem_addr(&ctl->empty[s]), 1);    // one tcgen05.commit frees it
            mbar_init(smem_addr(&ctl->xfull[s]), 1);    // the copying thread, and the bytes it announces
            mbar_init(smem_addr(&ctl->xempty[s]), 1);
        }
        mbar_init(smem_addr(&ctl->done), 1);
        ctl->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) {
        // 128 lanes x kTmemCols 32-bit columns
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&ctl->tmem_base)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    build_table<CODE>(lut, tlut);
    const int nb = n >> 5;                                  // 32-column blocks per row block
    const int r0 = blockIdx.x * kRows;                      // first output row of this CTA
    // 64-column tiles of this CTA: split over the CTAs of the cluster, not necessarily evenly; the last step may have one tile
    const int all_tiles = n / kTileCols;
    const int tile0 = all_tiles * (int)blockIdx.y / splitk, ntiles = all_tiles * ((int)blockIdx.y + 1) / splitk - tile0;
    const int nsteps = (ntiles + 1) >> 1, c0 = tile0 * kTileCols;

    // decode warps: this group fills steps group, group + kGroups, ...; a warp decodes two blocks of a step, rows 32 rb .. of the tile half
    const int group = warp >> 3, rb = warp & 3, half = (warp >> 2) & 1;
    const uint8_t *src = codes + ((size_t)(r0 / 32 + rb) * nb + (c0 / 32 + 2 * half + 4 * group)) * kBlockBytes + lane * (4 * K);
    // plain layout (V = 1 codes): tile (tile row, tile column) = 16K words at ((row/16)*(n/16) + col/16)*16K; this
    // lane decodes row lane >> 1 of tile row 2rb + (lane & 1), tile columns 4 half .. + 3 of the step
    const uint16_t *prow = reinterpret_cast<const uint16_t *>(codes) +
                           ((size_t)(r0 / 16 + 2 * rb + (lane & 1)) * (n >> 4) + (size_t)(c0 / 16 + 4 * half + 8 * group)) * (16 * K) +
                           (lane >> 1) * K;
    // codes of the current step and of the one after it
    StepCodes<K> now = {}, ahead = {};
    auto load_codes = [&](StepCodes<K> &c, int step) {
        if (2 * step + half >= ntiles) return;
        load_step<K, CODE>(c, src, prow);
        src += kGroups * 4 * kBlockBytes;
        prow += kGroups * (kStageCols / 16) * (16 * K);
    };
    if (warp < kDecodeWarps) {      // weights: before the wait for the launch that makes x
        load_codes(now, group);
        load_codes(ahead, group + kGroups);
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = ctl->tmem_base, tmem_d = tmem + kTmemD;
    asm volatile("griddepcontrol.wait;" ::: "memory");      // everything above touches weights only

    if (warp < kDecodeWarps) {
        // ---------------------------------- decode warps ------------------------------------------------
        const uint32_t lut_lane = CODE == QTIP_CODE_3INST ? mask_3inst(npad) : smem_addr(lut) + lane * 4;
        // this warp's 32 rows and 32 words of a stage (a warp reaches the 32 lanes of its index modulo four)
        const uint32_t tmem_warp = tmem + ((uint32_t)(32 * rb) << 16) + 32u * half;
        uint32_t s = group, parity = 1;                     // stage group, then group + kGroups, in turn
        for (int step = group; step < nsteps; step += kGroups) {
            const uint32_t ast = tmem_warp + s * kAStageCols;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                uint32_t wv[16];
                decode_half<K, CODE>(now, h, lut_lane, lane, wv);
                if (h == 0) {
                    // the first block is decoded before the stage is waited for; its last use was kStages steps ago (or none)
                    if (step >= kStages) mbar_wait(smem_addr(&ctl->empty[s]), parity, abort_flag, status, 1u);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    __syncwarp();
                }
                if constexpr (kHyb) {
                    tmem_st_16x128b_x4(ast + 16u * h, wv);
                    tmem_st_16x128b_x4(ast + 16u * h + (16u << 16), wv + 8);
                } else tmem_st_32x32b_x16(ast + 16u * h, wv);
            }
            now = ahead;
            load_codes(ahead, step + 2 * kGroups);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_addr(&ctl->full[s]));
            parity ^= s >= kGroups;                         // both stages have been used once more
            s = 2 * group + kGroups - s;
        }
    } else if (warp == kMmaWarp && elect_one()) {
        // ------------------------------------ MMA issue ---------------------------------------------------
        // instruction descriptor: D fp32, A/B fp16, both K-major, N = npad, M = 128
        const uint32_t idesc = (1u << 4) | ((uint32_t)(npad >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);
        int s = 0, round = 0, xs = 0, xround = 0;
        for (int step = 0; step < nsteps; step++) {
            // a wait that gave up ends the issue loop: no further MMA is started, and the commit below still
            // covers everything issued so far
            if (!mbar_wait<kMmaSleepNs>(smem_addr(&ctl->xfull[xs]), xround & 1, abort_flag, status, 4u)) break;
            if (!mbar_wait<kMmaSleepNs>(smem_addr(&ctl->full[s]), round & 1, abort_flag, status, 2u)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int tile = 0; tile < 2; tile++) {
                if (2 * step + tile < ntiles) {
                    const uint64_t bdesc = umma_desc(b_base + xs * x_stage_bytes + tile * tile_bytes);
#pragma unroll
                    for (int kk = 0; kk < 4; kk++)   // 16 columns = 32 bytes further inside the 128-byte swizzled row
                        umma_f16(tmem_d, tmem + (uint32_t)(s * kAStageCols + tile * 32 + kk * 8), bdesc + (uint64_t)(kk * 2), idesc,
                                 (step | tile | kk) != 0);
                }
            }
            umma_commit(smem_addr(&ctl->empty[s]));
            umma_commit(smem_addr(&ctl->xempty[xs]));
            if (++s == kStages) { s = 0; round++; }
            if (++xs == xstages) { xs = 0; xround++; }
        }
        umma_commit(smem_addr(&ctl->done));
    } else if (warp == kCopyWarp && elect_one()) {
        // ------------------------------------ copies of x -------------------------------------------------
        int xs = 0, xround = 0, step = 0;
        for (; step < nsteps; step++) {
            if (xround > 0 && !mbar_wait<kCopySleepNs>(smem_addr(&ctl->xempty[xs]), (xround - 1) & 1, abort_flag, status, 5u)) break;
            const uint32_t bar = smem_addr(&ctl->xfull[xs]), dst = b_base + xs * x_stage_bytes;
            const int c = c0 + step * kStageCols, tiles = min(2, ntiles - 2 * step);
            mbar_expect(bar, (uint32_t)(tiles * tile_bytes));
            copy_x_tile(dst, &xmap, c, 0, bar);
            if (tiles > 1) copy_x_tile(dst + tile_bytes, &xmap, c + kTileCols, 0, bar);
            if (++xs == xstages) { xs = 0; xround++; }
        }
        // nothing may be on its way when the CTA ends, whatever the other roles did: the last copy of each stage, with a limit
        for (int k = step - 1; k >= 0 && k >= step - xstages; k--) mbar_wait_bounded(smem_addr(&ctl->xfull[k % xstages]), (k / xstages) & 1);
    }

    if (warp < 4) {
        // ------------------------------------- epilogue ----------------------------------------------------
        mbar_wait(smem_addr(&ctl->done), 0u, abort_flag, status, 3u);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // tensor-memory lane -> row of the CTA: V = 1 codes keep row r of two tiles in lanes 2r and 2r + 1
        const int row = warp * 32 + (kHyb ? lane : 16 * (lane & 1) + (lane >> 1));
        float *part = reinterpret_cast<float *>(smem);      // [bs][128]: the ring is no longer needed (every MMA has completed)
        for (int col = 0; col < npad; col += 8) {
            uint32_t r[8];
            const uint32_t taddr = tmem_d + ((uint32_t)(warp * 32) << 16) + (uint32_t)col;
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                         : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                         : "r"(taddr)
                         : "memory");
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const int bcol = col + j;
                if (bcol < bs) {
                    const float v = __uint_as_float(r[j]);
                    if (splitk == 1) out[(size_t)bcol * m + r0 + row] = v;
                    else part[bcol * kRows + row] = v;
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == kMmaWarp) {
        // tensor memory is released only after the last commit has arrived, i.e. after every MMA that was issued has
        // completed - also on the abort path, where the epilogue warps did not wait for it
        if (lane == 0) mbar_wait_bounded(smem_addr(&ctl->done), 0u);
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
    // column splits: the cluster's CTAs add their parts in order, each its share of the outputs
    if (splitk > 1) {
        cluster_barrier();
        const int total = bs * kRows;
        const uint32_t part = smem_addr(smem);
        for (int i = (int)blockIdx.y * kGemmThreads + (int)threadIdx.x; i < total; i += splitk * kGemmThreads) {
            float v[kMaxSplit];
#pragma unroll
            for (int r = 0; r < kMaxSplit; r++)
                if (r < splitk) v[r] = cluster_load(part + i * 4u, r);
            float t = v[0];
#pragma unroll
            for (int r = 1; r < kMaxSplit; r++)
                if (r < splitk) t += v[r];
            out[(size_t)(i / kRows) * m + r0 + (i & (kRows - 1))] = t;
        }
        cluster_barrier();                                   // the parts are read
    }
}

__device__ __forceinline__ uint32_t b_tile(uint32_t base, int stage, int bytes) { return base + (uint32_t)(stage * bytes); }

// ---- more than 128 rows --------------------------------------------------------------------------------------------------
// The same roles over tiles of 128 output rows x up to 256 batch rows, fp16 results: a CTA per SM walks over the tiles (all row ranges of
// one batch group before the next), four more warps read the accumulator of a finished tile and write it.  Four stages of weights
// (tensor memory: 256 columns beside the accumulator's 256); x in a ring of single 64-column tiles.  Every batch group decodes the
// matrix again; 16 columns of a tile take the MMA 100 + 0.5 N cycles and the decode warps 140 (3INST 165, 1MAD 188; fitted, wide_cycles), so one
// group of 256 rows takes 228 where two of 128 take 328.  Measured against decode_hyb / decode_plain and
// a library product, HYB K = 2 unless stated (microseconds): 11008 x 4096 129 rows 44.7 -> 26.6, 512 rows 59.8 -> 50.7, 1000 rows
// 86.5 -> 81.1; 28672 x 8192 256 rows 214 -> 107, 512 rows 287 -> 230; K = 4 4096 x 4096 1000 rows 37.8 -> 33.1; 1MAD K = 4 8192 x 8192
// 256 rows 116 -> 56.  Bound: the MMAs (half of the tensor pipe's cycles are busy: a tensor-memory A operand takes twice the ideal interval),
// then the lookups (left out: 80.3 -> 69.6) and the copies of x (74.2); hence no sleeping between the control threads' polls here.
// Error against 64 bits at the shapes that the rule below sends here, 129 to 600 rows: the library product's to four digits (2.07e-4 to 2.10e-4 of
// the norm, 2.07e-4 of it the rounding to fp16).
constexpr int kWideN = 256, kWideStages = 4, kWideXMax = 8, kEpilogueWarp = kCopyWarp + 1;
constexpr int kWideThreads = (kEpilogueWarp + 4) * 32;

struct WideCtrl {
    unsigned long long full[kWideStages], empty[kWideStages];
    unsigned long long xfull[kWideXMax], xempty[kWideXMax];
    unsigned long long done, drained;      // the accumulator of a tile: complete; read
    uint32_t tmem_base;
    int abort_flag;
    int committed;                         // tiles whose last commit was issued
};
__host__ __device__ __forceinline__ int wide_x_stages(int npad) {
    const int fit = kXRingBytes / (npad * kTileCols * 2);
    return fit < kWideXMax ? fit : kWideXMax;
}

template <int K, int CODE>
__global__ void __launch_bounds__(kWideThreads, 1)
    decompress_gemm_wide_kernel(__half *__restrict__ out, const uint8_t *__restrict__ codes, const __grid_constant__ CUtensorMap xmap,
                                const uint32_t *__restrict__ tlut, int m, int n, int bs, int npad, int tiles, unsigned *__restrict__ status) {
    constexpr int kBlockBytes = 128 * K;
    constexpr bool kHyb = CODE == QTIP_CODE_HYB;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_addr(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t *smem = smem_raw + (base - raw);
    const int xstages = wide_x_stages(npad), xtile_bytes = npad * kTileCols * 2;
    uint32_t *lut = reinterpret_cast<uint32_t *>(smem + xstages * xtile_bytes);
    WideCtrl *ctl = reinterpret_cast<WideCtrl *>(smem + xstages * xtile_bytes + kLut512Bytes);
    volatile int *abort_flag = &ctl->abort_flag;
    const int warp = __shfl_sync(kFullMask, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    constexpr int kTmemD = kWideStages * kAStageCols, kTmemCols = 512;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kWideStages; s++) {
            mbar_init(smem_addr(&ctl->full[s]), 8);
            mbar_init(smem_addr(&ctl->empty[s]), 1);
        }
        for (int s = 0; s < kWideXMax; s++) {
            mbar_init(smem_addr(&ctl->xfull[s]), 1);
            mbar_init(smem_addr(&ctl->xempty[s]), 1);
        }
        mbar_init(smem_addr(&ctl->done), 1);
        mbar_init(smem_addr(&ctl->drained), 4);
        ctl->abort_flag = 0;
        ctl->committed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&ctl->tmem_base)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    build_table<CODE>(lut, tlut);
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = ctl->tmem_base, tmem_d = tmem + kTmemD;
    asm volatile("griddepcontrol.wait;" ::: "memory");

    const int nb = n >> 5, ntiles = n / kTileCols, nsteps = (ntiles + 1) >> 1, row_tiles = m / kRows;
    const int mine = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;      // tiles blockIdx.x, + gridDim.x, ...
    auto tile_at = [&](int i) { return (int)blockIdx.x + i * (int)gridDim.x; };

    if (warp < kDecodeWarps) {
        // the steps of all tiles in one sequence, which the groups take in turn
        const int group = warp >> 3, rb = warp & 3, half = (warp >> 2) & 1;
        const uint32_t lut_lane = CODE == QTIP_CODE_3INST ? mask_3inst(npad) : smem_addr(lut) + lane * 4;
        const uint32_t tmem_warp = tmem + ((uint32_t)(32 * rb) << 16) + 32u * half;
        int li = 0, lj = group;                             // tile and step of the next codes to be requested, and where they lie
        const uint8_t *src = nullptr;
        const uint16_t *prow = nullptr;
        auto seek = [&]() {
            while (lj >= nsteps) { lj -= nsteps; li++; }
            const int r0 = __shfl_sync(kFullMask, tile_at(li) % row_tiles * kRows, 0);
            if constexpr (kHyb) src = codes + ((size_t)(r0 / 32 + rb) * nb + 4 * lj + 2 * half) * kBlockBytes + lane * (4 * K);
            else prow = reinterpret_cast<const uint16_t *>(codes) +
                        ((size_t)(r0 / 16 + 2 * rb + (lane & 1)) * (n >> 4) + 8 * lj + 4 * half) * (16 * K) + (lane >> 1) * K;
        };
        auto load_codes = [&](StepCodes<K> &c) {
            if (lj >= nsteps) seek();
            if (li < mine && 2 * lj + half < ntiles) load_step<K, CODE>(c, src, prow);
            lj += kGroups;
            if constexpr (kHyb) src += kGroups * 4 * kBlockBytes;
            else prow += kGroups * (kStageCols / 16) * (16 * K);
        };
        seek();
        StepCodes<K> now = {}, ahead = {};
        load_codes(now);
        load_codes(ahead);
        const int total = mine * nsteps;
        for (int step = group; step < total; step += kGroups) {
            const uint32_t s = step % kWideStages;
            const uint32_t ast = tmem_warp + s * kAStageCols;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                uint32_t wv[16];
                decode_half<K, CODE>(now, h, lut_lane, lane, wv);
                if (h == 0) {
                    if (step >= kWideStages) mbar_wait(smem_addr(&ctl->empty[s]), (step / kWideStages - 1) & 1, abort_flag, status, 1u);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    __syncwarp();
                }
                if constexpr (kHyb) {
                    tmem_st_16x128b_x4(ast + 16u * h, wv);
                    tmem_st_16x128b_x4(ast + 16u * h + (16u << 16), wv + 8);
                } else tmem_st_32x32b_x16(ast + 16u * h, wv);
            }
            now = ahead;
            load_codes(ahead);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_addr(&ctl->full[s]));
        }
    } else if (warp == kMmaWarp && elect_one()) {
        const uint32_t idesc = (1u << 4) | ((uint32_t)(npad >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);
        int s = 0, round = 0, xs = 0, xround = 0;
        bool ok = true;
        for (int i = 0; i < mine && ok; i++) {
            // the accumulator of the tile before has been read
            if (i > 0 && !mbar_wait(smem_addr(&ctl->drained), (i - 1) & 1, abort_flag, status, 6u)) break;
            for (int step = 0; step < nsteps && ok; step++) {
                ok = mbar_wait(smem_addr(&ctl->full[s]), round & 1, abort_flag, status, 2u);
                for (int tile = 0; tile < 2 && ok && 2 * step + tile < ntiles; tile++) {
                    ok = mbar_wait(smem_addr(&ctl->xfull[xs]), xround & 1, abort_flag, status, 4u);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t bdesc = umma_desc(b_tile(base, xs, xtile_bytes));
#pragma unroll
                    for (int kk = 0; kk < 4; kk++)
                        umma_f16(tmem_d, tmem + (uint32_t)(s * kAStageCols + tile * 32 + kk * 8), bdesc + (uint64_t)(kk * 2), idesc,
                                 (step | tile | kk) != 0);
                    umma_commit(smem_addr(&ctl->xempty[xs]));
                    if (++xs == xstages) { xs = 0; xround++; }
                }
                umma_commit(smem_addr(&ctl->empty[s]));
                if (++s == kWideStages) { s = 0; round++; }
            }
            umma_commit(smem_addr(&ctl->done));
            ctl->committed = i + 1;
        }
    } else if (warp == kCopyWarp && elect_one()) {
        const int total = mine * ntiles;
        int xs = 0, xround = 0, k = 0, i = 0, t = 0;
        for (; k < total; k++) {
            if (xround > 0 && !mbar_wait(smem_addr(&ctl->xempty[xs]), (xround - 1) & 1, abort_flag, status, 5u)) break;
            const uint32_t bar = smem_addr(&ctl->xfull[xs]);
            mbar_expect(bar, (uint32_t)xtile_bytes);
            copy_x_tile(b_tile(base, xs, xtile_bytes), &xmap, t * kTileCols, tile_at(i) / row_tiles * npad, bar);
            if (++t == ntiles) { t = 0; i++; }
            if (++xs == xstages) { xs = 0; xround++; }
        }
        // nothing may be on its way when the CTA ends: the last copy of each stage, with a limit
        for (int j = k - 1; j >= 0 && j >= k - xstages; j--) mbar_wait_bounded(smem_addr(&ctl->xfull[j % xstages]), (j / xstages) & 1);
    } else if (warp >= kEpilogueWarp) {
        const int sub = warp & 3;                           // the tensor-memory lanes that a warp reaches: 32 sub ..
        const int row = sub * 32 + (kHyb ? lane : 16 * (lane & 1) + (lane >> 1));
        for (int i = 0; i < mine; i++) {
            const int tile = tile_at(i), r0 = tile % row_tiles * kRows, b0 = tile / row_tiles * npad, count = min(npad, bs - b0);
            if (!mbar_wait<kCopySleepNs>(smem_addr(&ctl->done), i & 1, abort_flag, status, 3u)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            __syncwarp();
            __half *dst = out + (size_t)b0 * m + r0 + row;
            for (int col = 0; col < npad; col += 16) {
                uint32_t r[16];
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                             : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                               "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                             : "r"(tmem_d + ((uint32_t)(sub * 32) << 16) + (uint32_t)col)
                             : "memory");
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (col + 16 >= npad) {                     // the last words are in registers: the next tile may begin
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_addr(&ctl->drained));
                }
#pragma unroll
                for (int j = 0; j < 16; j++)
                    if (col + j < count) dst[(size_t)(col + j) * m] = __float2half_rn(__uint_as_float(r[j]));
            }
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == kMmaWarp) {
        // tensor memory is released only after the last commit has arrived, on the abort path too (see above)
        if (lane == 0 && ctl->committed > 0) mbar_wait_bounded(smem_addr(&ctl->done), (ctl->committed - 1) & 1);
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
}

// Tensor map of x (bs, n) fp16 in boxes of npad rows x 64 columns, 128-byte swizzle
int encode_x(CUtensorMap *map, const __half *x, int n, int bs, int npad) {
    using Encode = decltype(&cuTensorMapEncodeTiled);
    static std::mutex mutex;
    static Encode encode = nullptr;
    Encode f;
    {
        std::lock_guard<std::mutex> lock(mutex);
        if (!encode) {
            void *p = nullptr;
            cudaDriverEntryPointQueryResult found;
            QTIP_CUDA_TRY(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &found));
            if (found != cudaDriverEntryPointSuccess) {
                set_last_cuda_error(cudaErrorSymbolNotFound);
                return QTIP_ERR_CUDA;
            }
            encode = reinterpret_cast<Encode>(p);
        }
        f = encode;
    }
    const cuuint64_t dims[2] = {(cuuint64_t)n, (cuuint64_t)bs}, strides[1] = {(cuuint64_t)n * sizeof(__half)};
    const cuuint32_t box[2] = {kTileCols, (cuuint32_t)npad}, step[2] = {1, 1};
    const CUresult r = f(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half *>(x), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r == CUDA_SUCCESS) return QTIP_OK;
    set_last_cuda_error(cudaErrorInvalidValue);
    return QTIP_ERR_CUDA;
}

// The launch may start while the one before it runs.  Both kernels read weights before they wait for it, so only where the caller says
// that those are settled; otherwise a plain launch (8192 x 8192, 27 rows, K = 2, after a transform: 19.7 -> 21.8 us for the two).
cudaLaunchAttribute overlap_attribute() {
    cudaLaunchAttribute a = {};
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    return a;
}

template <int K, int CODE>
int launch_gemm(float *out, const uint8_t *codes, const __half *x, const uint32_t *tlut, int m, int n, int bs, int npad,
                int splitk, unsigned *status, bool settled, cudaStream_t s) {
    const int smem = 1024 + x_stages(npad) * npad * kStageCols * 2 + kLut512Bytes + 256;
    static_assert(sizeof(GemmCtrl) <= 256 && 1024 + kXRingBytes + kLut512Bytes + 256 <= 227 * 1024, "shared memory");
    static bool attr_set[64] = {};
    static std::mutex attr_mutex;
    int dev = 0;
    QTIP_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return QTIP_ERR_BAD_ARG;
    {
        std::lock_guard<std::mutex> lock(attr_mutex);
        if (!attr_set[dev]) {
            QTIP_CUDA_TRY(cudaFuncSetAttribute(decompress_gemm_kernel<K, CODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
            attr_set[dev] = true;
        }
    }
    CUtensorMap xmap;
    const int st = encode_x(&xmap, x, n, bs, npad);
    if (st != QTIP_OK) return st;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(m / kRows, splitk);
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    cfg.attrs = attr;
    if (settled) attr[cfg.numAttrs++] = overlap_attribute();
    if (splitk > 1) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attr[cfg.numAttrs].val.clusterDim.x = 1;
        attr[cfg.numAttrs].val.clusterDim.y = splitk;
        attr[cfg.numAttrs++].val.clusterDim.z = 1;
    }
    QTIP_CUDA_TRY(cudaLaunchKernelEx(&cfg, decompress_gemm_kernel<K, CODE>, out, codes, xmap, tlut, m, n, bs, npad, splitk, status));
    return check_launch();
}

// CTAs per row range: as many as still fit the chip at once, in a cluster (at most the portable eight), each with a few steps
int column_splits(int m, int n) {
    int s = 1;
    while (s < kMaxSplit && (m / kRows) * s * 2 <= sm_count() && n / kTileCols >= 8 * s) s *= 2;
    return s;
}

// Time of a wide product on the busiest SM in cycles per 16 columns and wave of tiles: the MMA, or the decode warps.  (From timings: 11008 x 4096 129 rows
// 26.6 us, 256 rows 32.3, 1000 rows in five groups 81.1, in four 86; 8192 x 8192 129 rows 3INST 52, 1MAD 56.)
double wide_cycles(int code, int npad) { return std::max(100 + 0.5 * npad, code == QTIP_CODE_HYB ? 140.0 : code == QTIP_CODE_3INST ? 165.0 : 188.0); }
// Batch groups: as many as give the least time
int wide_groups(int code, int m, int bs, double *cost = nullptr) {
    const long row_tiles = m / kRows, sms = sm_count();
    int best = 0;
    double least = 0;
    for (int g = (bs + kWideN - 1) / kWideN; g <= (bs + 127) / 128; g++) {
        const int npad = ((bs + g - 1) / g + 15) & ~15;
        const double waves = (double)((row_tiles * ((bs + npad - 1) / npad) + sms - 1) / sms), t = waves * wide_cycles(code, npad);
        if (best == 0 || t < least) { best = g; least = t; }
    }
    if (cost) *cost = least;
    return best;
}

template <int K, int CODE>
int launch_gemm_wide(__half *out, const uint8_t *codes, const __half *x, const uint32_t *tlut, int m, int n, int bs, unsigned *status,
                     bool settled, cudaStream_t s) {
    static bool attr_set[64] = {};
    static std::mutex attr_mutex;
    int dev = 0;
    QTIP_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return QTIP_ERR_BAD_ARG;
    {
        std::lock_guard<std::mutex> lock(attr_mutex);
        if (!attr_set[dev]) {
            QTIP_CUDA_TRY(cudaFuncSetAttribute(decompress_gemm_wide_kernel<K, CODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
            attr_set[dev] = true;
        }
    }
    const int g = wide_groups(CODE, m, bs), npad = ((bs + g - 1) / g + 15) & ~15, groups = (bs + npad - 1) / npad;
    const long tiles = (long)(m / kRows) * groups;
    if (tiles >= 1L << 30) return QTIP_ERR_BAD_SHAPE;
    static_assert(sizeof(WideCtrl) <= 256, "control block");
    CUtensorMap xmap;
    const int st = encode_x(&xmap, x, n, bs, npad);
    if (st != QTIP_OK) return st;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles < sm_count() ? tiles : sm_count()));
    cfg.blockDim = dim3(kWideThreads);
    cfg.dynamicSmemBytes = 1024 + wide_x_stages(npad) * npad * kTileCols * 2 + kLut512Bytes + 256;
    cfg.stream = s;
    cudaLaunchAttribute attr = overlap_attribute();
    cfg.attrs = &attr;
    cfg.numAttrs = settled ? 1 : 0;
    QTIP_CUDA_TRY(cudaLaunchKernelEx(&cfg, decompress_gemm_wide_kernel<K, CODE>, out, codes, xmap, tlut, m, n, bs, npad, (int)tiles, status));
    return check_launch();
}
template <int CODE>
int launch_gemm_k(void *out, bool wide, const uint8_t *c, const __half *x, const uint32_t *t, int K, int m, int n, int bs, unsigned *status,
                  bool settled, cudaStream_t s) {
    if (wide) {
        auto *o = static_cast<__half *>(out);
        if (K == 2) return launch_gemm_wide<2, CODE>(o, c, x, t, m, n, bs, status, settled, s);
        if (K == 3) return launch_gemm_wide<3, CODE>(o, c, x, t, m, n, bs, status, settled, s);
        return launch_gemm_wide<4, CODE>(o, c, x, t, m, n, bs, status, settled, s);
    }
    auto *o = static_cast<float *>(out);
    const int npad = (bs + 15) & ~15, splitk = column_splits(m, n);
    if (K == 2) return launch_gemm<2, CODE>(o, c, x, t, m, n, bs, npad, splitk, status, settled, s);
    if (K == 3) return launch_gemm<3, CODE>(o, c, x, t, m, n, bs, npad, splitk, status, settled, s);
    return launch_gemm<4, CODE>(o, c, x, t, m, n, bs, npad, splitk, status, settled, s);
}

int gemm(void *out, bool wide, const void *codes, const void *x, const void *tlut, int code, int K, int m, int n, int bs, unsigned *status,
         bool settled, void *stream) {
    if (!out || !codes || !x || !status || K < 2 || K > 4 || bs < 1 || (!wide && bs > kMaxN)) return QTIP_ERR_BAD_ARG;
    if (code != QTIP_CODE_HYB && code != QTIP_CODE_3INST && code != QTIP_CODE_1MAD) return QTIP_ERR_BAD_ARG;
    if (code == QTIP_CODE_HYB && !tlut) return QTIP_ERR_BAD_ARG;
    if (m <= 0 || n <= 0 || (m % kRows) || (n % kTileCols)) return QTIP_ERR_BAD_SHAPE;
    if ((long)(m >> 5) * (n >> 5) >= (1L << 30)) return QTIP_ERR_BAD_SHAPE;
    if (!aligned(codes, 16) || !aligned(x, 16) || !aligned(out, wide ? 2 : 4) || (tlut && !aligned(tlut, 4)) || !aligned(status, 4))
        return QTIP_ERR_ALIGNMENT;
    auto *c = static_cast<const uint8_t *>(codes);
    auto *xh = static_cast<const __half *>(x);
    auto *t = static_cast<const uint32_t *>(tlut);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (code == QTIP_CODE_HYB) return launch_gemm_k<QTIP_CODE_HYB>(out, wide, c, xh, t, K, m, n, bs, status, settled, s);
    if (code == QTIP_CODE_3INST) return launch_gemm_k<QTIP_CODE_3INST>(out, wide, c, xh, nullptr, K, m, n, bs, status, settled, s);
    return launch_gemm_k<QTIP_CODE_1MAD>(out, wide, c, xh, nullptr, K, m, n, bs, status, settled, s);
}

}  // namespace
}  // namespace qtip

using namespace qtip;

extern "C" int qtip_decompress_gemm(float *out, const void *codes, const void *x, const void *tlut, int K, int m, int n, int bs,
                                    unsigned *status, void *stream) {
    return gemm(out, false, codes, x, tlut, QTIP_CODE_HYB, K, m, n, bs, status, false, stream);
}

extern "C" int qtip_decompress_gemm_plain(float *out, const void *codes, const void *x, int code, int K, int m, int n, int bs,
                                          unsigned *status, void *stream) {
    if (code == QTIP_CODE_HYB) return QTIP_ERR_BAD_ARG;
    return gemm(out, false, codes, x, nullptr, code, K, m, n, bs, status, false, stream);
}

extern "C" int qtip_decompress_gemm_f16(void *out, const void *codes, const void *x, const void *tlut, int code, int K, int m, int n, int bs,
                                        unsigned *status, void *stream) {
    return gemm(out, true, codes, x, tlut, code, K, m, n, bs, status, false, stream);
}

extern "C" int qtip_decompress_gemm_settled(void *out, int out_dtype, const void *codes, const void *x, const void *tlut, int code, int K, int m,
                                            int n, int bs, unsigned *status, void *stream) {
    if (out_dtype != QTIP_F16 && out_dtype != QTIP_F32) return QTIP_ERR_BAD_ARG;
    return gemm(out, out_dtype == QTIP_F16, codes, x, tlut, code, K, m, n, bs, status, true, stream);
}

// Rule: estimates of both ways in microseconds.  Wide: 6 to start and end, the cycles above at 1.965 GHz.  Dense: 5 for the launches, the
// decode at its write rate (3.9 TB/s HYB, settled weights, 2.8 3INST, 1.6 1MAD), the product at the rate of reading the matrix (4.2 TB/s) or 1430 TFLOP/s.
// Products of several hundred microseconds run at the power cap (28672 x 8192, 1000 rows: 400 to 458 us in three runs, dense 432 to 450): 10 % more.
// It errs by up to 10 %, on either side of the line (4096 x 4096: dense up to 512 rows, 26.2 against 27.0 us; 11008 x 4096: wide up to about 2000).
extern "C" int qtip_decompress_gemm_f16_faster(int code, int m, int n, int bs) {
    if (m <= 0 || n <= 0 || bs < 1 || (m % kRows) || (n % kTileCols)) return 0;
    double cycles;
    wide_groups(code, m, bs, &cycles);
    const double bytes = 2.0 * m * n;
    double wide = 6 + cycles * (n / 16) / 1965;
    if (wide > 300) wide *= 1.1;
    const double write = code == QTIP_CODE_HYB ? 3.9e6 : code == QTIP_CODE_3INST ? 2.8e6 : 1.6e6;
    const double dense = 5 + bytes / write + std::max(bytes / 4.2e6, bytes * bs / 1.43e9);
    return wide < dense;
}
