// Viterbi quantizer over the bitshift trellis with tail-biting: the encoder that produces the trellis states the
// decoders of this library consume (bitshift_codebook.quantize upstream, lib/codebook/bitshift.py:203-292).
//
// A sequence of T values is quantized to S = T/V states of L = 16 bits, consecutive states overlapping by 16 - KV bits
// (KV = K*V).  Upstream keeps one cost per state (2^16 floats per sequence and step) and, per step, gathers the
// 2^KV predecessors of every group of states that share them.  Here the cost vector is never materialised:
//     cost_i[p] = err_i(p) + best_i[p >> KV],      best_{i+1}[g] = min over d of cost_i[g + d * G],   G = 2^(16-KV)
// so the dynamic-programming state of a sequence is the G values best_i and lives in shared memory.  The arithmetic is
// upstream's, operation for operation in fp32 with round-to-nearest and no contraction (subtract, square, add over v, add
// best), so every cost is upstream's bit for bit.  Tail-biting as upstream: a first pass over the sequence rolled by half
// its length with free ends yields the 16 - KV bits where the original sequence starts; the second pass forces its first
// state to begin and its last state to end with them.
//
// The forward passes keep VALUES only: 65536 candidates per step, and a compare-and-select of the winning index would
// cost more than everything else a candidate needs.  Instead best_i is written to the workspace every `stride` steps by an
// asynchronous bulk copy, and the back-trace (one warp) recomputes the few candidates that lead to the state it is at: the
// 2^(KV*k) leaves of a tree k <= stride steps deep, combined with "the lower index wins ties" = torch.min's first minimal
// index, so the chosen states are identical to upstream's, not merely equally good.
//
// HYB forward.  The code's error takes only 1024 values per step (512 table entries x the sign), so they are computed
// once per step into a table E and a candidate is one lookup and one add.  Three properties of the hash h(p) = p*(p+1) mod
// 2^16, entry(p) = h >> 6, make the lookup cheap:
//   h(65535 - p) = h(p): one lookup serves two candidates (p and its complement);
//   entry(p + 64 l) mod 32 runs through all 32 values for l = 0..31: with lane l at p = y + 64 l + 2048 u the lookups of a
//     warp fall into 32 different banks, whatever y and u;
//   entry(y + 64 l + 2048 u) = entry(y + 64 l) + 32 * (u * (2y + 1) mod 32), wrapping in the upper five bits: with y mod 16
//     known at compile time and the table repeated once the address is register + immediate.
// best_i is stored under an XOR permutation of its index (pos()) that makes both the reads (stride 4 or 1 in lanes) and the
// writes (stride 64) conflict-free.  Four warps per sequence, four sequences per SM.  Bound: shared-memory wavefronts (32768
// lookups = 1024 wavefronts per step and sequence, plus reads of best) and issue (2.0 warp instructions per 32
// candidates, everything included), close to each other.
// 3INST / 1MAD forward.  65536 (1021) different values, so each candidate computes its error: LCG by constant increments,
// two values per packed fp32x2 instruction, minimum of three per instruction; issue bound at about 6.5 instructions per
// candidate.
//
// Measured on 4096 sequences of 256 values, milliseconds, before (index kept per candidate, byte back-pointers, 1024 threads
// per sequence) -> now:  HYB K=2 50.8 -> 7.0, 3INST K=2 98 -> 42, 1MAD K=2 97 -> 49.  HYB spends 1500 shared-memory
// wavefronts per step and sequence in 1700 cycles; the compute codes keep the fp32 / integer multiply pipe 80 % busy.
// Memory: the stored rows of every sequence in flight, at 256 values 1 / 1 / 0.25 MiB (HYB, K = 2 / 3 / 4) and 4 / 4 / 2 MiB (compute
// codes); with a full grid on 148 SMs 592 / 592 / 148 and 592 / 1184 / 592 MiB, where byte back-pointers of one sequence per SM took
// 74 / 18.5 / 4.6 and 592 / 296 / 148.
// Waits: CTA barriers, the bulk-store groups of thread 0, and the bounded waits of the back-trace (see there).
#include <climits>

#include "common.cuh"

namespace qtip {
namespace {

constexpr int kMaxT = 1024;
constexpr uint32_t kMaxSlots = 8;             // rows in flight during the back-trace
constexpr uint32_t kRowPolls = 1u << 20;      // polls of a wait for a row, and of each wait for what is in flight after one ran out
constexpr uint32_t kGivenUp = 0xFFFFFFFFu;    // no state and no overlap

// Threads per sequence, resident sequences per SM and steps between stored rows, per code and KV.
template <int CODE, int KV>
struct VitCfg {
    static constexpr bool kHyb = CODE == QTIP_CODE_HYB;
    static constexpr int kV = kHyb ? 2 : 1;
    static constexpr uint32_t G = 65536u >> KV, D = 1u << KV, Gs = G >> KV;      // (g + d*G) >> KV = (g >> KV) + d*Gs
    // HYB, KV > 4: a group's candidates split into a direct and a complemented half held by different warps; each writes
    // its own array and the minimum of the two is taken when best is read
    static constexpr int kHalves = kHyb && KV > 4 ? 2 : 1;
    static constexpr int kThreads = kHyb ? 128 : 512;
    // stored rows: a tree of `stride` steps has at most 2^8 leaves, eight per lane of the back-tracing warp
    static constexpr int kStride = 8 / KV;
    // HYB 4 x 54 KiB; compute codes: two cost buffers of 64 / 32 / 16 KiB
    static constexpr int kPerSm = kHyb ? 4 : (KV == 2 ? 1 : 2);
    static constexpr uint32_t kRowFloats = G * kHalves;
    // row slots of the back-trace: the two buffers of best and, HYB, the two error tables behind them
    static constexpr uint32_t kFit = (2 * kRowFloats * 4 + (kHyb ? 2 * 8192 : 0)) / (kRowFloats * 4);
    static constexpr uint32_t kSlots = kFit < kMaxSlots ? kFit : kMaxSlots;
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
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
__device__ __forceinline__ float lds(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}
template <int OFF>
__device__ __forceinline__ float lds_off(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1+%2];" : "=f"(v) : "r"(a), "n"(OFF));
    return v;
}
template <int OFF>
__device__ __forceinline__ void sts_off(uint32_t a, float v) {
    asm volatile("st.shared.f32 [%0+%1], %2;" ::"r"(a), "n"(OFF), "f"(v) : "memory");
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// packed fp32 pairs: each half rounds exactly like the scalar instruction
struct f2 { float x, y; };
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 d;
    asm("{\n\t.reg .b64 p, q;\n\tmov.b64 p, {%2, %3};\n\tmov.b64 q, {%4, %5};\n\tadd.rn.f32x2 p, p, q;\n\tmov.b64 {%0, %1}, p;\n\t}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 d;
    asm("{\n\t.reg .b64 p, q, r;\n\tmov.b64 p, {%2, %3};\n\tmov.b64 q, {%4, %5};\n\tmov.b64 r, {%6, %7};\n\tfma.rn.f32x2 p, p, q, r;\n\tmov.b64 {%0, %1}, p;\n\t}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}

// Word position of best[q] in its array (linear over XOR of index bits).  HYB: reads vary index bits 2..6 (KV = 4), 0..4
// (KV = 6), 0..2 (KV = 8) over the lanes of a warp, writes vary bits 6..10, 6..9, 6..7: the bank (low five bits) is the
// XOR of the two fields.
template <int CODE, int KV>
__host__ __device__ __forceinline__ constexpr uint32_t pos(uint32_t q) {
    if (CODE != QTIP_CODE_HYB) return q;
    if (KV == 4) {
        const uint32_t bank = (((q >> 2) ^ (q >> 7)) & 15u) | (((q >> 6) & 1u) << 4);
        return bank | ((q & 3u) << 5) | ((q >> 7) << 7);
    }
    if (KV == 6) return q ^ (q >> 6);
    return q ^ (q >> 6);
}

// reconstruction of state p: r0 (and r1 for V = 2), upstream's recons_state[:, p].  `tl` is the code's table in shared
// memory: HYB the 512 x 2 fp32 LUT; 1MAD the 1021 possible values (byte sum - 510) / 147.800537109375; 3INST needs none.
// Used where single candidates are evaluated (final step, back-trace).
template <int CODE>
__device__ __forceinline__ float err_of(uint32_t p, uint32_t tl, float x0, float x1) {
    float r0, r1 = 0.f;
    if constexpr (CODE == QTIP_CODE_HYB) {
        const uint32_t h = hyb_hash(p);
        float vx, vy;
        asm("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(vx), "=f"(vy) : "r"(tl + ((h >> 3) & 0xFF8u)));    // entry (h >> 6) & 511
        // quantlut_sym multiplies the first value by -1 when bit 15 of the hash is set: flip the sign bit
        r0 = __uint_as_float(__float_as_uint(vx) ^ ((h << 16) & 0x80000000u));
        r1 = vy;
    } else if constexpr (CODE == QTIP_CODE_3INST) {
        r0 = __half2float(decode_3inst(p));
    } else {
        const uint32_t x = p * 34038481u + 76625530u;
        asm("ld.shared.f32 %0, [%1];" : "=f"(r0) : "r"(tl + __vsadu4(x, 0u) * 4u));
    }
    const float d0 = __fsub_rn(r0, x0);
    float e = __fmul_rn(d0, d0);
    if constexpr (CODE == QTIP_CODE_HYB) {
        const float d1 = __fsub_rn(r1, x1);
        e = __fadd_rn(e, __fmul_rn(d1, d1));
    }
    return e;
}

struct __align__(16) Smem {    // sizeof is a multiple of 16: bulk copies and vector accesses follow it
    float red_v[32];
    uint32_t red_i[32];
    unsigned long long bar[kMaxSlots];
    uint32_t arg;
};

template <int CODE, int KV>
__device__ __forceinline__ float best_at(const float *row, uint32_t q) {     // a stored row or a shared-memory array
    using C = VitCfg<CODE, KV>;
    float b = row[pos<CODE, KV>(q)];
    if constexpr (C::kHalves == 2) b = fminf(b, row[C::G + pos<CODE, KV>(q)]);
    return b;
}

// Everything a pass needs that does not change within a launch.
struct PassCtx {
    const float *x;        // the sequence in shared memory (fp32)
    float *buf0, *buf1;    // best_i ping-pong, kRowFloats each
    uint32_t etab;         // HYB: two error tables of 2048 floats
    uint32_t tl;           // the code's value table
    float *rows;           // this CTA's slab: rows of best_i, i = 0, stride, 2 stride ...
    int T;
    float minus_zero;      // -0.0f as a run-time value (see v1_errors)
    uint32_t row_polls;
};

__device__ __forceinline__ void bulk_store(void *dst, uint32_t src, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

// index of the values that step i of a pass reads
template <int V>
__device__ __forceinline__ int x_index(int i, int xoff, int T) {
    const int t = i * V + xoff;       // T and xoff are multiples of V, xoff <= T
    return t >= T ? t - T : t;
}

// ---- HYB: one step ------------------------------------------------------------------------------------------------
// Error table of a step: entry e (10 bits: sign << 9 | index) at words e and e + 1024 (repeated so that the wrap of the
// upper five bits needs no arithmetic).  Thread t owns entries t + 128k; its four table rows stay in registers.
__device__ __forceinline__ void hyb_build_errors(uint32_t tab, const float2 (&lut)[4], float x0, float x1) {
    const uint32_t a = tab + threadIdx.x * 4u;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float d1 = __fsub_rn(lut[k].y, x1), s1 = __fmul_rn(d1, d1);
        const float dp = __fsub_rn(lut[k].x, x0), dn = __fsub_rn(-lut[k].x, x0);
        const float ep = __fadd_rn(__fmul_rn(dp, dp), s1), en = __fadd_rn(__fmul_rn(dn, dn), s1);
        asm volatile("st.shared.f32 [%0], %1;\n\tst.shared.f32 [%0+4096], %1;" ::"r"(a + k * 512u), "f"(ep) : "memory");
        asm volatile("st.shared.f32 [%0], %1;\n\tst.shared.f32 [%0+4096], %1;" ::"r"(a + k * 512u + 2048u), "f"(en) : "memory");
    }
}

// Minimum over the 16 candidates of one residue y = 16x + J and their complements: e[i] = E(entry of u = us*i), direct
// candidates add bd[i], complemented ones bm[i].
template <int J, int US>
__device__ __forceinline__ void hyb_residue(uint32_t ebase, const float (&bd)[16], const float (&bm)[16], float &md, float &mm) {
    constexpr uint32_t m = 2u * J + 1u;
    float e[16];
    e[0] = lds_off<128 * ((0u * US * m) & 31u)>(ebase);   e[1] = lds_off<128 * ((1u * US * m) & 31u)>(ebase);
    e[2] = lds_off<128 * ((2u * US * m) & 31u)>(ebase);   e[3] = lds_off<128 * ((3u * US * m) & 31u)>(ebase);
    e[4] = lds_off<128 * ((4u * US * m) & 31u)>(ebase);   e[5] = lds_off<128 * ((5u * US * m) & 31u)>(ebase);
    e[6] = lds_off<128 * ((6u * US * m) & 31u)>(ebase);   e[7] = lds_off<128 * ((7u * US * m) & 31u)>(ebase);
    e[8] = lds_off<128 * ((8u * US * m) & 31u)>(ebase);   e[9] = lds_off<128 * ((9u * US * m) & 31u)>(ebase);
    e[10] = lds_off<128 * ((10u * US * m) & 31u)>(ebase); e[11] = lds_off<128 * ((11u * US * m) & 31u)>(ebase);
    e[12] = lds_off<128 * ((12u * US * m) & 31u)>(ebase); e[13] = lds_off<128 * ((13u * US * m) & 31u)>(ebase);
    e[14] = lds_off<128 * ((14u * US * m) & 31u)>(ebase); e[15] = lds_off<128 * ((15u * US * m) & 31u)>(ebase);
    md = mm = INFINITY;
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
        const f2 ep = {e[i], e[i + 1]};
        const f2 a = add2(ep, f2{bd[i], bd[i + 1]}), b = add2(ep, f2{bm[i], bm[i + 1]});
        if (i == 0) { md = fminf(a.x, a.y); mm = fminf(b.x, b.y); }
        else { md = min3(md, a.x, a.y); mm = min3(mm, b.x, b.y); }
    }
}

// The per-thread constants of the HYB forward: warp w handles residues y = 16w + j, lane l the states y + 64l + 2048u.
template <int KV>
struct HybThread {
    uint32_t ebase[16];    // byte offset of entry(y + 64 l) in the error table, j = 0..15
    uint32_t rd, rm;       // byte offset of best[q], q = (y + 64 l) >> KV, and of its complement G - 1 - q
    uint32_t wd, wm;       // byte offset of best[g], g = (16w + 64 l) mod G (j = 0), and of its complement
};

template <int KV, int J>
__device__ __forceinline__ void hyb_residues(const HybThread<KV> &t, uint32_t etab, uint32_t nxt, const float (&bd)[16], const float (&bm)[16]) {
    if constexpr (J < 16) {
        using C = VitCfg<QTIP_CODE_HYB, KV>;
        float md, mm;
        hyb_residue<J, KV == 4 ? 2 : 1>(etab + t.ebase[J], bd, bm, md, mm);
        // group g = (y + 64 l) mod G and its complement; j enters the position by XOR in the bank bits and, above them, by
        // addition (the bits are 0 in wd) or subtraction (1 in the complement)
        constexpr uint32_t pj = pos<QTIP_CODE_HYB, KV>(J) * 4u, bank = pj & 127u;
        constexpr int rest = (int)(pj & ~127u);
        const int lane = threadIdx.x & 31;
        if constexpr (KV == 4) {
            sts_off<rest>(nxt + (t.wd ^ bank), md);
            sts_off<-rest>(nxt + (t.wm ^ bank), mm);
        } else {
            // lanes that share a group (the lane bits above the group's) hold different d: combine them
            constexpr int kGroupLanes = KV == 6 ? 16 : 4;
#pragma unroll
            for (int o = kGroupLanes; o < 32; o <<= 1) {
                md = fminf(md, __shfl_xor_sync(kFullMask, md, o));
                mm = fminf(mm, __shfl_xor_sync(kFullMask, mm, o));
            }
            if (lane < kGroupLanes) {
                sts_off<rest>(nxt + (t.wd ^ bank), md);                            // first array: direct candidates
                sts_off<(int)(C::G * 4u) - rest>(nxt + (t.wm ^ bank), mm);         // second: complemented ones
            }
        }
        hyb_residues<KV, J + 1>(t, etab, nxt, bd, bm);
    }
}

template <int KV>
__device__ __forceinline__ void hyb_step(const HybThread<KV> &t, uint32_t etab, uint32_t cur, uint32_t nxt) {
    using C = VitCfg<QTIP_CODE_HYB, KV>;
    // best of the 16 direct predecessors q + i*qs and of their complements, shared by all residues of the thread
    constexpr uint32_t qs = KV == 4 ? 256u : (KV == 6 ? 32u : 8u);
    float bd[16], bm[16];
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const uint32_t pi = pos<QTIP_CODE_HYB, KV>((uint32_t)i * qs) * 4u, bank = pi & 127u, rest = pi & ~127u;
        const uint32_t ad = cur + (t.rd ^ bank) + rest, am = cur + (t.rm ^ bank) - rest;
        bd[i] = lds(ad);
        bm[i] = lds(am);
        if constexpr (C::kHalves == 2) {
            bd[i] = fminf(bd[i], lds(ad + C::G * 4u));
            bm[i] = fminf(bm[i], lds(am + C::G * 4u));
        }
    }
    hyb_residues<KV, 0>(t, etab, nxt, bd, bm);
}

// ---- 3INST / 1MAD: one step ---------------------------------------------------------------------------------------
// Squared errors of the four states whose LCG values are x, x + A, x + 2A, x + 3A; nx = (-x0, -x0).
constexpr uint32_t k3instA = 89226354u, k3instB = 64248484u, k1madA = 34038481u, k1madB = 76625530u;
template <int CODE>
__device__ __forceinline__ void v1_errors(uint32_t x, f2 nx, float minus_zero, f2 (&e)[2]) {
    f2 r[2];
    float *rs = reinterpret_cast<float *>(r);
    if constexpr (CODE == QTIP_CODE_3INST) {
        // 0x8FFF8FFF, made at run time: a three-input logic instruction takes one literal, with two it becomes two instructions (K = 3 and 4
        // 3 % faster, K = 2 the same)
        const uint32_t mask = __float_as_uint(minus_zero) | 0x0FFF8FFFu;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            uint32_t v = ((x + (uint32_t)j * k3instA) & mask) ^ 0x3B603B60u;
            const __half2 h = *reinterpret_cast<__half2 *>(&v);
            rs[j] = __half2float(__hadd(__low2half(h), __high2half(h)));
        }
    } else {
        // byte sum as an exact float through the exponent trick (2^23 + sum), then (sum - 510) / 147.8005... with the
        // IEEE quotient from a rounded reciprocal and one exact residual (P. Markstein, "Computation of elementary
        // functions on the IBM RISC System/6000 processor", 1990); all 1021 sums are checked against the quotient
        // on the CPU and by the bit-exact state tests
        constexpr float c = 147.800537109375f, rc = 1.0f / 147.800537109375f;
#pragma unroll
        for (int j = 0; j < 4; j++) rs[j] = __uint_as_float(__dp4a(x + (uint32_t)j * k1madA, 0x01010101u, 0x4B000000u));
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const f2 y = add2(r[h], f2{-8389118.0f, -8389118.0f}), q = fma2(y, f2{rc, rc}, f2{-0.0f, -0.0f});
            r[h] = fma2(fma2(f2{-q.x, -q.y}, f2{c, c}, y), f2{rc, rc}, q);
        }
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const f2 d = add2(r[h], nx);
        // the square, rounded on its own: ptxas merges a packed multiply (and an fma with a literal -0) with the packed add
        // that follows in spite of .rn, but not an fma whose addend it cannot see
        e[h] = fma2(d, d, f2{minus_zero, minus_zero});
    }
}

// A thread owns four consecutive groups at a time: they share their predecessors' best values, and the result is one
// 16-byte store.
template <int CODE, int KV>
__device__ __forceinline__ void v1_step(const float *cur, float *nxt, float x0, float minus_zero) {
    using C = VitCfg<CODE, KV>;
    constexpr uint32_t A = CODE == QTIP_CODE_3INST ? k3instA : k1madA, B = CODE == QTIP_CODE_3INST ? k3instB : k1madB;
    const f2 nx = {-x0, -x0};
    static_assert(C::G % (4 * C::kThreads) == 0, "whole trips");
#pragma unroll 1
    for (uint32_t g = 4 * threadIdx.x; g < C::G; g += 4 * C::kThreads) {
        const uint32_t xg = g * A + B;
        const float *b = cur + (g >> KV);
        f2 m[2];
#pragma unroll
        for (uint32_t d = 0; d < C::D; d += 2) {
            f2 e0[2], e1[2];
            v1_errors<CODE>(xg + d * (C::G * A), nx, minus_zero, e0);
            v1_errors<CODE>(xg + (d + 1) * (C::G * A), nx, minus_zero, e1);
            const float b0 = b[d * C::Gs], b1 = b[(d + 1) * C::Gs];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const f2 c0 = add2(e0[h], f2{b0, b0}), c1 = add2(e1[h], f2{b1, b1});
                if (d == 0) m[h] = f2{fminf(c0.x, c1.x), fminf(c0.y, c1.y)};
                else m[h] = f2{min3(m[h].x, c0.x, c1.x), min3(m[h].y, c0.y, c1.y)};
            }
        }
        *reinterpret_cast<float4 *>(nxt + g) = make_float4(m[0].x, m[0].y, m[1].x, m[1].y);
    }
}

// ---- one pass of upstream's viterbi() -----------------------------------------------------------------------------
// Forward dynamic programming over the sequence read at offset xoff (the rolled sequence of the first pass); rows of best_i
// from step row_min on are stored for the back-trace.  Leaves the first minimal final state in sh->arg.
template <int CODE, int KV, class ThreadState>
__device__ __forceinline__ void viterbi_forward(Smem *sh, const PassCtx &P, const ThreadState &ts, const float2 (&lut)[4], int xoff,
                                                bool has_overlap, uint32_t overlap, int row_min, float *final_cost) {
    using C = VitCfg<CODE, KV>;
    constexpr int V = C::kV;
    const int S = P.T / V;
    const int tid = threadIdx.x;
    // best_0: adding 0 leaves the first step's error as it is; with an overlap only the states whose top bits equal it
    // may start the walk (upstream: min(cost + mask, inf))
    for (uint32_t q = tid; q < C::G; q += C::kThreads) {
        P.buf0[pos<CODE, KV>(q)] = (!has_overlap || q == overlap) ? 0.f : INFINITY;
        if constexpr (C::kHalves == 2) P.buf0[C::G + q] = INFINITY;
    }
    if constexpr (C::kHyb) {
        const int t0 = x_index<V>(0, xoff, P.T);
        hyb_build_errors(P.etab, lut, P.x[t0], P.x[t0 + 1]);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    float *cur = P.buf0, *nxt = P.buf1;
    for (int i = 0; i + 1 < S; i++) {
        if (tid == 0 && i % C::kStride == 0 && i >= row_min)
            bulk_store(P.rows + (size_t)(i / C::kStride) * C::kRowFloats, smem_u32(cur), C::kRowFloats * 4u);
        if constexpr (C::kHyb) {
            const int t1 = x_index<V>(i + 1, xoff, P.T);
            hyb_build_errors(P.etab + ((i + 1) & 1) * 8192u, lut, P.x[t1], P.x[t1 + 1]);
            hyb_step<KV>(ts, P.etab + (i & 1) * 8192u, smem_u32(cur), smem_u32(nxt));
        } else {
            v1_step<CODE, KV>(cur, nxt, P.x[x_index<V>(i, xoff, P.T)], P.minus_zero);
        }
        // the next step overwrites `cur`: its copy must have been read; the row stored next must be visible to the copy
        if ((i + 1) % C::kStride == 0) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        __syncthreads();
        float *t = cur; cur = nxt; nxt = t;
    }
    // final costs: err_{S-1}(s) + best_{S-1}[s >> KV], over the states that end with the overlap bits; first minimum
    const int tl = x_index<V>(S - 1, xoff, P.T);
    const float x0 = P.x[tl], x1 = V == 2 ? P.x[tl + 1] : 0.f;
    float bv = INFINITY;
    uint32_t bi = 0xFFFFFFFFu;
    const uint32_t count = has_overlap ? C::D : 65536u;
    for (uint32_t k = tid; k < count; k += C::kThreads) {
        const uint32_t s = has_overlap ? overlap + k * C::G : k;
        const float c = __fadd_rn(err_of<CODE>(s, P.tl, x0, x1), best_at<CODE, KV>(cur, s >> KV));
        if (bi == 0xFFFFFFFFu || c < bv) { bv = c; bi = s; }
    }
    auto reduce = [&]() {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(kFullMask, bv, o);
            const uint32_t oi = __shfl_xor_sync(kFullMask, bi, o);
            if (ov < bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
        }
    };
    reduce();
    if ((tid & 31) == 0) { sh->red_v[tid >> 5] = bv; sh->red_i[tid >> 5] = bi; }
    __syncthreads();
    if (tid < 32) {
        const int warps = C::kThreads / 32;
        bv = tid < warps ? sh->red_v[tid] : INFINITY;
        bi = tid < warps ? sh->red_i[tid] : 0xFFFFFFFFu;
        reduce();
        if (tid == 0) {
            sh->arg = bv < INFINITY ? bi : 0u;     // no reachable end (infinite inputs): the first of equals
            if (final_cost) *final_cost = bv;
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");       // the stored rows are complete
        }
    }
    asm volatile("fence.proxy.async;" ::: "memory");
    __syncthreads();
}

// One tree of the back-trace: from state st at step i to the best of the 2^(KV*k) paths that lead into it from the row of
// best_{i-k}.  Candidate c = the choices' digits, latest step most significant; lane l evaluates c = 8l .. 8l+7.  Minima are
// taken bit by bit from the lowest (earliest) digit up, the lower index winning ties, and the error of a step is added when
// its digit is complete - the recursion of the forward pass.  Returns the winning c (same in all lanes).
template <int KV>
__device__ __forceinline__ uint32_t path_state(uint32_t st, uint32_t c, int k, int t) {      // the state t steps back
    constexpr uint32_t G = 65536u >> KV, D = 1u << KV;
    uint32_t p = st;
#pragma unroll
    for (int q = 1; q <= t; q++) p = (p >> KV) + ((c >> (KV * (k - q))) & (D - 1u)) * G;
    return p;
}
template <int CODE, int KV, int k, class Row>
__device__ __forceinline__ uint32_t trace_tree(const PassCtx &P, uint32_t st, int i, int xoff, const Row &row) {
    constexpr int V = VitCfg<CODE, KV>::kV, n = k * KV;
    const int lane = threadIdx.x & 31;
    float xs[k + 1][2];
#pragma unroll
    for (int t = 1; t <= k; t++) {
        const int tx = x_index<V>(i - t, xoff, P.T);
        xs[t][0] = P.x[tx];
        xs[t][1] = V == 2 ? P.x[tx + 1] : 0.f;
    }
    float val[8];
    uint32_t idx[8];
#pragma unroll
    for (int r = 0; r < 8; r++) {
        idx[r] = (uint32_t)(lane * 8 + r) & ((1u << n) - 1u);      // lanes beyond the tree repeat it and are ignored
        const uint32_t p = path_state<KV>(st, idx[r], k, k);
        val[r] = __fadd_rn(err_of<CODE>(p, P.tl, xs[k][0], xs[k][1]), row(p >> KV));
    }
#pragma unroll
    for (int bit = 0; bit < n; bit++) {
        if (bit < 3) {
#pragma unroll
            for (int r = 0; r < (8 >> (bit + 1)); r++) {
                const bool hi = val[2 * r + 1] < val[2 * r];
                idx[r] = hi ? idx[2 * r + 1] : idx[2 * r];
                val[r] = hi ? val[2 * r + 1] : val[2 * r];
            }
        } else {
            const int o = 1 << (bit - 3);
            const float ov = __shfl_xor_sync(kFullMask, val[0], o);
            const uint32_t oi = __shfl_xor_sync(kFullMask, idx[0], o);
            const bool take = (lane & o) ? (ov <= val[0]) : (ov < val[0]);
            if (take) { val[0] = ov; idx[0] = oi; }
        }
        if ((bit + 1) % KV == 0 && bit + 1 < n) {
            const int t = k - (bit + 1) / KV;
#pragma unroll
            for (int r = 0; r < (bit < 3 ? (8 >> (bit + 1)) : 1); r++)
                val[r] = __fadd_rn(err_of<CODE>(path_state<KV>(st, idx[r], k, t), P.tl, xs[t][0], xs[t][1]), val[r]);
        }
    }
    return __shfl_sync(kFullMask, idx[0], 0);
}
template <int CODE, int KV, int k, class Row>
__device__ __forceinline__ uint32_t trace_tree_of_depth(int depth, const PassCtx &P, uint32_t st, int i, int xoff, const Row &row) {
    if constexpr (k == 1) return trace_tree<CODE, KV, 1>(P, st, i, xoff, row);
    else {
        if (depth == k) return trace_tree<CODE, KV, k>(P, st, i, xoff, row);
        return trace_tree_of_depth<CODE, KV, k - 1>(depth, P, st, i, xoff, row);
    }
}

// Back-trace by one warp: from state st at step i_from to the state at step i_stop (returned); states of the steps in
// between (i_stop included) go to out[step] if out is given.  The stored rows are streamed back through the shared memory
// that the forward pass no longer needs (kSlots rows in flight): a chain of dependent reads from global memory took
// 2.4 us per tree, 0.23 ms of a sequence's 0.6.  (cp.async groups, which need no polling, take the shared-memory pipe that the
// forward passes of the other CTAs are bound by: 4096 HYB sequences 7.07 -> 7.19 ms with one warp copying, 7.30 with all.)
// The waits are bounded: when one runs out nothing of the row is used, the rows still in flight are waited for, and kGivenUp is
// returned.
template <int CODE, int KV>
__device__ __forceinline__ uint32_t backtrace(Smem *sh, const PassCtx &P, uint32_t st, int i_from, int i_stop, int xoff, int *out) {
    using C = VitCfg<CODE, KV>;
    constexpr uint32_t kRowBytes = C::kRowFloats * 4u;
    const int lane = threadIdx.x & 31;
    const int r_first = (i_from - 1) / C::kStride, r_last = i_stop / C::kStride;      // rows used, descending
    const uint32_t slots = smem_u32(P.buf0), bars = smem_u32(sh->bar);
    auto fetch = [&](int r) {          // row r into its slot
        const uint32_t s = (uint32_t)(r_first - r) % C::kSlots;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bars + 8 * s), "r"(kRowBytes) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(slots + s * kRowBytes),
                     "l"(P.rows + (size_t)r * C::kRowFloats), "r"(kRowBytes), "r"(bars + 8 * s) : "memory");
    };
    if (lane == 0) {
        for (uint32_t s = 0; s < C::kSlots; s++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bars + 8 * s));
        asm volatile("fence.mbarrier_init.release.cluster;\n\tfence.proxy.async;" ::: "memory");
        for (int r = r_first; r >= r_last && r > r_first - (int)C::kSlots; r--) fetch(r);
    }
    __syncwarp();
    int i = i_from;
    for (int r = r_first; r >= r_last; r--) {
        const uint32_t s = (uint32_t)(r_first - r) % C::kSlots, parity = ((uint32_t)(r_first - r) / C::kSlots) & 1u;
        bool ready = false;
        for (uint32_t spin = 0; spin < P.row_polls && !ready; spin++) ready = mbar_try_wait(bars + 8 * s, parity);
        if (!__all_sync(kFullMask, ready)) {
            for (int q = r; q >= r_last && q > r - (int)C::kSlots; q--) {
                const uint32_t at = (uint32_t)(r_first - q) % C::kSlots, phase = ((uint32_t)(r_first - q) / C::kSlots) & 1u;
                for (uint32_t spin = 0; spin < kRowPolls && !mbar_try_wait(bars + 8 * at, phase); spin++) {}
            }
            return kGivenUp;
        }
        const float *slot = P.buf0 + s * C::kRowFloats;
        auto row = [&](uint32_t q) { return best_at<CODE, KV>(slot, q); };
        const int depth = i - r * C::kStride;
        const uint32_t c = trace_tree_of_depth<CODE, KV, C::kStride>(depth, P, st, i, xoff, row);
        __syncwarp();                  // every lane has read the slot
        if (lane == 0 && r - (int)C::kSlots >= r_last) fetch(r - (int)C::kSlots);
        const int steps = min(depth, i - i_stop);
        for (int t = 1; t <= steps; t++)
            if (out && lane == 0) out[i - t] = (int)path_state<KV>(st, c, depth, t);
        st = path_state<KV>(st, c, depth, steps);
        i -= steps;
    }
    __syncwarp();
    if (lane == 0)
        for (uint32_t s = 0; s < C::kSlots; s++) asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(bars + 8 * s) : "memory");
    return st;
}

template <int CODE, int KV>
__host__ __device__ constexpr int vit_table_bytes() { return CODE == QTIP_CODE_3INST ? 0 : 4096; }
template <int CODE, int KV>
inline int vit_smem_bytes(int T) {
    using C = VitCfg<CODE, KV>;
    return (int)sizeof(Smem) + 2 * (int)C::kRowFloats * 4 + (C::kHyb ? 2 * 8192 : 0) + vit_table_bytes<CODE, KV>() + ((T * 4 + 15) & ~15);
}

template <int CODE, int KV>
__global__ void __launch_bounds__(VitCfg<CODE, KV>::kThreads, VitCfg<CODE, KV>::kPerSm)
    viterbi_kernel(int *__restrict__ states, float *__restrict__ final_cost, const __half *__restrict__ X, long N, int T,
                   const float2 *__restrict__ tlut, float *__restrict__ workspace, float minus_zero, uint32_t row_polls) {
    using C = VitCfg<CODE, KV>;
    constexpr int V = C::kV;
    extern __shared__ __align__(128) uint8_t smem_raw[];
    Smem *sh = reinterpret_cast<Smem *>(smem_raw);
    static_assert(sizeof(Smem) % 16 == 0, "what follows the control block needs 16-byte alignment");
    const int S = T / V, tid = threadIdx.x;
    PassCtx P;
    uint8_t *at = smem_raw + sizeof(Smem);
    P.buf0 = reinterpret_cast<float *>(at); at += C::kRowFloats * 4;
    P.buf1 = reinterpret_cast<float *>(at); at += C::kRowFloats * 4;
    P.etab = smem_u32(at); at += C::kHyb ? 2 * 8192 : 0;
    float *table = reinterpret_cast<float *>(at); at += vit_table_bytes<CODE, KV>();
    float *x = reinterpret_cast<float *>(at);
    P.x = x; P.tl = smem_u32(table); P.T = T; P.minus_zero = minus_zero; P.row_polls = row_polls;
    P.rows = workspace + (size_t)blockIdx.x * ((S + C::kStride - 1) / C::kStride) * C::kRowFloats;

    float2 lut[4] = {};
    using ThreadState = HybThread<C::kHyb ? KV : 4>;
    ThreadState ts;
    if constexpr (C::kHyb) {
        for (int i = tid; i < 512; i += C::kThreads) reinterpret_cast<float2 *>(table)[i] = tlut[i];
#pragma unroll
        for (int k = 0; k < 4; k++) lut[k] = tlut[tid + 128 * k];
        const uint32_t w = tid >> 5, l = tid & 31;
#pragma unroll
        for (uint32_t j = 0; j < 16; j++) ts.ebase[j] = ((hyb_hash(16 * w + j + 64 * l) >> 6) & 1023u) * 4u;
        const uint32_t q = (16 * w + 64 * l) >> KV, g = (16 * w + 64 * l) & (C::G - 1u);
        ts.rd = pos<CODE, KV>(q) * 4u; ts.rm = pos<CODE, KV>(C::G - 1u - q) * 4u;
        ts.wd = pos<CODE, KV>(g) * 4u; ts.wm = pos<CODE, KV>(C::G - 1u - g) * 4u;
    }
    if constexpr (CODE == QTIP_CODE_1MAD)
        for (int i = tid; i < 1024; i += C::kThreads) table[i] = __fdiv_rn((float)(i - 510), 147.800537109375f);
    for (long b = blockIdx.x; b < N; b += gridDim.x) {
        for (int t = tid; t < T; t += C::kThreads) x[t] = __half2float(X[b * T + t]);
        __syncthreads();
        // first pass: the sequence rolled by T/(2V)*V (rolled[t] = x[t - roll]), free ends; the state at step T/(2V) of the
        // rolled walk is where the original sequence starts
        const int half = T / (2 * V), xoff = T - half * V;
        viterbi_forward<CODE, KV>(sh, P, ts, lut, xoff, false, 0u, half / C::kStride * C::kStride, nullptr);
        if (tid < 32) {
            const uint32_t st = backtrace<CODE, KV>(sh, P, sh->arg, S - 1, half, xoff, nullptr);
            __syncwarp();
            if (tid == 0) sh->arg = st == kGivenUp ? kGivenUp : st >> KV;
        }
        __syncthreads();
        const uint32_t overlap = sh->arg;
        __syncthreads();
        if (overlap != kGivenUp) {
            viterbi_forward<CODE, KV>(sh, P, ts, lut, 0, true, overlap, 0, final_cost ? final_cost + b : nullptr);
            if (tid < 32) {
                int *out = states + b * S;
                const uint32_t st = sh->arg;
                if (tid == 0) out[S - 1] = (int)st;
                const uint32_t first = backtrace<CODE, KV>(sh, P, st, S - 1, 0, 0, out);
                __syncwarp();
                if (tid == 0) sh->arg = first;
            }
            __syncthreads();
        }
        if (sh->arg == kGivenUp) {
            // this sequence and the CTA's remaining ones: negative states of which no two neighbours overlap, cost not a number
            for (; b < N; b += gridDim.x) {
                for (int i = tid; i < S; i += C::kThreads) states[b * S + i] = i & 1 ? INT_MIN : -1;
                if (tid == 0 && final_cost) final_cost[b] = __uint_as_float(0x7FC00000u);
            }
            return;
        }
    }
}

// CTAs of a launch: one per sequence, as far as the GPU holds them at once and the workspace has a slab of rows for each.
template <int CODE, int KV>
long vit_grid(long N) {
    const long cap = (long)sm_count() * VitCfg<CODE, KV>::kPerSm;
    return N < cap ? N : cap;
}
template <int CODE, int KV>
size_t vit_slab(int T) {
    using C = VitCfg<CODE, KV>;
    const int S = T / C::kV;
    return (size_t)((S + C::kStride - 1) / C::kStride) * C::kRowFloats * sizeof(float);
}

// The least workspace a call takes.  HYB K=2 stores 16 KiB at every second step but asks for 4096 bytes per step and sequence, what
// it has always asked for, so the least workspace of up to 1182 sequences has a slab for every second one (4 sequences of 256 values:
// 0.87 ms instead of 0.44).
template <int CODE, int KV>
size_t vit_workspace(int T, long N) {
    constexpr int kShare = VitCfg<CODE, KV>::kHyb && KV == 4 ? 2 : 1;
    return (size_t)vit_grid<CODE, KV>((N + kShare - 1) / kShare) * vit_slab<CODE, KV>(T);
}

template <int CODE, int KV>
int launch_viterbi(int *states, float *final_cost, const __half *X, long N, int T, const float2 *tlut, float *ws, size_t ws_bytes,
                   unsigned row_polls, cudaStream_t s) {
    QTIP_CUDA_TRY(cudaFuncSetAttribute(viterbi_kernel<CODE, KV>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    const long slabs = (long)(ws_bytes / vit_slab<CODE, KV>(T)), want = vit_grid<CODE, KV>(N);
    viterbi_kernel<CODE, KV><<<(unsigned)(want < slabs ? want : slabs), VitCfg<CODE, KV>::kThreads, vit_smem_bytes<CODE, KV>(T), s>>>(
        states, final_cost, X, N, T, tlut, ws, -0.0f, row_polls);
    return check_launch();
}

// calls F<CODE, KV>() for the code and rate of a call
template <class F>
auto vit_dispatch(int code, int K, F f) {
    if (code == QTIP_CODE_HYB) {
        if (K == 2) return f.template operator()<QTIP_CODE_HYB, 4>();
        if (K == 3) return f.template operator()<QTIP_CODE_HYB, 6>();
        return f.template operator()<QTIP_CODE_HYB, 8>();
    }
    if (code == QTIP_CODE_3INST) {
        if (K == 2) return f.template operator()<QTIP_CODE_3INST, 2>();
        if (K == 3) return f.template operator()<QTIP_CODE_3INST, 3>();
        return f.template operator()<QTIP_CODE_3INST, 4>();
    }
    if (K == 2) return f.template operator()<QTIP_CODE_1MAD, 2>();
    if (K == 3) return f.template operator()<QTIP_CODE_1MAD, 3>();
    return f.template operator()<QTIP_CODE_1MAD, 4>();
}

struct WorkspaceCall {
    int T;
    long N;
    template <int CODE, int KV>
    size_t operator()() const { return vit_workspace<CODE, KV>(T, N); }
};
struct FullWorkspaceCall {
    int T;
    long N;
    template <int CODE, int KV>
    size_t operator()() const { return (size_t)vit_grid<CODE, KV>(N) * vit_slab<CODE, KV>(T); }
};
struct LaunchCall {
    int *states;
    float *final_cost;
    const __half *X;
    long N;
    int T;
    const float2 *tlut;
    float *ws;
    size_t ws_bytes;
    unsigned row_polls;
    cudaStream_t s;
    template <int CODE, int KV>
    int operator()() const { return launch_viterbi<CODE, KV>(states, final_cost, X, N, T, tlut, ws, ws_bytes, row_polls, s); }
};

}  // namespace
}  // namespace qtip

using namespace qtip;

static bool vit_sizes_ok(int code, int K, int T, long N) {
    return K >= 2 && K <= 4 && T > 0 && N > 0 && code >= QTIP_CODE_HYB && code <= QTIP_CODE_1MAD;
}

extern "C" size_t qtip_viterbi_workspace_bytes(int code, int K, int T, long N) {
    return vit_sizes_ok(code, K, T, N) ? vit_dispatch(code, K, WorkspaceCall{T, N}) : 0;
}

extern "C" size_t qtip_viterbi_workspace_bytes_full(int code, int K, int T, long N) {
    return vit_sizes_ok(code, K, T, N) ? vit_dispatch(code, K, FullWorkspaceCall{T, N}) : 0;
}

extern "C" int qtip_viterbi_quantize_polls(int *states, float *final_cost, const void *X, long N, int T, int code, int K,
                                           const float *tlut, void *workspace, size_t workspace_bytes, unsigned row_polls, void *stream) {
    if (!states || !X || N <= 0 || K < 2 || K > 4) return QTIP_ERR_BAD_ARG;
    if (code != QTIP_CODE_HYB && code != QTIP_CODE_3INST && code != QTIP_CODE_1MAD) return QTIP_ERR_BAD_ARG;
    if (code == QTIP_CODE_HYB && !tlut) return QTIP_ERR_BAD_ARG;
    const int V = code == QTIP_CODE_HYB ? 2 : 1;
    // a tail-biting walk needs at least L = 16 stream bits (T*K): shorter sequences have no walk whose ends overlap
    if (T < 4 * V || T * K < 16 || T > kMaxT || (T % (2 * V))) return QTIP_ERR_BAD_SHAPE;
    if (!aligned(states, 4) || !aligned(X, 2) || (tlut && !aligned(tlut, 8)) || (final_cost && !aligned(final_cost, 4)) ||
        !aligned(workspace, 16))
        return QTIP_ERR_ALIGNMENT;
    if (!workspace || workspace_bytes < qtip_viterbi_workspace_bytes(code, K, T, N)) return QTIP_ERR_WORKSPACE;
    return vit_dispatch(code, K, LaunchCall{states, final_cost, static_cast<const __half *>(X), N, T,
                                            reinterpret_cast<const float2 *>(tlut), static_cast<float *>(workspace), workspace_bytes,
                                            row_polls, static_cast<cudaStream_t>(stream)});
}

extern "C" int qtip_viterbi_quantize(int *states, float *final_cost, const void *X, long N, int T, int code, int K,
                                     const float *tlut, void *workspace, size_t workspace_bytes, void *stream) {
    return qtip_viterbi_quantize_polls(states, final_cost, X, N, T, code, K, tlut, workspace, workspace_bytes, kRowPolls, stream);
}
