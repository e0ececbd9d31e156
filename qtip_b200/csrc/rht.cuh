// Arguments and element helpers shared by the Hadamard-transform kernels (rht.cu, rht_factor.cu, rht_pow2.cu).
#pragma once

#include "fwht.cuh"

namespace qtip {

struct RhtArgs {
    void *out; const void *in; const void *sign_in; const float *sign_out; const uint32_t *hadk_bits;
    const __half *residual; __half *residual_out; const __half *norm_weight; const __half *gate;
    long in_row_stride;  // elements between input rows (0 = every row reads the same input)
    int out_dtype, in_dtype, sign_in_dtype;
    int n, p, sign_rep, kfac, transpose;
    int rpc;             // hadK output rows per CTA (4, 8 or 16)
    int part_offset;     // float offset in shared memory of the partial-product buffer (short rows only)
    int sgn_offset;      // float offset of the staged sign_out slice (short rows only, else 0)
    int vec_ok;          // every buffer is 16-byte aligned and n, strides are multiples of 8: 8-wide loads / stores
    int settle;          // the next launch may start only when everything before this one is complete (see rht_wait)
    float scale, eps;
};

// Waits for the launch before and lets the next one start: at once (the decode loop, whose weights are old), or with `settle` (qtip_rht)
// only after the wait.  A product that reads its weights while the transform before it runs is then safe whatever wrote them before
// that.  It also measured faster where layer calls follow one another (28672 x 8192 K = 4, 1 row: 60.1 -> 50.8 us a call; 8192 x 8192,
// 5 rows 22.8 -> 22.1; 8192 x 8192 3INST, 16 rows 30.7 -> 31.1).
__device__ __forceinline__ void rht_wait(const RhtArgs &a) {
    if (!a.settle) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (a.settle) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ float load_elem(const void *p, int dtype, size_t i) {
    return dtype == QTIP_F16 ? __half2float(static_cast<const __half *>(p)[i]) : static_cast<const float *>(p)[i];
}

// 8 consecutive elements starting at element i (i % 8 == 0, base pointers 16-byte aligned)
__device__ __forceinline__ void load8(const void *p, int dtype, size_t i, float (&o)[8]) {
    if (dtype == QTIP_F16) load8_f16(static_cast<const __half *>(p), i, o);
    else load8_f32(static_cast<const float *>(p), i, o);
}
__device__ __forceinline__ void store8(void *p, int dtype, size_t i, const float (&o)[8]) {
    if (dtype == QTIP_F16) store8_f16(static_cast<__half *>(p), i, o);
    else store8_f32(static_cast<float *>(p), i, o);
}

// Eight elements of a row up to the transform.  load_row_vec: input and residual add; finish_row_vec: norm (with its
// statistics in rnorm), gate, sign.
__device__ __forceinline__ void load_row_vec(const RhtArgs &a, size_t in_off, size_t e, float (&x)[8]) {
    load8(a.in, a.in_dtype, in_off + e, x);
    if (a.residual) {
        float rs[8];
        load8_f16(a.residual, in_off + e, rs);
#pragma unroll
        for (int c = 0; c < 8; c++) x[c] = __half2float(__float2half_rn(x[c] + rs[c]));      // the residual stream is fp16
    }
}
__device__ __forceinline__ void finish_row_vec(const RhtArgs &a, size_t in_off, size_t sign_off, size_t e, float rnorm, float (&x)[8]) {
    if (a.norm_weight) {
        float w[8];
        load8_f16(a.norm_weight, e, w);
#pragma unroll
        for (int c = 0; c < 8; c++) x[c] = __half2float(__hmul(__float2half_rn(w[c]), __float2half_rn(x[c] * rnorm)));   // LlamaRMSNorm
    }
    if (a.gate) {
        float gt[8];
        load8_f16(a.gate, in_off + e, gt);
#pragma unroll
        for (int c = 0; c < 8; c++) x[c] = swiglu_fp16(gt[c], x[c]);
    }
    if (a.sign_in) {
        float sg[8];
        load8(a.sign_in, a.sign_in_dtype, sign_off + e, sg);
#pragma unroll
        for (int c = 0; c < 8; c++) x[c] *= sg[c];
    }
}

// Where the pair of columns e, e + 1 of a row lies in the matvec's fragment order (32-bit words)
__device__ __forceinline__ size_t fragment_word(long rows, long row, size_t e) {
    const size_t w = e >> 1;
    return ((w >> 4) * rows + row) * 16 + (w & 3) * 4 + ((w >> 2) & 3);
}

// ---- thread-block clusters ----------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t peer_smem(uint32_t addr, uint32_t rank) {
    uint32_t p;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(p) : "r"(addr), "r"(rank));
    return p;
}
__device__ __forceinline__ float2 peer_load2(uint32_t addr) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float peer_load(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
// sum over the CTA, then over the cluster (scratch: 33 floats)
__device__ __forceinline__ float cluster_sum(float x, float *scratch, int csize) {
    const float s = block_sum(x, scratch);
    if (threadIdx.x == 0) scratch[32] = s;
    cluster_sync();
    float t = 0.f;
    for (int r = 0; r < csize; r++) t += peer_load(peer_smem((uint32_t)__cvta_generic_to_shared(scratch + 32), r));
    return t;
}

// Shared memory that only one CTA per SM can have.  A launch of about one CTA per SM asks for it: with programmatic stream
// serialization it is placed while its predecessor still occupies most SMs, and would otherwise crowd onto the free ones.
constexpr int kOnePerSm = 120 * 1024;

// Launchers of the specialised kernels: false if the kernel does not apply, else `status` is the launch's result.
bool launch_rht_pow2(const RhtArgs &a, long rows, cudaStream_t s, int &status);       // rht_pow2.cu
bool launch_rht_cluster(const RhtArgs &a, long rows, cudaStream_t s, int &status);    // rht_factor.cu: few rows
bool launch_rht_rows(const RhtArgs &a, long rows, cudaStream_t s, int &status);       // rht_factor.cu: many rows

}  // namespace qtip
