// Hadamard transforms of power-of-two rows, 1024 to 65536 values.
//
// A thread owns 16 values; three radix passes (the first, of radix 16, on 16 consecutive values straight from the loads, one or
// two more bits by shuffles for the longest parts) with two exchanges through swizzled shared memory.  n / 16 threads per row,
// several rows per CTA below 4096.  CL > 0: a cluster of 2^CL CTAs shares a row (few long rows): each transforms its
// contiguous part and the last CL stages run over the cluster.
//
// Measured, microseconds per launch (fp16 -> fp16; before: a 1024-thread CTA per row, the whole row in registers with five
// shuffle stages twice for 4096 and 8192, radix-16 passes in shared memory otherwise):  1024 x 1000 rows 20.0 -> 3.6;
// 4096 x 1000 20.6 -> 7.5, x 120 3.4 -> 2.6, x 1 3.0 -> 2.4;  8192 x 1000 29.8 -> 15.1, x 8 4.3 -> 2.9;  16384 x 1 8.2 -> 3.1,
// x 120 8.6 -> 5.6;  32768 x 8 13.5 -> 3.8.  Few rows are latency (launch, load, two or three exchanges); 1000 rows of 4096 run
// at 2.2 TB/s of traffic, held back by shared-memory wavefronts and one load-compute-store phase per CTA.
#include "rht.cuh"

namespace qtip {
namespace {

// Shared-memory word of element e: its 16-byte chunk number is XORed with the bits above, so that both 16 consecutive values
// per thread (vector stores) and lanes on consecutive values, or on two groups of 16 that are 256 apart, use all banks.
// Linear in the bits of e: the register index contributes a constant.
__host__ __device__ __forceinline__ constexpr int pow2_at(int e) { return e ^ ((e >> 5 & 7) << 2) ^ ((e >> 8 & 1) << 4); }

template <int BITS>
__device__ __forceinline__ void radix(float (&v)[16]) {          // butterflies over the low BITS bits of the register index
#pragma unroll
    for (int s = 1; s < (1 << BITS); s <<= 1)
#pragma unroll
        for (int k = 0; k < 16; k++)
            if (!(k & s)) {
                const float x = v[k], y = v[k | s];
                v[k] = x + y;
                v[k | s] = x - y;
            }
}

template <int P, int CL>
struct Pow2Cfg {
    static constexpr int LP = P - CL;                      // log2 of the part a CTA transforms
    static constexpr int kRowThreads = 1 << (LP - 4);
    static constexpr int kThreads = kRowThreads < 256 && CL == 0 ? 256 : kRowThreads;
    static constexpr int kRows = kThreads / kRowThreads;
    static constexpr int SB = LP > 12 ? LP - 12 : 0;       // bits by shuffle after the first pass
    static constexpr int B2 = LP - 4 - SB < 8 ? (LP - 4 - SB + 1) / 2 : 4, B3 = LP - 4 - SB - B2;      // bits of passes two and three
    static constexpr int kRowFloats = 1 << LP;
    static constexpr int kSmem = (64 + kRows * kRowFloats) * (int)sizeof(float);
    static_assert(SB <= 2 && B3 >= 1 && B3 <= 4 && LP >= 10 && LP <= 14, "row length");
};

template <int P, int CL>
__global__ void __launch_bounds__(Pow2Cfg<P, CL>::kThreads) rht_pow2_kernel(const RhtArgs a, const long rows) {
    extern __shared__ __align__(16) float sm[];
    using C = Pow2Cfg<P, CL>;
    constexpr int LP = C::LP, n = 1 << P, SB = C::SB, B2 = C::B2, B3 = C::B3;
    const int sub = threadIdx.x / C::kRowThreads, tid = threadIdx.x % C::kRowThreads, lane = threadIdx.x & 31;
    float *scratch = sm;                                   // 64 floats
    float *buf = sm + 64 + sub * C::kRowFloats;
    rht_wait(a);
    const long row = CL ? (long)blockIdx.y : (long)blockIdx.x * C::kRows + sub;
    const bool live = row < rows;
    const long r = live ? row : rows - 1;                  // idle threads of the last CTA repeat the last row and store nothing
    const size_t part = CL ? (size_t)cluster_rank() << LP : 0;
    const size_t sign_off = (size_t)(r % a.sign_rep) * n, in_off = (size_t)r * a.in_row_stride;
    const size_t e0 = part + (size_t)tid * 16;
    float v[16];
    {
        float x[2][8];
#pragma unroll
        for (int h = 0; h < 2; h++) load_row_vec(a, in_off, e0 + 8 * h, x[h]);
        const bool write_res = live && a.residual_out && (a.in_row_stride != 0 || r == 0);
        float rnorm = 0.f;
        if (a.norm_weight || write_res) {
            float ss = 0.f;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                if (write_res) store8_f16(a.residual_out, in_off + e0 + 8 * h, x[h]);
#pragma unroll
                for (int c = 0; c < 8; c++) ss += x[h][c] * x[h][c];
            }
            if (a.norm_weight) {
                float total = 0.f;
                if constexpr (CL > 0) {
                    total = cluster_sum(ss, scratch, 1 << CL);
                } else {
                    constexpr int kRowWarps = C::kRowThreads / 32;
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(kFullMask, ss, o);
                    if (lane == 0) scratch[threadIdx.x >> 5] = ss;
                    __syncthreads();
#pragma unroll 8
                    for (int w = 0; w < kRowWarps; w++) total += scratch[sub * kRowWarps + w];
                }
                rnorm = rsqrtf(total / (float)n + a.eps);
            }
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            finish_row_vec(a, in_off, sign_off, e0 + 8 * h, rnorm, x[h]);
#pragma unroll
            for (int c = 0; c < 8; c++) v[8 * h + c] = x[h][c];
        }
    }
    radix<4>(v);
#pragma unroll
    for (int bit = 1; bit < (1 << SB); bit <<= 1)
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const float o = __shfl_xor_sync(kFullMask, v[k], bit);
            v[k] = (lane & bit) ? o - v[k] : v[k] + o;
        }
#pragma unroll
    for (int c = 0; c < 4; c++)
        *reinterpret_cast<float4 *>(buf + (pow2_at(tid * 16) ^ (4 * c))) = make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
    __syncthreads();
    // Passes two and three, B bits at position lo: register k holds the element whose bits [lo, lo + B) are k's low B bits (the
    // ones radix() works on) and whose low 4 - B bits are k's high ones.
    auto base = [&](int B, int lo) { const int t = tid << (4 - B); return ((t >> lo) << (lo + B)) | (t & ((1 << lo) - 1)); };
    auto reg = [](int B, int lo, int k) { return ((k & ((1 << B) - 1)) << lo) | (k >> B); };
    constexpr int lo2 = 4 + SB, lo3 = lo2 + B2;
    const int at2 = pow2_at(base(B2, lo2)), at3 = pow2_at(base(B3, lo3));
#pragma unroll
    for (int k = 0; k < 16; k++) v[k] = buf[at2 ^ pow2_at(reg(B2, lo2, k))];
    radix<B2>(v);
#pragma unroll
    for (int k = 0; k < 16; k++) buf[at2 ^ pow2_at(reg(B2, lo2, k))] = v[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 16; k++) v[k] = buf[at3 ^ pow2_at(reg(B3, lo3, k))];
    radix<B3>(v);
    if constexpr (CL == 0) {
        constexpr int W = 1 << (4 - B3);                   // consecutive values per strided position
        const size_t out_off = (size_t)row * n;
        if (!live) return;
#pragma unroll
        for (int k = 0; k < (1 << B3); k++) {
            const size_t e = base(B3, lo3) | reg(B3, lo3, k);
            float y[W];
#pragma unroll
            for (int c = 0; c < W; c++) {
                y[c] = v[k | (c << B3)] * a.scale;
                if (a.sign_out) y[c] *= __ldg(a.sign_out + sign_off + e + c);
            }
            if (a.out_dtype == QTIP_F16) {
                __half *o = static_cast<__half *>(a.out) + out_off + e;
                if constexpr (W == 1) *o = __float2half_rn(y[0]);
                else
#pragma unroll
                    for (int c = 0; c < W; c += 2) *reinterpret_cast<__half2 *>(o + c) = __floats2half2_rn(y[c], y[c + 1]);
            } else {      // fp32 (launch_pow2 refuses fragments here; a test of the type in this loop costs 2.5 us per launch)
                float *o = static_cast<float *>(a.out) + out_off + e;
                if constexpr (W == 1) *o = y[0];
                else
#pragma unroll
                    for (int c = 0; c < W; c += 2) *reinterpret_cast<float2 *>(o + c) = make_float2(y[c], y[c + 1]);
            }
        }
    } else {
        // the last CL stages: partners are the same local element of the other CTAs
#pragma unroll
        for (int k = 0; k < 16; k++) buf[at3 ^ pow2_at(reg(B3, lo3, k))] = v[k];
        constexpr int E = 1 << CL, items = 1 << (LP - 1);
        const uint32_t ob = (uint32_t)__cvta_generic_to_shared(buf);
        const int first = (int)cluster_rank() * C::kThreads + (int)threadIdx.x;
        float2 sg[E];
        auto signs = [&](int it) {
#pragma unroll
            for (int k = 0; k < E; k++) sg[k] = __ldg(reinterpret_cast<const float2 *>(a.sign_out + sign_off + ((size_t)k << LP) + 2 * it));
        };
        if (a.sign_out && first < items) signs(first);
        cluster_sync();
        for (int it = first; it < items; it += C::kThreads << CL) {
            float w[E][2];
#pragma unroll
            for (int k = 0; k < E; k++) {
                const float2 q = peer_load2(peer_smem(ob + (uint32_t)pow2_at(2 * it) * 4u, k));
                w[k][0] = q.x; w[k][1] = q.y;
            }
#pragma unroll
            for (int s = 1; s < E; s <<= 1)
#pragma unroll
                for (int k = 0; k < E; k++)
                    if (!(k & s))
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            const float x = w[k][h], y = w[k | s][h];
                            w[k][h] = x + y;
                            w[k | s][h] = x - y;
                        }
            if (a.sign_out && it != first) signs(it);
#pragma unroll
            for (int k = 0; k < E; k++) {
                const size_t col = ((size_t)k << LP) + 2 * it, e = (size_t)row * n + col;
                float y0 = w[k][0] * a.scale, y1 = w[k][1] * a.scale;
                if (a.sign_out) { y0 *= sg[k].x; y1 *= sg[k].y; }
                if (a.out_dtype == QTIP_F16) *reinterpret_cast<__half2 *>(static_cast<__half *>(a.out) + e) = __floats2half2_rn(y0, y1);
                else if (a.out_dtype == QTIP_F32) *reinterpret_cast<float2 *>(static_cast<float *>(a.out) + e) = make_float2(y0, y1);
                else static_cast<__half2 *>(a.out)[fragment_word(rows, row, col)] = __floats2half2_rn(y0, y1);
            }
        }
        cluster_sync();                                    // no CTA leaves while others read its part
    }
}

template <int P, int CL>
int launch_pow2(const RhtArgs &a, long rows, cudaStream_t s) {
    using C = Pow2Cfg<P, CL>;
    if (CL == 0 && a.out_dtype == QTIP_F16_FRAGMENTS) return QTIP_ERR_BAD_SHAPE;
    static bool attr_set[64] = {};
    int dev = 0;
    QTIP_CUDA_TRY(cudaGetDevice(&dev));
    if (dev >= 64 || !attr_set[dev]) {
        QTIP_CUDA_TRY(cudaFuncSetAttribute(rht_pow2_kernel<P, CL>, cudaFuncAttributeMaxDynamicSharedMemorySize, kOnePerSm));
        if (dev < 64) attr_set[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = CL ? dim3(1u << CL, (unsigned)rows) : dim3((unsigned)((rows + C::kRows - 1) / C::kRows));
    cfg.blockDim = dim3(C::kThreads);
    // about one CTA per SM: more than half an SM's shared memory keeps them on different SMs (see kOnePerSm; 8192 x 120 rows:
    // 5.7 -> 3.5 us)
    cfg.dynamicSmemBytes = !CL && (long)cfg.gridDim.x <= sm_count() && (long)cfg.gridDim.x * 2 > sm_count() ? kOnePerSm : C::kSmem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1u << CL;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = CL ? 2 : 1;
    QTIP_CUDA_TRY(cudaLaunchKernelEx(&cfg, rht_pow2_kernel<P, CL>, a, rows));
    return check_launch();
}

// log2 of the CTAs that share a row.  Short rows: one CTA, long ones: a cluster of eight.  In between a cluster while all of them
// run at once (three clusters of eight per sixteen SMs); fragments by the cluster kernels always: they alone write that order.
int pow2_cluster_log(int p, long rows, int out_dtype, int sms) {
    if (p < 13) return 0;
    return p > 14 || out_dtype == QTIP_F16_FRAGMENTS || rows <= (3 * sms / 2) >> 3 ? 3 : 0;
}

}  // namespace

bool launch_rht_pow2(const RhtArgs &a, long rows, cudaStream_t s, int &status) {
    if (a.kfac != 1 || !a.vec_ok) return false;
    const bool cluster = pow2_cluster_log(a.p, rows, a.out_dtype, sm_count()) > 0;
    switch (a.p) {
        case 10: status = launch_pow2<10, 0>(a, rows, s); return true;
        case 11: status = launch_pow2<11, 0>(a, rows, s); return true;
        case 12: status = launch_pow2<12, 0>(a, rows, s); return true;
        case 13: status = cluster ? launch_pow2<13, 3>(a, rows, s) : launch_pow2<13, 0>(a, rows, s); return true;
        case 14: status = cluster ? launch_pow2<14, 3>(a, rows, s) : launch_pow2<14, 0>(a, rows, s); return true;
        case 15: status = launch_pow2<15, 3>(a, rows, s); return true;
        case 16: status = launch_pow2<16, 3>(a, rows, s); return true;
        default: return false;
    }
}

}  // namespace qtip

extern "C" int qtip_rht_ctas_per_row(int n, long rows, int out_dtype, int sms) {
    int p = 0;
    while (p < 17 && (1 << p) < n) p++;
    if (n != 1 << p || p < 10 || p > 16 || rows < 1 || sms < 1) return 0;
    return 1 << qtip::pow2_cluster_log(p, rows, out_dtype, sms);
}
