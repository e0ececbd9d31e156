// Trellis decoders: packed codes -> dense fp16 (m, n).
//
// decode_hyb_kernel   HYB (L=16, V=2, Q=9) kernel layout; one warp per 2x2 block of 16x16 tiles,
//                     a lane reads its 4K contiguous bytes, gets the wrap-around bits from lane+1,
//                     and looks its 16 states up.  Same mapping as decode_compressed upstream (lib/utils/kernel_decompress.py:4-55).
//                     Bound: writing 2 bytes per weight.  With the 512 entries once per CTA the lookups' bank conflicts were the
//                     bound (shared-memory pipe at 77 %, issue at 35 %), so a persistent CTA of 32 warps keeps the matvec's 1024
//                     entries in 32 lane-private copies, and a tile's fragments go to the staging tile as matrices.
//                     Back to back, several matrices, microseconds at K = 2, 3, 4, the small kernel / this one / this one with settled
//                     weights, whose reads and table overlap the launch before:
//                       11008 x 4096  27.6 28.9 28.6 / 25.6 29.6 26.8 / 23.0 26.4 24.0 (3.9 TB/s of writes at K = 2)
//                       8192 x 8192   40.0 41.8 41.9 / 34.4 40.1 35.9 / 32.5 37.2 33.9
//                       28672 x 8192  131 138 137 / 109 130 114 / 106 127 111
// decode_hyb_small_kernel  the same with one copy of the table, for matrices of at most small_blocks() blocks, where building the
//                     128 KiB table costs more than the conflicts:
//                       2048 x 2048   5.0 5.0 5.1 / 5.9 6.2 6.1 / 4.8 5.0 5.0
//                       3072 x 2048   6.2 6.4 6.3 / 8.0 8.7 8.3 / 5.9 6.3 6.0
//                       4096 x 4096   11.7 12.2 12.3 / 12.3 14.0 12.8 / 10.4 11.6 10.8
//                       8192 x 4096   21.2 22.2 22.4 / 18.9 21.5 19.8 / 17.5 19.8 18.3
// decode_plain_kernel any code, plain layout (lib/codebook/bitshift.py:329-353, 378-381): one warp
//                     per tile, each lane decodes 8 consecutive sequence elements of one tile row half.
#include <mutex>

#include "common.cuh"

namespace qtip {
namespace {

constexpr int kDecodeThreads = 256;
constexpr int kHybThreads = 1024;
constexpr int kHybLutBytes = 1024 * 32 * 4;

// Row stride of a warp's staging tile in bytes: 64 of data + 16, so that the eight 16-byte rows of a matrix, and the rows of a
// read-back, fall into distinct banks.
constexpr int kStageStride = 80;
constexpr int kHybSmem = kHybLutBytes + kHybThreads / 32 * 32 * kStageStride;

template <int K>
__global__ void __launch_bounds__(kHybThreads, 1) decode_hyb_kernel(__half *__restrict__ W, const uint8_t *__restrict__ codes,
                                                                    const uint32_t *__restrict__ tlut, int m, int n) {
    extern __shared__ __align__(128) uint8_t smem[];
    // the warp index through a shuffle: the same in all lanes, so the loop control is scalar
    const int warp = __shfl_sync(kFullMask, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int nb = n >> 5, blocks = (m >> 5) * nb, warps = (int)gridDim.x * (kHybThreads / 32);
    int blk = (int)blockIdx.x * (kHybThreads / 32) + warp;
    const uint8_t *src = codes + (size_t)blk * (128 * K) + lane * (4 * K);
    LaneCodes<K> own = {};
    if (blk < blocks) own = load_lane_codes<K>(src);
    // entry e = sign << 9 | index, copy l at byte e*128 + l*4; the sign bit flips the first weight of the pair
    for (int i = threadIdx.x; i < 1024 * 8; i += kHybThreads) {
        const uint32_t e = __ldg(tlut + ((i >> 3) & 511)) ^ ((uint32_t)(i >> 12) << 15);
        reinterpret_cast<uint4 *>(smem)[i] = make_uint4(e, e, e, e);
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __syncthreads();
    asm volatile("griddepcontrol.wait;" ::: "memory");      // W may still be read by an earlier launch of the stream

    const uint32_t lut_lane = (uint32_t)__cvta_generic_to_shared(smem) + lane * 4;
    const uint32_t stage = (uint32_t)__cvta_generic_to_shared(smem) + kHybLutBytes + warp * (32 * kStageStride);
    // matrix q = lane >> 3 of a tile (column half q >> 1, row half q & 1), its row lane & 7
    const uint32_t put = stage + (8 * ((lane >> 3) & 1) + (lane & 7)) * kStageStride + (lane >> 4) * 16;
    const uint32_t get = stage + (lane >> 2) * kStageStride + (lane & 3) * 16;
    int M = __shfl_sync(kFullMask, blk / nb, 0), N = blk - M * nb;
    const int step_m = __shfl_sync(kFullMask, warps / nb, 0), step_n = warps - step_m * nb;
    const size_t lane_at = (size_t)(lane >> 2) * n + 8 * (lane & 3);
    for (; blk < blocks; blk += warps) {
        LaneCodes<K> cur = own, nxt;
        src += (size_t)warps * (128 * K);
        if (blk + warps < blocks) own = load_lane_codes<K>(src);
        nxt = shfl_next_lane<K>(cur, lane);
        __syncwarp();                                       // the tile of the block before has been read
#pragma unroll
        for (int t = 0; t < 4; t++) {                       // tile rows 16 (t & 1) .., columns 16 (t >> 1) ..
            uint32_t st[4], w[4];
            tile_states<K>(cur, nxt, t, st);
#pragma unroll
            for (int q = 0; q < 4; q++) w[q] = hyb_lookup(st[q], lut_lane);
            asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};"
                         ::"r"(put + 16 * (t & 1) * kStageStride + 32 * (t >> 1)), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
        }
        __syncwarp();
        // 64-byte row segments: one 16-byte store per lane covers 8 rows
        __half *dst = W + (size_t)M * 32 * n + (size_t)N * 32 + lane_at;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            uint4 v;
            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(get + 8 * i * kStageStride));
            *reinterpret_cast<uint4 *>(dst + (size_t)(8 * i) * n) = v;
        }
        M += step_m;
        N += step_n;
        if (N >= nb) { N -= nb; M++; }
    }
}

// where the two kernels meet (the figures above)
constexpr long small_blocks(bool settled) { return settled ? 4 << 10 : 16 << 10; }
constexpr int kSmallStride = kStageStride / 4;      // words

template <int K>
__global__ void __launch_bounds__(kDecodeThreads) decode_hyb_small_kernel(__half *__restrict__ W, const uint8_t *__restrict__ codes,
                                                                         const uint32_t *__restrict__ tlut, int m, int n) {
    __shared__ uint32_t lut[512];
    __shared__ __align__(16) uint32_t stage_all[kDecodeThreads / 32][32 * kSmallStride];
    for (int i = threadIdx.x; i < 512; i += blockDim.x) lut[i] = tlut[i];
    __syncthreads();

    const int lane = threadIdx.x & 31;
    uint32_t *stage = stage_all[threadIdx.x >> 5];
    const int warps = (gridDim.x * blockDim.x) >> 5;
    const int nb = n >> 5;
    const long blocks = (long)(m >> 5) * nb;
    const int a = lane >> 2, b = lane & 3;
    for (long blk = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; blk < blocks; blk += warps) {
        const int M = (int)(blk / nb), N = (int)(blk % nb);
        const LaneCodes<K> own = load_lane_codes<K>(codes + blk * (128 * K) + lane * (4 * K));
        const LaneCodes<K> nxt = shfl_next_lane<K>(own, lane);
        // decode into the warp's 32 x 32 staging tile (fragment order -> row-major) ...
#pragma unroll
        for (int t = 0; t < 4; t++) {
            const int ks = t >> 1, ms = t & 1;
            uint32_t st[4];
            tile_states<K>(own, nxt, t, st);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int c = q >> 1, d = q & 1;
                const uint32_t h = hyb_hash(st[q]);
                stage[(16 * ms + 8 * d + a) * kSmallStride + 8 * ks + 4 * c + b] = lut[(h >> 6) & 511u] ^ (h & 0x8000u);
            }
        }
        __syncwarp();
        // ... and write it out as 64-byte row segments: one 16-byte store per lane covers 8 rows x 64 bytes
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int r = 8 * i + a;
            const uint4 v = *reinterpret_cast<const uint4 *>(stage + r * kSmallStride + 4 * b);
            *reinterpret_cast<uint4 *>(W + ((size_t)32 * M + r) * n + (size_t)32 * N + 8 * b) = v;
        }
        __syncwarp();
    }
}

int decode_grid(long warps_needed) {
    long ctas = (warps_needed + (kDecodeThreads / 32) - 1) / (kDecodeThreads / 32);
    long cap = (long)sm_count() * 8;
    return (int)(ctas < cap ? (ctas < 1 ? 1 : ctas) : cap);
}

template <int K>
int launch_decode_hyb(__half *W, const uint8_t *codes, const uint32_t *tlut, int m, int n, bool settled, cudaStream_t s) {
    const long blocks = (long)(m >> 5) * (n >> 5);
    if (blocks <= small_blocks(settled)) {
        decode_hyb_small_kernel<K><<<decode_grid(blocks), kDecodeThreads, 0, s>>>(W, codes, tlut, m, n);
        return check_launch();
    }
    static bool attr_set[64] = {};
    static std::mutex attr_mutex;
    int dev = 0;
    QTIP_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return QTIP_ERR_BAD_ARG;
    {
        std::lock_guard<std::mutex> lock(attr_mutex);
        if (!attr_set[dev]) {
            QTIP_CUDA_TRY(cudaFuncSetAttribute(decode_hyb_kernel<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, kHybSmem));
            attr_set[dev] = true;
        }
    }
    const long ctas = (blocks + kHybThreads / 32 - 1) / (kHybThreads / 32);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(ctas < sm_count() ? ctas : sm_count()));
    cfg.blockDim = dim3(kHybThreads);
    cfg.dynamicSmemBytes = kHybSmem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = settled ? 1 : 0;       // codes and table are read before the wait
    QTIP_CUDA_TRY(cudaLaunchKernelEx(&cfg, decode_hyb_kernel<K>, W, codes, tlut, m, n));
    return check_launch();
}

// 48 stream bits of a tile starting at bit `pos` (circular over nbits = 256*K), first bit at bit 47.
__device__ __forceinline__ uint64_t tile_bits48(const uint16_t *__restrict__ words, int nwords, int pos) {
    int w = pos >> 4;
    uint64_t v = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        int wi = w + i;
        if (wi >= nwords) wi -= nwords;
        v = (v << 16) | words[wi];
    }
    return (v << (pos & 15)) >> 16;  // drop the bits before pos, keep 48
}

template <int CODE>
__global__ void __launch_bounds__(kDecodeThreads) decode_plain_kernel(__half *__restrict__ W,
                                                                     const uint16_t *__restrict__ codes,
                                                                     const uint32_t *__restrict__ tlut, int K, int m,
                                                                     int n) {
    __shared__ uint32_t lut[CODE == QTIP_CODE_HYB ? 512 : 1];
    if constexpr (CODE == QTIP_CODE_HYB) {
        for (int i = threadIdx.x; i < 512; i += blockDim.x) lut[i] = tlut[i];
        __syncthreads();
    }
    const int lane = threadIdx.x & 31;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    const int tn = n >> 4;
    const long tiles = (long)(m >> 4) * tn;
    const int nwords = 16 * K;
    const int r = lane >> 1, hf = lane & 1;  // tile row, half of the row (8 elements)
    for (long tile = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; tile < tiles; tile += warps) {
        const uint16_t *words = codes + tile * nwords;
        const int e0 = r * 16 + hf * 8;  // first sequence element of this lane
        __half out[8];
        if constexpr (CODE == QTIP_CODE_HYB) {
            // V = 2: state i covers elements 2i, 2i+1; window starts at bit i*2K
#pragma unroll
            for (int j = 0; j < 4; j++) {
                int i = (e0 >> 1) + j;
                uint32_t s = (uint32_t)(tile_bits48(words, nwords, i * 2 * K) >> 32) & 0xFFFFu;
                uint32_t h = hyb_hash(s);
                uint32_t w = lut[(h >> 6) & 511u] ^ (h & 0x8000u);
                *reinterpret_cast<uint32_t *>(&out[2 * j]) = w;
            }
        } else {
            // V = 1: 8 states from 7K+16 <= 44 consecutive bits
            uint64_t bits = tile_bits48(words, nwords, e0 * K);
#pragma unroll
            for (int j = 0; j < 8; j++) {
                uint32_t s = (uint32_t)(bits >> (32 - j * K)) & 0xFFFFu;
                out[j] = (CODE == QTIP_CODE_3INST) ? decode_3inst(s) : decode_1mad(s);
            }
        }
        size_t row = (size_t)(tile / tn) * 16 + r, col = (size_t)(tile % tn) * 16 + hf * 8;
        *reinterpret_cast<uint4 *>(W + row * n + col) = *reinterpret_cast<uint4 *>(out);
    }
}

int decode_hyb(void *W, const void *codes, const void *tlut, int K, int m, int n, bool settled, void *stream) {
    if (!W || !codes || !tlut || K < 2 || K > 4) return QTIP_ERR_BAD_ARG;
    if (m <= 0 || n <= 0 || (m & 31) || (n & 31)) return QTIP_ERR_BAD_SHAPE;
    if (!aligned(codes, 16) || !aligned(W, 16) || !aligned(tlut, 4)) return QTIP_ERR_ALIGNMENT;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    auto *Wh = static_cast<__half *>(W);
    auto *c = static_cast<const uint8_t *>(codes);
    auto *t = static_cast<const uint32_t *>(tlut);
    if (K == 2) return launch_decode_hyb<2>(Wh, c, t, m, n, settled, s);
    if (K == 3) return launch_decode_hyb<3>(Wh, c, t, m, n, settled, s);
    return launch_decode_hyb<4>(Wh, c, t, m, n, settled, s);
}

}  // namespace
}  // namespace qtip

using namespace qtip;

extern "C" int qtip_decode_hyb(void *W, const void *codes, const void *tlut, int K, int m, int n, void *stream) {
    return decode_hyb(W, codes, tlut, K, m, n, false, stream);
}

extern "C" int qtip_decode_hyb_settled(void *W, const void *codes, const void *tlut, int K, int m, int n, void *stream) {
    return decode_hyb(W, codes, tlut, K, m, n, true, stream);
}

extern "C" int qtip_decode_plain(void *W, const void *codes, int code, const void *tlut, int K, int m, int n,
                                 void *stream) {
    if (!W || !codes || K < 2 || K > 4) return QTIP_ERR_BAD_ARG;
    if (code == QTIP_CODE_HYB && !tlut) return QTIP_ERR_BAD_ARG;
    if (m <= 0 || n <= 0 || (m & 15) || (n & 15)) return QTIP_ERR_BAD_SHAPE;
    if (!aligned(codes, 2) || !aligned(W, 16)) return QTIP_ERR_ALIGNMENT;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int grid = decode_grid((long)(m >> 4) * (n >> 4));
    auto *Wh = static_cast<__half *>(W);
    auto *c = static_cast<const uint16_t *>(codes);
    auto *t = static_cast<const uint32_t *>(tlut);
    switch (code) {
        case QTIP_CODE_HYB: decode_plain_kernel<QTIP_CODE_HYB><<<grid, kDecodeThreads, 0, s>>>(Wh, c, t, K, m, n); break;
        case QTIP_CODE_3INST: decode_plain_kernel<QTIP_CODE_3INST><<<grid, kDecodeThreads, 0, s>>>(Wh, c, t, K, m, n); break;
        case QTIP_CODE_1MAD: decode_plain_kernel<QTIP_CODE_1MAD><<<grid, kDecodeThreads, 0, s>>>(Wh, c, t, K, m, n); break;
        default: return QTIP_ERR_BAD_ARG;
    }
    return check_launch();
}
