// Channel mixer for sm_100a: token-shift mix -> key projection -> relu^2 -> value
// projection, the two projections on the tcgen05 tensor cores with the activation
// applied in the first one's epilogue.
//
// Replaces ChannelMixerBackend::fused_channel_mixer
// (crates/rwkv-nn/src/kernels/train/channel_mixer/forward.rs:52-88; semantic definition
// channel_mixer_reference, mod.rs:96-128; elementwise kernels kernel.rs:4-45):
//     shifted[b,t,:] = x[b,t-1,:] (zero at t == 0)
//     key_input = x + (shifted - x) * key_scale
//     hidden    = relu(key_input . key_weight^T)^2        key_weight   [F, C]
//     output    = hidden . value_weight^T                 value_weight [C, F]
// The reference runs two elementwise kernels around two library matmuls; here the
// hidden activation never exists unactivated: the first GEMM's epilogue squares the
// rectified accumulator before it is rounded to bf16.
//
// GEMM: out[M,N] = act(A[M,K] . B[N,K]^T), A and B row-major bf16 (both "K-major"), fp32 accumulation in TMEM, bf16 output.
// From 129 rows on mostly by pairs of CTAs (gemm_tn_bf16_pair_kernel, see gemm_plan::pair_width and sm100_pair_gemm.cuh).  Few rows, and
// rows that fill their blocks of 256 badly, by single CTAs: persistent, one per SM; a tile is 128 x 256;
// tiles are walked with the column block fastest, so that the CTAs running together share a
// few row blocks of A and sweep all of B, and both stay in L2.  Warp roles as in the LM-head
// kernel: warp 0 requests A and B tiles by TMA (128-byte swizzle, K slices of 64, 4-stage
// ring), warp 1 issues tcgen05.mma (M=128, N=256, kind::f16) into one of two 256-column
// TMEM buffers, warps 2..5 read the finished buffer back (thread = row, 32 columns at a
// time), apply the activation and store 64 contiguous bytes per thread while the next tile
// multiplies.  Every mbarrier wait is bounded.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "gemm_plan.h"
#include "kernels.h"
#include "launch.h"
#include "rwkv7_b200.h"
#include "sm100_pair_gemm.cuh"
#include "sm100_umma.cuh"

namespace rwkv7 {
namespace {

using namespace sm100;

constexpr int kBM = 128, kBN = 256, kBK = 64, kStages = 4;
static_assert(kBM == gemm_plan::kRows && kBN == gemm_plan::kCols && kBK == gemm_plan::kSlice && kPairM == gemm_plan::kPairRows, "as planned");
constexpr int kThreads = 192;  // TMA warp, MMA warp, four epilogue warps
constexpr uint32_t kABytes = kBM * kBK * 2, kBBytes = kBN * kBK * 2;
constexpr uint32_t kStageBytes = kABytes + kBBytes;
constexpr uint32_t kSmemBytes = kStages * kStageBytes + 1024 /*barriers*/ + 1024 /*alignment slack*/;

struct GemmMaps {
    CUtensorMap a;  // [M, K] bf16, box 128 x 64
    CUtensorMap b;  // [N, K] bf16, box 256 x 64
};

enum { kEpiNone = 0, kEpiReluSquare = 1, kEpiPartial = 2 };   // partial: fp32 sums over one piece of K

// 32 neighbouring accumulators of a row, from column c0 of N on (a multiple of 8), activated, rounded and stored: `nvec` pieces of eight.
template <int EPI>
__device__ __forceinline__ void store_row(const uint32_t (&v)[32], __nv_bfloat16 *dst, int nvec) {
    uint4 pk[4];
    unsigned *pw = &pk[0].x;
#pragma unroll
    for (int e = 0; e < 32; e += 2) {
        float x0 = __uint_as_float(v[e]), x1 = __uint_as_float(v[e + 1]);
        if constexpr (EPI == kEpiReluSquare) {
            x0 = fmaxf(x0, 0.f); x0 *= x0;
            x1 = fmaxf(x1, 0.f); x1 *= x1;
        }
        const __nv_bfloat162 h = __floats2bfloat162_rn(x0, x1);
        pw[e >> 1] = *reinterpret_cast<const unsigned *>(&h);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
        if (q < nvec) *reinterpret_cast<uint4 *>(dst + q * 8) = pk[q];
}

template <int EPI>
__global__ void __launch_bounds__(kThreads, 1)
gemm_tn_bf16_kernel(const __grid_constant__ GemmMaps maps, void *__restrict__ out, int64_t M, int N,
                    int K, int n_tiles, int mn_tiles, int splits, int *status) {
    extern __shared__ __align__(1024) unsigned char smem[];   // swizzled TMA tiles need 1024-byte alignment
    if (smem_u32(smem) & 1023u) {
        if (threadIdx.x == 0) atomicExch(status, (int)kDevInternal);
        return;
    }
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + kStages * kStageBytes);
    uint64_t *empty = full + kStages;
    uint64_t *tmem_full = empty + kStages;
    uint64_t *tmem_empty = tmem_full + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(tmem_empty + 2);

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // (uniform, for elect_one)
    const int all_ksteps = (K + kBK - 1) / kBK;   // the K tail is zero-filled by TMA
    // A work item is an output tile, or (splits > 1) one of `splits` pieces of K of it.
    const int total_tiles = mn_tiles * splits, per_split = (all_ksteps + splits - 1) / splits;
    auto first_kstep = [&](int item) { return item / mn_tiles * per_split; };
    auto count_ksteps = [&](int item) { return max(0, min(per_split, all_ksteps - first_kstep(item))); };

    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&tmem_full[b], 1); mbar_init(&tmem_empty[b], 4); }
        mbar_fence_init();
        tma_prefetch_desc(&maps.a);
        tma_prefetch_desc(&maps.b);
    }
    if (warp == 1) tmem_alloc(tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    bool timed_out = false;
    if (warp != 0) {
        wait_for_previous();
        let_next_in();
    }

    if (warp == 0) {
        if (elect_one()) {
            uint32_t it = 0;
            // the weights' first tiles are on their way while the kernel before this one finishes (see launch_channel_mixer)
            const int first = blockIdx.x, ahead = first < total_tiles ? min(kStages, count_ksteps(first)) : 0;
            for (int j = 0; j < ahead; ++j) {
                mbar_expect_tx(&full[j], kStageBytes);
                tma_load_2d(smem + j * kStageBytes + kABytes, &maps.b, (first_kstep(first) + j) * kBK, first % mn_tiles % n_tiles * kBN, &full[j]);
            }
            wait_for_previous();
            for (int j = 0; j < ahead; ++j)
                tma_load_2d(smem + j * kStageBytes, &maps.a, (first_kstep(first) + j) * kBK, first % mn_tiles / n_tiles * kBM, &full[j]);
            for (int tile = blockIdx.x; tile < total_tiles && !timed_out; tile += gridDim.x) {
                const int nt = tile % mn_tiles % n_tiles, mt = tile % mn_tiles / n_tiles, k0 = first_kstep(tile), ksteps = count_ksteps(tile);
                for (int ks = k0; ks < k0 + ksteps; ++ks, ++it) {
                    if (it < (uint32_t)ahead) continue;
                    const uint32_t s = it % kStages, ph = (it / kStages) & 1;
                    if (!mbar_wait(&empty[s], ph ^ 1)) { timed_out = true; break; }
                    unsigned char *a = smem + s * kStageBytes, *b = a + kABytes;
                    mbar_expect_tx(&full[s], kStageBytes);
                    tma_load_2d(a, &maps.a, ks * kBK, mt * kBM, &full[s]);
                    tma_load_2d(b, &maps.b, ks * kBK, nt * kBN, &full[s]);
                }
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            constexpr uint32_t idesc = make_idesc(kFmtBF16, kBM, kBN, false, false);
            uint32_t it = 0, local = 0;
            for (int tile = blockIdx.x; tile < total_tiles && !timed_out; tile += gridDim.x, ++local) {
                const uint32_t buf = local & 1, bph = (local >> 1) & 1;
                const int ksteps = count_ksteps(tile);
                if (!mbar_wait(&tmem_empty[buf], bph ^ 1)) { timed_out = true; break; }
                tc_fence_after();
                for (int ks = 0; ks < ksteps; ++ks, ++it) {
                    const uint32_t s = it % kStages, ph = (it / kStages) & 1;
                    if (!mbar_wait(&full[s], ph)) { timed_out = true; break; }
                    tc_fence_after();
                    const uint32_t a = smem_u32(smem + s * kStageBytes), b = a + kABytes;
#pragma unroll
                    for (int k = 0; k < kBK / 16; ++k)
                        umma_f16(tmem + buf * kBN, make_smem_desc(a + k * 32, 16, 1024),
                                 make_smem_desc(b + k * 32, 16, 1024), idesc, ks > 0 || k > 0);
                    umma_commit(&empty[s]);   // the stage may be refilled once these MMAs have read it
                }
                if (timed_out) break;
                umma_commit(&tmem_full[buf]);
            }
        }
    } else {
        const int quarter = warp & 3;
        uint32_t local = 0;
        for (int tile = blockIdx.x; tile < total_tiles && !timed_out; tile += gridDim.x, ++local) {
            const int nt = tile % mn_tiles % n_tiles, mt = tile % mn_tiles / n_tiles;
            const uint32_t buf = local & 1, bph = (local >> 1) & 1;
            if (!mbar_wait(&tmem_full[buf], bph)) { timed_out = true; break; }
            tc_fence_after();
            const int64_t row = (int64_t)mt * kBM + quarter * 32 + lane;
            __nv_bfloat16 *orow = static_cast<__nv_bfloat16 *>(out) + row * N + (int64_t)nt * kBN;
            float *prow = static_cast<float *>(out) + ((int64_t)(tile / mn_tiles) * M + row) * N + (int64_t)nt * kBN;
#pragma unroll 1
            for (int ch = 0; ch < kBN / 32; ++ch) {
                uint32_t v[32];
                tmem_ld32(tmem + ((uint32_t)(quarter * 32) << 16) + buf * kBN + ch * 32, v);
                tmem_ld_wait();
                const int c0 = nt * kBN + ch * 32;
                if (row >= M || c0 >= N) continue;            // padding rows / columns of edge tiles
                const int nvec = min(32, N - c0) / 8;          // N is a multiple of 8
                if constexpr (EPI == kEpiPartial) {
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if (q < 2 * nvec) *reinterpret_cast<uint4 *>(prow + ch * 32 + q * 4) = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                    continue;
                }
                store_row<EPI>(v, orow + ch * 32, nvec);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tmem_empty[buf]);
        }
    }
    if (timed_out) atomicExch(status, (int)kDevTimeout);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 512);
}

// The same on pairs of CTAs (see sm100_pair_gemm.cuh), tiles of 256 x width, K uncut; persistent pairs, column block fastest.
template <int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
gemm_tn_bf16_pair_kernel(const __grid_constant__ PairMaps maps, __nv_bfloat16 *__restrict__ out, int64_t M, int N, int K, int width, int n_tiles,
                         int tiles, int *status) {
    extern __shared__ __align__(1024) unsigned char smem[];
    if (smem_u32(smem) & 1023u) {
        if (threadIdx.x == 0) atomicExch(status, (int)kDevInternal);
        return;
    }
    const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);
    const int first = blockIdx.x >> 1, step = gridDim.x >> 1;
    auto items = [&](int i, PairItem &w) {
        const int tile = first + i * step;
        w = PairItem{tile / n_tiles * kPairM, tile % n_tiles * width, 0, (K + kPairK - 1) / kPairK};
        return tile < tiles;
    };
    PairGemm gemm;
    gemm.begin(smem, maps, warp);
    bool ok = true;
    // (the weights' first tiles are on their way while the kernel before this one finishes, see launch_channel_mixer)
    if (warp == 0) {
        if (elect_one()) ok = gemm.produce(maps, width, items, [] { wait_for_previous(); });
        __syncwarp();
    }
    wait_for_previous();
    let_next_in();
    if (warp == 0) {
        // (done)
    } else if (warp == 1) {
        if (gemm.rank == 0 && elect_one()) ok = gemm.multiply(width, items);
    } else {
        const int quarter = warp & 3;
        PairItem w;
        for (int i = 0; items(i, w); ++i) {
            if (!gemm.complete(i)) { ok = false; break; }
            const int64_t row = (int64_t)w.m0 + gemm.rank * 128 + quarter * 32 + lane;
            const int n1 = min(N, w.n0 + width);
            __nv_bfloat16 *orow = out + row * N + w.n0;
#pragma unroll 1
            for (int c = 0; c < n1 - w.n0; c += 32) {
                uint32_t v[32];
                tmem_ld32(gemm.tmem + ((uint32_t)(quarter * 32) << 16) + (i & 1) * kPairN + c, v);
                tmem_ld_wait();
                if (row < M) store_row<EPI>(v, orow + c, min(32, n1 - w.n0 - c) / 8);
            }
            gemm.release(i);
        }
    }
    __syncwarp();
    if (!ok) atomicExch(status, (int)kDevTimeout);
    gemm.end(warp);
}

// Sums the pieces of K and applies the activation; one thread per four columns.
template <int EPI>
__global__ void __launch_bounds__(256)
gemm_reduce_kernel(const float *__restrict__ parts, int splits, __nv_bfloat16 *__restrict__ out, int64_t quads) {
    wait_for_previous();
    let_next_in();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= quads) return;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int s = 0; s < splits; ++s) {
        const float4 x = __ldcs(reinterpret_cast<const float4 *>(parts) + (int64_t)s * quads + i);
        a.x += x.x;
        a.y += x.y;
        a.z += x.z;
        a.w += x.w;
    }
    if constexpr (EPI == kEpiReluSquare) {
        a.x = fmaxf(a.x, 0.f); a.x *= a.x;
        a.y = fmaxf(a.y, 0.f); a.y *= a.y;
        a.z = fmaxf(a.z, 0.f); a.z *= a.z;
        a.w = fmaxf(a.w, 0.f); a.w *= a.w;
    }
    const __nv_bfloat162 lo = __floats2bfloat162_rn(a.x, a.y), hi = __floats2bfloat162_rn(a.z, a.w);
    reinterpret_cast<uint2 *>(out)[i] = make_uint2(*reinterpret_cast<const unsigned *>(&lo), *reinterpret_cast<const unsigned *>(&hi));
}

// key_input = x + (shifted - x) * key_scale, shifted = previous token (zero at t == 0)
// (channel_mixer/kernel.rs:4-25).  A thread owns one 16-byte channel vector of kRows consecutive rows, and all of them and the row in
// front are on their way before the first is used.  Bound by latency at the sizes of a prefill: 4096 rows of 2048 channels took 14.3 us with
// two rows a CTA, one after the other, and a 64-bit division for each, 10.2 with shares of three or four; the whole call 220.6 -> 216.7 us so.
constexpr int kMixRows = 4;
template <int kRows>
__global__ void __launch_bounds__(256)
channel_mixer_mix_kernel(const __nv_bfloat16 *__restrict__ x, const __nv_bfloat16 *__restrict__ scale,
                         __nv_bfloat16 *__restrict__ out, int64_t rows, int64_t Tlen, int64_t C) {
    wait_for_previous();
    let_next_in();
    const int64_t row0 = (int64_t)blockIdx.x * kRows;
    const int count = (int)min((int64_t)kRows, rows - row0);
    const int64_t t0 = row0 % Tlen;
    auto unpack = [](const uint4 &u, float (&f)[8]) {
        const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            f[2 * i] = __uint_as_float(w[i] << 16);
            f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        }
    };
    for (int64_t c = (int64_t)threadIdx.x * 8; c < C; c += (int64_t)blockDim.x * 8) {
        const __nv_bfloat16 *from = x + row0 * C + c;
        uint4 raw[kRows + 1];   // the row in front, then this CTA's
        raw[0] = t0 == 0 ? make_uint4(0u, 0u, 0u, 0u) : *reinterpret_cast<const uint4 *>(from - C);
#pragma unroll
        for (int i = 0; i < kRows; ++i)
            if (i < count) raw[i + 1] = *reinterpret_cast<const uint4 *>(from + i * C);
        float mu[8], prev[8], cur[8];
        unpack(*reinterpret_cast<const uint4 *>(scale + c), mu);
        unpack(raw[0], prev);
        int64_t t = t0;
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
            if (i >= count) break;
            unpack(raw[i + 1], cur);
            if (t == Tlen) t = 0;
            if (t == 0) {
#pragma unroll
                for (int e = 0; e < 8; ++e) prev[e] = 0.f;   // first token of a sequence
            }
            ++t;
            uint4 o;
            unsigned *ow = &o.x;
#pragma unroll
            for (int e = 0; e < 8; e += 2) {
                const __nv_bfloat162 h = __floats2bfloat162_rn(fmaf(prev[e] - cur[e], mu[e], cur[e]),
                                                               fmaf(prev[e + 1] - cur[e + 1], mu[e + 1], cur[e + 1]));
                ow[e >> 1] = *reinterpret_cast<const unsigned *>(&h);
            }
            *reinterpret_cast<uint4 *>(out + (row0 + i) * C + c) = o;
#pragma unroll
            for (int e = 0; e < 8; ++e) prev[e] = cur[e];
        }
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

EncodeTiledFn gemm_encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    });
    return fn;
}

int encode_rows_by_k(EncodeTiledFn encode, CUtensorMap *map, const void *base, int64_t rows, int64_t K, int box_rows) {
    const cuuint32_t estr[2] = {1, 1};
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
    const cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)box_rows};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
               ? 0
               : (int)cudaErrorInvalidValue;
}

// out[M,N] = act(A[M,K] . B[N,K]^T); K and N multiples of 8, all pointers 16-byte aligned.
template <int EPI>
int launch_gemm(const void *a, const void *b, void *out, float *partials, size_t room, int64_t M, int64_t N, int64_t K, int num_sms,
                int *status, cudaStream_t stream) {
    EncodeTiledFn encode = gemm_encode_fn();
    if (encode == nullptr) return (int)cudaErrorNotSupported;
    const int splits = gemm_plan::k_pieces(M, N, K, std::min(num_sms, gemm_plan::kMostSms), room);
    if (const int width = gemm_plan::pair_width(M, N, K, num_sms, splits)) {
        PairMaps maps;
        if (int e = encode_rows_by_k(encode, &maps.a, a, M, K, kPairM / 2)) return e;
        if (int e = encode_rows_by_k(encode, &maps.b, b, N, K, width / 2)) return e;
        const int n_tiles = (int)((N + width - 1) / width), tiles = (int)((M + kPairM - 1) / kPairM) * n_tiles;
        cudaError_t e = cudaFuncSetAttribute(gemm_tn_bf16_pair_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPairSmem);
        if (e == cudaSuccess)
            e = launch_serialized(gemm_tn_bf16_pair_kernel<EPI>, 2u * (unsigned)std::min(tiles, num_sms / 2), (unsigned)kPairThreads, kPairSmem, stream, maps,
                                  (__nv_bfloat16 *)out, M, (int)N, (int)K, width, n_tiles, tiles, status);
        return (int)e;
    }
    GemmMaps maps;
    if (int e = encode_rows_by_k(encode, &maps.a, a, M, K, kBM)) return e;
    if (int e = encode_rows_by_k(encode, &maps.b, b, N, K, kBN)) return e;
    const int m_tiles = (int)((M + kBM - 1) / kBM), n_tiles = (int)((N + kBN - 1) / kBN);
    const int tiles = m_tiles * n_tiles;
    const int items = tiles * splits;
    const unsigned grid = (unsigned)(items < num_sms ? items : num_sms);
    auto kernel = splits > 1 ? gemm_tn_bf16_kernel<kEpiPartial> : gemm_tn_bf16_kernel<EPI>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
    if (e == cudaSuccess)
        e = launch_serialized(kernel, grid, kThreads, kSmemBytes, stream, maps, splits > 1 ? (void *)partials : out, M, (int)N, (int)K,
                              n_tiles, tiles, splits, status);
    if (e != cudaSuccess || splits == 1) return (int)e;
    const int64_t quads = M * N / 4;
    return (int)launch_serialized(gemm_reduce_kernel<EPI>, (unsigned)((quads + 255) / 256), 256u, 0, stream, (const float *)partials, splits,
                                  (__nv_bfloat16 *)out, quads);
}

inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

}  // namespace

// key_input and hidden; the partial sums behind them take what room there is (a workspace laid out for the largest batch serves a
// smaller one, which may cut K into more pieces).
size_t channel_mixer_min_workspace_bytes(int64_t rows, int64_t C, int64_t F) {
    if (rows <= 0 || C <= 0 || F <= 0) return 0;
    return align256((size_t)rows * C * 2) + align256((size_t)rows * F * 2);
}

size_t channel_mixer_workspace_bytes(int64_t rows, int64_t C, int64_t F) {
    if (rows <= 0 || C <= 0 || F <= 0) return 0;
    const size_t p1 = gemm_plan::partial_bytes(rows, F, C), p2 = gemm_plan::partial_bytes(rows, C, F);
    return channel_mixer_min_workspace_bytes(rows, C, F) + align256(p1 > p2 ? p1 : p2);
}

int launch_channel_mixer(const ChannelMixerArgs &p, void *workspace, size_t workspace_bytes, cudaStream_t stream) {
    const int64_t rows = p.B * p.T;
    if (rows == 0) return 0;
    if (workspace_bytes < channel_mixer_min_workspace_bytes(rows, p.C, p.F)) return (int)cudaErrorInvalidValue;
    __nv_bfloat16 *key_input = static_cast<__nv_bfloat16 *>(workspace);
    __nv_bfloat16 *hidden = reinterpret_cast<__nv_bfloat16 *>(static_cast<unsigned char *>(workspace) +
                                                              align256((size_t)rows * p.C * 2));
    const size_t least = channel_mixer_min_workspace_bytes(rows, p.C, p.F), room = workspace_bytes - least;
    float *partials = reinterpret_cast<float *>(static_cast<unsigned char *>(workspace) + least);
    int threads = 32;
    while (threads < 256 && threads < p.C / 8) threads <<= 1;
    // The products request weights before the kernel in front of them is complete.  That is one of this call's, which writes no weights
    // and lets its successor in only when everything before it is complete.
    const bool several = rows >= 4 * kMixRows * (int64_t)p.num_sms / 2;   // (few rows: one a CTA, so that more SMs have some)
    const cudaError_t e = launch_serialized(several ? channel_mixer_mix_kernel<kMixRows> : channel_mixer_mix_kernel<1>,
                                            (unsigned)(several ? (rows + kMixRows - 1) / kMixRows : rows), (unsigned)threads, 0, stream,
                                            (const __nv_bfloat16 *)p.x, (const __nv_bfloat16 *)p.key_scale, key_input, rows, p.T, p.C);
    if (e != cudaSuccess) return (int)e;
    if (int e = launch_gemm<kEpiReluSquare>(key_input, p.key_weight, hidden, partials, room, rows, p.F, p.C, p.num_sms, p.status, stream))
        return e;
    return launch_gemm<kEpiNone>(hidden, p.value_weight, p.out, partials, room, rows, p.C, p.F, p.num_sms, p.status, stream);
}

}  // namespace rwkv7
