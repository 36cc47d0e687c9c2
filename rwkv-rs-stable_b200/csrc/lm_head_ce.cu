// Fused LM-head cross entropy for sm_100a: z = x W^T on the tcgen05 tensor cores
// with an online log-sum-exp epilogue, so the [R, V] logits are never written.
//
// The reference reserves this operator but ships no implementation
// (crates/rwkv-nn/src/kernels/train/lm_head_l2wrap_ce/mod.rs is empty; the config
// switch is crates/rwkv-config/src/raw/train.rs:59-60), so the definition is the
// one stated in rwkv7_b200.h: per row the triple (max_v z_v, sum_v exp(z_v - max),
// z_target) over a vocabulary shard, then a combine over shards.
//
// One CTA owns a block of 128 rows, or a pair of CTAs 256 (lm_head_ce_pair_kernel, most
// calls of more than 128 rows), and a contiguous range of vocabulary tiles of up to 256
// columns.  Warp roles: warp 0 requests the x and W tiles (TMA, 128-byte swizzle, K
// slices of 64 bf16, 4-stage ring); warp 1 issues the UMMAs (M=128, bf16 in,
// fp32 accumulators, two 256-column TMEM buffers); warps 2..5 are the epilogue:
// thread = row, it reads its accumulator row 32 columns at a time and keeps the
// running (max, sum-exp, target logit) in registers while the next tile is being
// multiplied.  CTAs that run together walk the vocabulary in the same order, so a
// W tile is fetched from HBM once per wave and served to the others from L2.
// Every mbarrier wait is bounded.
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
constexpr float kLog2e = 1.4426950408889634f;

struct LmMaps {
    CUtensorMap x;  // [R, C] bf16, box 128 x 64
    CUtensorMap w;  // [V, C] bf16, box 256 x 64
};

__device__ __forceinline__ int64_t load_target(const void *t, int dtype, int64_t row) {
    return dtype == RWKV7_I64 ? reinterpret_cast<const int64_t *>(t)[row]
                              : (int64_t) reinterpret_cast<const int32_t *>(t)[row];
}

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// The wait for a TMEM read, with its registers: nothing that uses them moves in front of it while others are in flight.
__device__ __forceinline__ void tmem_ld_wait_for(uint32_t (&v)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]), "+r"(v[9]),
                   "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]), "+r"(v[16]), "+r"(v[17]), "+r"(v[18]),
                   "+r"(v[19]), "+r"(v[20]), "+r"(v[21]), "+r"(v[22]), "+r"(v[23]), "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27]),
                   "+r"(v[28]), "+r"(v[29]), "+r"(v[30]), "+r"(v[31])
                 :
                 : "memory");
}

// What a thread keeps of its row of logits.
struct RowSums {
    float m = -INFINITY, ssum = 0.f, zt = 0.f;
    // 32 neighbouring logits from column c0 on, of which those below `end` count; `tgt` is the target's column in this shard
    __device__ __forceinline__ void take(uint32_t (&v)[32], int c0, int end, int64_t tgt) {
        const int ncol = min(32, end - c0);
        if (ncol < 32) {
#pragma unroll
            for (int e = 0; e < 32; ++e)
                if (e >= ncol) v[e] = __float_as_uint(-INFINITY);
        }
        // (four chains each for the maximum and the sum: one warp a scheduler does this, nothing else covers its latency)
        float most[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) most[e] = __uint_as_float(v[e]);
#pragma unroll
        for (int e = 4; e < 32; ++e) most[e & 3] = fmaxf(most[e & 3], __uint_as_float(v[e]));
        const float m_new = fmaxf(m, fmaxf(fmaxf(most[0], most[1]), fmaxf(most[2], most[3])));
        const float mb = m_new * kLog2e;
        ssum *= ex2(m * kLog2e - mb);               // 2^-inf = 0 on the first chunk
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int e = 0; e < 32; ++e) acc[e & 3] += ex2(fmaf(__uint_as_float(v[e]), kLog2e, -mb));   // (at most 1: subnormal terms are nothing)
        ssum += (acc[0] + acc[1]) + (acc[2] + acc[3]);
        m = m_new;
        if (tgt >= c0 && tgt < c0 + ncol) {
            const int off = (int)(tgt - c0);
#pragma unroll
            for (int e = 0; e < 32; ++e)
                if (e == off) zt = __uint_as_float(v[e]);
        }
    }
    // The accumulators of columns col0 .. end - 1, from TMEM address `at` on: the next 32 are read while these are summed up.
    __device__ __forceinline__ void take_row(uint32_t at, int col0, int end, int64_t tgt) {
        uint32_t v0[32], v1[32];
        auto from = [&](int c) { return at + (uint32_t)min(c - col0, kBN - 32); };   // (always a read: one under a condition would be copied in flight)
        tmem_ld32(at, v0);
        tmem_ld_wait_for(v0);
#pragma unroll 1
        for (int c = col0; c < end; c += 64) {
            tmem_ld32(from(c + 32), v1);
            take(v0, c, end, tgt);
            tmem_ld_wait_for(v1);
            tmem_ld32(from(c + 64), v0);
            if (c + 32 < end) take(v1, c + 32, end, tgt);
            tmem_ld_wait_for(v0);
        }
    }
};

__global__ void __launch_bounds__(kThreads, 1)
lm_head_ce_kernel(const __grid_constant__ LmMaps maps, const void *__restrict__ targets, int targets_dtype,
                  int64_t vocab_offset, float *__restrict__ out /* [splits][R][3] */, int64_t R, int C, int V,
                  int row_blocks, int width, int tiles_per_split, int *status) {
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
    // consecutive CTAs share a vocabulary split and differ in the row block
    const int rb = blockIdx.x % row_blocks, split = blockIdx.x / row_blocks;
    const int total_tiles = (V + width - 1) / width;
    const int tile0 = split * tiles_per_split;
    const int ntiles = min(tiles_per_split, total_tiles - tile0);
    const int ksteps = C / kBK;

    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&tmem_full[b], 1); mbar_init(&tmem_empty[b], 4); }
        mbar_fence_init();
        tma_prefetch_desc(&maps.x);
        tma_prefetch_desc(&maps.w);
    }
    if (warp == 1) tmem_alloc(tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    bool timed_out = false;
    wait_for_previous();
    let_next_in();

    if (warp == 0) {
        if (elect_one()) {
            uint32_t it = 0;
            for (int t = 0; t < ntiles && !timed_out; ++t) {
                for (int ks = 0; ks < ksteps; ++ks, ++it) {
                    const uint32_t s = it % kStages, ph = (it / kStages) & 1;
                    if (!mbar_wait(&empty[s], ph ^ 1)) { timed_out = true; break; }
                    unsigned char *a = smem + s * kStageBytes, *b = a + kABytes;
                    mbar_expect_tx(&full[s], kABytes + (uint32_t)width * kBK * 2);
                    tma_load_2d(a, &maps.x, ks * kBK, rb * kBM, &full[s]);
                    tma_load_2d(b, &maps.w, ks * kBK, (tile0 + t) * width, &full[s]);
                }
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            const uint32_t idesc = make_idesc(kFmtBF16, kBM, width, false, false);
            uint32_t it = 0;
            for (int t = 0; t < ntiles && !timed_out; ++t) {
                const uint32_t buf = t & 1, bph = (t >> 1) & 1;
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
        const int row_local = quarter * 32 + lane;
        const int64_t row = (int64_t)rb * kBM + row_local;
        const bool row_ok = row < R;
        int64_t tgt = -1;
        if (row_ok) tgt = load_target(targets, targets_dtype, row);
        const int64_t tgt_local = (tgt >= 0) ? tgt - vocab_offset : -1;   // column inside this shard
        RowSums sums;
        for (int t = 0; t < ntiles && !timed_out; ++t) {
            const uint32_t buf = t & 1, bph = (t >> 1) & 1;
            if (!mbar_wait(&tmem_full[buf], bph)) { timed_out = true; break; }
            tc_fence_after();
            const int col0 = (tile0 + t) * width, end = min(V, col0 + width);
            sums.take_row(tmem + ((uint32_t)(quarter * 32) << 16) + buf * kBN, col0, end, tgt_local);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tmem_empty[buf]);
        }
        if (row_ok && !timed_out) {
            float *o = out + ((size_t)split * R + row) * 3;
            o[0] = sums.m;
            o[1] = sums.ssum;
            o[2] = sums.zt;
        }
    }
    if (timed_out) atomicExch(status, (int)kDevTimeout);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 512);
}

// The same on pairs of CTAs (see sm100_pair_gemm.cuh): a pair owns 256 rows, each CTA 128 of them.
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
lm_head_ce_pair_kernel(const __grid_constant__ PairMaps maps, const void *__restrict__ targets, int targets_dtype, int64_t vocab_offset,
                       float *__restrict__ out /* [splits][R][3] */, int64_t R, int C, int V, int row_blocks, int width, int tiles_per_split, int *status) {
    extern __shared__ __align__(1024) unsigned char smem[];
    if (smem_u32(smem) & 1023u) {
        if (threadIdx.x == 0) atomicExch(status, (int)kDevInternal);
        return;
    }
    const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);
    const int pair = blockIdx.x >> 1, rb = pair % row_blocks, split = pair / row_blocks;
    const int total_tiles = (V + width - 1) / width, tile0 = split * tiles_per_split;
    const int ntiles = min(tiles_per_split, total_tiles - tile0);
    auto items = [&](int i, PairItem &w) {
        w = PairItem{rb * kPairM, (tile0 + i) * width, 0, C / kPairK};
        return i < ntiles;
    };
    PairGemm gemm;
    gemm.begin(smem, maps, warp);
    wait_for_previous();
    let_next_in();
    bool ok = true;
    if (warp == 0) {
        if (elect_one()) ok = gemm.produce(maps, width, items, [] {});
    } else if (warp == 1) {
        if (gemm.rank == 0 && elect_one()) ok = gemm.multiply(width, items);
    } else {
        const int quarter = warp & 3;
        const int64_t row = (int64_t)rb * kPairM + gemm.rank * 128 + quarter * 32 + lane;
        const int64_t tgt = row < R ? load_target(targets, targets_dtype, row) : -1, tgt_local = tgt >= 0 ? tgt - vocab_offset : -1;
        RowSums sums;
        for (int t = 0; t < ntiles; ++t) {
            if (!gemm.complete(t)) { ok = false; break; }
            const int col0 = (tile0 + t) * width, end = min(V, col0 + width);
            sums.take_row(gemm.tmem + ((uint32_t)(quarter * 32) << 16) + (t & 1) * kPairN, col0, end, tgt_local);
            gemm.release(t);
        }
        if (row < R && ok) {
            float *o = out + ((size_t)split * R + row) * 3;
            o[0] = sums.m;
            o[1] = sums.ssum;
            o[2] = sums.zt;
        }
    }
    __syncwarp();
    if (!ok) atomicExch(status, (int)kDevTimeout);
    gemm.end(warp);
}

// Combines `nparts` partial triples per row: out[row] = (M, sum_g s_g exp(m_g - M), sum_g zt_g).  A warp per row: a thread per row walked up
// to 148 triples one after the other, 16 us behind the 54 of 16 rows' product; now 4.6.
__global__ void __launch_bounds__(256) lm_head_combine_kernel(const float *__restrict__ parts, int nparts, float *__restrict__ out, int64_t R) {
    wait_for_previous();
    let_next_in();
    const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (row >= R) return;
    float M = -INFINITY;
    for (int g = lane; g < nparts; g += 32) M = fmaxf(M, parts[((size_t)g * R + row) * 3]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
    float s = 0.f, zt = 0.f;
    for (int g = lane; g < nparts; g += 32) {
        const float *p = parts + ((size_t)g * R + row) * 3;
        if (p[0] > -INFINITY) s += p[1] * expf(p[0] - M);
        zt += p[2];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        zt += __shfl_xor_sync(0xffffffffu, zt, o);
    }
    if (lane < 3) out[row * 3 + lane] = lane == 0 ? M : lane == 1 ? s : zt;
}

__global__ void lm_head_finalize_kernel(const float *__restrict__ parts, int nparts, const void *__restrict__ targets,
                                        int targets_dtype, float *__restrict__ lse, float *__restrict__ loss,
                                        int64_t R) {
    wait_for_previous();
    let_next_in();
    const int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= R) return;
    float M = -INFINITY;
    for (int g = 0; g < nparts; ++g) M = fmaxf(M, parts[((size_t)g * R + row) * 3]);
    float s = 0.f, zt = 0.f;
    for (int g = 0; g < nparts; ++g) {
        const float *p = parts + ((size_t)g * R + row) * 3;
        if (p[0] > -INFINITY) s += p[1] * expf(p[0] - M);
        zt += p[2];
    }
    const float l = M + logf(s);
    lse[row] = l;
    loss[row] = load_target(targets, targets_dtype, row) >= 0 ? l - zt : 0.f;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

EncodeTiledFn lm_encode_fn() {
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

}  // namespace

// Upper bound for any device: one triple per row per vocabulary split, at most max_splits of them.  (Fewer rows may have more
// splits: a workspace laid out for the largest batch serves a smaller one with as many as it has room for.)
size_t lm_head_ce_workspace_bytes(int64_t R, int64_t C, int64_t V) {
    (void)C;
    return gemm_plan::split_bytes(R, V, gemm_plan::max_splits(R));
}
size_t lm_head_ce_min_workspace_bytes(int64_t R, int64_t C, int64_t V) {
    (void)C;
    return gemm_plan::split_bytes(R, V, gemm_plan::kFewSplits);
}

int launch_lm_head_ce_partial(const LmHeadArgs &p, void *workspace, size_t workspace_bytes, cudaStream_t stream) {
    EncodeTiledFn encode = lm_encode_fn();
    if (encode == nullptr) return (int)cudaErrorNotSupported;
    if ((reinterpret_cast<uintptr_t>(p.x) & 15u) || (reinterpret_cast<uintptr_t>(p.w) & 15u))
        return (int)cudaErrorMisalignedAddress;
    const int64_t room = workspace == nullptr ? 1 : std::max<int64_t>(1, (int64_t)(workspace_bytes / ((size_t)p.R * 3 * sizeof(float))));
    const gemm_plan::LmHeadCut cut = gemm_plan::lm_head_cut(p.R, p.C, p.V, p.num_sms, room);
    auto describe = [&](CUtensorMap *map, const void *ptr, int64_t rows, int box_rows) {
        const cuuint32_t estr[2] = {1, 1}, box[2] = {(cuuint32_t)kBK, (cuuint32_t)box_rows};
        const cuuint64_t dims[2] = {(cuuint64_t)p.C, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)p.C * 2};
        return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(ptr), dims, strides, box, estr,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    const int splits = cut.splits;
    float *parts = splits == 1 ? p.partials : static_cast<float *>(workspace);
    cudaError_t e;
    if (cut.pairs) {
        PairMaps maps;
        if (!describe(&maps.a, p.x, p.R, kPairM / 2) || !describe(&maps.b, p.w, p.V, cut.width / 2)) return (int)cudaErrorInvalidValue;
        e = cudaFuncSetAttribute(lm_head_ce_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPairSmem);
        if (e != cudaSuccess) return (int)e;
        e = launch_serialized(lm_head_ce_pair_kernel, (unsigned)(2 * cut.row_blocks * splits), (unsigned)kPairThreads, kPairSmem, stream, maps, p.targets,
                              p.targets_dtype, p.vocab_offset, parts, p.R, (int)p.C, (int)p.V, cut.row_blocks, cut.width, cut.tiles_per_split, p.status);
    } else {
        LmMaps maps;
        if (!describe(&maps.x, p.x, p.R, kBM) || !describe(&maps.w, p.w, p.V, cut.width)) return (int)cudaErrorInvalidValue;
        e = cudaFuncSetAttribute(lm_head_ce_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
        if (e != cudaSuccess) return (int)e;
        e = launch_serialized(lm_head_ce_kernel, (unsigned)(cut.row_blocks * splits), (unsigned)kThreads, kSmemBytes, stream, maps, p.targets, p.targets_dtype,
                              p.vocab_offset, parts, p.R, (int)p.C, (int)p.V, cut.row_blocks, cut.width, cut.tiles_per_split, p.status);
    }
    if (e == cudaSuccess && splits > 1)
        e = launch_serialized(lm_head_combine_kernel, (unsigned)((p.R + 7) / 8), 256u, 0, stream, (const float *)parts, splits, p.partials, p.R);
    return (int)e;
}

int launch_lm_head_ce_finalize(const float *partials_all, int num_shards, const void *targets, int targets_dtype,
                               float *lse, float *loss, int64_t R, cudaStream_t stream) {
    return (int)launch_serialized(lm_head_finalize_kernel, (unsigned)((R + 255) / 256), 256u, 0, stream, partials_all, num_shards, targets, targets_dtype, lse,
                                  loss, R);
}

}  // namespace rwkv7
