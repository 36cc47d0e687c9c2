// Last part of the WKV7 training step (N == 64, bf16 tensors, 64-token chunks): from the state S in front of every chunk
// (kept by the forward scan) and the gradient G of the state behind it (kept by the gradient scan) the gradients of
// receptance, decay, keys, removal key and replacement, all chunks in parallel.
//
// Gradient definitions: the reference's wkv7_backward_kernel (crates/rwkv-nn/src/kernels/train/time_mixer/wkv7/kernel.rs:395-690).
// In matrices over a 16-token block, with the decay D_t from the block's start to token t (inclusive), D its value at the
// end, and a reference point mu per channel, the power of two nearest sqrt(D) (so that no factor leaves e^+-6):
//     a~_t = a_t D_{t-1} / mu   r~_t = r_t D_t / mu   b^_s = b_s mu / D_s   k^_s = k_s mu / D_s
//     A_ab[t][s] = a~_t . b^_s (s < t)   A_ak = a~_t . k^_s (s < t)   A_rb[t][s] = r~_t . b^_s (s <= t)
//     U = T (a~ (S mu)^T + A_ak V)                         T = (I - A_ab)^-1,  u_t = S_{t-1} a_t
//     S' = (D / mu) (S mu + U^T b^ + V^T k^)               state at the block's end
//     dU = T^T (b^ (G rho)^T + A_rb^T dY)                  rho = D / mu
//     G' = mu (G rho + dY^T r~ + dU^T a~)                  gradient of the state at the block's start
//     dr = (D_t / mu) (dY (S mu) + B_rb b^ + B_rk k^)      B_rb = dY U^T, B_rk = dY V^T   (s <= t)
//     da = (D_{t-1} / mu) (dU (S mu) + B_ab b^ + B_ak k^)  B_ab = dU U^T, B_ak = dU V^T   (s < t)
//     db = (mu / D_s) (U (G rho) + B_rb^T r~ + B_ab^T a~)  dk = (mu / D_s) (V (G rho) + B_rk^T r~ + B_ak^T a~)
// The decay's gradient follows from phi_t = colsum(Gh_t . S_t) at a block's boundary: with x_t = b_t db_t + k_t dk_t - r_t dr_t
//     d_t dd_t = phi_t - x_t,   phi_{t-1} = phi_t - x_t + a_t da_t,   dw_t = -exp(w_t) d_t dd_t.
// dv is an output of the gradient scan.
//
// States, accumulators, decays and sums are fp32; matrix operands are fp16 (11 significant bits), S with V and G with dY scaled
// by a power of two per chunk, k and r by what then is between the two (see below).  A chunk whose decay leaves the range of the
// reference points, where a value leaves that of fp16, or with rows of a or b that are all below 2^-12 (u and du are as small, and
// db and da are made of them; a model's are of length one), is recomputed token by token in fp32.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "kernels.h"
#include "launch.h"
#include "sm100_mma.cuh"
#include "sm100_umma.cuh"
#include "trace.h"
#include "wkv7_tiles.cuh"

namespace rwkv7 {
namespace {

using namespace sm100;

constexpr int kThreads = 256;
constexpr float kTiny = 2.44140625e-4f;   // 2^-12
enum { TA = 0, TR, TB, TK, TV, TY, TW, kTensors };
constexpr uint32_t kTilesBytes = kTensors * kPanel;             // one of two buffers of input tiles
constexpr uint32_t kF = 2 * kTilesBytes;                         // D_{t-1} / mu and D_t / mu, fp16 tiles [token][channel]
constexpr uint32_t kS = kF + 2 * kPanel;                         // [4] S mu of block q, fp16 tiles [value row][channel]
constexpr uint32_t kG = kS + 4 * kPanel;                         // [4] G rho, the same
constexpr uint32_t kU = kG + 4 * kPanel;                         // U and dU, tiles [token][value row]
constexpr uint32_t kDU = kU + kPanel;
constexpr uint32_t kAak = kDU + kPanel;                          // [4] blocks each of A_ak, A_rb, T
constexpr uint32_t kArb = kAak + 4 * kBlk;
constexpr uint32_t kT = kArb + 4 * kBlk;
constexpr uint32_t kDiag = kT + 4 * kBlk;                        // [4] A_ab in fp32
constexpr uint32_t kMu = kDiag + 4 * 1024;                       // [4][64] fp32 each
constexpr uint32_t kRho = kMu + 1024;
constexpr uint32_t kFactorRow = 320;                             // (16 floats for each lane of a row group and 16 bytes: their banks differ)
constexpr uint32_t kFactors = kRho + 1024;                       // [8][80] fp32: from block to block, S then G; channel order of factor_place
constexpr uint32_t kE = kFactors + 8 * kFactorRow;                         // [8][64] fp32: decay over half a block
constexpr uint32_t kTop = kE + 2048;                             // [16] largest magnitudes: of S and V, of G and dY, by warp
constexpr uint32_t kBars = kTop + 64;
constexpr uint32_t kSmem = kBars + 64;
static_assert(kS % 1024 == 0 && kSmem <= 232448, "shared memory");

struct ChunkMaps {
    CUtensorMap in[kTensors];   // [B*T, H*N] bf16, box 64 x 64, 128-byte swizzle
    CUtensorMap out[5];         // da, dr, db, dk, dw, the same
    CUtensorMap block[5];       // and with box 64 x 16, for a chunk that ends early
};
struct ChunkArgs {
    const __nv_bfloat16 *in[kTensors];
    __nv_bfloat16 *out[5];
    const unsigned char *records;   // [chain][chunk], of which the exponents of r and k rows are read
    // [chain][chunk][64 x 64], in the order of accumulator_place; behind them eight largest magnitudes each, as float bits
    const float *states, *gradients;
    int T, H, nchunks;
    int units;
    int *status;
};

__device__ __forceinline__ void stsm4(uint32_t addr, const uint32_t (&r)[4]) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}
// transposed 16 x 16 block, A order to A order
__device__ __forceinline__ void transpose16(uint32_t (&y)[4], const uint32_t (&x)[4]) {
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y[0]) : "r"(x[0]));
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y[1]) : "r"(x[2]));
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y[2]) : "r"(x[1]));
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y[3]) : "r"(x[3]));
}
__device__ __forceinline__ void pack_block(uint32_t (&x)[4], const float (&c0)[4], const float (&c1)[4]) {
    x[0] = pack_half2(c0[0], c0[1]);
    x[1] = pack_half2(c0[2], c0[3]);
    x[2] = pack_half2(c1[0], c1[1]);
    x[3] = pack_half2(c1[2], c1[3]);
}
// Channels 8 n + 2 q, + 1 of all n next to one another: what lane q of a row group multiplies its accumulators with.
__device__ __forceinline__ int factor_place(int j) { return ((j & 7) >> 1) * 20 + (j >> 3) * 2 + (j & 1); }
__device__ __forceinline__ uint32_t pack_bf2(float lo, float hi) {
    const __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&b);
}

// Largest of four signed bytes.
__device__ __forceinline__ int most_of_four(uint32_t x) {
    return max(max((int)(signed char)x, (int)(signed char)(x >> 8)), max((int)(signed char)(x >> 16), (int)(signed char)(x >> 24)));
}
// Whether eight rows of a removal key or replacement are below what its products keep their bits at, but not zero.
__device__ __forceinline__ bool tiny(const uint32_t (&x)[8]) {
    __nv_bfloat162 m = __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll
    for (int u = 0; u < 8; ++u) m = __hmax2(m, __habs2(*reinterpret_cast<const __nv_bfloat162 *>(&x[u])));
    const float most = fmaxf(__low2float(m), __high2float(m));
    return !__any_sync(0xffffffffu, most >= kTiny) && __any_sync(0xffffffffu, most > 0.f);
}

// One chunk in fp32, token by token.  Four lanes per value row, columns c0 + 16 kk + e, for u = S a and du = G b; then four lanes per
// column, rows c0 + 16 kk + e, where with u and du known the state and its gradient need no sum over a row any more, and the sums over
// rows that the gradients are stay within four lanes.  `raw`: 56 KB of shared memory for the chunk's tensors, `d`: 16 KB, `sums`: 64 KB.
__device__ __noinline__ void chunk_by_token(const ChunkArgs &p, int unit, __nv_bfloat16 *raw, float *d, float *sums) {
    const int tid = threadIdx.x;
    const int own = tid >> 2, c0 = (tid & 3) * 4;   // row, or column; of the other
    const int chain = unit / p.nchunks, chunk = unit % p.nchunks;
    const int valid = min(kL, p.T - chunk * kL);
    const size_t base = (((size_t)(chain / p.H) * p.T + chunk * kL) * p.H + chain % p.H) * kN, step = (size_t)p.H * kN;
    float *u = sums, *du = u + kL * kN, *dr = du + kL * kN, *da = dr + kL * kN;
    __syncthreads();   // (the tiles and the operands are no longer read)
    for (int idx = tid; idx < kTensors * kL * 8; idx += kThreads) {
        const int x = idx / (kL * 8), t = idx / 8 % kL, c = idx % 8 * 8;
        if (t < valid) *reinterpret_cast<uint4 *>(raw + (x * kL + t) * kN + c) = *reinterpret_cast<const uint4 *>(p.in[x] + base + t * step + c);
    }
    __syncthreads();
    for (int i = tid; i < valid * kN; i += kThreads) d[i] = expf(-expf(__bfloat162float(raw[TW * kL * kN + i])));
    __syncthreads();
    auto one = [&](int x, int t) -> float { return __bfloat162float(raw[(x * kL + t) * kN + own]); };
    struct Four { float v[4]; };
    auto four = [&](int x, int t, int kk) {
        const uint2 w = *reinterpret_cast<const uint2 *>(raw + (x * kL + t) * kN + c0 + 16 * kk);
        const float2 lo = unpack_bf2(w.x), hi = unpack_bf2(w.y);
        return Four{{lo.x, lo.y, hi.x, hi.y}};
    };
    auto four_f32 = [&](const float *v, int t, int kk) {
        const float4 w = *reinterpret_cast<const float4 *>(v + t * kN + c0 + 16 * kk);
        return Four{{w.x, w.y, w.z, w.w}};
    };
    auto over_four = [](float x) {
        x += __shfl_xor_sync(0xffffffffu, x, 1);
        return x + __shfl_xor_sync(0xffffffffu, x, 2);
    };
    float M[4][4];
    auto load = [&](const float *src, bool by_row) {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int other = c0 + 16 * kk + e;
                M[kk][e] = src[(size_t)unit * kN * kN + (by_row ? accumulator_place(own, other) : accumulator_place(other, own))];
            }
    };
    // rows: u, then du
    load(p.states, true);
    for (int t = 0; t < valid; ++t) {
        float sa = 0.f;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            const Four a = four(TA, t, kk);
#pragma unroll
            for (int e = 0; e < 4; ++e) sa = fmaf(M[kk][e], a.v[e], sa);
        }
        sa = over_four(sa);
        if (c0 == 0) u[t * kN + own] = sa;
        const float vi = one(TV, t);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            const Four dd = four_f32(d, t, kk), b = four(TB, t, kk), k = four(TK, t, kk);
#pragma unroll
            for (int e = 0; e < 4; ++e) M[kk][e] = fmaf(M[kk][e], dd.v[e], fmaf(sa, b.v[e], vi * k.v[e]));
        }
    }
    load(p.gradients, true);
    for (int t = valid - 1; t >= 0; --t) {
        const float dy = one(TY, t);
        float dsa = 0.f;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            const Four r = four(TR, t, kk), b = four(TB, t, kk);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                M[kk][e] = fmaf(dy, r.v[e], M[kk][e]);
                dsa = fmaf(M[kk][e], b.v[e], dsa);
            }
        }
        dsa = over_four(dsa);
        if (c0 == 0) du[t * kN + own] = dsa;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            const Four dd = four_f32(d, t, kk), a = four(TA, t, kk);
#pragma unroll
            for (int e = 0; e < 4; ++e) M[kk][e] = fmaf(M[kk][e], dd.v[e], dsa * a.v[e]);
        }
    }
    __syncthreads();
    // columns: da and dr forwards, then the rest backwards
    load(p.states, false);
    for (int t = 0; t < valid; ++t) {
        const float dj = d[t * kN + own], b = one(TB, t), k = one(TK, t);
        float sum_a = 0.f, sum_r = 0.f;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            const Four ui = four_f32(u, t, kk), dui = four_f32(du, t, kk), v = four(TV, t, kk), dy = four(TY, t, kk);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                sum_a = fmaf(M[kk][e], dui.v[e], sum_a);
                M[kk][e] = fmaf(M[kk][e], dj, fmaf(ui.v[e], b, v.v[e] * k));
                sum_r = fmaf(M[kk][e], dy.v[e], sum_r);
            }
        }
        sum_a = over_four(sum_a);
        sum_r = over_four(sum_r);
        if (c0 == 0) {
            da[t * kN + own] = sum_a;
            dr[t * kN + own] = sum_r;
        }
    }
    float phi = 0.f, end[4][4];
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
#pragma unroll
        for (int e = 0; e < 4; ++e) end[kk][e] = M[kk][e];
    load(p.gradients, false);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
#pragma unroll
        for (int e = 0; e < 4; ++e) phi = fmaf(end[kk][e], M[kk][e], phi);
    phi = over_four(phi);
    __syncwarp();   // (da and dr are this quad's own)
    for (int t = valid - 1; t >= 0; --t) {
        const float dj = d[t * kN + own], r = one(TR, t), a = one(TA, t);
        float sum_k = 0.f, sum_b = 0.f;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            const Four ui = four_f32(u, t, kk), dui = four_f32(du, t, kk), v = four(TV, t, kk), dy = four(TY, t, kk);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                M[kk][e] = fmaf(dy.v[e], r, M[kk][e]);
                sum_k = fmaf(M[kk][e], v.v[e], sum_k);
                sum_b = fmaf(M[kk][e], ui.v[e], sum_b);
                M[kk][e] = fmaf(M[kk][e], dj, dui.v[e] * a);
            }
        }
        sum_k = over_four(sum_k);
        sum_b = over_four(sum_b);
        const float sum_a = da[t * kN + own], sum_r = dr[t * kN + own];
        const float x = one(TB, t) * sum_b + one(TK, t) * sum_k - r * sum_r;
        const size_t o = base + t * step + own;
        const int q = tid & 3;   // (a lane of the four stores one of the gradients)
        (q == 0 ? p.out[TA] : q == 1 ? p.out[TR] : q == 2 ? p.out[TB] : p.out[TK])[o] =
            __float2bfloat16_rn(q == 0 ? sum_a : q == 1 ? sum_r : q == 2 ? sum_b : sum_k);
        if (q == 0) p.out[4][o] = __float2bfloat16_rn(-expf(one(TW, t)) * (phi - x));
        phi -= x - a * sum_a;
    }
    __syncthreads();
}

// One CTA of eight warps per SM, chunk after chunk; the next chunk's tiles arrive in the other buffer meanwhile.  Warp = 16 value
// rows of S (warps 0-3) or G (warps 4-7): a row of the state never needs another row, so the state stays in the matrix
// instructions' accumulators over the four blocks of the chunk, S forwards and G backwards, without a barrier.  What the gradients need of
// it (S mu, G rho, U, dU) is left in shared memory, and then warp = (block, half of the channels) sums over value rows.
//
// Bound by the shared-memory port, busy two thirds of the time (9 k wavefronts of 13.5 k cycles a chunk), and by latency with two warps per
// scheduler (225 KB of shared memory leave room for one CTA); the matrix instructions take 4.3 k of a scheduler.  Measured, 6144 chunks:
// 335 us; the fp32 replay per 16 tokens that this replaced took 880, and 90 for the reversed copies it needed.  Not kept: four more warps
// that prepare the next chunk meanwhile (they share the port and the issue slots), sixteen warps with half the channels or tokens each (57 us
// more: every warp reads its first operands itself), U and V moved in registers to be second operands instead of read again (4 us more).
__global__ void __launch_bounds__(kThreads, 1)
wkv7_chunk_gradients_kernel(const __grid_constant__ ChunkMaps maps, const __grid_constant__ ChunkArgs p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    if (smem_u32(smem) & 1023u) {
        if (threadIdx.x == 0) atomicExch(p.status, (int)kDevInternal);
        return;
    }
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int g = lane >> 2, c2 = 2 * (lane & 3);
    const uint32_t sb = smem_u32(smem);
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + kBars);   // [2] a buffer's tiles have landed
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + kBars + 16);
    if (tid == 0) {
        mbar_init(bar, 1);
        mbar_init(bar + 1, 1);
        mbar_fence_init();
        *abort_flag = 0;
    }
    auto coordinates = [&](int unit, int &x, int &y) {
        const int chain = unit / p.nchunks;
        x = (chain % p.H) * kN;
        y = (chain / p.H) * p.T + unit % p.nchunks * kL;
    };
    auto request = [&](int unit, int buf) {
        int x, y;
        coordinates(unit, x, y);
        mbar_expect_tx(bar + buf, kTilesBytes);
#pragma unroll
        for (int i = 0; i < kTensors; ++i) tma_load_2d(smem + buf * kTilesBytes + i * kPanel, &maps.in[i], x, y, bar + buf);
    };
    __syncthreads();
    // (the call's inputs are requested while the gradient scan in front, which writes none of them, finishes: see launch.h)
    if (warp == 7 && elect_one() && (int)blockIdx.x < p.units) request(blockIdx.x, 0);
    __syncwarp();
    wait_for_previous();
    // this warp's 16 rows of S or G, in accumulator order: c[n] = rows g, g + 8, columns 8 n + c2, + 1
    const int wr = warp & 3;
    const bool g_side = warp >= 4;
    float c[8][4];
    auto fetch = [&](int unit) {
        const float *src = (g_side ? p.gradients : p.states) + (size_t)unit * kN * kN + (wr * 256 + lane) * 4;
        if (RWKV7_IN_RANGE(unit >= 0 && unit < p.units, p.status)) {
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                const float4 x = __ldcs(reinterpret_cast<const float4 *>(src + n * 128));
                c[n][0] = x.x; c[n][2] = x.y; c[n][1] = x.z; c[n][3] = x.w;
            }
        }
    };
    if ((int)blockIdx.x < p.units) fetch(blockIdx.x);
    const uint32_t *tops_s = reinterpret_cast<const uint32_t *>(p.states + (size_t)p.units * kN * kN);
    const uint32_t *tops_g = reinterpret_cast<const uint32_t *>(p.gradients + (size_t)p.units * kN * kN);
    auto row_exponents = [&](int unit) { return *reinterpret_cast<const uint2 *>(p.records + (size_t)unit * kRecord + kDecayAt + kRowExpAt); };
    uint2 row_exp_next = (int)blockIdx.x < p.units ? row_exponents(blockIdx.x) : make_uint2(0u, 0u);
    int seq = 0;
    for (int unit = blockIdx.x; unit < p.units; unit += (int)gridDim.x, ++seq) {
        const int buf = seq & 1;
        const uint32_t tiles = sb + buf * kTilesBytes;
        const int valid = min(kL, p.T - unit % p.nchunks * kL), nblk = valid / 16;
        const uint2 row_exp = row_exp_next;   // (a line of its own in memory for every chunk: fetched a chunk ahead)
        if (unit + (int)gridDim.x < p.units) row_exp_next = row_exponents(unit + (int)gridDim.x);
        const uint32_t state_top = lane < 16 ? (lane < 8 ? tops_s : tops_g)[(size_t)unit * 8 + (lane & 7)] : 0u;
        if (!mbar_wait(bar + buf, (uint32_t)((seq >> 1) & 1))) *abort_flag = 1;
        __syncwarp();
        // ---------------- 1. decays of half a block per warp, lane = channel pair; largest magnitudes
        const int tb = wr, hf = warp >> 2, ch = 2 * lane, t_first = 16 * tb + 8 * hf;
        const int nv = min(8, max(0, valid - t_first));       // 0 or 8
        // (t_first is a multiple of eight: the swizzle depends on u alone)
        auto at = [&](int x, int u) -> uint32_t { return tiles + t_first * 128 + x * kPanel + off16(u, ch); };
        uint32_t rv[8], ry[8];
        float2 d[8], e = make_float2(1.f, 1.f);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const uint32_t w = lds32(at(TW, u));
            rv[u] = nv ? lds32(at(TV, u)) : 0u;
            ry[u] = nv ? lds32(at(TY, u)) : 0u;
            d[u] = nv ? decay2(unpack_bf2(w)) : make_float2(1.f, 1.f);
            e = mul2(e, d[u]);
        }
        sts_f2(sb + kE + ((2 * tb + hf) * 64 + ch) * 4, e.x, e.y);
        {
            __nv_bfloat162 m = __floats2bfloat162_rn(0.f, 0.f), my = m;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                m = __hmax2(m, __habs2(*reinterpret_cast<const __nv_bfloat162 *>(&rv[u])));
                my = __hmax2(my, __habs2(*reinterpret_cast<const __nv_bfloat162 *>(&ry[u])));
            }
            const uint32_t a = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(__low2float(m), __high2float(m)))),
                           b = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(__low2float(my), __high2float(my))));
            if (lane == 0) {
                sts32(sb + kTop + warp * 4, a);
                sts32(sb + kTop + 32 + warp * 4, b);
            }
        }
        __syncthreads();
        if (*abort_flag) break;
        // ---------------- 2. scaled fp16 operands, in place; D_t / mu
        // V and dY are scaled alone (dk, dr are made of them); S and G with what V k^T and dY r^T add to them, and k and r by
        // what is left between the two: V 2^-ev, S 2^-es, k 2^(ev - es), dY 2^-ey, G 2^-eg, r 2^(ey - eg).
        int es, ev, eg, ey;
        {
            const int er = most_of_four(__byte_perm(row_exp.x, row_exp.y, 0x6420)), ek = most_of_four(__byte_perm(row_exp.x, row_exp.y, 0x7531));
            const uint32_t own = lane < 16 ? 0u : lds32(sb + kTop + (lane - 16) * 4);
            auto largest = [&](uint32_t x, int &e) {
                const uint32_t m = __reduce_max_sync(0xffffffffu, x);
                e = min(max((int)(m >> 23) - 127, -60), 60);
                return m != 0u;
            };
            const bool has_s = largest(lane < 8 ? state_top : 0u, es), has_v = largest(lane >= 16 && lane < 24 ? own : 0u, ev);
            const bool has_g = largest(lane >= 8 && lane < 16 ? state_top : 0u, eg), has_y = largest(lane >= 24 ? own : 0u, ey);
            es = has_v ? max(has_s ? es : -60, max(ev + ek, -60)) : has_s ? es : 0;
            eg = has_y ? max(has_g ? eg : -60, max(ey + er, -60)) : has_g ? eg : 0;
            if (!has_v) ev = es;
            if (!has_y) ey = eg;
        }
        const float scale_s = exp2_of(-es), scale_g = exp2_of(-eg);
        bool over;
        {
            const float2 e0 = lds_f2(sb + kE + (2 * tb * 64 + ch) * 4), e1 = lds_f2(sb + kE + ((2 * tb + 1) * 64 + ch) * 4);
            const float2 D = mul2(e0, e1);
            over = !(D.x >= kBlockDecay && D.y >= kBlockDecay);
            // mu = 2^-h, h half of D's exponent
            const int hx = (127 - exponent_of(D.x)) >> 1, hy = (127 - exponent_of(D.y)) >> 1;
            const float2 mu = make_float2(exp2_of(-hx), exp2_of(-hy)), up = make_float2(exp2_of(hx), exp2_of(hy));
            const float2 rho = mul2(D, up);
            if (hf == 0) {
                sts_f2(sb + kMu + (tb * 64 + ch) * 4, mu.x, mu.y);
                sts_f2(sb + kRho + (tb * 64 + ch) * 4, rho.x, rho.y);
            }
            float2 f = hf ? mul2(e0, up) : up;
            const float2 rs = make_float2(exp2_of(ey - eg), exp2_of(ey - eg)), ks = make_float2(exp2_of(ev - es), exp2_of(ev - es));
            uint32_t x0[8], x1[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                x0[u] = nv ? lds32(at(TA, u)) : 0u;
                x1[u] = nv ? lds32(at(TR, u)) : 0u;
            }
            over |= tiny(x0);
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const uint32_t o = t_first * 128 + off16(u, ch);
                sts32(at(TA, u), pack2(mul2(unpack_bf2(x0[u]), f)));
                sts32(sb + kF + o, pack2(f));
                f = mul2(f, d[u]);
                sts32(at(TR, u), pack2(mul2(mul2(unpack_bf2(x1[u]), rs), f)));
                sts32(sb + kF + kPanel + o, pack2(f));
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                x0[u] = nv ? lds32(at(TB, u)) : 0u;
                x1[u] = nv ? lds32(at(TK, u)) : 0u;
            }
            over |= tiny(x0);
            f = make_float2(rcp(rho.x), rcp(rho.y));
            if (!hf) f = mul2(f, e1);
            const float2 vs = make_float2(exp2_of(-ev), exp2_of(-ev)), ys = make_float2(exp2_of(-ey), exp2_of(-ey));
#pragma unroll
            for (int u = 7; u >= 0; --u) {
                sts32(at(TB, u), pack2(mul2(unpack_bf2(x0[u]), f)));
                sts32(at(TK, u), pack2(mul2(mul2(unpack_bf2(x1[u]), ks), f)));
                f = mul2(f, d[u]);
                sts32(at(TV, u), pack2(mul2(unpack_bf2(rv[u]), vs)));
                sts32(at(TY, u), pack2(mul2(unpack_bf2(ry[u]), ys)));
            }
        }
        over = __syncthreads_or(over);
        bool bad = false;
        if (unit + (int)gridDim.x < p.units) {   // the next chunk: its tiles into the other buffer, its states into L2
            const int next = unit + (int)gridDim.x;
            if (warp == 7 && elect_one()) {
                bulk_wait_group_read<0>();   // the other buffer's gradients have left
                request(next, buf ^ 1);
            }
            __syncwarp();
            asm volatile("prefetch.global.L2 [%0];" ::"l"((tid < 128 ? p.states : p.gradients) + (size_t)next * kN * kN + (tid & 127) * 32));
        }
        if (!over) {
            // ---------------- 3. warps 0-3: A_ab of a block and T; warps 4-7: A_ak, A_rb
            {
                const int q = wr;
                float m[2][2][4] = {};
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    uint32_t A[4], B[4];
                    ldsm4(A, tiles + TA * kPanel + tile_plain(lane, 16 * q, kk));
                    ldsm4(B, tiles + (g_side ? TK : TB) * kPanel + tile_cols(lane, 16 * q, kk));
                    mma16816(m[0][0], A, B[0], B[1]);
                    mma16816(m[0][1], A, B[2], B[3]);
                    if (g_side) {
                        ldsm4(A, tiles + TR * kPanel + tile_plain(lane, 16 * q, kk));
                        ldsm4(B, tiles + TB * kPanel + tile_cols(lane, 16 * q, kk));
                        mma16816(m[1][0], A, B[0], B[1]);
                        mma16816(m[1][1], A, B[2], B[3]);
                    }
                }
                if (g_side) {
                    {   // factors from the block before (S: mu rho', G: rho mu') to this one
                        const uint32_t own = sb + (q * 64 + ch) * 4;
                        const float2 mu = lds_f2(own + kMu), rho = lds_f2(own + kRho);
                        const float2 fs = q == 0 ? make_float2(scale_s, scale_s) : lds_f2(own + kRho - 256), fg = q == 3 ? make_float2(scale_g, scale_g) : lds_f2(own + kMu + 256);
                        const uint32_t o = sb + kFactors + q * kFactorRow + factor_place(ch) * 4;
                        sts_f2(o, mu.x * fs.x, mu.y * fs.y);
                        sts_f2(o + 4 * kFactorRow, rho.x * fg.x, rho.y * fg.y);
                    }
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        const uint32_t o = sb + (x ? kArb : kAak) + q * kBlk + lane * 4;
#pragma unroll
                        for (int h = 0; h < 2; ++h)
#pragma unroll
                            for (int r = 0; r < 2; ++r) {
                                const int t = g + 8 * r + x, s = 8 * h + c2;   // kept: s < t (A_ak), s <= t (A_rb)
                                sts32(o + h * 256 + r * 128, pack_half2(s < t ? m[x][h][2 * r] : 0.f, s + 1 < t ? m[x][h][2 * r + 1] : 0.f));
                            }
                    }
                } else {
                    const uint32_t src = sb + kDiag + q * 1024;
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            const int t = g + 8 * r, piece = 2 * h + (c2 >> 2);
                            sts_f2(src + t * 64 + ((piece ^ ((t >> 1) & 3)) << 4) + (c2 & 2) * 4, m[0][h][2 * r], m[0][h][2 * r + 1]);
                        }
                    __syncwarp();
                    // forward substitution, a column per lane (both half-warps the same)
                    const int cc = lane & 15;
                    float x[16];
#pragma unroll
                    for (int t = 0; t < 16; ++t) {
                        float acc0 = 0.f, acc1 = 0.f;
#pragma unroll
                        for (int s4 = 0; s4 < (t + 3) / 4; ++s4) {
                            const float4 a4 = lds_f4(src + t * 64 + ((s4 ^ ((t >> 1) & 3)) << 4));
                            if (4 * s4 + 0 < t) acc0 = fmaf(a4.x, x[4 * s4 + 0], acc0);
                            if (4 * s4 + 1 < t) acc1 = fmaf(a4.y, x[4 * s4 + 1], acc1);
                            if (4 * s4 + 2 < t) acc0 = fmaf(a4.z, x[4 * s4 + 2], acc0);
                            if (4 * s4 + 3 < t) acc1 = fmaf(a4.w, x[4 * s4 + 3], acc1);
                        }
                        x[t] = (t == cc) ? 1.f : acc0 + acc1;
                    }
                    if (lane < 16) {
                        unsigned char *dst = smem + kT + q * kBlk + (cc >> 3) * 256 + (cc & 7) * 2;
#pragma unroll
                        for (int t = 0; t < 16; ++t) *reinterpret_cast<__half *>(dst + t * 16) = __float2half_rn(x[t]);
                    }
                }
            }
            __syncthreads();
            // ---------------- 4. the state, block by block: S forwards, G backwards
            {
                const uint32_t own = sb + (g_side ? kG : kS), rows = sb + (g_side ? kDU : kU);
                const uint32_t left = tiles + (g_side ? TY : TV) * kPanel;      // V or dY
                const uint32_t with = tiles + (g_side ? TB : TA) * kPanel;      // what S or G is multiplied with: a~ or b^
                const uint32_t mat = sb + (g_side ? kArb : kAak);
                const uint32_t up_u = tiles + (g_side ? TA : TB) * kPanel, up_l = tiles + (g_side ? TR : TK) * kPanel;
#pragma unroll 1
                for (int i = 0; i < 4; ++i) {
                    const int q = g_side ? 3 - i : i;
                    {
                        const uint32_t f0 = sb + kFactors + (g_side ? 4 * kFactorRow : 0) + q * kFactorRow + (lane & 3) * 80;
#pragma unroll
                        for (int n = 0; n < 8; n += 2) {
                            const float4 f = lds_f4(f0 + n * 8);
#pragma unroll
                            for (int r = 0; r < 4; r += 2) {
                                const float2 a = mul2(make_float2(c[n][r], c[n][r + 1]), make_float2(f.x, f.y));
                                const float2 b = mul2(make_float2(c[n + 1][r], c[n + 1][r + 1]), make_float2(f.z, f.w));
                                c[n][r] = a.x; c[n][r + 1] = a.y;
                                c[n + 1][r] = b.x; c[n + 1][r + 1] = b.y;
                            }
                        }
                    }
                    uint32_t L[4], M[4];
                    float o[2][2][4] = {};
                    ldsm4_t(L, left + tile_cols(lane, 16 * q, wr));
                    if (g_side) ldsm4_t(M, mat + q * kBlk + blk_plain(lane));
                    else ldsm4(M, mat + q * kBlk + blk_cols(lane));
                    mma16816(o[0][0], L, M[0], M[1]);
                    mma16816(o[0][1], L, M[2], M[3]);
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk) {
                        uint32_t A[4], B[4];
                        pack_block(A, c[2 * kk], c[2 * kk + 1]);
                        stsm4(own + q * kPanel + tile_plain(lane, 16 * wr, kk), A);
                        ldsm4(B, with + tile_cols(lane, 16 * q, kk));
                        mma16816(o[kk & 1][0], A, B[0], B[1]);
                        mma16816(o[kk & 1][1], A, B[2], B[3]);
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int x = 0; x < 4; ++x) o[0][h][x] += o[1][h][x];
                    uint32_t X[4], U[4];
                    pack_block(X, o[0][0], o[0][1]);
                    if (g_side) ldsm4_t(M, sb + kT + q * kBlk + blk_plain(lane));
                    else ldsm4(M, sb + kT + q * kBlk + blk_cols(lane));
                    mma16816_first(o[0][0], X, M[0], M[1]);
                    mma16816_first(o[0][1], X, M[2], M[3]);
                    pack_block(U, o[0][0], o[0][1]);
                    stsm4_t(rows + tile_cols(lane, 16 * q, wr), U[0], U[1], U[2], U[3]);
                    if (i < 3) {
#pragma unroll
                        for (int jj = 0; jj < 4; ++jj) {
                            uint32_t B[4];
                            ldsm4_t(B, up_l + tile_plain(lane, 16 * q, jj));
                            mma16816(c[2 * jj], L, B[0], B[1]);
                            mma16816(c[2 * jj + 1], L, B[2], B[3]);
                            ldsm4_t(B, up_u + tile_plain(lane, 16 * q, jj));
                            mma16816(c[2 * jj], U, B[0], B[1]);
                            mma16816(c[2 * jj + 1], U, B[2], B[3]);
                        }
                    }
                }
            }
            __syncthreads();
            // ---------------- 5. gradients of block q, channels 32 jh ..
            const int q = wr, jh = warp >> 2;
            if (q < nblk) {
                float acc[4][4][4] = {}, sc[4][2][4] = {};   // dr, da, db, dk; B_rb, B_rk, B_ab, B_ak
                // phi at the block's start, from its S and the G of the block before; at the first block's end, the other way round
                float2 phi[4] = {};
                const uint32_t other = sb + (q == 0 ? kS + kPanel : kG + (q - 1) * kPanel);
                const int bd = max(q, 1);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    uint32_t Y[4], D[4], U[4], V[4], X[2][4];
                    const uint32_t o = tile_plain(lane, 16 * q, kk);
                    ldsm4(Y, tiles + TY * kPanel + o);
                    ldsm4(D, sb + kDU + o);
                    ldsm4(U, sb + kU + o);
                    ldsm4(V, tiles + TV * kPanel + o);
                    uint32_t Z[2][4];
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        const uint32_t ox = tile_plain(lane, 16 * kk, 2 * jh + x);
                        ldsm4_t(X[x], sb + kS + q * kPanel + ox);
                        ldsm4_t(Z[x], other + ox);
                    }
                    auto boundary = [&] {
#pragma unroll
                        for (int x = 0; x < 2; ++x)
#pragma unroll
                            for (int i = 0; i < 4; ++i) phi[2 * x + (i >> 1)] = __ffma2_rn(unpack_half2(X[x][i]), unpack_half2(Z[x][i]), phi[2 * x + (i >> 1)]);
                    };
#pragma unroll
                    for (int n = 0; n < 4; ++n) {
                        mma16816(acc[0][n], Y, X[n >> 1][(n & 1) * 2], X[n >> 1][(n & 1) * 2 + 1]);
                        mma16816(acc[1][n], D, X[n >> 1][(n & 1) * 2], X[n >> 1][(n & 1) * 2 + 1]);
                    }
                    if (q > 0) boundary();
#pragma unroll
                    for (int x = 0; x < 2; ++x) ldsm4_t(X[x], sb + kG + q * kPanel + tile_plain(lane, 16 * kk, 2 * jh + x));
                    if (q == 0) boundary();
#pragma unroll
                    for (int n = 0; n < 4; ++n) {
                        mma16816(acc[2][n], U, X[n >> 1][(n & 1) * 2], X[n >> 1][(n & 1) * 2 + 1]);
                        mma16816(acc[3][n], V, X[n >> 1][(n & 1) * 2], X[n >> 1][(n & 1) * 2 + 1]);
                    }
                    // (as second operands a register pair holds both halves of k: read in that order, not moved)
                    const uint32_t oc = tile_cols(lane, 16 * q, kk);
                    ldsm4(X[0], sb + kU + oc);
                    ldsm4(X[1], tiles + TV * kPanel + oc);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        mma16816(sc[0][h], Y, X[0][2 * h], X[0][2 * h + 1]);
                        mma16816(sc[1][h], Y, X[1][2 * h], X[1][2 * h + 1]);
                        mma16816(sc[2][h], D, X[0][2 * h], X[0][2 * h + 1]);
                        mma16816(sc[3][h], D, X[1][2 * h], X[1][2 * h + 1]);
                    }
                }
                uint32_t P[4][4], Q[4][4];
#pragma unroll
                for (int m = 0; m < 4; ++m) {
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int x = 0; x < 4; ++x)
                            if (8 * h + c2 + (x & 1) > g + 8 * (x >> 1) - (m >> 1)) sc[m][h][x] = 0.f;
                    pack_block(P[m], sc[m][0], sc[m][1]);
                    transpose16(Q[m], P[m]);
                }
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    uint32_t B[4];
                    const uint32_t o = tile_plain(lane, 16 * q, 2 * jh + x);
                    auto both = [&](int i0, const uint32_t (&A0)[4], int i1, const uint32_t (&A1)[4]) {
#pragma unroll
                        for (int n = 0; n < 2; ++n) {
                            mma16816(acc[i0][2 * x + n], A0, B[2 * n], B[2 * n + 1]);
                            mma16816(acc[i1][2 * x + n], A1, B[2 * n], B[2 * n + 1]);
                        }
                    };
                    ldsm4_t(B, tiles + TB * kPanel + o);
                    both(0, P[0], 1, P[2]);
                    ldsm4_t(B, tiles + TK * kPanel + o);
                    both(0, P[1], 1, P[3]);
                    ldsm4_t(B, tiles + TR * kPanel + o);
                    both(2, Q[0], 3, Q[1]);
                    ldsm4_t(B, tiles + TA * kPanel + o);
                    both(2, Q[2], 3, Q[3]);
                }
                const float sigma = exp2_of(es + eg), sigma_r = exp2_of(ey + es), sigma_k = exp2_of(ev + eg);
                float finite = 0.f;
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const uint32_t o = tile_plain(lane, 16 * q, 2 * jh + x);
                    uint32_t ta[4], tr[4], tbb[4], tk[4], tw[4], fe[4], fi[4], out[5][4];
                    ldsm4(ta, tiles + TA * kPanel + o);
                    ldsm4(tr, tiles + TR * kPanel + o);
                    ldsm4(tbb, tiles + TB * kPanel + o);
                    ldsm4(tk, tiles + TK * kPanel + o);
                    ldsm4(tw, tiles + TW * kPanel + o);
                    ldsm4(fe, sb + kF + o);
                    ldsm4(fi, sb + kF + kPanel + o);
#pragma unroll
                    for (int n2 = 0; n2 < 2; ++n2) {
                        const int n = 2 * x + n2, j = 32 * jh + 8 * n + c2;
                        float2 xs[2], z[2], suf[2];
#pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            const int i = n2 * 2 + r;
                            const float2 dr = make_float2(acc[0][n][2 * r], acc[0][n][2 * r + 1]), da = make_float2(acc[1][n][2 * r], acc[1][n][2 * r + 1]);
                            const float2 db = make_float2(acc[2][n][2 * r], acc[2][n][2 * r + 1]), dk = make_float2(acc[3][n][2 * r], acc[3][n][2 * r + 1]);
                            const float2 rr = unpack_half2(tr[i]), aa = unpack_half2(ta[i]);
                            xs[r] = __ffma2_rn(unpack_half2(tbb[i]), db, __ffma2_rn(unpack_half2(tk[i]), dk, mul2(make_float2(-rr.x, -rr.y), dr)));
                            z[r] = __ffma2_rn(make_float2(-aa.x, -aa.y), da, xs[r]);
                            suf[r] = z[r];
                        }
                        // sums of z over this token and the later ones of its half of the block (over g), then the block
#pragma unroll
                        for (int s = 4; s <= 16; s <<= 1)
#pragma unroll
                            for (int r = 0; r < 2; ++r) {
                                const float vx = __shfl_down_sync(0xffffffffu, suf[r].x, s), vy = __shfl_down_sync(0xffffffffu, suf[r].y, s);
                                if (lane + s < 32) { suf[r].x += vx; suf[r].y += vy; }
                            }
                        const float hx = __shfl_sync(0xffffffffu, suf[1].x, lane & 3), hy = __shfl_sync(0xffffffffu, suf[1].y, lane & 3);
                        suf[0].x += hx;
                        suf[0].y += hy;
                        // (phi: lane (g, q') holds the rows of its q' of column 8 n + g)
                        float pc = phi[n].x + phi[n].y;
                        pc += __shfl_xor_sync(0xffffffffu, pc, 1);
                        pc += __shfl_xor_sync(0xffffffffu, pc, 2);
                        const float2 m0 = lds_f2(sb + kMu + (bd * 64 + j) * 4), m1 = lds_f2(sb + kRho + ((bd - 1) * 64 + j) * 4);
                        float2 ph = make_float2(__shfl_sync(0xffffffffu, pc, 4 * c2) * rcp(m0.x * m1.x), __shfl_sync(0xffffffffu, pc, 4 * c2 + 4) * rcp(m0.y * m1.y));
                        if (q > 0) {   // from the block's start: the whole block's sum on top
                            ph.x += __shfl_sync(0xffffffffu, suf[0].x, lane & 3);
                            ph.y += __shfl_sync(0xffffffffu, suf[0].y, lane & 3);
                        }
#pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            const int i = n2 * 2 + r;
                            const float2 s2 = make_float2(sigma, sigma), f = unpack_half2(fi[i]);
                            const float2 inv = make_float2(rcp(f.x), rcp(f.y));
                            const float2 fa = mul2(unpack_half2(fe[i]), s2), fr = mul2(f, make_float2(sigma_r, sigma_r)), fb = mul2(inv, s2), fk = mul2(inv, make_float2(sigma_k, sigma_k));
                            const float2 w = unpack_bf2(tw[i]);
                            constexpr float kLog2e = 1.4426950408889634f;
                            out[TA][i] = pack_bf2(acc[1][n][2 * r] * fa.x, acc[1][n][2 * r + 1] * fa.y);
                            out[TR][i] = pack_bf2(acc[0][n][2 * r] * fr.x, acc[0][n][2 * r + 1] * fr.y);
                            out[TB][i] = pack_bf2(acc[2][n][2 * r] * fb.x, acc[2][n][2 * r + 1] * fb.y);
                            out[TK][i] = pack_bf2(acc[3][n][2 * r] * fk.x, acc[3][n][2 * r + 1] * fk.y);
                            // d_t dd_t = phi_t - x_t, phi_t = phi at the boundary - the later tokens' z
                            const float px = ph.x - (suf[r].x - z[r].x) - xs[r].x, py = ph.y - (suf[r].y - z[r].y) - xs[r].y;
                            finite += fabsf(px) + fabsf(py);   // (every product above is part of it)
                            out[4][i] = pack_bf2(-ex2(w.x * kLog2e) * px * sigma, -ex2(w.y * kLog2e) * py * sigma);
                        }
                    }
                    __syncwarp();
                    // (the gradients take the place of the operands, which no other warp reads)
#pragma unroll
                    for (int i = 0; i < 4; ++i) stsm4(tiles + i * kPanel + o, out[i]);
                    stsm4(tiles + TW * kPanel + o, out[4]);
                }
                bad = !(finite <= 3.0e38f);
            }
            fence_proxy_async();
            if (unit + (int)gridDim.x < p.units) fetch(unit + (int)gridDim.x);   // (behind the fence, which waits for what was issued before it)
            bad = __syncthreads_or(bad);
            if (!bad && warp == 7 && elect_one()) {
                int x, y;
                coordinates(unit, x, y);
                const unsigned char *from = smem + buf * kTilesBytes;
                if (nblk == 4) {
#pragma unroll
                    for (int i = 0; i < 5; ++i) tma_store_2d(&maps.out[i], x, y, from + (i < 4 ? i : TW) * kPanel);
                } else {
                    for (int b = 0; b < nblk; ++b)
#pragma unroll
                        for (int i = 0; i < 5; ++i) tma_store_2d(&maps.block[i], x, y + 16 * b, from + (i < 4 ? i : TW) * kPanel + b * 2048);
                }
                bulk_commit_group();
            }
            __syncwarp();
        }
        if (over || bad) {
            if (over && unit + (int)gridDim.x < p.units) fetch(unit + (int)gridDim.x);
            chunk_by_token(p, unit, reinterpret_cast<__nv_bfloat16 *>(smem + buf * kTilesBytes), reinterpret_cast<float *>(smem + kF), reinterpret_cast<float *>(smem + kS));
            fence_proxy_async();
            __syncthreads();
        }
    }
    if (warp == 7 && elect_one()) {
        if (*abort_flag) {   // what is in flight lands before the CTA leaves
            mbar_wait(bar + (seq & 1), (uint32_t)((seq >> 1) & 1), 100000u);
            atomicExch(p.status, (int)kDevTimeout);
        }
        bulk_wait_group_read<0>();
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

}  // namespace

// Enqueues the chunk kernel behind the gradient scan.
int launch_wkv7_chunk_gradients(const Wkv7TrainingBackwardArgs &p, const unsigned char *records, const float *states, const float *gradients,
                                cudaStream_t stream) {
    static const EncodeTiledFn encode = [] {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        return cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess
                   ? reinterpret_cast<EncodeTiledFn>(fn) : nullptr;
    }();
    if (encode == nullptr) return (int)cudaErrorNotSupported;
    ChunkMaps maps{};
    ChunkArgs args{};
    const cuuint64_t dims[2] = {(cuuint64_t)(p.H * kN), (cuuint64_t)(p.B * p.T)};
    const cuuint64_t strides[1] = {(cuuint64_t)(p.H * kN * 2)};
    const cuuint32_t estr[2] = {1, 1};
    auto describe = [&](CUtensorMap *map, const void *ptr, cuuint32_t rows) {
        const cuuint32_t box[2] = {(cuuint32_t)kN, rows};
        return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                      CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    const void *in[kTensors] = {p.a, p.r, p.b, p.k, p.v, p.dy, p.w};
    void *out[5] = {p.da, p.dr, p.db, p.dk, p.dw};
    for (int i = 0; i < kTensors; ++i) {
        if (!describe(&maps.in[i], in[i], (cuuint32_t)kL)) return (int)cudaErrorInvalidValue;
        args.in[i] = static_cast<const __nv_bfloat16 *>(in[i]);
    }
    for (int i = 0; i < 5; ++i) {
        if (!describe(&maps.out[i], out[i], (cuuint32_t)kL) || !describe(&maps.block[i], out[i], 16u)) return (int)cudaErrorInvalidValue;
        args.out[i] = static_cast<__nv_bfloat16 *>(out[i]);
    }
    args.records = records;
    args.states = states;
    args.gradients = gradients;
    args.T = (int)p.T;
    args.H = (int)p.H;
    args.nchunks = (int)((p.T + kL - 1) / kL);
    args.units = (int)(p.B * p.H * args.nchunks);   // (33 KB are kept for each: far fewer than 2^31)
    if (int e = device_status_ptr(p.device, &args.status)) return e;
    cudaError_t e = cudaFuncSetAttribute(wkv7_chunk_gradients_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
    if (e != cudaSuccess) return (int)e;
    return (int)launch_serialized(wkv7_chunk_gradients_kernel, (unsigned)(args.units < p.num_sms ? args.units : p.num_sms), (unsigned)kThreads, kSmem, stream,
                                  maps, args);
}

}  // namespace rwkv7
