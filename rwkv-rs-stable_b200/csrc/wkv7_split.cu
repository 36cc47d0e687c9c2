// Two-kernel WKV7 prefill for sm_100a (N == 64, bf16 or fp32 tensors, 64-token chunks, fp16 tensor-core
// operands): everything that does not depend on the running state is computed for all chunks in
// parallel by `wkv7_chunk_operator_kernel`, which folds a chunk into one linear operator, and
// `wkv7_state_scan_kernel` then walks each (b,h) chain chunk by chunk.
//
// Reference semantics: crates/rwkv-nn/src/kernels/train/time_mixer/wkv7/mod.rs:179-242 (token
// recurrence; the reference kernel, kernel.rs:82-195, scans token by token).
//
// Per chain and chunk, with the in-chunk inclusive prefix c_t of the log-decay l_t = -exp(w_t) and its value c_L at
// the chunk's end:
//     A_ab[t][s] = sum_n a_t[n] b_s[n] e^{c_{t-1}[n] - c_s[n]}  (s < t), A_ak likewise with k_s,
//     A_rb[t][s] = sum_n r_t[n] b_s[n] e^{c_t[n] - c_s[n]}      (s <= t), A_rk likewise with k_s
//     [A~ | A~k] = (I - A_ab)^-1 [a_t e^{c_{t-1}} | A_ak]       (u_t = S_{t-1} a_t = A~ S^T + A~k V)
//     Be_s = b_s e^{c_L - c_s}, Ke_s = k_s e^{c_L - c_s}
//     P  = A~^T Be     Kt = Ke + A~k^T Be     W = r_t e^{c_t} + A_rb A~     Ark = A_rk + A_rb A~k
// so that, for the state S[i][j] entering the chunk and V[s][i]:
//     S'[i][j'] = e^{c_L} S[i][j'] + sum_j S[i][j] P[j][j'] + sum_s V[s][i] Kt[s][j']
//     y[t][i]   = sum_j W[t][j] S[i][j] + sum_s Ark[t][s] V[s][i].
//
// Every tensor-core operand is fp16 (the same 11-bit significand as tf32).  The products of a chunk that depend on one another
// run on warp-level matrix instructions (see sm100_mma.cuh), the 128 x 128 one in front of them and all of the scan's on
// tcgen05.  fp16 has a narrow exponent range, and the factors of the four A matrices, e^{c_t} and e^{-c_s}, do not.  A chunk whose decay exceeds what the references below resolve is marked
// and its chain flagged; non-finite values (keys or values beyond fp16) are detected in the scan.
// Small values do not lose bits below fp16's normal numbers: r and k rows go in times a power of two where a 16-token block of
// them stays below 2 (the factor comes out again in the scan), and the scan scales V and the state likewise per chunk.
// Without, values of 1e-5 came out with an error of 1.1e-2 (tf32 operands: 1.7e-3, the rounding of y to bf16).
//
// References.  The factor e^{c_t - c_s} of an A matrix is split between its two operands at a reference point, per
// channel, chosen as e^{c_L} times a power of two.  Then
//   - b and k operands differ from Be and Ke by powers of two only, so one tile serves the A matrices and P, Kt;
//   - the a and r operands carry the factor 1/fx, fx[j] = e^{c_L} 2^..., which is the same for everything in column j of
//     A~ and R: the operator's rows P[j][.] and W[.][j] are stored divided by fx[j], and the scan multiplies the state
//     by fx[j] in fp32 before it rounds it to fp16.
// Where the decay of both halves of the chunk is mild (kMildDecay) one point near the middle serves all blocks and every
// power of two is the same per channel (it is applied in the scan too).  Otherwise each 16-token block has points of its
// own at its two ends, so that no factor exceeds 2, and the power of two of a pair of blocks is multiplied into one of the
// fp16 operands on its way into the matrix instruction, which is exact.  That resolves decays of e^-12 per block
// (kBlockDecay); the model's range (w < -0.5, weight_prepare.rs:272-274) ends at e^-9.7.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <type_traits>

#include "kernels.h"
#include "launch.h"
#include "sm100_mma.cuh"
#include "sm100_umma.cuh"
#include "trace.h"
#include "wkv7_overlap.h"
#include "wkv7_tiles.cuh"

namespace rwkv7 {

int launch_wkv7_sequential_flagged(const Wkv7Args &p, const int *flags, cudaStream_t stream);

namespace {

using namespace sm100;

constexpr float kMildDecay = 9.118820e-4f;    // e^-7: both halves of the chunk at or above it take one reference point
                                              // (factors up to 2200: room for entries of 29 and, below, down to 6e-2)
constexpr float kNarrowDecay = 1.522998e-8f;  // e^-18: least decay over a chunk when the wide range is switched off
constexpr int kWideShift = 6;                 // block-wise references: operands are stored times 2^6, because there the
constexpr float kWideScale = 64.f;            // factors reach down to e^-12 and a typical entry has to stay a normal number
__host__ __device__ constexpr int tri(int t) { return t * (t + 1) / 2; }

// ------------------------------------------------------------------------------------------
// Kernel 1: the operator of every chunk.  One CTA of four warps per chunk at a time, four CTAs per SM.
//
// Bound by the latency of a chunk's phases, which the four CTAs of an SM cover for one another in part: no unit is saturated (shared-memory
// port 63 %, issue slots 50 %, DRAM 65 %).  What a phase reads from shared memory is its length; hence few warps per chunk, each with
// the largest tile its registers hold (eight warps per chunk read a quarter more and were slower: 153 against 121 us).  Measured, 6144 chunks (8 x
// 4096 tokens x 12 heads): 107.4 us, 4.2 TB/s; the form on six tcgen05 products per chunk that this replaced took 170.  Per chunk:
//   1. decays: warp = 16-token block, lane = channel pair; prefix and suffix products within the block
//   2. scaled fp16 operands, in place over the bf16 tiles that TMA delivered
//   3. the A matrices: one 128 x 128 tcgen05 product [a; r] [b; k]^T, read back a row per thread, lower triangle only; with
//      block-wise references on warp-level instructions, warp = one of A_ab, A_ak, A_rb, A_rk
//   4. two warps: inverses of the four diagonal blocks I - A_bb in fp32 (forward substitution, a column per lane)
//   5. warp = 16 columns j and 16 columns s of [A~ | A~k]: block forward substitution on the transposed system, where
//      these columns are independent of all others, then every operator row from the same registers, and out.
// The next chunk's tiles are requested behind phase 5, w first.  (Bringing them into L2 during phase 2, through the same TMA unit, made
// the loads of the SM's other chunks wait: 118.5 us, 112.5 without.)
// ------------------------------------------------------------------------------------------
constexpr int kOpThreads = 128;
enum { XA = 0, XR = 1, XB = 2, XK = 3, XW = 4 };
constexpr uint32_t kTiles = 0;                        // a, r, b, k, w; w's place is part of the next region
// Compact lower triangles.  A_ab: six blocks below the diagonal, then the diagonal in fp32 (4 x [16][16]), each block
// replaced by its fp16 inverse; A_ak, A_rb, A_rk: ten blocks each.
constexpr uint32_t kAab = kTiles + 4 * kPanel;
constexpr uint32_t kDiag = kAab + 6 * kBlk;
constexpr uint32_t kAak = kDiag + 4 * 1024;
constexpr uint32_t kArb = kAak + 10 * kBlk;
constexpr uint32_t kArk = kArb + 10 * kBlk;
constexpr uint32_t kE = kArk;                         // block decays [4][64] (dead before A_rk is written; beyond w's tile)
constexpr uint32_t kPow = kArk + 10 * kBlk;           // powers of two (block-wise references): 11 x [64] fp16,
constexpr uint32_t kPowExp = kPow + 11 * 128;         // and exponents of further ones: 8 x [64] bytes
constexpr uint32_t kBar1 = kPowExp + 8 * 64;
constexpr uint32_t kSmem1 = kBar1 + 64;
static_assert(kE >= kTiles + 5 * kPanel, "the decays must not lie under w's tile");
static_assert(4 * (kSmem1 + 1024) <= 233472, "four CTAs per SM");
__host__ __device__ constexpr int below(int t) { return t * (t - 1) / 2; }   // first block of row t of A_ab
// kPow rows: the a/r side and the b/k side of a diagonal block, block pairs (2,0) (3,0) (3,1); kPowExp rows: per block what takes
// an a/r operand to the scale of its column of A~ (PX) and a b/k operand to Be, Ke (PE).
// (The first go with every matrix load of phase 3, 88 pairs a warp: as bytes, widened there, they were a fifth of a chunk's
// instructions.  The last are multiplied into b and k once, by the warps that the inverses leave idle.  Measured, 3 x 2047 tokens x 32
// heads at a model's decays: 73.9 -> 71.8 us.  There is no room for all of them as fp16.)
enum { PA = 0, PB = 4, PF = 8, PX = 0, PE = 4 };

struct OperatorMaps {
    CUtensorMap m[5];   // a, r, b, k, w as [B*T, H*N] bf16, box 64 x 64, 128-byte swizzle (bf16 tensors only)
};
struct OperatorPtrs {
    const void *p[5];   // the same tensors
};

__device__ __forceinline__ int lds_s8(uint32_t addr) {
    int v;
    asm volatile("ld.shared.s8 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t power_pair(uint32_t addr) {   // 2^e of two neighbouring exponents
    return pack_half2(exp2_of(lds_s8(addr)), exp2_of(lds_s8(addr + 1)));
}
__device__ __forceinline__ uint32_t power_twice(uint32_t addr) {
    const float f = exp2_of(lds_s8(addr));
    return pack_half2(f, f);
}

template <typename TIn>
__global__ void __launch_bounds__(kOpThreads, 4)
wkv7_chunk_operator_kernel(const __grid_constant__ OperatorMaps maps, OperatorPtrs ptrs, unsigned char *__restrict__ records,
                           int Tlen, int H, int chunk0, int seg_chunks, int nchains, int wide_range, int *status) {
    extern __shared__ __align__(1024) unsigned char smem[];
    constexpr bool kTma = sizeof(TIn) == 2;
    // How rows of the diagonal blocks are moved so that the half-warps and column halves that share an access lie in different banks.  (bf16
    // tensors: 111.2 -> 107.4 us.  The fp32 kernel has no registers for the addresses: 14.2 -> 15.0 us for 2 x 1000 tokens x 12 heads.)
    constexpr int kSpread = kTma ? 1 : 0;
    if (smem_u32(smem) & 1023u) {
        if (threadIdx.x == 0) atomicExch(status, (int)kDevInternal);
        return;
    }
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // (uniform: no divergence handling around what depends on it)
    const int g = lane >> 2, q = lane & 3;
    const uint32_t sb = smem_u32(smem);
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + kBar1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + kBar1 + 32);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + kBar1 + 40);
    if (warp == 0) tmem_alloc(tmem_slot, 128);
    if (tid == 0) {
        mbar_init(bar, 1);       // w
        mbar_init(bar + 1, 1);   // a, r, b, k
        mbar_init(bar + 2, 1);   // the tcgen05 product
        mbar_fence_init();
        *abort_flag = 0;
    }
    const long long units = (long long)nchains * seg_chunks;
    auto tile = [&](int x, long long unit, uint64_t *b) {
        const int chain = (int)(unit / seg_chunks), chunk = chunk0 + (int)(unit % seg_chunks);
        tma_load_2d(smem + kTiles + x * kPanel, &maps.m[x], (chain % H) * kN, (chain / H) * Tlen + chunk * kL, b);
    };
    auto request = [&](long long unit) {
        mbar_expect_tx(bar, kPanel);
        tile(XW, unit, bar);
        mbar_expect_tx(bar + 1, 4 * kPanel);
#pragma unroll
        for (int x = 0; x < 4; ++x) tile(x, unit, bar + 1);
    };
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // (set up while the kernel in front of it drains: 1 x 333 tokens x 32 heads 20.5 -> 16.8 us a call, back to back)
    wait_for_previous();
    if (kTma && tid == 0 && blockIdx.x < units) request(blockIdx.x);
    uint32_t mma_phase = 0;
    uint32_t phase = 0;
    int seq = 0;                               // chunks this CTA has begun
    const int tb = warp;                       // token block of phases 1 and 2
    const int ch = 2 * lane;                   // channel pair
    uint32_t po[8];                            // this thread's place in row u (mod 8) of its block of a tile
#pragma unroll
    for (int u = 0; u < 8; ++u) po[u] = sb + kTiles + off16(16 * tb + u, ch);
    auto at = [&](int x, int u) -> uint32_t { return po[u & 7] + (uint32_t)x * kPanel + (uint32_t)(u >> 3) * 1024u; };

    for (long long unit = blockIdx.x; unit < units; unit += gridDim.x, ++seq, phase ^= 1u) {
        const bool more = unit + gridDim.x < units;
        const int chain = (int)(unit / seg_chunks), chunk = chunk0 + (int)(unit % seg_chunks);
        const int valid = min(kL, Tlen - chunk * kL);
        const int nv = min(16, max(0, valid - 16 * tb));   // tokens of this block that exist
        const size_t gbase = (((size_t)(chain / H) * Tlen + chunk * kL + 16 * tb) * H + chain % H) * kN + ch;
        const size_t gstep = (size_t)H * kN;
        // (token u of this warp's block, channel pair) of a tensor; tokens past the end are no-ops: w = -inf, the rest zero
        using Raw = std::conditional_t<kTma, uint32_t, float2>;
        auto load16 = [&](int x, Raw (&v)[16]) {   // (all loads first: what follows stores to the same memory)
#pragma unroll
            for (int u = 0; u < 16; ++u) {
                if constexpr (kTma) v[u] = lds32(at(x, u));
                else {
                    const float none = x == XW ? -INFINITY : 0.f;
                    v[u] = make_float2(none, none);
                    if (u < nv && RWKV7_IN_RANGE(chain < nchains && chunk * kL + 16 * tb + u < Tlen, status))
                        v[u] = *reinterpret_cast<const float2 *>(static_cast<const float *>(ptrs.p[x]) + gbase + u * gstep);
                }
            }
        };
        auto value = [&](Raw v) -> float2 {
            if constexpr (kTma) return unpack_bf2(v);
            else return v;
        };
        if constexpr (kTma) {
            if (!mbar_wait(bar, phase)) *abort_flag = 1;
            __syncwarp();
            if (valid < kL)   // (each thread rewrites only what it reads itself)
                for (int u = nv; u < 16; ++u) sts32(sb + kTiles + XW * kPanel + off16(16 * tb + u, ch), 0xff80ff80u);
        }
        // ---------------- 1. decays
        float2 d[16];
        float2 e = make_float2(1.f, 1.f);
        {
            Raw w[16];
            load16(XW, w);
#pragma unroll
            for (int u = 0; u < 16; ++u) {
                d[u] = decay2(value(w[u]));
                e = mul2(e, d[u]);
            }
        }
        sts_f2(sb + kE + (tb * 64 + ch) * 4, e.x, e.y);
        __syncthreads();
        if (*abort_flag) break;
        // Every warp sees the whole chunk's decays (its 32 lanes hold all channels): no further agreement is needed.
        float E[2][4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const float2 v = lds_f2(sb + kE + (b * 64 + ch) * 4);
            E[0][b] = v.x;
            E[1][b] = v.y;
        }
        bool over = false, strong = false;
#pragma unroll
        for (int x = 0; x < 2; ++x) {
#pragma unroll
            for (int b = 0; b < 4; ++b) over |= !(E[x][b] >= kBlockDecay);
            const float h0 = E[x][0] * E[x][1], h1 = E[x][2] * E[x][3];
            strong |= !(h0 >= kMildDecay && h1 >= kMildDecay);
            if (!wide_range) over |= !(h0 * h1 >= kNarrowDecay);
        }
        over = __any_sync(0xffffffffu, over);
        const bool wide = __any_sync(0xffffffffu, strong);
        unsigned char *record = records + (size_t)unit * kRecord;
        if (tid == 0 && RWKV7_IN_RANGE(unit >= 0 && unit < units, status)) *reinterpret_cast<int *>(record + kMarkAt) = over;
        if constexpr (kTma) {
            if (!mbar_wait(bar + 1, phase)) *abort_flag = 1;
            __syncwarp();
            if (valid < kL)
                for (int u = nv; u < 16; ++u)
#pragma unroll
                    for (int x = 0; x < 4; ++x) sts32(sb + kTiles + x * kPanel + off16(16 * tb + u, ch), 0u);
        }
        auto note = [&](int er, int ek) {
            if (lane == 0 && RWKV7_IN_RANGE(unit >= 0 && unit < units, status))
                *reinterpret_cast<char2 *>(record + kDecayAt + kRowExpAt + 2 * tb) = make_char2((signed char)er, (signed char)ek);
        };
        if (over) {   // the chain is recomputed elsewhere: nothing more to do for this chunk
            note(0, 0);   // (read by the kernel of the chunk gradients, whose range may differ by a rounding)
            if (kTma) fence_proxy_async();
            __syncthreads();   // (everyone has read the decays)
            if (kTma && tid == 0 && more) request(unit + gridDim.x);
            continue;
        }
        // ---------------- 2. scaled operands
        {
            float mA[2], mB[2], dec[2];
            int ef[2], eg[2];
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const float p1 = E[x][0], p2 = p1 * E[x][1], p3 = p2 * E[x][2], p4 = p3 * E[x][3];
                const float pre = tb == 0 ? 1.f : tb == 1 ? p1 : tb == 2 ? p2 : p3;    // decay up to this block's start,
                const float post = tb == 0 ? p1 : tb == 1 ? p2 : tb == 2 ? p3 : p4;    // to its end,
                const float tail = tb == 3 ? 1.f : tb == 2 ? E[x][3] : tb == 1 ? E[x][2] * E[x][3] : E[x][1] * E[x][2] * E[x][3];   // and from there to the chunk's
                const int x4 = exponent_of(p4);
                dec[x] = p4;
                if (!wide) {
                    ef[x] = eg[x] = exponent_of(p2) - x4;
                    const float up = exp2_of(ef[x]);
                    mA[x] = pre * rcp(p4 * up);
                    mB[x] = tail * up;
                } else {
                    const int xs = exponent_of(pre), xe = exponent_of(post);
                    mA[x] = pre * exp2_of(kWideShift) * rcp(p4 * exp2_of(xs - x4));
                    mB[x] = tail * exp2_of(xe - x4 + kWideShift);
                    ef[x] = 127 - x4;
                    eg[x] = 0;
                    __half *pw = reinterpret_cast<__half *>(smem + kPow) + ch + x;
                    signed char *pe = reinterpret_cast<signed char *>(smem + kPowExp) + ch + x;
                    auto power = [&](int row, int e) { pw[row * 64] = __float2half_rn(exp2_of(max(e, -100))); };   // (fp16 ends at 2^-24)
                    auto exponent = [&](int row, int e) { pe[row * 64] = (signed char)max(e, -100); };
                    const int ha = (xs - xe) >> 1;
                    power(PA + tb, ha - kWideShift);
                    power(PB + tb, xs - xe - ha - kWideShift);
                    if (tb < 3)   // (2,0), (3,0), (3,1): start of the row block over the end of the column block
                        power(PF + tb, exponent_of(tb == 0 ? p2 : p3) - exponent_of(tb == 2 ? p2 : p1));
                    exponent(PX + tb, xs - 127 - kWideShift);
                    exponent(PE + tb, x4 - xe - kWideShift);
                }
            }
            if (tb == 3 && RWKV7_IN_RANGE(unit >= 0 && unit < units, status)) {
                *reinterpret_cast<float2 *>(record + kDecayAt + ch * 4) = make_float2(dec[0], dec[1]);
                *reinterpret_cast<char2 *>(record + kExpAt + ch) = make_char2((signed char)ef[0], (signed char)ef[1]);
                *reinterpret_cast<char2 *>(record + kExpAt + 64 + ch) = make_char2((signed char)eg[0], (signed char)eg[1]);
            }
            Raw v0[16], v1[16];
            // Rows of small values (largest magnitude below 2) times the power of two that brings it to [2, 4); its exponent.
            auto raise_small = [&](Raw (&v)[16]) -> int {
                uint32_t bits = 0u;   // (a magnitude of 2 and above has the top bit of its exponent)
#pragma unroll
                for (int u = 0; u < 16; ++u) {
                    if constexpr (kTma) bits |= v[u];
                    else bits |= __float_as_uint(v[u].x) | __float_as_uint(v[u].y);
                }
                if (__any_sync(0xffffffffu, (bits & (kTma ? 0x40004000u : 0x40000000u)) != 0u)) return 0;
                uint32_t most;
                if constexpr (kTma) {
                    __nv_bfloat162 m = __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll
                    for (int u = 0; u < 16; ++u) m = __hmax2(m, __habs2(*reinterpret_cast<const __nv_bfloat162 *>(&v[u])));
                    most = __float_as_uint(fmaxf(__low2float(m), __high2float(m)));
                } else {
                    float m = 0.f;
#pragma unroll
                    for (int u = 0; u < 16; ++u) m = fmaxf(m, fmaxf(fabsf(v[u].x), fabsf(v[u].y)));
                    most = __float_as_uint(m);
                }
                const int x = (int)(__reduce_max_sync(0xffffffffu, most) >> 23);
                const int ex = max(min(x - 128, 0), -60);   // (rows of zeros: whatever)
#pragma unroll
                for (int u = 0; u < 16; ++u) {
                    if constexpr (kTma) v[u] = raise_bf2(v[u], -ex);
                    else v[u] = mul2(v[u], make_float2(exp2_of(-ex), exp2_of(-ex)));
                }
                return ex;
            };
            load16(XA, v0);
            load16(XR, v1);
            const int er = raise_small(v1);
            float2 f = make_float2(mA[0], mA[1]);
#pragma unroll
            for (int u = 0; u < 16; ++u) {
                sts32(at(XA, u), pack2(mul2(value(v0[u]), f)));
                f = mul2(f, d[u]);
                sts32(at(XR, u), pack2(mul2(value(v1[u]), f)));
            }
            load16(XB, v0);
            load16(XK, v1);
            note(er, raise_small(v1));
            f = make_float2(mB[0], mB[1]);
#pragma unroll
            for (int u = 15; u >= 0; --u) {
                sts32(at(XB, u), pack2(mul2(value(v0[u]), f)));
                sts32(at(XK, u), pack2(mul2(value(v1[u]), f)));
                f = mul2(f, d[u]);
            }
        }
        fence_proxy_async();
        __syncthreads();
        // ---------------- 3. the A matrices, lower triangles
        if (!wide) {
            if (warp == 0 && elect_one()) {
                tc_fence_after();
#pragma unroll
                for (int ks = 0; ks < 4; ++ks)
                    umma_f16(tmem, make_smem_desc(sb + kTiles + XA * kPanel + ks * 32u, 16u, 1024u), make_smem_desc(sb + kTiles + XB * kPanel + ks * 32u, 16u, 1024u),
                             make_idesc(kFmtF16, 128, 128, false, false), ks > 0);
                umma_commit(bar + 2);
            }
            __syncwarp();
            if (!mbar_wait_tight(bar + 2, mma_phase, 4000000u)) *abort_flag = 1;
            __syncwarp();
            mma_phase ^= 1u;
            tc_fence_after();
            // This thread's row t of [A_ab | A_ak] (warps 0, 1) or [A_rb | A_rk]; block row bt, the other half-warp's is bt0 or bt0 + 1.
            const int bt0 = 2 * (warp & 1), bt = bt0 + (lane >> 4), r = lane & 15;
            const bool top = warp < 2;                 // strictly lower
            const uint32_t col0 = tmem + ((uint32_t)(warp * 32) << 16);
            uint32_t keep[8];                          // column pairs of a diagonal block that this row keeps
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int n = r + (top ? 0 : 1) - 2 * e;   // of these two columns, how many
                keep[e] = n <= 0 ? 0u : n == 1 ? 0xffffu : ~0u;
            }
            const uint32_t sub = r * 16, row = sub + tri(bt) * kBlk;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int m = i >> 1, sp = i & 1;
                if (sp == 1 && bt0 == 0) continue;     // (uniform) above the diagonal for the whole warp
                const bool ab = m == 0 && top;
                const uint32_t out = m == 0 ? (top ? sb + kAab + sub + below(bt) * kBlk : sb + kArb + row) : (top ? sb + kAak : sb + kArk) + row;
                uint32_t d[32];
                tmem_ld32(col0 + i * 32, d);
                tmem_ld_wait();
#pragma unroll
                for (int s1 = 0; s1 < 2; ++s1) {
                    const int sc = 2 * sp + s1;
                    if (sc == bt && ab) {          // fp32 for the inverse (which reads below the diagonal only)
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const uint32_t x[4] = {d[16 * s1 + 4 * e], d[16 * s1 + 4 * e + 1], d[16 * s1 + 4 * e + 2], d[16 * s1 + 4 * e + 3]};
                            sts128(sb + kDiag + bt * 1024 + (r ^ (bt & kSpread)) * 64 + ((e ^ ((r >> 1) & 3)) << 4), x);
                        }
                    } else if (sc <= bt) {
                        const uint32_t all = sc == bt ? 0u : ~0u;
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            uint32_t x[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e)
                                x[e] = pack_half2(__uint_as_float(d[16 * s1 + 8 * h + 2 * e]), __uint_as_float(d[16 * s1 + 8 * h + 2 * e + 1])) & (keep[4 * h + e] | all);
                            sts128(out + sc * kBlk + h * 256, x);
                        }
                    }
                }
            }
            tc_fence_before();
        } else {
            const uint32_t rows = sb + kTiles + (warp < 2 ? XA : XR) * kPanel, cols = sb + kTiles + (warp & 1 ? XK : XB) * kPanel;
            const uint32_t mat = sb + (warp == 0 ? kAab : warp == 1 ? kAak : warp == 2 ? kArb : kArk) + lane * 4;
            const int keep = warp >= 2 ? 0 : -1;    // r rows keep the diagonal
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                float c[4][2][4] = {};
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    uint32_t A[4];
                    ldsm4(A, rows + tile_plain(lane, 16 * t, kk));
#pragma unroll
                    for (int s = 0; s <= t; ++s) {
                        uint32_t As[4] = {A[0], A[1], A[2], A[3]}, Bs[4];
                        ldsm4(Bs, cols + tile_cols(lane, 16 * s, kk));
                        const uint32_t f = sb + kPow + kk * 32 + 4 * q;
                        if (t != s + 1) {
                            const int pa = (s == t ? PA + t : PF + (t == 2 ? 0 : 1 + s)) * 128;
                            const uint32_t lo = lds32(f + pa), hi = lds32(f + pa + 16);
                            As[0] = mul_half2(As[0], lo);
                            As[1] = mul_half2(As[1], lo);
                            As[2] = mul_half2(As[2], hi);
                            As[3] = mul_half2(As[3], hi);
                        }
                        if (t == s) {
                            const uint32_t lo = lds32(f + (PB + t) * 128), hi = lds32(f + (PB + t) * 128 + 16);
                            Bs[0] = mul_half2(Bs[0], lo);
                            Bs[1] = mul_half2(Bs[1], hi);
                            Bs[2] = mul_half2(Bs[2], lo);
                            Bs[3] = mul_half2(Bs[3], hi);
                        }
                        mma16816(c[s][0], As, Bs[0], Bs[1]);
                        mma16816(c[s][1], As, Bs[2], Bs[3]);
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (8 * h + 2 * q + (e & 1) > g + (e >> 1) * 8 + keep) c[t][h][e] = 0.f;
                // (the diagonal blocks' powers have taken the operands' common scale out already)
#pragma unroll
                for (int s = 0; s < t; ++s)
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int e = 0; e < 4; ++e) c[s][h][e] *= 1.f / (kWideScale * kWideScale);
#pragma unroll
                for (int s = 0; s <= t; ++s) {
                    if (s == t && warp == 0) {   // fp32 for the inverse
#pragma unroll
                        for (int h = 0; h < 2; ++h)
#pragma unroll
                            for (int r = 0; r < 2; ++r) {
                                const int row = g + 8 * r, piece = 2 * h + (q >> 1);
                                sts_f2(sb + kDiag + t * 1024 + (row ^ (t & kSpread)) * 64 + ((piece ^ ((row >> 1) & 3)) << 4) + (q & 1) * 8, c[s][h][2 * r], c[s][h][2 * r + 1]);
                            }
                    } else {
                        const uint32_t o = mat + ((warp == 0 ? below(t) : tri(t)) + s) * kBlk;
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            sts32(o + h * 256, pack_half2(c[s][h][0], c[s][h][1]));
                            sts32(o + h * 256 + 128, pack_half2(c[s][h][2], c[s][h][3]));
                        }
                    }
                }
            }
        }
        __syncthreads();
        // ---------------- 4. T_bb = (I - A_bb)^-1: two warps, a half-warp per diagonal block, a column per lane.  The other two
        // take b and k to Be and Ke (block-wise references).
        {
            const int pair = (warp + seq) & 3;   // (which two warps changes from chunk to chunk: each sits on its own scheduler)
            if (pair < 2) {
                const int cc = lane & 15, b = 2 * pair + (lane >> 4);
                // (rows of blocks 1 and 3 are exchanged in pairs: the two half-warps read different banks)
                const uint32_t src = sb + kDiag + b * 1024, even = src + (lane >> 4) * 64 * kSpread, odd = src - (lane >> 4) * 64 * kSpread;
                float x[16];
#pragma unroll
                for (int t = 0; t < 16; ++t) {
                    float acc0 = 0.f, acc1 = 0.f;
#pragma unroll
                    for (int s4 = 0; s4 < (t + 3) / 4; ++s4) {
                        const float4 a4 = lds_f4(((t & 1) ? odd : even) + t * 64 + ((s4 ^ ((t >> 1) & 3)) << 4));
                        if (4 * s4 + 0 < t) acc0 = fmaf(a4.x, x[4 * s4 + 0], acc0);
                        if (4 * s4 + 1 < t) acc1 = fmaf(a4.y, x[4 * s4 + 1], acc1);
                        if (4 * s4 + 2 < t) acc0 = fmaf(a4.z, x[4 * s4 + 2], acc0);
                        if (4 * s4 + 3 < t) acc1 = fmaf(a4.w, x[4 * s4 + 3], acc1);
                    }
                    x[t] = (t == cc) ? 1.f : acc0 + acc1;   // (zero above: every term up to there is)
                }
                __syncwarp();   // (every lane has read the block that the inverse replaces)
                // (rows in an order of their own per half and parity of the block, four and two apart: a store of the warp's 32 halves is conflict-free)
                const uint32_t dst = (kDiag + b * 1024 + (cc >> 3) * 256 + (cc & 7) * 2) ^ ((uint32_t)(cc >> 3) << 6) * kSpread ^ ((uint32_t)(lane >> 4) << 5) * kSpread;
                static_assert(kDiag % 256 == 0, "exclusive or of the rows");
#pragma unroll
                for (int t = 0; t < 16; ++t) *reinterpret_cast<__half *>(smem + (dst ^ (uint32_t)(t << 4))) = __float2half_rn(x[t]);
            } else if (wide) {
                const uint32_t rows = sb + kTiles + (pair == 2 ? XB : XK) * kPanel + (lane >> 3) * 128, piece = lane & 7;   // eight channels of every fourth token
#pragma unroll 1
                for (int b = 0; b < 4; ++b) {
                    uint32_t f[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) f[e] = power_pair(sb + kPowExp + (PE + b) * 64 + piece * 8 + 2 * e);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint32_t o = rows + (16 * b + 4 * i) * 128 + ((piece ^ ((4 * i + (lane >> 3)) & 7)) << 4);
                        uint32_t x[4];
                        lds128(x, o);
#pragma unroll
                        for (int e = 0; e < 4; ++e) x[e] = mul_half2(x[e], f[e]);
                        sts128(o, x);
                    }
                }
            }
        }
        // The tiles and what lies in w's place are only read from here on: handed back to TMA now, because behind the stores of phase 5 this
        // fence would wait for them too.
        if (kTma) fence_proxy_async();
        __syncthreads();
        // ---------------- 5. [A~ | A~k]^T for columns j = 16 ct.. and s = 16 ct.., then the operator's rows they are
        auto finish = [&](auto block_wise) {
            constexpr bool kWide = decltype(block_wise)::value;
            const int ct = (warp + seq) & 3;   // (block ct of s has 4 - ct row blocks to do: the share goes round)
            uint32_t U[2][4][4];   // A order, rows = own columns (0: j, 1: s), columns = tokens of block b
            auto unpack8 = [&](const uint32_t (&X)[4], float (&c)[2][4]) {
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const float2 v = unpack_half2(X[2 * h + r]);
                        c[h][2 * r] = v.x;
                        c[h][2 * r + 1] = v.y;
                    }
            };
            // a/r or b/k operand block, rows = channels 16 c.., times its row's power of two (block-wise references)
            auto row_power = [&](int table, int c, uint32_t (&X)[4]) {
                const uint32_t f0 = power_twice(sb + kPowExp + table * 64 + 16 * c + g), f1 = power_twice(sb + kPowExp + table * 64 + 16 * c + g + 8);
                X[0] = mul_half2(X[0], f0);
                X[1] = mul_half2(X[1], f1);
                X[2] = mul_half2(X[2], f0);
                X[3] = mul_half2(X[3], f1);
            };
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                uint32_t X[2][4];
                float c[2][2][4];
                ldsm4_t(X[0], sb + kTiles + XA * kPanel + tile_cols(lane, 16 * b, ct));
                if constexpr (kWide) row_power(PX + b, ct, X[0]);
                const bool live = b >= ct;   // A~k[t][s] is zero above the diagonal
                if (live) ldsm4_t(X[1], sb + kAak + (tri(b) + ct) * kBlk + blk_cols(lane));
                else X[1][0] = X[1][1] = X[1][2] = X[1][3] = 0;
                if (b > 0) {
                    unpack8(X[0], c[0]);
                    unpack8(X[1], c[1]);
#pragma unroll
                    for (int p = 0; p < b; ++p) {
                        uint32_t M[4];
                        ldsm4(M, sb + kAab + (below(b) + p) * kBlk + blk_cols(lane));
                        mma16816(c[0][0], U[0][p], M[0], M[1]);
                        mma16816(c[0][1], U[0][p], M[2], M[3]);
                        mma16816(c[1][0], U[1][p], M[0], M[1]);   // (zero for p < ct: cheaper than a branch)
                        mma16816(c[1][1], U[1][p], M[2], M[3]);
                    }
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        X[x][0] = pack_half2(c[x][0][0], c[x][0][1]);
                        X[x][1] = pack_half2(c[x][0][2], c[x][0][3]);
                        X[x][2] = pack_half2(c[x][1][0], c[x][1][1]);
                        X[x][3] = pack_half2(c[x][1][2], c[x][1][3]);
                    }
                }
                uint32_t Tb[4];
                ldsm4(Tb, sb + kDiag + b * 1024 + (blk_cols(lane) ^ ((uint32_t)((lane >> 3) & 1) << 6) * kSpread ^ ((uint32_t)(b & 1) << 5) * kSpread));
                float o[2][2][4];
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    mma16816_first(o[x][0], X[x], Tb[0], Tb[1]);
                    mma16816_first(o[x][1], X[x], Tb[2], Tb[3]);
                }
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    U[x][b][0] = pack_half2(o[x][0][0], o[x][0][1]);
                    U[x][b][1] = pack_half2(o[x][0][2], o[x][0][3]);
                    U[x][b][2] = pack_half2(o[x][1][0], o[x][1][1]);
                    U[x][b][3] = pack_half2(o[x][1][2], o[x][1][3]);
                }
            }
            // Sixteen rows n of the operator, columns k of this warp's two blocks (see kRecord).  A lane has four k of rows g and g + 8; two
            // neighbours exchange theirs, and each stores eight k of one row: whole 32-byte sectors.
            unsigned char *dst = record + ct * 256 + (q >> 1) * 128;
            const int row_state = (g >> 2) * 2048 + ((g >> 1) & 1) * 64 + (q & 1) * 32 + (g & 1) * 16, row_out = (q & 1) * 2048 + g * 16;
            auto put = [&](int n16, const float (&c)[2][2][4]) {
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const uint32_t lo[2] = {pack_half2(c[x][0][0], c[x][0][1]), pack_half2(c[x][1][0], c[x][1][1])};
                    const uint32_t hi[2] = {pack_half2(c[x][0][2], c[x][0][3]), pack_half2(c[x][1][2], c[x][1][3])};
                    const uint32_t t0 = __shfl_xor_sync(0xffffffffu, (q & 1) ? lo[0] : hi[0], 1), t1 = __shfl_xor_sync(0xffffffffu, (q & 1) ? lo[1] : hi[1], 1);
                    if (RWKV7_IN_RANGE(unit >= 0 && unit < units && n16 < 8, status))
                        *reinterpret_cast<uint4 *>(dst + n16 * 4096 + (n16 < 4 ? row_state : row_out) + x * 1024) =
                            (q & 1) ? make_uint4(t0, t1, hi[0], hi[1]) : make_uint4(lo[0], lo[1], t0, t1);
                }
            };
            // (This loop, like the one over the quarters of the product above, is kept as a loop: a chunk's straight-line code is
            // larger than the SM's instruction cache, and sixteen warps in different phases of it waited for instructions.)
            // rows j' of the next state: P^T = Be^T A~, Kt^T = Ke^T + Be^T A~k
#pragma unroll 1
            for (int n = 0; n < 4; ++n) {
                float c[2][2][4];
                uint32_t X[4];
                ldsm4_t(X, sb + kTiles + XK * kPanel + tile_cols(lane, 16 * ct, n));
                unpack8(X, c[1]);
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    uint32_t A[4];
                    ldsm4_t(A, sb + kTiles + XB * kPanel + tile_cols(lane, 16 * b, n));
                    if (b == 0) {
                        mma16816_first(c[0][0], A, U[0][b][0], U[0][b][2]);
                        mma16816_first(c[0][1], A, U[0][b][1], U[0][b][3]);
                    } else {
                        mma16816(c[0][0], A, U[0][b][0], U[0][b][2]);
                        mma16816(c[0][1], A, U[0][b][1], U[0][b][3]);
                    }
                    mma16816(c[1][0], A, U[1][b][0], U[1][b][2]);
                    mma16816(c[1][1], A, U[1][b][1], U[1][b][3]);
                }
                put(n, c);
            }
            // rows t of the output: W = r e^{c} + A_rb A~, Ark = A_rk + A_rb A~k
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                float c[2][2][4];
                uint32_t X[4];
                ldsm4(X, sb + kTiles + XR * kPanel + tile_plain(lane, 16 * n, ct));
                if constexpr (kWide) {
                    const uint32_t fa = sb + kPowExp + (PX + n) * 64 + 16 * ct + 2 * q;
                    const uint32_t f0 = power_pair(fa), f1 = power_pair(fa + 8);
                    X[0] = mul_half2(X[0], f0);
                    X[1] = mul_half2(X[1], f0);
                    X[2] = mul_half2(X[2], f1);
                    X[3] = mul_half2(X[3], f1);
                }
                unpack8(X, c[0]);
                if (n >= ct) ldsm4(X, sb + kArk + (tri(n) + ct) * kBlk + blk_plain(lane));
                else X[0] = X[1] = X[2] = X[3] = 0;
                unpack8(X, c[1]);
#pragma unroll
                for (int b = 0; b <= n; ++b) {
                    uint32_t A[4];
                    ldsm4(A, sb + kArb + (tri(n) + b) * kBlk + blk_plain(lane));
                    mma16816(c[0][0], A, U[0][b][0], U[0][b][2]);
                    mma16816(c[0][1], A, U[0][b][1], U[0][b][3]);
                    mma16816(c[1][0], A, U[1][b][0], U[1][b][2]);
                    mma16816(c[1][1], A, U[1][b][1], U[1][b][3]);
                }
                put(4 + n, c);
            }
        };
        if (wide) finish(std::true_type{});   // (two copies: merging them costs the common one a move per operand register)
        else finish(std::false_type{});
        __syncthreads();
        if (kTma && tid == 0 && more) request(unit + gridDim.x);
        // (the last chunk of this CTA: the scan may be set up)
        if (!more) let_next_in();
    }
    if (tid == 0 && *abort_flag) {
        if (kTma) {   // what is in flight lands before the CTA leaves
            mbar_wait(bar, phase, 100000u);
            mbar_wait(bar + 1, phase, 100000u);
        }
        atomicExch(status, (int)kDevTimeout);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 128);
}

// ------------------------------------------------------------------------------------------
// Kernel 2: the scan, one CTA per chain.  D[n][i] = sum_k O[n][k] [Z; V][k][i] per chunk, four tcgen05 products of M = 128,
// N = 64, K = 16 over V, issued a chunk ahead, and four over Z: TMEM lanes 0-63 are the rows j' of the next state (fp32 state Z[j'][i] = S[i][j'] in registers, two
// warps per column half), lanes 64-127 the output tokens.  Warps 0-7 own the lanes twice over (two column halves), warp 8
// streams records and V tiles into a ring, warp 9 issues, warps 10 to 13 turn V tiles into scaled fp16 rows of [Z; V] ahead of time.
//
// Bound by the serial step of a chain: TMEM read, multiply-add with the decays, fp16 rows of Z, hand-over to the issuing
// warp, the products over Z, their completion.  Hand-overs are hardware barriers (16 cycles; a satisfied mbarrier wait
// written as a C loop costs a warp 127, with its loop in one asm statement 53): one that the state warps arrive on when
// Z is written, one for the V products (tile converted, accumulator read back).  Only the completion of products and the
// arrival of a stage go through an mbarrier.  (A version on warp-level matrix instructions, the state in their
// accumulators, was bound by shared-memory bandwidth: each warp reads its operator columns and all of Z and V, 1.8 k
// cycles a chunk.)  Rows of the accumulator are in the order of the contraction index (k_at_position), so that a warp's lanes write
// neighbouring rows of the operand tile: with two or four of them in one bank a chunk of the chain took 70 (gradients 270) cycles more.
// Measured: 57.8 us for 64 chunks of 96 chains (60.2 in channel order); 512 chains 6.1 TB/s, the roof.
// ------------------------------------------------------------------------------------------
constexpr int kConverters = 4;                    // (one per token block of a chunk; with two the prefill's scan took 60.5 us, not 58.8)
constexpr int kScanThreads = (10 + kConverters) * 32;
template <typename TIO>
struct Scan {
    static constexpr bool kF32 = sizeof(TIO) == 4;
    static constexpr int kStages = kF32 ? 3 : 4;
    static constexpr uint32_t kVBytes = kL * kN * sizeof(TIO);
    static constexpr uint32_t kV = kOperatorBytes;                // stage: operator, V tile, vectors
    static constexpr uint32_t kVec = kV + kVBytes;
    static constexpr uint32_t kStage = kVec + 1024;
    static constexpr uint32_t kZV = kStages * kStage;             // two tiles each of Z and V, 64 rows k of 64 channels, 128-byte swizzle
    static constexpr uint32_t kYTile = kL * kN * sizeof(TIO);
    static constexpr uint32_t kY = kZV + 2 * 2 * kPanel;          // two output tiles (fp32: each two panels of 32 channels)
    static constexpr uint32_t kBars = kY + 2 * kYTile;
    static constexpr uint32_t kBytes = kBars + 384;
    static_assert(kBytes <= 232448, "the scan exceeds an SM");
};

struct ScanMaps {
    CUtensorMap v;   // [B*T, H*N], 128-byte swizzle: bf16, box 64 x 64; fp32, box 32 channels x 64 tokens (two per tile)
    CUtensorMap y;   // the output, the same
};

// Row of the Z tile (and position of the contraction index in the operator) of state column j, or of the V tile of token s.
__device__ __forceinline__ int k_position(int j) {
    return (j >> 4) * 16 + ((j & 7) >> 1) * 4 + ((j & 8) >> 2) + (j & 1);
}

// ... and the state column or token of a position.
__device__ __forceinline__ int k_at_position(int p) {
    return (p >> 4) * 16 + ((p >> 1) & 1) * 8 + ((p >> 2) & 3) * 2 + (p & 1);
}

// Descriptor of the operator as A operand without swizzle: 8 x 16-byte core matrices, 128 bytes apart along k, 2048
// along n.  Forwards the rows are n and a K-step is two core matrices along k; for gradients the operator is transposed: the
// rows are k (contiguous, "MN-major") and a K-step is two core matrices along n.
template <bool kTransposed>
__device__ __forceinline__ uint64_t desc_operator(uint32_t addr, int ks) {
    const uint32_t step = kTransposed ? 4096u : 256u, along_k = kTransposed ? 2048u : 128u, along_m = kTransposed ? 128u : 2048u;
    return (uint64_t)(((addr + (uint32_t)ks * step) >> 4) & 0x3fffu) | (uint64_t)(along_k >> 4) << 16 | (uint64_t)(along_m >> 4) << 32 | (uint64_t)1 << 46;
}

__device__ __forceinline__ float max3_abs(float a, float b, float c) {
    float y;
    asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
    return y;
}

// A warp's largest magnitude of a state, as float bits.
__device__ __forceinline__ void keep_top(uint32_t *tops, const float (&S)[4][4]) {
    float m = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) m = fmaxf(m, fabsf(S[i >> 2][i & 3]));
    const uint32_t most = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
    if ((threadIdx.x & 31) == 0) tops[threadIdx.x >> 5] = most;
}

// Tiles of 32 tokens of a chain's tensors (a, r, b, k, w, and v or dY) in shared memory, one fetched while the one before is
// used, with the decays of the current one.  For the 256 threads that recompute a chain.
template <typename TIO>
struct TokenTiles {
    static constexpr int kTokens = 32, kPiece = 16 / (int)sizeof(TIO), kPieces = kN / kPiece, kTile = kTokens * kN;
    const OperatorPtrs &in;
    const TIO *x;
    size_t base, step;   // of token 0, from token to token
    TIO *room;
    float *d;
    __device__ TokenTiles(const OperatorPtrs &in, const TIO *x, unsigned char *smem, int bi, int h, int H, int Tlen)
        : in(in), x(x), base(((size_t)bi * Tlen * H + h) * kN), step((size_t)H * kN), room(reinterpret_cast<TIO *>(smem)), d(reinterpret_cast<float *>(room + 12 * kTile)) {}
    static __device__ void together() { asm volatile("bar.sync 9, 256;" ::: "memory"); }
    __device__ const TIO *tile(int i, int tensor) const { return room + ((i & 1) * 6 + tensor) * kTile; }
    __device__ void fetch(int i, int t0, int t1) const {
#pragma unroll
        for (int tensor = 0; tensor < 6; ++tensor)
#pragma unroll
            for (int idx = threadIdx.x; idx < kTokens * kPieces; idx += 256) {
                const int tok = idx / kPieces, at = idx % kPieces * kPiece;
                if (t0 + tok < t1) {
                    const TIO *src = (tensor < 5 ? static_cast<const TIO *>(in.p[tensor]) : x) + base + (size_t)(t0 + tok) * step + at;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(tile(i, tensor) + tok * kN + at)), "l"(src) : "memory");
                }
            }
    }
    // tile i is there and its decays are known
    __device__ void arrived(int i) const {
        asm volatile("cp.async.wait_all;" ::: "memory");
        together();
        const TIO *w = tile(i, XW) + threadIdx.x * 8;
#pragma unroll
        for (int e = 0; e < 8; ++e) d[threadIdx.x * 8 + e] = expf(-expf(static_cast<float>(w[e])));
        together();
    }
    // four neighbouring channels of a token
    static __device__ float4 four(const TIO *at) {
        if constexpr (sizeof(TIO) == 4) return *reinterpret_cast<const float4 *>(at);
        else {
            const uint2 u = *reinterpret_cast<const uint2 *>(at);
            const float2 lo = unpack_bf2(u.x), hi = unpack_bf2(u.y);
            return make_float4(lo.x, lo.y, hi.x, hi.y);
        }
    }
};
// (the tiles, and behind them the state that the recomputation goes on from, lie where the stages were)
constexpr uint32_t kStateThen = 12 * 32 * kN * sizeof(float) + 32 * kN * sizeof(float);
static_assert(kStateThen + kN * kN * sizeof(float) <= Scan<float>::kZV && kStateThen + kN * kN * sizeof(float) <= Scan<__nv_bfloat16>::kZV, "shared memory");

// Token-by-token recomputation of one chain over tokens t0 .. t1 - 1, fp32 throughout: what a
// CTA does when a value overflowed fp16 on the way, or the chain is flagged and no later kernel is there to take it.  Four
// lanes per row; columns and sums in the order of the sequential scan (wkv7_seq.cu), whose bits it reproduces.
template <typename TIO>
__device__ __noinline__ void scan_rows_by_token(const OperatorPtrs &in, const TIO *v, TIO *y, const float *s_in, float *s_out, float *snapshots,
                                                uint32_t *tops, unsigned char *smem, int bi, int h, int H, int Tlen, int t0, int t1) {
    using Tiles = TokenTiles<TIO>;
    const Tiles tiles(in, v, smem, bi, h, H, Tlen);
    const int row = (int)threadIdx.x >> 2, c0 = ((int)threadIdx.x & 3) * 4;   // columns c0 + 16 kk + e
    tiles.fetch(0, t0, t1);
    float S[4][4];
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[kk][e] = s_in ? s_in[row * kN + c0 + 16 * kk + e] : 0.f;
    for (int i = 0, first = t0; first < t1; ++i, first += Tiles::kTokens) {
        tiles.arrived(i);
        tiles.fetch(i + 1, first + Tiles::kTokens, t1);
        if (snapshots != nullptr && first % kL == 0) {
            keep_top(tops + first / kL * 8, S);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                for (int e = 0; e < 4; ++e) snapshots[(size_t)(first / kL) * kN * kN + accumulator_place(row, c0 + 16 * kk + e)] = S[kk][e];
        }
        const int count = min(Tiles::kTokens, t1 - first);
        for (int u = 0; u < count; ++u) {
            auto f = [&](int x, int kk) { return Tiles::four(tiles.tile(i, x) + u * kN + c0 + 16 * kk); };
            float p[4] = {}, yy[4] = {};
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                const float4 a = f(XA, kk);
                p[0] = fmaf(S[kk][0], a.x, p[0]);
                p[1] = fmaf(S[kk][1], a.y, p[1]);
                p[2] = fmaf(S[kk][2], a.z, p[2]);
                p[3] = fmaf(S[kk][3], a.w, p[3]);
            }
            float sa = (p[0] + p[1]) + (p[2] + p[3]);
            sa += __shfl_xor_sync(0xffffffffu, sa, 1);
            sa += __shfl_xor_sync(0xffffffffu, sa, 2);
            const float vi = static_cast<float>(tiles.tile(i, 5)[u * kN + row]);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                const float4 d = *reinterpret_cast<const float4 *>(tiles.d + u * kN + c0 + 16 * kk), b = f(XB, kk), k = f(XK, kk), r = f(XR, kk);
                S[kk][0] = fmaf(S[kk][0], d.x, fmaf(sa, b.x, vi * k.x));
                S[kk][1] = fmaf(S[kk][1], d.y, fmaf(sa, b.y, vi * k.y));
                S[kk][2] = fmaf(S[kk][2], d.z, fmaf(sa, b.z, vi * k.z));
                S[kk][3] = fmaf(S[kk][3], d.w, fmaf(sa, b.w, vi * k.w));
                yy[0] = fmaf(S[kk][0], r.x, yy[0]);
                yy[1] = fmaf(S[kk][1], r.y, yy[1]);
                yy[2] = fmaf(S[kk][2], r.z, yy[2]);
                yy[3] = fmaf(S[kk][3], r.w, yy[3]);
            }
            float out = (yy[0] + yy[1]) + (yy[2] + yy[3]);
            out += __shfl_xor_sync(0xffffffffu, out, 1);
            out += __shfl_xor_sync(0xffffffffu, out, 2);
            if (c0 == 0) {
                TIO *o = y + tiles.base + (size_t)(first + u) * tiles.step + row;
                if constexpr (sizeof(TIO) == 4) *o = out;
                else *o = __float2bfloat16_rn(out);
            }
        }
    }
    if (s_out != nullptr) {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
            for (int e = 0; e < 4; ++e) s_out[row * kN + c0 + 16 * kk + e] = S[kk][e];
    }
}

// The same for the gradient of the state, backwards from token t_end - 1 on; dv comes with it.  Snapshots: the gradient of the state
// at the end of every chunk.
__device__ __noinline__ void scan_gradients_by_token(const OperatorPtrs &in, const __nv_bfloat16 *dy, __nv_bfloat16 *dv, const float *g_in, float *g_out,
                                                     float *snapshots, uint32_t *tops, unsigned char *smem, int bi, int h, int H, int Tlen, int t_end) {
    using Tiles = TokenTiles<__nv_bfloat16>;
    const Tiles tiles(in, dy, smem, bi, h, H, Tlen);
    const int row = (int)threadIdx.x >> 2, c0 = ((int)threadIdx.x & 3) * 4;
    const int last = (t_end - 1) / Tiles::kTokens * Tiles::kTokens;
    tiles.fetch(0, last, t_end);
    float G[4][4];
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
#pragma unroll
        for (int e = 0; e < 4; ++e) G[kk][e] = g_in ? g_in[row * kN + c0 + 16 * kk + e] : 0.f;
    for (int i = 0, first = last; first >= 0; ++i, first -= Tiles::kTokens) {
        tiles.arrived(i);
        if (first > 0) tiles.fetch(i + 1, first - Tiles::kTokens, t_end);
        for (int u = min(Tiles::kTokens, t_end - first) - 1; u >= 0; --u) {
            const int t = first + u;
            if (t == t_end - 1 || t % kL == kL - 1) {
                keep_top(tops + t / kL * 8, G);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                    for (int e = 0; e < 4; ++e) snapshots[(size_t)(t / kL) * kN * kN + accumulator_place(row, c0 + 16 * kk + e)] = G[kk][e];
            }
            auto f = [&](int x, int kk) { return Tiles::four(tiles.tile(i, x) + u * kN + c0 + 16 * kk); };
            const float dyi = __bfloat162float(tiles.tile(i, 5)[u * kN + row]);
            float dsa = 0.f, out = 0.f;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                const float4 r = f(XR, kk), b = f(XB, kk), k = f(XK, kk);
                const float rr[4] = {r.x, r.y, r.z, r.w}, bb[4] = {b.x, b.y, b.z, b.w}, kv[4] = {k.x, k.y, k.z, k.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    G[kk][e] = fmaf(dyi, rr[e], G[kk][e]);
                    dsa = fmaf(G[kk][e], bb[e], dsa);
                    out = fmaf(G[kk][e], kv[e], out);
                }
            }
#pragma unroll
            for (int x = 1; x <= 2; x <<= 1) {
                dsa += __shfl_xor_sync(0xffffffffu, dsa, x);
                out += __shfl_xor_sync(0xffffffffu, out, x);
            }
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                const float4 d = *reinterpret_cast<const float4 *>(tiles.d + u * kN + c0 + 16 * kk), a = f(XA, kk);
                const float dd[4] = {d.x, d.y, d.z, d.w}, aa[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) G[kk][e] = fmaf(G[kk][e], dd[e], dsa * aa[e]);
            }
            if (c0 == 0) dv[tiles.base + (size_t)t * tiles.step + row] = __float2bfloat16_rn(out);
        }
    }
    if (g_out != nullptr) {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
            for (int e = 0; e < 4; ++e) g_out[row * kN + c0 + 16 * kk + e] = G[kk][e];
    }
}

// What a scan is for.  Training needs the state every chunk starts with (kForTraining); its backward pass is the same scan
// over the transposed operators, last chunk first (kGradients): with G[j'][i] the gradient of the state behind a chunk and
// dY[t][i] that of its output,
//     D'[k][i] = sum_n O[n][k] [G; dY][n][i]
// has the rows j of the gradient in front of the chunk and the rows s of dV.
//
// Scales.  Values and states may be far smaller than fp16 resolves well, and gradients also larger than it holds: the state and V of a
// chunk (G and dY) go in times a power of two, chosen by the converting warps from the largest magnitudes of V in this chunk and the three
// before it in the scan's order and of the state as it entered the chunk three steps back, which the state warps publish.
// Forwards values are only scaled up: a chain that overflows fp16 is recomputed in fp32.  The choice does not depend on where a call
// is cut into segments: what the first three chunks of the next segment look back on is handed on with the chain's flag.
// Measured, training, 96 chains x 64 chunks: 71 and 67 us (gradients in channel order 76).
enum ScanKind { kPrefill, kForTraining, kGradients };

template <typename TIO, int kKind>
__global__ void __launch_bounds__(kScanThreads, 1)
wkv7_state_scan_kernel(const __grid_constant__ ScanMaps maps, OperatorPtrs ptrs, const TIO *__restrict__ v,
                       const unsigned char *__restrict__ records, const float *state_in, float *state_out,
                       TIO *__restrict__ y, float *__restrict__ snapshots, uint32_t *__restrict__ tops, int *flags, int Tlen, int H, int chunk0, int n, int resolve_flagged,
                       int *status) {
    constexpr bool kGrad = kKind == kGradients;
    using SM = Scan<TIO>;
    constexpr int NS = SM::kStages;
    extern __shared__ __align__(1024) unsigned char smem[];
    if (smem_u32(smem) & 1023u) {
        if (threadIdx.x == 0) atomicExch(status, (int)kDevInternal);
        return;
    }
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t sb = smem_u32(smem);
    uint64_t *bar_full = reinterpret_cast<uint64_t *>(smem + SM::kBars);   // [NS] a stage has landed
    uint64_t *bar_empty = bar_full + NS;                                   // [NS] its products are done
    uint64_t *bar_acc = bar_empty + NS;                                    // [2] an accumulator is complete
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bar_acc + 2);
    volatile int *bad = reinterpret_cast<volatile int *>(tmem_slot + 1);   // bit 0: a wait expired, bit 1: a value is not finite
    uint64_t *bar_scale = bar_acc + 3;                                     // [2] the scale of a chunk is known
    // Its exponent, by chunk mod 4; largest magnitude of the state as float bits, by chunk mod 4
    // (and at the start) and state warp; exponent of the largest V by chunk mod 2 and converting warp; what an output row of each
    // 16-token block is multiplied by, by chunk mod 4
    volatile int *scale_exp = reinterpret_cast<volatile int *>(smem + SM::kBars + 128);
    volatile uint32_t *top_z = reinterpret_cast<volatile uint32_t *>(smem + SM::kBars + 144);
    volatile int *top_v = reinterpret_cast<volatile int *>(smem + SM::kBars + 224);
    volatile float *row_up = reinterpret_cast<volatile float *>(smem + SM::kBars + 256);
    int *first_marked = reinterpret_cast<int *>(smem + SM::kBars + 320);
    float *state_then = reinterpret_cast<float *>(smem + kStateThen);   // behind the last step run, if the chain goes on token by token
    static_assert(8 * (2 * NS + 5) <= 128, "the barriers' place");
    // chunk of step c (gradients run from the last to the first)
    auto at_step = [&](int c) { return kGrad ? n - 1 - c : c; };
    const int chain = blockIdx.x;
    const int bi = chain / H, h = chain % H;
    if (tid == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(bar_full + s, 1);
            mbar_init(bar_empty + s, 1);
        }
        mbar_init(bar_acc, 1);
        mbar_init(bar_acc + 1, 1);
        mbar_init(bar_scale, 1);
        mbar_init(bar_scale + 1, 1);
        mbar_fence_init();
        *bad = 0;
        *first_marked = n;
        for (int i = 0; i < 8; ++i) top_v[i] = 0;
        tma_prefetch_desc(&maps.v);
        tma_prefetch_desc(&maps.y);
    }
    if (warp == 0) tmem_alloc(tmem_slot, 128);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // (launched behind the operator kernel with programmatic stream serialization: everything below reads what it wrote)
    wait_for_previous();
    let_next_in();
    const float *s_in = state_in ? state_in + (size_t)chain * kN * kN : nullptr;
    float *s_out = state_out ? state_out + (size_t)chain * kN * kN : nullptr;
    const unsigned char *rec = records + (size_t)chain * n * kRecord;
    // A chain is flagged by any of its chunks, in this segment or (as the scan of that segment left it, bit 0) an earlier one.
    // Above it, for the first three chunks of a segment: the exponent of what their scales have to cover from before it, 0 where
    // that is not known (then it is the state's at the start).
    const uint32_t left = chunk0 > 0 ? *reinterpret_cast<volatile uint32_t *>(&flags[chain]) : 0u;
    int mark = (int)(left & 1u);
    int first = n;   // step of the first marked chunk
    for (int c = tid; c < n; c += kScanThreads)
        if (*reinterpret_cast<const int *>(rec + (size_t)at_step(c) * kRecord + kMarkAt)) {
            mark = 1;
            first = min(first, c);
        }
    const bool flagged = __syncthreads_or(mark) != 0;
    // Steps to run here: all; none for a chain that later kernels take; those in front of the first marked chunk for one that is
    // continued token by token below.
    int run = flagged ? 0 : n;
    if (flagged && resolve_flagged) {
        if (first < n) atomicMin(first_marked, first);
        __syncthreads();
        run = *reinterpret_cast<volatile int *>(first_marked);
    }
    run = __shfl_sync(0xffffffffu, run, 0);   // (uniform, as the warp's number)
    uint32_t leave = flagged && !resolve_flagged ? 1u : 0u;   // (warp 10 writes it at the end)
    const int t_end = min(Tlen, (chunk0 + n) * kL);
    // Z of a chunk is written: four state warps arrive, the issuing warp waits.  V of chunk c is converted and the chunk's
    // accumulator, the one of two chunks before, read back: four converters and four output warps arrive.
    auto z_arrive = [] { asm volatile("bar.arrive 3, 160;" ::: "memory"); };
    auto v_arrive = [](int c) { asm volatile("bar.arrive %0, 288;" ::"r"(4 + (c & 1)) : "memory"); };
    uint32_t limit = 4000000u;   // polls a wait may take; after the first that expires this thread stops waiting, and the call reports it
    auto wait = [&](uint64_t *b, uint32_t parity) { limit = mbar_wait_tight(b, parity, limit) ? limit : 1u; };
    if (run == 0) {
        // (recomputed below, or by the next kernel in line)
    } else if (warp == 8) {
        // ---------------- loader
        if (lane == 0) {
            int issued = 0;
            for (int c = 0; c < run; ++c, ++issued) {
                const int s = c % NS;
                if (c >= NS) wait(bar_empty + s, (uint32_t)((c / NS - 1) & 1));
                if (limit == 1u) break;
                const uint32_t st = sb + s * SM::kStage;
                mbar_expect_tx(bar_full + s, kOperatorBytes + kVectorBytes + SM::kVBytes);
                const unsigned char *src = rec + (size_t)at_step(c) * kRecord;
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                             ::"r"(st), "l"(src), "r"(kOperatorBytes), "r"(smem_u32(bar_full + s))
                             : "memory");
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                             ::"r"(st + SM::kVec), "l"(src + kDecayAt), "r"(kVectorBytes), "r"(smem_u32(bar_full + s))
                             : "memory");
                const int trow = bi * Tlen + (chunk0 + at_step(c)) * kL;
                tma_load_2d(smem + s * SM::kStage + SM::kV, &maps.v, h * kN, trow, bar_full + s);
                if (SM::kF32) tma_load_2d(smem + s * SM::kStage + SM::kV + SM::kVBytes / 2, &maps.v, h * kN + 32, trow, bar_full + s);
            }
            // what has been requested lands before the CTA leaves, whatever became of the warps that read it
            for (int c = max(0, issued - NS); c < issued; ++c) mbar_wait(bar_full + c % NS, (uint32_t)((c / NS) & 1));
        }
        __syncwarp();
    } else if (warp == 9) {
        // ---------------- issuing warp
        constexpr uint32_t id = make_idesc(kFmtF16, 128, 64, kGrad, true);
        auto v_products = [&](int c) {
            const int s = c % NS, a = c & 1;
            wait(bar_full + s, (uint32_t)((c / NS) & 1));
            asm volatile("bar.sync %0, 288;" ::"r"(4 + a) : "memory");
            if (elect_one()) {
                tc_fence_after();
                const uint32_t op = sb + s * SM::kStage, vt = sb + SM::kZV + a * 2 * kPanel + kPanel;
#pragma unroll
                for (int ks = 0; ks < 4; ++ks)
                    umma_f16(tmem + a * 64, desc_operator<kGrad>(op, 4 + ks), make_smem_desc(vt + ks * 2048u, kPanel, 1024u), id, ks > 0);
            }
            __syncwarp();
        };
        v_products(0);
        for (int c = 0; c < run; ++c) {
            const int s = c % NS, a = c & 1;
            asm volatile("bar.sync 3, 160;" ::: "memory");
            if (elect_one()) {
                tc_fence_after();
                const uint32_t op = sb + s * SM::kStage, zt = sb + SM::kZV + a * 2 * kPanel;
#pragma unroll
                for (int ks = 0; ks < 4; ++ks)
                    umma_f16(tmem + a * 64, desc_operator<kGrad>(op, ks), make_smem_desc(zt + ks * 2048u, kPanel, 1024u), id, true);
                umma_commit(bar_acc + a);
                umma_commit(bar_empty + s);
            }
            __syncwarp();
            if (c + 1 < run) v_products(c + 1);
        }
    } else if (warp >= 10) {
        // ---------------- V converters: tile -> fp16 rows in the order of the contraction index, 16-byte pieces; rows past the sequence's end belong to
        // another one, whatever they hold stays out of the sums
        constexpr int kShare = kL * kN / 8 / 32 / kConverters;
        // What is largest, the state or eight times V (a state gathers a chunk's V times k; a gradient dY times r), comes to lie in
        // [32, 64): eleven binary orders to overflow, and a state that falls by nineteen within three chunks is still resolved.
        constexpr int kAbove = 3, kUnscaled = 127 + 5;
        const int own = warp - 10;                  // this warp's token block
        int carried[3], before[3] = {0, 0, 0};      // exponents; of V (dY) one, two and three chunks ago
        auto most_at = [&](uint32_t at) {   // of four words
            uint32_t x[4];
            lds128(x, sb + SM::kBars + at);
            return max(max(x[0], x[1]), max(x[2], x[3]));
        };
        auto top_state = [&](int slot) { return (int)(most_at(144 + slot * 16) >> 23); };
        asm volatile("bar.sync 7, 256;" ::: "memory");   // the state warps have published the start
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const int x = (int)(left >> (8 + 8 * i)) & 255;
            carried[i] = x ? x : top_state(4);
        }
        for (int c = 0; c < run; ++c) {
            const int s = c % NS, a = c & 1;
            wait(bar_full + s, (uint32_t)((c / NS) & 1));
            const uint32_t vt = sb + s * SM::kStage + SM::kV, out = sb + SM::kZV + a * 2 * kPanel + kPanel;
            const int valid = Tlen - (chunk0 + at_step(c)) * kL;
            const signed char *row_exp = reinterpret_cast<const signed char *>(smem + s * SM::kStage + SM::kVec + kRowExpAt);
            const int e_in = row_exp[2 * own + (kGrad ? 0 : 1)];
            auto token = [&](int k) { return ((own * kShare + k) * 32 + lane) >> 3; };
            // eight channels of a token (fp32: two pieces of a panel of 32 channels)
            constexpr int kWords = SM::kF32 ? 8 : 4;
            uint32_t x[kShare][kWords];
            __nv_bfloat162 m[4];
            float m32[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int e = 0; e < 4; ++e) m[e] = __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll
            for (int k = 0; k < kShare; ++k) {
                const int t = token(k), cg = lane & 7;
                if constexpr (!SM::kF32) lds128(x[k], vt + off16(t, cg * 8));
                else {
                    const uint32_t row = vt + (cg >> 2) * (SM::kVBytes / 2) + t * 128;
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const float4 f = lds_f4(row + (((2 * cg & 7) + i) ^ (t & 7)) * 16);
                        x[k][4 * i] = __float_as_uint(f.x); x[k][4 * i + 1] = __float_as_uint(f.y);
                        x[k][4 * i + 2] = __float_as_uint(f.z); x[k][4 * i + 3] = __float_as_uint(f.w);
                    }
                }
#pragma unroll
                for (int e = 0; e < kWords; ++e) {
                    if (t >= valid) x[k][e] = 0;
                    if constexpr (!SM::kF32) m[e] = __hmax2(m[e], __habs2(*reinterpret_cast<const __nv_bfloat162 *>(&x[k][e])));
                    else m32[e & 3] = fmaxf(m32[e & 3], fabsf(__uint_as_float(x[k][e])));
                }
            }
            const __nv_bfloat162 mm = __hmax2(__hmax2(m[0], m[1]), __hmax2(m[2], m[3]));
            const float most = SM::kF32 ? fmaxf(fmaxf(m32[0], m32[1]), fmaxf(m32[2], m32[3])) : fmaxf(__low2float(mm), __high2float(mm));
            int top = (int)(__reduce_max_sync(0xffffffffu, __float_as_uint(most)) >> 23);
            if (top > 0) top = max(top + e_in, 1);
            if (lane == 0) top_v[a * 4 + own] = top;
            asm volatile("bar.sync 6, 128;" ::: "memory");
            if (c >= 2) wait(bar_acc + a, (uint32_t)(((c >> 1) - 1) & 1));   // the products that last read this tile
            const int now = (int)most_at(224 + a * 16);
            const int v_most = max(max(now, before[0]), max(before[1], before[2]));
            const int all = max(c < 3 ? (c == 0 ? carried[0] : c == 1 ? carried[1] : carried[2]) : top_state((c - 3) & 3), v_most > 0 ? v_most + kAbove : 0);
            const int ex = all > 0 ? min(max(all - kUnscaled, -96), kGrad ? 96 : 0) : 0;
            before[2] = before[1];
            before[1] = before[0];
            before[0] = now;
            if (own == 0) {
                if (lane < 4) row_up[(c & 3) * 4 + lane] = exp2_of(ex) * exp2_of(row_exp[2 * lane + (kGrad ? 1 : 0)]);
                if (lane == 0) scale_exp[c & 3] = ex;
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_scale + a);   // (a hardware barrier would have the state warps wait for one another too)
            }
#pragma unroll
            for (int k = 0; k < kShare; ++k) {
                const float f1 = exp2_of(max(e_in - ex, -126));
                uint32_t y[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float2 v2;
                    if constexpr (!SM::kF32) v2 = unpack_bf2(x[k][e]);
                    else v2 = make_float2(__uint_as_float(x[k][2 * e]), __uint_as_float(x[k][2 * e + 1]));
                    y[e] = pack2(mul2(v2, make_float2(f1, f1)));
                }
                // (dY of a chunk: rows in token order)
                sts128(out + off16(kGrad ? token(k) : k_position(token(k)), (lane & 7) * 8), y);
            }
            fence_proxy_async();
            v_arrive(c);
        }
        if (!flagged && (chunk0 + n) * kL < Tlen) {   // what the next segment's first chunks look back on
            asm volatile("bar.sync 7, 256;" ::: "memory");   // (the state warps have published every chunk)
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                int x = n + i >= 3 ? top_state((n + i - 3) & 3) : n + i == 1 ? carried[1] : carried[2];
#pragma unroll
                for (int k = 0; k < 3 - i; ++k) x = max(x, before[k] > 0 ? before[k] + kAbove : 0);
                leave |= (uint32_t)min(x, 255) << (8 + 8 * i);
            }
        }
    } else {
        const int quarter = warp & 3, hf = warp >> 2;
        const uint32_t acc = tmem + ((uint32_t)(quarter * 32) << 16) + hf * 32;
        const int i0 = hf * 32;                       // this thread's 32 value channels
        if (quarter < 2) {
            // ---------------- state rows j'
            // (accumulator rows are in the order of the contraction index, so that neighbouring lanes write neighbouring operand rows)
            const int zr = quarter * 32 + lane, jp = k_at_position(zr);
            const uint32_t zrow = sb + SM::kZV + off16(zr, 0);
            const uint32_t sw = ((uint32_t)zr & 7u) << 4;
            float2 Z[16];
#pragma unroll
            for (int e = 0; e < 16; ++e)
                Z[e] = s_in ? make_float2(s_in[(i0 + 2 * e) * kN + jp], s_in[(i0 + 2 * e + 1) * kN + jp]) : make_float2(0.f, 0.f);
            // this row's scalars of a chunk: e^{c_L}, and what the operand and the product are multiplied by: fx and the factor of P
            // and Kt, or, for gradients, the other way round; both with the chunk's scale
            auto load_vec = [&](int c, float &gx, float &fx, float &g2) {
                const int s = c % NS;
                wait(bar_full + s, (uint32_t)((c / NS) & 1));
                const unsigned char *vec = smem + s * SM::kStage + SM::kVec;
                gx = *reinterpret_cast<const float *>(vec + jp * 4);
                const int ef = *reinterpret_cast<const signed char *>(vec + 256 + jp), eg = *reinterpret_cast<const signed char *>(vec + 320 + jp);
                wait(bar_scale + (c & 1), (uint32_t)((c >> 1) & 1));
                const float up = exp2_of(scale_exp[c & 3]), down = exp2_of(-scale_exp[c & 3]);
                if constexpr (kGrad) {
                    fx = exp2_of(-eg) * down;
                    g2 = gx * exp2_of(ef) * up;
                } else {
                    fx = gx * exp2_of(ef) * down;
                    g2 = exp2_of(-eg) * up;
                }
            };
            // largest magnitude of the state in this warp's share
            auto largest = [&] {
                float m[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int e = 0; e < 16; ++e) m[e & 3] = max3_abs(m[e & 3], Z[e].x, Z[e].y);
                return __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3]))));
            };
            auto keep = [&](int c, uint32_t most) {   // the state that step c starts from, for the kernel of the chunks (see accumulator_place)
                if (lane < 2) tops[((size_t)chain * n + at_step(c)) * 8 + quarter * 2 + hf + 4 * lane] = lane ? 0u : most;
                float *dst = snapshots + ((size_t)chain * n + at_step(c)) * kN * kN + accumulator_place(i0, jp);
#pragma unroll
                for (int m = 0; m < 32; m = m == 7 ? 16 : m + 1) {
                    if (m >= 24) break;
                    const float2 lo = Z[m >> 1], hi = Z[(m + 8) >> 1];
                    if (RWKV7_IN_RANGE(c < n && i0 + m + 8 < kN && jp < kN, status))
                        *reinterpret_cast<float2 *>(dst + (m >> 4) * 1024 + (m & 7) * 16) = m & 1 ? make_float2(lo.y, hi.y) : make_float2(lo.x, hi.x);
                }
            };
            // the state a chunk starts with, as operand: times fx, fp16
            auto put_z = [&](int c, float fx) {
                const float2 f = make_float2(fx, fx);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const uint32_t x[4] = {pack2(mul2(Z[4 * e], f)), pack2(mul2(Z[4 * e + 1], f)), pack2(mul2(Z[4 * e + 2], f)), pack2(mul2(Z[4 * e + 3], f))};
                    // (16-byte pieces XOR-ed with the row: zrow is piece 0's place)
                    sts128((zrow ^ sw) + (c & 1) * 2 * kPanel + ((uint32_t)((i0 / 8 + e) << 4) ^ sw), x);
                }
                fence_proxy_async();
                tc_fence_before();
                z_arrive();
            };
            float gx, fx, g2, gxn = 1.f, fxn = 1.f, g2n = 0.f;
            {
                const uint32_t most = largest();
                if (lane == 0) top_z[16 + quarter * 2 + hf] = most;
                asm volatile("bar.sync 7, 256;" ::: "memory");
            }
            load_vec(0, gx, fx, g2);
            put_z(0, fx);
            for (int c = 0; c < run; ++c) {
                const int a = c & 1;
                const uint32_t most = largest();
                if (lane == 0) top_z[(c & 3) * 4 + quarter * 2 + hf] = most;   // for the converting warps
                if constexpr (kKind != kPrefill) keep(c, most);
                if (c + 1 < run) load_vec(c + 1, gxn, fxn, g2n);   // (while the products run)
                wait(bar_acc + a, (uint32_t)((c >> 1) & 1));
                tc_fence_after();
                uint32_t d[32];
                tmem_ld32(acc + a * 64, d);
                tmem_ld_wait();
                const float2 gx2 = make_float2(gx, gx), gg = make_float2(g2, g2);
#pragma unroll
                for (int e = 0; e < 16; ++e)
                    Z[e] = __ffma2_rn(gx2, Z[e], mul2(gg, make_float2(__uint_as_float(d[2 * e]), __uint_as_float(d[2 * e + 1]))));
                if (c + 1 < run) put_z(c + 1, fxn);
                gx = gxn;
                g2 = g2n;
            }
            if (!flagged && (chunk0 + n) * kL < Tlen) asm volatile("bar.sync 7, 256;" ::: "memory");
            bool off = false;   // a non-finite operand upstream stays in the state for good
#pragma unroll
            for (int e = 0; e < 16; ++e) off |= !(fabsf(Z[e].x) <= 3.0e38f) | !(fabsf(Z[e].y) <= 3.0e38f);
            if (off) atomicOr(const_cast<int *>(bad), 2);
            if (limit == 1u) atomicOr(const_cast<int *>(bad), 1);
            // the eight compute warps have all reported before the state is written: it may alias what a recomputation
            // starts from
            asm volatile("bar.sync 1, 256;" ::: "memory");
            if (flagged) {
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    state_then[(i0 + 2 * e) * kN + jp] = Z[e].x;
                    state_then[(i0 + 2 * e + 1) * kN + jp] = Z[e].y;
                }
            } else if (*bad == 0 && s_out != nullptr) {
#pragma unroll
                for (int e = 0; e < 16; ++e)
                    if (RWKV7_IN_RANGE(i0 + 2 * e + 1 < kN && jp < kN, status)) {
                        s_out[(i0 + 2 * e) * kN + jp] = Z[e].x;
                        s_out[(i0 + 2 * e + 1) * kN + jp] = Z[e].y;
                    }
            }
        } else {
            // ---------------- output tokens t.  A chunk's y tile is staged in shared memory (one of two buffers) and leaves
            // by a bulk tensor store; a partial last chunk is stored by the threads themselves.
            const int tq = kGrad ? k_at_position((quarter - 2) * 32 + lane) : (quarter - 2) * 32 + lane;   // token within the chunk
            const bool elected = warp == 2 && lane == 0;
            float ysum = 0.f;    // a non-finite output makes the sum non-finite for good
            v_arrive(0);
            if (run > 1) v_arrive(1);
            for (int c = 0; c < run; ++c) {
                const int a = c & 1;
                wait(bar_acc + a, (uint32_t)((c >> 1) & 1));
                tc_fence_after();
                uint32_t d[32];
                tmem_ld32(acc + a * 64, d);
                tmem_ld_wait();
                const float up = row_up[(c & 3) * 4 + (tq >> 4)];
#pragma unroll
                for (int e = 0; e < 32; e += 2) {
                    const float2 y2 = mul2(make_float2(__uint_as_float(d[e]), __uint_as_float(d[e + 1])), make_float2(up, up));
                    d[e] = __float_as_uint(y2.x);
                    d[e + 1] = __float_as_uint(y2.y);
                }
                tc_fence_before();
                if (c + 2 < run) v_arrive(c + 2);
                const int t0 = (chunk0 + at_step(c)) * kL;
                float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int e = 0; e < 32; ++e) sum[e & 3] += fabsf(__uint_as_float(d[e]));
                ysum += (sum[0] + sum[1]) + (sum[2] + sum[3]);
                constexpr int kPieces = SM::kF32 ? 8 : 4;   // 16-byte pieces of this thread's channels
                uint32_t w[4 * kPieces];
                if constexpr (!SM::kF32) {
#pragma unroll
                    for (int e2 = 0; e2 < 16; ++e2) {
                        const __nv_bfloat162 b2 = __floats2bfloat162_rn(__uint_as_float(d[2 * e2]), __uint_as_float(d[2 * e2 + 1]));
                        w[e2] = *reinterpret_cast<const uint32_t *>(&b2);
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < 32; ++e) w[e] = d[e];
                }
                if (t0 + kL <= Tlen) {
                    // (bf16: 128-byte rows of 64 channels; fp32: two panels of 32 channels)
                    const uint32_t stage = sb + SM::kY + a * SM::kYTile + (SM::kF32 ? hf * (SM::kYTile / 2) : 0u) + (uint32_t)tq * 128u;
                    if (elected) bulk_wait_group_read<1>();   // the store that last read this buffer (two chunks ago) is done with it
                    asm volatile("bar.sync 2, 128;" ::: "memory");
#pragma unroll
                    for (int e = 0; e < kPieces; ++e) {
                        const uint32_t x[4] = {w[4 * e], w[4 * e + 1], w[4 * e + 2], w[4 * e + 3]};
                        const uint32_t o = (uint32_t)(((SM::kF32 ? 0 : i0 / 8) + e) ^ (tq & 7)) << 4;
                        if (RWKV7_IN_RANGE(o + 16 <= 128u, status)) sts128(stage + o, x);
                    }
                    fence_proxy_async();
                    asm volatile("bar.sync 2, 128;" ::: "memory");
                    if (elected) {
                        unsigned char *tile = smem + SM::kY + a * SM::kYTile;
                        tma_store_2d(&maps.y, h * kN, bi * Tlen + t0, tile);
                        if (SM::kF32) tma_store_2d(&maps.y, h * kN + 32, bi * Tlen + t0, tile + SM::kYTile / 2);
                        bulk_commit_group();
                    }
                } else if (t0 + tq < Tlen) {
                    TIO *dst = y + (((size_t)bi * Tlen + t0 + tq) * H + h) * kN + i0;
#pragma unroll
                    for (int e = 0; e < kPieces; ++e)
                        *reinterpret_cast<uint4 *>(dst + e * (16 / sizeof(TIO))) = make_uint4(w[4 * e], w[4 * e + 1], w[4 * e + 2], w[4 * e + 3]);
                }
            }
            if (elected) bulk_wait_group<0>();   // (a recomputation below may write the same rows)
            if (!(ysum <= 3.0e38f)) atomicOr(const_cast<int *>(bad), 2);
            if (limit == 1u) atomicOr(const_cast<int *>(bad), 1);
            asm volatile("bar.sync 1, 256;" ::: "memory");
        }
    }
    if (limit == 1u) atomicOr(const_cast<int *>(bad), 1);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 128);
    if (warp == 10 && lane == 0) flags[chain] = (int)(*bad ? leave & 1u : leave);   // (a chain redone below starts afresh)
    if (*bad & 1) {
        if (tid == 0) atomicExch(status, (int)kDevTimeout);
        return;
    }
    // A value beyond fp16: the chain once more, token by token, from the state this launch started with, which is still
    // untouched.  A flagged chain that nobody else takes: on from its first marked chunk.
    if (((flagged && resolve_flagged) || (*bad & 2)) && tid < 256) {
        float *own = snapshots + (kKind == kPrefill ? 0 : (size_t)chain * n * kN * kN);
        uint32_t *top = tops + (kKind == kPrefill ? 0 : (size_t)chain * n * 8);
        const int done = (*bad & 2) ? 0 : run;
        const float *from = done > 0 ? state_then : s_in;
        if constexpr (kGrad) scan_gradients_by_token(ptrs, v, y, from, s_out, own, top, smem, bi, h, H, Tlen, min(Tlen, (n - done) * kL));
        else scan_rows_by_token<TIO>(ptrs, v, y, from, s_out, kKind == kPrefill ? nullptr : own, top, smem, bi, h, H, Tlen, (chunk0 + done) * kL, t_end);
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
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

// A [B,T,H,64] tensor as rows of channels, in tiles of 64 tokens by 128 bytes.
bool describe_rows(CUtensorMap *map, const void *ptr, int64_t B, int64_t T, int64_t H, bool bf16) {
    const EncodeTiledFn encode = encode_fn();
    const size_t esize = bf16 ? 2 : 4;
    const cuuint64_t dims[2] = {(cuuint64_t)(H * kN), (cuuint64_t)(B * T)};
    const cuuint64_t strides[1] = {(cuuint64_t)(H * kN * esize)};
    const cuuint32_t box[2] = {(cuuint32_t)(128 / esize), (cuuint32_t)kL};
    const cuuint32_t estr[2] = {1, 1};
    return encode != nullptr &&
           encode(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void *>(ptr), dims, strides, box,
                  estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

constexpr size_t kAlign = 256;
size_t align_up(size_t x) { return (x + kAlign - 1) / kAlign * kAlign; }
// Operator storage the launcher aims for: beyond this a call is cut into segments of chunks.
constexpr size_t kOperatorBudget = (size_t)768 << 20;

}  // namespace

// ---- host side ------------------------------------------------------------------------------
//
// Workspace: [flags: one int per chain][carried fp32 state per chain][records of buffer 0][records of buffer 1]; a call of one
// segment carries nothing.  A call is cut into segments of chunks.  With at most as many chains as SMs the scan of a segment
// leaves most of the GPU idle (one latency-bound CTA per chain), so it runs on a second stream beside
// the operator kernel of the next segment, which writes the other buffer.

namespace {

constexpr int kMaxSegments = 1024;

struct WorkspaceLayout {
    size_t flags, carry, records[2], total;
    size_t seg;      // chunks per segment
    int buffers;     // 1 or 2
};

// What lies in front of the records.  (4 KB of a cut call's are not used; callers who work out the least size have counted them.)
size_t fixed_part(size_t chains, bool cut) {
    return align_up(chains * sizeof(int)) + (cut ? 4096 + align_up(chains * kN * kN * sizeof(float)) : 0);
}

WorkspaceLayout layout_for(size_t chains, size_t seg, int buffers, bool cut) {
    WorkspaceLayout l{};
    l.seg = seg;
    l.buffers = buffers;
    l.flags = 0;
    l.carry = align_up(chains * sizeof(int)) + 4096;
    size_t off = fixed_part(chains, cut);
    for (int b = 0; b < 2; ++b) {
        l.records[b] = off;
        if (b < buffers) off += chains * seg * kRecord;
    }
    l.total = off;
    return l;
}

// How a call is cut: the number of segments that balances the scan of the last segment (which nothing
// overlaps) against the few microseconds a segment boundary costs, within the operator budget.
//
// When the scan of a segment may run beside the operator kernel of the next one: see wkv7_overlap.h.
bool overlap_applies(size_t chains, size_t nchunks, int num_sms) {
    return wkv7_split_overlap() != 0 && partition_overlap_pays(chains, nchunks, num_sms);
}

size_t preferred_segment(size_t chains, size_t nchunks, bool overlap) {
    size_t seg = nchunks;
    if (overlap) {
        size_t nseg = 1;
        while ((nseg + 1) * (nseg + 1) * 16 <= nchunks && nseg < 32) ++nseg;   // about sqrt(nchunks / 16): measured best (1024 chunks: 8 segments)
        seg = (nchunks + nseg - 1) / nseg;
    }
    const size_t per_chunk = chains * kRecord * (overlap ? 2 : 1);
    if (seg * per_chunk > kOperatorBudget) seg = kOperatorBudget / per_chunk;
    if ((nchunks + seg - 1) / (seg ? seg : 1) > (size_t)kMaxSegments) seg = (nchunks + kMaxSegments - 1) / kMaxSegments;
    return seg < 1 ? 1 : seg;
}

// Second stream and events of a device, created on first use.
struct DeviceStreams {
    cudaStream_t side = nullptr;
    cudaEvent_t fork = nullptr, built[2] = {nullptr, nullptr}, scanned[2] = {nullptr, nullptr};
    bool ok = false;
};

std::mutex g_streams_mu;
DeviceStreams g_streams[64];

// (the caller holds g_streams_mu and has made `device` current)
DeviceStreams *device_streams(int device) {
    if (device < 0 || device >= 64) return nullptr;
    DeviceStreams &d = g_streams[device];
    if (!d.ok) {
        int least = 0, greatest = 0;
        if (cudaDeviceGetStreamPriorityRange(&least, &greatest) != cudaSuccess) return nullptr;
        if (cudaStreamCreateWithPriority(&d.side, cudaStreamNonBlocking, greatest) != cudaSuccess) return nullptr;
        cudaEvent_t *evs[5] = {&d.fork, &d.built[0], &d.built[1], &d.scanned[0], &d.scanned[1]};
        for (cudaEvent_t *e : evs)
            if (cudaEventCreateWithFlags(e, cudaEventDisableTiming) != cudaSuccess) return nullptr;
        d.ok = true;
    }
    return &d;
}

// ---- SM partitions (green contexts) for the overlapped schedule ----------------------------------
// The scan of a segment and the operator kernel of the next one want different things from an SM: a scan CTA is
// one latency-bound chain that needs an SM to itself, an operator CTA is throughput work, four to an SM, and holds up a scan
// that waits for its SM.  Where the driver offers it, the device's SMs are therefore split once into two partitions, each with
// a stream of its own, and neither kernel sees the other's CTAs.
struct GreenApi {
    CUresult (*deviceGet)(CUdevice *, int) = nullptr;
    CUresult (*getRes)(CUdevice, CUdevResource *, CUdevResourceType) = nullptr;
    CUresult (*split)(CUdevResource *, unsigned int *, const CUdevResource *, CUdevResource *, unsigned int, unsigned int) = nullptr;
    CUresult (*genDesc)(CUdevResourceDesc *, CUdevResource *, unsigned int) = nullptr;
    CUresult (*create)(CUgreenCtx *, CUdevResourceDesc, CUdevice, unsigned int) = nullptr;
    CUresult (*streamCreate)(CUstream *, CUgreenCtx, unsigned int, int) = nullptr;
    CUresult (*ctxFromGreen)(CUcontext *, CUgreenCtx) = nullptr;
    CUresult (*ctxPush)(CUcontext) = nullptr;
    CUresult (*ctxPop)(CUcontext *) = nullptr;
    bool ok = false;
};

const GreenApi &green_api() {
    static GreenApi api;
    static std::once_flag once;
    std::call_once(once, [] {
        auto get = [](const char *name, void **out) {
            cudaDriverEntryPointQueryResult q;
            return cudaGetDriverEntryPoint(name, out, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess &&
                   *out != nullptr;
        };
        api.ok = get("cuDeviceGet", reinterpret_cast<void **>(&api.deviceGet)) &&
                 get("cuDeviceGetDevResource", reinterpret_cast<void **>(&api.getRes)) &&
                 get("cuDevSmResourceSplitByCount", reinterpret_cast<void **>(&api.split)) &&
                 get("cuDevResourceGenerateDesc", reinterpret_cast<void **>(&api.genDesc)) &&
                 get("cuGreenCtxCreate", reinterpret_cast<void **>(&api.create)) &&
                 get("cuGreenCtxStreamCreate", reinterpret_cast<void **>(&api.streamCreate)) &&
                 get("cuCtxFromGreenCtx", reinterpret_cast<void **>(&api.ctxFromGreen)) &&
                 get("cuCtxPushCurrent", reinterpret_cast<void **>(&api.ctxPush)) &&
                 get("cuCtxPopCurrent", reinterpret_cast<void **>(&api.ctxPop));
        (void)cudaGetLastError();
    });
    return api;
}

struct DevicePartition {
    int scan_sms = 0, op_sms = 0;          // SMs of the two partitions as the driver cut them
    cudaStream_t scan_stream = nullptr, op_stream = nullptr;
    // (an event is recorded only on a stream of the context it was created in; waits may cross contexts)
    cudaEvent_t built[2] = {nullptr, nullptr}, scanned[2] = {nullptr, nullptr};
    bool tried = false, ok = false;
};

// per device, per size of the scan partition in units of eight SMs (the granularity of a split)
DevicePartition g_partitions[64][10];

// (the caller holds g_streams_mu and has made `device` current)  Null when the driver does not offer it.
DevicePartition *device_partition(int device, int want_scan_sms, int num_sms) {
    const GreenApi &api = green_api();
    const int slot = (want_scan_sms + 7) / 8;
    // A tool injected into the process (a profiler, a memory checker: they announce themselves through these
    // variables) may not support kernels in green contexts: Nsight Compute 2025.2 fails to prepare them for
    // profiling and ends the application.  Under such a tool the partitions are not used.
    static const bool injected = std::getenv("CUDA_INJECTION64_PATH") != nullptr ||
                                 std::getenv("NV_NSIGHT_INJECTION_PORT_BASE") != nullptr ||
                                 std::getenv("NV_COMPUTE_PROFILER_PERFWORKS_DIR") != nullptr;
    if (!api.ok || injected || device < 0 || device >= 64 || slot < 1 || slot >= 10) return nullptr;
    DevicePartition &d = g_partitions[device][slot];
    if (d.tried) return d.ok ? &d : nullptr;
    d.tried = true;
    CUdevice dev;
    CUdevResource all, scan_res, op_res;
    unsigned int nb = 1;
    if (api.deviceGet(&dev, device) != CUDA_SUCCESS) return nullptr;
    if (api.getRes(dev, &all, CU_DEV_RESOURCE_TYPE_SM) != CUDA_SUCCESS) return nullptr;
    if (api.split(&scan_res, &nb, &all, &op_res, 0, (unsigned int)(slot * 8)) != CUDA_SUCCESS || nb != 1) return nullptr;
    d.scan_sms = (int)scan_res.sm.smCount;
    d.op_sms = (int)op_res.sm.smCount;
    if (d.scan_sms < want_scan_sms || d.op_sms < num_sms / 2) return nullptr;
    int least = 0, greatest = 0;
    if (cudaDeviceGetStreamPriorityRange(&least, &greatest) != cudaSuccess) return nullptr;
    struct Half { CUdevResource *res; cudaStream_t *stream; cudaEvent_t *events; int priority; };
    const Half halves[2] = {{&scan_res, &d.scan_stream, d.scanned, greatest}, {&op_res, &d.op_stream, d.built, least}};
    for (const Half &h : halves) {
        CUdevResourceDesc desc;
        CUgreenCtx green;
        CUcontext ctx, popped;
        CUstream st;
        if (api.genDesc(&desc, h.res, 1) != CUDA_SUCCESS) return nullptr;
        if (api.create(&green, desc, dev, CU_GREEN_CTX_DEFAULT_STREAM) != CUDA_SUCCESS) return nullptr;
        if (api.streamCreate(&st, green, CU_STREAM_NON_BLOCKING, h.priority) != CUDA_SUCCESS) return nullptr;
        *h.stream = reinterpret_cast<cudaStream_t>(st);
        if (api.ctxFromGreen(&ctx, green) != CUDA_SUCCESS || api.ctxPush(ctx) != CUDA_SUCCESS) return nullptr;
        bool made = true;
        for (int i = 0; i < 2; ++i) made = made && cudaEventCreateWithFlags(&h.events[i], cudaEventDisableTiming) == cudaSuccess;
        api.ctxPop(&popped);
        if (!made) return nullptr;
    }
    d.ok = true;
    return &d;
}

std::atomic<int> g_split_overlap{1};

}  // namespace

int wkv7_split_overlap() { return g_split_overlap.load(); }
// 0: everything on the caller's stream; 1: overlapped, on SM partitions where the driver offers them;
// 2: overlapped on the second stream without partitions.
void wkv7_set_split_overlap(int on) { g_split_overlap.store(on < 0 || on > 2 ? 1 : on); }

size_t wkv7_split_min_workspace_bytes(int64_t B, int64_t T, int64_t H, int64_t N) {
    if (N != kN) return 0;
    return layout_for((size_t)(B * H), 1, 1, T > kL).total;
}

bool wkv7_split_in_budget(int64_t B, int64_t H) { return (size_t)(B * H) * kRecord <= kOperatorBudget; }

size_t wkv7_split_workspace_bytes(int64_t B, int64_t T, int64_t H, int64_t N, int num_sms) {
    if (N != kN) return 0;
    const size_t chains = (size_t)(B * H);
    const size_t nchunks = (size_t)((T + kL - 1) / kL);
    const bool overlap = overlap_applies(chains, nchunks, num_sms);
    const size_t seg = preferred_segment(chains, nchunks, overlap);
    return layout_for(chains, seg, overlap ? 2 : 1, seg < nchunks).total;
}

bool wkv7_split_supported(const Wkv7Args &p) {
    auto aligned = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
    return p.N == kN && aligned(p.r) && aligned(p.w) && aligned(p.k) && aligned(p.v) && aligned(p.a) &&
           aligned(p.b) && aligned(p.y) && p.B * p.T < (int64_t(1) << 31) && p.B * p.H < (int64_t(1) << 24);
}

// Enqueues the two kernels, once per segment of chunks, and leaves one flag per chain in the first
// B*H ints of the workspace: 1 for chains that the caller's next kernel must recompute (their final
// state is not written: it may alias the initial state that the recomputation starts from).
int launch_wkv7_split(const Wkv7Args &p, void *workspace, size_t workspace_bytes, bool wide_range, bool resolve_flagged,
                      cudaStream_t stream) {
    if (encode_fn() == nullptr) return (int)cudaErrorNotSupported;
    const size_t chains = (size_t)(p.B * p.H);
    const int nchunks = (int)((p.T + kL - 1) / kL);
    // The plan: overlapped (two buffers) when it applies and the workspace holds two segments of a useful
    // length, else one buffer with the longest segment that fits.
    // (fp32 tensors stay in sequence: the schedules have not been measured with their kernels)
    bool overlap = p.bf16 && overlap_applies(chains, (size_t)nchunks, p.num_sms);
    // The second stream and its events, or the two SM partitions with theirs, are shared by all calls on a device:
    // the enqueueing of an overlapped call is serialised per process from here on.
    std::unique_lock<std::mutex> lock(g_streams_mu, std::defer_lock);
    DevicePartition *part = nullptr;
    if (overlap) {
        lock.lock();
        // (a stream that is being captured into a graph stays within its own context: no partitions then)
        cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(stream, &capturing) != cudaSuccess) capturing = cudaStreamCaptureStatusActive;
        if (wkv7_split_overlap() == 1 && capturing == cudaStreamCaptureStatusNone)
            part = device_partition(p.device, (int)chains, p.num_sms);
        if (part == nullptr && !shared_sm_overlap_pays(chains, (size_t)nchunks, p.num_sms)) overlap = false;
    }
    size_t seg = preferred_segment(chains, (size_t)nchunks, overlap);
    const size_t per_chunk = chains * kRecord, fixed = fixed_part(chains, true), room = workspace_bytes > fixed ? workspace_bytes - fixed : 0;
    if (overlap && layout_for(chains, seg, 2, true).total > workspace_bytes) {
        const size_t fit = room / (2 * per_chunk);
        if (fit >= 8) seg = fit;
        else overlap = false;
    }
    if (!overlap) {
        seg = preferred_segment(chains, (size_t)nchunks, false);
        if (seg < (size_t)nchunks || layout_for(chains, seg, 1, false).total > workspace_bytes) {
            const size_t fit = room / per_chunk;
            if (fit < 1) return (int)cudaErrorInvalidValue;
            if (seg > fit) seg = fit;
        }
    }
    if (seg > (size_t)nchunks) seg = (size_t)nchunks;
    const int nsegments = (int)(((size_t)nchunks + seg - 1) / seg);
    if (nsegments > kMaxSegments) return (int)cudaErrorInvalidValue;
    if (nsegments < 2) overlap = false;
    const WorkspaceLayout lay = layout_for(chains, seg, overlap ? 2 : 1, nsegments > 1);
    unsigned char *ws = static_cast<unsigned char *>(workspace);
    int *flags = reinterpret_cast<int *>(ws + lay.flags);
    float *carry = reinterpret_cast<float *>(ws + lay.carry);

    OperatorMaps omaps{};
    ScanMaps smaps{};
    const OperatorPtrs optrs{{p.a, p.r, p.b, p.k, p.w}};
    auto describe = [&](CUtensorMap *map, const void *ptr) { return describe_rows(map, ptr, p.B, p.T, p.H, p.bf16); };
    for (int i = 0; p.bf16 && i < 5; ++i)   // (fp32 tensors are read by the threads themselves)
        if (!describe(&omaps.m[i], optrs.p[i])) return (int)cudaErrorInvalidValue;
    if (!describe(&smaps.v, p.v) || !describe(&smaps.y, p.y)) return (int)cudaErrorInvalidValue;
    int *status = nullptr;
    if (int e = device_status_ptr(p.device, &status)) return e;

    auto k1 = p.bf16 ? wkv7_chunk_operator_kernel<__nv_bfloat16> : wkv7_chunk_operator_kernel<float>;
    cudaError_t e = cudaFuncSetAttribute(k1, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem1);
    if (e != cudaSuccess) return (int)e;
    if (!overlap) part = nullptr;
    cudaStream_t op_stream = part ? part->op_stream : stream;
    auto launch_scan = [&](cudaStream_t st, int buf, const float *s_in, float *s_out, int c0, int n) -> cudaError_t {
        const unsigned char *records = ws + lay.records[buf];
        auto go = [&](auto kern, auto ytype, size_t smem_bytes) -> cudaError_t {
            cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes);
            if (err != cudaSuccess) return err;
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3((unsigned)chains);
            cfg.blockDim = dim3((unsigned)kScanThreads);
            cfg.dynamicSmemBytes = smem_bytes;
            cfg.stream = st;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[0].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = attr;
            cfg.numAttrs = st == stream ? 1 : 0;   // directly behind its operator kernel on the caller's stream
            using T = std::remove_pointer_t<decltype(ytype)>;
            err = cudaLaunchKernelEx(&cfg, kern, smaps, optrs, static_cast<const T *>(p.v), records, s_in, s_out,
                                     static_cast<T *>(p.y), (float *)nullptr, (uint32_t *)nullptr, flags, (int)p.T, (int)p.H, c0, n, resolve_flagged ? 1 : 0, status);
            if (err == cudaSuccess) count_launch();
            return err;
        };
        using bf = __nv_bfloat16;
        if (!p.bf16) return go(wkv7_state_scan_kernel<float, kPrefill>, (float *)nullptr, Scan<float>::kBytes);
        return go(wkv7_state_scan_kernel<bf, kPrefill>, (bf *)nullptr, Scan<bf>::kBytes);
    };
    auto launch_operators = [&](int buf, int c0, int n) -> cudaError_t {
        const long long units = (long long)chains * n;
        // (see overlap_applies; on its own partition the kernel fills every SM it has)
        const long long places = part ? 4LL * part->op_sms : overlap ? 4LL * (p.num_sms - (long long)chains) : 4LL * p.num_sms;
        const unsigned grid = (unsigned)(units < places ? units : places);
        // (the operator of (chain, chunk) sits at index chain * n + chunk - c0 of the buffer in both kernels)
        if (!overlap)
            return launch_serialized(k1, grid, (unsigned)kOpThreads, kSmem1, op_stream, omaps, optrs, ws + lay.records[buf], (int)p.T, (int)p.H, c0, n, (int)chains,
                                     wide_range ? 1 : 0, status);
        k1<<<grid, kOpThreads, kSmem1, op_stream>>>(omaps, optrs, ws + lay.records[buf], (int)p.T, (int)p.H, c0, n, (int)chains, wide_range ? 1 : 0, status);
        count_launch();
        return cudaGetLastError();
    };

    if (!overlap) {
        for (int c0 = 0; c0 < nchunks; c0 += (int)seg) {
            const int n = (int)((size_t)(nchunks - c0) < seg ? (size_t)(nchunks - c0) : seg);
            e = launch_operators(0, c0, n);
            if (e != cudaSuccess) return (int)e;
            const bool first = c0 == 0, last = c0 + n >= nchunks;
            e = launch_scan(stream, 0, first ? p.s0 : carry, last ? p.s_out : carry, c0, n);
            if (e != cudaSuccess) return (int)e;
        }
        return 0;
    }
    // Overlapped: operator kernels on the caller's stream (or the stream of the operator partition), scans on the
    // device's second, high-priority stream (or the stream of the scan partition); events order a scan after its
    // operators, and an operator kernel after the scan that last read the buffer it is about to overwrite.
    DeviceStreams *ds = device_streams(p.device);
    if (ds == nullptr) return (int)cudaErrorUnknown;
    cudaStream_t scan_stream = part ? part->scan_stream : ds->side;
    cudaEvent_t *built = part ? part->built : ds->built, *scanned = part ? part->scanned : ds->scanned;
    e = cudaEventRecord(ds->fork, stream);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(scan_stream, ds->fork, 0);
    if (e == cudaSuccess && part) e = cudaStreamWaitEvent(op_stream, ds->fork, 0);
    if (e != cudaSuccess) return (int)e;
    int segment = 0;
    for (int c0 = 0; c0 < nchunks; c0 += (int)seg, ++segment) {
        const int n = (int)((size_t)(nchunks - c0) < seg ? (size_t)(nchunks - c0) : seg);
        const int buf = segment & 1;
        if (segment >= 2) {
            e = cudaStreamWaitEvent(op_stream, scanned[buf], 0);
            if (e != cudaSuccess) return (int)e;
        }
        e = launch_operators(buf, c0, n);
        if (e == cudaSuccess) e = cudaEventRecord(built[buf], op_stream);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(scan_stream, built[buf], 0);
        if (e != cudaSuccess) return (int)e;
        const bool first = c0 == 0, last = c0 + n >= nchunks;
        e = launch_scan(scan_stream, buf, first ? p.s0 : carry, last ? p.s_out : carry, c0, n);
        if (e == cudaSuccess) e = cudaEventRecord(scanned[buf], scan_stream);
        if (e != cudaSuccess) return (int)e;
    }
    // join: the caller's stream continues after the last scan (scans run in order on their stream, and every
    // operator kernel is ordered before the scan of its segment)
    e = cudaStreamWaitEvent(stream, scanned[(segment - 1) & 1], 0);
    return (int)e;
}

// ---- a training step ------------------------------------------------------------------------------
//
// Kept between the passes: [records of all chunks][state in front of every chunk][eight largest magnitudes for each][one int per
// chain]; workspace of the backward pass: the same without records, for the gradient of the state behind every chunk.

namespace {

struct TrainingLayout {
    size_t chains, nchunks, states, flags, total;
};
TrainingLayout training_layout(int64_t B, int64_t T, int64_t H, bool with_records) {
    TrainingLayout l{};
    l.chains = (size_t)(B * H);
    l.nchunks = (size_t)((T + kL - 1) / kL);
    l.states = with_records ? align_up(l.chains * l.nchunks * kRecord) : 0;
    l.flags = l.states + align_up(l.chains * l.nchunks * (kN * kN * sizeof(float) + 32));
    l.total = l.flags + align_up(l.chains * sizeof(int));
    return l;
}

template <int kKind>
int launch_training_scan(const ScanMaps &maps, const OperatorPtrs &ptrs, const void *in, const unsigned char *records, const float *s_in,
                         float *s_out, void *out, float *states, int *flags, const TrainingLayout &l, int64_t T, int64_t H, int *status,
                         cudaStream_t stream) {
    using bf = __nv_bfloat16;
    auto kern = wkv7_state_scan_kernel<bf, kKind>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Scan<bf>::kBytes);
    if (e != cudaSuccess) return (int)e;
    return (int)launch_serialized(kern, (unsigned)l.chains, (unsigned)kScanThreads, Scan<bf>::kBytes, stream, maps, ptrs, static_cast<const bf *>(in), records, s_in,
                                  s_out, static_cast<bf *>(out), states, reinterpret_cast<uint32_t *>(states + l.chains * l.nchunks * kN * kN), flags, (int)T,
                                  (int)H, 0, (int)l.nchunks, 1, status);
}

}  // namespace

bool wkv7_training_supported(int64_t B, int64_t T, int64_t H, int64_t N, bool bf16) {
    return bf16 && N == kN && T >= kL && T % 16 == 0 && B * T < (int64_t(1) << 31) && B * H < (int64_t(1) << 24);
}
size_t wkv7_training_saved_bytes(int64_t B, int64_t T, int64_t H) { return training_layout(B, T, H, true).total; }
size_t wkv7_training_workspace_bytes(int64_t B, int64_t T, int64_t H) { return training_layout(B, T, H, false).total; }

int launch_wkv7_training_forward(const Wkv7Args &p, void *saved, cudaStream_t stream) {
    const TrainingLayout l = training_layout(p.B, p.T, p.H, true);
    unsigned char *base = static_cast<unsigned char *>(saved);
    OperatorMaps omaps{};
    ScanMaps smaps{};
    const OperatorPtrs optrs{{p.a, p.r, p.b, p.k, p.w}};
    for (int i = 0; i < 5; ++i)
        if (!describe_rows(&omaps.m[i], optrs.p[i], p.B, p.T, p.H, true)) return (int)cudaErrorInvalidValue;
    if (!describe_rows(&smaps.v, p.v, p.B, p.T, p.H, true) || !describe_rows(&smaps.y, p.y, p.B, p.T, p.H, true)) return (int)cudaErrorInvalidValue;
    int *status = nullptr;
    if (int e = device_status_ptr(p.device, &status)) return e;
    auto k1 = wkv7_chunk_operator_kernel<__nv_bfloat16>;
    cudaError_t e = cudaFuncSetAttribute(k1, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem1);
    if (e != cudaSuccess) return (int)e;
    const long long units = (long long)(l.chains * l.nchunks), places = 4LL * p.num_sms;
    e = launch_serialized(k1, (unsigned)(units < places ? units : places), (unsigned)kOpThreads, kSmem1, stream, omaps, optrs, base, (int)p.T, (int)p.H, 0,
                          (int)l.nchunks, (int)l.chains, 1, status);
    if (e != cudaSuccess) return (int)e;
    return launch_training_scan<kForTraining>(smaps, optrs, p.v, base, p.s0, p.s_out, p.y, reinterpret_cast<float *>(base + l.states),
                                              reinterpret_cast<int *>(base + l.flags), l, p.T, p.H, status, stream);
}

int launch_wkv7_training_backward(const Wkv7TrainingBackwardArgs &p, const void *saved, void *workspace, cudaStream_t stream) {
    const TrainingLayout ls = training_layout(p.B, p.T, p.H, true), lw = training_layout(p.B, p.T, p.H, false);
    const unsigned char *base = static_cast<const unsigned char *>(saved);
    unsigned char *ws = static_cast<unsigned char *>(workspace);
    float *gradients = reinterpret_cast<float *>(ws + lw.states);
    ScanMaps smaps{};
    const OperatorPtrs optrs{{p.a, p.r, p.b, p.k, p.w}};
    if (!describe_rows(&smaps.v, p.dy, p.B, p.T, p.H, true) || !describe_rows(&smaps.y, p.dv, p.B, p.T, p.H, true)) return (int)cudaErrorInvalidValue;
    int *status = nullptr;
    if (int e = device_status_ptr(p.device, &status)) return e;
    if (int e = launch_training_scan<kGradients>(smaps, optrs, p.dy, base, p.next_state_grad, p.initial_state_grad, p.dv, gradients,
                                                 reinterpret_cast<int *>(ws + lw.flags), lw, p.T, p.H, status, stream))
        return e;
    return launch_wkv7_chunk_gradients(p, base, reinterpret_cast<const float *>(base + ls.states), gradients, stream);
}

}  // namespace rwkv7
