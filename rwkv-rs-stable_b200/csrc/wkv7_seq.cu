// Sequential WKV7 scan and decode sweep.
//
// Semantics: crates/rwkv-nn/src/kernels/train/time_mixer/wkv7/mod.rs:179-242 of
// the reference (per token: sa = S a; S = S diag(d) + sa b^T + v k^T; y = S r,
// d = exp(-exp(w))).  Unlike the reference kernel (kernel.rs:82-195), which
// re-reads its state row from global memory every token, the fp32 state here
// stays in registers for the whole call and is read from / written to HBM once.
//
// N == 64: a CTA owns ROWS value rows of one (b,h); 4 threads share a row, each
// holding 16 key columns (interleaved in groups of 4 so that the per-token
// vectors are read from shared memory with conflict-free 128-bit loads).  Token
// vectors are staged 16 tokens at a time through a double-buffered shared tile,
// converted to fp32 once (decay computed once per element).
// Any other N <= 128: one thread per row, state in shared memory.
//
// Bound by the chain from one token's state to the next with few chains (0.21 us a token: eight multiply-adds deep, two shuffles,
// the update) and by shared memory and the packed multiply-adds with many.  Measured (B200), fp32, 511 tokens: 32 chains 108
// us, 1600 chains 900 us (with a row per thread throughout and the output summed in the chain: 191 and 2385).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdlib>

#include "kernels.h"
#include "launch.h"

namespace rwkv7 {
namespace {

constexpr int kN = 64;
// Tokens staged per shared tile; fewer where a thread has several rows, so that more CTAs fit an SM.
__host__ __device__ constexpr int seq_tile(int rows_per_thread) { return rows_per_thread == 1 ? 16 : 8; }
constexpr size_t seq_smem(int rows, int rows_per_thread) {
    return sizeof(float) * (size_t)(2 * seq_tile(rows_per_thread) * 6 * 64 + 4 * seq_tile(rows_per_thread) * rows);
}

enum { VR = 0, VD = 1, VK = 2, VV = 3, VA = 4, VB = 5 };

struct SeqPtrs {
    const void *in[6];  // r, w, k, v, a, b
};

template <typename T>
struct Vec16;
template <>
struct Vec16<float> {
    static constexpr int kElems = 4;
    static __device__ __forceinline__ void unpack(const uint4 &u, float *f) {
        f[0] = __uint_as_float(u.x);
        f[1] = __uint_as_float(u.y);
        f[2] = __uint_as_float(u.z);
        f[3] = __uint_as_float(u.w);
    }
};
template <>
struct Vec16<__nv_bfloat16> {
    static constexpr int kElems = 8;
    static __device__ __forceinline__ void unpack(const uint4 &u, float *f) {
        const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            f[2 * i] = __uint_as_float(w[i] << 16);
            f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        }
    }
};

template <typename T>
__device__ __forceinline__ T from_f32(float x);
template <>
__device__ __forceinline__ float from_f32<float>(float x) { return x; }
template <>
__device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float x) {
    return __float2bfloat16_rn(x);
}

// Tensors a training forward saves for the backward pass (wkv7/forward.rs:368-375):
// snapshots [B,H,T/chunk_len,N,N] = the state after the last token of every chunk (fp32 here),
// state_replacement [B,T,H,N] = sa_t = S_{t-1} a_t, in the sequence dtype.
struct SavePtrs {
    float *snapshots;
    void *state_replacement;
    int chunk_len;
};

// ROWS value rows per CTA, RPT of them per group of four threads (RPT 1, 2 or 4).
template <typename T, int ROWS, int RPT = 1, bool SAVE = false>
__global__ void __launch_bounds__(ROWS / RPT * 4)
wkv7_seq64_kernel(SeqPtrs ptrs, const float *s0, T *__restrict__ y,
                  float *s_out, int Tlen, int H, const int *__restrict__ flags, SavePtrs save = SavePtrs{}) {
    constexpr int THREADS = ROWS / RPT * 4, GROUPS = THREADS / 4;
    constexpr int SPLITS = kN / ROWS;
    constexpr int kTile = seq_tile(RPT);
    // fp32 tensors land in shared memory as they are where registers are short.  (With a row per thread the registers a tile
    // passes through cost nothing, and the compiler then keeps more of a token's loads ahead of its sums: 125 against 146 us at 511 tokens x 32 heads.)
    constexpr bool kDirect = sizeof(T) == 4 && RPT > 1;
    constexpr int EPV = Vec16<T>::kElems;
    constexpr int VPR = kN / EPV;                 // 16-byte vectors per token row
    constexpr int VECS = kTile * 6 * VPR;         // vectors per tile
    constexpr int NV = (VECS + THREADS - 1) / THREADS;
    static_assert(RPT == 1 || !SAVE, "the saving variant has a row per thread");

    extern __shared__ __align__(16) unsigned char smem_raw[];
    float *vec = reinterpret_cast<float *>(smem_raw);             // [2][kTile][6][kN]
    float *ytile = vec + 2 * kTile * 6 * kN;                      // [2][kTile][ROWS]
    float *satile = ytile + 2 * kTile * ROWS;                     // [2][kTile][ROWS], SAVE only

    const int bh = blockIdx.x / SPLITS;
    // Fallback mode: only the chains another kernel flagged are (re)computed.
    // (launched behind the kernel in front of it, which writes the flags, possibly before that has finished; a no-op for an ordinary launch)
    wait_for_previous();
    // The kernel behind is not let in early: the next call's CTAs would take the places that are free beside this one's, which
    // need not be where its load is even (short calls back to back: 12 tokens x 264 chains 7.7 us so, 10.5 let in at once, 9.4 launched in the ordinary way; 16 x 84
    // 7.1 / 8.8 / 8.6; fp32 22 x 80 9.7 / 12.2 / 12.4; 45 x 896 64.4 / 64.4 / 66.1).
    if (flags != nullptr) {
        // (Nor behind the pass over flagged chains: there may come the next call's operator kernel, four CTAs of 57 KB to an SM.  Those that
        // start beside CTAs of this kernel lie unevenly for as long as they run: 3 x 2047 tokens x 32 heads 98.7 -> 105.3 us, 113 where an SM that
        // holds CTAs of this kernel keeps a smaller share of its memory as shared memory; 8 x 4096 x 12 166 -> 181.)
        if (flags[bh] == 0) return;
    }
    const int split = blockIdx.x % SPLITS;
    const int bi = bh / H, h = bh % H;
    const int row0 = split * ROWS;
    const int tid = threadIdx.x;
    const int i0 = tid >> 2, q = tid & 3;         // rows i0 + m GROUPS

    float2 S[RPT][4][2];   // columns 16 kk + 4 q + {0, 1}, {2, 3}
#pragma unroll
    for (int m = 0; m < RPT; ++m)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
            if (s0 != nullptr) x = reinterpret_cast<const float4 *>(s0 + ((size_t)bh * kN + row0 + i0 + m * GROUPS) * kN)[kk * 4 + q];
            S[m][kk][0] = make_float2(x.x, x.y);
            S[m][kk][1] = make_float2(x.z, x.w);
        }

    const size_t seq_base = ((size_t)bi * Tlen * H + h) * kN;  // element offset of (b, t=0, h, 0)
    const size_t tok_stride = (size_t)H * kN;
    const int ntiles = (Tlen + kTile - 1) / kTile;

    // Vectors of a tile in the order (tensor, token, piece): a thread's n-th is of a tensor known at compile time (or uniform for
    // its warp).
    uint4 stage[kDirect ? 1 : NV];
    auto place = [&](int n, int &c, int &tok, int &tensor) {
        const int idx = tid + n * THREADS;
        c = idx % VPR;
        tok = idx / VPR % kTile;
        tensor = idx / (VPR * kTile);
        return idx < VECS;
    };
    auto issue_loads = [&](int tile) {
#pragma unroll
        for (int n = 0; n < NV; ++n) {
            int c, tok, tensor;
            const bool mine = place(n, c, tok, tensor);
            const int t = tile * kTile + tok;
            if constexpr (!kDirect) stage[n] = make_uint4(0, 0, 0, 0);
            if (mine && t < Tlen) {
                const T *p = reinterpret_cast<const T *>(ptrs.in[tensor]) + seq_base + (size_t)t * tok_stride + c * EPV;
                if constexpr (kDirect) {
                    const unsigned dst = (unsigned)__cvta_generic_to_shared(vec + (((size_t)(tile & 1) * kTile + tok) * 6 + tensor) * kN + c * EPV);
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(p) : "memory");
                } else {
                    stage[n] = __ldg(reinterpret_cast<const uint4 *>(p));
                }
            }
        }
    };
    auto commit_stage = [&](int buf) {
        if constexpr (kDirect) asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
        for (int n = 0; n < NV; ++n) {
            int c, tok, tensor;
            if (place(n, c, tok, tensor) && (!kDirect || tensor == VD)) {   // (a thread converts what it fetched itself)
                float4 *dst = reinterpret_cast<float4 *>(vec + (((size_t)buf * kTile + tok) * 6 + tensor) * kN + c * EPV);
                float f[EPV];
                if constexpr (kDirect) {
                    const float4 x = *dst;
                    f[0] = x.x; f[1] = x.y; f[2] = x.z; f[3] = x.w;
                } else {
                    Vec16<T>::unpack(stage[n], f);
                }
                if (tensor == VD) {
#pragma unroll
                    for (int e = 0; e < EPV; ++e) f[e] = expf(-expf(f[e]));
                }
#pragma unroll
                for (int e = 0; e < EPV / 4; ++e) dst[e] = make_float4(f[4 * e], f[4 * e + 1], f[4 * e + 2], f[4 * e + 3]);
            }
        }
    };

    issue_loads(0);
    commit_stage(0);
    __syncthreads();

    for (int tile = 0; tile < ntiles; ++tile) {
        const int buf = tile & 1;
        if (tile + 1 < ntiles) issue_loads(tile + 1);
        const int ntok = min(kTile, Tlen - tile * kTile);
        const float *tv = vec + (size_t)buf * kTile * 6 * kN;
        float *yt = ytile + (size_t)buf * kTile * ROWS;
        float *sat = satile + (size_t)buf * kTile * ROWS;

        // (the removal key of the next token is fetched while this one's is used, which takes its latency out of the chain from state
        // to state: 125 -> 108 us at 511 fp32 tokens x 32 heads; fetching the other vectors as early cost registers, 117.  Behind a
        // tile's last token it reads what follows the tile and nobody uses it.)
        float4 ahead[4];
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) ahead[kk] = reinterpret_cast<const float4 *>(tv + VA * kN)[kk * 4 + q];
        // One token: the step of the state; this thread's parts of y.  (Packed multiply-adds: the sums are those of single ones.)
        auto step = [&](int tt, float (&part)[RPT]) {
            const float *base = tv + (size_t)tt * 6 * kN;
            auto vec4 = [&](int x, int kk) { return reinterpret_cast<const float4 *>(base + x * kN)[kk * 4 + q]; };
            float2 s01[RPT], s23[RPT], sa[RPT], vi[RPT], y01[RPT], y23[RPT];
#pragma unroll
            for (int m = 0; m < RPT; ++m) s01[m] = s23[m] = y01[m] = y23[m] = make_float2(0.f, 0.f);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                const float4 x = ahead[kk];
                ahead[kk] = vec4(6 + VA, kk);   // the next token's
#pragma unroll
                for (int m = 0; m < RPT; ++m) {
                    s01[m] = __ffma2_rn(S[m][kk][0], make_float2(x.x, x.y), s01[m]);
                    s23[m] = __ffma2_rn(S[m][kk][1], make_float2(x.z, x.w), s23[m]);
                }
            }
#pragma unroll
            for (int m = 0; m < RPT; ++m) {
                float sum = (s01[m].x + s01[m].y) + (s23[m].x + s23[m].y);
                sum += __shfl_xor_sync(0xffffffffu, sum, 1);
                sum += __shfl_xor_sync(0xffffffffu, sum, 2);
                if constexpr (SAVE) {
                    if (q == 0) sat[tt * ROWS + i0] = sum;
                }
                const float v = base[VV * kN + row0 + i0 + m * GROUPS];
                sa[m] = make_float2(sum, sum);
                vi[m] = make_float2(v, v);
            }
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                const float4 d = vec4(VD, kk), b = vec4(VB, kk), k = vec4(VK, kk), r = vec4(VR, kk);
#pragma unroll
                for (int m = 0; m < RPT; ++m) {
                    float2 &s0 = S[m][kk][0], &s1 = S[m][kk][1];
                    s0 = __ffma2_rn(s0, make_float2(d.x, d.y), __ffma2_rn(sa[m], make_float2(b.x, b.y), __fmul2_rn(vi[m], make_float2(k.x, k.y))));
                    s1 = __ffma2_rn(s1, make_float2(d.z, d.w), __ffma2_rn(sa[m], make_float2(b.z, b.w), __fmul2_rn(vi[m], make_float2(k.z, k.w))));
                    y01[m] = __ffma2_rn(s0, make_float2(r.x, r.y), y01[m]);
                    y23[m] = __ffma2_rn(s1, make_float2(r.z, r.w), y23[m]);
                }
            }
            if constexpr (SAVE) {
                const int t = tile * kTile + tt;
                if ((t + 1) % save.chunk_len == 0) {   // state after the last token of a chunk
                    const int chunk = t / save.chunk_len, nchunks = Tlen / save.chunk_len;
                    float4 *dst = reinterpret_cast<float4 *>(
                        save.snapshots + (((size_t)bh * nchunks + chunk) * kN + row0 + i0) * kN);
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk) dst[kk * 4 + q] = make_float4(S[0][kk][0].x, S[0][kk][0].y, S[0][kk][1].x, S[0][kk][1].y);
                }
            }
#pragma unroll
            for (int m = 0; m < RPT; ++m) part[m] = (y01[m].x + y01[m].y) + (y23[m].x + y23[m].y);
        };
        // Four outputs at a time (of 4 / RPT tokens) are summed over the four lanes of a row group together: lane q ends up with
        // the q-th, by the additions a sum of its own would have.  With a row per thread nothing but the state's own chain then
        // lies between one token and the next three.
        constexpr int TOKENS = 4 / RPT;
        int tt = 0;
        for (; tt + TOKENS <= ntok; tt += TOKENS) {
            float part[TOKENS][RPT];
#pragma unroll
            for (int u = 0; u < TOKENS; ++u) step(tt + u, part[u]);
            const float p0 = part[0][0], p1 = part[1 / RPT][1 % RPT], p2 = part[2 / RPT][2 % RPT], p3 = part[3 / RPT][3 % RPT];
            const bool odd = q & 1, high = q & 2;
            const float r0 = (odd ? p1 : p0) + __shfl_xor_sync(0xffffffffu, odd ? p0 : p1, 1);
            const float r1 = (odd ? p3 : p2) + __shfl_xor_sync(0xffffffffu, odd ? p2 : p3, 1);
            yt[(tt + q / RPT) * ROWS + i0 + q % RPT * GROUPS] = (high ? r1 : r0) + __shfl_xor_sync(0xffffffffu, high ? r0 : r1, 2);
        }
        for (; tt < ntok; ++tt) {
            float part[RPT];
            step(tt, part);
#pragma unroll
            for (int m = 0; m < RPT; ++m) {
                part[m] += __shfl_xor_sync(0xffffffffu, part[m], 1);
                part[m] += __shfl_xor_sync(0xffffffffu, part[m], 2);
                if (q == 0) yt[tt * ROWS + i0 + m * GROUPS] = part[m];
            }
        }

        if (tile + 1 < ntiles) commit_stage(buf ^ 1);
        __syncthreads();
        for (int idx = tid; idx < ntok * ROWS; idx += THREADS) {
            const int tt = idx / ROWS, rr = idx % ROWS;
            const size_t o = seq_base + (size_t)(tile * kTile + tt) * tok_stride + row0 + rr;
            y[o] = from_f32<T>(yt[tt * ROWS + rr]);
            if constexpr (SAVE) reinterpret_cast<T *>(save.state_replacement)[o] = from_f32<T>(sat[tt * ROWS + rr]);
        }
    }

    if (s_out != nullptr) {
#pragma unroll
        for (int m = 0; m < RPT; ++m) {
            float4 *dst = reinterpret_cast<float4 *>(s_out + ((size_t)bh * kN + row0 + i0 + m * GROUPS) * kN);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) dst[kk * 4 + q] = make_float4(S[m][kk][0].x, S[m][kk][0].y, S[m][kk][1].x, S[m][kk][1].y);
        }
    }
}

// Any head size N <= 128: thread i owns state row i, kept in shared memory with
// a padded row pitch; the six token vectors are staged per token.
template <typename T, bool SAVE = false>
__global__ void wkv7_seq_generic_kernel(SeqPtrs ptrs, const float *s0,
                                        T *__restrict__ y, float *s_out, int Tlen,
                                        int H, int N, SavePtrs save = SavePtrs{}) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int pitch = N + 1;
    float *S = reinterpret_cast<float *>(smem_raw);  // [N][N+1]
    float *vec = S + (size_t)N * pitch;              // [6][N]
    const int bh = blockIdx.x;
    const int bi = bh / H, h = bh % H;
    const int tid = threadIdx.x;

    for (int idx = tid; idx < N * N; idx += blockDim.x) {
        const int i = idx / N, j = idx % N;
        S[i * pitch + j] = s0 ? s0[(size_t)bh * N * N + idx] : 0.f;
    }
    const size_t seq_base = ((size_t)bi * Tlen * H + h) * N;
    const size_t tok_stride = (size_t)H * N;
    __syncthreads();
    for (int t = 0; t < Tlen; ++t) {
        const size_t o = seq_base + (size_t)t * tok_stride;
        for (int idx = tid; idx < 6 * N; idx += blockDim.x) {
            const int tensor = idx / N, j = idx % N;
            float x = static_cast<float>(reinterpret_cast<const T *>(ptrs.in[tensor])[o + j]);
            if (tensor == VD) x = expf(-expf(x));
            vec[idx] = x;
        }
        __syncthreads();
        if (tid < N) {
            float *Si = S + tid * pitch;
            float sa = 0.f;
            for (int j = 0; j < N; ++j) sa = fmaf(Si[j], vec[VA * N + j], sa);
            const float vi = vec[VV * N + tid];
            float acc = 0.f;
            for (int j = 0; j < N; ++j) {
                const float s = fmaf(Si[j], vec[VD * N + j], fmaf(sa, vec[VB * N + j], vi * vec[VK * N + j]));
                Si[j] = s;
                acc = fmaf(s, vec[VR * N + j], acc);
            }
            y[o + tid] = from_f32<T>(acc);
            if constexpr (SAVE) {
                reinterpret_cast<T *>(save.state_replacement)[o + tid] = from_f32<T>(sa);
                if ((t + 1) % save.chunk_len == 0) {
                    float *dst = save.snapshots +
                                 (((size_t)bh * (Tlen / save.chunk_len) + t / save.chunk_len) * N + tid) * N;
                    for (int j = 0; j < N; ++j) dst[j] = Si[j];
                }
            }
        }
        __syncthreads();
    }
    if (s_out != nullptr)
        for (int idx = tid; idx < N * N; idx += blockDim.x) {
            const int i = idx / N, j = idx % N;
            s_out[(size_t)bh * N * N + idx] = S[i * pitch + j];
        }
}

template <typename T, int ROWS, int RPT>
int launch_seq64(const Wkv7Args &p, cudaStream_t stream, const int *flags = nullptr) {
    SeqPtrs ptrs{{p.r, p.w, p.k, p.v, p.a, p.b}};
    constexpr size_t smem = seq_smem(ROWS, RPT);
    constexpr unsigned threads = ROWS / RPT * 4;
    auto kern = wkv7_seq64_kernel<T, ROWS, RPT, false>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    // (as many CTAs on an SM as its shared memory holds: 19 tokens x 108 chains of fp32 tensors 8.3 -> 7.7 us back to back)
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return (int)e;
    const unsigned grid = (unsigned)(p.B * p.H * (kN / ROWS));
    return (int)launch_serialized(kern, grid, threads, smem, stream, ptrs, p.s0, reinterpret_cast<T *>(p.y), p.s_out, (int)p.T, (int)p.H, flags, SavePtrs{});
}

template <typename T>
int launch_seq(const Wkv7Args &p, cudaStream_t stream) {
    if (p.N == kN) {
        // Rows of S never interact.  A token's five column vectors cost a warp 84 wavefronts of shared memory however many
        // rows its threads have: 672 cycles of an SM per chain and token with a row per thread, 336 with two, 168 with
        // four.  The chain of one token to the next takes about 400, so threads take as few rows as keep an SM's
        // chains below that, and a chain is spread over as many CTAs as that leaves.
        const int64_t chains = p.B * p.H;
        if (chains * 5 <= 3 * (int64_t)p.num_sms) return launch_seq64<T, 16, 1>(p, stream);
        if (chains * 5 <= 6 * (int64_t)p.num_sms) return launch_seq64<T, 32, 2>(p, stream);
        return launch_seq64<T, 64, 4>(p, stream);
    }
    SeqPtrs ptrs{{p.r, p.w, p.k, p.v, p.a, p.b}};
    const int N = (int)p.N;
    const size_t smem = sizeof(float) * ((size_t)N * (N + 1) + 6 * N);
    auto kern = wkv7_seq_generic_kernel<T, false>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    const int threads = ((N + 31) / 32) * 32;
    kern<<<(unsigned)(p.B * p.H), threads, smem, stream>>>(ptrs, p.s0, reinterpret_cast<T *>(p.y),
                                                          p.s_out, (int)p.T, (int)p.H, N, SavePtrs{});
    count_launch();
    return (int)cudaGetLastError();
}

// Training forward: the scan above, also writing the tensors the backward pass needs.
template <typename T>
int launch_seq_saved(const Wkv7Args &p, float *snapshots, void *state_replacement, int chunk_len,
                     cudaStream_t stream) {
    SeqPtrs ptrs{{p.r, p.w, p.k, p.v, p.a, p.b}};
    SavePtrs save{snapshots, state_replacement, chunk_len};
    if (p.N == kN) {
        constexpr int ROWS = 16;   // four CTAs per chain: rows of S never interact
        const size_t smem = seq_smem(ROWS, 1);
        auto kern = wkv7_seq64_kernel<T, ROWS, 1, true>;
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        kern<<<(unsigned)(p.B * p.H * (kN / ROWS)), ROWS * 4, smem, stream>>>(
            ptrs, p.s0, reinterpret_cast<T *>(p.y), p.s_out, (int)p.T, (int)p.H, nullptr, save);
    } else {
        const int N = (int)p.N;
        const size_t smem = sizeof(float) * ((size_t)N * (N + 1) + 6 * N);
        auto kern = wkv7_seq_generic_kernel<T, true>;
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        kern<<<(unsigned)(p.B * p.H), ((N + 31) / 32) * 32, smem, stream>>>(
            ptrs, p.s0, reinterpret_cast<T *>(p.y), p.s_out, (int)p.T, (int)p.H, N, save);
    }
    count_launch();
    return (int)cudaGetLastError();
}

}  // namespace

int launch_wkv7_forward_saved(const Wkv7Args &p, float *snapshots, void *state_replacement, int chunk_len,
                              cudaStream_t stream) {
    return p.bf16 ? launch_seq_saved<__nv_bfloat16>(p, snapshots, state_replacement, chunk_len, stream)
                  : launch_seq_saved<float>(p, snapshots, state_replacement, chunk_len, stream);
}

// N == 64 only: the flagged chains again, with the saved tensors of the training forward.
int launch_wkv7_sequential_flagged_saved(const Wkv7Args &p, const int *flags, float *snapshots,
                                         void *state_replacement, int chunk_len, cudaStream_t stream) {
    SeqPtrs ptrs{{p.r, p.w, p.k, p.v, p.a, p.b}};
    SavePtrs save{snapshots, state_replacement, chunk_len};
    constexpr int ROWS = 16;
    const size_t smem = seq_smem(ROWS, 1);
    const unsigned grid = (unsigned)(p.B * p.H * (kN / ROWS));
    cudaError_t e;
    if (p.bf16) {
        auto kern = wkv7_seq64_kernel<__nv_bfloat16, ROWS, 1, true>;
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        kern<<<grid, ROWS * 4, smem, stream>>>(ptrs, p.s0, reinterpret_cast<__nv_bfloat16 *>(p.y), p.s_out, (int)p.T,
                                               (int)p.H, flags, save);
    } else {
        auto kern = wkv7_seq64_kernel<float, ROWS, 1, true>;
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        kern<<<grid, ROWS * 4, smem, stream>>>(ptrs, p.s0, reinterpret_cast<float *>(p.y), p.s_out, (int)p.T, (int)p.H,
                                               flags, save);
    }
    count_launch();
    return (int)cudaGetLastError();
}

// N == 64 only: recomputes the chains with flags[b*H+h] != 0, 16 value rows per CTA.
int launch_wkv7_sequential_flagged(const Wkv7Args &p, const int *flags, cudaStream_t stream) {
    return p.bf16 ? launch_seq64<__nv_bfloat16, 16, 1>(p, stream, flags) : launch_seq64<float, 16, 1>(p, stream, flags);
}

int launch_wkv7_sequential(const Wkv7Args &p, cudaStream_t stream) {
    // A handful of tokens per chain is the decode case: the state sweep dominates.
    if (p.N == kN && p.T <= 4) return launch_wkv7_decode(p, stream);
    return p.bf16 ? launch_seq<__nv_bfloat16>(p, stream) : launch_seq<float>(p, stream);
}

}  // namespace rwkv7
