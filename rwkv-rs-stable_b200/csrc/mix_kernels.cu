// Token-shift mixing kernels: mix6, addcmul / addcmul5, token_shift_diff.
//
// All three are pure streaming kernels bound by HBM bandwidth.  A thread owns one
// 16-byte channel vector of every row it takes and keeps the per-channel scales in
// registers; every access is a coalesced 128-bit load or store.  A CTA of addcmul and
// token_shift_diff owns consecutive token rows, and the latter carries the previous
// row in registers (one halo row per CTA is read again).  mix6 moves the whole grid
// over the tensor as a window of neighbouring rows and reads the row in front from
// L2.  Arithmetic is fp32, rounded once on store.
//
// Reference semantics (paths inside the rwkv-rs repository):
//   mix6              crates/rwkv-nn/src/kernels/train/time_mixer/mix6/kernel.rs:25-57
//   addcmul/addcmul5  crates/rwkv-nn/src/kernels/template/addcmul/kernel.rs:4-65
//   token_shift_diff  crates/rwkv-nn/src/kernels/template/token_shift_diff/kernel.rs:16-45
//                     (there one thread walks T serially; here T is parallel and
//                     only the t == 0 row touches the carried state)
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.h"
#include "launch.h"
#include "rwkv7_b200.h"

namespace rwkv7 {
namespace {

// Rows per CTA: 16, or with few rows (a decode step) as few as give every SM two CTAs, since a CTA walks its rows one after the
// other: five scales over 16 rows of 2048 channels took one CTA 10 us.
constexpr int kMostRows = 16;
int rows_per_block(int64_t rows, int num_sms) {
    const int64_t r = rows / (2 * (int64_t)(num_sms > 0 ? num_sms : 1));
    return (int)(r < 1 ? 1 : r < kMostRows ? r : kMostRows);
}

// CTAs of mix6 on an SM.  With one element a thread (odd channel counts, tensors off 16 bytes) two of them have too little in flight:
// 4 x 2049 tokens of 2049 channels, bf16 / fp32 tensors, 140 / 168 us with two, 92 / 124 with four, 68 / 121 with six, 75 / 147 with eight.
template <int EPV>
constexpr int kMixPerSm = EPV == 1 ? 6 : 2;

__host__ __device__ __forceinline__ int64_t imin(int64_t a, int64_t b) { return a < b ? a : b; }

// EPV elements per vector: 8 (bf16, 16 B), 4 (f32, 16 B) or 1 (scalar fallback
// for channel counts or pointers that are not 16-byte aligned).
template <typename T, int EPV>
struct Pack {
    float f[EPV];
    __device__ __forceinline__ void load(const T *p) {
        if constexpr (EPV == 1) {
            f[0] = static_cast<float>(*p);
        } else if constexpr (sizeof(T) == 4) {
            const float4 x = *reinterpret_cast<const float4 *>(p);
            f[0] = x.x; f[1] = x.y; f[2] = x.z; f[3] = x.w;
        } else {
            const uint4 u = *reinterpret_cast<const uint4 *>(p);
            const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                f[2 * i] = __uint_as_float(w[i] << 16);
                f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
            }
        }
    }
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < EPV; ++i) f[i] = 0.f;
    }
    __device__ __forceinline__ void store(T *p) const {
        if constexpr (EPV == 1) {
            if constexpr (sizeof(T) == 4) *p = f[0];
            else *p = __float2bfloat16_rn(f[0]);
        } else if constexpr (sizeof(T) == 4) {
            *reinterpret_cast<float4 *>(p) = make_float4(f[0], f[1], f[2], f[3]);
        } else {
            uint4 u;
            unsigned *w = &u.x;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
                w[i] = *reinterpret_cast<const unsigned *>(&h);
            }
            *reinterpret_cast<uint4 *>(p) = u;
        }
    }
};

// A vector as it lies in memory: bf16 scales take half the registers so, which leaves room for the rows on their way (124 registers, two CTAs an SM).
template <typename T, int EPV>
struct Raw {
    Pack<T, EPV> v;
    __device__ __forceinline__ void load(const T *p) { v.load(p); }
    __device__ __forceinline__ void unpack(Pack<T, EPV> &o) const { o = v; }
};
template <>
struct Raw<__nv_bfloat16, 8> {
    uint4 v;
    __device__ __forceinline__ void load(const __nv_bfloat16 *p) { v = *reinterpret_cast<const uint4 *>(p); }
    __device__ __forceinline__ void unpack(Pack<__nv_bfloat16, 8> &o) {
        // (not hoisted out of the loop over the rows)
        asm volatile("" : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w));
        const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            o.f[2 * i] = __uint_as_float(w[i] << 16);
            o.f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        }
    }
};

struct Mix6Ptrs {
    const void *mu[6];
    void *out[6];
};

// Bound by HBM, six rows written for each that is read.  The grid is a window of neighbouring rows that moves over the tensor, a thread always
// at the same channels of it: with shares of consecutive rows for every CTA the writes went to thousands of places in DRAM at a time.  The row
// in front is read again, from L2; a thread's next two vectors are on their way while it writes six, and the scales stay as they lie in
// memory.  Measured, 4 x 2049 tokens of 2048 channels: 46.5 us (5.05 TB/s) with shares of 14 rows, 40.9 (5.75).
template <typename T, int EPV>
__global__ void __launch_bounds__(256, kMixPerSm<EPV>)
mix6_kernel(const T *__restrict__ x, Mix6Ptrs ptrs, int64_t rows, int64_t Tlen, int64_t C) {
    wait_for_previous();
    let_next_in();
    const unsigned CV = (unsigned)(C / EPV), at = blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t step = gridDim.x * blockDim.x / CV, c = (int64_t)(at % CV) * EPV;   // rows of the window (the grid has a row's threads at least)
    int64_t row = at / CV;
    if (row >= step || row >= rows) return;
    Raw<T, EPV> scale[6];
#pragma unroll
    for (int s = 0; s < 6; ++s) scale[s].load(reinterpret_cast<const T *>(ptrs.mu[s]) + c);
    const int64_t t_step = step % Tlen;
    int64_t t = row % Tlen;
    Raw<T, EPV> ahead, ahead_prev;   // the next row and the one in front of it
    auto request = [&](int64_t row, int64_t t) {
        ahead.load(x + row * C + c);
        if (t > 0) ahead_prev.load(x + (row - 1) * C + c);
    };
    request(row, t);
#pragma unroll 1
    for (; row < rows; row += step) {
        Pack<T, EPV> cur, prev;
        ahead.unpack(cur);
        ahead_prev.unpack(prev);
        if (t == 0) prev.zero();  // first token of a sequence: x_{-1} = 0
        t += t_step;
        if (t >= Tlen) t -= Tlen;
        if (row + step < rows) request(row + step, t);
#pragma unroll
        for (int s = 0; s < 6; ++s) {
            Pack<T, EPV> o, mu;
            scale[s].unpack(mu);
#pragma unroll
            for (int e = 0; e < EPV; ++e)
                o.f[e] = fmaf(prev.f[e] - cur.f[e], mu.f[e], cur.f[e]);
            o.store(reinterpret_cast<T *>(ptrs.out[s]) + row * C + c);
        }
    }
}

struct AddcmulPtrs {
    const void *scale[5];
    void *out[5];
};

template <typename T, int EPV, int NS>
__global__ void __launch_bounds__(256)
addcmul_kernel(const T *base, const T *__restrict__ diff, AddcmulPtrs ptrs, int64_t rows, int64_t C, int per_block) {
    wait_for_previous();
    // The next kernel is not let in early.  Where that is the next call of this one, its CTAs would take the places that are free beside this
    // call's, and lie unevenly over the SMs when their turn comes: 4700 rows of 2049 channels in bf16, each call with an output of its own, 26.0 us so, 42.2 let in at
    // once, 28.7 launched in the ordinary way; 16 000 of 511 9.5, 16.0, 11.8; 3000 of 2048 4.8, 7.5, 6.3; 4800 of 2048 9.1, 11.8, 11.2.
    const int64_t CV = C / EPV;
    const int64_t row_begin = (int64_t)blockIdx.x * per_block;
    const int64_t row_end = imin(rows, row_begin + per_block);
    for (int64_t cv = threadIdx.x; cv < CV; cv += blockDim.x) {
        const int64_t c = cv * EPV;
        Pack<T, EPV> sc[NS];
#pragma unroll
        for (int s = 0; s < NS; ++s) sc[s].load(reinterpret_cast<const T *>(ptrs.scale[s]) + c);
        // five scale vectors already fill 40 registers: a shorter unroll keeps three CTAs per SM
#pragma unroll(NS == 1 ? 4 : 2)
        for (int64_t row = row_begin; row < row_end; ++row) {
            Pack<T, EPV> bs, df;
            if constexpr (NS == 1) {
                bs.load(base + row * C + c);  // `out[0]` may alias `base`: read before write, same thread
            } else {
                // the five outputs never alias the inputs: let loads of later rows pass earlier stores
                const T *__restrict__ base_noalias = base;
                bs.load(base_noalias + row * C + c);
            }
            df.load(diff + row * C + c);
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                Pack<T, EPV> o;
#pragma unroll
                for (int e = 0; e < EPV; ++e) o.f[e] = fmaf(df.f[e], sc[s].f[e], bs.f[e]);
                o.store(reinterpret_cast<T *>(ptrs.out[s]) + row * C + c);
            }
        }
    }
}

__device__ __forceinline__ int64_t load_id(const void *ids, int dtype, int64_t b) {
    if (dtype == RWKV7_I64) return reinterpret_cast<const int64_t *>(ids)[b];
    if (dtype == RWKV7_U32) return (int64_t) reinterpret_cast<const uint32_t *>(ids)[b];
    return (int64_t) reinterpret_cast<const int32_t *>(ids)[b];
}

// `next` == `state`: the carried tokens are updated in place.  Otherwise the CTAs behind those of the sequences write `next`, some slots
// each: the last token of the sequence that names a slot, else what `state` holds.  Each of them reads all ids once, so there
// are no more than four per SM, but for kMostSlots slots each, and then a warp copies a slot.
constexpr int kMostSlots = 256;
template <typename T, int EPV>
__global__ void __launch_bounds__(256)
token_shift_diff_kernel(const T *__restrict__ x, const T *state, T *next, const void *__restrict__ ids, int ids_dtype,
                        T *__restrict__ diff, int64_t B, int64_t Tlen, int64_t C, int64_t S, int per_block, int slots_per_block, int *status) {
    wait_for_previous();
    if constexpr (EPV > 1) let_next_in();   // (one element a thread: as in addcmul_kernel, 4700 tokens of 2049 channels 19.6 us, 22.1 let in at once)
    const int64_t CV = C / EPV;
    const int64_t blocks_per_seq = (Tlen + per_block - 1) / per_block;
    if (blockIdx.x >= B * blocks_per_seq) {
        const int64_t slot0 = (blockIdx.x - B * blocks_per_seq) * slots_per_block;
        const int slots = (int)imin(slots_per_block, S - slot0);
        __shared__ int named_by[kMostSlots];
        for (int s = threadIdx.x; s < slots; s += blockDim.x) named_by[s] = -1;
        __syncthreads();
        for (int64_t b0 = threadIdx.x; b0 < B; b0 += 8 * blockDim.x) {
            int64_t s[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) s[u] = b0 + u * blockDim.x < B ? load_id(ids, ids_dtype, b0 + u * blockDim.x) - slot0 : -1;
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (s[u] >= 0 && s[u] < slots) atomicMax(&named_by[s[u]], (int)(b0 + u * blockDim.x));
        }
        __syncthreads();
        const int threads = slots == 1 ? blockDim.x : 32;   // of a slot
        const int first = slots == 1 ? threadIdx.x : threadIdx.x & 31;
        for (int s = slots == 1 ? 0 : threadIdx.x >> 5; s < slots; s += blockDim.x >> 5) {
            const T *from = named_by[s] < 0 ? state + (slot0 + s) * C : x + ((int64_t)named_by[s] * Tlen + Tlen - 1) * C;
            T *to = next + (slot0 + s) * C;
            for (int64_t c0 = first; c0 < CV; c0 += 4 * threads) {
                Pack<T, EPV> v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (c0 + u * threads < CV) v[u].load(from + (c0 + u * threads) * EPV);
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (c0 + u * threads < CV) v[u].store(to + (c0 + u * threads) * EPV);
            }
        }
        return;
    }
    const int64_t b = blockIdx.x / blocks_per_seq;
    const int64_t t_begin = (blockIdx.x % blocks_per_seq) * per_block;
    const int64_t t_end = imin(Tlen, t_begin + per_block);
    const int64_t slot = load_id(ids, ids_dtype, b);
    const bool slot_ok = slot >= 0 && slot < S;
    if (!slot_ok && threadIdx.x == 0 && t_begin == 0) atomicExch(status, (int)kDevBadIndex);
    const T *xb = x + b * Tlen * C;
    T *db = diff + b * Tlen * C;
    for (int64_t cv = threadIdx.x; cv < CV; cv += blockDim.x) {
        const int64_t c = cv * EPV;
        Pack<T, EPV> prev;
        if (t_begin == 0) {
            if (slot_ok) prev.load(state + slot * C + c);
            else prev.zero();
        } else {
            prev.load(xb + (t_begin - 1) * C + c);
        }
#pragma unroll 4
        for (int64_t t = t_begin; t < t_end; ++t) {
            Pack<T, EPV> cur, o;
            cur.load(xb + t * C + c);
#pragma unroll
            for (int e = 0; e < EPV; ++e) o.f[e] = prev.f[e] - cur.f[e];
            o.store(db + t * C + c);
            prev = cur;
        }
        // In place the thread that read the carried token of this (slot, channel vector) is the only one that
        // overwrites it, after its read.
        if (t_begin == 0 && slot_ok && next == state) {
            Pack<T, EPV> last;
            if (t_end == Tlen) last = prev;
            else last.load(xb + (Tlen - 1) * C + c);
            last.store(next + slot * C + c);
        }
    }
}

inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

inline int pick_threads(int64_t CV) {
    int t = 32;
    while (t < 256 && t < CV) t <<= 1;
    return t;
}

template <typename First, typename... Rest>
First first_parameter(void (*)(First, Rest...));

}  // namespace

int launch_mix6(const MixArgs &p, cudaStream_t stream) {
    const int64_t rows = p.B * p.T;
    if (rows == 0 || p.C == 0) return 0;
    Mix6Ptrs ptrs;
    bool vec_ok = aligned16(p.x);
    for (int s = 0; s < 6; ++s) {
        ptrs.mu[s] = p.mu[s];
        ptrs.out[s] = p.out[s];
        vec_ok = vec_ok && aligned16(p.mu[s]) && aligned16(p.out[s]);
    }
    auto go = [&](auto kernel, int per_sm, int64_t vectors) {
        // so many CTAs an SM, or as many as there are vectors, and a row's at least
        const int64_t most = (rows * vectors + 255) / 256, fill = std::max<int64_t>(per_sm * (int64_t)(p.num_sms > 0 ? p.num_sms : 1), (vectors + 255) / 256);
        return (int)launch_serialized(kernel, (unsigned)imin(most, fill), 256u, 0, stream, (decltype(first_parameter(kernel)))p.x, ptrs, rows, p.T, p.C);
    };
    using bf = __nv_bfloat16;
    if (p.bf16) return vec_ok && p.C % 8 == 0 ? go(mix6_kernel<bf, 8>, kMixPerSm<8>, p.C / 8) : go(mix6_kernel<bf, 1>, kMixPerSm<1>, p.C);
    return vec_ok && p.C % 4 == 0 ? go(mix6_kernel<float, 4>, kMixPerSm<4>, p.C / 4) : go(mix6_kernel<float, 1>, kMixPerSm<1>, p.C);
}

template <typename T, int EPV>
static cudaError_t launch_addcmul_t(const AddcmulArgs &p, const AddcmulPtrs &ptrs, cudaStream_t stream) {
    const int threads = pick_threads(p.C / EPV), per = rows_per_block(p.rows, p.num_sms);
    const unsigned grid = (unsigned)((p.rows + per - 1) / per);
    return launch_serialized(p.nscale == 1 ? addcmul_kernel<T, EPV, 1> : addcmul_kernel<T, EPV, 5>, grid, (unsigned)threads, 0, stream, (const T *)p.base,
                             (const T *)p.diff, ptrs, p.rows, p.C, per);
}

int launch_addcmul(const AddcmulArgs &p, cudaStream_t stream) {
    if (p.rows == 0 || p.C == 0) return 0;
    AddcmulPtrs ptrs{};
    bool vec_ok = aligned16(p.base) && aligned16(p.diff);
    for (int s = 0; s < p.nscale; ++s) {
        ptrs.scale[s] = p.scale[s];
        ptrs.out[s] = p.out[s];
        vec_ok = vec_ok && aligned16(p.scale[s]) && aligned16(p.out[s]);
    }
    using bf = __nv_bfloat16;
    if (p.bf16) return (int)(vec_ok && p.C % 8 == 0 ? launch_addcmul_t<bf, 8>(p, ptrs, stream) : launch_addcmul_t<bf, 1>(p, ptrs, stream));
    return (int)(vec_ok && p.C % 4 == 0 ? launch_addcmul_t<float, 4>(p, ptrs, stream) : launch_addcmul_t<float, 1>(p, ptrs, stream));
}

template <typename T, int EPV>
static cudaError_t launch_token_shift_t(const TokenShiftArgs &p, cudaStream_t stream) {
    const int per = rows_per_block(p.B * p.T, p.num_sms);
    const int64_t fair = p.S / (4 * (int64_t)(p.num_sms > 0 ? p.num_sms : 1));
    const int slots = (int)(fair < 1 ? 1 : imin(fair, kMostSlots));
    const int threads = slots == 1 ? pick_threads(p.C / EPV) : 256;
    const int64_t blocks = p.B * ((p.T + per - 1) / per) + (p.next != p.state ? (p.S + slots - 1) / slots : 0);
    return launch_serialized(token_shift_diff_kernel<T, EPV>, (unsigned)blocks, (unsigned)threads, 0, stream, (const T *)p.x, (const T *)p.state, (T *)p.next,
                             p.ids, p.ids_dtype, (T *)p.diff, p.B, p.T, p.C, p.S, per, slots, p.status);
}

int launch_token_shift_diff(const TokenShiftArgs &p, cudaStream_t stream) {
    if (p.B == 0 || p.T == 0 || p.C == 0) return 0;  // T == 0: diff empty, state unchanged
    const bool vec_ok = aligned16(p.x) && aligned16(p.state) && aligned16(p.next) && aligned16(p.diff);
    using bf = __nv_bfloat16;
    if (p.bf16) return (int)(vec_ok && p.C % 8 == 0 ? launch_token_shift_t<bf, 8>(p, stream) : launch_token_shift_t<bf, 1>(p, stream));
    return (int)(vec_ok && p.C % 4 == 0 ? launch_token_shift_t<float, 4>(p, stream) : launch_token_shift_t<float, 1>(p, stream));
}

}  // namespace rwkv7
