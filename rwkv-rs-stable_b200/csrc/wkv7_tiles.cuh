// What the tensor-core kernels of a 64-token chunk share: tiles of [64][64] 16-bit elements and 16 x 16 blocks in shared
// memory, the lane addresses of matrix loads on them, and the arithmetic of the decays.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "sm100_mma.cuh"
#include "sm100_umma.cuh"

namespace rwkv7 {
namespace sm100 {

constexpr int kN = 64;   // head size
constexpr int kL = 64;   // tokens per chunk
constexpr float kBlockDecay = 6.144212e-6f;   // e^-12: a block below it (or a NaN) marks the chunk
constexpr uint32_t kPanel = 8192;             // one [64][64] 16-bit tile, 128-byte rows, 16-byte pieces XOR-ed with (row & 7)
constexpr uint32_t kBlk = 512;                // one 16 x 16 fp16 block: two halves of 8 columns, each [16 rows][16 bytes]

__device__ __forceinline__ uint32_t off16(int row, int col) {
    return (uint32_t)row * 128u + ((((uint32_t)col >> 3) ^ ((uint32_t)row & 7u)) << 4) + ((uint32_t)col & 7u) * 2u;
}
__device__ __forceinline__ float2 unpack_bf2(uint32_t u) {
    return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}

// Lane addresses of ldmatrix.x4 for a 16 x 16 block, as byte offsets.  In a swizzled tile the block starts at (row0,
// column 16 c); in a compact block the rows are 16 bytes and the halves 256.  "plain" gives A order; "cols" swaps the
// two middle matrices: B order for a block stored [column][k], and, with .trans, A order of the transposed block.
// (row0 is a multiple of eight, so the swizzle depends on the lane alone and the column block is one exclusive or.)
__device__ __forceinline__ uint32_t tile_plain(int lane, int row0, int c) {
    const uint32_t own = (uint32_t)(lane & 15) * 128u + (uint32_t)(((lane >> 4) ^ (lane & 7)) << 4);
    return (uint32_t)row0 * 128u + (own ^ (uint32_t)(c << 5));
}
__device__ __forceinline__ uint32_t tile_cols(int lane, int row0, int c) {
    const uint32_t own = (uint32_t)((lane & 7) + ((lane >> 4) << 3)) * 128u + (uint32_t)((((lane >> 3) & 1) ^ (lane & 7)) << 4);
    return (uint32_t)row0 * 128u + (own ^ (uint32_t)(c << 5));
}
__device__ __forceinline__ uint32_t blk_plain(int lane) { return (uint32_t)lane * 16u; }
__device__ __forceinline__ uint32_t blk_cols(int lane) {
    return (uint32_t)((lane >> 3) & 1) * 256u + (uint32_t)((lane & 7) + ((lane >> 4) << 3)) * 16u;
}

// Place of element (i, j) of a [64][64] fp32 matrix kept in the order of matrix-instruction accumulators: a warp's 16 rows i in
// turn, in them eight columns j at a time, four elements per lane (rows g and g + 8 of column 2q, then of 2q + 1).
__device__ __forceinline__ int accumulator_place(int i, int j) {
    return (((i >> 4) * 8 + (j >> 3)) * 32 + (i & 7) * 4 + ((j & 7) >> 1)) * 4 + (j & 1) * 2 + ((i >> 3) & 1);
}

// What the builder leaves of a chunk in global memory: the 128 x 128 fp16 operator O[n][k], n = (j' in the order of k | t), as the core
// matrices (eight rows n, eight k, 128 bytes) of a K-major tcgen05 operand without swizzle, 16 of them along k and 16 along n.
// The contraction index (64 j, then 64 s) is ordered so that a lane of the builder holds four neighbouring k of a row in its
// accumulators: the eight of core 2 c + m are {2q, 2q+1, 2q+8, 2q+9} of the 16-block c for q = 2 m, then for q = 2 m + 1.  Behind
// the operator e^{c_L}[64] in fp32, two signed exponents per channel (fx = e^{c_L} 2^ef; P and Kt are stored times 2^eg), two
// per 16-token block (its r rows were taken times 2^-er, its k rows times 2^-ek), and the mark.
constexpr uint32_t kOperatorBytes = 4 * kPanel;
constexpr uint32_t kDecayAt = kOperatorBytes, kExpAt = kDecayAt + 256;
constexpr uint32_t kVectorBytes = 256 + 128 + 16;
constexpr uint32_t kRowExpAt = 384;                      // of er, ek of every block in turn, from kDecayAt on
constexpr uint32_t kMarkAt = kDecayAt + kVectorBytes;   // int: the chunk is beyond what fp16 operands resolve
constexpr size_t kRecord = 33280;                        // bytes per chunk in the workspace

// Bounded wait for a whole warp without compiler-made divergence handling around the loop.
__device__ __forceinline__ bool mbar_wait_tight(uint64_t *bar, uint32_t parity, uint32_t limit) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p, r;\n\t.reg .u32 n;\n\t"
        "mov.u32 n, %3;\n"
        "POLL_%=:\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "@p bra DONE_%=;\n\t"
        "sub.u32 n, n, 1;\n\t"
        "setp.ne.u32 r, n, 0;\n\t"
        "@r bra POLL_%=;\n"
        "DONE_%=:\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(limit)
        : "memory");
    return ok != 0;
}

// d = exp(-exp(w)) of a channel pair
// (subnormal results flushed: without that every exponential costs a compare and two more multiplications)
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float2 decay2(float2 w) {
    constexpr float kLog2e = 1.4426950408889634f;
    const float2 x = mul2(w, make_float2(kLog2e, kLog2e));
    const float2 z = mul2(make_float2(ex2(x.x), ex2(x.y)), make_float2(-kLog2e, -kLog2e));
    return make_float2(ex2(z.x), ex2(z.y));
}
// A bf16 pair times 2^e, 0 <= e <= 60: exact
__device__ __forceinline__ uint32_t raise_bf2(uint32_t v, int e) {
    const uint32_t f = (uint32_t)(127 + e) * 0x00800080u;
    const __nv_bfloat162 y = __hmul2(*reinterpret_cast<const __nv_bfloat162 *>(&v), *reinterpret_cast<const __nv_bfloat162 *>(&f));
    return *reinterpret_cast<const uint32_t *>(&y);
}
__device__ __forceinline__ uint32_t pack2(float2 v) { return pack_half2(v.x, v.y); }
__device__ __forceinline__ int exponent_of(float v) { return (int)(__float_as_uint(v) >> 23); }   // biased; v > 0
__device__ __forceinline__ float exp2_of(int e) { return __uint_as_float((uint32_t)(e + 127) << 23); }   // -126 <= e <= 127

}  // namespace sm100
}  // namespace rwkv7
