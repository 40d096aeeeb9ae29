// bc1_decode.cu -- decode_bc1 / evaluate_bc1_error and the reference's
// decode_bc3 / evaluate_bc3_error over many blocks.
#include <cuda_runtime.h>

#include "bc1_kernels.h"

namespace icbc_gpu {

constexpr unsigned kFullWarp = 0xffffffffu;

// A warp takes 32 blocks.  Each lane decodes the palette of one; the texels
// are then moved a block row (16 bytes) a lane, 8 blocks at a time, with the
// block's palette and indices by shuffle, so that every load and store of the
// warp covers 512 consecutive bytes.  With a block a lane each access touched
// 32 half sectors 64 bytes apart: 2^22 blocks took 68 us to decode (4.4 TB/s)
// and 74 to evaluate (4.3), now 47 (6.5) and 51 (6.3); both on 2^20 blocks, one
// after the other, 45 and now 33-34.  Bound by DRAM, evaluate by its shuffles
// and selects too.
//
// Row `lane & 3` of the block that lane `src` holds: its 4 texels.
__device__ __forceinline__ uint4 block_row(const uint32_t pk[4], uint32_t indices, int src) {
    const uint32_t p0 = __shfl_sync(kFullWarp, pk[0], src), p1 = __shfl_sync(kFullWarp, pk[1], src),
                   p2 = __shfl_sync(kFullWarp, pk[2], src), p3 = __shfl_sync(kFullWarp, pk[3], src);
    const uint32_t bits = __shfl_sync(kFullWarp, indices, src) >> (8 * (threadIdx.x & 3));
    uint32_t q[4];
#pragma unroll
    for (int x = 0; x < 4; x++) {
        const uint32_t i = bits >> (2 * x);
        q[x] = (i & 2) ? ((i & 1) ? p3 : p2) : ((i & 1) ? p1 : p0);
    }
    return make_uint4(q[0], q[1], q[2], q[3]);
}

// Writes the 32 blocks at `base` (palette and indices of block base + lane in
// pk, indices) as RGBA8.
__device__ __forceinline__ void store_blocks(uint4 *rgba, int64_t base, int64_t n, const uint32_t pk[4],
                                             uint32_t indices) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int it = 0; it < 4; it++) {
        const int src = 8 * it + (lane >> 2);
        const uint4 q = block_row(pk, indices, src);
        if (base + src < n) rgba[4 * base + 32 * it + lane] = q;
    }
}

// decode_bc1 (icbc.h:2915-2927).
__global__ void k_decode(const uint2 *blocks, uint4 *rgba, int64_t n, int decoder) {
    const int lane = threadIdx.x & 31;
    const int64_t base = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) - lane;
    if (base >= n) return;
    const uint2 v = base + lane < n ? blocks[base + lane] : make_uint2(0u, 0u);
    const Pal32 p = palette32(v.x & 0xffff, v.x >> 16, decoder);
    const bool four = (v.x & 0xffff) > (v.x >> 16);
    uint32_t pk[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t a = (i == 3 && !four) ? 0u : 255u;
        pk[i] = (uint32_t)p.r[i] | ((uint32_t)p.g[i] << 8) | ((uint32_t)p.b[i] << 16) | (a << 24);
    }
    store_blocks(rgba, base, n, pk, v.y);
}

// evaluate_bc1_error (icbc.h:3030-3046): integer squared error per texel,
// accumulated as float in texel order.  The sums are integers of at most 16 *
// 3 * 255^2 < 2^24, exact in float, so integer sums in any order give the
// same value.
__global__ void k_evaluate(const uint4 *rgba, const uint2 *blocks, float *errors, int64_t n, int decoder) {
    const int lane = threadIdx.x & 31;
    const int64_t base = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) - lane;
    if (base >= n) return;
    uint4 texels[4];
#pragma unroll
    for (int it = 0; it < 4; it++) {
        const int src = 8 * it + (lane >> 2);
        texels[it] = base + src < n ? rgba[4 * base + 32 * it + lane] : make_uint4(0u, 0u, 0u, 0u);
    }
    const uint2 v = base + lane < n ? blocks[base + lane] : make_uint2(0u, 0u);
    const Pal32 p = palette32(v.x & 0xffff, v.x >> 16, decoder);
    uint32_t pk[4];
#pragma unroll
    for (int i = 0; i < 4; i++) pk[i] = (uint32_t)p.r[i] | ((uint32_t)p.g[i] << 8) | ((uint32_t)p.b[i] << 16);
    // Per row sum (a - c)^2 as a.a + c.c - 2 a.c, byte dot products.
    int sum[4];
#pragma unroll
    for (int it = 0; it < 4; it++) {
        const uint4 q = block_row(pk, v.y, 8 * it + (lane >> 2));
        const uint32_t a[4] = {q.x, q.y, q.z, q.w},
                       c[4] = {texels[it].x, texels[it].y, texels[it].z, texels[it].w};
        unsigned squares = 0, cross = 0;
#pragma unroll
        for (int x = 0; x < 4; x++) {
            squares = __dp4a(a[x], a[x], squares);
            squares = __dp4a(c[x] & 0xffffffu, c[x] & 0xffffffu, squares);
            cross = __dp4a(a[x], c[x], cross);  // a's fourth byte is 0
        }
        sum[it] = (int)(squares - 2 * cross);
    }
    // The 4 lanes of a block share its rows for each `it`: two exchanges leave
    // lane l with the sum of block 8 (l & 3) + l / 4.
    const bool odd = lane & 1, upper = lane & 2;
    const int s0 = (odd ? sum[1] : sum[0]) + __shfl_xor_sync(kFullWarp, odd ? sum[0] : sum[1], 1);
    const int s1 = (odd ? sum[3] : sum[2]) + __shfl_xor_sync(kFullWarp, odd ? sum[2] : sum[3], 1);
    const int total = (upper ? s1 : s0) + __shfl_xor_sync(kFullWarp, upper ? s0 : s1, 2);
    const int64_t b = base + 8 * (lane & 3) + (lane >> 2);
    if (b < n) errors[b] = (float)total;
}

// decode_bc3 (icbc.h:2929-2947): a 16-byte block is the BC4 alpha half
// (alpha0, alpha1, 6 index bytes) and a BC1 block.  The colour palette is
// always the 4-colour form; the reference's alpha index is always 0, so every
// texel takes alpha0.
__global__ void k_decode_bc3(const uint4 *blocks, uint4 *rgba, int64_t n, int decoder) {
    const int lane = threadIdx.x & 31;
    const int64_t base = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) - lane;
    if (base >= n) return;
    const uint4 v = base + lane < n ? blocks[base + lane] : make_uint4(0u, 0u, 0u, 0u);
    const Pal32 p = palette32_form(v.z & 0xffff, v.z >> 16, decoder, true);
    const uint32_t a = (v.x & 255u) << 24;
    uint32_t pk[4];
#pragma unroll
    for (int i = 0; i < 4; i++) pk[i] = (uint32_t)p.r[i] | ((uint32_t)p.g[i] << 8) | ((uint32_t)p.b[i] << 16) | a;
    store_blocks(rgba, base, n, pk, v.w);
}

// evaluate_bc3_error (icbc.h:3048-3071): per texel in order, the integer
// colour error (scaled by alpha / 255.0f when alpha_blend), then the squared
// difference of alpha0 and the texel's alpha, accumulated as float.
__global__ void k_evaluate_bc3(const uint4 *rgba, const uint4 *blocks, float *errors, int64_t n, int alpha_blend,
                               int decoder) {
    const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= n) return;
    const uint4 v = blocks[b];
    const Pal32 p = palette32_form(v.z & 0xffff, v.z >> 16, decoder, true);
    const int alpha0 = (int)(v.x & 255u);
    float error = 0.0f;
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const uint4 q = rgba[4 * b + r];
        const uint32_t px[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int x = 0; x < 4; x++) {
            const int i = (v.w >> (2 * (4 * r + x))) & 3;
            const int dr = p.r[i] - (int)(px[x] & 255), dg = p.g[i] - (int)((px[x] >> 8) & 255),
                      db = p.b[i] - (int)((px[x] >> 16) & 255), ta = (int)(px[x] >> 24);
            const float scale = alpha_blend ? __fdiv_rn((float)ta * 1.0f, 255.0f) : 1.0f;
            error += scale * (float)(dr * dr + dg * dg + db * db);
            error += (float)((alpha0 - ta) * (alpha0 - ta));
        }
    }
    errors[b] = error;
}

cudaError_t launch_decode_bc3(const void *blocks, void *rgba, int64_t n, int decoder, cudaStream_t stream) {
    if (n == 0) return cudaSuccess;
    const int threads = 256;
    k_decode_bc3<<<(unsigned)((n + threads - 1) / threads), threads, 0, stream>>>(
        reinterpret_cast<const uint4 *>(blocks), reinterpret_cast<uint4 *>(rgba), n, decoder);
    return cudaGetLastError();
}

cudaError_t launch_evaluate_bc3(const void *rgba, const void *blocks, float *errors, int64_t n, int alpha_blend,
                                int decoder, cudaStream_t stream) {
    if (n == 0) return cudaSuccess;
    const int threads = 256;
    k_evaluate_bc3<<<(unsigned)((n + threads - 1) / threads), threads, 0, stream>>>(
        reinterpret_cast<const uint4 *>(rgba), reinterpret_cast<const uint4 *>(blocks), errors, n, alpha_blend,
        decoder);
    return cudaGetLastError();
}

cudaError_t launch_decode(const void *blocks, void *rgba, int64_t n, int decoder, cudaStream_t stream) {
    if (n == 0) return cudaSuccess;
    const int threads = 256;
    k_decode<<<(unsigned)((n + threads - 1) / threads), threads, 0, stream>>>(
        reinterpret_cast<const uint2 *>(blocks), reinterpret_cast<uint4 *>(rgba), n, decoder);
    return cudaGetLastError();
}

cudaError_t launch_evaluate(const void *rgba, const void *blocks, float *errors, int64_t n, int decoder,
                            cudaStream_t stream) {
    if (n == 0) return cudaSuccess;
    const int threads = 256;
    k_evaluate<<<(unsigned)((n + threads - 1) / threads), threads, 0, stream>>>(
        reinterpret_cast<const uint4 *>(rgba), reinterpret_cast<const uint2 *>(blocks), errors, n, decoder);
    return cudaGetLastError();
}

}  // namespace icbc_gpu
