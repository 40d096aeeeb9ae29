// bc1_refine.cu -- endpoint refinement of level 9 as its own pass.
//
// refine_endpoints (icbc.h:3574-3651) runs 33 to 256 sequential steps per
// block, different for every block.  The encoder leaves, per block, the error
// refinement starts from and whether it applies (RefineSlot); these kernels
// then run the reference's steps.  Many blocks: a block a lane, with a queue
// per lane (k_refine).  Few: a warp a block (k_refine_warp).
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "bc1_loaders.cuh"

namespace icbc_gpu {

// One float block (the compress_bc1 layout) into a lane's texel row.
__device__ __forceinline__ void load_float_block_lane(const BlocksSrc &s, int64_t b, float *row) {
    const float4 *c = reinterpret_cast<const float4 *>(s.colors) + b * 16;
#pragma unroll 4
    for (int t = 0; t < 16; t++) {
        const float4 v = __ldg(c + t);
        row[4 * t + 0] = v.x;
        row[4 * t + 1] = v.y;
        row[4 * t + 2] = v.z;
    }
    if (s.weights) {
        const float4 *w4 = reinterpret_cast<const float4 *>(s.weights) + b * 4;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float4 v = __ldg(w4 + j);
            row[16 * j + 3] = v.x;
            row[16 * j + 7] = v.y;
            row[16 * j + 11] = v.z;
            row[16 * j + 15] = v.w;
        }
    } else {
#pragma unroll
        for (int t = 0; t < 16; t++) row[4 * t + 3] = 1.0f;
    }
}

constexpr size_t kRefineLutBytes = 256 * sizeof(float);
// Texel rows of 68 floats (16-byte aligned, 17 float4): a texel's colour and
// weight are one 16-byte load, and the 16-byte accesses of any 8 lanes to
// the same texel of their rows fall in 8 different bank groups.
constexpr int kRefineStride = 68;
constexpr size_t kRefineRowBytes = kWarpsPerCta * sizeof(float) * 32 * kRefineStride;
// Then each warp's candidate palettes, 4 entries x 32 lanes of float4
// (block_error_pal): 44 KB per CTA, five CTAs per SM.
constexpr size_t kRefineSmem = kRefineLutBytes + kRefineRowBytes + kWarpsPerCta * 4 * 32 * sizeof(float4);

constexpr int kRefillBatch = 16;  // 4: 3% slower, 8: 0.4%, 12: as 16 (hard mixture, level 9)

__device__ __forceinline__ V3 shfl3(V3 v, int src) {
    return v3(__shfl_sync(kFull, v.x, src), __shfl_sync(kFull, v.y, src), __shfl_sync(kFull, v.z, src));
}

// Bit t of x (t < 16) to bit 2t.
__device__ __forceinline__ uint32_t spread_bits(uint32_t x) {
    x = (x | (x << 8)) & 0x00ff00ffu;
    x = (x | (x << 4)) & 0x0f0f0f0fu;
    x = (x | (x << 2)) & 0x33333333u;
    return (x | (x << 1)) & 0x55555555u;
}

// A block a lane: a lane that finishes a block takes the next pending one
// (warp-aggregated atomics on one counter), so lanes stay busy until the
// queue is empty.
// MODE 0: float blocks (s), 1: one image (d), 2: the deferred level-9 blocks
// of a batch (images + map), each lane with its own image's decoder and
// parameters.
template <int MODE>
__global__ void __launch_bounds__(kWarpsPerCta * 32) k_refine(const GlobalTables *G, ImageDesc d, BlocksSrc s,
                                                              EncodeParams p, uint2 *out, float *errors,
                                                              const RefineSlot *st, int64_t n,
                                                              unsigned long long *counter, const ImageDesc *images,
                                                              RefineMap map) {
    // Shared memory: the u8 table (all refinement needs of the staged
    // tables), each warp's 32 float texel rows, then its candidate palettes.
    extern __shared__ __align__(16) unsigned char smem[];
    float *lut = reinterpret_cast<float *>(smem);
    for (int i = threadIdx.x; i < 256; i += blockDim.x) lut[i] = G->s.lut255[i];
    __syncthreads();
    WarpCtx w{};
    w.D = &G->dec[p.decoder];
    w.in = reinterpret_cast<float *>(smem + kRefineLutBytes) + (threadIdx.x >> 5) * 32 * kRefineStride;
    w.lane = threadIdx.x & 31;
    const int lane = w.lane;
    float *row = w.in + lane * kRefineStride;
    float4 *pal = reinterpret_cast<float4 *>(smem + kRefineLutBytes + kRefineRowBytes) + (threadIdx.x >> 5) * 128 + lane;
    EncodeParams lp = p;
    RefineLane r;
    uint2 *o = nullptr;
    float *er = nullptr;
    bool have = false, exhausted = false;
    // The last accepted candidate's palette times the colour weights, the
    // source of the index update the warp computes for this lane.
    V3 q0 = v3(0.0f, 0.0f, 0.0f), q1 = q0, q2 = q0, q3 = q0;
    for (;;) {
        // Lanes without a block take the next ones; blocks that need no
        // refinement are skipped (their error and bytes are final already).
        // Refills run in batches: a lane that finished waits until
        // kRefillBatch lanes (or all) need a block, so the divergent refill
        // code runs for many lanes at once instead of one at a time.
        unsigned need = __ballot_sync(kFull, !have && !exhausted);
        if (__popc(need) < kRefillBatch && __any_sync(kFull, have)) need = 0;
        while (need) {
            const int leader = __ffs(need) - 1;
            unsigned long long base = 0;
            if (lane == leader) base = atomicAdd(counter, (unsigned long long)__popc(need));
            base = __shfl_sync(kFull, base, leader);
            if (!have && !exhausted) {
                const int64_t mine = (int64_t)base + __popc(need & ((1u << lane) - 1u));
                if (mine >= n) {
                    exhausted = true;
                } else {
                    const RefineSlot sl = st[mine];
                    if (sl.pending) {
                        if (MODE == 2) {
                            int lo = 0, hi = map.n;
                            while (hi - lo > 1) {
                                const int mid = (lo + hi) >> 1;
                                if (map.map_start[mid] <= mine) lo = mid;
                                else hi = mid;
                            }
                            const ImageDesc &di = images[map.map_image[lo]];
                            const int64_t b = mine - map.map_start[lo];
                            lp.decoder = di.decoder;
                            lp.three_color_mode = di.three_color_mode;
                            lp.three_color_black = di.three_color_black;
                            lp.cw = v3(di.cw[0], di.cw[1], di.cw[2]);
                            w.D = &G->dec[di.decoder];
                            load_image_block(di, b, row, lut);
                            o = di.out + b;
                            er = di.errors ? di.errors + b : nullptr;
                        } else {
                            if (MODE == 1) load_image_block(d, mine, row, lut);
                            else load_float_block_lane(s, mine, row);
                            o = out + mine;
                            er = errors ? errors + mine : nullptr;
                        }
                        const uint2 cur = *o;
                        refine_begin(w, lut, FloatRow4{row}, lp, sl.error, cur.x & 0xffff, cur.x >> 16, cur.y, r);
                        have = true;
                    }
                }
            }
            need = __ballot_sync(kFull, !have && !exhausted);
        }
        if (!__any_sync(kFull, have)) break;
        bool accepted = false, stop = false;
        if (have) {
            PalF pr;
            accepted = refine_try(w, lut, FloatRow4{row}, lp, r, pr, stop, pal);
            if (accepted) {
                q0 = pr.c[0] * lp.cw;
                q1 = pr.c[1] * lp.cw;
                q2 = pr.c[2] * lp.cw;
                q3 = pr.c[3] * lp.cw;
            }
        }
        // An accepted step's lane needs indices_generic of its new palette
        // before its next step.  Each texel's index depends on that texel
        // alone, so the warp computes them for two such lanes at a time: the
        // half-warp of lane l takes texel l & 15 of one block, and two ballots
        // pack the 2-bit indices in texel order.
        unsigned m = __ballot_sync(kFull, accepted);
        while (m) {
            const int l0 = __ffs(m) - 1;
            m &= m - 1;
            const int l1 = m ? __ffs(m) - 1 : l0;
            m &= m - 1;
            const int src = lane < 16 ? l0 : l1;
            const V3 p0 = shfl3(q0, src), p1 = shfl3(q1, src), p2 = shfl3(q2, src), p3 = shfl3(q3, src);
            const V3 cw = shfl3(lp.cw, src);
            const uint32_t x =
                index_generic(FloatRow4{w.in + src * kRefineStride}.color(lane & 15), cw, p0, p1, p2, p3);
            const unsigned lo = __ballot_sync(kFull, x & 1u), hi = __ballot_sync(kFull, x >> 1);
            if (lane == l0) r.base_idx = spread_bits(lo & 0xffffu) | (spread_bits(hi & 0xffffu) << 1);
            else if (lane == l1) r.base_idx = spread_bits(lo >> 16) | (spread_bits(hi >> 16) << 1);
        }
        if (have && stop) {
            *o = make_uint2(r.c0 | (r.c1 << 16), r.idx);
            if (er) *er = r.best;
            have = false;
        }
    }
}

// Shared memory of a CTA: the u8 table, then per warp its block's 16 texels
// (r, g, b, weight) and every lane's candidate palette, entry-major, so that
// the 16-byte accesses of any 8 lanes fall in 8 bank groups.
constexpr int kRefineWarpWarps = 8;
constexpr size_t kRefineWarpFloat4 = 16 + 4 * 32;
constexpr size_t kRefineWarpSmem = 256 * sizeof(float) + kRefineWarpWarps * kRefineWarpFloat4 * sizeof(float4);

// The weighted error of the block's texels under this lane's palette, summed
// in texel order (icbc.h:3006-3028), `indices` the same for the whole warp.
__device__ __forceinline__ float warp_block_error(const float4 *texels, V3 cw, const float4 *pal, uint32_t indices) {
    float error = 0.0f;
#pragma unroll
    for (int t = 0; t < 16; t++) {
        const float4 q = pal[32 * ((indices >> (2 * t)) & 3)], c = texels[t];
        error += c.w * texel_mse(v3(q.x, q.y, q.z), v3(c.x, c.y, c.z), cw);
    }
    return error;
}

// indices_generic (icbc.h:3179-3235) of the warp's block under `pal`, a texel
// a lane: two ballots pack the 2-bit indices in texel order.
__device__ __forceinline__ uint32_t warp_indices(const float4 *texels, V3 cw, V3 p0, V3 p1, V3 p2, V3 p3) {
    const float4 c = texels[threadIdx.x & 15];
    const uint32_t x = index_generic(v3(c.x, c.y, c.z), cw, p0 * cw, p1 * cw, p2 * cw, p3 * cw);
    const unsigned lo = __ballot_sync(kFull, x & 1u), hi = __ballot_sync(kFull, x >> 1);
    return spread_bits(lo & 0xffffu) | (spread_bits(hi & 0xffffu) << 1);
}

// A warp a block, for fewer blocks than k_refine has lanes.  The steps up to
// the next accepted one all start from the same block, so a warp tries 32 of
// them at once, a step a lane, and takes the first that is accepted; 32 steps
// are every delta of both endpoints, so a round without an accepted step is
// the end (the 33rd would repeat the first).  Warps take chunks of slots from
// one counter.
//
// Bound by FP32 issue: a round is about 450 instructions (the candidate's
// palette, 16 texels of 21), 1.5 rounds a block on smooth images and 11 on
// the hard mixture, where k_refine's lanes need a third of the instructions.
// But k_refine runs a block's steps one after another, however few blocks
// there are: the pass took 133 us for 64 x 64, 277 for 1,000 blocks of the
// hard mixture and 377 for 40,000; here 21, 34 and 291.  At 200,000 k_refine
// takes 723 us and this kernel 1018, so k_refine keeps the work that gives
// each of its lanes a block.
template <int MODE>
__global__ void __launch_bounds__(kRefineWarpWarps * 32) k_refine_warp(const GlobalTables *G, ImageDesc d, BlocksSrc s,
                                                              EncodeParams p, uint2 *out, float *errors,
                                                              const RefineSlot *st, int64_t n, int chunk,
                                                              unsigned long long *counter, const ImageDesc *images,
                                                              RefineMap map) {
    extern __shared__ __align__(16) unsigned char smem[];
    float *lut = reinterpret_cast<float *>(smem);
    for (int i = threadIdx.x; i < 256; i += blockDim.x) lut[i] = G->s.lut255[i];
    __syncthreads();
    const int lane = threadIdx.x & 31;
    float4 *texels = reinterpret_cast<float4 *>(lut + 256) + (threadIdx.x >> 5) * kRefineWarpFloat4;
    float4 *pals = texels + 16;
    const DecoderTables *D = &G->dec[p.decoder];
    // The delta of step `lane` (and of lane + 16), each channel plus one in two bits.
    const int8_t *own = c_deltas[lane & 15];
    const int delta = (own[0] + 1) | ((own[1] + 1) << 2) | ((own[2] + 1) << 4);
    for (;;) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(counter, (unsigned long long)chunk);
        base = __shfl_sync(kFull, base, 0);
        if ((int64_t)base >= n) break;
        // This chunk's slots, one a lane; blocks that need no refinement are
        // final already.
        const int64_t mine = (int64_t)base + lane;
        RefineSlot sl{0.0f, 0u};
        if (lane < chunk && mine < n) sl = st[mine];
        int image = 0;
        int64_t local = mine;
        if (MODE == 2 && sl.pending) {
            int lo = 0, hi = map.n;
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (map.map_start[mid] <= mine) lo = mid;
                else hi = mid;
            }
            image = (int)map.map_image[lo];
            local = mine - map.map_start[lo];
        }
        for (unsigned todo = __ballot_sync(kFull, sl.pending != 0); todo; todo &= todo - 1) {
            const int src = __ffs(todo) - 1;
            const int64_t b = __shfl_sync(kFull, local, src);
            float best = __shfl_sync(kFull, sl.error, src);
            uint2 *o = out + b;
            float *er = errors ? errors + b : nullptr;
            const ImageDesc *im = &d;
            if (MODE == 2) {
                im = images + __shfl_sync(kFull, image, src);
                p.decoder = im->decoder;
                p.three_color_mode = im->three_color_mode;
                p.three_color_black = im->three_color_black;
                p.cw = v3(im->cw[0], im->cw[1], im->cw[2]);
                D = &G->dec[p.decoder];
                o = im->out + b;
                er = im->errors ? im->errors + b : nullptr;
            }
            const uint2 cur = *o;
            uint32_t c0 = cur.x & 0xffff, c1 = cur.x >> 16, idx = cur.y;
            __syncwarp();  // the previous block's texels and palettes are read
            if (lane < 16) {
                if (MODE == 0) {
                    const float4 v = __ldg(reinterpret_cast<const float4 *>(s.colors) + b * 16 + lane);
                    texels[lane] = make_float4(v.x, v.y, v.z, s.weights ? __ldg(s.weights + b * 16 + lane) : 1.0f);
                } else {
                    texels[lane] = load_image_texel(*im, b, lane, lut);
                }
            }
            __syncwarp();
            PalF pr = palette_f(c0, c1, p.decoder, lut, D);
            uint32_t base_idx = warp_indices(texels, p.cw, pr.c[0], pr.c[1], pr.c[2], pr.c[3]);
            // Steps i .. i + 31 from the block (c0, c1, base_idx, best).
            for (int i = 0;;) {
                uint32_t r0 = c0, r1 = c1;
                const int dl = __shfl_sync(kFull, delta, i + lane);
                refine_candidate(i + lane, (dl & 3) - 1, ((dl >> 2) & 3) - 1, (dl >> 4) - 1, p, r0, r1);
                pr = palette_f(r0, r1, p.decoder, lut, D);
#pragma unroll
                for (int e = 0; e < 4; e++) pals[32 * e + lane] = make_float4(pr.c[e].x, pr.c[e].y, pr.c[e].z, 0.0f);
                const float e = warp_block_error(texels, p.cw, pals + lane, base_idx);
                const unsigned accepted = __ballot_sync(kFull, e < best && i + lane < 256);
                if (!accepted) break;
                const int a = __ffs(accepted) - 1;
                best = __shfl_sync(kFull, e, a);
                c0 = __shfl_sync(kFull, r0, a);
                c1 = __shfl_sync(kFull, r1, a);
                idx = base_idx;
                i += a + 1;
                if (i >= 256) break;
                __syncwarp();
                const float4 q0 = pals[a], q1 = pals[32 + a], q2 = pals[64 + a], q3 = pals[96 + a];
                base_idx = warp_indices(texels, p.cw, v3(q0.x, q0.y, q0.z), v3(q1.x, q1.y, q1.z),
                                        v3(q2.x, q2.y, q2.z), v3(q3.x, q3.y, q3.z));
                __syncwarp();
            }
            if (lane == 0) {
                *o = make_uint2(c0 | (c1 << 16), idx);
                if (er) *er = best;
            }
        }
    }
}

namespace {

std::mutex g_pool_mutex;
cudaMemPool_t g_pool[64] = {};

}  // namespace

// The library-owned pool of the current device, created on first use.
static cudaError_t device_pool(cudaMemPool_t *out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    if (!g_pool[dev]) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        e = cudaMemPoolCreate(&g_pool[dev], &props);
        if (e != cudaSuccess) return e;
        uint64_t keep = 1ull << 30;
        cudaMemPoolSetAttribute(g_pool[dev], cudaMemPoolAttrReleaseThreshold, &keep);
    }
    *out = g_pool[dev];
    return cudaSuccess;
}

// Creates the pool of the current device if it does not exist yet.  Pool
// creation is not allowed while a stream captures, so code that captures
// launches which take scratch calls this first.
cudaError_t scratch_prepare() {
    cudaMemPool_t pool;
    return device_pool(&pool);
}

// Stream-ordered scratch from a library-owned pool of the current device
// (freed memory stays cached in the pool for the next call).
cudaError_t scratch_alloc(void **ptr, size_t bytes, cudaStream_t stream) {
    cudaMemPool_t pool;
    const cudaError_t e = device_pool(&pool);
    if (e != cudaSuccess) return e;
    return cudaMallocFromPoolAsync(ptr, bytes, pool, stream);
}

cudaError_t scratch_free(void *ptr, cudaStream_t stream) { return cudaFreeAsync(ptr, stream); }

// CTAs of k_refine per SM (0: not known yet).
template <int MODE>
static int &refine_resident() {
    static int resident = 0;
    return resident;
}

template <int MODE>
static cudaError_t refine_grid(int64_t n, int sms, size_t smem, int *grid) {
    int &resident = refine_resident<MODE>();
    cudaError_t e = cudaFuncSetAttribute(k_refine<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    if (!resident) {
        int per_sm = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_refine<MODE>, kWarpsPerCta * 32, smem);
        if (e != cudaSuccess) return e;
        resident = per_sm > 0 ? per_sm : 1;
    }
    const int64_t want = (n + kWarpsPerCta * 32 - 1) / (kWarpsPerCta * 32);
    const int64_t cap = (int64_t)sms * resident;
    *grid = (int)(want < cap ? (want > 0 ? want : 1) : cap);
    return cudaSuccess;
}

// Launches the pass over n slots: k_refine when each of its resident lanes
// gets a block, else k_refine_warp.
template <int MODE>
static cudaError_t refine_pass(const GlobalTables *G, const ImageDesc &d, const BlocksSrc &s, const EncodeParams &p,
                               uint2 *out, float *errors, const RefineSlot *st, int64_t n, unsigned long long *counter,
                               const ImageDesc *images, RefineMap map, cudaStream_t stream, int sms) {
    int grid = 0;
    cudaError_t e = refine_grid<MODE>(n, sms, kRefineSmem, &grid);
    if (e != cudaSuccess) return e;
    if (n >= (int64_t)sms * refine_resident<MODE>() * kWarpsPerCta * 32) {
        k_refine<MODE><<<grid, kWarpsPerCta * 32, kRefineSmem, stream>>>(G, d, s, p, out, errors, st, n, counter,
                                                                         images, map);
        return cudaGetLastError();
    }
    // One slot a warp at a time, or as many as give every resident warp one chunk.
    static int resident = 0;
    if (!resident) {
        int per_sm = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_refine_warp<MODE>, kRefineWarpWarps * 32,
                                                          kRefineWarpSmem);
        if (e != cudaSuccess) return e;
        resident = per_sm > 0 ? per_sm : 1;
    }
    const int64_t warps = (int64_t)sms * resident * kRefineWarpWarps;
    const int chunk = (int)std::max<int64_t>(1, std::min<int64_t>(32, (n + warps - 1) / warps));
    const int64_t want = (n + (int64_t)chunk * kRefineWarpWarps - 1) / ((int64_t)chunk * kRefineWarpWarps);
    const int ctas = (int)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)sms * resident));
    k_refine_warp<MODE><<<ctas, kRefineWarpWarps * 32, kRefineWarpSmem, stream>>>(G, d, s, p, out, errors, st, n, chunk,
                                                                                  counter, images, map);
    return cudaGetLastError();
}

cudaError_t launch_refine(const GlobalTables *G, const ImageDesc *image, const BlocksSrc *blocks,
                          const EncodeParams &p, uint2 *out, float *errors, const RefineSlot *st, int64_t n,
                          unsigned long long *counter, cudaStream_t stream, int sms) {
    const ImageDesc dd = image ? *image : ImageDesc{};
    const BlocksSrc ss = blocks ? *blocks : BlocksSrc{nullptr, nullptr};
    const RefineMap none{nullptr, nullptr, 0};
    return image ? refine_pass<1>(G, dd, ss, p, out, errors, st, n, counter, nullptr, none, stream, sms)
                 : refine_pass<0>(G, dd, ss, p, out, errors, st, n, counter, nullptr, none, stream, sms);
}

cudaError_t launch_refine_batch(const GlobalTables *G, const ImageDesc *images, RefineMap map,
                                const RefineSlot *slots, int64_t total, unsigned long long *counter,
                                cudaStream_t stream, int sms) {
    return refine_pass<2>(G, ImageDesc{}, BlocksSrc{nullptr, nullptr}, EncodeParams{}, nullptr, nullptr, slots, total,
                          counter, images, map, stream, sms);
}

}  // namespace icbc_gpu
