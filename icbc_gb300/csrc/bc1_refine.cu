// bc1_refine.cu -- endpoint refinement of level 9 as its own pass.
//
// refine_endpoints (icbc.h:3574-3651) tries up to 256 steps in order, each
// moving one endpoint of the best block so far by one of 16 deltas, and stops
// 33 steps after the last one that helped.  The encoder leaves, per block, the
// error refinement starts from and whether it applies (RefineSlot).
//
// The steps up to the next accepted one all start from the same block, so the
// LANES lanes of a group try that many at once, a step a lane, and take the
// first that is accepted; 32 steps are every delta of both endpoints, so 32
// without an accepted one are the end (the 33rd would repeat the first).  A
// warp holds 32 / LANES groups, each with a block of its own.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "bc1_loaders.cuh"

namespace icbc_gpu {

// Shared memory of a CTA: the u8 table, then per warp its groups' blocks (16
// texels each as r, g, b, weight; 17 float4 apart, so that the groups of a
// quarter-warp read different banks) and every lane's candidate palette,
// entry-major, so that the 16-byte accesses of any 8 lanes fall in 8 bank
// groups.
constexpr int kRefineWarps = 8;
template <int LANES>
constexpr int kRefineFloat4 = 32 / LANES * 17 + 4 * 32;
template <int LANES>
constexpr size_t kRefineSmem = 256 * sizeof(float) + kRefineWarps * kRefineFloat4<LANES> * sizeof(float4);

constexpr int kRefillLanes = 8;  // 16: 2-4% slower on the hard mixture, 24: 13% (LANES 4)

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

// The weighted error of a block's texels under this lane's palette, summed in
// texel order (icbc.h:3006-3028).
__device__ __forceinline__ float group_block_error(const float4 *texels, V3 cw, const float4 *pal, uint32_t indices) {
    float error = 0.0f;
#pragma unroll
    for (int t = 0; t < 16; t++) {
        const float4 q = pal[32 * ((indices >> (2 * t)) & 3)], c = texels[t];
        error += c.w * texel_mse(v3(q.x, q.y, q.z), v3(c.x, c.y, c.z), cw);
    }
    return error;
}

// MODE 0: float blocks (s), 1: one image (d), 2: the deferred level-9 blocks
// of a batch (images + map), each with its own image's decoder and parameters.
// Warps take chunks of slots from one counter, groups take their blocks from
// the warp's chunk; groups without a block wait until kRefillLanes lanes do.
//
// Bound by issue (80% of cycles): a pass is about 550 instructions (the
// candidates' palettes, 16 texels of 21) and refills and new indices another
// 250.  A smooth block has 0.3 accepted steps of 36, one of the hard mixture 8
// of 69; what a pass tries after an accepted step is lost, so in units of a
// warp's pass a block takes 1.10 / 2.6 with 4 lanes, 1.13 / 3.4 with 8, 1.29 /
// 8.8 with 32, and its own steps one after another 9 / 21, 4.5 / 14 and 1.3 /
// 8.8 passes.  With a block a lane and the steps one by one 4096 x 4096 at
// level 9 took 3992 us, the hard mixture 4665, 200,000 float blocks of it
// 1287; with 4 lanes 3773, 4442 and 1171.
template <int MODE, int LANES>
__global__ void __launch_bounds__(kRefineWarps * 32) k_refine(const GlobalTables *G, ImageDesc d, BlocksSrc s,
                                                              EncodeParams p, uint2 *out, float *errors,
                                                              const RefineSlot *st, int64_t n, int chunk,
                                                              unsigned long long *counter, const ImageDesc *images,
                                                              RefineMap map) {
    extern __shared__ __align__(16) unsigned char smem[];
    float *lut = reinterpret_cast<float *>(smem);
    for (int i = threadIdx.x; i < 256; i += blockDim.x) lut[i] = G->s.lut255[i];
    __syncthreads();
    const int lane = threadIdx.x & 31, sub = lane % LANES, first = lane - sub;  // first: the group's first lane
    float4 *rows = reinterpret_cast<float4 *>(lut + 256) + (threadIdx.x >> 5) * kRefineFloat4<LANES>;
    float4 *texels = rows + lane / LANES * 17;
    float4 *pals = rows + 32 / LANES * 17;
    const DecoderTables *D = &G->dec[p.decoder];
    // The delta of step `lane` (and of lane + 16), each channel plus one in two bits.
    const int8_t *own = c_deltas[lane & 15];
    const int delta = (own[0] + 1) | ((own[1] + 1) << 2) | ((own[2] + 1) << 4);
    // The warp's chunk: slot base + lane is this lane's; todo: those still to refine.
    float slot_error = 0.0f;
    int64_t slot_block = 0;
    int slot_image = 0;
    unsigned todo = 0;
    bool drained = false;
    // The group's block, the same in all its lanes.
    bool have = false, reindex = false;
    uint32_t c0 = 0, c1 = 0, idx = 0, base_idx = 0;
    float best = 0.0f;
    int i = 0, left = 0, from = 0;  // next step, steps until the end, the lane whose palette slot is the block's
    uint2 *o = nullptr;
    float *er = nullptr;
    for (;;) {
        unsigned idle = __ballot_sync(kFull, !have);
        if (idle && !(drained && !todo) && (__popc(idle) >= kRefillLanes || idle == kFull)) {
            while (!todo && !drained) {
                unsigned long long base = 0;
                if (lane == 0) base = atomicAdd(counter, (unsigned long long)chunk);
                base = __shfl_sync(kFull, base, 0);
                drained = (int64_t)base >= n;
                const int64_t mine = (int64_t)base + lane;
                RefineSlot sl{0.0f, 0u};
                if (lane < chunk && mine < n) sl = st[mine];
                slot_error = sl.error;
                slot_block = mine;
                if (MODE == 2 && sl.pending) {
                    int lo = 0, hi = map.n;
                    while (hi - lo > 1) {
                        const int mid = (lo + hi) >> 1;
                        if (map.map_start[mid] <= mine) lo = mid;
                        else hi = mid;
                    }
                    slot_image = (int)map.map_image[lo];
                    slot_block = mine - map.map_start[lo];
                }
                todo = __ballot_sync(kFull, sl.pending != 0);
            }
            // The k-th idle group takes the k-th slot still to do.
            int src = -1;
            while (todo && idle) {
                const int at = __ffs(idle) - 1;
                if (first == at) src = __ffs(todo) - 1;
                todo &= todo - 1;
                idle &= ~((LANES == 32 ? ~0u : (1u << LANES) - 1u) << at);
            }
            const int from_lane = src < 0 ? 0 : src;
            const int64_t b = __shfl_sync(kFull, slot_block, from_lane);
            const float error = __shfl_sync(kFull, slot_error, from_lane);
            const int image = MODE == 2 ? __shfl_sync(kFull, slot_image, from_lane) : 0;
            if (src >= 0) {
                have = reindex = true;
                best = error;
                i = 0;
                left = 32;
                from = first;
                const ImageDesc *im = &d;
                if (MODE == 2) {
                    im = images + image;
                    p.decoder = im->decoder;
                    p.three_color_mode = im->three_color_mode;
                    p.three_color_black = im->three_color_black;
                    p.cw = v3(im->cw[0], im->cw[1], im->cw[2]);
                    D = &G->dec[p.decoder];
                    o = im->out + b;
                    er = im->errors ? im->errors + b : nullptr;
                } else {
                    o = out + b;
                    er = errors ? errors + b : nullptr;
                }
                const uint2 cur = *o;
                c0 = cur.x & 0xffff;
                c1 = cur.x >> 16;
                idx = cur.y;
#pragma unroll
                for (int t = sub; t < 16; t += LANES) {
                    if (MODE == 0) {
                        const float4 v = __ldg(reinterpret_cast<const float4 *>(s.colors) + b * 16 + t);
                        texels[t] = make_float4(v.x, v.y, v.z, s.weights ? __ldg(s.weights + b * 16 + t) : 1.0f);
                    } else {
                        texels[t] = load_image_texel(*im, b, t, lut);
                    }
                }
                if (sub == 0) {
                    const PalF pr = palette_f(c0, c1, p.decoder, lut, D);
#pragma unroll
                    for (int e = 0; e < 4; e++) pals[32 * e + lane] = make_float4(pr.c[e].x, pr.c[e].y, pr.c[e].z, 0.0f);
                }
            }
        }
        if (!__any_sync(kFull, have)) {
            if (drained && !todo) break;
            continue;
        }
        __syncwarp();
        // indices_generic (icbc.h:3179-3235) of the blocks whose palette is
        // new, two at a time: a half-warp takes a block, a lane a texel, and
        // two ballots pack the 2-bit indices in texel order.
        unsigned m = __ballot_sync(kFull, reindex && sub == 0);
        reindex = false;
        while (m) {
            const int l0 = __ffs(m) - 1;
            m &= m - 1;
            const int l1 = m ? __ffs(m) - 1 : l0;
            m &= m - 1;
            const int src = lane < 16 ? l0 : l1;
            const float4 *pal = pals + __shfl_sync(kFull, from, src);
            const V3 cw = MODE == 2 ? shfl3(p.cw, src) : p.cw;
            const float4 q0 = pal[0], q1 = pal[32], q2 = pal[64], q3 = pal[96], c = rows[src / LANES * 17 + (lane & 15)];
            const uint32_t x = index_generic(v3(c.x, c.y, c.z), cw, v3(q0.x, q0.y, q0.z) * cw, v3(q1.x, q1.y, q1.z) * cw,
                                             v3(q2.x, q2.y, q2.z) * cw, v3(q3.x, q3.y, q3.z) * cw);
            const unsigned lo = __ballot_sync(kFull, x & 1u), hi = __ballot_sync(kFull, x >> 1);
            if (first == l0) base_idx = spread_bits(lo & 0xffffu) | (spread_bits(hi & 0xffffu) << 1);
            else if (first == l1) base_idx = spread_bits(lo >> 16) | (spread_bits(hi >> 16) << 1);
        }
        __syncwarp();  // the palettes are rewritten
        // Steps i .. i + LANES - 1 from the block (c0, c1, base_idx, best).
        uint32_t r0 = c0, r1 = c1;
        const int dl = __shfl_sync(kFull, delta, i + sub);
        refine_candidate(i + sub, (dl & 3) - 1, ((dl >> 2) & 3) - 1, (dl >> 4) - 1, p, r0, r1);
        const PalF pr = palette_f(r0, r1, p.decoder, lut, D);
#pragma unroll
        for (int e = 0; e < 4; e++) pals[32 * e + lane] = make_float4(pr.c[e].x, pr.c[e].y, pr.c[e].z, 0.0f);
        const float e = group_block_error(texels, p.cw, pals + lane, base_idx);
        const unsigned accepted = __ballot_sync(kFull, have && e < best && i + sub < 256);
        const unsigned mine = LANES == 32 ? accepted : (accepted >> first) & ((1u << (LANES & 31)) - 1u);
        const int a = mine ? __ffs(mine) - 1 : 0;
        const float ne = __shfl_sync(kFull, e, first + a);
        const uint32_t n0 = __shfl_sync(kFull, r0, first + a), n1 = __shfl_sync(kFull, r1, first + a);
        if (mine) {
            best = ne;
            c0 = n0;
            c1 = n1;
            idx = base_idx;
            i += a + 1;
            left = 32;
            from = first + a;
            reindex = true;
        } else {
            i += LANES;
            left -= LANES;
        }
        if (have && (left <= 0 || i >= 256)) {
            if (sub == 0) {
                *o = make_uint2(c0 | (c1 << 16), idx);
                if (er) *er = best;
            }
            have = reindex = false;
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

template <int MODE, int LANES>
static cudaError_t refine_launch(const GlobalTables *G, const ImageDesc &d, const BlocksSrc &s, const EncodeParams &p,
                                 uint2 *out, float *errors, const RefineSlot *st, int64_t n,
                                 unsigned long long *counter, const ImageDesc *images, RefineMap map,
                                 cudaStream_t stream, int sms) {
    static int resident = 0;
    if (!resident) {
        int per_sm = 0;
        const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_refine<MODE, LANES>,
                                                                            kRefineWarps * 32, kRefineSmem<LANES>);
        if (e != cudaSuccess) return e;
        resident = per_sm > 0 ? per_sm : 1;
    }
    // A warp takes 32 slots at a time, or as few as give every resident warp a chunk.
    const int64_t warps = (int64_t)sms * resident * kRefineWarps;
    const int chunk = (int)std::max<int64_t>(1, std::min<int64_t>(32, (n + warps - 1) / warps));
    const int64_t want = (n + (int64_t)chunk * kRefineWarps - 1) / ((int64_t)chunk * kRefineWarps);
    const int ctas = (int)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)sms * resident));
    k_refine<MODE, LANES><<<ctas, kRefineWarps * 32, kRefineSmem<LANES>, stream>>>(
        G, d, s, p, out, errors, st, n, chunk, counter, images, map);
    return cudaGetLastError();
}

// The pass over n slots.  Few blocks leave the GPU idle while each runs its
// passes one after another, so they take more lanes (us for the whole call at
// level 9, 32 / 8 / 4 lanes a block: 64 x 64 64 / 70 / 80; 4,000 float blocks
// of the hard mixture 147 / 166 / 196, 10,000 215 / 203 / 235, 40,000 539 /
// 376 / 402, 200,000 1797 / 1203 / 1171; 1024 x 1024 328 / 314 / 323, 4096 x
// 4096 3920 / 3800 / 3773; a block a lane one step at a time: 133 us for 64 x
// 64's pass alone).  n counts slots, with something to refine or not.
template <int MODE>
static cudaError_t refine_pass(const GlobalTables *G, const ImageDesc &d, const BlocksSrc &s, const EncodeParams &p,
                               uint2 *out, float *errors, const RefineSlot *st, int64_t n, unsigned long long *counter,
                               const ImageDesc *images, RefineMap map, cudaStream_t stream, int sms) {
    if (n < 8192) return refine_launch<MODE, 32>(G, d, s, p, out, errors, st, n, counter, images, map, stream, sms);
    if (n < 98304) return refine_launch<MODE, 8>(G, d, s, p, out, errors, st, n, counter, images, map, stream, sms);
    return refine_launch<MODE, 4>(G, d, s, p, out, errors, st, n, counter, images, map, stream, sms);
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
