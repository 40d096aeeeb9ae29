// bc1_level.cu -- encoder kernels of one quality level.
//
// Compiled once per level with -DICBC_LEVEL=<0..9> so the ten
// specialisations build in parallel.  -fmad=false keeps every multiply and
// add separately rounded, as the reference's scalar build does.
#include <cuda_runtime.h>

#include <algorithm>

#include "bc1_batch_task.cuh"

#ifndef ICBC_LEVEL
#error "compile with -DICBC_LEVEL=<0..9>"
#endif

namespace icbc_gpu {

// ------------------------------------------------------------- kernels --

// With DEFER (level 9 only) refinement is left to k_refine: the kernel
// records each block's starting error and whether refinement applies.
template <int L, bool DEFER>
__global__ void __launch_bounds__(kWarpsPerCta * 32) k_encode_blocks(const GlobalTables *G, BlocksSrc s, EncodeParams p,
                                                                     uint2 *out, float *errors, int64_t n, int per_warp,
                                                                     RefineSlot *st) {
    extern __shared__ __align__(16) unsigned char smem[];
    SharedTables &T = *reinterpret_cast<SharedTables *>(smem);
    stage_tables(T, G);
    const WarpCtx w = warp_ctx<L>(smem, T, G, p.decoder);
    if (L < 2) per_warp = 32;  // a constant: these kernels take microseconds
    const int64_t groups = (n + per_warp - 1) / per_warp;
    for (int64_t g = (int64_t)blockIdx.x * kWarpsPerCta + (threadIdx.x >> 5); g < groups;
         g += (int64_t)gridDim.x * kWarpsPerCta) {
        const int64_t base = g * per_warp;
        const int nb = (int)(n - base < per_warp ? n - base : per_warp);
        __syncwarp();
        load_float_blocks(s, base, nb, w.in, w.lane);
        __syncwarp();
        const bool active = w.lane < nb;
        const int64_t b = base + w.lane;
        uint32_t c0 = 0, c1 = 0, idx = 0;
        if (L >= 4 && active) {
            const uint2 prev = out[b];
            c0 = prev.x & 0xffff;
            c1 = prev.x >> 16;
            idx = prev.y;
        }
        bool pending;
        const float e = encode_warp_ex<L, DEFER>(w, float_row(w), p, active, c0, c1, idx, pending);
        if (active) {
            out[b] = make_uint2(c0 | (c1 << 16), idx);
            if (errors) errors[b] = e;
            if (DEFER) st[b] = RefineSlot{e, pending ? 1u : 0u};
        }
    }
}

// Levels 0-1 take ImageRows: one 16-byte load a texel and pass instead of four
// loads, the chosen palette entry by a load instead of a 4-way select, four
// texels at a time in flight (2: 2% slower, 8: 12%, 16: 70%, instruction
// fetch).  Bound by issue (3,580 instructions a warp, 4,330 before): 4096 x
// 4096 at level 1 134 us, before 161; at level 0 80, before 93.
template <int L, bool DEFER>
__global__ void __launch_bounds__(kWarpsPerCta * 32) k_encode_image(const GlobalTables *G, ImageDesc d, EncodeParams p,
                                                                    int per_warp, RefineSlot *st) {
    extern __shared__ __align__(16) unsigned char smem[];
    SharedTables &T = *reinterpret_cast<SharedTables *>(smem);
    WarpCtx w;
    if constexpr (L < 2) {
        stage_color_tables(T, G);
        w = warp_ctx_image(smem, T, G, p.decoder);
    } else {
        stage_tables(T, G);
        w = warp_ctx<L>(smem, T, G, p.decoder);
    }
    if (L < 2) per_warp = 32;
    const int64_t groups = (d.nblocks + per_warp - 1) / per_warp;
    for (int64_t g = (int64_t)blockIdx.x * kWarpsPerCta + (threadIdx.x >> 5); g < groups;
         g += (int64_t)gridDim.x * kWarpsPerCta) {
        const int64_t b = g * per_warp + w.lane;
        const bool active = w.lane < per_warp && b < d.nblocks;
        __syncwarp();
        if (active) {
            if constexpr (L < 2) load_image_row(d, b, w.sat + w.lane * kSatStride, T.lut255);
            else load_image_block(d, b, w.in + w.lane * kInStride, T.lut255);
        }
        __syncwarp();
        uint32_t c0 = 0, c1 = 0, idx = 0;
        if (L >= 4 && active) {
            const uint2 prev = d.out[b];
            c0 = prev.x & 0xffff;
            c1 = prev.x >> 16;
            idx = prev.y;
        }
        bool pending;
        float e;
        if constexpr (L < 2) e = encode_warp_ex<L, DEFER>(w, image_row(w), p, active, c0, c1, idx, pending);
        else e = encode_warp_ex<L, DEFER>(w, float_row(w), p, active, c0, c1, idx, pending);
        if (active) {
            d.out[b] = make_uint2(c0 | (c1 << 16), idx);
            if (d.errors) d.errors[b] = e;
            if (DEFER) st[b] = RefineSlot{e, pending ? 1u : 0u};
        }
    }
}

// k_encode_image with byte texel rows, for RGBA8 images with uniform or alpha
// weights at levels 2..9: 11 KB of shared memory per warp and at most 128
// registers per thread, so four CTAs (16 warps) fit on an SM instead of three.
template <int L, bool DEFER>
__global__ void __launch_bounds__(kWarpsPerCta * 32, 4) k_encode_image_bytes(const GlobalTables *G, ImageDesc d,
                                                                             EncodeParams p, int per_warp,
                                                                             RefineSlot *st) {
    extern __shared__ __align__(16) unsigned char smem[];
    SharedTables &T = *reinterpret_cast<SharedTables *>(smem);
    stage_tables(T, G);
    const WarpCtx w = warp_ctx_byte_rows(smem, T, G, p.decoder);
    const ByteRow row = byte_row(w, d.weight_mode == ICBC_GPU_WEIGHTS_ALPHA);
    const int64_t groups = (d.nblocks + per_warp - 1) / per_warp;
    for (int64_t g = (int64_t)blockIdx.x * kWarpsPerCta + (threadIdx.x >> 5); g < groups;
         g += (int64_t)gridDim.x * kWarpsPerCta) {
        const int64_t b = g * per_warp + w.lane;
        const bool active = w.lane < per_warp && b < d.nblocks;
        __syncwarp();
        if (active) load_image_block_bytes(d, b, reinterpret_cast<uint32_t *>(w.in) + w.lane * kInWordsByte);
        __syncwarp();
        uint32_t c0 = 0, c1 = 0, idx = 0;
        if (L >= 4 && active) {
            const uint2 prev = d.out[b];
            c0 = prev.x & 0xffff;
            c1 = prev.x >> 16;
            idx = prev.y;
        }
        bool pending;
        const float e = encode_warp_ex<L, DEFER>(w, row, p, active, c0, c1, idx, pending);
        if (active) {
            d.out[b] = make_uint2(c0 | (c1 << 16), idx);
            if (d.errors) d.errors[b] = e;
            if (DEFER) st[b] = RefineSlot{e, pending ? 1u : 0u};
        }
    }
}

// Levels 2..9 in two passes (RGBA8 images, byte rows).  Many blocks reduce
// to 0 or 1 colours (on the quality-sweep image 99% at level 2, 86% at level
// 4, 61% at level 5, 21-29% at levels 6-9), and a warp with one other block
// among them runs that block's whole cluster fit with some lanes idle (with
// one lane busy at the low levels).  Pass 1 finishes the blocks of 0 or 1
// colours and lists the rest; pass 2 runs the full encoder over the list, 32
// listed blocks per warp.  Each block's computation is the single-pass one
// (pass 2 reduces again).  Levels 2-4 take half the time, levels 5-8 2-25%
// less.
// Pass 1 needs only to tell blocks of 0 or 1 reduced colours from the rest.
// Levels 8-9 compare bytes (one_byte_colour).  Levels 2-7 follow reduce_colors
// (icbc.h:1683-1728) only while one colour has been kept: the texels and the
// running colour stay in registers (a ByteRow over a register array, every
// index known at compile time), and a block is listed as soon as a second
// colour appears.  For the blocks it finishes the arithmetic is reduce_colors'
// (every texel merged into the first colour).  Shared memory holds only the i / 255 table; six CTAs per SM
// (80 registers) beat both four (126 registers) and eight (more spills).
template <int L>
__global__ void __launch_bounds__(kWarpsPerCta * 32, 6) k_image_trivial(const GlobalTables *G, ImageDesc d, EncodeParams p,
                                                                     uint32_t *list, unsigned int *listed,
                                                                     RefineSlot *st) {
    __shared__ float lut[256];
    for (int i = threadIdx.x; i < 256; i += blockDim.x) lut[i] = G->s.lut255[i];
    __syncthreads();
    const DecoderTables *D = &G->dec[p.decoder];
    const int lane = threadIdx.x & 31;
    const int alpha = d.weight_mode == ICBC_GPU_WEIGHTS_ALPHA;
    const int64_t groups = (d.nblocks + 31) / 32;
    for (int64_t g = (int64_t)blockIdx.x * kWarpsPerCta + (threadIdx.x >> 5); g < groups;
         g += (int64_t)gridDim.x * kWarpsPerCta) {
        const int64_t b = g * 32 + lane;
        const bool active = b < d.nblocks;
        bool other = false;
        if (active) {
            uint32_t px[16];
            fetch_image_block(d, b, px);
            const ByteRow row{px, lut, alpha};
            V3 c;
            int count;
            other = L >= 8 ? !one_byte_colour(px, lut, alpha, c, count)
                           : !reduce_to_one(row, Level<L>::threshold, c, count);
            if (!other) {
                uint32_t c0, c1, idx;
                const float e = trivial_block<16>(D, lut, row, p, c, count, c0, c1, idx);
                d.out[b] = make_uint2(c0 | (c1 << 16), idx);
                if (d.errors) d.errors[b] = e;
                if (st) st[b] = RefineSlot{e, 0u};  // level 9: nothing to refine
            }
        }
        const unsigned m = __ballot_sync(kFull, other);
        if (m) {
            unsigned base = 0;
            if (lane == 0) base = atomicAdd(listed, (unsigned)__popc(m));
            base = __shfl_sync(kFull, base, 0);
            if (other) list[base + __popc(m & ((1u << lane) - 1u))] = (uint32_t)b;
        }
    }
}

template <int L, bool DEFER>
__global__ void __launch_bounds__(kWarpsPerCta * 32, 4) k_image_listed(const GlobalTables *G, ImageDesc d,
                                                                       EncodeParams p, const uint32_t *list,
                                                                       const unsigned int *listed, RefineSlot *st) {
    const int64_t n = *listed;
    const int per_warp = image_share(n, (int64_t)gridDim.x * kWarpsPerCta, L);
    const int64_t groups = (n + per_warp - 1) / per_warp;
    if ((int64_t)blockIdx.x * kWarpsPerCta >= groups) return;  // the whole CTA has no work
    extern __shared__ __align__(16) unsigned char smem[];
    SharedTables &T = *reinterpret_cast<SharedTables *>(smem);
    stage_tables(T, G);
    const WarpCtx w = warp_ctx_byte_rows(smem, T, G, p.decoder);
    const ByteRow row = byte_row(w, d.weight_mode == ICBC_GPU_WEIGHTS_ALPHA);
    for (int64_t g = (int64_t)blockIdx.x * kWarpsPerCta + (threadIdx.x >> 5); g < groups;
         g += (int64_t)gridDim.x * kWarpsPerCta) {
        const int64_t k = g * per_warp + w.lane;
        const bool active = w.lane < per_warp && k < n;
        const int64_t b = active ? (int64_t)list[k] : 0;
        __syncwarp();
        if (active) load_image_block_bytes(d, b, reinterpret_cast<uint32_t *>(w.in) + w.lane * kInWordsByte);
        __syncwarp();
        uint32_t c0 = 0, c1 = 0, idx = 0;
        if (L >= 4 && active) {
            const uint2 prev = d.out[b];
            c0 = prev.x & 0xffff;
            c1 = prev.x >> 16;
            idx = prev.y;
        }
        bool pending;
        const float e = encode_warp_ex<L, DEFER>(w, row, p, active, c0, c1, idx, pending);
        if (active) {
            d.out[b] = make_uint2(c0 | (c1 << 16), idx);
            if (d.errors) d.errors[b] = e;
            if (DEFER) st[b] = RefineSlot{e, pending ? 1u : 0u};
        }
    }
}

// k_image_listed with the CTA as the unit: NW warps take 32 * NW listed
// blocks at a time and move through the encoder's stages together -- colour
// reduction and summed-area tables one block per lane, then the cluster
// searches over all the CTA's blocks at once (flat_search_group), then the
// output blocks.  All warps of an SM run the same stage's code at the same
// time, and a search balances over 32 * NW blocks instead of 32.  Same
// arithmetic and the same winner per block as k_image_listed.  Shared memory:
// the tables, then the CTA's byte rows, SAT rows and the sentinel's SAT row,
// argmin slots, info words with the sentinel's (padded to 16 bytes) and NW
// scan sums (group_smem_bytes).
template <int NW>
__host__ __device__ constexpr size_t group_smem_bytes() {
    return sizeof(SharedTables) + (size_t)NW * 32 * (kInWordsByte * 4 + kSatStride * 4 + 8 + 4) + NW * 4 +
           kSatStride * 4 + 16;
}

// The batched CTA-wide kernel's layout: the group layout (16-byte aligned
// size), NW 16-byte round keys, the round's tasks and their number.
template <int NW>
__host__ __device__ constexpr size_t batch_smem_bytes() {
    return group_smem_bytes<NW>() + NW * 16 + (NW + 4) * 4;
}
static_assert(group_smem_bytes<8>() % 16 == 0 && group_smem_bytes<16>() % 16 == 0, "round keys need 16-byte alignment");

// The warp's and the CTA's contexts in the group layout, and the scan sums.
template <int NW>
__device__ __forceinline__ void group_ctx(unsigned char *smem, const SharedTables &T, const DecoderTables *D,
                                          WarpCtx &w, WarpCtx &g, int *&sums) {
    uint32_t *in = reinterpret_cast<uint32_t *>(smem + sizeof(SharedTables));
    float *sat = reinterpret_cast<float *>(in + NW * 32 * kInWordsByte);
    unsigned long long *slots = reinterpret_cast<unsigned long long *>(sat + (NW * 32 + 1) * kSatStride);
    int *info = reinterpret_cast<int *>(slots + NW * 32);
    sums = info + NW * 32 + 4;
    // The group search's sentinel block (flat_search_group), read only after
    // the search's first barrier.
    const float nan = __int_as_float(0x7fffffff);
    if (threadIdx.x < 17) st4(sat + NW * 32 * kSatStride + 4 * threadIdx.x, make_float4(nan, nan, nan, nan));
    if (threadIdx.x == 0) info[NW * 32] = 16 << kInfoShift;
    const int warp = threadIdx.x >> 5;
    g.T = &T;
    g.D = D;
    g.in = reinterpret_cast<float *>(in);
    g.sat = sat;
    g.slots = slots;
    g.info = info;
    g.lane = threadIdx.x;
    w = g;
    w.in = reinterpret_cast<float *>(in + warp * 32 * kInWordsByte);
    w.sat = sat + warp * 32 * kSatStride;
    w.slots = slots + warp * 32;
    w.info = info + warp * 32;
    w.lane = threadIdx.x & 31;
}

template <int L, bool DEFER, int NW>
__global__ void __launch_bounds__(NW * 32, 512 / (NW * 32))
    k_image_listed_cta(const GlobalTables *G, ImageDesc d, EncodeParams p, const uint32_t *list,
                       const unsigned int *listed, RefineSlot *st) {
    // Up to level 7: no list (one_cta_pass) means every block of the image, and
    // a band of a larger image leaves its last round's SMs to the next band.
    constexpr bool WHOLE = L <= 7;
    const int64_t n = WHOLE && !list ? d.nblocks : (int64_t)*listed;
    const int per_cta = WHOLE && d.overlapped && n > (int64_t)gridDim.x * 32 * NW
                            ? 32 * NW
                            : balanced_share(n, gridDim.x, 32 * NW, 1);
    const int64_t groups = (n + per_cta - 1) / per_cta;
    if ((int64_t)blockIdx.x >= groups) return;  // the whole CTA has no work
    extern __shared__ __align__(16) unsigned char smem[];
    SharedTables &T = *reinterpret_cast<SharedTables *>(smem);
    stage_tables(T, G);
    WarpCtx w, g;
    int *sums;
    group_ctx<NW>(smem, T, &G->dec[p.decoder], w, g, sums);
    uint32_t *in = reinterpret_cast<uint32_t *>(g.in);
    const ByteRow row = byte_row(w, d.weight_mode == ICBC_GPU_WEIGHTS_ALPHA);
    for (int64_t grp = blockIdx.x; grp < groups; grp += gridDim.x) {
        const int64_t k = grp * per_cta + threadIdx.x;
        const bool active = (int)threadIdx.x < per_cta && k < n;
        const int64_t b = !active ? 0 : WHOLE && !list ? k : (int64_t)list[k];
        __syncwarp();
        if (active) load_image_block_bytes(d, b, in + threadIdx.x * kInWordsByte);
        __syncwarp();
        uint32_t c0 = 0, c1 = 0, idx = 0;
        if (L >= 4 && active) {
            const uint2 prev = d.out[b];
            c0 = prev.x & 0xffff;
            c1 = prev.x >> 16;
            idx = prev.y;
        }
        bool pending;
        const float e = encode_warp_ex<L, DEFER, false, NW>(w, row, p, active, c0, c1, idx, pending, &g, sums);
        if (active) {
            d.out[b] = make_uint2(c0 | (c1 << 16), idx);
            if (d.errors) d.errors[b] = e;
            if (DEFER) st[b] = RefineSlot{e, pending ? 1u : 0u};
        }
    }
}

// k_batch_level with the CTA as the unit: the CTA takes NW tasks at a time
// (one per warp; past the end of the queue a warp has no blocks, but its
// threads still walk the round's combinations) and moves through the
// encoder's stages together, the cluster searches over all its blocks at
// once -- when every task of the round has the same decoder and colour
// weights (every walker must use the same fit weights); otherwise each warp
// searches its own blocks that round.  Levels 2-9 of a byte-row batch; at
// level 9 every image refines in k_refine's batch mode (the planner gives
// each level-9 image of the shared kernel a slot range).
template <int LV, int NW>
__global__ void __launch_bounds__(NW * 32, 512 / (NW * 32))
    k_batch_level_cta(const GlobalTables *G, const ImageDesc *images, const BatchTask *tasks, int task0, int ntasks,
                      int *counter, const int64_t *refine_base, RefineSlot *slots, BatchLists lists) {
    extern __shared__ __align__(16) unsigned char smem[];
    SharedTables &T = *reinterpret_cast<SharedTables *>(smem);
    stage_tables(T, G);
    WarpCtx w, g;
    int *sums;
    group_ctx<NW>(smem, T, &G->dec[0], w, g, sums);
    // Round state past the group layout (batch_smem_bytes): each warp's
    // (decoder, colour weights), then its tasks and their number.
    uint4 *warp_key = reinterpret_cast<uint4 *>(smem + group_smem_bytes<NW>());
    int *round = reinterpret_cast<int *>(warp_key + NW);
    uint32_t *in = reinterpret_cast<uint32_t *>(g.in);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (;;) {
        // Warp 0 draws tasks until the round has one for every warp or the
        // queue is empty; those past their list's end have nothing to do and
        // take no place in it (400,000 blocks at level 6 292 us with NW tasks
        // a round as they come, 280 so; of the hard mixture 1295 and 1212).
        if (warp == 0) {
            int have = 0;
            for (bool more = true; have < NW && more;) {
                const int want = NW - have;
                int t = 0;
                if (lane == 0) t = atomicAdd(counter, want);
                t = __shfl_sync(kFull, t, 0);
                more = t + want < ntasks;
                t += lane;
                bool useful = lane < want && t < ntasks;
                if (useful && lists.list) {
                    const BatchTask c = tasks[task0 + t];
                    useful = lists.list_base[c.image] < 0 || c.first_block < lists.listed[c.image];
                }
                const unsigned m = __ballot_sync(kFull, useful);
                if (useful) round[have + __popc(m & ((1u << lane) - 1u))] = t;
                have += __popc(m);
            }
            if (lane == 0) round[NW] = have;
        }
        __syncthreads();
        const int have = round[NW];
        if (have == 0) break;
        const bool has_task = warp < have;
        const BatchTask task = has_task ? load_task(tasks + task0 + round[warp]) : BatchTask{};
        const ImageDesc &d = images[task.image];
        const int64_t lb = lists.list ? lists.list_base[task.image] : -1;
        int64_t b = (int64_t)task.first_block + lane;
        bool active = has_task && lane < (int)task.blocks && b < d.nblocks;
        if (has_task && lb >= 0) {
            const int64_t n = lists.listed[task.image];
            active = lane < (int)task.blocks && b < n;  // tasks past the list's end: finished by the first pass
            b = active ? (int64_t)lists.list[lb + b] : 0;
        }
        if (lane == 0)
            warp_key[warp] = has_task ? make_uint4((uint32_t)d.decoder, __float_as_uint(d.cw[0]),
                                                   __float_as_uint(d.cw[1]), __float_as_uint(d.cw[2]))
                                      : make_uint4(0xffffffffu, 0u, 0u, 0u);
        __syncthreads();
        // One search over the CTA when every warp with a task has the same key.
        bool group = true;
        uint4 first = make_uint4(0xffffffffu, 0u, 0u, 0u);
#pragma unroll
        for (int k = 0; k < NW; k++) {
            const uint4 v = warp_key[k];
            if (v.x == 0xffffffffu) continue;
            if (first.x == 0xffffffffu) first = v;
            group &= v.x == first.x && v.y == first.y && v.z == first.z && v.w == first.w;
        }
        // Every thread walks the group's combinations with its own fit
        // weights, so a warp without a task takes the round's (decoder,
        // colour weights); warp 0 always has a task.
        EncodeParams p;
        p.decoder = has_task ? d.decoder : (int)first.x;
        p.three_color_mode = d.three_color_mode;
        p.three_color_black = d.three_color_black;
        p.cw = has_task ? v3(d.cw[0], d.cw[1], d.cw[2])
                        : v3(__uint_as_float(first.y), __uint_as_float(first.z), __uint_as_float(first.w));
        w.D = &G->dec[p.decoder];
        const ByteRow row = byte_row(w, d.weight_mode == ICBC_GPU_WEIGHTS_ALPHA);
        __syncwarp();
        if (active) load_image_block_bytes(d, b, in + threadIdx.x * kInWordsByte);
        __syncwarp();
        uint32_t c0 = 0, c1 = 0, idx = 0;
        if (LV >= 4 && active) {
            const uint2 prev = d.out[b];
            c0 = prev.x & 0xffff;
            c1 = prev.x >> 16;
            idx = prev.y;
        }
        bool pending = false;
        const float e = encode_warp_ex<LV, LV == 9, false, NW>(w, row, p, active, c0, c1, idx, pending, &g, sums,
                                                                group);
        if (active) {
            d.out[b] = make_uint2(c0 | (c1 << 16), idx);
            if (d.errors) d.errors[b] = e;
            if (LV == 9) slots[refine_base[task.image] + b] = RefineSlot{e, pending ? 1u : 0u};
        }
        __syncthreads();  // round and warp_key are rewritten next round
    }
}

// The batched form's kernel for this level's tasks of a byte-row batch:
// run_batch with the level fixed, so the kernel holds one level's code as the
// plain kernels do (the all-levels kernel stalls about twice as often on
// instruction fetch for the same blocks).
template <int LV>
__global__ void __launch_bounds__(kWarpsPerCta * 32, 4)
    k_batch_level(const GlobalTables *G, const ImageDesc *images, const BatchTask *tasks, int task0, int ntasks,
                  int *counter, const int64_t *refine_base, RefineSlot *slots, BatchLists lists) {
    extern __shared__ __align__(16) unsigned char smem[];
    run_batch<true, LV>(G, smem, images, tasks, nullptr, 0, task0, ntasks, counter, refine_base, slots, lists);
}

constexpr int L = ICBC_LEVEL;

// CTAs for n blocks and the blocks a warp takes at a time.  An image of many
// rounds takes the level's launch shape: every warp takes groups_per_warp
// groups of 32 blocks; a persistent grid is exactly the resident CTAs (from
// the occupancy API), each warp striding over the image, otherwise there are
// enough CTAs for the work and the hardware balances them (better when block
// costs vary, as they do from level 2 on).  From level 2 on, one of fewer than
// kBalancedRounds rounds gives each warp one group of a balanced size.
constexpr int kBalancedRounds = 8;
template <class K>
static int grid_for(K kernel, int64_t n, int sms, size_t smem, int &resident, bool image = true,
                    int *per_warp = nullptr) {
    const LaunchShape shape = launch_shape(L);
    if (!resident) {
        int per_sm = 0;
        if (smem) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kWarpsPerCta * 32, smem) != cudaSuccess ||
            per_sm < 1)
            per_sm = 1;
        resident = per_sm;
    }
    const int64_t cap = (int64_t)sms * resident;
    if (per_warp) {
        *per_warp = 32;
        if (L >= 2 && n < cap * kWarpsPerCta * 32 * kBalancedRounds) {
            *per_warp = image ? image_share(n, cap * kWarpsPerCta, L)
                              : balanced_share(n, cap * kWarpsPerCta, 32, least_per_warp(L));
            return (int)((n + (int64_t)*per_warp * kWarpsPerCta - 1) / ((int64_t)*per_warp * kWarpsPerCta));
        }
    }
    const int64_t groups = (n + 31) / 32;
    const int64_t per_cta = (int64_t)kWarpsPerCta * shape.groups_per_warp;
    int64_t ctas = (groups + per_cta - 1) / per_cta;
    if (shape.persistent) {
        const int64_t all = (groups + kWarpsPerCta - 1) / kWarpsPerCta;
        ctas = all < cap ? all : cap;
    }
    return (int)(ctas < 1 ? 1 : ctas < 0x7fffffff ? ctas : 0x7fffffff);
}

#define ICBC_CAT2(a, b) a##b
#define ICBC_CAT(a, b) ICBC_CAT2(a, b)

// Level 9 encodes in two launches: the encoder without refinement, then
// k_refine, handing over through a RefineSlot per block in stream-ordered
// scratch.  Other levels are one launch.
constexpr bool kDefer = Level<L>::refine;

// The level-9 hand-over lives in stream-ordered scratch, or in the caller's
// `ext_st` (n slots) and `ext_counter` when given (graph captures, where
// nothing is allocated).
template <class Kernel, class Launch>
static cudaError_t run(Kernel kernel, size_t smem, int &resident, int64_t n, int sms, cudaStream_t stream,
                       Launch launch, const GlobalTables *G, const ImageDesc *image, const BlocksSrc *blocks,
                       const EncodeParams &p, uint2 *out, float *errors, RefineSlot *ext_st = nullptr,
                       unsigned long long *ext_counter = nullptr) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int per_warp = 32;
    const int grid = grid_for(kernel, n, sms, smem, resident, image != nullptr, &per_warp);
    if (!kDefer) {
        launch(grid, smem, per_warp, nullptr);
        return cudaGetLastError();
    }
    void *scratch = nullptr;
    RefineSlot *st = ext_st;
    unsigned long long *counter = ext_counter;
    if (!st) {
        const size_t slots = ((size_t)n * sizeof(RefineSlot) + 15) / 16 * 16;
        e = scratch_alloc(&scratch, slots + 16, stream);
        if (e != cudaSuccess) return e;
        st = reinterpret_cast<RefineSlot *>(scratch);
        counter = reinterpret_cast<unsigned long long *>(static_cast<char *>(scratch) + slots);
    }
    e = cudaMemsetAsync(counter, 0, sizeof(unsigned long long), stream);
    if (e == cudaSuccess) {
        launch(grid, smem, per_warp, st);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = launch_refine(G, image, blocks, p, out, errors, st, n, counter, stream, sms);
    if (!scratch) return e;
    const cudaError_t f = scratch_free(scratch, stream);
    return e != cudaSuccess ? e : f;
}

// Resident CTAs per SM of each kernel (persistent launch shapes), found once.
static int g_resident_blocks = 0, g_resident_image = 0;

#if ICBC_LEVEL >= 2  // the cluster-fit levels, up to `#endif`
static_assert(Level<L>::cluster, "");

// Byte rows apply to the cluster-fit levels and to RGBA8 weights (uniform or
// alpha); weight planes need float rows.
static bool use_byte_rows(const ImageDesc &d) { return d.weight_mode != ICBC_GPU_WEIGHTS_PLANE; }

static int g_resident_bytes = 0, g_resident_trivial = 0, g_resident_listed = 0, g_resident_listed8 = 0;
static int g_resident_listed16 = 0, g_resident_batch8 = 0, g_resident_batch16 = 0;

// The listed pass's CTA size at this level: the launch shape's, else the
// level's default -- 4 warps at levels 2-3, whose short lists gain nothing from
// CTA-wide searches, 8 at levels 4-5, 16 above.  Where few blocks are listed, a
// 16-warp CTA has work for a few of its warps only: level 4 with 16 / 8 warps,
// 1448 x 1448 60 / 55 us, one seventh of it textured 75 / 61 (4 warps 50), the
// hard mixture 269 / 272; 4096 x 4096 203 / 200, 1794 / 1792; at levels 6-7 16 is
// 2% faster on the mixture and as fast on the others.
static int listed_cta_warps() {
    const int c = launch_shape(L).cta_warps;
    if (c == 4 || c == 8 || c == 16) return c;
    return L >= 6 ? 16 : L >= 4 ? 8 : 4;
}

// The CTA size for an image of `nblocks` blocks.  A CTA-wide pass shares the
// blocks out evenly over the resident CTAs (balanced_share), so it pays from
// few blocks a warp on: 8-warp CTAs from 96 blocks an SM (512 x 512 at level 7
// 66 us, 4-warp CTAs 78; 1024 x 1024 at levels 6 / 8 76 / 241 us, 4-warp 88 /
// 269; at 256 x 256, 27 an SM, 4-warp CTAs are 2-10% faster), 16-warp ones
// from a full round of them on (2048 x 2048 at levels 6 / 8 197 / 825 us,
// 8-warp 203 / 845; at 768 x 768 8-warp CTAs are 2-7% faster).
static int listed_cta_warps(int64_t nblocks, int sms) {
    const int c = listed_cta_warps();
    if (c == 16 && nblocks >= (int64_t)sms * 32 * 16) return 16;
    return c > 4 && nblocks >= (int64_t)sms * 96 ? 8 : 4;
}

// The batched form's per-level kernel's CTA size: the launch shape's, else the
// batch's plan (batch_shape): 8 where the CTA's stages in step keep the long
// per-block code in the instruction cache (300 images of 64 to 2048 a side,
// all levels: 7.21 ms with 4-warp CTAs, 6.23 with 8, 6.43 with 16; 400 of the
// mixed batch 6.53 / 6.34 / 6.45).
static int batch_cta_warps(int planned) {
    const int c = launch_shape(L).batch_cta_warps;
    return c == 4 || c == 8 || c == 16 ? c : planned;
}

// Whether the CTA-wide pass takes all of an image's blocks instead of a list,
// at levels 4-7: up to 512 blocks an SM, 900 at levels 6-7, where the first
// pass costs more (its allocation, memset and wait included) than it keeps out
// of the CTA's stages.  With / without, us: level 5 at 512 x 512 37 / 51, 1100
// x 1100 45 / 57, 1448 x 1448 82 / 70; level 7 49 / 62, 81 / 92, 140 / 154,
// 2048 x 2048 283 / 271.  At levels 8-9, where a CTA's blocks of 0 or 1
// colours unbalance the searches, the list stays (level 8 at 1100 x 1100 274 /
// 252).
static bool one_cta_pass(int64_t nblocks, int sms) {  // L <= 7: k_image_listed_cta's WHOLE
    return L >= 4 && L <= 7 && nblocks < (int64_t)sms * (L >= 6 ? 900 : 512);
}

// Shared-memory limit of a listed-pass kernel and, once, its resident CTAs per SM.
template <class K>
static cudaError_t listed_attributes(K kernel, int warps, size_t smem, int *resident) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess && !*resident) {
        int per_sm = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, warps * 32, smem);
        *resident = per_sm > 0 ? per_sm : 1;
    }
    return e;
}

// The two passes -- the CTA-wide one alone for smaller images (one_cta_pass) --
// with the list (and at level 9 the refinement hand-over, unless the caller
// gives one) in stream-ordered scratch; level 9 then runs its refinement pass
// over every block.
static cudaError_t launch_image_compacted(const GlobalTables *G, const ImageDesc &d, const EncodeParams &p,
                                          cudaStream_t stream, int sms, RefineSlot *ext_st,
                                          unsigned long long *ext_counter) {
    const int cta_warps = listed_cta_warps(d.nblocks, sms);
    const size_t smem = cta_warps == 16 ? group_smem_bytes<16>()
                        : cta_warps == 8 ? group_smem_bytes<8>()
                                         : smem_bytes_byte_rows();
    cudaError_t e = cudaSuccess;
    int *resident = cta_warps == 16 ? &g_resident_listed16 : cta_warps == 8 ? &g_resident_listed8 : &g_resident_listed;
    if (cta_warps == 16) e = listed_attributes(k_image_listed_cta<L, kDefer, 16>, 16, smem, resident);
    else if (cta_warps == 8) e = listed_attributes(k_image_listed_cta<L, kDefer, 8>, 8, smem, resident);
    else e = listed_attributes(k_image_listed<L, kDefer>, kWarpsPerCta, smem, resident);
    if (e != cudaSuccess) return e;
    const bool listing = cta_warps == 4 || !one_cta_pass(d.nblocks, sms);
    const size_t list_bytes = listing ? ((size_t)d.nblocks * 4 + 15) / 16 * 16 + 16 : 0;
    const size_t slot_bytes = (kDefer && !ext_st) ? ((size_t)d.nblocks * sizeof(RefineSlot) + 15) / 16 * 16 + 16 : 0;
    void *scratch = nullptr;
    if (list_bytes + slot_bytes) e = scratch_alloc(&scratch, list_bytes + slot_bytes, stream);
    if (e != cudaSuccess) return e;
    char *base = static_cast<char *>(scratch);
    uint32_t *list = listing ? reinterpret_cast<uint32_t *>(base) : nullptr;
    unsigned int *listed = listing ? reinterpret_cast<unsigned int *>(base + list_bytes - 16) : nullptr;
    RefineSlot *st = ext_st;
    unsigned long long *counter = ext_counter;
    if (kDefer && !ext_st) {
        st = reinterpret_cast<RefineSlot *>(base + list_bytes);
        counter = reinterpret_cast<unsigned long long *>(base + list_bytes + slot_bytes - 16);
    }
    if (listing) e = cudaMemsetAsync(listed, 0, sizeof(unsigned int), stream);
    if (e == cudaSuccess && kDefer) e = cudaMemsetAsync(counter, 0, sizeof(unsigned long long), stream);
    if (e == cudaSuccess && listing) {
        const int grid = grid_for(k_image_trivial<L>, d.nblocks, sms, 0, g_resident_trivial);
        k_image_trivial<L><<<grid, kWarpsPerCta * 32, 0, stream>>>(G, d, p, list, listed, kDefer ? st : nullptr);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
        // Persistent over the list, whose length only the device knows.
        const int per_cta = cta_warps == 4 ? kWarpsPerCta * least_per_warp(L) : 32;
        const int64_t most = ((int64_t)d.nblocks + per_cta - 1) / per_cta;
        const int64_t cap = (int64_t)sms * *resident;
        const int grid = (int)(most < cap ? most : cap);
        if (cta_warps == 16)
            k_image_listed_cta<L, kDefer, 16><<<grid, 16 * 32, smem, stream>>>(G, d, p, list, listed, st);
        else if (cta_warps == 8)
            k_image_listed_cta<L, kDefer, 8><<<grid, 8 * 32, smem, stream>>>(G, d, p, list, listed, st);
        else
            k_image_listed<L, kDefer><<<grid, kWarpsPerCta * 32, smem, stream>>>(G, d, p, list, listed, st);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess && kDefer) e = launch_refine(G, &d, nullptr, p, d.out, d.errors, st, d.nblocks, counter, stream, sms);
    const cudaError_t f = scratch ? scratch_free(scratch, stream) : cudaSuccess;
    return e != cudaSuccess ? e : f;
}

// Whether an image of `nblocks` blocks is encoded in one pass of 4-warp CTAs.
// Two passes keep blocks of 0 or 1 colours out of the searching warps, but
// cost a scratch allocation, a memset and a second kernel that waits for the
// first.  One pass below 96 blocks an SM, where the CTA-wide kernels begin;
// at levels 2-3, which do not take those, up to 512.  One / two passes, us:
// level 3 at 64 x 64 22 / 35, 1024 x 1024 33 / 40, 1448 x 1448 60 / 44; level
// 6 27 / 41; level 8 30 / 43, 384 x 384 84 / 88, 512 x 512 115 / 105.
static bool one_pass(int64_t nblocks, int sms) { return nblocks < (int64_t)sms * (L >= 4 ? 96 : 512); }

// Whether launch_image_compacted's kernels take the image.
static bool compacted(const ImageDesc &d, int sms) {
    return use_byte_rows(d) && d.nblocks < (int64_t(1) << 32) && !one_pass(d.nblocks, sms);
}
#endif

static cudaError_t launch_image(const GlobalTables *G, const ImageDesc &d, const EncodeParams &p, cudaStream_t stream,
                                int sms, RefineSlot *ext_st, unsigned long long *ext_counter) {
#if ICBC_LEVEL >= 2
    if (compacted(d, sms)) return launch_image_compacted(G, d, p, stream, sms, ext_st, ext_counter);
    if (use_byte_rows(d))
        return run(k_encode_image_bytes<L, kDefer>, smem_bytes_byte_rows(), g_resident_bytes, d.nblocks, sms, stream,
                   [&](int grid, size_t smem, int per_warp, RefineSlot *slots) {
                       k_encode_image_bytes<L, kDefer><<<grid, kWarpsPerCta * 32, smem, stream>>>(G, d, p, per_warp, slots);
                   },
                   G, &d, nullptr, p, d.out, d.errors, ext_st, ext_counter);
#endif
    return run(k_encode_image<L, kDefer>, L < 2 ? smem_bytes_image() : smem_bytes(Level<L>::cluster), g_resident_image, d.nblocks, sms, stream,
               [&](int grid, size_t smem, int per_warp, RefineSlot *slots) {
                   k_encode_image<L, kDefer><<<grid, kWarpsPerCta * 32, smem, stream>>>(G, d, p, per_warp, slots);
               },
               G, &d, nullptr, p, d.out, d.errors, ext_st, ext_counter);
}

// The kernels launch_image takes and what of the launch shape reaches them.
icbc_gpu_launch_info ICBC_CAT(image_plan_l, ICBC_LEVEL)(const ImageDesc &d, int sms) {
    int per_warp = 32;
#if ICBC_LEVEL >= 2
    if (compacted(d, sms)) {
        const int cta_warps = listed_cta_warps(d.nblocks, sms);
        if (cta_warps != 4 && one_cta_pass(d.nblocks, sms)) return {1, cta_warps, 0};
        return {2, cta_warps, grid_for(k_image_trivial<L>, d.nblocks, sms, 0, g_resident_trivial)};
    }
    if (use_byte_rows(d))
        return {1, kWarpsPerCta, grid_for(k_encode_image_bytes<L, kDefer>, d.nblocks, sms, smem_bytes_byte_rows(),
                                          g_resident_bytes, true, &per_warp)};
#endif
    const int grid = grid_for(k_encode_image<L, kDefer>, d.nblocks, sms,
                              L < 2 ? smem_bytes_image() : smem_bytes(Level<L>::cluster), g_resident_image, true, &per_warp);
    return {1, kWarpsPerCta, grid};
}

cudaError_t ICBC_CAT(launch_blocks_l, ICBC_LEVEL)(const GlobalTables *G, const BlocksSrc &s, const EncodeParams &p,
                                                  void *out, float *errors, int64_t n, cudaStream_t stream, int sms) {
    uint2 *o = reinterpret_cast<uint2 *>(out);
    return run(k_encode_blocks<L, kDefer>, smem_bytes(Level<L>::cluster), g_resident_blocks, n, sms, stream,
               [&](int grid, size_t smem, int per_warp, RefineSlot *st) {
                   k_encode_blocks<L, kDefer><<<grid, kWarpsPerCta * 32, smem, stream>>>(G, s, p, o, errors, n, per_warp, st);
               },
               G, nullptr, &s, p, o, errors);
}

cudaError_t ICBC_CAT(launch_batch_level_l, ICBC_LEVEL)(const GlobalTables *G, const ImageDesc *images,
                                                        const BatchTask *tasks, int task0, int ntasks, int planned_warps,
                                                        int *counter, cudaStream_t stream, int grid, const int64_t *refine_base,
                                                        RefineSlot *slots, BatchLists lists) {
#if ICBC_LEVEL >= 2
    // `grid` counts 4-warp CTAs; a CTA-wide kernel gets as many warps in all.
    const int cta_warps = L < 9 || refine_base ? batch_cta_warps(planned_warps) : 4;
    if (cta_warps != 4) {
        const size_t smem = cta_warps == 16 ? batch_smem_bytes<16>() : batch_smem_bytes<8>();
        int *resident = cta_warps == 16 ? &g_resident_batch16 : &g_resident_batch8;
        cudaError_t e = cta_warps == 16 ? listed_attributes(k_batch_level_cta<L, 16>, 16, smem, resident)
                                        : listed_attributes(k_batch_level_cta<L, 8>, 8, smem, resident);
        if (e != cudaSuccess) return e;
        const int want = (grid * kWarpsPerCta + cta_warps - 1) / cta_warps;
        const int ctas = std::max(1, std::min(want, current_sm_count() * *resident));
        if (cta_warps == 16)
            k_batch_level_cta<L, 16><<<ctas, 16 * 32, smem, stream>>>(G, images, tasks, task0, ntasks, counter,
                                                                       refine_base, slots, lists);
        else
            k_batch_level_cta<L, 8><<<ctas, 8 * 32, smem, stream>>>(G, images, tasks, task0, ntasks, counter,
                                                                     refine_base, slots, lists);
        return cudaGetLastError();
    }
#endif
    const size_t smem = smem_bytes_byte_rows();
    cudaError_t e = cudaFuncSetAttribute(k_batch_level<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k_batch_level<L><<<grid, kWarpsPerCta * 32, smem, stream>>>(G, images, tasks, task0, ntasks, counter, refine_base,
                                                               slots, lists);
    return cudaGetLastError();
}

cudaError_t ICBC_CAT(launch_image_l, ICBC_LEVEL)(const GlobalTables *G, const ImageDesc &d, const EncodeParams &p,
                                                 cudaStream_t stream, int sms) {
    return launch_image(G, d, p, stream, sms, nullptr, nullptr);
}

// As launch_image_l<L>, with level 9's hand-over in the caller's memory
// (d.nblocks slots and a counter; unused at the other levels).
cudaError_t ICBC_CAT(launch_image_ext_l, ICBC_LEVEL)(const GlobalTables *G, const ImageDesc &d, const EncodeParams &p,
                                                     cudaStream_t stream, int sms, RefineSlot *st,
                                                     unsigned long long *counter) {
    return launch_image(G, d, p, stream, sms, st, counter);
}

}  // namespace icbc_gpu
