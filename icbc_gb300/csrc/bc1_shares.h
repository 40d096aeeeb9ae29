// bc1_shares.h -- how work is shared out: blocks per warp or CTA, blocks per
// task of a batch, bands of a host-buffer call.  Plain arithmetic on counts,
// for host and device code alike.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define ICBC_HD __host__ __device__
#else
#define ICBC_HD
#endif

namespace icbc_gpu {

// How many of n blocks a worker (a warp of 32 lanes, or a CTA) takes at a
// time when `workers` share them: as few as the rounds they need anyway allow,
// at most `most`.  A last round that is nearly empty costs as much as a full
// one, and an image too small for 32 blocks a warp leaves most SMs without a
// warp while the others run long ones (the cluster search spreads a warp's
// blocks over its 32 lanes however many they are).  Against 32 blocks a warp
// always, in us: level 8 at 64 x 64 187 -> 48, 512 x 512 194 -> 116, 2048 x
// 2048 (the 16-warp CTAs' last round) 1018 -> 826, 4096 x 4096 3342 -> 3114;
// with a weight plane 1000 x 600 431 -> 237; 40,000 float blocks 303 -> 155.
// A warp takes at least `least` blocks: below level 4, where the search is a
// small part of a block's work, warps with few blocks only add lanes without
// one (level 3 at 1024 x 1024: 45 us with 16, 51 with 1; level 7 at 64 x 64:
// 79 with 16, 48 with 1).
ICBC_HD constexpr int balanced_share(int64_t n, int64_t workers, int most, int least) {
    const int64_t rounds = (n + workers * most - 1) / (workers * most);
    const int64_t share = rounds < 1 ? 1 : (n + workers * rounds - 1) / (workers * rounds);
    return (int)(share < least ? least : share);
}
ICBC_HD constexpr int least_per_warp(int level) { return level >= 4 ? 1 : 16; }

// The share of an image's n blocks.  Below level 4 an image of more than one
// round of the workers takes 32 a warp: its warps take much the same time
// however few blocks they have, so even rounds only make more of them (levels
// 2 / 3, even / 32, us: 1100 x 1100 with a weight plane 55 / 51 and 60 / 56,
// 1448 x 1448 of the hard mixture 322 / 305 and 317 / 314).  Float blocks keep
// even rounds (65,000 of the mixture at level 2 199, 218 with 32 a warp).
ICBC_HD constexpr int image_share(int64_t n, int64_t workers, int level) {
    return level < 4 && n > workers * 32 ? 32 : balanced_share(n, workers, 32, least_per_warp(level));
}

// How a batch is cut into tasks and launched, per level.
//
// A task is a warp's work, and its time grows with its blocks where the search
// is most of it: levels 8-9 take as few blocks a task as give each task a warp
// of its own (20,000 blocks at level 8 128 us, with 32 a task 204; 50,000 with
// a weight plane, whose kernel has 12 warps an SM instead of 16, 300 with 28
// or 32, but 411 in two rounds of 21).  At levels 0-1, where there is none, a
// warp takes the same time for 1 block as for 32, and smaller tasks only share
// the SMs with more of them (20,000 blocks at level 1: 12.5 us, 17.2 with 9 a
// task).  Between them the gain depends on the content: levels 2-5 take
// smaller tasks only while they leave most warps without one (3/8: 20,000
// smooth blocks at level 3 46 us with 17 to 32 a task and 58 with 9, of the
// hard mixture 145, 168 and 140), levels 6-7 down to 8 blocks.
//
// With several levels in a batch their kernels share the SMs.  Levels 8-9 are
// then the longest, and small tasks at the others stand in their way: 80,000
// blocks of all levels 192 us, 371 with one size of task for all.  They leave a
// quarter of the warps to the others, and take no more than 16 blocks while
// all of them would fit in one round of 32 (200,000 blocks of all levels: 327
// us with 16, 414 with 32; 400,000 of levels 6-9: 971 with 16, 886 with 32).
//
// 8-warp CTAs search for their 8 tasks together: better at levels 6-9 from few
// blocks a task on (level 8, 4 / 8 warps: 1,500 blocks 48 / 57 us, 10,000 111 /
// 94, 400,000 1310 / 1211), at levels 2-5 only beside those (levels 3-6, 160,000
// blocks: 127 us with 8 warps at level 6 alone, 94 at all four; level 4 alone
// 133 / 148 at 400,000), and with few blocks in all not at all.
struct BatchShape {
    int task_blocks[10];  // blocks per task, 1 to 32
    int cta_warps[10];    // 8: the CTA-wide kernel, 4: a warp a task
};
// From the images' levels and block counts and the resident warps of the GPU;
// level_kernels: byte rows, a kernel per level, all at once (else one kernel
// takes the tasks of every level, most expensive first).
inline BatchShape batch_shape(const int *levels, const int64_t *blocks, int n, int64_t warps, bool level_kernels) {
    BatchShape s;
    const auto tasks = [&](int lo, int hi, int size) {
        int64_t t = 0;
        for (int i = 0; i < n; i++)
            if (levels[i] >= lo && levels[i] <= hi) t += (blocks[i] + size - 1) / size;
        return t;
    };
    // The smallest size from `size` on that makes at most `room` tasks, else `most`.
    const auto fit = [&](int lo, int hi, int size, int most, int64_t room) {
        while (size < most && tasks(lo, hi, size) > room) size++;
        return size;
    };
    const auto set = [&](int lo, int hi, int size, bool wide) {
        for (int l = lo; l <= hi; l++) s.task_blocks[l] = size, s.cta_warps[l] = level_kernels && wide ? 8 : 4;
    };
    const bool mixed = tasks(0, 7, 32) > 0;
    const int heavy = !mixed          ? fit(8, 9, 1, 32, warps)
                      : level_kernels ? fit(8, 9, 2, tasks(8, 9, 1) <= 32 * warps ? 16 : 32, 3 * warps / 4)
                                      : fit(8, 9, 1, 32, warps / 2);
    const int64_t heavy_tasks = tasks(8, 9, heavy);
    set(8, 9, heavy, heavy >= 2);  // 2 at least when mixed
    int64_t used = heavy_tasks + tasks(0, 1, 32);
    const int mid = fit(6, 7, level_kernels ? 8 : 4, 32, warps - used - tasks(2, 5, 32));
    const int64_t mid_tasks = tasks(6, 7, mid);
    const int64_t light = tasks(2, 5, 1);
    const bool wide = mid > 8 || heavy_tasks > 0 || (light > 0 && light + tasks(6, 7, 1) >= 6 * warps);
    set(6, 7, mid, wide);
    used += mid_tasks;
    set(2, 5, fit(2, 5, 1, 32, 3 * warps / 8 - used), heavy_tasks > 0 || (mid_tasks > 0 && wide));
    set(0, 1, 32, false);
    return s;
}

// Bands that a host-buffer call cuts an image of `blocks` blocks into: enough
// to overlap the upload, most of the light levels' call, with the encode, but
// each large enough for the encoder, for which blocks count and not rows.  In
// us, by bands: level 1, 16384 x 512 272 (1) 239 (2) 222 (5) 223 (8); 2048 x
// 2048 155 (1) 128 (4) 140 (8); 1024 x 1024 60 (1) 58 (2) 65 (4).  Level 3, 4096
// x 4096 508 (1) 438 (4) 423 (6).  Level 8, 2048 x 2048 897 (1) 849 (3) 876 (4);
// 4096 x 4096 3343 / 3100 / 3093; level 9 3992 / 3777 / 3761.
//
// Levels 4-7 take bands that one CTA-wide pass takes whole (512 blocks an SM,
// one_cta_pass) where that makes at most five: level 4, 2048 x 2048 194 (1) 193
// (2) 204 (3) 177 (4); 2400 x 2400 239 (1) 216 (2) 237 (3) 213 (5).  Above, large
// ones at levels 4-5, which list their blocks again (4096 x 4096 at level 5 603
// (2) 553 (4) 529 (6)), and five at levels 6-7, each of which leaves its last
// round's SMs to the next (level 6 823 (2) 756 (4) 728 (5) 742 (8)).
inline int host_bands(int level, int64_t blocks, int sms) {
    constexpr int64_t k = 1024;
    const auto bands = [&](int64_t first, int64_t each, int most) {
        const int64_t b = blocks / each;
        return blocks < first ? 1 : b < 2 ? 2 : b < most ? (int)b : most;
    };
    if (level < 2) return bands(48 * k, 64 * k, 5);
    if (level < 4) return blocks < 640 * k ? bands(80 * k, 64 * k, 4) : bands(0, 160 * k, 6);
    if (level >= 8) return bands(96 * k, 80 * k, 4);
    const int64_t whole = (blocks + 512 * (int64_t)sms - 1) / (512 * (int64_t)sms);
    if (whole <= 5) return (int)whole;
    return level >= 6 ? 5 : bands(0, 160 * k, 6);
}

}  // namespace icbc_gpu
