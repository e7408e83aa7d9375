#pragma once
// ---------------------------------------------------------------------------
// bh_launch_rules.h -- how the tile kernel's launch goes by the frame's size (plain C++:
// shared by bh_trace.cu and the CPU tests).
// ---------------------------------------------------------------------------

// Whether the hole and its disk leave most of the view empty: the half height of the view at the
// hole's distance against the disk's outer radius (no disk: 0) or 16 M.  Then few warps hold the long
// rays, and the frame lasts as long as they do; otherwise nearly all do, and the frame's work counts.
inline bool bh_wide_view(float distance, float tanHalfFov, float M, float diskOuter)
{
    const float reach = 16.f * M > diskOuter ? 16.f * M : diskOuter;
    return distance * tanHalfFov >= 1.2f * reach;
}

// Rays a warp of the tile kernel takes at a time; `known`: the host knows the number of rays.
// A small frame lasts as long as the warp of its longest rays, and a warp's steps cost the union
// of its lanes' paths (disk samples above all, which come at different steps); while there are few
// warps, fewer rays a warp shorten that.  The smallest power of two that makes at most 8192 (a
// wide view) or 1024 groups.  With the warps below, us of one wide view at 32 / 16 / 8 / 4 / 2 / 1 rays a
// warp: Kerr-Newman orbit 128 x 72 1133 / 981 / 869 / 858 / 668 / 778 (2 taken), 320 x 180 1651 / 1518 / 1423 /
// 1568 / 2008 / 3885 (8 taken), 480 x 270 1589 / 1409 / 1520 / 2294 (16 taken), 640 x 360 1688 / 1632 / 2115 (32
// taken); Reissner-Nordstroem 128 x 72 729 -> 355, 320 x 180 672 -> 575.  Close views at the width of 8192
// groups ran at 0.55 .. 0.97 of their speed at 32, at that of 1024 groups at 0.96 and more.
// Means over 14 random views a size, 96 x 54 .. 640 x 360, against 32 rays and all the warps that fit:
// 1.02 .. 1.43x, mixed precision 1.01 .. 1.52x; least view 0.96x.
// (A list whose length only the device knows is traced 32 at a time.)
inline int bh_rays_per_warp(unsigned rays, bool known, bool wide)
{
    int width = 32;
    if (known)
        while (width > 1 && ((unsigned long long)rays * 2u) / (unsigned)width <= (wide ? 8192u : 1024u)) width >>= 1;
    return width;
}

// Warps an SM of the tile kernel for a small or middling frame (0: as many as fit).  Up to some
// tens of thousands of tiles a frame ends with a few warps whose rays go round the hole; those
// started first and ran all the while next to 25 .. 28 others, so fewer warps an SM let them
// through sooner (1283 x 719 Reissner-Nordstroem: the queue empty at 1.17 ms, the last warp,
// begun at 0, at 1.77).  Geometric means (least) over 16 random views, against all that fit:
// spherical 96 x 54 .. 640 x 360 at 12 warps 1.04 .. 1.08x (0.86, where the hole fills the view) and at 16
// 1.03 .. 1.06x (0.91), 800 x 450 and 960 x 540 at 16 1.03 .. 1.06x (0.91), 1040 x 585 .. 1283 x 719 at 20
// 1.03 .. 1.04x (0.95), 1500 x 843 at 20 1.00x (not taken); rotating up to 128 x 72 at 10 1.06 .. 1.09x
// (0.97), 240 x 135 .. 960 x 540 at 15 1.03 .. 1.07x (0.97), 1283 x 719 at 15 0.99x (not taken).  Mixed
// precision: 1.02 .. 1.10x (0.87).  The anchors of a surrogate frame, 640 x 360 .. 4K: 0.99 .. 1.03x.
inline int bh_warps_per_sm(unsigned rays, bool known, bool kerr, bool wide)
{
    if (!known) return 0;
    const unsigned tiles = rays / 32u;
    if (tiles <= 512u && kerr) return 10;
    if (tiles <= 8192u && !kerr) return wide ? 12 : 16;
    if (tiles <= 16384u) return kerr ? 15 : 16;
    return tiles <= 32768u && !kerr ? 20 : 0;
}

// Resident CTAs an SM: as many as fit (`fit`), but no more than the rule's warps nor than
// bhSetTuning's number (each 0: no limit).  A set number is a limit and does not turn the rule
// off: the autotuner sets one for all later frames of the family from the one frame it timed, and
// with a 4K frame's number in the rule's place a 128 x 72 frame took 481 us instead of 442.
inline int bh_blocks_per_sm(int fit, int ruleWarps, int warpsPerBlock, int set)
{
    int n = fit < 1 ? 1 : fit;
    if (ruleWarps > 0 && ruleWarps / warpsPerBlock < n) n = ruleWarps / warpsPerBlock;
    if (set > 0 && set < n) n = set;
    return n < 1 ? 1 : n;
}
