// config.h -- compile-time limits shared by host and device code.
#pragma once

// Traversal stack entries per ray.  The reference's ordered DFS needs at most (tree depth + 1)
// entries; pt_scene_create records the depth and calls refuse trees that do not fit.
#define PT_TRAVERSAL_STACK 64
// Top-level stack entries of a two-level scene (pt_scene_create_two_level refuses deeper trees).
#define PT_TOP_STACK 64

// Warp rounds of the persistent walks (walk_round, traverse.cuh): the lanes of a warp take node
// steps together until this many of them hold a leaf or have ended their walk (32 = every walking
// lane), then test faces together; 0 walks each lane on its own to its next leaf instead (no vote,
// fewer live registers).  One value per kernel: the ray-query kernel, the persistent path kernel
// and the wavefront extend/shadow kernel.  Measured on a B200 (each against the per-lane walk):
// ray queries on the 1.3 M-face microbench 1722 -> 1985 Mrays/s at 16 (12: 1937, 24: slower);
// whole paths on the 6.5 M-face frame 1595 -> 1678 Msamples/s at 12 (8 and 16 slower); the
// wavefront kernel on the 256-scene batch 1806 -> 2024 Mrays/s at 12 with its first 16 stack
// entries in shared memory (16: 1954, 20: 1801; with the stack in local memory the vote lost 17 %
// at this kernel's 64 registers).
#ifndef PT_LEAF_BATCH_TRACE
#define PT_LEAF_BATCH_TRACE 16
#endif
#ifndef PT_LEAF_BATCH_PATHS
#define PT_LEAF_BATCH_PATHS 12
#endif
#ifndef PT_LEAF_BATCH_WAVEFRONT
#define PT_LEAF_BATCH_WAVEFRONT 12
#endif

// Persistent path kernel (wf_path_kernel): lanes whose ray has ended wait until this many lanes of
// the warp can shade together (or no lane still walks), and the resident-block floor given to the
// register allocator (blocks of 128 threads per SM).  With the lighter node steps (the box form
// chosen per warp round, sign-mask child order, paired pushes) 7 blocks (72 registers) overtook 8
// on a B200: the 6.5 M-face frame 1884-1888 against 1800-1805 Msamples/s, the saturated serving mix
// 4624 against 4411 Mrays/s (the 256-scene plain frames 1551 against 1567); 6 blocks (80
// registers) 1847 and 4574; shade batches of 12 or 24 measured 1706 / 1703 (at 8 blocks).
#ifndef PT_SHADE_BATCH_PATHS
#define PT_SHADE_BATCH_PATHS 16
#endif
#ifndef PT_PATH_MIN_BLOCKS
#define PT_PATH_MIN_BLOCKS 7
#endif

// Walks over four-wide records: resident blocks of 128 threads a SM, lanes at a leaf before faces are
// tested, ended lanes before new rays are taken, and visits a lane makes between votes.  Measured on a
// B200 (us; 16.7 M rays on 1.3 M faces / 1 M rays on 100 k box faces / 1 M occlusion rays on 330 k
// faces): 4 visits 4926 / 500 / 483, 1: 5293 / 523 / 511, 2: 5126 / 513 / 493, 8: 5082 / 520 / 517; at 4
// visits, 4 blocks 5778 / 566 / 516, 6 blocks (80 registers) 4590 / 478 / 477, but 37.2 against 36.6 on 1 k
// rays (chosen when the walk spilled there, 5484 against 5190 on the first); leaf batch 12 5039 / 498 /
// 478, 20 5011 / 514 / 497.
#ifndef PT_WIDE_BLOCKS
#define PT_WIDE_BLOCKS 5
#endif
#ifndef PT_WIDE_BATCH
#define PT_WIDE_BATCH 16
#endif
#ifndef PT_WIDE_REFILL
#define PT_WIDE_REFILL 8
#endif
#ifndef PT_WIDE_STEPS
#define PT_WIDE_STEPS 4
#endif
// A warp that has no more rays to take is as slow as its slowest lane: there fewer lanes wait for faces to
// be tested, and a lane may test a second leaf at once.  1 k rays 36.6 us, 100 k on box faces 94.7, 1 M
// occlusion rays 483, 16.7 M rays 4926; a batch of 16 there, as elsewhere, gives 48.5 / 97.0 / 499 / 4921, of 4
// 36.5 / 95.0 / 467 / 4930; one leaf 36.9 / 92.6 / 491 / 4936, four 39.1 / 95.9 / 483 / 4930.  (With all rays,
// and before the frames were halved, a second leaf cost 7 % on 16.7 M; two-level queries were 1 % slower with
// these and keep the constants above.)
#ifndef PT_WIDE_LAST_BATCH
#define PT_WIDE_LAST_BATCH 8
#endif
#ifndef PT_WIDE_LAST_LEAVES
#define PT_WIDE_LAST_LEAVES 2
#endif

// Resident blocks of 128 and leaf batch of the extend and shadow kernels (wf_wide_kernel).  Their rays come
// from one wave and are alike, so more warps pay although the walk spills (72 registers, about 100 B;
// launched with 256 threads they are three blocks of those a SM, 80 registers, and as fast).  Measured on
// a B200 (ms, four renders of depth 6; scenes of 500 k box faces / 20 k box faces / instanced spheres,
// 33.5 M paths in one wave; the binary walk's kernel 52.2 / 74.1 / 38.5): 7 blocks and 12 46.1 / 69.0 /
// 29.4, 6 and 12 46.5 / 69.9 / 30.0, 8 and 12 47.5 / 69.5 / 29.3, 5 and 16 48.6 / 72.1 / 30.9; with waves of
// 4.2 M paths 6.50 / 9.55 / 5.25, 5 and 16 6.68 / 9.85 / 5.32.
#ifndef PT_WIDE_WF_BLOCKS
#define PT_WIDE_WF_BLOCKS 7
#endif
#ifndef PT_WIDE_WF_BATCH
#define PT_WIDE_WF_BATCH 12
#endif

// The same for the persistent path kernel (wf_wide_path_kernel), with the lanes that must have a ray to
// end or start, or a hit to shade, before those steps run.  Measured on a B200 (ms; 1920x1080x16 frame
// of 3.9 M faces / 641x479x4 frame of 20 k box faces / 24 served requests): 8.34 / 2.39 / 6.1 (the binary
// walk's kernel about 1.4 times that).  One visit between votes 8.77 / 2.68 / 6.55; 4 blocks 9.22 / 2.54 /
// 6.41, 6 blocks 8.60 / 2.55 / 6.44; turns from 4 lanes on 8.52 / 2.44 / 6.28, from 16 8.33 / 2.40 / 6.10 (and
// 320x240x8 frames 5 % slower); shading from 10 lanes on 9.08 / 2.40 / 6.30, from 24 8.48 / 2.46 / 6.14.
#ifndef PT_WIDE_PATH_BLOCKS
#define PT_WIDE_PATH_BLOCKS 5
#endif
#ifndef PT_WIDE_BATCH_PATHS
#define PT_WIDE_BATCH_PATHS 12
#endif
#ifndef PT_WIDE_TURNS
#define PT_WIDE_TURNS 8
#endif
#ifndef PT_WIDE_SHADES
#define PT_WIDE_SHADES 16
#endif
#ifndef PT_WIDE_PATH_STEPS
#define PT_WIDE_PATH_STEPS 4
#endif

// Two-level scenes over four-wide records (queries and the persistent path kernel): resident blocks, and
// lanes that must stand at an instance or an exit before those steps run.  Measured on a B200 (us, 1 M rays
// on five instances of 82 k faces / ms, 1280x720x8 frame of five instances of 330 k faces through the
// persistent kernel, 33.6 over the binary trees): 4 blocks 324 / 12.8, 3 blocks 370 / 15.0, 5 blocks 351 /
// 13.4, 6 blocks 386 / 15.4; entering from 4 lanes on 328 / 12.9, from 16 356 / 14.1.
#ifndef PT_WIDE_TL_BLOCKS
#define PT_WIDE_TL_BLOCKS 4
#endif
#ifndef PT_WIDE_ENTERS
#define PT_WIDE_ENTERS 8
#endif

// Paths per bounce up to which a wave over four-wide records runs as whole paths in the persistent path
// kernel instead of bounce by bounce: a bounce costs six launches, each as long as its slowest ray, which
// few paths don't cover.  Bounce by bounce / whole paths on a B200 (ms; eight scenes of 20 k faces each):
// depth 0 (one bounce), 131 k paths 0.15 / 0.15, 524 k 0.26 / 0.25; depth 2, 131 k 0.54 / 0.43, 390 k 0.84 /
// 0.80, 783 k 1.27 / 1.32; depth 6, 131 k 1.22 / 0.80, 913 k 2.70 / 2.57; depth 12, 131 k 2.07 / 1.17, 2.1 M
// 6.69 / 6.28.  Far above the line the waves were 8 % ahead (24 uneven renders, 24.5 against 26.3).
#ifndef PT_WIDE_WAVE_PATHS
#define PT_WIDE_WAVE_PATHS (1u << 17)
#endif
