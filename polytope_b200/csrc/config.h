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
// faces): 4 visits 5190 / 427 / 562, 1: 5450 / 464 / 578, 2: 5357 / 438 / 568, 8: 5387 / 438 / 605; at 4
// visits, 6 blocks (80 registers, spills) 5484 / 437 / 586, 4 blocks 5696 / 447 / 552; leaf batch 12
// 5280 / 427 / 554, 20 5328 / 441 / 590.
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
// be tested, and a lane may test a second leaf at once.  1 k rays 26.9 -> 25.6 us, 100 k on box faces 97 ->
// 95, 1 M occlusion rays 565 -> 517, 16.7 M rays 5187 -> 5128 (the path kernel's 1920x1080x16 frame, a
// second leaf only: 9.24 -> 9.12 ms).  With all rays a second leaf costs 7 % on 16.7 M.  A batch of 16 there
// gives 25.7 / 92.5 / 540 / 5119, of 4 27.4 / 95.7 / 505 / 5161; four leaves 25.7 / 93.1 / 543 / 5135; 8
// visits between votes 25.5 / 91.5 / 543 / 5147 at 16.  Two-level queries are 1 % slower with it and keep
// the constants above.
#ifndef PT_WIDE_LAST_BATCH
#define PT_WIDE_LAST_BATCH 8
#endif
#ifndef PT_WIDE_LAST_LEAVES
#define PT_WIDE_LAST_LEAVES 2
#endif

// Resident blocks of 128 and leaf batch of the extend and shadow kernels (wf_wide_kernel).  Their rays come
// from one wave and are alike, so more warps pay although the walk spills (72 registers, about 150 B).
// Measured on a B200 (ms, four renders of depth 6; scenes of 500 k box faces / 20 k box faces / instanced
// spheres, 33.5 M paths in one wave; the binary walk's kernel 61.0 / 65.0 / 16.1): 7 blocks and 12 59.5 /
// 66.0 / 12.9, 6 and 12 60.5 / 67.0 / 13.1, 8 and 12 60.6 / 66.6 / 13.0, 5 and 16 65.3 / 71.0 / 13.6; with
// waves of 4.2 M paths (binary 9.39 / 9.89 / 4.75) 8.68 / 9.30 / 2.93, 5 and 16 9.20 / 9.73 / 2.92.
#ifndef PT_WIDE_WF_BLOCKS
#define PT_WIDE_WF_BLOCKS 7
#endif
#ifndef PT_WIDE_WF_BATCH
#define PT_WIDE_WF_BATCH 12
#endif

// The same for the persistent path kernel (wf_wide_path_kernel), with the lanes that must have a ray to
// end or start, or a hit to shade, before those steps run.  Measured on a B200 (ms; 1920x1080x16 frame
// of 3.9 M faces / 641x479x4 frame of 20 k box faces / 24 served requests), before the binary walk's
// kernel and after: 12.9 / 3.35 / 9.0 -> 9.4 / 2.7 / 6.1 (9.1 / 2.5 / 5.9 with the last paths handed out in
// small lots, wide_take).  One visit between votes 9.5 / 3.0 / 6.5; 4 blocks
// 10.2 / 2.85 / 6.2, 6 blocks 9.4 / 2.7 / 6.1 (one visit: 11.1 / 3.3 / 7.1); turns from 4 or 16 lanes on
// within 2 %, shading from 10 or 24 lanes on 3 to 7 % slower on the first.
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
// persistent kernel), over the binary trees before 633 / 14.5: 4 blocks 338 / 5.8, 3 blocks 390 / 7.6, 5
// blocks 417 / 6.6, 6 blocks 473 / 7.5; entering from 4 or 16 lanes on within 2 %.
#ifndef PT_WIDE_TL_BLOCKS
#define PT_WIDE_TL_BLOCKS 4
#endif
#ifndef PT_WIDE_ENTERS
#define PT_WIDE_ENTERS 8
#endif

// Paths per bounce up to which a wave over four-wide records runs as whole paths in the persistent path
// kernel instead of bounce by bounce: a bounce costs six launches, each as long as its slowest ray, which
// few paths don't cover.  Bounce by bounce / whole paths on a B200 (ms; eight scenes of 20 k faces each):
// depth 0 (one bounce), 131 k paths 0.13 / 0.13, 524 k 0.26 / 0.27; depth 2, 131 k 0.65 / 0.48, 393 k 0.93 /
// 0.90, 786 k 1.44 / 1.49; depth 6, 131 k 1.04 / 0.57, 917 k 2.16 / 1.95; depth 12, 131 k 3.11 / 1.24, 2.1 M
// 7.66 / 6.89.  Scenes of 1 k faces gain more, of 500 k faces the same; far above the line the waves are
// 8 % ahead (24 uneven renders, 24.5 against 26.3).
#ifndef PT_WIDE_WAVE_PATHS
#define PT_WIDE_WAVE_PATHS (1u << 17)
#endif
