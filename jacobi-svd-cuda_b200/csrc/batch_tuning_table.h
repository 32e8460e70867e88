/* Built-in launch shapes of the batched solver, one entry per size class:
 * {threads per CTA, persistent CTAs per SM, grid cap (0 = none)}.
 *
 * Generated by jacobi-svd-cuda_b200/batch_autotune.py on NVIDIA B200
 * (148 SMs), 2026-12-03, from jsvd_batch_autotune over 4000 FP32-stored matrices m ~ U{16..256}, n ~ U{8..m} (seed 3);
 * 2 runs per shape, L2 flushed before each, minimum kept.  A shape
 * replaces the previous built-in one only when it is more than 2% faster.
 *
 * class: members timed / in batch, shapes tried, ms previous -> chosen
 *   0 (A and V in <= 48 KiB of shared memory): 7400 / 7400, 5 shapes, 6.41 -> 5.71
 *   1 (A and V in <= 100 KiB of shared memory): 3610 / 3610, 5 shapes, 14.88 -> 14.88
 *   2 (A and V in <= ~226 KiB of shared memory): 397 / 397, 3 shapes, 17.68 -> 17.68
 *   3 (A in shared memory, V in global memory): 485 / 485, 9 shapes, 76.49 -> 76.49
 *   4 (A and V in global memory): 506 / 506, 9 shapes, 240.89 -> 240.89
 * (classes 0 and 1 on 2026-12-05 over 11,010 FP32-stored members of the same
 * distribution, class 2 over 2000; classes 3 and 4 as generated)
 *
 * CTAs per matrix: the classes whose bit is set in JSVD_BATCH_CLUSTER_CLASSES
 * are solved by a thread-block cluster per matrix (2, 4 or 8 CTAs; class 3
 * only while its members are few), the others by one CTA per matrix; a class
 * goes over only when that is more than 2% faster.
 * Timed on NVIDIA B200 (148 SMs), 2026-12-05, over 2000 FP32-stored matrices (m ~ U{16..256}, n ~ U{8..m}), all classes, mean of 3 runs.
 * class: ms one CTA per matrix, ms clusters -> chosen
 *   2: 17.6, 22.7 -> one CTA
 *   3: 25.3 -> clusters while few
 *   4: 119.5, 95.7 -> clusters
 */
#pragma once

#define JSVD_BATCH_TUNING_TABLE \
    { {128, 4, 0}, {256, 2, 0}, {512, 1, 0}, {512, 1, 0}, {512, 1, 0} }

#define JSVD_BATCH_CLUSTER_CLASSES 0x18
