/* Built-in launch shapes of the batched solver, one entry per size class:
 * {threads per CTA, persistent CTAs per SM, grid cap (0 = none)}.
 *
 * Generated by jacobi-svd-cuda_b200/batch_autotune.py on NVIDIA B200
 * (148 SMs), 2026-12-05, from jsvd_batch_autotune over 20000 FP32-stored matrices m ~ U{16..256}, n ~ U{8..m} (seed 3);
 * 2 runs per shape, L2 flushed before each, minimum kept.  A shape
 * replaces the previous built-in one only when it is more than 2% faster.
 *
 * class: members timed / in batch, shapes tried, ms previous -> chosen
 *   0 (A and V in <= 48 KiB of shared memory): 7599 / 7599, 9 shapes, 8.81 -> 8.81
 *   1 (A and V in <= 100 KiB of shared memory): 3383 / 3383, 6 shapes, 26.27 -> 26.27
 *   2 (A and V in <= ~226 KiB of shared memory): 3932 / 3932, 3 shapes, 115.45 -> 115.45
 *   3 (A in shared memory, V in global memory): 2550 / 2550, 9 shapes, 218.30 -> 218.30
 *   4 (A and V in global memory): 2536 / 2536, 9 shapes, 709.05 -> 709.05
 *
 * CTAs per matrix: the classes whose bit is set in JSVD_BATCH_CLUSTER_CLASSES
 * are solved by a thread-block cluster per matrix (2, 4 or 8 CTAs; class 3
 * only while its members are few), the others by one CTA per matrix; a class
 * goes over only when that is more than 2% faster.
 * Timed on the same batch, all classes, mean of 3 runs, L2 flushed.
 * class: ms one CTA per matrix, ms clusters -> chosen
 *   2: 115.5, 160.7 -> one CTA
 *   3: 218.6, 218.4 -> clusters
 *   4: 752.8, 709.1 -> clusters
 */
#pragma once

#define JSVD_BATCH_TUNING_TABLE \
    { {128, 4, 0}, {256, 2, 0}, {512, 1, 0}, {512, 1, 0}, {512, 1, 0} }

#define JSVD_BATCH_CLUSTER_CLASSES 0x18
