// Batched solves of many small systems of uneven size (n <= 256, k <= 8) in one persistent
// launch: float32 LU with partial pivoting + float64 refinement per system, falling back to a
// float64 LU for the systems whose refinement stalls, all inside the same kernel.
//
// rustymath solves a stack of systems one LuWork per thread (Stacked::solve,
// src/linalg/stacked.rs:88-101, over parallel::stack, core/src/parallel.rs:118-192), each an
// lu_factor + lu_solve (core/src/linalg/factor.rs:617-641) and, when `regular` fails
// (factor.rs:221-226), least squares. Here a CTA takes one system at a time from a shared
// counter (systems sorted by size, largest first, so the long ones start early) and:
//   - loads A (float64, row-major) into a float32 working copy W in its own slice of a global
//     scratch (W stays in L2 while the CTA works on it); thread r owns row r;
//   - factors W with partial pivoting, implicitly: rows never move, a row chosen as pivot of
//     logical column c records pos = c and leaves the candidates; in panels of NB columns
//     (16 or 32, picked per size bucket by the tuner) each thread keeps its row's panel in
//     registers and each column costs one barrier (every warp posts its best candidate row,
//     every thread picks the winner among the posts: largest |pivot|, lowest row on ties, NaN
//     never chosen over a number); then U12 of the panel's pivot rows (a column per thread)
//     and the update of the rows not chosen yet;
//   - solves L U x = P b with the rows' right-hand sides in registers, block by block (a warp
//     per right-hand side solves each NB x NB diagonal block with shuffles);
//   - refines in float64: r = b - A x (a warp per row of A, x in shared memory), the normwise
//     backward error max_c ||r_c|| / (||A|| ||x_c|| + ||b_c||), and corrections from the
//     float32 factors until it is at most the tolerance (n * 2^-53 by default);
//   - on a stall (the error not halving) or the step limit, redoes the system in float64
//     (the same code on float64 items, reusing the slice) and reports the fallback; a pivot
//     at most eps * n * max|a| there marks the system not regular, as rustymath's `regular`.
#define RM_BT_NS bt
#define RM_BT_NMAX 256
#define RM_BT_MIN_BLOCKS 2
#include "batched_kernels.cuh"
