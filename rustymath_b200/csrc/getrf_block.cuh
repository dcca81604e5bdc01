// The kernels of one 128-column block of the blocked float64 LU (getrf_block.cu), for getrf.cu.
#pragma once
#include <cstdint>

#include <cuda_runtime.h>

namespace rm {

constexpr int kLeaf = 32;    // columns of a leaf
constexpr int kOuter = 128;  // columns of a block (the trailing update's rank)

// Where a leaf's pivoting moves rows (absolute row indices): position j0 + e takes the old row
// piv_src[e], and position disp_dst[d] the old row disp_src[d], one of j0 .. j0 + 31 that a pivot
// displaced. Every other row stays.
struct LeafMoves {
  int j0, jb, disp;
  int piv_src[kLeaf], disp_src[kLeaf], disp_dst[kLeaf];
};

// What a block's kernels hand to each other, in global memory.
struct BlockScratch {
  LeafMoves moves[kOuter / kLeaf];
  // the rows a leaf moves (pivot e in row e, displaced row d in row 32 + d), the block's columns
  alignas(16) double rows[2 * kLeaf][kOuter];
};

// Where the leaves have run: sm[i] is the last leaf (its first column plus one) with a CTA on SM i,
// latest the last leaf of all.
constexpr unsigned kSmMarks = 1024;
struct LeafMarks {
  int latest;
  int sm[kSmMarks];
};

// Rows that leaf_f64 takes: a thread per row, 512 threads in each of 16 CTAs, or of as many as the current
// device places in one cluster.
constexpr int kLeafMaxRows = 8192;
int leaf_max_rows();

// Factors the leaf of columns j0 .. j0 + jb (of the block J0 .. J1) over rows j0 .. n - 1, its rows
// left at their final positions; fills s->moves[(j0 - J0) / kLeaf] and s->rows. The block's last
// leaf (j0 + jb == J1) also moves the rows of the block's columns left of it. With marks, its CTAs
// note the SMs that they run on.
int leaf_f64(double* w, int64_t ldw, int n, int j0, int jb, int J0, int J1, BlockScratch* s, LeafMarks* marks,
             unsigned* status, cudaStream_t stream);
// The same from the swaps ipiv[j0 ..] of a leaf that has been factored with its rows swapped.
int leaf_moves_f64(double* w, int64_t ldw, int j0, int jb, int J0, int J1, const int64_t* ipiv, BlockScratch* s,
                   cudaStream_t stream);
// After a leaf that is not the block's last: its moves on the block's other columns, its rows of
// the later columns (U12), and those columns' update below them.
int leaf_tail_f64(double* w, int64_t ldw, int n, int j0, int J0, int J1, const BlockScratch* s, cudaStream_t stream);
// After the block's leaves: their moves on the columns left of the block (with left), on columns
// lo .. hi - 1 right of it and on perm (not NULL), and the block's rows of those right columns, U12 =
// L11^-1 A12.
int block_rows_f64(double* w, int64_t ldw, int J0, int nb, bool left, int lo, int hi, const BlockScratch* s, int64_t* perm,
                   cudaStream_t stream);

// C -= A B (row-major m x k and k x n; dgemm.cu; C 16-byte aligned, ldc even), by a persistent grid
// that leaves the SMs of the latest leaf, `most` at most, to the next one. *counters (two ints) is
// zero on entry.
int dgemm_update_f64(int m, int n, int k, const double* a, int64_t lda, const double* b, int64_t ldb, double* c,
                     int64_t ldc, const LeafMarks* marks, int most, int* counters, unsigned* status,
                     cudaStream_t stream);

}  // namespace rm
