// LU with partial pivoting on the B200: the plain float64 path.
//
// Replaces lu_factor / lu_panel (core/src/linalg/factor.rs:580-630). The reference halves
// columns recursively down to 16-column leaves on a column-major copy. Here the working
// copy stays row-major (row swaps are contiguous and coalesced) and the factorization is
// right-looking in blocks of kOuter columns, so the trailing update is a rank-128 FP64
// product (compute-bound on DMMA) instead of the rank-16..n/2 products of the recursion:
//
//   for each block of kOuter columns at J0 (getrf_block.cu):
//     for each 32-column leaf at j0 inside it:
//       leaf_kernel       : pivot search, scale and rank-1 updates of the leaf, the rows in the
//                           shared memory of up to 16 CTAs (taller than 512 rows for each CTA of
//                           the largest cluster: panel_kernel)
//       leaf_tail_kernel  : the leaf's row moves on the block's other columns, U = L^-1 A for the
//                           leaf's rows of the block's later columns, and those columns' update
//     block_rows_kernel   : the block's row moves on every column outside it, and perm; U12 =
//                           L11^-1 A12
//     dgemm               : A22 -= L21 U12: the next block's 128 columns first; for n >= 1024 the
//                           rest runs on a side stream while the next block's leaves factor
//                           (look-ahead)
//
// The pivot rule is the reference's `largest` (factor.rs:476): the first row of greatest
// magnitude, NaN never chosen, the diagonal itself when every candidate is NaN; a zero
// pivot leaves its column unreduced (factor.rs:606); `divide` multiplies by the
// reciprocal unless the pivot is subnormal (factor.rs:506-508).
#include <climits>

#include <mutex>
#include <vector>

#include "getrf_block.cuh"
#include "rm_cluster.cuh"
#include "rm_internal.h"
#include "short_pivot.cuh"
#include "small_solve.cuh"

namespace rm {

constexpr int kPanelThreads = 256;
constexpr int kPanelWarps = kPanelThreads / 32;
constexpr int kPanelStride = kLeaf + 1;  // shared row stride (odd: conflict-free column reads)
constexpr int kMaxCluster = 16;
constexpr int kPanelSmemBudget = 200 * 1024;

template <typename T>
__device__ __forceinline__ T min_normal() {
  if constexpr (sizeof(T) == 8) return 2.2250738585072014e-308;
  else return 1.17549435e-38f;
}

// Keeps the larger magnitude, and on equal magnitudes the lower row (the first index).
template <typename T>
__device__ __forceinline__ void argmax_merge(T& v, int& i, T ov, int oi) {
  if (ov > v || (ov == v && oi < i)) {
    v = ov;
    i = oi;
  }
}
template <typename T>
__device__ __forceinline__ void warp_argmax(T& v, int& i) {
#pragma unroll
  for (int off = 16; off; off >>= 1) {
    const T ov = __shfl_xor_sync(0xffffffffu, v, off);
    const int oi = __shfl_xor_sync(0xffffffffu, i, off);
    argmax_merge(v, i, ov, oi);
  }
}

template <typename T>
struct PanelShared {
  T red_v[kPanelWarps];
  int red_i[kPanelWarps];
  T slot_v[2][kMaxCluster];
  int slot_i[2][kMaxCluster];
  T cand[2][kLeaf];
  T diag[2][kLeaf];
  T piv[kLeaf];
  T old[kLeaf];
  int p;
};

// One leaf of up to kLeaf columns: rows j0..n-1, columns j0..j0+jb-1 of W. CTA `rank` of
// the cluster holds rows [rank*rpc, (rank+1)*rpc) of the leaf (in shared memory when
// IN_SMEM, else read and written in place); thread t owns the rows t, t+256, ...
template <typename T, bool IN_SMEM>
__global__ void __launch_bounds__(kPanelThreads)
    panel_kernel(T* __restrict__ w, int64_t ldw, int n, int j0, int jb, int rpc, int64_t* __restrict__ ipiv) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int P = (int)cluster_nctarank();
  const int rank = (int)cluster_ctarank();
  const int M = n - j0;
  const int base = rank * rpc;
  const int cnt = max(0, min(rpc, M - base));
  T* S = reinterpret_cast<T*>(smem);
  const size_t rows_bytes = IN_SMEM ? ((size_t)rpc * kPanelStride * sizeof(T) + 15) / 16 * 16 : 0;
  PanelShared<T>* sh = reinterpret_cast<PanelShared<T>*>(smem + rows_bytes);
  T* g0 = w + (int64_t)(j0 + base) * ldw + j0;  // this CTA's first row, first leaf column

  auto at = [&](int lr, int cc) -> T& {
    if constexpr (IN_SMEM) return S[lr * kPanelStride + cc];
    else return g0[(int64_t)lr * ldw + cc];
  };

  if constexpr (IN_SMEM) {
    for (int e = tid; e < cnt * jb; e += kPanelThreads) {
      const int lr = e / jb, cc = e - lr * jb;
      S[lr * kPanelStride + cc] = g0[(int64_t)lr * ldw + cc];
    }
  }
  __syncthreads();
  if (P > 1) cluster_sync_all();  // every CTA of the cluster runs before any DSMEM access

  for (int c = 0; c < jb; ++c) {
    const int par = c & 1;
    const int d = j0 + c;  // the diagonal row
    // ---- this thread's candidate: first greatest magnitude among its rows >= d
    T bv = T(-1);
    int bi = INT_MAX;
    for (int lr = tid; lr < cnt; lr += kPanelThreads) {
      const int gi = j0 + base + lr;
      if (gi >= d) {
        const T v = fabs(at(lr, c));
        if (v > bv) {  // NaN never compares greater
          bv = v;
          bi = gi;
        }
      }
    }
    warp_argmax(bv, bi);
    if (lane == 0) {
      sh->red_v[warp] = bv;
      sh->red_i[warp] = bi;
    }
    __syncthreads();
    if (warp == 0) {
      bv = lane < kPanelWarps ? sh->red_v[lane] : T(-1);
      bi = lane < kPanelWarps ? sh->red_i[lane] : INT_MAX;
      warp_argmax(bv, bi);
      if (lane < jb) {
        if (bi != INT_MAX) sh->cand[par][lane] = at(bi - j0 - base, lane);
        const int dl = d - j0 - base;
        if (dl >= 0 && dl < cnt) sh->diag[par][lane] = at(dl, lane);
      }
      if (P > 1) {
        if (lane < P) {
          st_cluster(map_rank(&sh->slot_v[par][rank], lane), bv);
          st_cluster(map_rank(&sh->slot_i[par][rank], lane), bi);
        }
      } else if (lane == 0) {
        sh->slot_v[par][0] = bv;
        sh->slot_i[par][0] = bi;
      }
    }
    if (P > 1) cluster_sync_all();
    else __syncthreads();
    if (warp == 0) {
      T v = lane < P ? sh->slot_v[par][lane] : T(-1);
      int i = lane < P ? sh->slot_i[par][lane] : INT_MAX;
      warp_argmax(v, i);
      const int p = i == INT_MAX ? d : i;
      const int owner_p = (p - j0) / rpc, owner_d = (d - j0) / rpc;
      if (lane < jb) {
        T dv, pv;
        if (P > 1) {
          dv = ld_cluster_f64(map_rank(&sh->diag[par][lane], owner_d));
          pv = p == d ? dv : ld_cluster_f64(map_rank(&sh->cand[par][lane], owner_p));
        } else {
          dv = sh->diag[par][lane];
          pv = p == d ? dv : sh->cand[par][lane];
        }
        sh->piv[lane] = pv;
        sh->old[lane] = dv;
      }
      if (lane == 0) sh->p = p;
    }
    __syncthreads();
    const int p = sh->p;
    const T pivot = sh->piv[c];
    if (p != d) {
      const int dl = d - j0 - base, pl = p - j0 - base;
      if (dl >= 0 && dl < cnt && dl % kPanelThreads == tid)
        for (int cc = 0; cc < jb; ++cc) at(dl, cc) = sh->piv[cc];
      if (pl >= 0 && pl < cnt && pl % kPanelThreads == tid)
        for (int cc = 0; cc < jb; ++cc) at(pl, cc) = sh->old[cc];
    }
    if (pivot != T(0)) {
      const bool sub = fabs(pivot) < min_normal<T>();
      const T r = sub ? T(0) : T(1) / pivot;
      for (int lr = tid; lr < cnt; lr += kPanelThreads) {
        if (j0 + base + lr > d) {
          T l = at(lr, c);
          l = sub ? l / pivot : l * r;
          at(lr, c) = l;
#pragma unroll 8
          for (int cc = c + 1; cc < jb; ++cc) at(lr, cc) = fma(l, -sh->piv[cc], at(lr, cc));
        }
      }
    }
    if (rank == 0 && tid == 0) ipiv[d] = p;
  }

  if constexpr (IN_SMEM) {
    __syncthreads();
    for (int e = tid; e < cnt * jb; e += kPanelThreads) {
      const int lr = e / jb, cc = e - lr * jb;
      g0[(int64_t)lr * ldw + cc] = S[lr * kPanelStride + cc];
    }
  }
  if (P > 1) cluster_sync_all();  // no CTA leaves while a peer may still read its memory
}

// ------------------------------------------------------------------ a whole matrix in a cluster
// n <= 256: the whole matrix lives in the shared memory of one cluster of C <= 8 CTAs (a power
// of two, at most 32 rows per CTA; 66 KB per CTA at n = 256) and is factored in one launch,
// column by column, right-looking, with one cluster barrier per pivot column, in place of the
// blocked path's chain of dependent launches (leaves, swaps, inversions, block products). Each
// item takes the fmas of rustymath's packed products in the same order (one per pivot column,
// in column order), so the factors are the oracle's bits, which is why these sizes stay here: the
// blocked path, whose block rows go through inverted diagonal blocks, does not give them, but has become
// the faster one (a factorization at n = 64 / 128 / 192 / 256: 0.132 / 0.203 / 0.308 / 0.422 ms here,
// 0.106 / 0.165 / 0.243 / 0.307 ms there). A column costs ~1.1 us at C = 2 and ~2.2 us at C = 16 (the cluster
// barrier and the pivot row's reads from one CTA's shared memory).
//
// Rows do not move. Every warp of a CTA tracks the positions of the CTA's rows (lane = row), so
// a pivot choice only exchanges two positions, as in leaf_kernel; at the end each row is
// stored at its final position. Per pivot column j, after the barrier that publishes column j's
// candidates:
//   - every warp reduces the C posts (largest key, lowest position among equals; when every
//     candidate is NaN, the row at position j, which its CTA posts beside its candidate) and
//     forms its rows' multipliers l = a_ij / pivot (the reciprocal as the other panels form it);
//   - warp 0 updates column j + 1 (the pivot row's item read from the winner's shared memory),
//     keeps it, finds its CTA's candidate for column j + 1 and posts it into every CTA's slot;
//   - the other warps update columns j + 2 .. n - 1, 32 columns per warp, the pivot row's items
//     read from the winner's shared memory a lane each and passed on by shuffles.
// Posts are double-buffered by the column's parity: a CTA writes the slot of column j + 2 only
// after the barrier of column j + 1, which every CTA reaches after it has read column j's posts.
// Each item takes one fma per pivot column, in column order; a zero pivot leaves its column
// unreduced (factor.rs:606); the multipliers of column j are written into column j at the next
// step, when no warp reads that column any more. Every CTA runs the same n barriers, so the
// barrier cannot be left waiting.
constexpr int kClusterLuMax = 256;
constexpr int kClusterLuRows = 32;  // rows per CTA at most (a lane each)

struct alignas(16) ClusterPost {
  unsigned long long key;  // |candidate| bits + 1; 0 for NaN or no row left
  double piv;              // the candidate's item
  double dpiv;             // the item of the row at the diagonal's position, when this CTA holds it
  int pos;                 // the candidate's position
  int lrow;                // its row within the CTA
  int drow;                // the CTA's row at the diagonal's position, or -1
  int pad;
};

struct ClusterLuShared {
  ClusterPost post[2][kMaxCluster];  // [column parity][posting CTA]
};

// Warp 0 of each CTA: the CTA's candidate for column `col` (y = this lane's row's item) and, if
// the CTA holds it, the row at position `col`, stored into slot `slot` of every CTA's posts.
__device__ __forceinline__ void cluster_lu_post(ClusterLuShared& sh, int slot, double y, int pos, bool active,
                                                int col, int C, int rank, int lane) {
  const double a = fabs(y);
  const unsigned long long key = (active && a == a) ? (unsigned long long)__double_as_longlong(a) + 1ull : 0ull;
  bool none;
  const int wl = short_reduce(key, (unsigned)pos, none);
  const unsigned long long wkey = __shfl_sync(0xffffffffu, key, wl);
  const double wpiv = __shfl_sync(0xffffffffu, y, wl);
  const int wpos = __shfl_sync(0xffffffffu, pos, wl);
  const unsigned db = __ballot_sync(0xffffffffu, pos == col);
  const int dl = db ? __ffs(db) - 1 : -1;
  const double dpiv = __shfl_sync(0xffffffffu, y, dl < 0 ? 0 : dl);
  if (lane < C) {
    const uint32_t d = map_rank(&sh.post[slot][rank], (uint32_t)lane);
    st_cluster_u64(d + offsetof(ClusterPost, key), wkey);
    st_cluster(d + offsetof(ClusterPost, piv), wpiv);
    st_cluster(d + offsetof(ClusterPost, dpiv), dpiv);
    st_cluster(d + offsetof(ClusterPost, pos), wpos);
    st_cluster(d + offsetof(ClusterPost, lrow), wl);
    st_cluster(d + offsetof(ClusterPost, drow), dl);
  }
}

// The n x n row-major a (lda; it may be W) is factored into W (row-major, ldw): on return row i of W
// holds row i of the factors (the
// source row perm[i]); ipiv[j] is the position exchanged with j at step j. R rows per CTA, ld
// the shared row stride (odd: a warp's column reads hit distinct banks).
__global__ void __launch_bounds__(32 * (1 + kClusterLuMax / 32), 1)
    cluster_lu_kernel(const double* a, int64_t lda, double* w, int64_t ldw, int n, int R, int ld,
                      int64_t* __restrict__ ipiv, int64_t* __restrict__ perm, double* amax) {
  extern __shared__ __align__(16) uint8_t smem[];
  ClusterLuShared& sh = *reinterpret_cast<ClusterLuShared*>(smem);
  double* S = reinterpret_cast<double*>(smem + sizeof(ClusterLuShared));
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int nwarps = blockDim.x >> 5;
  const int rank = (int)cluster_ctarank(), C = (int)cluster_nctarank();
  const int g0 = rank * R;
  const int rows = max(0, min(R, n - g0));
  double top = 0.0;
  for (int i = warp; i < rows; i += nwarps)
    for (int c = lane; c < n; c += 32) {
      const double v = a[(int64_t)(g0 + i) * lda + c];
      S[i * ld + c] = v;
      if (fabs(v) > top) top = fabs(v);  // NaN never is
    }
  if (amax != nullptr) {
    __shared__ double tops[1 + kClusterLuMax / 32];
#pragma unroll
    for (int off = 16; off; off >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, off));
    if (lane == 0) tops[warp] = top;
    __syncthreads();
    if (t == 0) {
      for (int v = 1; v < nwarps; ++v) top = fmax(top, tops[v]);
      amax[rank] = top;
    }
  }
  const bool valid = lane < rows;
  int pos = valid ? g0 + lane : INT_MAX;
  double* myrow = S + (valid ? lane : 0) * ld;
  cluster_sync_all();  // the rows are in, and every CTA of the cluster runs before any DSMEM access
  if (warp == 0) cluster_lu_post(sh, 0, valid ? myrow[0] : 0.0, pos, valid, 0, C, rank, lane);
  cluster_sync_all();
  double lprev = 0.0;  // warp 0: the multiplier of the step before, written one step late
  bool lprev_set = false;
#pragma unroll 1
  for (int j = 0; j < n; ++j) {
    const ClusterPost* pp = sh.post[j & 1];
    const unsigned long long k2 = lane < C ? pp[lane].key : 0ull;
    const unsigned p2 = lane < C ? (unsigned)pp[lane].pos : 0xffffffffu;
    bool none;
    int wr = short_reduce(k2, p2, none);
    int lr, pr;
    double piv;
    if (!none) {
      lr = pp[wr].lrow;
      pr = pp[wr].pos;
      piv = pp[wr].piv;
    } else {  // every candidate is NaN: the row at position j is the pivot row
      const unsigned b = __ballot_sync(0xffffffffu, lane < C && pp[lane].drow >= 0);
      wr = __ffs(b) - 1;
      lr = pp[wr].drow;
      pr = j;
      piv = pp[wr].dpiv;
    }
    if (pos == pr) pos = j;
    else if (pos == j) pos = pr;
    const bool active = valid && pos > j;
    const bool skip = piv == 0.0;
    const bool sub = fabs(piv) < 2.2250738585072014e-308;
    const double rcp = short_rcp(piv);
    double l = 0.0;
    if (active && !skip) {
      const double a = myrow[j];
      l = sub ? a / piv : a * rcp;
    }
    const uint32_t prow = map_rank(S + lr * ld, (uint32_t)wr);  // the pivot row, in CTA wr
    if (warp == 0) {
      if (lprev_set) myrow[j - 1] = lprev;
      lprev = l;
      lprev_set = active && !skip;
      if (j + 1 < n) {
        double y = valid ? myrow[j + 1] : 0.0;
        if (!skip) {
          const double u = ld_cluster_f64(prow + (uint32_t)(j + 1) * 8u);
          if (active) {
            y = fma(l, -u, y);
            myrow[j + 1] = y;
          }
        }
        cluster_lu_post(sh, (j + 1) & 1, y, pos, active, j + 1, C, rank, lane);
      }
    } else if (!skip) {
#pragma unroll 1
      for (int c0 = j + 2 + (warp - 1) * 32; c0 < n; c0 += (nwarps - 1) * 32) {
        const int cc = c0 + lane;
        const double ul = cc < n ? ld_cluster_f64(prow + (uint32_t)cc * 8u) : 0.0;
        const int cend = min(32, n - c0);
        double* rp = myrow + c0;
        if (cend == 32) {
#pragma unroll 8
          for (int q = 0; q < 32; ++q) {
            const double u = __shfl_sync(0xffffffffu, ul, q);
            if (active) rp[q] = fma(l, -u, rp[q]);
          }
        } else {
          for (int q = 0; q < cend; ++q) {
            const double u = __shfl_sync(0xffffffffu, ul, q);
            if (active) rp[q] = fma(l, -u, rp[q]);
          }
        }
      }
    }
    if (rank == 0 && t == 0) ipiv[j] = pr;
    cluster_sync_all();
  }
  // every row to its final position: a warp per row, lanes along it
  for (int i = warp; i < rows; i += nwarps) {
    const int pi = __shfl_sync(0xffffffffu, pos, i);
    for (int c = lane; c < n; c += 32) w[(int64_t)pi * ldw + c] = S[i * ld + c];
  }
  if (warp == 0 && valid) perm[pos] = g0 + lane;
}

constexpr size_t cluster_lu_smem(int R, int ld) {
  return sizeof(ClusterLuShared) + (size_t)R * ld * sizeof(double);
}

// ------------------------------------------------------------------ small solves in one CTA
// x = U^-1 L^-1 b[perm] for n <= 256 and k <= 8 from W (rows at their final positions), in one
// CTA: a thread per row holds its row of x; per column one barrier. The order is that of
// rustymath's single-column solve (`single` on the transposed factors, factor.rs:725-748):
// forward, column j after column j - 1, x_i = fma(l_ij, -x_j, x_i) for i > j; backward, from the
// last column, x_j = x_j / u_jj, then x_i = fma(u_ij, -x_j, x_i) for i < j. With one right-hand
// side the result is the oracle's bits; with more, each column is solved the same way. W comes
// in 32-column blocks through two shared-memory buffers, the next block's copies in flight
// while the current one is used.
constexpr int kSmallSolveMax = 256;
constexpr int kSmallSolveK = 8;
constexpr int kSsCols = 32;
constexpr int kSsStride = kSsCols + 2;  // doubles per staged row (16-byte aligned rows)

__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// COLMAJOR: the factors in rustymath's order (item (i, j) at w[j * ldw + i], exactly n columns),
// staged as columns ([32][n] per buffer); else W row-major ([n][kSsStride] per buffer). A row
// position outside 0..n-1 sets RM_DEV_BAD_INDEX in *status (when given) and that row's right-hand
// side is taken as zero.
template <bool COLMAJOR>
__global__ void __launch_bounds__(kSmallSolveMax, 1)
    small_solve_kernel(const double* __restrict__ w, int64_t ldw, int n, const int64_t* __restrict__ perm,
                       const double* b, int k, double* x, unsigned* status, const double* amax, int parts,
                       SmallSolveResults* results) {
  extern __shared__ __align__(16) uint8_t smem[];
  double* buf = reinterpret_cast<double*>(smem);  // two staging buffers of kSsCols * kSsStride * ... doubles
  __shared__ double xs[2][kSmallSolveK];
  const int t = threadIdx.x;
  const bool own = t < n;
  const int nblk = (n + kSsCols - 1) / kSsCols;
  double v[kSmallSolveK];
  {
    const int64_t src = own ? perm[t] : 0;
    const bool in = src >= 0 && src < n;
    if (own && !in && status) flag_error(status, RM_DEV_BAD_INDEX);
#pragma unroll
    for (int c = 0; c < kSmallSolveK; ++c) v[c] = (own && in && c < k) ? b[src * k + c] : 0.0;
  }
  const size_t bufsz = COLMAJOR ? (size_t)kSsCols * n : (size_t)n * kSsStride;
  // stage q: forward blocks 0..nblk-1, then backward blocks nblk-1..0
  auto stage = [&](int q) {
    const int blk = q < nblk ? q : 2 * nblk - 1 - q;
    double* dst = buf + (q & 1) * bufsz;
    if constexpr (COLMAJOR) {  // columns blk*32 .. min(n, blk*32 + 32) - 1, a row item each
      const int c0 = blk * kSsCols, cols = min(kSsCols, n - c0);
      for (int e = t; e < cols * n; e += kSmallSolveMax) {
        const int c = e / n, r = e % n;
        cp_async8(dst + (size_t)c * n + r, w + (int64_t)(c0 + c) * ldw + r);
      }
    } else {
      const double* src = w + (int64_t)blk * kSsCols;
      for (int e = t; e < n * (kSsCols / 2); e += kSmallSolveMax) {
        const int r = e / (kSsCols / 2), h = e % (kSsCols / 2);
        cp_async16(dst + r * kSsStride + 2 * h, src + (int64_t)r * ldw + 2 * h);
      }
    }
    cp_async_commit();
  };
  stage(0);
  for (int q = 0; q < 2 * nblk; ++q) {
    cp_async_wait<0>();
    __syncthreads();  // stage q is in; every thread is done with stage q - 1's buffer
    if (q + 1 < 2 * nblk) stage(q + 1);
    const double* S = buf + (q & 1) * bufsz;
    // item (t, c0 + i) of the staged block is mine[i * step]
    const double* mine = COLMAJOR ? S + (own ? t : 0) : S + (own ? t : 0) * kSsStride;
    const int step = COLMAJOR ? n : 1;
    if (q < nblk) {
      const int c0 = q * kSsCols, c1 = min(n, c0 + kSsCols);
      for (int j = c0; j < c1; ++j) {
        double* xj = xs[j & 1];
        if (t == j)
#pragma unroll
          for (int c = 0; c < kSmallSolveK; ++c)
            if (c < k) xj[c] = v[c];
        __syncthreads();
        if (own && t > j) {
          const double l = mine[(j - c0) * step];
#pragma unroll
          for (int c = 0; c < kSmallSolveK; ++c)
            if (c < k) v[c] = fma(l, -xj[c], v[c]);
        }
      }
    } else {
      const int blk = 2 * nblk - 1 - q, c0 = blk * kSsCols, c1 = min(n, c0 + kSsCols);
      for (int j = c1 - 1; j >= c0; --j) {
        double* xj = xs[j & 1];
        if (t == j) {  // the divisions are on the critical path: only the k columns in use
          const double d = mine[(j - c0) * step];
#pragma unroll
          for (int c = 0; c < kSmallSolveK; ++c)
            if (c < k) xj[c] = v[c] = v[c] / d;
        }
        __syncthreads();
        if (own && t < j) {
          const double u = mine[(j - c0) * step];
#pragma unroll
          for (int c = 0; c < kSmallSolveK; ++c)
            if (c < k) v[c] = fma(u, -xj[c], v[c]);
        }
      }
    }
  }
  if (own)
#pragma unroll
    for (int c = 0; c < kSmallSolveK; ++c)
      if (c < k) x[(int64_t)t * k + c] = v[c];
  if (results != nullptr) {
    // LuWork::regular (regular_kernel), and what the caller reads, straight into its host memory
    double top = 0.0;
    for (int i = 0; i < parts; ++i) top = fmax(top, amax[i]);
    const bool bad = own && fabs(w[(int64_t)t * ldw + t]) <= 2.220446049250313e-16 * (double)n * top;
    const int any = __syncthreads_or(bad ? 1 : 0);
    if (t == 0) {
      results->flag = any ? 0 : 1;
      results->status = *status;
      __threadfence_system();
    }
  }
}

// The plain solve takes this kernel up to n = 192, where one right-hand side gives the oracle's bits. Whole
// solves with it and with the block-chained solves in its place (n = 64 / 128 / 192 / 256): one right-hand
// side 0.192 / 0.288 / 0.424 / 0.586 against 0.207 / 0.283 / 0.406 / 0.519 ms, eight 0.220 / 0.348 / 0.514 /
// 0.697 against 0.207 / 0.283 / 0.407 / 0.522 ms.
constexpr int kSmallSolveRoute = 192;
bool small_solve_fits(int64_t n, int64_t k) { return n >= 1 && n <= kSmallSolveRoute && k >= 1 && k <= kSmallSolveK; }

int small_solve_f64(const double* w, int64_t ldw, bool colmajor, int64_t n, const int64_t* perm, const double* b,
                    int64_t k, double* x, unsigned* status, cudaStream_t stream) {
  if (n < 1 || n > kSmallSolveMax || k < 1 || k > kSmallSolveK) return RM_BAD_ARG;
  if (colmajor) {
    RM_TRY(smem_attribute(small_solve_kernel<true>, (size_t)2 * kSsCols * kSmallSolveMax * sizeof(double)));
    small_solve_kernel<true><<<1, kSmallSolveMax, (size_t)2 * kSsCols * n * sizeof(double), stream>>>(
        w, ldw, (int)n, perm, b, (int)k, x, status, nullptr, 0, nullptr);
  } else {
    RM_TRY(smem_attribute(small_solve_kernel<false>, (size_t)2 * kSmallSolveMax * kSsStride * sizeof(double)));
    small_solve_kernel<false><<<1, kSmallSolveMax, (size_t)2 * n * kSsStride * sizeof(double), stream>>>(
        w, ldw, (int)n, perm, b, (int)k, x, status, nullptr, 0, nullptr);
  }
  RM_LAUNCHED();
  return RM_OK;
}

// ------------------------------------------------------------------ driver

// The largest cluster (<= kMaxCluster CTAs of kPanelSmemBudget bytes) this device can place.
template <typename T>
static int find_panel_cluster_limit() {
  int limit = 0;
  auto k = panel_kernel<T, true>;
  if (smem_attribute(k, kPanelSmemBudget + 4096) != RM_OK ||
      func_attribute(reinterpret_cast<const void*>(k), cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != RM_OK ||
      func_attribute(reinterpret_cast<const void*>(panel_kernel<T, false>),
                     cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != RM_OK) {
    cudaGetLastError();
    return limit = 8;
  }
  for (int P = kMaxCluster; P >= 1; P /= 2) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = P;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(P);
    cfg.blockDim = dim3(kPanelThreads);
    cfg.dynamicSmemBytes = kPanelSmemBudget;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, k, &cfg) == cudaSuccess && clusters > 0) return limit = P;
    cudaGetLastError();
  }
  return limit = 1;
}

// Found once per device (the attributes and the answer belong to that device).
template <typename T>
static int panel_cluster_limit() {
  static std::mutex mu;
  static std::vector<int> limits;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 1;
  {
    std::lock_guard<std::mutex> lock(mu);
    if ((int)limits.size() > dev && limits[dev]) return limits[dev];
  }
  const int limit = find_panel_cluster_limit<T>();
  std::lock_guard<std::mutex> lock(mu);
  if ((int)limits.size() <= dev) limits.resize(dev + 1, 0);
  limits[dev] = limit;
  return limit;
}


// Whether this device can place the largest cluster cluster_lu_kernel takes (8 CTAs of 288
// threads and 66 KB of shared memory); found once per device.
constexpr int kClusterLuMaxCtas = kClusterLuMax / kClusterLuRows;
static bool find_cluster_lu_ok() {
  const size_t smem = cluster_lu_smem(kClusterLuRows, kClusterLuMax + 1);
  if (smem_attribute(cluster_lu_kernel, smem) != RM_OK) {
    cudaGetLastError();
    return false;
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kClusterLuMaxCtas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(kClusterLuMaxCtas);
  cfg.blockDim = dim3(32 * (1 + kClusterLuMax / 32));
  cfg.dynamicSmemBytes = smem;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, cluster_lu_kernel, &cfg) == cudaSuccess && clusters > 0) return true;
  cudaGetLastError();
  return false;
}

static bool cluster_lu_ok() {
  static std::mutex mu;
  static std::vector<int> state;  // 0 unknown, 1 yes, 2 no
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  {
    std::lock_guard<std::mutex> lock(mu);
    if ((int)state.size() > dev && state[dev]) return state[dev] == 1;
  }
  const bool ok = find_cluster_lu_ok();
  std::lock_guard<std::mutex> lock(mu);
  if ((int)state.size() <= dev) state.resize(dev + 1, 0);
  state[dev] = ok ? 1 : 2;
  return ok;
}

// n <= kClusterLuMax in one launch: C CTAs (the least power of two giving at most 32 rows each).
static int launch_cluster_lu(const double* a, int64_t lda, double* w, int64_t ldw, int n, int64_t* ipiv, int64_t* perm,
                             double* amax, cudaStream_t stream) {
  const int need = (n + kClusterLuRows - 1) / kClusterLuRows;
  int C = 1;
  while (C < need) C *= 2;
  const int R = (n + C - 1) / C;
  const int ld = n | 1;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(C);
  cfg.blockDim = dim3(32 * (1 + (n + 31) / 32));
  cfg.dynamicSmemBytes = cluster_lu_smem(R, ld);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  RM_CUDA_TRY(cudaLaunchKernelEx(&cfg, cluster_lu_kernel, a, lda, w, ldw, n, R, ld, ipiv, perm, amax));
  note_launch();
  return RM_OK;
}

template <typename T>
static int launch_panel(T* w, int64_t ldw, int n, int j0, int jb, int64_t* ipiv, cudaStream_t stream) {
  const int M = n - j0;
  const size_t sh = (sizeof(PanelShared<T>) + 15) / 16 * 16;
  const int rows_cap = (int)((kPanelSmemBudget - sh) / (kPanelStride * sizeof(T)));
  const int pmax = panel_cluster_limit<T>();
  int P = 1;
  while (P < pmax && (M + P - 1) / P > rows_cap) P *= 2;
  // spread tall leaves over more CTAs: about 2 rows per thread
  while (P < pmax && (M + P - 1) / P > 2 * kPanelThreads) P *= 2;
  const int rpc = (M + P - 1) / P;
  const bool in_smem = rpc <= rows_cap;
  const size_t smem = (in_smem ? ((size_t)rpc * kPanelStride * sizeof(T) + 15) / 16 * 16 : 0) + sh;

  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = P;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(P);
  cfg.blockDim = dim3(kPanelThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (in_smem) {
    RM_CUDA_TRY(cudaLaunchKernelEx(&cfg, panel_kernel<T, true>, w, ldw, n, j0, jb, rpc, ipiv));
  } else {
    RM_CUDA_TRY(cudaLaunchKernelEx(&cfg, panel_kernel<T, false>, w, ldw, n, j0, jb, rpc, ipiv));
  }
  note_launch();
  return RM_OK;
}

__global__ void iota_kernel(int64_t* perm, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    perm[i] = i;
}

namespace {
struct GetrfScratch {
  BlockScratch block[2];         // by the block's parity: the side stream still reads the last one's
  LeafMarks marks;
};
}  // namespace

// the look-ahead's counters follow: two ints per block
size_t getrf_f64_scratch_bytes(int64_t n) {
  return sizeof(GetrfScratch) + (size_t)((n + kOuter - 1) / kOuter) * 2 * sizeof(int);
}

namespace {
// The look-ahead's streams: the critical chain (hp) at the device's highest stream priority, the
// rest of each trailing update (side) at its lowest, so that the chain's panel clusters take
// SMs first as the update's tiles finish. Released on return (queued work completes first).
struct F64LookAhead {
  cudaStream_t hp = nullptr, side = nullptr;
  cudaEvent_t leaves_done = nullptr, rest_done = nullptr, entry = nullptr;
  int open() {
    int least = 0, greatest = 0;
    RM_CUDA_TRY(cudaDeviceGetStreamPriorityRange(&least, &greatest));
    RM_CUDA_TRY(cudaStreamCreateWithPriority(&hp, cudaStreamNonBlocking, greatest));
    RM_CUDA_TRY(cudaStreamCreateWithPriority(&side, cudaStreamNonBlocking, least));
    RM_CUDA_TRY(cudaEventCreateWithFlags(&leaves_done, cudaEventDisableTiming));
    RM_CUDA_TRY(cudaEventCreateWithFlags(&rest_done, cudaEventDisableTiming));
    RM_CUDA_TRY(cudaEventCreateWithFlags(&entry, cudaEventDisableTiming));
    RM_CUDA_TRY(cudaEventRecord(rest_done, side));  // complete at first, so the first wait passes
    return RM_OK;
  }
  ~F64LookAhead() {
    if (leaves_done) cudaEventDestroy(leaves_done);
    if (rest_done) cudaEventDestroy(rest_done);
    if (entry) cudaEventDestroy(entry);
    if (hp) cudaStreamDestroy(hp);
    if (side) cudaStreamDestroy(side);
  }
};
}  // namespace

int getrf_f64(double* w, int64_t ldw, int64_t n64, int64_t* ipiv, int64_t* perm, void* scratch, unsigned* status,
              cudaStream_t caller) {
  if (n64 <= 0) return RM_OK;
  if (n64 > INT32_MAX / 2) return RM_BAD_ARG;
  const int n = (int)n64;
  if (n <= kClusterLuMax && cluster_lu_ok()) return launch_cluster_lu(w, ldw, w, ldw, n, ipiv, perm, nullptr, caller);
  GetrfScratch* gs = reinterpret_cast<GetrfScratch*>(scratch);
  int* counters = reinterpret_cast<int*>(gs + 1);
  iota_kernel<<<std::max(1, std::min(n / 256 + 1, 1024)), 256, 0, caller>>>(perm, n);
  RM_LAUNCHED();
  // Look-ahead (n >= 1024): the chain's stream does only what the next block's leaves wait for: the
  // block's rows and the trailing update of the next block's 128 columns. The same on all other
  // columns, and the row moves of the columns left of the block, run on a side stream while the
  // next block's leaves factor; the chain waits for the side stream before it touches columns that
  // the side's update wrote.
  //
  // The leaves' clusters need up to 16 free SMs of one GPC at once, which a trailing update that
  // fills the GPU never leaves: with a plain grid for it, chain and update ran one after the other
  // (n = 8192: 34 ms, the chain alone 20, the update alone 11). So the update is a persistent grid
  // whose CTAs do not stay on the SMs where the latest leaf ran.
  F64LookAhead la;
  const bool ahead = n >= 1024;
  const int leaf_rows = leaf_max_rows();
  cudaStream_t stream = caller;
  if (ahead) {
    RM_CUDA_TRY(cudaMemsetAsync(&gs->marks, 0, sizeof gs->marks, caller));
    RM_CUDA_TRY(cudaMemsetAsync(counters, 0, (size_t)((n + kOuter - 1) / kOuter) * 2 * sizeof(int), caller));
    RM_TRY(la.open());
    RM_CUDA_TRY(cudaEventRecord(la.entry, caller));
    RM_CUDA_TRY(cudaStreamWaitEvent(la.hp, la.entry, 0));
    stream = la.hp;
  }
  for (int J0 = 0; J0 < n; J0 += kOuter) {
    const int nb = std::min(kOuter, n - J0);
    const int J1 = J0 + nb;
    BlockScratch* bs = &gs->block[J0 / kOuter & 1];
    for (int j0 = J0; j0 < J1; j0 += kLeaf) {
      const int jb = std::min(kLeaf, J1 - j0);
      if (n - j0 <= leaf_rows) {
        RM_TRY(leaf_f64(w, ldw, n, j0, jb, J0, J1, bs, ahead ? &gs->marks : nullptr, status, stream));
      } else {
        RM_TRY(launch_panel<double>(w, ldw, n, j0, jb, ipiv, stream));
        RM_TRY(leaf_moves_f64(w, ldw, j0, jb, J0, J1, ipiv, bs, stream));
      }
      if (j0 + jb < J1) RM_TRY(leaf_tail_f64(w, ldw, n, j0, J0, J1, bs, stream));
    }
    const double* a12 = w + (int64_t)J0 * ldw + J1;
    const double* l21 = w + (int64_t)J1 * ldw + J0;
    double* a22 = w + (int64_t)J1 * ldw + J1;
    const int rest = n - J1;
    if (!ahead) {
      RM_TRY(block_rows_f64(w, ldw, J0, nb, true, J1, n, bs, perm, stream));
      if (rest > 0)
        RM_TRY(dgemm_device(false, false, rest, rest, nb, -1.0, l21, ldw, a12, ldw, 1.0, a22, ldw, status, stream));
      continue;
    }
    // the side stream needs the leaves, not the chain's part of the block's end
    const int nn = std::min(kOuter, rest);
    RM_CUDA_TRY(cudaEventRecord(la.leaves_done, stream));
    RM_CUDA_TRY(cudaStreamWaitEvent(la.side, la.leaves_done, 0));
    if (nn > 0) {
      if (J0 > 0) RM_CUDA_TRY(cudaStreamWaitEvent(stream, la.rest_done, 0));
      RM_TRY(block_rows_f64(w, ldw, J0, nb, false, J1, J1 + nn, bs, nullptr, stream));
      RM_TRY(dgemm_device(false, false, rest, nn, nb, -1.0, l21, ldw, a12, ldw, 1.0, a22, ldw, status, stream));
    }
    RM_TRY(block_rows_f64(w, ldw, J0, nb, true, J1 + nn, n, bs, perm, la.side));
    if (rest > nn) {
      const int64_t tiles = (int64_t)((rest + 127) / 128) * ((rest - nn + 127) / 128);
      if (tiles >= device_sm_count())
        RM_TRY(dgemm_update_f64(rest, rest - nn, nb, l21, ldw, a12 + nn, ldw, a22 + nn, ldw, &gs->marks, kMaxCluster,
                                counters + 2 * (J0 / kOuter), status, la.side));
      else
        RM_TRY(dgemm_device(false, false, rest, rest - nn, nb, -1.0, l21, ldw, a12 + nn, ldw, 1.0, a22 + nn, ldw, status,
                            la.side));
    }
    RM_CUDA_TRY(cudaEventRecord(la.rest_done, la.side));
  }
  if (ahead) {
    RM_CUDA_TRY(cudaStreamWaitEvent(stream, la.rest_done, 0));
    RM_CUDA_TRY(cudaEventRecord(la.entry, stream));  // the caller's stream continues after both
    RM_CUDA_TRY(cudaStreamWaitEvent(caller, la.entry, 0));
  }
  return RM_OK;
}

// The whole plain solve of a small system in two launches: a into W factored, then the solves, the
// regular test and the results (in page-locked host memory, complete once the stream has
// synchronised). False when the size or the device does not take it. Copying a into W, the regular
// test and reading two words back were three more launches and two copies, about half of the time of
// a solve at n = 8.
bool small_plain_solve_f64(const double* a, double* w, int64_t ldw, int64_t n, const double* b, int64_t k, double* x,
                           int64_t* ipiv, int64_t* perm, double* amax, unsigned* status, SmallSolveResults* results,
                           cudaStream_t stream, int* st) {
  if (!small_solve_fits(n, k) || !cluster_lu_ok()) return false;
  *st = launch_cluster_lu(a, n, w, ldw, (int)n, ipiv, perm, amax, stream);
  if (*st != RM_OK) return true;
  *st = smem_attribute(small_solve_kernel<false>, (size_t)2 * kSmallSolveMax * kSsStride * sizeof(double));
  if (*st != RM_OK) return true;
  int parts = 1;  // CTAs of the cluster
  while (parts * kClusterLuRows < (int)n) parts *= 2;
  small_solve_kernel<false><<<1, kSmallSolveMax, (size_t)2 * n * kSsStride * sizeof(double), stream>>>(
      w, ldw, (int)n, perm, b, (int)k, x, status, amax, parts, results);
  note_launch();
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_last_error(e, "small_solve_kernel", __FILE__, __LINE__);
    *st = RM_CUDA_ERROR;
  }
  return true;
}

// ------------------------------------------------------------------ load / store / regular

__global__ void load_matrix_kernel(const double* __restrict__ a, int64_t lda, double* __restrict__ w, int64_t ldw,
                                   int64_t n, double* amax) {
  double top = 0.0;
  const int64_t total = n * ldw;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = e / ldw, j = e - i * ldw;
    double v = 0.0;
    if (j < n) {
      v = a[i * lda + j];
      const double m = fabs(v);
      if (m > top) top = m;
    }
    w[e] = v;
  }
#pragma unroll
  for (int off = 16; off; off >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, off));
  if ((threadIdx.x & 31) == 0 && top > 0.0)  // non-negative doubles order like their bits
    atomicMax(reinterpret_cast<unsigned long long*>(amax), (unsigned long long)__double_as_longlong(top));
}

int load_matrix_f64(const double* a, int64_t lda, double* w, int64_t ldw, int64_t n, double* amax,
                    cudaStream_t stream) {
  RM_CUDA_TRY(cudaMemsetAsync(amax, 0, sizeof(double), stream));
  if (n == 0) return RM_OK;
  const int64_t total = n * ldw;
  const int blocks = (int)std::min<int64_t>((total + 255) / 256, 8 * device_sm_count());
  load_matrix_kernel<<<blocks, 256, 0, stream>>>(a, lda, w, ldw, n, amax);
  RM_LAUNCHED();
  return RM_OK;
}

// factors[j*n + i] = W[i][j]: a 32x32-tiled transpose through shared memory
__global__ void store_factors_kernel(const double* __restrict__ w, int64_t ldw, int64_t n, double* __restrict__ f) {
  __shared__ double tile[32][33];
  const int64_t i0 = (int64_t)blockIdx.y * 32, j0 = (int64_t)blockIdx.x * 32;
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int64_t i = i0 + r, j = j0 + threadIdx.x;
    if (i < n && j < n) tile[r][threadIdx.x] = w[i * ldw + j];
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int64_t j = j0 + r, i = i0 + threadIdx.x;
    if (i < n && j < n) f[j * n + i] = tile[threadIdx.x][r];
  }
}

int store_factors_f64(const double* w, int64_t ldw, int64_t n, double* factors, cudaStream_t stream) {
  if (n == 0) return RM_OK;
  dim3 grid((unsigned)((n + 31) / 32), (unsigned)((n + 31) / 32));
  store_factors_kernel<<<grid, dim3(32, 8), 0, stream>>>(w, ldw, n, factors);
  RM_LAUNCHED();
  return RM_OK;
}

__global__ void regular_kernel(const double* __restrict__ w, int64_t ldw, int64_t n, const double* amax,
                               int32_t* flag) {
  __shared__ int bad;
  if (threadIdx.x == 0) bad = 0;
  __syncthreads();
  const double negligible = 2.220446049250313e-16 * (double)n * *amax;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x)
    if (fabs(w[i * ldw + i]) <= negligible) bad = 1;  // NaN compares false: a NaN pivot is regular
  __syncthreads();
  if (threadIdx.x == 0) *flag = (n > 0 && !bad) ? 1 : 0;
}

int regular_flag_f64(const double* w, int64_t ldw, int64_t n, const double* amax, int32_t* flag,
                     cudaStream_t stream) {
  regular_kernel<<<1, 1024, 0, stream>>>(w, ldw, n, amax, flag);
  RM_LAUNCHED();
  return RM_OK;
}

}  // namespace rm
