// One 128-column block of the blocked float64 LU: leaves of 32 columns, and the block's rows.
//
// A block is a chain of small dependent steps, so what counts is the number of launches and the
// latency inside each. Per leaf: leaf_kernel (pivoting and factorization, the rows in shared memory)
// and leaf_tail_kernel (the row moves, U12 and the rank-32 update of the block's later columns in
// one launch); per block: block_rows_kernel (the row moves of all four leaves on the other
// columns and U12 = L11^-1 A12). The trailing update is dgemm's.
//
// No kernel swaps rows one after another. Rows keep their threads while a leaf is factored; at
// its end each is stored at its final position, and the moves (at most 32 pivot rows and 32 rows
// that they displaced) are handed on as a list. The moved rows' items of the block's other columns
// go through a small buffer, so the kernel that moves them never reads a row that another CTA
// has already overwritten.
#include <algorithm>
#include <climits>
#include <mutex>
#include <vector>

#include "getrf_block.cuh"
#include "rm_cluster.cuh"
#include "rm_internal.h"

namespace rm {

// D += A B for one m16n8k8 tile; per item one fma per k in increasing k.
__device__ __forceinline__ void dmma(double (&d)[4], const double (&a)[4], double b0, double b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b0), "d"(b1));
}

// ------------------------------------------------------------------ the leaf
// The leaf's rows stay in shared memory, a thread per row, and are factored 8 columns at a time: a
// sub-leaf's 8 items are in the thread's registers, so a column's update reads only 8 items of the
// pivot row; after the sub-leaf its pivot rows' later columns are solved (a thread per column) and
// every row not yet chosen takes the rank-8 update on DMMA. (Holding all 32 items in registers was
// slower: every warp reads the whole pivot row from shared memory at each column, and at 512 rows
// those reads alone were ~1000 cycles of the SM's one pipe.)
//
// Per column: each warp reduces its rows' keys and posts its winner; after one CTA barrier every
// warp reduces the warps' posts. With more than one CTA (rows > 512) the CTA's winner then goes to
// every CTA of the cluster by asynchronous stores that complete on the receiver's mbarrier (one
// per column, so none is armed twice), a warp per receiver; the wait for the C posts is the
// column's only cluster-wide step. Posts are double-buffered by the column's parity: a CTA sends
// column c + 2's post only after it has every post of column c + 1, which each CTA sends after a
// CTA barrier that its warps reach once they have read column c's. At a sub-leaf's end each CTA
// sends the pivot rows it holds, from the sub-leaf's columns on, to every CTA.
//
// A column is a chain of dependent instructions in every warp (~5 cycles each), so what a column
// does is kept to what the next one needs; the rest waits for the sub-leaf's end.
//
// Each item takes one fma per pivot column in column order; a zero pivot's column is skipped.
constexpr int kSub = 8;
constexpr int kLeafMaxThreads = 512;
constexpr int kLeafMaxCtas = kLeafMaxRows / kLeafMaxThreads;
// doubles per row in shared memory: 16-byte rows, and DMMA fragment loads that hit 16 distinct
// 8-byte banks per half-warp
constexpr int kLeafStride = kLeaf + 4;

enum : unsigned { kPivotInvert = 0u, kPivotZero = 1u, kPivotDivide = 2u };

struct alignas(16) LeafPost {
  double row[kSub];              // the candidate's sub-leaf items: multipliers, then items not yet reduced
  unsigned hi, lo, pos, kind;    // its key, its position (relative to j0), what its pivot does
  double rcp, pad;
};
constexpr int kPostPieces = sizeof(LeafPost) / 16;

struct LeafShared {
  LeafPost warp_post[2][kLeafMaxThreads / 32];
  LeafPost cta_post[2][kLeafMaxCtas];
  alignas(16) double prow[kSub][kLeafStride];  // the sub-leaf's pivot rows, from its columns on; then U12
  uint64_t bar[kLeaf], row_bar[kLeaf / kSub];
  int chosen[kLeaf];                           // this CTA's row that became pivot c, or -1
  int pos[kLeafMaxThreads];
  unsigned char active[kLeafMaxThreads];
  int disp, disp_src[kLeaf], disp_dst[kLeaf];
  // the block's other columns: of the rows chosen here (by pivot), and of rows j0 .. j0 + 31
  alignas(16) double piv_other[kLeaf][kOuter];
  alignas(16) double top_other[kLeaf][kOuter];
};
// the self-test's column whose posts come short (in the CTAs of `hold`)
constexpr int kHoldColumn = 11;
constexpr uint64_t kSelfTestWaitNs = 1000000;

constexpr size_t leaf_smem(int threads) {
  return (sizeof(LeafShared) + 15) / 16 * 16 + (size_t)threads * kLeafStride * sizeof(double);
}
static_assert(leaf_smem(kLeafMaxThreads) <= 227 * 1024, "a CTA's shared memory");

// 1 / a, correctly rounded; 0 where rustymath divides by the pivot instead (a subnormal one). Every lane
// forms its own beside the reduction. Rows that are no candidates give 1 to the intrinsic, so that it
// leaves its short path for extreme pivots only.
__device__ __forceinline__ double leaf_rcp(double a, bool candidate) {
  const bool normal = ((unsigned)__double2hiint(a) & 0x7ff00000u) != 0u;
  const double r = __drcp_rn(candidate && normal ? a : 1.0);
  return normal ? r : 0.0;
}

// A candidate's key: the bits of its magnitude, the high word plus 2. 0: no candidate; 1: a NaN at
// the diagonal's position, the pivot when every candidate is NaN. The lane of the warp's largest
// key, and of equal keys the lowest position; nearly always the high words decide.
__device__ __forceinline__ int leaf_best(unsigned hi, unsigned lo, unsigned pos) {
  const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
  unsigned top = __ballot_sync(0xffffffffu, hi == mhi);
  if (top & (top - 1u)) {
    const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? lo : 0u);
    const bool tie = hi == mhi && lo == mlo;
    const unsigned pmin = __reduce_min_sync(0xffffffffu, tie ? pos : 0xffffffffu);
    top = __ballot_sync(0xffffffffu, tie && pos == pmin);
  }
  return __ffs(top) - 1;
}

template <bool CLUSTER>
__global__ void __launch_bounds__(kLeafMaxThreads, 1)
    leaf_kernel(double* w, int64_t ldw, int n, int j0, int jb, int J0, int J1, BlockScratch* s, LeafMarks* marks,
                unsigned* status, uint64_t wait_ns, unsigned hold) {
  extern __shared__ __align__(16) uint8_t smem[];
  LeafShared& sh = *reinterpret_cast<LeafShared*>(smem);
  double* S = reinterpret_cast<double*>(smem + (sizeof(LeafShared) + 15) / 16 * 16);
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, warps = blockDim.x >> 5, T = blockDim.x;
  const int C = CLUSTER ? (int)cluster_nctarank() : 1, rank = CLUSTER ? (int)cluster_ctarank() : 0;
  const int M = n - j0, r0 = rank * T, rows = max(0, min(T, M - r0));
  if (t < kLeaf) sh.chosen[t] = -1;
  if (marks != nullptr && t == 0) {
    unsigned sm;
    asm("mov.u32 %0, %%smid;" : "=r"(sm));
    if (sm < kSmMarks) marks->sm[sm] = j0 + 1;
    if (rank == 0) marks->latest = j0 + 1;
  }
  if (CLUSTER) {
    if (t < kLeaf) {
      mbar_init(&sh.bar[t], 1);
      if (t < kLeaf / kSub) mbar_init(&sh.row_bar[t], 1);
      fence_barrier_init();
      const uint32_t held = t == kHoldColumn && ((hold >> rank) & 1u) ? 16u : 0u;  // bytes that nobody sends
      mbar_arrive_expect_tx(&sh.bar[t], (uint32_t)C * sizeof(LeafPost) + held);
      if (t < kLeaf / kSub) mbar_arrive_expect_tx(&sh.row_bar[t], kSub * (kLeaf - kSub * t) * 8);
    }
  }
  griddep_wait();  // the kernel before this one in the stream has completed
  // A list that moves nothing, for the launches behind this one should a wait give up before the moves
  // are known; each CTA's own part of the list replaces it at the end, behind a cluster barrier.
  if (CLUSTER && rank == 0 && t < jb) {
    LeafMoves& mv = s->moves[(j0 - J0) / kLeaf];
    mv.piv_src[t] = j0 + t;
    if (t == 0) mv.j0 = j0, mv.jb = jb, mv.disp = 0;
  }
  // the rows into shared memory: 16 lanes per row (coalesced), then a row per thread
  const double* g = w + (int64_t)(j0 + r0) * ldw + j0;
  for (int e = t; e < rows * (kLeaf / 2); e += T) {
    const int r = e / (kLeaf / 2), q = e % (kLeaf / 2) * 2;
    cp_async16(S + r * kLeafStride + q, g + (int64_t)r * ldw + q);  // columns past n are W's padding
  }
  cp_async_commit();
  // a row's other columns of the block, 64 pieces of 16 bytes but the leaf's own, in the background
  const int leaf_piece = (j0 - J0) / 2, pieces = (J1 - J0 + 1) / 2;
  auto fetch_other = [&](double* dst, int row, int q) {
    if (q < pieces && (q < leaf_piece || q >= leaf_piece + kLeaf / 2))
      cp_async16(dst + 2 * q, w + (int64_t)(j0 + row) * ldw + J0 + 2 * q);
  };
  if (rank == 0)
    for (int e = t; e < min(jb, rows) * (kOuter / 2); e += T)
      fetch_other(sh.top_other[e / (kOuter / 2)], e / (kOuter / 2), e % (kOuter / 2));
  cp_async_commit();
  cp_async_wait<1>();  // the rows have landed
  if (CLUSTER) cluster_sync_all();  // every CTA's barriers are set before any post arrives
  else __syncthreads();
  // where this warp sends its CTA's posts: CTA `warp` (and warp + warps, ... of a wide cluster)
  const uint32_t rpost = CLUSTER ? map_rank(&sh.cta_post[0][rank], min(warp, C - 1)) + lane * 16u : 0u;
  const uint32_t rbar = CLUSTER ? map_rank(&sh.bar[0], min(warp, C - 1)) : 0u;
  // Whether this thread's waits have all ended in time. A thread whose wait gave up stays in step (the
  // others may have seen the same posts arrive, and count on it at the CTA's barriers) but sends no
  // post, waits for none and takes no position from one; the CTA agrees at the sub-leaf's barriers.
  bool ok = true;
  // the CTA leaves together: once no copy of its own is in flight, no CTA sends to it any more, and
  // what was sent to it before (microseconds at most) has landed
  auto give_up = [] {
    cp_async_wait<0>();
    cluster_sync_all();
    for (const uint64_t start = global_ns(); global_ns() - start < 20000;) {
    }
  };
  double* srow = S + t * kLeafStride;
  bool active = t < rows;
  int pos = active ? r0 + t : INT_MAX;
#pragma unroll 1
  for (int c0 = 0; c0 < jb; c0 += kSub) {
    double p[kSub];
#pragma unroll
    for (int i = 0; i < kSub; i += 2) {
      const double2 v = t < rows ? *reinterpret_cast<const double2*>(srow + c0 + i) : make_double2(0.0, 0.0);
      p[i] = v.x;
      p[i + 1] = v.y;
    }
    unsigned skip = 0;  // the sub-leaf's columns whose pivot was zero
#pragma unroll
    for (int i = 0; i < kSub; ++i) {
      const int c = c0 + i;
      if (c >= jb) break;
      constexpr unsigned kNone = 0xffffffffu;
      const unsigned long long mag = (unsigned long long)__double_as_longlong(p[i]) & 0x7fffffffffffffffull;
      unsigned hi = 0u;
      if (active) hi = mag <= 0x7ff0000000000000ull ? (unsigned)(mag >> 32) + 2u : (pos == c ? 1u : 0u);
      const unsigned lo = (unsigned)mag;
      const double rcp = leaf_rcp(p[i], active);
      LeafPost* wp = sh.warp_post[i & 1];
      if (lane == leaf_best(hi, lo, (unsigned)pos)) {
        LeafPost& post = wp[warp];
#pragma unroll
        for (int q = i & ~1; q < kSub; q += 2) *reinterpret_cast<double2*>(&post.row[q]) = make_double2(p[q], p[q + 1]);
        const unsigned kind = mag == 0ull ? kPivotZero : (__double2hiint(rcp) == 0 ? kPivotDivide : kPivotInvert);
        *reinterpret_cast<uint4*>(&post.hi) = make_uint4(hi, lo, (unsigned)pos, kind);
        post.rcp = rcp;
      }
      __syncthreads();
      uint4 m = lane < warps ? *reinterpret_cast<const uint4*>(&wp[lane].hi) : make_uint4(0u, 0u, kNone, 0u);
      const LeafPost* win = &wp[leaf_best(m.x, m.y, m.z)];
      if (CLUSTER) {
        if (ok && warp < C && lane < kPostPieces) {
          const double2 v = reinterpret_cast<const double2*>(win)[lane];
          st_async16(rpost + (i & 1) * (uint32_t)sizeof(sh.cta_post[0]), v, rbar + c * 8u);
          for (int dst = warp + warps; dst < C; dst += warps)
            st_async16(map_rank(&sh.cta_post[i & 1][rank], dst) + lane * 16u, v, map_rank(&sh.bar[c], dst));
        }
        ok = ok && mbar_wait_cluster(&sh.bar[c], 0, status, wait_ns);
        __syncwarp();
        const LeafPost* cp = sh.cta_post[i & 1];
        m = lane < C ? *reinterpret_cast<const uint4*>(&cp[lane].hi) : make_uint4(0u, 0u, kNone, 0u);
        win = &cp[leaf_best(m.x, m.y, m.z)];
      }
      // the winner: everything the update reads, in flight at once
      const uint2 meta = *reinterpret_cast<const uint2*>(&win->pos);
      const double r = win->rcp;
      double2 u[kSub / 2];
#pragma unroll
      for (int q = i / 2; q < kSub / 2; ++q) u[q] = reinterpret_cast<const double2*>(win->row)[q];
      if (ok) {
        if (pos == (int)meta.x) {
          active = false;
          pos = c;
          sh.chosen[c] = t;
        } else if (pos == c) {
          pos = (int)meta.x;
        }
      }
      double l = p[i] * r;
      if (meta.y != kPivotInvert) {
        if (meta.y == kPivotZero) skip |= 1u << i;
        else l = p[i] / (i & 1 ? u[i / 2].y : u[i / 2].x);
      }
      if (active && meta.y != kPivotZero) {
        p[i] = l;
#pragma unroll
        for (int q = (i + 1) / 2; q < kSub / 2; ++q) {
          if (2 * q > i) p[2 * q] = fma(l, -u[q].x, p[2 * q]);
          p[2 * q + 1] = fma(l, -u[q].y, p[2 * q + 1]);
        }
      }
    }
    if (t < rows) {
#pragma unroll
      for (int i = 0; i < kSub; i += 2) *reinterpret_cast<double2*>(srow + c0 + i) = make_double2(p[i], p[i + 1]);
    }
    sh.active[t] = active;
    if (CLUSTER) {
      if (!__syncthreads_and(ok)) return give_up();
    } else {
      __syncthreads();
    }
    // the pivot rows held here: their other columns of the block in the background; to every CTA,
    // the row from the sub-leaf's columns on
    for (int k = warp; k < kSub; k += warps) {
      const int row = c0 + k < jb ? sh.chosen[c0 + k] : -1;
      if (row < 0) continue;
      const double* src = S + row * kLeafStride;
      if (CLUSTER) {
        if (lane < (kLeaf - c0) / 2 && c0 + kSub < jb) {
          const double2 v = *reinterpret_cast<const double2*>(src + c0 + 2 * lane);
          for (int dst = 0; dst < C; ++dst)
            st_async16(map_rank(&sh.prow[k][c0 + 2 * lane], dst), v, map_rank(&sh.row_bar[c0 / kSub], dst));
        }
      } else if (lane >= c0) {
        sh.prow[k][lane] = src[lane];
      }
      fetch_other(sh.piv_other[c0 + k], r0 + row, lane);
      fetch_other(sh.piv_other[c0 + k], r0 + row, lane + 32);
    }
    cp_async_commit();
    const int rc0 = c0 + kSub;
    if (rc0 >= jb) break;
    if (CLUSTER) {
      ok = mbar_wait_cluster(&sh.row_bar[c0 / kSub], 0, status, wait_ns);
      __syncwarp();
    } else {
      __syncthreads();
    }
    // U12: the sub-leaf's pivot rows' later columns against their unit lower triangle, a thread per
    // column; a skipped column's row is left as it is, and zero for the update
    if (t < kLeaf - rc0) {
      const int col = rc0 + t;
      double u[kSub], l[kSub][kSub];
#pragma unroll
      for (int k = 0; k < kSub; ++k) u[k] = sh.prow[k][col];
#pragma unroll
      for (int k = 1; k < kSub; ++k)
#pragma unroll
        for (int q = 0; q < k; ++q) l[k][q] = sh.prow[k][c0 + q];
#pragma unroll
      for (int q = 0; q < kSub - 1; ++q)
        if (!((skip >> q) & 1u)) {
#pragma unroll
          for (int k = q + 1; k < kSub; ++k) u[k] = fma(l[k][q], -u[q], u[k]);
        }
#pragma unroll
      for (int k = 0; k < kSub; ++k) {
        const int own = sh.chosen[c0 + k];
        if (own >= 0) S[own * kLeafStride + col] = u[k];
        sh.prow[k][col] = ((skip >> k) & 1u) ? 0.0 : u[k];
      }
    }
    if (CLUSTER) {
      if (!__syncthreads_and(ok)) return give_up();
    } else {
      __syncthreads();
    }
    // the rows not yet chosen: later columns -= L U12, an m16 tile of rows per warp at a time
    {
      const int g2 = lane >> 2, q = lane & 3;
      const bool s0 = (skip >> q) & 1u, s4 = (skip >> (q + 4)) & 1u;
      for (int m = warp * 16; m < rows; m += warps * 16) {
        double* xa = S + (m + g2) * kLeafStride;
        double* xb = xa + 8 * kLeafStride;
        const double a[4] = {s0 ? 0.0 : -xa[c0 + q], s0 ? 0.0 : -xb[c0 + q], s4 ? 0.0 : -xa[c0 + q + 4],
                             s4 ? 0.0 : -xb[c0 + q + 4]};
        const bool sa = sh.active[m + g2], sb = sh.active[m + g2 + 8];
        double2 va[kLeaf / 8 - 1], vb[kLeaf / 8 - 1];
#pragma unroll
        for (int j = 0; j < kLeaf / 8 - 1; ++j)
          if (rc0 + 8 * j < kLeaf) {
            va[j] = *reinterpret_cast<const double2*>(xa + rc0 + 8 * j + 2 * q);
            vb[j] = *reinterpret_cast<const double2*>(xb + rc0 + 8 * j + 2 * q);
          }
#pragma unroll
        for (int j = 0; j < kLeaf / 8 - 1; ++j)
          if (rc0 + 8 * j < kLeaf) {
            const int col = rc0 + 8 * j;
            double d[4] = {va[j].x, va[j].y, vb[j].x, vb[j].y};
            dmma(d, a, sh.prow[q][col + g2], sh.prow[q + 4][col + g2]);
            if (sa) *reinterpret_cast<double2*>(xa + col + 2 * q) = make_double2(d[0], d[1]);
            if (sb) *reinterpret_cast<double2*>(xb + col + 2 * q) = make_double2(d[2], d[3]);
          }
      }
    }
    __syncthreads();
  }

  // only now may the next kernel's CTAs come: any earlier they would wait on SMs that the trailing
  // update on the side stream can use
  griddep_launch_dependents();
  // the moves: rows of the diagonal block that a pivot displaced (all in warp 0 of CTA 0)
  sh.pos[t] = pos;
  if (rank == 0 && warp == 0) {
    const bool moved = t < min(jb, rows) && pos >= jb;
    const unsigned b = __ballot_sync(0xffffffffu, moved);
    const int d = __popc(b & ((1u << lane) - 1u));
    if (moved) sh.disp_src[d] = t, sh.disp_dst[d] = pos;
    if (lane == 0) sh.disp = __popc(b);
  }
  cp_async_wait<0>();
  __syncthreads();
  const bool last = j0 + jb == J1 && j0 > J0;
  if (CLUSTER && !last) cluster_arrive();
  // every CTA has loaded its rows (it has posted for the last column): rows to their positions
  if (jb == kLeaf) {
    for (int e = t; e < rows * (kLeaf / 2); e += T) {
      const int r = e / (kLeaf / 2), q = e % (kLeaf / 2) * 2;
      *reinterpret_cast<double2*>(w + (int64_t)(j0 + sh.pos[r]) * ldw + j0 + q) =
          *reinterpret_cast<const double2*>(S + r * kLeafStride + q);
    }
  } else {
    for (int r = warp; r < rows; r += warps)
      if (lane < jb) w[(int64_t)(j0 + sh.pos[r]) * ldw + j0 + lane] = S[r * kLeafStride + lane];
  }
  // the moved rows' other columns and the lists, for the block's next kernel
  LeafMoves& mv = s->moves[(j0 - J0) / kLeaf];
  const int disp = rank == 0 ? sh.disp : 0;
  for (int e = t; e < (jb + disp) * (kOuter / 2); e += T) {
    const int k = e / (kOuter / 2), q = e % (kOuter / 2) * 2;
    if (k < jb ? sh.chosen[k] >= 0 : true)
      *reinterpret_cast<double2*>(&s->rows[k < jb ? k : kLeaf + k - jb][q]) =
          *reinterpret_cast<const double2*>(k < jb ? &sh.piv_other[k][q] : &sh.top_other[sh.disp_src[k - jb]][q]);
  }
  if (t < jb && sh.chosen[t] >= 0) mv.piv_src[t] = j0 + r0 + sh.chosen[t];
  if (rank == 0) {
    if (t == 0) mv.j0 = j0, mv.jb = jb, mv.disp = disp;
    if (t < disp) mv.disp_src[t] = j0 + sh.disp_src[t], mv.disp_dst[t] = j0 + sh.disp_dst[t];
  }
  if (last) {
    // the block's last leaf: nothing later moves the columns left of it. Every CTA has its moved
    // rows in shared memory (this barrier).
    if (CLUSTER) cluster_sync_all();
    else __syncthreads();
    for (int e = t; e < (jb + disp) * leaf_piece; e += T) {
      const int k = e / leaf_piece, q = e % leaf_piece * 2;
      if (k < jb ? sh.chosen[k] >= 0 : true)
        *reinterpret_cast<double2*>(w + (int64_t)(j0 + (k < jb ? k : sh.disp_dst[k - jb])) * ldw + J0 + q) =
            *reinterpret_cast<const double2*>(k < jb ? &sh.piv_other[k][q] : &sh.top_other[sh.disp_src[k - jb]][q]);
    }
  } else if (CLUSTER) {
    cluster_wait();  // no CTA leaves while another may still send to it
  }
}

// CTAs of a leaf of M rows: one up to 512 rows; then, as the CTAs' own part of a column (512 rows:
// ~500 cycles more than 128) costs more than a wider exchange, 256 rows each up to 16 CTAs.
constexpr int kLeafRows = 256;

static cudaLaunchConfig_t leaf_config(cudaLaunchAttribute* attr, int ctas, int threads) {
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = ctas;
  attr->val.clusterDim.y = 1;
  attr->val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = leaf_smem(threads);
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// The largest cluster of whole leaf CTAs that this device can place; a single CTA needs none.
static int find_leaf_cluster_limit() {
  if (smem_attribute(leaf_kernel<true>, leaf_smem(kLeafMaxThreads)) == RM_OK &&
      func_attribute(reinterpret_cast<const void*>(leaf_kernel<true>),
                     cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == RM_OK)
    for (int C = kLeafMaxCtas; C > 1; C /= 2) {
      cudaLaunchAttribute attr;
      const cudaLaunchConfig_t cfg = leaf_config(&attr, C, kLeafMaxThreads);
      int clusters = 0;
      if (cudaOccupancyMaxActiveClusters(&clusters, leaf_kernel<true>, &cfg) == cudaSuccess && clusters > 0) return C;
      cudaGetLastError();
    }
  cudaGetLastError();
  return 1;
}

static thread_local int g_leaf_ctas = kLeafMaxCtas;  // lowered by tests only

// Found once per device.
static int leaf_cluster_limit() {
  static std::mutex mu;
  static std::vector<int> limits;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 1;
  std::lock_guard<std::mutex> lock(mu);
  if ((int)limits.size() <= dev) limits.resize(dev + 1, 0);
  if (!limits[dev]) limits[dev] = find_leaf_cluster_limit();
  return std::min(limits[dev], g_leaf_ctas);
}

int leaf_max_rows() { return leaf_cluster_limit() * kLeafMaxThreads; }

int leaf_f64(double* w, int64_t ldw, int n, int j0, int jb, int J0, int J1, BlockScratch* s, LeafMarks* marks,
             unsigned* status, cudaStream_t stream) {
  const int M = n - j0;
  int C = 1;
  if (M > kLeafMaxThreads) {
    const int limit = leaf_cluster_limit();
    while (C < limit && M > C * kLeafRows) C *= 2;
    if (M > C * kLeafMaxThreads) return RM_BAD_ARG;
  }
  const int T = std::max(32, ((M + C - 1) / C + 31) / 32 * 32);
  if (C == 1) {
    RM_TRY(smem_attribute(leaf_kernel<false>, leaf_smem(kLeafMaxThreads)));
    RM_CUDA_TRY(launch_dependent(leaf_kernel<false>, dim3(1), dim3(T), leaf_smem(T), stream, w, ldw, n, j0, jb, J0, J1, s,
                                 marks, status, kWaitLimitNs, 0u));
    note_launch();
    return RM_OK;
  }
  cudaLaunchAttribute attr;  // the kernel's attributes are set since the limit was found
  cudaLaunchConfig_t cfg = leaf_config(&attr, C, T);
  cfg.stream = stream;
  unsigned hold = 0u;  // a self-test's leaf, with a short limit
  if (injected_failure(RM_INJECT_LEAF_TIMEOUT)) hold = 0xffffffffu;
  else if (injected_failure(RM_INJECT_LEAF_CTA_TIMEOUT)) hold = 1u << (C - 1);
  RM_CUDA_TRY(cudaLaunchKernelEx(&cfg, leaf_kernel<true>, w, ldw, n, j0, jb, J0, J1, s, marks, status,
                                 hold ? kSelfTestWaitNs : kWaitLimitNs, hold));
  note_launch();
  return RM_OK;
}

// The block's other columns of the cnt moved rows into s->rows (or, with SCATTER, the columns left of the
// leaf from there to their new positions), 16 bytes per thread and four in flight. pos: the rows relative
// to j0; at: the first row's slot.
template <bool SCATTER>
__device__ __forceinline__ void move_rows(double* w, int64_t ldw, int j0, int J0, BlockScratch* s, const int* pos,
                                          int cnt, int at) {
  constexpr int kPer = kOuter / 2;  // 16-byte pieces of a row
  const int total = cnt * kPer;
  const int lc = (j0 - J0) / 2;  // the leaf's first piece
  for (int e0 = threadIdx.x; e0 < total; e0 += 4 * (int)blockDim.x) {
    double2 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = e0 + u * (int)blockDim.x, i = e / kPer, q = e % kPer;
      if (e < total && (q < lc || (!SCATTER && q >= lc + kLeaf / 2)))
        v[u] = SCATTER ? *reinterpret_cast<const double2*>(&s->rows[at + i][2 * q])
                       : *reinterpret_cast<const double2*>(w + (int64_t)(j0 + pos[i]) * ldw + J0 + 2 * q);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = e0 + u * (int)blockDim.x, i = e / kPer, q = e % kPer;
      if (e < total && (q < lc || (!SCATTER && q >= lc + kLeaf / 2))) {
        if constexpr (SCATTER) *reinterpret_cast<double2*>(w + (int64_t)(j0 + pos[i]) * ldw + J0 + 2 * q) = v[u];
        else *reinterpret_cast<double2*>(&s->rows[at + i][2 * q]) = v[u];
      }
    }
  }
}

// The moves of a leaf whose rows were swapped one after another (ipiv, absolute): their net
// effect, then the same buffer and lists. One CTA; only leaves taller than leaf_max_rows() come here.
__global__ void __launch_bounds__(256) leaf_moves_kernel(double* w, int64_t ldw, int j0, int jb, int J0, int J1,
                                                         const int64_t* __restrict__ ipiv, BlockScratch* s) {
  __shared__ int pos[2 * kLeaf], src[2 * kLeaf], cnt_s;
  const int t = threadIdx.x;
  if (t == 0) {
    int cnt = jb;
    for (int q = 0; q < jb; ++q) pos[q] = src[q] = q;
    for (int i = 0; i < jb; ++i) {
      const int p = (int)(ipiv[j0 + i] - j0);
      if (p == i) continue;
      int e = p;
      if (p >= jb) {
        for (e = jb; e < cnt && pos[e] != p; ++e) {
        }
        if (e == cnt) pos[cnt] = src[cnt] = p, ++cnt;
      }
      const int v = src[i];
      src[i] = src[e];
      src[e] = v;
    }
    // a position past the leaf that ends with a row from past the leaf would be a third kind of
    // move; one swap per pivot, each with the diagonal's position, never makes one
    cnt_s = cnt;
  }
  __syncthreads();
  const int disp = cnt_s - jb;
  move_rows<false>(w, ldw, j0, J0, s, src, jb, 0);
  move_rows<false>(w, ldw, j0, J0, s, src + jb, disp, kLeaf);
  LeafMoves& mv = s->moves[(j0 - J0) / kLeaf];
  if (t == 0) mv.j0 = j0, mv.jb = jb, mv.disp = disp;
  if (t < jb) mv.piv_src[t] = j0 + src[t];
  if (t < disp) mv.disp_src[t] = j0 + src[jb + t], mv.disp_dst[t] = j0 + pos[jb + t];
  __syncthreads();
  if (j0 + jb == J1 && j0 > J0) {
    move_rows<true>(w, ldw, j0, J0, s, pos, jb, 0);
    move_rows<true>(w, ldw, j0, J0, s, pos + jb, disp, kLeaf);
  }
}

int leaf_moves_f64(double* w, int64_t ldw, int j0, int jb, int J0, int J1, const int64_t* ipiv, BlockScratch* s,
                   cudaStream_t stream) {
  leaf_moves_kernel<<<1, 256, 0, stream>>>(w, ldw, j0, jb, J0, J1, ipiv, s);
  RM_LAUNCHED();
  return RM_OK;
}

// ------------------------------------------------------------------ the rest of the block
// The leaf's rows of the block's later columns and those columns' update, a CTA per 64 rows. Every
// CTA forms U12 (32 x up to 96) for itself from the moved rows' buffer: a thread per column, its
// 32 items in registers, the same fmas in the same order as the reference's rank-1 updates. The
// CTA with the diagonal rows stores it. Then C -= L21 U12 on DMMA, 8 warps of 16 x 48.
constexpr int kTailRows = 64;
constexpr int kTailLda = 36;   // row strides whose fragment loads hit 16 distinct 8-byte banks
constexpr int kTailLdu = 100;
constexpr size_t kTailSmem = ((size_t)kLeaf * kTailLdu + (size_t)kTailRows * kTailLda + kLeaf * kLeaf) * sizeof(double);

__global__ void __launch_bounds__(256) leaf_tail_kernel(double* w, int64_t ldw, int n, int j0, int J0, int J1,
                                                        const BlockScratch* __restrict__ s) {
  extern __shared__ __align__(16) double tsm[];
  double* U = tsm;                      // [32][kTailLdu]
  double* A = U + kLeaf * kTailLdu;     // [64][kTailLda], negated multipliers
  double* Lc = A + kTailRows * kTailLda;  // [32][32], Lc[i][r] = L11(r, i)
  __shared__ int from[kTailRows];         // the row's row of the buffer, or -1
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r0 = j0 + blockIdx.x * kTailRows, c0 = j0 + kLeaf, cols = J1 - c0, off = c0 - J0;
  griddep_launch_dependents();
  griddep_wait();  // the kernel before this one in the stream has completed
  const LeafMoves& mv = s->moves[(j0 - J0) / kLeaf];
  if (warp == 0) {
    const int disp = mv.disp, dst = mv.disp_dst[lane] - r0;
    from[lane] = blockIdx.x == 0 ? lane : -1;
    from[lane + kLeaf] = -1;
    __syncwarp();
    if (lane < disp && dst >= 0 && dst < kTailRows) from[dst] = kLeaf + lane;
  }
  double x[kLeaf];
  if (tid < cols)
#pragma unroll
    for (int i = 0; i < kLeaf; ++i) x[i] = s->rows[i][off + tid];
  {
    double lv[kLeaf / 8], av[kTailRows / 8];
#pragma unroll
    for (int i = 0; i < kLeaf / 8; ++i) lv[i] = w[(int64_t)(j0 + warp + 8 * i) * ldw + j0 + lane];
#pragma unroll
    for (int i = 0; i < kTailRows / 8; ++i) {
      const int r = r0 + warp + 8 * i;
      av[i] = r < n ? -w[(int64_t)r * ldw + j0 + lane] : 0.0;
    }
#pragma unroll
    for (int i = 0; i < kLeaf / 8; ++i) Lc[lane * kLeaf + warp + 8 * i] = lv[i];
#pragma unroll
    for (int i = 0; i < kTailRows / 8; ++i) A[(warp + 8 * i) * kTailLda + lane] = av[i];
  }
  __syncthreads();
  // The update's rows and the moved rows' columns left of the leaf (at most 64) are asked for here, to
  // arrive behind U12: loaded one after another where they are used, they were most of this kernel.
  const int g = lane >> 2, q = lane & 3, m0 = 16 * (warp >> 1);
  const bool update = blockIdx.x != 0 || m0 >= kLeaf;  // not the diagonal rows
  const int ra = m0 + g, rb = ra + 8;
  const bool va = update && r0 + ra < n, vb = update && r0 + rb < n;
  double acc[6][4];
  {
    const double* srca = from[ra] >= 0 ? s->rows[from[ra]] + off : w + (int64_t)(r0 + ra) * ldw + c0;
    const double* srcb = from[rb] >= 0 ? s->rows[from[rb]] + off : w + (int64_t)(r0 + rb) * ldw + c0;
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      const int c = 48 * (warp & 1) + 8 * j + 2 * q;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        acc[j][h] = va && c + h < cols ? srca[c + h] : 0.0;
        acc[j][2 + h] = vb && c + h < cols ? srcb[c + h] : 0.0;
      }
    }
  }
  constexpr int kLeft = (kOuter - 2 * kLeaf) / 32;
  double moved[kTailRows / 8][kLeft];
#pragma unroll
  for (int i = 0; i < kTailRows / 8; ++i)
#pragma unroll
    for (int h = 0; h < kLeft; ++h) {
      const int e = from[warp + 8 * i], c = lane + 32 * h;
      moved[i][h] = e >= 0 && c < j0 - J0 ? s->rows[e][c] : 0.0;
    }
  if (tid < cols) {
#pragma unroll
    for (int i = 0; i < kLeaf - 1; ++i) {
      const double* l = Lc + i * kLeaf;
#pragma unroll
      for (int r = i + 1; r < kLeaf; ++r) x[r] = fma(l[r], -x[i], x[r]);
    }
#pragma unroll
    for (int i = 0; i < kLeaf; ++i) U[i * kTailLdu + tid] = x[i];
    if (blockIdx.x == 0)
#pragma unroll
      for (int i = 0; i < kLeaf; ++i) w[(int64_t)(j0 + i) * ldw + c0 + tid] = x[i];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kTailRows / 8; ++i)
#pragma unroll
    for (int h = 0; h < kLeft; ++h) {
      const int r = warp + 8 * i, c = lane + 32 * h;
      if (from[r] >= 0 && c < j0 - J0) w[(int64_t)(r0 + r) * ldw + J0 + c] = moved[i][h];
    }
  if (!update) return;
#pragma unroll
  for (int k = 0; k < kLeaf; k += 8) {
    const double a[4] = {A[ra * kTailLda + k + q], A[rb * kTailLda + k + q], A[ra * kTailLda + k + q + 4],
                         A[rb * kTailLda + k + q + 4]};
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      const int c = 48 * (warp & 1) + 8 * j + g;
      dmma(acc[j], a, U[(k + q) * kTailLdu + c], U[(k + q + 4) * kTailLdu + c]);
    }
  }
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    const int c = 48 * (warp & 1) + 8 * j + 2 * q;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (va && c + h < cols) w[(int64_t)(r0 + ra) * ldw + c0 + c + h] = acc[j][h];
      if (vb && c + h < cols) w[(int64_t)(r0 + rb) * ldw + c0 + c + h] = acc[j][2 + h];
    }
  }
}

int leaf_tail_f64(double* w, int64_t ldw, int n, int j0, int J0, int J1, const BlockScratch* s, cudaStream_t stream) {
  RM_TRY(smem_attribute(leaf_tail_kernel, kTailSmem));
  const int grid = (n - j0 + kTailRows - 1) / kTailRows;
  RM_CUDA_TRY(launch_dependent(leaf_tail_kernel, dim3(grid), dim3(256), kTailSmem, stream, w, ldw, n, j0, J0, J1, s));
  note_launch();
  return RM_OK;
}

// ------------------------------------------------------------------ the block's rows
// A CTA per 64 columns outside the block (all of those left of it, or none, and lo .. hi - 1 of
// those right of it): the net moves of the block's four leaves, then, right of the block, U12 =
// L11^-1 A12 in shared memory: the four 32 x 32 diagonal blocks of L11 are inverted by a warp each
// (a lane per column) while the other warps work out the moves, and per block row X_b = D_b^-1 (A_b -
// sum) and the rows below it are updated, all on DMMA. One launch in place of a swap, an inversion
// of the whole L11 and a product with it. 64 columns: the lists, L11 and its inverses are per CTA,
// and at 8192 columns the CTAs still fit one wave.
constexpr int kBrCols = 64;
constexpr int kBrLdx = kBrCols + 4;   // fragment loads of both operands hit 16 distinct 8-byte banks
constexpr int kBrLda = kOuter + 4;
// where the inverse of L11's diagonal block b lies: blocks (0, 1), (1, 2), (2, 3) and (0, 3)
__device__ __forceinline__ int inverse_at(int b) {
  return b < kOuter / kLeaf - 1 ? kLeaf * b * kBrLda + kLeaf * (b + 1) : kLeaf * b;
}
constexpr size_t kBrSmem = ((size_t)kOuter * kBrLdx + (size_t)kOuter * kBrLda) * sizeof(double);

__global__ void __launch_bounds__(256) block_rows_kernel(double* w, int64_t ldw, int J0, int nb, int left_cols, int lo,
                                                         int hi, const BlockScratch* __restrict__ s, int64_t* perm) {
  extern __shared__ __align__(16) double bsm[];
  double* X = bsm;                      // [128][kBrLdx]: the block's rows
  double* L = bsm + kOuter * kBrLdx;    // [128][kBrLda]: L11, D_b^-1 in its diagonal blocks
  __shared__ LeafMoves mv[kOuter / kLeaf];
  __shared__ int4 dsts[kOuter / kLeaf][kLeaf / 4];  // disp_dst, -1 past disp
  __shared__ int src[kOuter], xdst[kOuter], xsrc[kOuter], extra;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int leaves = (nb + kLeaf - 1) / kLeaf, J1 = J0 + nb;
  griddep_launch_dependents();
  griddep_wait();  // the kernel before this one in the stream has completed
  // CTAs 0 .. left - 1 take the columns left of the block, the others lo .. hi - 1, right of it (and
  // then the block is whole: nb = 128)
  const int left = (left_cols + kBrCols - 1) / kBrCols;
  const bool solve = (int)blockIdx.x >= left;
  const int c0 = solve ? lo + ((int)blockIdx.x - left) * kBrCols : (int)blockIdx.x * kBrCols;
  const int cols = min(kBrCols, (solve ? hi : left_cols) - c0);  // <= 0 when only perm is left to move
  if (solve && cols > 0) {
    for (int e = tid; e < kOuter * kOuter / 2; e += 256) {
      const int r = e / (kOuter / 2), c = e % (kOuter / 2) * 2;
      if (c <= r) cp_async16(L + r * kBrLda + c, w + (int64_t)(J0 + r) * ldw + J0 + c);
    }
  }
  for (int e = tid; e < leaves * (int)(sizeof(LeafMoves) / 4); e += 256)
    reinterpret_cast<int*>(mv)[e] = reinterpret_cast<const int*>(s->moves)[e];
  if (tid < kOuter) {
    const int l = tid / kLeaf, d = tid % kLeaf;
    reinterpret_cast<int*>(dsts)[tid] = l < leaves && d < s->moves[l].disp ? s->moves[l].disp_dst[d] : -1;
  }
  if (tid == 0) extra = 0;
  cp_async_wait_all();
  __syncthreads();
  // the displaced row of leaf l that ends at position p, or -1
  auto find = [&](int p, int l) {
    int at = -1;
#pragma unroll
    for (int i = 0; i < kLeaf / 4; ++i) {
      const int4 v = dsts[l][i];
      if (v.x == p) at = 4 * i;
      if (v.y == p) at = 4 * i + 1;
      if (v.z == p) at = 4 * i + 2;
      if (v.w == p) at = 4 * i + 3;
    }
    return at;
  };
  // the row that ends at position p after all leaves was at position back(p, leaves) before them
  auto back = [&](int p, int l) {
    for (--l; l >= 0; --l) {
      const LeafMoves& m = mv[l];
      if (p >= m.j0 && p < m.j0 + m.jb) {
        p = m.piv_src[p - m.j0];
      } else {
        const int d = find(p, l);
        if (d >= 0) p = m.disp_src[d];
      }
    }
    return p;
  };
  const bool invert_ahead = solve && cols > 0;
  const int lt = invert_ahead ? tid - kOuter : tid;  // the lists by warps 4..7 beside the inverses, or by all
  if (invert_ahead && warp < 4) {
    // D_b^-1 of the diagonal block b = warp, a lane per column, into a block of L's unused upper part
    const double* D = L + (kLeaf * warp) * kBrLda + kLeaf * warp;
    double x[kLeaf];
#pragma unroll
    for (int i = 0; i < kLeaf; ++i) x[i] = i == lane ? 1.0 : 0.0;
#pragma unroll
    for (int i = 0; i < kLeaf - 1; ++i)
#pragma unroll
      for (int r = i + 1; r < kLeaf; ++r) x[r] = fma(D[r * kBrLda + i], -x[i], x[r]);
    double* V = L + inverse_at(warp);
#pragma unroll
    for (int i = 0; i < kLeaf; ++i) V[i * kBrLda + lane] = x[i];
  }
  if (lt >= 0 && lt < kOuter) src[lt] = lt < nb ? back(J0 + lt, leaves) : J0 + lt;
  if (tid >= kOuter) {
    // positions below the block, each once: by the last leaf that moved a row there
    const int l = (tid - kOuter) / kLeaf, d = (tid - kOuter) % kLeaf;
    if (l < leaves && d < mv[l].disp && mv[l].disp_dst[d] >= J1) {
      const int p = mv[l].disp_dst[d];
      bool last = true;
      for (int l2 = l + 1; l2 < leaves; ++l2) last &= find(p, l2) < 0;
      const int from = last ? back(p, leaves) : p;
      if (last && from != p) {
        const int e = atomicAdd(&extra, 1);
        xdst[e] = p;
        xsrc[e] = from;
      }
    }
  }
  __syncthreads();
  const int extras = extra;
  if (perm != nullptr && blockIdx.x == 0) {
    const bool mine = tid < kOuter ? tid < nb : tid - kOuter < extras;
    int64_t v = 0;
    if (mine) v = perm[tid < kOuter ? src[tid] : xsrc[tid - kOuter]];
    __syncthreads();
    if (mine) perm[tid < kOuter ? J0 + tid : xdst[tid - kOuter]] = v;
  }
  if (cols <= 0) return;
  // every moved row's items of these columns, a pair per lane, before any is stored
  const int c = 2 * lane;
  const bool one = c < cols, two = c + 1 < cols;
  auto get = [&](int row) {
    double2 v = make_double2(0.0, 0.0);
    const double* p = w + (int64_t)row * ldw + c0 + c;
    if (two) v = *reinterpret_cast<const double2*>(p);
    else if (one) v.x = *p;
    return v;
  };
  auto put = [&](int row, double2 v) {
    double* p = w + (int64_t)row * ldw + c0 + c;
    if (two) *reinterpret_cast<double2*>(p) = v;
    else if (one) *p = v.x;
  };
  double2 xv[kOuter / 8];
#pragma unroll
  for (int q = 0; q < kOuter / 8; ++q) {
    const int e = warp + 8 * q;
    xv[q] = e < extras ? get(xsrc[e]) : make_double2(0.0, 0.0);
  }
  bool plain = true;  // neither infinities nor NaN in the block's rows
#pragma unroll
  for (int q = 0; q < kOuter / 8; ++q) {
    const int e = warp + 8 * q;
    if (e < nb) {
      const double2 v = get(src[e]);
      *reinterpret_cast<double2*>(X + e * kBrLdx + c) = v;
      plain = plain && fabs(v.x) < INFINITY && fabs(v.y) < INFINITY;
    }
  }
  // A product with the inverses' zeros would spread an infinity or a NaN to rows that rustymath's
  // substitution leaves alone: such columns are substituted, a thread per column.
  const bool invert = solve && __syncthreads_and(plain ? 1 : 0);
  if (solve && !invert) {
    if (tid < kBrCols)
      for (int i = 1; i < kOuter; ++i)
        for (int r = 0; r < i; ++r) X[i * kBrLdx + tid] = fma(L[i * kBrLda + r], -X[r * kBrLdx + tid], X[i * kBrLdx + tid]);
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kOuter / 8; ++q) {
    const int e = warp + 8 * q;
    if (e < extras) put(xdst[e], xv[q]);
  }
  if (invert) {
    const int g = lane >> 2, q = lane & 3;
    // warp: an m16 tile of the block row and two n8 tiles of columns
    const int n0 = 16 * (warp & 3);
    for (int b = 0; b < kOuter / kLeaf; ++b) {
      const int m0 = kLeaf * b + 16 * (warp >> 2);
      double d[2][4] = {{0.0, 0.0, 0.0, 0.0}, {0.0, 0.0, 0.0, 0.0}};
#pragma unroll
      for (int k = 0; k < kLeaf; k += 8) {
        const double* a0 = L + inverse_at(b) + (16 * (warp >> 2) + g) * kBrLda + k + q;
        const double a[4] = {a0[0], a0[8 * kBrLda], a0[4], a0[8 * kBrLda + 4]};
        const double* x0 = X + (kLeaf * b + k + q) * kBrLdx + n0 + g;
        dmma(d[0], a, x0[0], x0[4 * kBrLdx]);
        dmma(d[1], a, x0[8], x0[4 * kBrLdx + 8]);
      }
      __syncthreads();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        *reinterpret_cast<double2*>(X + (m0 + g) * kBrLdx + n0 + 8 * h + 2 * q) = make_double2(d[h][0], d[h][1]);
        *reinterpret_cast<double2*>(X + (m0 + g + 8) * kBrLdx + n0 + 8 * h + 2 * q) = make_double2(d[h][2], d[h][3]);
      }
      __syncthreads();
      if (b + 1 == kOuter / kLeaf) break;
      // the rows below: X_c -= L_cb X_b
      double xb[kLeaf / 8][2][2];
#pragma unroll
      for (int k = 0; k < kLeaf / 8; ++k)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const double* x0 = X + (kLeaf * b + 8 * k + q) * kBrLdx + n0 + 8 * h + g;
          xb[k][h][0] = -x0[0];
          xb[k][h][1] = -x0[4 * kBrLdx];
        }
      for (int m = kLeaf * (b + 1) + 16 * (warp >> 2); m < kOuter; m += 32) {
        double* xr = X + (m + g) * kBrLdx + n0 + 2 * q;
        double acc[2][4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const double2 u = *reinterpret_cast<const double2*>(xr + 8 * h), v = *reinterpret_cast<const double2*>(xr + 8 * kBrLdx + 8 * h);
          acc[h][0] = u.x, acc[h][1] = u.y, acc[h][2] = v.x, acc[h][3] = v.y;
        }
#pragma unroll
        for (int k = 0; k < kLeaf; k += 8) {
          const double* a0 = L + (m + g) * kBrLda + kLeaf * b + k + q;
          const double a[4] = {a0[0], a0[8 * kBrLda], a0[4], a0[8 * kBrLda + 4]};
          dmma(acc[0], a, xb[k / 8][0][0], xb[k / 8][0][1]);
          dmma(acc[1], a, xb[k / 8][1][0], xb[k / 8][1][1]);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          *reinterpret_cast<double2*>(xr + 8 * h) = make_double2(acc[h][0], acc[h][1]);
          *reinterpret_cast<double2*>(xr + 8 * kBrLdx + 8 * h) = make_double2(acc[h][2], acc[h][3]);
        }
      }
      __syncthreads();
    }
  }
#pragma unroll
  for (int q = 0; q < kOuter / 8; ++q) {
    const int e = warp + 8 * q;
    if (e < nb) put(J0 + e, *reinterpret_cast<const double2*>(X + e * kBrLdx + c));
  }
}

int block_rows_f64(double* w, int64_t ldw, int J0, int nb, bool left, int lo, int hi, const BlockScratch* s, int64_t* perm,
                   cudaStream_t stream) {
  const int left_cols = left ? J0 : 0;
  const int grid = std::max(perm ? 1 : 0, (left_cols + kBrCols - 1) / kBrCols + std::max(0, hi - lo + kBrCols - 1) / kBrCols);
  if (grid == 0) return RM_OK;
  RM_TRY(smem_attribute(block_rows_kernel, kBrSmem));
  RM_CUDA_TRY(launch_dependent(block_rows_kernel, dim3(grid), dim3(256), kBrSmem, stream, w, ldw, J0, nb, left_cols, lo,
                               hi, s, perm));
  note_launch();
  return RM_OK;
}

}  // namespace rm

extern "C" int rm_test_limit_leaf_ctas(int ctas) {
  if (ctas < 0 || ctas > rm::kLeafMaxCtas || (ctas & (ctas - 1))) return RM_BAD_ARG;
  rm::g_leaf_ctas = ctas ? ctas : rm::kLeafMaxCtas;
  return RM_OK;
}
