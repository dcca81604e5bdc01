// FP64 GEMM on the B200's FP64 tensor path: TMA-fed shared-memory tiles, mma.sync f64.
//
// Replaces rustymath's packed product (core/src/linalg.rs:1353-1426) and its AVX2 6x8
// micro-kernel (linalg.rs:1282); the operation is Tiled::gemm (linalg.rs:772-774),
// C = alpha*op(A)*op(B) + beta*C on row-major views. tcgen05 has no f64 kind, so the FP64
// tensor cores are reached through warp-level mma.sync.m16n8k8.f64 (DMMA).
//
// Pipeline: thread 0 issues cp.async.bulk.tensor loads (128-byte swizzle) STAGES-1 k-tiles
// ahead into a ring of stages guarded by full/empty mbarriers; the warps read fragments with
// 8-byte shared loads and run DMMA. (No separate producer warp: a ninth warp would cut every
// thread's register budget to 168 and spill the 64x32 accumulator tile.) The mma row/column each thread's fragment covers
// is mapped to a tile row/column (fragment maps below) so that every fragment load of a
// half-warp touches 16 distinct 8-byte bank pairs under the 128-byte swizzle.
#include <climits>

#include "dgemm_lower.cuh"
#include "getrf_block.cuh"
#include "rm_internal.h"

namespace rm {

// Columns of a 16-wide swizzled slice that mma column g (0..7) of the slice's first (h=0)
// or second (h=1) n8 tile reads: {0,1,8,9,2,3,10,11} and the same plus 4.
__device__ __forceinline__ uint32_t rho(uint32_t g, uint32_t h) {
  return ((g & 1u) | ((g & 2u) << 2) | ((g & 4u) >> 1)) + 4u * h;
}

template <int BM_, int BN_, int WM_, int WN_, int STAGES_, bool TA_, bool TB_>
struct DgemmCfg {
  static constexpr int BM = BM_, BN = BN_, WM = WM_, WN = WN_, STAGES = STAGES_;
  static constexpr bool TA = TA_, TB = TB_;
  static constexpr int BK = 16;
  static constexpr int WARPS_M = BM / WM, WARPS_N = BN / WN;
  static constexpr int COMPUTE_WARPS = WARPS_M * WARPS_N;
  static constexpr int THREADS = COMPUTE_WARPS * 32;
  static constexpr int A_BYTES = BM * BK * 8, B_BYTES = BN * BK * 8;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int SMEM = STAGES * STAGE_BYTES + 1024 + 2 * STAGES * 8;
  static constexpr int MI = WM / 16, NJ = WN / 8;
  static constexpr bool PIPE = MI * NJ <= 2;  // few products per step, few warps: fetch a step ahead
  static_assert(BM % 16 == 0 && BN % 16 == 0 && WM % 16 == 0 && WN % 16 == 0, "tile shape");
  static_assert(BM <= 256 && BN <= 256, "TMA box extent");
};

// Byte offset of operand item (mn, k) in a stage's tile: K-major tiles hold one 128-byte
// row per M/N index; MN-major tiles hold 16-wide boxes of 16 k rows (2 KB each).
template <bool KMAJOR>
__device__ __forceinline__ uint32_t tile_off(uint32_t mn, uint32_t k) {
  if (KMAJOR) return swz128_f64(mn, k);
  return (mn >> 4) * 2048u + swz128_f64(k, mn & 15u);
}

template <class C>
__global__ void __launch_bounds__(C::THREADS, 1)
    dgemm_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                 double* __restrict__ c, int64_t ldc, int m, int n, int k, double alpha, double beta, bool lower,
                 unsigned* status) {
  if (lower && (int)(blockIdx.x * C::BN) >= (int)(blockIdx.y + 1) * C::BM) return;  // strictly above the diagonal
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::STAGES * C::STAGE_BYTES);
  uint64_t* empty = full + C::STAGES;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.y * C::BM, n0 = blockIdx.x * C::BN;
  const int ktiles = (k + C::BK - 1) / C::BK;
  griddep_launch_dependents();
  griddep_wait();  // the kernel before this one in the stream has completed

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], C::COMPUTE_WARPS);
    }
    fence_barrier_init();
  }
  __syncthreads();

  // Thread 0 also issues the TMA loads: k-tile kt goes to stage kt % STAGES once every warp
  // has released that stage's previous k-tile (kt - STAGES).
  bool producing = true;
  auto issue = [&](int kt) {
    const int s = kt % C::STAGES;
    if (kt >= C::STAGES && !mbar_wait(&empty[s], ((kt - C::STAGES) / C::STAGES) & 1u, status)) {
      producing = false;
      return;
    }
    uint8_t* sa = smem + s * C::STAGE_BYTES;
    uint8_t* sb = sa + C::A_BYTES;
    mbar_arrive_expect_tx(&full[s], C::STAGE_BYTES);
    const int k0 = kt * C::BK;
    if (!C::TA) {
      tma_load_2d(sa, &tma_a, &full[s], k0, m0);
    } else {
#pragma unroll
      for (int b = 0; b < C::BM / 16; ++b) tma_load_2d(sa + b * 2048, &tma_a, &full[s], m0 + 16 * b, k0);
    }
    if (C::TB) {
      tma_load_2d(sb, &tma_b, &full[s], k0, n0);
    } else {
#pragma unroll
      for (int b = 0; b < C::BN / 16; ++b) tma_load_2d(sb + b * 2048, &tma_b, &full[s], n0 + 16 * b, k0);
    }
  };
  int issued = 0;
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tma_a);
    tma_prefetch_desc(&tma_b);
    for (; issued < C::STAGES - 1 && issued < ktiles && producing; ++issued) issue(issued);
  }

  // ---------------- compute warps
  const int wm0 = (warp / C::WARPS_N) * C::WM, wn0 = (warp % C::WARPS_N) * C::WN;
  const uint32_t g = lane >> 2, t = lane & 3;

  // Fragment maps: tile row of mma row r (0..15) of m16 tile i; tile column of mma column
  // q (0..7) of n8 tile j.
  auto arow = [&](int i, uint32_t r) -> uint32_t {
    return C::TA ? (wm0 + 16 * i + rho(r & 7u, r >> 3)) : (wm0 + 16 * i + 2 * (r & 7u) + (r >> 3));
  };
  auto bcol = [&](int j, uint32_t q) -> uint32_t {
    return C::TB ? (wn0 + 16 * (j >> 1) + 2 * q + (j & 1)) : (wn0 + 16 * (j >> 1) + rho(q, j & 1));
  };

  double acc[C::MI][C::NJ][4];
#pragma unroll
  for (int i = 0; i < C::MI; ++i)
#pragma unroll
    for (int j = 0; j < C::NJ; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0;

  // The fragments of 8 k's. k offsets kk and kk + 4 change the swizzled chunk by XOR, so they are
  // recomputed per k.
  auto load_frags = [&](int st, int kk, double (&af)[C::MI][4], double (&bf)[C::NJ][2]) {
    const uint8_t* sa = smem + st * C::STAGE_BYTES;
    const uint8_t* sb = sa + C::A_BYTES;
#pragma unroll
    for (int i = 0; i < C::MI; ++i) {
      const uint32_t r0 = arow(i, g), r1 = arow(i, g + 8);
      af[i][0] = *reinterpret_cast<const double*>(sa + tile_off<!C::TA>(r0, kk + t));
      af[i][1] = *reinterpret_cast<const double*>(sa + tile_off<!C::TA>(r1, kk + t));
      af[i][2] = *reinterpret_cast<const double*>(sa + tile_off<!C::TA>(r0, kk + t + 4));
      af[i][3] = *reinterpret_cast<const double*>(sa + tile_off<!C::TA>(r1, kk + t + 4));
    }
#pragma unroll
    for (int j = 0; j < C::NJ; ++j) {
      const uint32_t q = bcol(j, g);
      bf[j][0] = *reinterpret_cast<const double*>(sb + tile_off<C::TB>(q, kk + t));
      bf[j][1] = *reinterpret_cast<const double*>(sb + tile_off<C::TB>(q, kk + t + 4));
    }
  };
  auto multiply = [&](const double (&af)[C::MI][4], const double (&bf)[C::NJ][2]) {
#pragma unroll
    for (int i = 0; i < C::MI; ++i)
#pragma unroll
      for (int j = 0; j < C::NJ; ++j)
        asm volatile(
            "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
            "{%0,%1,%2,%3};"
            : "+d"(acc[i][j][0]), "+d"(acc[i][j][1]), "+d"(acc[i][j][2]), "+d"(acc[i][j][3])
            : "d"(af[i][0]), "d"(af[i][1]), "d"(af[i][2]), "d"(af[i][3]), "d"(bf[j][0]), "d"(bf[j][1]));
  };

  bool ok = true;
  if constexpr (C::PIPE) {
    // few warps per SM: the next 8 k's fragments are loaded before this step's products, so that
    // neither the shared loads' latency nor a stage's barrier stands between products
    double af[2][C::MI][4], bf[2][C::NJ][2];
    ok = mbar_wait(&full[0], 0u, status);
    if (ok) load_frags(0, 0, af[0], bf[0]);
    for (int kt = 0; ok && kt < ktiles; ++kt) {
      if (threadIdx.x == 0 && producing && issued < ktiles) issue(issued++);
      const int s = kt % C::STAGES;
      load_frags(s, 8, af[1], bf[1]);
      multiply(af[0], bf[0]);
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[s]);  // the stage has been read
      if (kt + 1 < ktiles) {
        const int s1 = (kt + 1) % C::STAGES;
        ok = mbar_wait(&full[s1], ((kt + 1) / C::STAGES) & 1u, status);
        if (ok) load_frags(s1, 0, af[0], bf[0]);
      }
      multiply(af[1], bf[1]);
    }
  } else {
    for (int kt = 0; kt < ktiles; ++kt) {
      if (threadIdx.x == 0 && producing && issued < ktiles) issue(issued++);
      const int s = kt % C::STAGES;
      if (!mbar_wait(&full[s], (kt / C::STAGES) & 1u, status)) {
        ok = false;
        break;
      }
      const uint8_t* sa = smem + s * C::STAGE_BYTES;
      const uint8_t* sb = sa + C::A_BYTES;
#pragma unroll
      for (int kk = 0; kk < C::BK; kk += 8) {
        double af[C::MI][4], bf[C::NJ][2];
#pragma unroll
        for (int i = 0; i < C::MI; ++i) {
          const uint32_t r0 = arow(i, g), r1 = arow(i, g + 8);
          af[i][0] = *reinterpret_cast<const double*>(sa + tile_off<!C::TA>(r0, kk + t));
          af[i][1] = *reinterpret_cast<const double*>(sa + tile_off<!C::TA>(r1, kk + t));
          af[i][2] = *reinterpret_cast<const double*>(sa + tile_off<!C::TA>(r0, kk + t + 4));
          af[i][3] = *reinterpret_cast<const double*>(sa + tile_off<!C::TA>(r1, kk + t + 4));
        }
#pragma unroll
        for (int j = 0; j < C::NJ; ++j) {
          const uint32_t q = bcol(j, g);
          bf[j][0] = *reinterpret_cast<const double*>(sb + tile_off<C::TB>(q, kk + t));
          bf[j][1] = *reinterpret_cast<const double*>(sb + tile_off<C::TB>(q, kk + t + 4));
        }
#pragma unroll
        for (int i = 0; i < C::MI; ++i)
#pragma unroll
          for (int j = 0; j < C::NJ; ++j)
            asm volatile(
                "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                "{%0,%1,%2,%3};"
                : "+d"(acc[i][j][0]), "+d"(acc[i][j][1]), "+d"(acc[i][j][2]), "+d"(acc[i][j][3])
                : "d"(af[i][0]), "d"(af[i][1]), "d"(af[i][2]), "d"(af[i][3]), "d"(bf[j][0]), "d"(bf[j][1]));
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[s]);
    }
  }
  if (!ok) {
    // leave no copy in flight behind: wait (bounded) for every issued stage's bytes
    if (threadIdx.x == 0)
      for (int kt = (issued > C::STAGES ? issued - C::STAGES : 0); kt < issued; ++kt)
        mbar_wait(&full[kt % C::STAGES], (kt / C::STAGES) & 1u, status);
    return;
  }

  // ---------------- epilogue: C = alpha*acc + beta*C, an m16 row of tiles at a time: all its
  // items of C are in flight before the first is used
#pragma unroll
  for (int i = 0; i < C::MI; ++i) {
    double old[C::NJ][4];
    if (beta != 0.0) {
#pragma unroll
      for (int j = 0; j < C::NJ; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int row = m0 + arow(i, g + 8 * (e >> 1)), col = n0 + bcol(j, 2 * t + (e & 1));
          old[j][e] = row < m && col < n ? c[(int64_t)row * ldc + col] : 0.0;
        }
    }
#pragma unroll
    for (int j = 0; j < C::NJ; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = m0 + arow(i, g + 8 * (e >> 1)), col = n0 + bcol(j, 2 * t + (e & 1));
        const double v = alpha * acc[i][j][e];
        if (row < m && col < n) c[(int64_t)row * ldc + col] = beta == 0.0 ? v : fma(beta, old[j][e], v);
      }
  }
}

// ------------------------------------------------------------------ the LU's trailing update
// C -= A B with A m x k and B k x n row-major and k small (128): a tile's share of C takes nearly a
// third as long to cross HBM as its products take, so C comes by TMA like the operands, through the
// tile's products, into a buffer of its own (128 KB; three operand stages beside it). Reading C from
// global memory at the end, as dgemm_kernel does, ran a 7552 x 7552 rank-128 update at 15.7 TFLOP/s;
// two CTAs per SM with C read at the start, 23.8; this, 27. The arithmetic is dgemm_kernel's: the
// products of a tile are summed by themselves and then subtracted from C (starting the sums from C
// rounds at C's magnitude once per k, and nearly doubled the error of a solve at n = 8192).
//
// Persistent: CTAs take tiles from a counter, thread 0 fetching two tiles ahead; it
// writes a tile into `ring` before it arms the first stage of the tile before it, which every warp
// waits for, so there is no CTA barrier per tile.
//
// A CTA that starts on an SM where the factorization's latest leaf has run (marks) leaves it to the
// next leaf. While short kernels before it still hold the other SMs, the CTAs yet to start all try
// those free ones, so the grid is three times the SMs, and all but (SMs - `most`) of its CTAs may
// leave: the tiles always have that many takers. With one CTA per SM and `most` leaving, the ones
// turned away came back and kept the marked SMs (n = 8192: 28 ms a factorization against 22).
using UpdateCfg = DgemmCfg<128, 128, 64, 32, 3, false, false>;
constexpr int kUpdateC = UpdateCfg::BM * UpdateCfg::BN * 8;
constexpr size_t kUpdateSmem = UpdateCfg::STAGES * UpdateCfg::STAGE_BYTES + kUpdateC + 1024 + (2 * UpdateCfg::STAGES + 2) * 8;

__global__ void __launch_bounds__(UpdateCfg::THREADS, 1)
    dgemm_update_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                        const __grid_constant__ CUtensorMap tma_c, double* __restrict__ c, int64_t ldc, int m, int n,
                        int k, const LeafMarks* marks, int may_leave, int* counters, unsigned* status) {
  using C = UpdateCfg;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* cbuf = smem + C::STAGES * C::STAGE_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(cbuf + kUpdateC);
  uint64_t* empty = full + C::STAGES;
  uint64_t* cfull = empty + C::STAGES;
  uint64_t* cempty = cfull + 1;
  __shared__ int ring[4];  // this CTA's tiles, by their order
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ktiles = (k + C::BK - 1) / C::BK;
  const int tiles_n = (n + C::BN - 1) / C::BN, tiles = tiles_n * ((m + C::BM - 1) / C::BM);
  griddep_launch_dependents();
  griddep_wait();  // the kernel before this one in the stream has completed
  if (threadIdx.x == 0) {
    unsigned sm;
    asm("mov.u32 %0, %%smid;" : "=r"(sm));
    const volatile LeafMarks* mk = marks;
    const bool leave = sm < kSmMarks && mk->latest != 0 && mk->sm[sm] == mk->latest && atomicAdd(&counters[1], 1) < may_leave;
    ring[0] = leave ? INT_MAX : atomicAdd(&counters[0], 1);
    ring[1] = leave ? INT_MAX : atomicAdd(&counters[0], 1);
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], C::COMPUTE_WARPS);
    }
    mbar_init(cfull, 1);
    mbar_init(cempty, C::COMPUTE_WARPS);
    fence_barrier_init();
    tma_prefetch_desc(&tma_a);
    tma_prefetch_desc(&tma_b);
    tma_prefetch_desc(&tma_c);
  }
  __syncthreads();
  // step st = (tile in this CTA's order) * ktiles + k-tile goes to stage st % STAGES
  bool producing = true;
  auto issue = [&](int st, int tile) {
    const int s = st % C::STAGES;
    if (st >= C::STAGES && !mbar_wait(&empty[s], ((st - C::STAGES) / C::STAGES) & 1u, status)) {
      producing = false;
      return;
    }
    uint8_t* sa = smem + s * C::STAGE_BYTES;
    uint8_t* sb = sa + C::A_BYTES;
    mbar_arrive_expect_tx(&full[s], C::STAGE_BYTES);
    const int k0 = st % ktiles * C::BK, m0 = tile / tiles_n * C::BM, n0 = tile % tiles_n * C::BN;
    tma_load_2d(sa, &tma_a, &full[s], k0, m0);
#pragma unroll
    for (int b = 0; b < C::BN / 16; ++b) tma_load_2d(sb + b * 2048, &tma_b, &full[s], n0 + 16 * b, k0);
  };
  int c_issued = 0;  // tiles whose C has been asked for
  auto issue_c = [&](int tile) {
    if (c_issued > 0 && !mbar_wait(cempty, (c_issued - 1) & 1u, status)) {
      producing = false;
      return;
    }
    mbar_arrive_expect_tx(cfull, kUpdateC);
    const int m0 = tile / tiles_n * C::BM, n0 = tile % tiles_n * C::BN;
#pragma unroll
    for (int b = 0; b < C::BN / 16; ++b) tma_load_2d(cbuf + b * C::BM * 128, &tma_c, cfull, n0 + 16 * b, m0);
    ++c_issued;
  };
  const int wm0 = (warp / C::WARPS_N) * C::WM, wn0 = (warp % C::WARPS_N) * C::WN;
  const uint32_t g = lane >> 2, t = lane & 3;
  auto arow = [&](int i, uint32_t r) -> uint32_t { return wm0 + 16 * i + 2 * (r & 7u) + (r >> 3); };
  auto bcol = [&](int j, uint32_t q) -> uint32_t { return wn0 + 16 * (j >> 1) + rho(q, j & 1); };

  int tile = ring[0], issued = 0, step = 0;
  bool ok = true;
  for (int seq = 0; tile < tiles; ++seq) {
    int next = ring[(seq + 1) & 3], after = INT_MAX;  // thread 0's own; the others read next below
    if (threadIdx.x == 0) {
      after = atomicAdd(&counters[0], 1);
      for (; issued < step + C::STAGES - 1 && issued < step + ktiles && producing; ++issued) issue(issued, tile);
      if (producing) issue_c(tile);  // once every warp has read the tile before's
    }
    double acc[C::MI][C::NJ][4];
#pragma unroll
    for (int i = 0; i < C::MI; ++i)
#pragma unroll
      for (int j = 0; j < C::NJ; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0;
    const int end = step + ktiles;
    for (; step < end; ++step) {
      if (threadIdx.x == 0 && producing) {
        if (issued < end) {
          issue(issued, tile), ++issued;
        } else if (next < tiles && issued < end + ktiles) {
          if (issued == end) ring[(seq + 2) & 3] = after;
          issue(issued, next), ++issued;
        }
      }
      const int s = step % C::STAGES;
      if (!mbar_wait(&full[s], (step / C::STAGES) & 1u, status)) {
        ok = false;
        break;
      }
      const uint8_t* sa = smem + s * C::STAGE_BYTES;
      const uint8_t* sb = sa + C::A_BYTES;
#pragma unroll
      for (int kk = 0; kk < C::BK; kk += 8) {
        double af[C::MI][4], bf[C::NJ][2];
#pragma unroll
        for (int i = 0; i < C::MI; ++i) {
          const uint32_t r0 = arow(i, g), r1 = arow(i, g + 8);
          af[i][0] = *reinterpret_cast<const double*>(sa + tile_off<true>(r0, kk + t));
          af[i][1] = *reinterpret_cast<const double*>(sa + tile_off<true>(r1, kk + t));
          af[i][2] = *reinterpret_cast<const double*>(sa + tile_off<true>(r0, kk + t + 4));
          af[i][3] = *reinterpret_cast<const double*>(sa + tile_off<true>(r1, kk + t + 4));
        }
#pragma unroll
        for (int j = 0; j < C::NJ; ++j) {
          const uint32_t q = bcol(j, g);
          bf[j][0] = *reinterpret_cast<const double*>(sb + tile_off<false>(q, kk + t));
          bf[j][1] = *reinterpret_cast<const double*>(sb + tile_off<false>(q, kk + t + 4));
        }
#pragma unroll
        for (int i = 0; i < C::MI; ++i)
#pragma unroll
          for (int j = 0; j < C::NJ; ++j)
            asm volatile(
                "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                "{%0,%1,%2,%3};"
                : "+d"(acc[i][j][0]), "+d"(acc[i][j][1]), "+d"(acc[i][j][2]), "+d"(acc[i][j][3])
                : "d"(af[i][0]), "d"(af[i][1]), "d"(af[i][2]), "d"(af[i][3]), "d"(bf[j][0]), "d"(bf[j][1]));
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[s]);
    }
    if (!ok) break;
    next = ring[(seq + 1) & 3];
    if (!mbar_wait(cfull, seq & 1u, status)) {
      ok = false;
      break;
    }
    // rows g and g + 8 of each m16 tile, two neighbouring columns each
    const int m0 = tile / tiles_n * C::BM, n0 = tile % tiles_n * C::BN;
#pragma unroll
    for (int i = 0; i < C::MI; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = arow(i, g + 8 * h), row = m0 + r;
        double* p = c + (int64_t)row * ldc + n0;
#pragma unroll
        for (int j = 0; j < C::NJ; ++j) {
          const int col = bcol(j, 2 * t);
          double2 v = *reinterpret_cast<const double2*>(cbuf + (col >> 4) * (C::BM * 128) + swz128_f64(r, col & 15));
          v.x -= acc[i][j][2 * h];
          v.y -= acc[i][j][2 * h + 1];
          if (row < m) {
            if (n0 + col + 1 < n) *reinterpret_cast<double2*>(p + col) = v;
            else if (n0 + col < n) p[col] = v.x;
          }
        }
      }
    __syncwarp();
    if (lane == 0) mbar_arrive(cempty);
    tile = next;
  }
  // leave no copy in flight behind: wait (bounded) for every issued stage's bytes
  if (!ok && threadIdx.x == 0) {
    for (int st = (issued > C::STAGES ? issued - C::STAGES : 0); st < issued; ++st)
      mbar_wait(&full[st % C::STAGES], (st / C::STAGES) & 1u, status);
    if (c_issued > 0) mbar_wait(cfull, (c_issued - 1) & 1u, status);
  }
}

int dgemm_update_f64(int m, int n, int k, const double* a, int64_t lda, const double* b, int64_t ldb, double* c,
                     int64_t ldc, const LeafMarks* marks, int most, int* counters, unsigned* status,
                     cudaStream_t stream) {
  CUtensorMap ta, tb, tc;
  RM_TRY(make_tensor_map_2d(&ta, a, 8, k, m, lda * 8, 16, UpdateCfg::BM, true));
  RM_TRY(make_tensor_map_2d(&tb, b, 8, n, k, ldb * 8, 16, 16, true));
  RM_TRY(make_tensor_map_2d(&tc, c, 8, n, m, ldc * 8, 16, UpdateCfg::BM, true));  // checks C's alignment too
  RM_TRY(smem_attribute(dgemm_update_kernel, kUpdateSmem));
  const int sms = device_sm_count();
  RM_CUDA_TRY(launch_dependent(dgemm_update_kernel, dim3(3 * sms), dim3(UpdateCfg::THREADS), kUpdateSmem,
                               stream, ta, tb, tc, c, ldc, m, n, k, marks, 2 * sms + most, counters, status));
  note_launch();
  return RM_OK;
}

// ------------------------------------------------------------------ host side

template <class C>
static int launch_cfg(const double* a, int64_t lda, const double* b, int64_t ldb, double* c, int64_t ldc, int m,
                      int n, int k, double alpha, double beta, unsigned* status, cudaStream_t stream, bool lower = false) {
  CUtensorMap ta, tb;
  // A: op(A) is m x k. Not transposed: stored m rows of k; transposed: k rows of m.
  if (!C::TA) {
    RM_TRY(make_tensor_map_2d(&ta, a, 8, k, m, lda * 8, 16, C::BM, true));
  } else {
    RM_TRY(make_tensor_map_2d(&ta, a, 8, m, k, lda * 8, 16, 16, true));
  }
  if (!C::TB) {
    RM_TRY(make_tensor_map_2d(&tb, b, 8, n, k, ldb * 8, 16, 16, true));
  } else {
    RM_TRY(make_tensor_map_2d(&tb, b, 8, k, n, ldb * 8, 16, C::BN, true));
  }
  RM_TRY(smem_attribute(dgemm_kernel<C>, C::SMEM));
  dim3 grid((n + C::BN - 1) / C::BN, (m + C::BM - 1) / C::BM);
  RM_CUDA_TRY(launch_dependent(dgemm_kernel<C>, grid, dim3(C::THREADS), C::SMEM, stream, ta, tb, c, ldc, m, n, k, alpha,
                               beta, lower, status));
  note_launch();
  return RM_OK;
}

// The tile by the number of tiles: a launch lasts as long as its fullest SM does, so the tile is the
// smallest whose tiles come to at most two or three per SM, and the stages are as many as leave room
// for just that many CTAs (deeper stages hide more of the operands' latency, and the CTAs spread
// evenly). Measured (us, one 64 x 64 tile of four warps before): 512^3 37 -> 18 with 32 x 32 tiles
// at two per SM, 12 stages (27 with 6 stages and room for four); 640^3 72 -> 26 at three per SM;
// 768^3 88 -> 37 with 64 x 32; 1024^3 128 -> 79 and 2135 x 3926 x 462 463 -> 294 with 64 x 64 at
// two per SM (6 stages) in a stream of products, alone 90 and 320 either way; 1200^3 161 -> 144 at
// three per SM (4 stages). From 148 tiles of 128 x 128 on, those.
// whole_rows: the tile must span all n <= 128 columns (C may then be A: a CTA has read its rows'
// items before it stores them).
template <bool TA, bool TB>
static int launch_t(const double* a, int64_t lda, const double* b, int64_t ldb, double* c, int64_t ldc, int m, int n,
                    int k, double alpha, double beta, unsigned* status, cudaStream_t stream, bool whole_rows,
                    bool lower = false) {
  const int64_t sms = device_sm_count();
  auto tiles = [&](int bm, int bn) {
    const int64_t t = (int64_t)((m + bm - 1) / bm) * ((n + bn - 1) / bn);
    return lower ? (t + 1) / 2 : t;
  };
  using Mid = DgemmCfg<64, 64, 32, 32, 6, TA, TB>;
  using Big = DgemmCfg<128, 128, 64, 32, 4, TA, TB>;
  if (whole_rows) {
    if (n > Big::BN) return RM_BAD_ARG;
    if (n <= Mid::BN) return launch_cfg<Mid>(a, lda, b, ldb, c, ldc, m, n, k, alpha, beta, status, stream, lower);
    return launch_cfg<Big>(a, lda, b, ldb, c, ldc, m, n, k, alpha, beta, status, stream, lower);
  }
  if (tiles(128, 128) >= sms)
    return launch_cfg<Big>(a, lda, b, ldb, c, ldc, m, n, k, alpha, beta, status, stream, lower);
  if (tiles(32, 32) <= 2 * sms)
    return launch_cfg<DgemmCfg<32, 32, 16, 16, 12, TA, TB>>(a, lda, b, ldb, c, ldc, m, n, k, alpha, beta, status, stream,
                                                            lower);
  if (tiles(32, 32) <= 3 * sms)
    return launch_cfg<DgemmCfg<32, 32, 16, 16, 8, TA, TB>>(a, lda, b, ldb, c, ldc, m, n, k, alpha, beta, status, stream,
                                                           lower);
  if (tiles(64, 32) <= 2 * sms)
    return launch_cfg<DgemmCfg<64, 32, 16, 16, 8, TA, TB>>(a, lda, b, ldb, c, ldc, m, n, k, alpha, beta, status, stream,
                                                           lower);
  const int64_t t64 = tiles(64, 64);
  if (t64 > 2 * sms && t64 <= 3 * sms)
    return launch_cfg<DgemmCfg<64, 64, 32, 32, 4, TA, TB>>(a, lda, b, ldb, c, ldc, m, n, k, alpha, beta, status, stream,
                                                           lower);
  return launch_cfg<Mid>(a, lda, b, ldb, c, ldc, m, n, k, alpha, beta, status, stream, lower);
}

int dgemm_device(bool ta, bool tb, int64_t m, int64_t n, int64_t k, double alpha, const double* a, int64_t lda,
                 const double* b, int64_t ldb, double beta, double* c, int64_t ldc, unsigned* status,
                 cudaStream_t stream, bool wide) {
  if (m == 0 || n == 0) return RM_OK;
  if (k == 0 || alpha == 0.0) return scale_device(c, ldc, m, n, beta, stream);
  if (m > INT32_MAX || n > INT32_MAX || k > INT32_MAX) return RM_BAD_ARG;
  if (ta) {
    if (tb) return launch_t<true, true>(a, lda, b, ldb, c, ldc, (int)m, (int)n, (int)k, alpha, beta, status, stream, wide);
    return launch_t<true, false>(a, lda, b, ldb, c, ldc, (int)m, (int)n, (int)k, alpha, beta, status, stream, wide);
  }
  if (tb) return launch_t<false, true>(a, lda, b, ldb, c, ldc, (int)m, (int)n, (int)k, alpha, beta, status, stream, wide);
  return launch_t<false, false>(a, lda, b, ldb, c, ldc, (int)m, (int)n, (int)k, alpha, beta, status, stream, wide);
}

int dgemm_lower_device(int64_t n, int64_t k, double alpha, const double* a, int64_t lda, const double* b, int64_t ldb,
                       double beta, double* c, int64_t ldc, unsigned* status, cudaStream_t stream) {
  if (n == 0) return RM_OK;
  if (n > INT32_MAX || k < 1 || k > INT32_MAX) return RM_BAD_ARG;
  return launch_t<false, true>(a, lda, b, ldb, c, ldc, (int)n, (int)n, (int)k, alpha, beta, status, stream, false, true);
}

// C = beta*C (beta == 0 writes zeros), the reference's `scale` (linalg.rs:1000-1008).
__global__ void scale_kernel(double* c, int64_t ldc, int64_t m, int64_t n, double beta) {
  const int64_t total = m * n;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = idx / n, j = idx % n;
    double* p = c + i * ldc + j;
    *p = beta == 0.0 ? 0.0 : beta * *p;
  }
}

int scale_device(double* c, int64_t ldc, int64_t m, int64_t n, double beta, cudaStream_t stream) {
  if (beta == 1.0 || m == 0 || n == 0) return RM_OK;
  const int64_t total = m * n;
  const int blocks = (int)std::min<int64_t>((total + 255) / 256, 4 * device_sm_count());
  scale_kernel<<<blocks, 256, 0, stream>>>(c, ldc, m, n, beta);
  RM_LAUNCHED();
  return RM_OK;
}

}  // namespace rm
