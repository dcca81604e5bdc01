// FP64-accurate GEMM from int8 tensor-core products (the Ozaki split scheme).
//
// C = A B for float64 A (m x k) and B (k x n), row-major. Each row i of A is scaled by a
// power of two 2^-ea[i] into (-1, 1) and cut into `s` signed 7-bit slices:
//   a_ij = 2^ea[i] sum_{p<s} t_p 2^-7(p+1) + (remainder below 2^(ea[i]-7s)),  t_p in [-127, 127],
// each slice exact in int8 (the scaling and the digit extraction are exact in float64);
// likewise each column j of B with 2^eb[j]. Then
//   C_ij ~= 2^(ea[i]+eb[j]) sum_{d<s} 2^-7(d+2) sum_{p+q=d} (A_p B_q)_ij,
// dropping the products of order p + q >= s (below 2^-7s relative, as the truncation). The
// inner sums are int8 x int8 products accumulated in int32 by tcgen05.mma kind::i8 - exact
// while (d+1) k 127^2 < 2^31, so k is cut into chunks that keep it so - and two orders
// d, d - 1 are one persistent launch whose epilogue adds 2^(ea+eb-7(d+2)) acc of each to C in float64,
// the smallest first. With s = 8 the truncation (2^-56 relative to 2^(ea+eb)) is below
// float64 rounding.
//
// The slices live in one scratch buffer: A's as s stacked (mp x kp) int8 planes, B's
// transposed (K-major) as s stacked (np x kp) planes, all of whole tiles. A's columns past k are zeros; the rest
// of the padding is not written, as it meets only those or what is not stored.
// rustymath's matmul is float64 throughout (core/src/linalg.rs:1119-1132); this is the
// split-precision product measured against the native float64 GEMM (rm_dgemm).
#include <algorithm>
#include <cfloat>
#include <climits>

#include "rm_internal.h"
#include "rm_tcgen05.cuh"

namespace rm {
namespace oz {

constexpr int BM = 128, BK = 128;            // BK int8 = 128 bytes: one swizzle row
constexpr int A_BYTES = BM * BK;             // 16 KB
constexpr int EPI_WARPS = 8;                 // two per TMEM lane quarter, half the columns each
constexpr int THREADS = 64 + 32 * EPI_WARPS; // TMA warp, MMA warp, epilogue warps
constexpr int STG = 33;                      // epilogue staging: 32 x 33 int32 per warp
constexpr int STG_BYTES = EPI_WARPS * 32 * STG * 4;
constexpr int kPadN = 128;                   // B's planes are padded to whole 128-row tiles
template <int BN>
struct Tile {
  static constexpr int kStages = BN == 256 ? 4 : 6;
  static constexpr int kStageBytes = A_BYTES + BN * BK;
  static constexpr uint32_t kTmemCols = 2 * BN;  // two accumulators: orders d and d - 1
  static constexpr size_t kSmem = 1024 + (size_t)kStages * kStageBytes + STG_BYTES + 512;
};
constexpr int MAX_SLICES = 8;

// Instruction descriptor, kind::i8: D s32, A and B signed int8, both K-major.
__host__ __device__ constexpr uint32_t idesc_i8(int m, int n) {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void mma_i8(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(da), "l"(db), "r"(idesc), "r"(acc));
}

// frexp-style exponent of the largest |x| of a row: max|x| < 2^e (e = 0 for an all-zero row)
__device__ __forceinline__ int exponent_of(double v) {
  if (v == 0.0 || !(v == v)) return INT_MIN;
  int e;
  frexp(v, &e);
  return e;
}

// The largest finite magnitude first, then its exponent once: frexp an element costs more than
// the pass over memory. A NaN never compares greater; an infinity (its exponent is not above that
// of every finite entry) sends the caller through the entries one by one.
__device__ __forceinline__ void max_magnitude(double& top, double v) {
  v = fabs(v);
  if (v > top) top = v;
}

// eb[j] (pre-set to INT_MIN) for each column of the k x n row-major b: 32 x 32 tiles, atomics
__global__ void col_exponent_kernel(const double* __restrict__ b, int64_t ldb, int k, int n, int* __restrict__ eb) {
  __shared__ int cm[32];
  const int j = blockIdx.x * 32 + threadIdx.x;
  if (threadIdx.y == 0) cm[threadIdx.x] = INT_MIN;
  __syncthreads();
  int e = INT_MIN;
  if (j < n) {
    const int r0 = blockIdx.y * 32 + threadIdx.y, step = gridDim.y * 32;
    double top = 0.0;
#pragma unroll 4
    for (int r = r0; r < k; r += step) max_magnitude(top, b[(int64_t)r * ldb + j]);
    e = exponent_of(top);
    if (isinf(top))
      for (int r = r0; r < k; r += step) e = max(e, exponent_of(fabs(b[(int64_t)r * ldb + j])));
  }
  atomicMax(&cm[threadIdx.x], e);
  __syncthreads();
  if (threadIdx.y == 0 && j < n && cm[threadIdx.x] != INT_MIN) atomicMax(&eb[j], cm[threadIdx.x]);
}

__global__ void fix_exponent_kernel(int* e, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && e[i] == INT_MIN) e[i] = 0;
}

// 2^e for -1022 <= e <= 1023
__device__ __forceinline__ double pow2(int e) { return __hiloint2double((e + 1023) << 20, 0); }

// Four bytes of 7 bits from 28 bits, the top ones in the high byte, each negated if neg
__device__ __forceinline__ uint32_t spread7(uint32_t v, bool neg) {
  v = (v & 0x3fffu) | ((v << 2) & 0x3fff0000u);
  v = (v & 0x007f007fu) | ((v << 1) & 0x7f007f00u);
  return neg ? (0x80808080u - v) ^ 0x80808080u : v;
}

// The digits of a value that is not below 1 in magnitude (a row or column with an infinity, a
// NaN), one by one
__device__ __noinline__ uint2 digits_rare(double t) {
  uint32_t w[2] = {0u, 0u};
  for (int p = 0; p < MAX_SLICES; ++p) {
    t *= 128.0;
    const double d = trunc(t);
    t -= d;
    w[p >> 2] |= (uint32_t)(uint8_t)(int8_t)d << (8 * (3 - (p & 3)));
  }
  return make_uint2(w[0], w[1]);
}

// Eight signed base-128 digits of 2^-e x, truncated toward zero: x.x holds the first four, the
// first in the high byte. They are the digits of one 56-bit fixed-point number, which costs one
// conversion where a digit at a time costs two roundings each.
__device__ __forceinline__ uint2 digits(double x, int e) {
  const double r = (unsigned)(e + 1022) <= 2044u ? x * pow2(-e) : ldexp(x, -e);
  if (!(fabs(r) < 1.0)) return digits_rare(r);
  const uint64_t v = (uint64_t)__double2ll_rz(fabs(r) * 0x1p56);
  return make_uint2(spread7((uint32_t)(v >> 28), r < 0.0), spread7((uint32_t)v & 0xfffffffu, r < 0.0));
}

// Words of planes 0..3 from the digit words of four elements: byte 3 - p of each, the first
// element's lowest
__device__ __forceinline__ void transpose4(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3, uint32_t* out) {
  const uint32_t a = __byte_perm(w0, w1, 0x6273), b = __byte_perm(w2, w3, 0x6273);  // planes 1 | 0
  const uint32_t c = __byte_perm(w0, w1, 0x4051), d = __byte_perm(w2, w3, 0x4051);  // planes 3 | 2
  out[0] = __byte_perm(a, b, 0x5410);
  out[1] = __byte_perm(a, b, 0x7632);
  out[2] = __byte_perm(c, d, 0x5410);
  out[3] = __byte_perm(c, d, 0x7632);
}
__device__ __forceinline__ void plane_words(const double (&x)[4], int e, uint32_t (&out)[MAX_SLICES]) {
  uint2 w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) w[i] = digits(x[i], e);
  transpose4(w[0].x, w[1].x, w[2].x, w[3].x, out);
  transpose4(w[0].y, w[1].y, w[2].y, w[3].y, out + 4);
}

// ea[i] and the s slices of row i of a into planes [p][i][kk] (row stride kp, plane stride
// mp * kp), zero from k to kp: a block per row, so that the second pass over the row finds it
// in L2, and four columns a lane, so that a warp's stores are 128 bytes in each plane. Rows
// from m to mp stay unwritten: they only meet rows of C that are not stored. HBM-bound but for the
// second pass: 8192 x 8192, 198 us (157 for the bytes; with a digit at a time 421, and 410 : 244 for
// the columns' kernel).
__global__ void __launch_bounds__(256)
    split_rows_kernel(const double* __restrict__ a, int64_t lda, int k, int* __restrict__ ea, int s,
                      int8_t* __restrict__ out, int64_t kp, int64_t plane) {
  __shared__ int part[8];
  const int64_t row = blockIdx.x;
  const double* ar = a + row * lda;
  double top = 0.0;
#pragma unroll 8
  for (int j = threadIdx.x; j < k; j += 256) max_magnitude(top, ar[j]);
  int e = exponent_of(top);
  if (isinf(top))
    for (int j = threadIdx.x; j < k; j += 256) e = max(e, exponent_of(fabs(ar[j])));
  e = __reduce_max_sync(0xffffffffu, e);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = e;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; ++w) e = max(e, part[w]);
  if (e == INT_MIN) e = 0;
  if (threadIdx.x == 0) ea[row] = e;
  for (int64_t j = 4 * threadIdx.x; j < kp; j += 1024) {
    double x[4];
    uint32_t w[MAX_SLICES];
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = j + i < k ? ar[j + i] : 0.0;
    plane_words(x, e, w);
#pragma unroll
    for (int p = 0; p < MAX_SLICES; ++p)
      if (p < s) *reinterpret_cast<uint32_t*>(out + p * plane + row * kp + j) = w[p];
  }
}

// The s slices of column j of b (scaled by 2^-eb[j]), transposed: planes [q][j][kk] (row
// stride kp). A block takes 128 rows and 32 columns through shared memory: reads along b's
// rows, four of them a thread, and 128-byte stores along k. What lies past k meets A's zeros,
// so nothing else of the planes is written.
__global__ void __launch_bounds__(256)
    split_cols_kernel(const double* __restrict__ b, int64_t ldb, int k, int n, const int* __restrict__ eb, int s,
                      int8_t* __restrict__ out, int64_t kp, int64_t plane) {
  __shared__ uint32_t t8[MAX_SLICES][32][33];
  const int r0 = blockIdx.y * 128, j0 = blockIdx.x * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int j = j0 + tx;
  const int e = j < n ? eb[j] : 0;
#pragma unroll
  for (int g = ty; g < 32; g += 8) {
    double x[4];
    uint32_t w[MAX_SLICES];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = r0 + 4 * g + i;
      x[i] = (r < k && j < n) ? b[(int64_t)r * ldb + j] : 0.0;
    }
    plane_words(x, e, w);
#pragma unroll
    for (int q = 0; q < MAX_SLICES; ++q)
      if (q < s) t8[q][tx][g] = w[q];
  }
  __syncthreads();
  for (int i = ty; i < 32 * s; i += 8) {
    const int q = i >> 5, jj = i & 31;
    if (j0 + jj < n)
      *reinterpret_cast<uint32_t*>(out + q * plane + (int64_t)(j0 + jj) * kp + r0 + 4 * tx) = t8[q][jj][tx];
  }
}

// Output tile t of a persistent walk -> (tile row, tile column), in bands of kBand tile rows:
// down a band's rows first, then across its columns, so that the ~148 tiles in flight at once
// read about kBand row panels of A's slices and 148 / kBand column panels of B's (some tens of
// MB, resident in L2) instead of one row panel and 148 column panels.
constexpr int kBand = 8;
__device__ __forceinline__ void tile_coords(int t, int ntm, int ntn, int& tm, int& tn) {
  const int per_band = kBand * ntn;
  const int band = t / per_band, in = t - band * per_band;
  const int rows = min(kBand, ntm - band * kBand);
  tm = band * kBand + in % rows;
  tn = in / rows;
}

// 2^e v for an integer |v| < 2^31 and any e: the first factor keeps the product exact, the
// second rounds (or underflows, or overflows) once
__device__ __forceinline__ double scale_any(double v, int e) {
  const int e1 = min(max(e, -1000), 1000);
  return v * pow2(e1) * pow2(min(max(e - e1, -1022), 1023));
}

// Orders d and (TWO) d - 1 of the split product over the k-range [k0, k0 + kc):
//   C (+)= 2^(ea[i] + eb[j] - 7(d+2)) sum_{p+q=d} A_p B_q^T, then the same of d - 1.
// Persistent: warp 0 loads slice tiles by TMA (rows p*mp + m0 of A's planes, q*np + n0 of
// B's), warp 1 issues kind::i8 MMAs, warps 2..9 drain the accumulators (int32 -> float64,
// scaled, added to C in coalesced rows through shared memory).
//
// An SM reads about 64 bytes a cycle from L2 and 128 from shared memory, and an int8 tile
// product 128 x N x 128 takes 2 N cycles. One order at a time on 128 x 128 tiles loads 32 KB
// for 256 cycles: twice what L2 delivers (the tensor pipe stood at 48%). Here a stage holds
// A_p and B_{d-p}, and B_{d-p} also meets the A_{p-1} of the stage before it for the order
// d - 1, so a loaded tile is used twice; with N = 256 that is 48 KB for 1024 cycles. Both
// accumulators take all 512 TMEM columns, so the epilogue is not overlapped with the tile's
// successor; it is under 3% of the 2d + 1 products, and C is read and written half as often.
// 8192^3, 8 slices, the whole call: 22.7 ms before, 15.2 after, 14.9 with the split kernels above; the
// tensor pipe then runs at 3.7 POPS (12.5 ms alone, 4.9 for the first launch) and the power cap binds.
template <int BN, bool TWO>
__global__ void __launch_bounds__(THREADS, 1)
    ozaki_order_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b,
                       double* __restrict__ c, int64_t ldc, int m, int n, int mp, int np, int k0, int kc, int d,
                       const int* __restrict__ ea, const int* __restrict__ eb, int first, unsigned* status) {
  using T = Tile<BN>;
  constexpr int STAGES = T::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  int* stg_all = reinterpret_cast<int*>(smem + STAGES * T::kStageBytes);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * T::kStageBytes + STG_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* tfull = empty + STAGES;
  uint64_t* tempty = tfull + 1;
  uint64_t* mma_done = tempty + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mma_done + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ntn = (n + BN - 1) / BN, ntm = (m + BM - 1) / BM;
  const int tiles = ntm * ntn;
  const int ktiles = (kc + BK - 1) / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tfull, 1);
    mbar_init(tempty, EPI_WARPS);
    mbar_init(mma_done, 1);
    fence_barrier_init();
  }
  if (warp == 1) {
    tc::tmem_alloc(tmem_slot, T::kTmemCols);
    tc::fence_before();
  }
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&tm_a);
      tma_prefetch_desc(&tm_b);
      int it = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        int tmi, tni;
        tile_coords(tile, ntm, ntn, tmi, tni);
        const int m0 = tmi * BM, n0 = tni * BN;
        for (int kt = 0; kt < ktiles && ok; ++kt)
          for (int p = 0; p <= d; ++p, ++it) {
            const int s = it % STAGES;
            if (!mbar_wait(&empty[s], ((it / STAGES) & 1u) ^ 1u, status)) {
              ok = false;
              break;
            }
            uint8_t* st = smem + s * T::kStageBytes;
            mbar_arrive_expect_tx(&full[s], T::kStageBytes);
            tma_load_2d(st, &tm_a, &full[s], k0 + kt * BK, p * mp + m0);
            tma_load_2d(st + A_BYTES, &tm_b, &full[s], k0 + kt * BK, (d - p) * np + n0);
          }
      }
      for (int j = (it > STAGES ? it - STAGES : 0); j < it; ++j) mbar_wait(&full[j % STAGES], (j / STAGES) & 1u, status);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = idesc_i8(BM, BN);
      const uint32_t base = smem_u32(smem);
      int it = 0, lt = 0, prev = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x, ++lt) {
        if (!mbar_wait(tempty, (lt & 1u) ^ 1u, status)) break;
        tc::fence_after();
        for (int kt = 0; kt < ktiles && ok; ++kt)
          for (int p = 0; p <= d; ++p, ++it) {
            const int s = it % STAGES;
            if (!mbar_wait(&full[s], (it / STAGES) & 1u, status)) {
              ok = false;
              break;
            }
            tc::fence_after();
            const uint32_t sa = base + s * T::kStageBytes, sb = sa + A_BYTES;
#pragma unroll
            for (int kk = 0; kk < BK / 32; ++kk)  // K = 32 int8 = 32 bytes per MMA
              mma_i8(tmem, tc::smem_desc(sa + kk * 32), tc::smem_desc(sb + kk * 32), idesc,
                     (kt == 0 && p == 0 && kk == 0) ? 0u : 1u);
            if (TWO && p > 0) {
              const uint32_t sp = base + prev * T::kStageBytes;
#pragma unroll
              for (int kk = 0; kk < BK / 32; ++kk)
                mma_i8(tmem + BN, tc::smem_desc(sp + kk * 32), tc::smem_desc(sb + kk * 32), idesc,
                       (kt == 0 && p == 1 && kk == 0) ? 0u : 1u);
              tc::mma_commit(&empty[prev]);
            }
            if (!TWO || p == d) tc::mma_commit(&empty[s]);
            prev = s;
          }
        if (ok) tc::mma_commit(tfull);
      }
      tc::mma_commit(mma_done);
      mbar_wait(mma_done, 0u, status);
    }
  } else {
    // epilogue: warps 2..9, TMEM lane quarter warp % 4, half of the columns
    const int q = warp & 3, half = (warp - 2) >> 2;
    int* stg = stg_all + (warp - 2) * 32 * STG;
    int lt = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++lt) {
      int tmi, tni;
      tile_coords(tile, ntm, ntn, tmi, tni);
      const int row0 = tmi * BM + q * 32;
      const int er = row0 + lane < m ? ea[row0 + lane] : 0;
      const int ermin = __reduce_min_sync(0xffffffffu, er), ermax = __reduce_max_sync(0xffffffffu, er);
      const uint32_t tq = tmem + ((uint32_t)(q * 32) << 16);
      bool waited = false;
#pragma unroll 1
      for (int cb = half * (BN / 2); cb < (half + 1) * (BN / 2); cb += 32) {
        const int col = tni * BN + cb + lane;
        double cv[32];
#pragma unroll
        for (int rr = 0; rr < 32; ++rr)
          cv[rr] = (!first && row0 + rr < m && col < n) ? c[(int64_t)(row0 + rr) * ldc + col] : 0.0;
        const int ecol = (col < n ? eb[col] : 0) - 7 * (d + 2);
        const bool plain = __all_sync(0xffffffffu, ermin + ecol >= -1022 && ermax + ecol + 7 <= 1023);
        if (!waited) {  // after the first chunk of C has been asked for
          if (!__all_sync(0xffffffffu, mbar_wait(tfull, lt & 1u, status))) goto out;
          tc::fence_after();
          waited = true;
        }
#pragma unroll
        for (int o = 0; o < (TWO ? 2 : 1); ++o) {
          uint32_t v[32];
          tc::tmem_ld32(tq + o * BN + cb, v);
          if (o == (TWO ? 1 : 0) && cb == (half + 1) * (BN / 2) - 32) {
            tc::fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty);
          }
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 32; ++j) stg[lane * STG + j] = (int)v[j];
          __syncwarp();
          if (plain) {
#pragma unroll
            for (int rr = 0; rr < 32; ++rr)
              cv[rr] += (double)stg[rr * STG + lane] * pow2(__shfl_sync(0xffffffffu, er, rr) + ecol + 7 * o);
          } else {
#pragma unroll
            for (int rr = 0; rr < 32; ++rr)
              cv[rr] += scale_any((double)stg[rr * STG + lane], __shfl_sync(0xffffffffu, er, rr) + ecol + 7 * o);
          }
        }
#pragma unroll
        for (int rr = 0; rr < 32; ++rr)
          if (row0 + rr < m && col < n) c[(int64_t)(row0 + rr) * ldc + col] = cv[rr];
      }
    }
  out:;
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after();
    tc::tmem_free(tmem, T::kTmemCols);
  }
}

// Every order of every k chunk, the smallest terms first, two orders to a launch
template <int BN>
int orders(int64_t m, int64_t n, int64_t k, double* c, int64_t ldc, int s, const int8_t* asl, const int8_t* bsl,
           int64_t mp, int64_t np, int64_t kp, int64_t kmax, const int* ea, const int* eb, unsigned* status,
           cudaStream_t stream) {
  constexpr size_t smem = Tile<BN>::kSmem;
  RM_TRY(smem_attribute(ozaki_order_kernel<BN, true>, smem));
  RM_TRY(smem_attribute(ozaki_order_kernel<BN, false>, smem));
  CUtensorMap ta, tb;
  RM_TRY(make_tensor_map_2d(&ta, asl, 1, kp, s * mp, kp, BK, BM, true));
  // a 256-row box may reach into the next plane or past the last one: columns beyond n, not stored
  RM_TRY(make_tensor_map_2d(&tb, bsl, 1, kp, s * np, kp, BK, BN, true));
  const int64_t tiles = (mp / BM) * ((n + BN - 1) / BN);
  const unsigned grid = (unsigned)std::min<int64_t>(tiles, device_sm_count());
  int first = 1;
  for (int64_t k0 = 0; k0 < k; k0 += kmax) {
    const int kc = (int)std::min<int64_t>(kmax, k - k0);
    for (int d = s - 1; d >= 0; d -= 2) {
      auto kernel = d > 0 ? ozaki_order_kernel<BN, true> : ozaki_order_kernel<BN, false>;
      kernel<<<grid, THREADS, smem, stream>>>(ta, tb, c, ldc, (int)m, (int)n, (int)mp, (int)np, (int)k0, kc, d, ea, eb,
                                              first, status);
      RM_LAUNCHED();
      first = 0;
    }
  }
  return RM_OK;
}

}  // namespace oz

size_t ozaki_scratch_bytes(int64_t m, int64_t n, int64_t k, int s) {
  const int64_t mp = (m + oz::BM - 1) / oz::BM * oz::BM, np = (n + oz::kPadN - 1) / oz::kPadN * oz::kPadN;
  const int64_t kp = (k + oz::BK - 1) / oz::BK * oz::BK;
  return (size_t)s * (mp + np) * kp + (size_t)(m + n) * sizeof(int) + 1024;
}

__global__ void fill_int_kernel(int* p, int n, int v) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = v;
}

int dgemm_ozaki(int64_t m, int64_t n, int64_t k, const double* a, int64_t lda, const double* b, int64_t ldb,
                double* c, int64_t ldc, int s, void* scratch, unsigned* status, cudaStream_t stream) {
  if (m == 0 || n == 0) return RM_OK;
  if (s < 1 || s > oz::MAX_SLICES || m > INT_MAX / 2 || n > INT_MAX / 2 || k > INT_MAX / 2) return RM_BAD_ARG;
  if (k == 0) {
    RM_CUDA_TRY(cudaMemset2DAsync(c, ldc * sizeof(double), 0, n * sizeof(double), m, stream));
    return RM_OK;
  }
  const int64_t mp = (m + oz::BM - 1) / oz::BM * oz::BM, np = (n + oz::kPadN - 1) / oz::kPadN * oz::kPadN;
  const int64_t kp = (k + oz::BK - 1) / oz::BK * oz::BK;
  int8_t* asl = reinterpret_cast<int8_t*>(scratch);
  int8_t* bsl = asl + (size_t)s * mp * kp;
  int* ea = reinterpret_cast<int*>(bsl + (size_t)s * np * kp);
  int* eb = ea + m;
  const int ni = (int)n, ki = (int)k;
  // exponents and slices; int8 planes hold no value that could spread, so only A's columns from
  // k to kp are cleared
  oz::split_rows_kernel<<<(unsigned)m, 256, 0, stream>>>(a, lda, ki, ea, s, asl, kp, mp * kp);
  RM_LAUNCHED();
  fill_int_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(eb, ni, INT_MIN);
  RM_LAUNCHED();
  oz::col_exponent_kernel<<<dim3((unsigned)((n + 31) / 32), (unsigned)std::min<int64_t>((k + 31) / 32, 64)),
                            dim3(32, 32), 0, stream>>>(b, ldb, ki, ni, eb);
  RM_LAUNCHED();
  oz::fix_exponent_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(eb, ni);
  RM_LAUNCHED();
  oz::split_cols_kernel<<<dim3((unsigned)((n + 31) / 32), (unsigned)(kp / 128)), 256, 0, stream>>>(
      b, ldb, ki, ni, eb, s, bsl, kp, np * kp);
  RM_LAUNCHED();
  // k chunks short enough that an order's int32 sums cannot overflow: s k 127^2 < 2^31
  const int64_t kmax = std::max<int64_t>(oz::BK, ((int64_t)INT_MAX / ((int64_t)s * 127 * 127)) / oz::BK * oz::BK);
  // 128 x 256 tiles need less traffic per product, 128 x 128 tiles spread a small product over
  // more SMs: by the waves that each takes, a wide tile costing two narrow ones over 1.3 (wide
  // against narrow, us: 1300 x 1300, k = 1024, one wave of either, 221 : 172; 1700 x 1400,
  // k = 1700, one : two, 319 : 402; 2200 x 2200, k = 1000, two : three, 418 : 399; 2500 x 2500,
  // k = 3000, 896 : 926; 3500^3, three : six, 1477 : 2007; 8192^3 14.2 : 19.3 ms)
  const int64_t sms = device_sm_count();
  const int64_t narrow = (mp / oz::BM) * ((n + 127) / 128), wide = (mp / oz::BM) * ((n + 255) / 256);
  const bool use_wide = 20 * ((wide + sms - 1) / sms) <= 13 * ((narrow + sms - 1) / sms);
  return use_wide ? oz::orders<256>(m, n, k, c, ldc, s, asl, bsl, mp, np, kp, kmax, ea, eb, status, stream)
                  : oz::orders<128>(m, n, k, c, ldc, s, asl, bsl, mp, np, kp, kmax, ea, eb, status, stream);
}

}  // namespace rm
