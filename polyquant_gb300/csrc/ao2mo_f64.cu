// FP64 AO->MO transform on the tcgen05 tensor cores.
//
// The two pair-symmetric half transforms of ao2mo.cu: for every slice S_b (the symmetric matrix of one ket pair in
// half 1, of one MO bra pair in half 2), T_b = C^T S_b C, kept for i >= j.  The FP64 pipe of this GPU runs at 1.1
// TFLOP/s (DGEMM) beside 1 900 TFLOP/s of FP16 products, so both products of a slice run as 36 exact FP16 digit
// products each (pq_digits.cuh): the result carries the rounding of U to 62 bits below its row bound and one final
// rounding to FP64, where DGEMM rounds at every term.
//
//   digits of S   rows (b, nu), one exponent per slice              slice_digits_kernel
//   product 1     U_b = S_b C: rows (b, nu) x rows m of C^T         digit_gemm_kernel<OUT_U>
//                 written as digits, rows (m, b), exponent from
//                 the bound |U| <= |C_m| max_nu |S_b[nu]|
//   product 2     T = U C: rows (m, b) x rows of C^T                digit_gemm_kernel<OUT_T>
//                 written as FP64 at [pair (m, n)][b]
//
// With rows (m, b) a warp's 32 accumulator lanes are 32 slices of one m, so the packed result goes out transposed in
// whole lines: half 1 leaves H1[ij][ket] as half 2 reads it and half 2 leaves (ij|kl) in its final place, with no
// transpose pass and no second half-transformed copy; column tiles right of the diagonal are skipped.
//
// Bound: L2 reads of the A operand (64 KB of digits per K chunk and column tile) in product 1, the accumulator drain,
// which cannot overlap the MMAs because eight orders fill TMEM, in product 2, and the digit writes in the slice pass.
// Measured at n = 150, 141 MOs: 11.8 ms against 336.6 ms with batched library DGEMM (product 1 5.2, product 2 3.5,
// slices 2.7 ms); n = 256: 153 ms against 4.16 s.  Against quadruple precision the 2-norm error is 7e-17 where
// DGEMM's is 3e-16 to 5e-16 (n = 24 and 40; normal, decaying, constant and eight-decade inputs).
#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

#include "pq_digits.cuh"
#include "pq_internal.h"
#include "pq_tc.cuh"

namespace pq {
namespace f64 {

using namespace tcx;

constexpr int BM = 128;                       // accumulator rows per tile (TMEM lanes)
constexpr int BN = 64;                        // accumulator columns per order; 8 orders fill TMEM's 512
constexpr int STAGES = 2;
constexpr int A_BOX = BM * 128, B_BOX = BN * 128;  // two digits of 32 K values: 128-byte rows
constexpr int BOXES = digits::N / 2;
constexpr int STAGE_BYTES = BOXES * (A_BOX + B_BOX);  // 96 KB
constexpr int EPI_WARPS = 16;                 // four per TMEM lane quadrant, a quarter of the columns each
constexpr int THREADS = 64 + 32 * EPI_WARPS;  // producer, MMA issuer, epilogue
constexpr int NBARS = 2 * STAGES + 3;         // full, empty, acc_full, acc_empty, drain
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 128;
static_assert(SMEM_BYTES <= 232448, "shared memory per CTA");

constexpr int STAGED_MAX = 220 * 1024;       // largest slice staged in shared memory (n <= 236)

enum { OUT_U = 0, OUT_T = 1 };
enum { ERR_FULL = 1, ERR_EMPTY = 2, ERR_ACC = 3 };

struct Args {
  int64_t m_tiles;
  int64_t M;        // accumulator rows: nb * kp (OUT_U) or n_mo * nbp (OUT_T)
  int n_tiles, bn;  // column tiles of bn columns (a multiple of 16, at most BN)
  int chunks;       // K chunks of 32
  int n_mo;         // columns
  int kp;           // OUT_U: rows per slice (n_ao up to a multiple of 32); the K length of U
  int nb, nbp;      // slices of this batch, and up to a multiple of 32
  const int *eS;    // exponent of each slice, of each row of C^T
  const int *eC;
  const float *nS;  // norm bounds: max row norm of each slice and norm of each row of C^T, in units of 2^e
  const float *nC;
  __half *U;        // OUT_U: digit rows (m, b)
  double *T;        // OUT_T: [pair][ld_t], slice b of this batch at column b
  int64_t ld_t;
  long long wait;
  int *err;
};

// exponent f with |U row| < 2^f in units of 2^(eS + eC)
__device__ __forceinline__ int bound_exp(float nS, float nC) {
  const float b = nS * nC * 1.0001f;
  return max(-1, (int)(__float_as_uint(b) >> 23) - 126);
}

// accumulator block of order l: the even orders, then the odd ones
__device__ __forceinline__ constexpr int order_block(int l) { return (l & 1) * (digits::N / 2) + (l >> 1); }

// Roles: warp 0 lane 0 loads stages (four 64-column boxes of A and of B: the eight digits of 32 K values), warp 1
// lane 0 issues the MMAs into the eight order accumulators, warps 2 .. 17 drain them.  The B boxes lie one behind
// the other, so digits of one parity are one operand of up to 4 bn rows: one MMA multiplies a digit of A with all of
// them, into neighbouring order blocks, and a K step takes 16 MMAs and A reads instead of 36.  The accumulators
// fill TMEM, so a tile's MMAs wait for the drain of the last one while the loads run ahead.  Every wait is bounded;
// one that runs out records an error and an abort flag that every role polls, the loads and MMAs in flight are
// waited for (bounded), and TMEM is freed.
template <int OUT>
__global__ void __launch_bounds__(THREADS, 1)
    digit_gemm_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, Args g) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + STAGES * STAGE_BYTES);
  uint64_t *full = bars, *empty = bars + STAGES, *accf = bars + 2 * STAGES, *acce = accf + 1, *drain = accf + 2;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + NBARS);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t tiles = g.m_tiles * g.n_tiles;

  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; i++) {
      mbar_init(smem_u32(full + i), 1);
      mbar_init(smem_u32(empty + i), 1);
    }
    mbar_init(smem_u32(accf), 1);
    mbar_init(smem_u32(acce), EPI_WARPS);
    mbar_init(smem_u32(drain), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  // a column tile right of the diagonal for every row of the tile holds nothing that is kept
  auto skip = [&](int64_t mt, int nt) {
    return OUT == OUT_T && nt * g.bn > (int)(min(mt * BM + BM, g.M) - 1) / g.nbp;
  };

  if (warp == 0 && lane == 0) {
    int gs = 0;
    for (int64_t t = blockIdx.x; t < tiles && !*abort_flag; t += gridDim.x) {
      const int64_t mt = t / g.n_tiles;
      const int nt = (int)(t - mt * g.n_tiles);
      if (skip(mt, nt)) continue;
      for (int c = 0; c < g.chunks; c++, gs++) {
        const int slot = gs % STAGES;
        if (!mbar_wait(smem_u32(empty + slot), (uint32_t)((gs / STAGES) & 1) ^ 1u, g.wait)) {
          atomicCAS(g.err, 0, ERR_EMPTY);
          *abort_flag = 1;
          break;
        }
        if (*abort_flag) break;
        const uint32_t st = smem_u32(smem + slot * STAGE_BYTES), bar = smem_u32(full + slot);
        mbar_expect_tx(bar, BOXES * (A_BOX + g.bn * 128));
        for (int i = 0; i < BOXES; i++) {
          const int x = c * (digits::CHUNK * digits::N) + 64 * i;
          tma_load_2d(st + i * A_BOX, &mapA, x, (int)(mt * BM), bar);
          tma_load_2d(st + BOXES * A_BOX + i * g.bn * 128, &mapB, x, nt * g.bn, bar);
        }
      }
    }
    // the loads in flight land before the CTA exits
    for (int j = gs > STAGES ? gs - STAGES : 0; j < gs; j++)
      mbar_wait(smem_u32(full + (j % STAGES)), (uint32_t)((j / STAGES) & 1), WAIT_CYCLES);
  } else if (warp == 1 && lane == 0) {
    uint32_t idesc[BOXES];  // N = 1 .. 4 blocks
    for (int j = 0; j < BOXES; j++) idesc[j] = idesc_f16((j + 1) * g.bn);
    int gs = 0, i = 0;
    bool ok = true;
    for (int64_t t = blockIdx.x; t < tiles && ok && !*abort_flag; t += gridDim.x) {
      const int64_t mt = t / g.n_tiles;
      const int nt = (int)(t - mt * g.n_tiles);
      if (skip(mt, nt)) continue;
      if (!mbar_wait(smem_u32(acce), (uint32_t)(i & 1) ^ 1u, g.wait)) {
        atomicCAS(g.err, 0, ERR_ACC);
        ok = false;
        break;
      }
      i++;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int c = 0; c < g.chunks; c++, gs++) {
        const int slot = gs % STAGES;
        if (!mbar_wait(smem_u32(full + slot), (uint32_t)((gs / STAGES) & 1), g.wait)) {
          atomicCAS(g.err, 0, ERR_FULL);
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a = smem_u32(smem + slot * STAGE_BYTES), b = a + BOXES * A_BOX;
        // digit i of a 32-value chunk: box i / 2, 64-byte half i % 2 of its rows; k steps of 16 values
#pragma unroll
        for (int k = 0; k < 2; k++)
#pragma unroll
          for (int da = 0; da < digits::N; da++)
#pragma unroll
            for (int par = 0; par < 2; par++) {
              // digits par, par + 2, .. of B as far as the order stays below 8
              if (da + par >= digits::N) continue;
              const int nj = (digits::N - 1 - da - par) / 2 + 1;
              mma_f16(tmem + order_block(da + par) * g.bn, smem_desc(a + (da >> 1) * A_BOX + (da & 1) * 64 + k * 32),
                      smem_desc(b + par * 64 + k * 32), idesc[nj - 1], (c | k | da) ? 1u : 0u);
            }
        mma_commit(smem_u32(empty + slot));
      }
      if (ok) mma_commit(smem_u32(accf));
    }
    if (!ok) *abort_flag = 1;
    mma_commit(smem_u32(drain));
    mbar_wait(smem_u32(drain), 0, WAIT_CYCLES);
  } else if (warp >= 2) {
    const int q = warp & 3, part = (warp - 2) >> 2;
    int i = 0;
    for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
      const int64_t mt = t / g.n_tiles;
      const int nt = (int)(t - mt * g.n_tiles);
      if (skip(mt, nt)) continue;
      const bool ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(accf), (uint32_t)(i & 1), g.wait));
      i++;
      if (!ok || __any_sync(0xffffffffu, *abort_flag != 0)) {
        if (!ok && lane == 0) atomicCAS(g.err, 0, ERR_ACC);
        *abort_flag = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16);
      // rows come in groups of 32 that share their slice (OUT_U) or their m (OUT_T)
      const int64_t r0 = mt * BM + q * 32;
      const bool rows_in = r0 < g.M;
      const int per = OUT == OUT_U ? g.kp : g.nbp;
      const int outer = rows_in ? (int)(r0 / per) : 0, inner = rows_in ? (int)(r0 - (int64_t)outer * per) : 0;
      // column groups of 8, in turn between the warps of a quadrant
      for (int c0 = 8 * part; c0 < g.bn; c0 += 8 * (EPI_WARPS / 4)) {
        uint32_t acc[digits::N][8];
#pragma unroll
        for (int l = 0; l < digits::N; l++) tmem_ld8(taddr + order_block(l) * g.bn + c0, acc[l]);
        tmem_wait();
        const int col0 = nt * g.bn + c0;
        if (!rows_in || col0 >= g.n_mo || (OUT == OUT_T && col0 > outer)) continue;
        int eS = 0, eC = 0;
        float nS = 0.0f;
        if (OUT == OUT_T) {
          const int b = min(inner + lane, g.nb - 1);
          eS = __ldg(g.eS + b), nS = __ldg(g.nS + b);
          eC = __ldg(g.eC + outer);
          eS += eC + bound_exp(nS, __ldg(g.nC + outer)) - 68;
        } else {
          nS = __ldg(g.nS + outer);
        }
#pragma unroll
        for (int c = 0; c < 8; c++) {
          const int m = col0 + c;
          if (m >= g.n_mo || (OUT == OUT_T && m > outer)) break;
          float a[digits::N];
#pragma unroll
          for (int l = 0; l < digits::N; l++) a[l] = __uint_as_float(acc[l][c]);
          int64_t hi, lo;
          digits::combine(a, hi, lo);
          if constexpr (OUT == OUT_U) {
            // digits of U relative to its row's bound; row (m, b), K = inner + lane
            const int sh = 6 + bound_exp(nS, __ldg(g.nC + m));
            __half2 d[4];
            digits::to_half((hi << (32 - sh)) + (lo >> sh), d);
            // lane pairs exchange digits, so that each lane stores two neighbouring K values of four digits
            const bool odd = lane & 1;
            const uint32_t d0 = *reinterpret_cast<uint32_t *>(d), d1 = *reinterpret_cast<uint32_t *>(d + 1);
            const uint32_t d2 = *reinterpret_cast<uint32_t *>(d + 2), d3 = *reinterpret_cast<uint32_t *>(d + 3);
            const uint32_t x0 = __shfl_xor_sync(0xffffffffu, odd ? d0 : d2, 1), x1 = __shfl_xor_sync(0xffffffffu, odd ? d1 : d3, 1);
            // even lanes: (own, neighbour) of digits 0 .. 3; odd lanes: (neighbour, own) of digits 4 .. 7
            const uint32_t f0 = odd ? x0 : d0, s0 = odd ? d2 : x0, f1 = odd ? x1 : d1, s1 = odd ? d3 : x1;
            uint32_t *u = reinterpret_cast<uint32_t *>(g.U + ((int64_t)m * g.nbp + outer) * (int64_t)(g.kp * digits::N) +
                                                       (int64_t)inner * digits::N) +
                          (odd ? 4 * (digits::CHUNK / 2) : 0) + (lane >> 1);
            u[0] = __byte_perm(f0, s0, 0x5410);
            u[digits::CHUNK / 2] = __byte_perm(f0, s0, 0x7632);
            u[2 * (digits::CHUNK / 2)] = __byte_perm(f1, s1, 0x5410);
            u[3 * (digits::CHUNK / 2)] = __byte_perm(f1, s1, 0x7632);
          } else {
            const int e = eS + __ldg(g.eC + m);
            const double v = e >= digits::BAD / 2 ? __longlong_as_double(0x7ff8000000000000LL) : digits::to_double(hi, lo, e);
            if (inner + lane < g.nb)
              g.T[((int64_t)outer * (outer + 1) / 2 + m) * g.ld_t + inner + lane] = v;
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(acce));
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

__device__ __forceinline__ int64_t tri(int64_t i, int64_t j) { return i > j ? i * (i + 1) / 2 + j : j * (j + 1) / 2 + i; }

// two neighbouring K values of a digit row: the lane pair (2 l, 2 l + 1) of a 32-value chunk
__device__ __forceinline__ void store_pair(__half *chunk, int l, int64_t t0, int64_t t1) {
  __half2 a[4], b[4];
  digits::to_half(t0, a);
  digits::to_half(t1, b);
  __half2 *o = reinterpret_cast<__half2 *>(chunk) + l;
#pragma unroll
  for (int p = 0; p < 4; p++) {
    o[(2 * p) * (digits::CHUNK / 2)] = __lows2half2(a[p], b[p]);
    o[(2 * p + 1) * (digits::CHUNK / 2)] = __highs2half2(a[p], b[p]);
  }
}

__device__ __forceinline__ uint32_t block_max(uint32_t x, uint32_t *red) {
  x = __reduce_max_sync(0xffffffffu, x);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
  __syncthreads();
  uint32_t m = 0;
  for (unsigned w = 0; w < blockDim.x / 32; w++) m = max(m, red[w]);
  return m;
}

// Digit rows of C^T: block per row m, its exponent and norm
__global__ void __launch_bounds__(128) ct_digits_kernel(const double *C, int64_t ldc, int n, int kp, __half *out, int *e,
                                                       float *nrm) {
  __shared__ uint32_t red[4];
  const int m = blockIdx.x;
  const double *c = C + (int64_t)m * ldc;
  uint32_t hi = 0;
  for (int k = threadIdx.x; k < n; k += blockDim.x) hi = max(hi, (uint32_t)__double2hiint(c[k]) & 0x7fffffffu);
  const int ex = digits::exponent_of(block_max(hi, red));
  float s = 0.0f;
  for (int k = 2 * threadIdx.x; k < kp; k += 2 * blockDim.x) {
    const int64_t t0 = k < n && ex != digits::BAD ? digits::fixed_point(c[k], ex) : 0;
    const int64_t t1 = k + 1 < n && ex != digits::BAD ? digits::fixed_point(c[k + 1], ex) : 0;
    store_pair(out + (int64_t)m * kp * digits::N + (k / digits::CHUNK) * (digits::CHUNK * digits::N), (k % digits::CHUNK) / 2,
               t0, t1);
    const float x = (float)(int)(t0 >> 32) * 0x1p-30f, y = (float)(int)(t1 >> 32) * 0x1p-30f;
    s += x * x + y * y;
  }
  // the norm of the row in units of 2^ex: a sum of at most 256 FP32 squares, raised past its rounding
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = __float_as_uint(s);
  __syncthreads();
  if (threadIdx.x == 0) {
    float tot = 0.0f;
    for (int w = 0; w < 4; w++) tot += __uint_as_float(red[w]);
    e[m] = ex;
    nrm[m] = sqrtf(tot) * 1.0001f;
  }
}

// Digit rows of the slices b0 .. b0 + gridDim.x - 1: block per slice, kp rows of kp values (zero past n), one exponent
// per slice and the largest row norm.  src is 8-fold packed or a pair matrix with columns of ld pairs.  STAGED: the
// slice's pairs are converted once to fixed point in shared memory, which both triangles read; larger slices are
// read again from L1/L2.
template <bool STAGED>
__global__ void __launch_bounds__(512) slice_digits_kernel(const double *src, int packed, int64_t ld, int n, int kp,
                                                          int64_t b0, __half *out, int *e, float *nrm) {
  extern __shared__ int64_t pairs[];
  __shared__ uint32_t red[16], top;
  const int64_t b = blockIdx.x, ket = b0 + b;
  const int np = n * (n + 1) / 2;
  auto value = [&](int bra) { return __ldg(packed ? src + tri(bra, ket) : src + bra + ket * ld); };
  uint32_t hi = 0;
  for (int i = threadIdx.x; i < np; i += blockDim.x) {
    const double x = value(i);
    if (STAGED) pairs[i] = __double_as_longlong(x);
    hi = max(hi, (uint32_t)__double2hiint(x) & 0x7fffffffu);
  }
  const int ex = digits::exponent_of(block_max(hi, red));
  if (threadIdx.x == 0) top = 0;
  if (STAGED)
    for (int i = threadIdx.x; i < np; i += blockDim.x)  // the entries this thread stored
      pairs[i] = ex == digits::BAD ? 0 : digits::fixed_point(__longlong_as_double(pairs[i]), ex);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  __half *rows = out + b * (int64_t)kp * kp * digits::N;
  for (int nu = threadIdx.x >> 5; nu < kp; nu += blockDim.x >> 5) {
    float s = 0.0f;
    for (int k = 2 * lane; k < kp; k += 64) {
      int64_t t[2] = {0, 0};
#pragma unroll
      for (int j = 0; j < 2; j++)
        if (nu < n && k + j < n) {
          const int i = (int)tri(nu, k + j);
          if (STAGED)
            t[j] = pairs[i];
          else if (ex != digits::BAD)
            t[j] = digits::fixed_point(value(i), ex);
        }
      store_pair(rows + (int64_t)nu * kp * digits::N + (k / digits::CHUNK) * (digits::CHUNK * digits::N),
                 (k % digits::CHUNK) / 2, t[0], t[1]);
      const float x = (float)(int)(t[0] >> 32) * 0x1p-30f, y = (float)(int)(t[1] >> 32) * 0x1p-30f;
      s += x * x + y * y;
    }
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) atomicMax(&top, __float_as_uint(s));
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    e[b] = ex;
    nrm[b] = sqrtf(__uint_as_float(top)) * 1.0001f;
  }
}

}  // namespace f64

// digit rows: boxes of 64 FP16 (two digits of a chunk) x box_rows, 128-byte swizzle, zeros past the last row
static pq_status f64_map(CUtensorMap *m, const void *base, int64_t rows, int64_t row_len, int box_rows) {
  auto fn = tcx::encode_fn();
  if (!fn) {
    set_error("cuTensorMapEncodeTiled is not available from the driver");
    return PQ_ERR_CUDA;
  }
  cuuint64_t dims[2] = {(cuuint64_t)row_len, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)row_len * 2};
  cuuint32_t box[2] = {64, (cuuint32_t)box_rows}, es[2] = {1, 1};
  const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(base), dims, strides, box, es,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed (%d): %lld digit rows of %lld", (int)r, (long long)rows, (long long)row_len);
    return PQ_ERR_CUDA;
  }
  return PQ_OK;
}

static int64_t up(int64_t x, int64_t m) { return (x + m - 1) / m * m; }

// One half transform: T[pair of C's columns][b] for the nket slices of src.
static pq_status f64_half(Ao2moF64 &w, const double *src, int packed, int64_t ld, int n, int64_t nket, const double *C,
                          int64_t ldc, int m, double *T, int sms, cudaStream_t st) {
  using namespace f64;
  const int kp = (int)up(n, digits::CHUNK);
  const int64_t rl = (int64_t)kp * digits::N;  // FP16 per digit row
  // slices per batch: about 1.5 GB of digits, and whole tiles of one m in product 2
  const int64_t per = (int64_t)sizeof(__half) * rl * (kp + m);
  const int64_t bt = std::min<int64_t>(up(nket, 32), std::max<int64_t>(128, (((int64_t)3 << 29) / per) / 128 * 128));
  PQ_TRY(w.ct.ensure(sizeof(__half) * rl * m));
  PQ_TRY(w.s.ensure(sizeof(__half) * rl * kp * bt));
  PQ_TRY(w.u.ensure(sizeof(__half) * rl * m * bt));
  PQ_TRY(w.e.ensure((sizeof(int) + sizeof(float)) * (size_t)(bt + m)));
  int *eS = w.e.as<int>(), *eC = eS + bt;
  float *nS = reinterpret_cast<float *>(eC + m), *nC = nS + bt;
  ct_digits_kernel<<<m, 128, 0, st>>>(C, ldc, n, kp, w.ct.as<__half>(), eC, nC);
  PQ_CUDA_TRY(cudaGetLastError());
  Args g{};
  g.n_tiles = (m + BN - 1) / BN;
  g.bn = (int)up((m + g.n_tiles - 1) / g.n_tiles, 16);
  g.chunks = kp / digits::CHUNK;
  g.n_mo = m;
  g.kp = kp;
  g.eS = eS, g.eC = eC, g.nS = nS, g.nC = nC;
  g.U = w.u.as<__half>();
  g.ld_t = nket;
  g.wait = ao2mo_wait_cycles();
  g.err = w.err.as<int>();
  const int staged = (int)sizeof(int64_t) * n * (n + 1) / 2;
  CUtensorMap mapC;
  PQ_TRY(f64_map(&mapC, w.ct.ptr, m, rl, g.bn));
  for (int64_t b0 = 0; b0 < nket; b0 += bt) {
    g.nb = (int)std::min(bt, nket - b0);
    g.nbp = (int)up(g.nb, 32);
    if (staged <= STAGED_MAX)
      slice_digits_kernel<true><<<(unsigned)g.nb, 512, staged, st>>>(src, packed, ld, n, kp, b0, w.s.as<__half>(), eS, nS);
    else
      slice_digits_kernel<false><<<(unsigned)g.nb, 512, 0, st>>>(src, packed, ld, n, kp, b0, w.s.as<__half>(), eS, nS);
    PQ_CUDA_TRY(cudaGetLastError());
    CUtensorMap mapS, mapU;
    g.M = (int64_t)g.nb * kp;
    g.m_tiles = (g.M + BM - 1) / BM;
    PQ_TRY(f64_map(&mapS, w.s.ptr, g.M, rl, BM));
    digit_gemm_kernel<OUT_U><<<(unsigned)std::min<int64_t>(g.m_tiles * g.n_tiles, sms), THREADS, SMEM_BYTES, st>>>(mapS, mapC, g);
    PQ_CUDA_TRY(cudaGetLastError());
    g.M = (int64_t)m * g.nbp;
    g.m_tiles = (g.M + BM - 1) / BM;
    g.T = T + b0;
    PQ_TRY(f64_map(&mapU, w.u.ptr, g.M, rl, BM));
    digit_gemm_kernel<OUT_T><<<(unsigned)std::min<int64_t>(g.m_tiles * g.n_tiles, sms), THREADS, SMEM_BYTES, st>>>(mapU, mapC, g);
    PQ_CUDA_TRY(cudaGetLastError());
  }
  return PQ_OK;
}

// n_ao <= 256 per species (one exact K range); w is this device's workspace, held by the caller's lock
pq_status ao2mo_f64(Ao2moF64 &w, const double *eri_ao, int layout, int64_t n_ao_a, int64_t n_ao_b, const double *Ca,
                    int64_t lda, int64_t nmo_a, const double *Cb, int64_t ldb, int64_t nmo_b, double *eri_mo,
                    cudaStream_t st) {
  using namespace f64;
  int dev = 0, sms = 0;
  PQ_CUDA_TRY(cudaGetDevice(&dev));
  PQ_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  PQ_CUDA_TRY(cudaFuncSetAttribute(digit_gemm_kernel<OUT_U>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
  PQ_CUDA_TRY(cudaFuncSetAttribute(digit_gemm_kernel<OUT_T>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
  PQ_CUDA_TRY(cudaFuncSetAttribute(slice_digits_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, STAGED_MAX));
  const int64_t npa = n_ao_a * (n_ao_a + 1) / 2, npb = n_ao_b * (n_ao_b + 1) / 2, nma = nmo_a * (nmo_a + 1) / 2;
  PQ_TRY(w.h1.ensure(sizeof(double) * npb * nma));
  PQ_TRY(w.err.ensure(sizeof(int)));
  PQ_CUDA_TRY(cudaMemsetAsync(w.err.ptr, 0, sizeof(int), st));
  // half 1 over AO ket pairs: H1[ij][ket]; half 2 over MO bra pairs: (ij|kl) at [kl][ij]
  PQ_TRY(f64_half(w, eri_ao, layout == PQ_AO_PACKED8, npa, (int)n_ao_a, npb, Ca, lda, (int)nmo_a, w.h1.as<double>(), sms, st));
  PQ_TRY(f64_half(w, w.h1.as<double>(), 0, npb, (int)n_ao_b, nma, Cb, ldb, (int)nmo_b, eri_mo, sms, st));
  int herr = 0;
  PQ_CUDA_TRY(cudaMemcpyAsync(&herr, w.err.ptr, sizeof(int), cudaMemcpyDeviceToHost, st));
  PQ_CUDA_TRY(cudaStreamSynchronize(st));
  if (herr) {
    set_error("ao2mo FP64 digit product: bounded wait gave up (code %d)", herr);
    return PQ_TIMEOUT;
  }
  return PQ_OK;
}

}  // namespace pq
