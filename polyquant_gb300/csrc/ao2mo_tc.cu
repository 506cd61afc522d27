// Split-precision AO->MO transform on the tcgen05 tensor cores.
//
// Same two pair-symmetric half transforms as the FP64 path (ao2mo.cu): for
// each slice S (a symmetric n x n matrix: one ket AO pair in half 1, one bra MO
// pair in half 2), T = C^T S C, written packed (i >= j).  Each slice costs two
// GEMMs, both in the "A (M x K, K-major) times B (N x K, K-major)^T" form:
//   GEMM 1:  U^T[m][nu] = sum_mu Ct[m][mu] S[nu][mu]    (A = C^T shared, B = S per slice)
//   GEMM 2:  T[m][n]   = sum_nu U^T[m][nu] Ct[n][nu]    (A = U^T of all slices, B = C^T shared)
// GEMM 1 leaves U^T with rows (m, slice).  A tile of GEMM 2 then holds 128 slices of one m, or a few m: it loads and
// multiplies only the columns n <= m, half of the work, and its 32 lanes hold 32 slices, so that a pair (m, n) is
// written along the slices, as half 2 reads it and as the result wants it, and no transpose is left (256 AOs, BF16x3:
// two transposes of 13 + 8.7 GB and the FP64 expansion, 35.8 ms in all; without them 24.7).  In BF16 GEMM 1 reads the
// slices from their pair rows (slice_gemm_kernel); in TF32 they are split in memory first.
// Operands are split into a high and a low part (x = x_hi + x_lo) in BF16 or
// TF32 and each product is formed as hi*hi + hi*lo + lo*hi with FP32
// accumulation in tensor memory (three MMAs per K step).  BF16 and TF32 keep
// FP32's 8-bit exponent, so no per-block scaling is needed for range.
//
// GEMM kernel: persistent, one CTA per SM looping over 128 x 256 output
// tiles, warp-specialised: one thread issues TMA tile loads (128-byte
// swizzle, a ring of two stages of K = 128 bytes of each of A_hi, A_lo, B_hi,
// B_lo), one thread issues the tcgen05.mma instructions into one of two TMEM
// accumulators (128 lanes x 256 FP32 columns each; as many columns as the tile has), and four warps drain the
// other accumulator with tcgen05.ld for the epilogue (BF16/TF32 split of the
// result for the next GEMM, or the packed lower triangle).  Every mbarrier
// wait is bounded; a wait that runs out records an error code and the kernel
// winds down (waits, bounded again, for its own loads and MMAs, frees TMEM).
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "pq_internal.h"
#include "pq_tc.cuh"

namespace pq {

namespace tc {

using namespace tcx;

constexpr int BM = 128;          // output rows per CTA (TMEM lanes)
constexpr int BN = 256;          // output columns per CTA (TMEM columns, UMMA N)
constexpr int ROW_BYTES = 128;   // K extent of one stage, in bytes (one swizzle span)
// Persistent warp-specialised GEMM: one CTA per SM, a ring of two 96 KB
// operand stages, and two TMEM accumulators (2 x 256 columns) so the epilogue
// of one tile overlaps the loads and MMAs of the next.
constexpr int STAGES = 2;
constexpr int A_TILE = BM * ROW_BYTES;  // 16 KB
constexpr int B_TILE = BN * ROW_BYTES;  // 32 KB
constexpr int B_BOX = 64;               // B rows per load: a tile loads the boxes that it has columns for
constexpr int STAGE_BYTES = 2 * A_TILE + 2 * B_TILE;
constexpr int EPI_WARPS = 4;
constexpr int EPI_LD = 33;                                  // per-warp 32 x 32 staging, odd stride
constexpr int EPI_BYTES = EPI_WARPS * 32 * EPI_LD * 4;      // 16.5 KB
constexpr int NBARS = 2 * STAGES + 4 + 1;                   // full, empty, acc_full[2], acc_empty[2], drain
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + EPI_BYTES + 1024 /*align*/ + 256 /*barriers, slots*/;
constexpr int GEMM_THREADS = 64 + 32 * EPI_WARPS;           // producer warp, MMA warp, epilogue warps

enum { EPI_SPLIT = 0, EPI_PACK = 1 };
enum { ERR_TIMEOUT_FULL = 1, ERR_TIMEOUT_MMA = 2, ERR_TIMEOUT_ACC = 3 };

struct GemmArgs {
  int M, N, K;                 // logical sizes (EPI_PACK: M = n_mo * nbp rows)
  int m_tiles;                 // ceil(M / BM)
  int nbatch;                  // EPI_SPLIT: slices, one B operand of b_rows rows each (tiles = nbatch * m_tiles)
  int b_rows;
  int nb, nbp;                 // slices of this batch, and up to a multiple of 32
  int ld_out;                  // EPI_SPLIT: row length of the split output
  float *out_hi, *out_lo;      // EPI_SPLIT outputs (TF32), rows (m, slice)
  void *out_pack;              // EPI_PACK output [pair (m, n)][ld_pack], slice b of this batch in column b
  int64_t ld_pack;
  long long wait_cycles;       // budget of the pipeline waits (the wind-down waits keep WAIT_CYCLES)
  int *err;
};

// EPI_PACK: rows (m, slice), so a tile holds few m; only columns n <= m are kept, and the tile takes a whole number of
// B boxes up to the last of them
// (the widest tiles come first, so that the last ones even the SMs out)
template <int EPI> __device__ __forceinline__ void tile_at(const GemmArgs &g, int t, int &b, int &mt) {
  b = EPI == EPI_SPLIT ? t / g.m_tiles : 0;
  mt = EPI == EPI_SPLIT ? t - b * g.m_tiles : g.m_tiles - 1 - t;
}
template <int EPI> __device__ __forceinline__ int tile_cols(const GemmArgs &g, int64_t row0) {
  if (EPI == EPI_SPLIT) return g.N;
  const int64_t last = row0 + BM < g.M ? row0 + BM : g.M;
  const int n = (int)((last - 1) / g.nbp) + 1;
  return n < g.N ? n : g.N;
}

// instruction descriptor: D = F32, A/B format (1 = BF16 for kind::f16, 2 = TF32), K-major A and B, n columns
__host__ __device__ constexpr uint32_t instr_desc(uint32_t ab_format, int n) {
  return (1u << 4) | (ab_format << 7) | (ab_format << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}

template <bool TF32>
__device__ __forceinline__ void mma(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accum) {
  if constexpr (TF32) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(accum)
        : "memory");
  } else {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(accum)
        : "memory");
  }
}

__device__ __forceinline__ float tf32_round(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}

// TF32 = operands stored as FP32 (tf32-rounded); otherwise BF16.
// Roles: warp 0 lane 0 issues TMA loads into the stage ring, warp 1 lane 0
// issues the MMAs (tile i into accumulator i & 1), warps 2..5 drain the
// accumulators (warp w reads TMEM lanes 32 (w & 3) .. + 31) through a
// per-warp shared-memory staging block into coalesced row stores.  Barriers:
// full[s] (loads landed), empty[s] (MMAs reading stage s done), acc_full[a]
// (tile's MMAs done), acc_empty[a] (epilogue done with accumulator a).  Every
// wait is bounded; a wait that runs out sets the error word and an abort flag
// that every role polls, the producer then waits (bounded) for its own loads
// in flight, the MMA thread for its own MMAs, and the CTA frees TMEM.
template <bool TF32, int EPI, typename TO>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
    tc_gemm_kernel(const __grid_constant__ CUtensorMap tmA_hi, const __grid_constant__ CUtensorMap tmA_lo,
                   const __grid_constant__ CUtensorMap tmB_hi, const __grid_constant__ CUtensorMap tmB_lo, GemmArgs g) {
  static_assert(TF32 || EPI == EPI_PACK, "BF16 slices go through slice_gemm_kernel");
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // 1024-byte alignment of the shared-window address (128-byte swizzle atoms)
  unsigned char *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  float *epi = reinterpret_cast<float *>(smem + STAGES * STAGE_BYTES);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + STAGES * STAGE_BYTES + EPI_BYTES);
  uint64_t *full = bars, *empty = bars + STAGES, *accf = bars + 2 * STAGES, *acce = bars + 2 * STAGES + 2;
  uint64_t *drain = bars + 2 * STAGES + 4;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + NBARS);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int ESZ = TF32 ? 4 : 2;
  constexpr int BK = ROW_BYTES / ESZ;  // K elements per stage
  constexpr int UK = TF32 ? 8 : 16;    // K per MMA instruction
  const int nst = (g.K + BK - 1) / BK;
  const int n_tiles = g.nbatch * g.m_tiles;

  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; i++) {
      mbar_init(smem_u32(full + i), 1);
      mbar_init(smem_u32(empty + i), 1);
    }
    for (int a = 0; a < 2; a++) {
      mbar_init(smem_u32(accf + a), 1);
      mbar_init(smem_u32(acce + a), EPI_WARPS);
    }
    mbar_init(smem_u32(drain), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(2 * BN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  if (warp == 0 && lane == 0) {
    // ---- producer
    int gs = 0;
    for (int t = blockIdx.x; t < n_tiles && !*abort_flag; t += gridDim.x) {
      int b, mt;
      tile_at<EPI>(g, t, b, mt);
      const int ya = mt * BM, yb = b * g.b_rows;
      const int boxes = (tile_cols<EPI>(g, ya) + B_BOX - 1) / B_BOX;
      for (int s = 0; s < nst; s++, gs++) {
        const int slot = gs % STAGES;
        const uint32_t ph = (uint32_t)((gs / STAGES) & 1);
        if (!mbar_wait(smem_u32(empty + slot), ph ^ 1u, g.wait_cycles)) {
          atomicCAS(g.err, 0, ERR_TIMEOUT_MMA);
          *abort_flag = 1;
          break;
        }
        if (*abort_flag) break;
        unsigned char *st = smem + slot * STAGE_BYTES;
        const uint32_t bar = smem_u32(full + slot);
        mbar_expect_tx(bar, 2 * A_TILE + 2 * boxes * B_BOX * ROW_BYTES);
        const int x = s * BK;
        tma_load_2d(smem_u32(st), &tmA_hi, x, ya, bar);
        tma_load_2d(smem_u32(st + A_TILE), &tmA_lo, x, ya, bar);
        for (int i = 0; i < boxes; i++) {
          tma_load_2d(smem_u32(st + 2 * A_TILE + i * B_BOX * ROW_BYTES), &tmB_hi, x, yb + i * B_BOX, bar);
          tma_load_2d(smem_u32(st + 2 * A_TILE + B_TILE + i * B_BOX * ROW_BYTES), &tmB_lo, x, yb + i * B_BOX, bar);
        }
      }
    }
    // the loads of the last stages must have landed before the CTA exits
    for (int j = gs > STAGES ? gs - STAGES : 0; j < gs; j++)
      mbar_wait(smem_u32(full + (j % STAGES)), (uint32_t)((j / STAGES) & 1), WAIT_CYCLES);
  } else if (warp == 1 && lane == 0) {
    // ---- MMA issuer
    int gs = 0, i = 0;
    for (int t = blockIdx.x; t < n_tiles && !*abort_flag; t += gridDim.x, i++) {
      const int a = i & 1;
      const uint32_t aph = (uint32_t)((i >> 1) & 1);
      if (!mbar_wait(smem_u32(acce + a), aph ^ 1u, g.wait_cycles)) {
        atomicCAS(g.err, 0, ERR_TIMEOUT_ACC);
        *abort_flag = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t d = tmem + (uint32_t)(a * BN);
      int b, mt;
      tile_at<EPI>(g, t, b, mt);
      const uint32_t idesc = instr_desc(TF32 ? 2u : 1u, (tile_cols<EPI>(g, (int64_t)mt * BM) + 15) / 16 * 16);
      bool ok = true;
      for (int s = 0; s < nst; s++, gs++) {
        const int slot = gs % STAGES;
        const uint32_t ph = (uint32_t)((gs / STAGES) & 1);
        if (!mbar_wait(smem_u32(full + slot), ph, g.wait_cycles)) {
          atomicCAS(g.err, 0, ERR_TIMEOUT_FULL);
          *abort_flag = 1;
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        unsigned char *st = smem + slot * STAGE_BYTES;
        const uint32_t a_hi = smem_u32(st), a_lo = smem_u32(st + A_TILE);
        const uint32_t b_hi = smem_u32(st + 2 * A_TILE), b_lo = smem_u32(st + 2 * A_TILE + B_TILE);
#pragma unroll
        for (int kk = 0; kk < BK / UK; kk++) {
          const uint32_t off = kk * UK * ESZ;  // bytes along K inside the swizzle span
          const uint32_t acc0 = (s > 0 || kk > 0) ? 1u : 0u;
          mma<TF32>(d, smem_desc(a_hi + off), smem_desc(b_hi + off), idesc, acc0);
          mma<TF32>(d, smem_desc(a_hi + off), smem_desc(b_lo + off), idesc, 1u);
          mma<TF32>(d, smem_desc(a_lo + off), smem_desc(b_hi + off), idesc, 1u);
        }
        mma_commit(smem_u32(empty + slot));  // frees the stage once these MMAs completed
      }
      if (!ok) break;
      mma_commit(smem_u32(accf + a));
    }
    // every MMA issued by this thread has completed before TMEM is freed
    mma_commit(smem_u32(drain));
    mbar_wait(smem_u32(drain), 0, WAIT_CYCLES);
  } else if (warp >= 2) {
    // ---- epilogue
    const int q = warp & 3;  // TMEM lane quadrant of this warp
    float *stg = epi + (warp - 2) * 32 * EPI_LD;
    int i = 0;
    for (int t = blockIdx.x; t < n_tiles; t += gridDim.x, i++) {
      const int a = i & 1;
      const uint32_t aph = (uint32_t)((i >> 1) & 1);
      const bool ok = warp_wait(smem_u32(accf + a), aph, g.wait_cycles);
      if (!ok || warp_aborted(abort_flag)) {
        if (!ok && lane == 0) atomicCAS(g.err, 0, ERR_TIMEOUT_ACC);
        *abort_flag = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      int b, mt;
      tile_at<EPI>(g, t, b, mt);
      const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(a * BN);
      const int row0 = mt * BM + q * 32;
      const int cols = tile_cols<EPI>(g, (int64_t)mt * BM);
      // EPI_PACK: 32 rows of one m, lanes are slices
      const int pm = EPI == EPI_PACK ? row0 / g.nbp : 0, pb = EPI == EPI_PACK ? row0 - pm * g.nbp + lane : 0;
      for (int c0 = 0; c0 < cols; c0 += 32) {
        float v[32];
        tmem_ld32(taddr + c0, v);  // v[j] = D[row0 + lane][c0 + j]
        if constexpr (EPI == EPI_SPLIT) {
#pragma unroll
          for (int j = 0; j < 32; j++) stg[lane * EPI_LD + j] = v[j];
          __syncwarp();
          // four lanes per row, eight consecutive columns per lane: 16-byte stores
          // (rows of ld_out = a multiple of 8 elements, so n0 keeps them aligned)
          const int cq = (lane & 3) * 8, n0 = c0 + cq;
#pragma unroll
          for (int it = 0; it < 4; it++) {
            const int rr = it * 8 + (lane >> 2), m = row0 + rr;
            if (m >= g.M || n0 >= g.N) continue;
            float x[8];
#pragma unroll
            for (int k = 0; k < 8; k++) x[k] = stg[rr * EPI_LD + cq + k];
            const int64_t o = ((int64_t)m * g.nbp + b) * g.ld_out + n0;
            float h[8], l[8];
#pragma unroll
            for (int k = 0; k < 8; k++) {
              h[k] = tf32_round(x[k]);
              l[k] = tf32_round(x[k] - h[k]);
            }
            float *oh = g.out_hi + o, *ol = g.out_lo + o;
            if (n0 + 8 <= g.N) {
              reinterpret_cast<float4 *>(oh)[0] = make_float4(h[0], h[1], h[2], h[3]);
              reinterpret_cast<float4 *>(oh)[1] = make_float4(h[4], h[5], h[6], h[7]);
              reinterpret_cast<float4 *>(ol)[0] = make_float4(l[0], l[1], l[2], l[3]);
              reinterpret_cast<float4 *>(ol)[1] = make_float4(l[4], l[5], l[6], l[7]);
            } else {
              for (int k = 0; k < g.N - n0; k++) oh[k] = h[k], ol[k] = l[k];
            }
          }
          __syncwarp();
        } else if (row0 < g.M && pb < g.nb) {
          TO *o = static_cast<TO *>(g.out_pack) + ((int64_t)pm * (pm + 1) / 2 + c0) * g.ld_pack + pb;
#pragma unroll
          for (int j = 0; j < 32; j++)
            if (c0 + j <= pm) o[(int64_t)j * g.ld_pack] = (TO)v[j];
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(acce + a));
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * BN) : "memory");
}

// ---------------------------------------------------------------------------
// operand preparation
template <bool TF32> struct Split;
// The split works in FP32: hi + lo carry at most 2 x 8 (BF16) or 2 x 11
// (TF32) significant bits, fewer than FP32's 24, and GB300 runs FP64
// arithmetic at a small fraction of the FP32 rate (one FP64 -> FP32
// conversion per element remains for FP64 sources).
template <> struct Split<false> {
  using T = __nv_bfloat16;
  static __device__ __forceinline__ void run(float x, T &h, T &l) {
    h = __float2bfloat16_rn(x);
    l = __float2bfloat16_rn(x - __bfloat162float(h));
  }
};
template <> struct Split<true> {
  using T = float;
  static __device__ __forceinline__ void run(float x, T &h, T &l) {
    h = tf32_round(x);
    l = tf32_round(x - h);
  }
};

// Ct[m][mu] = C[mu + m*ldc], split, row length ld (>= n_ao)
template <bool TF32>
__global__ void split_ct_kernel(const double *C, int64_t ldc, int n_ao, int n_mo, int ld, typename Split<TF32>::T *hi,
                                typename Split<TF32>::T *lo) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (int64_t)n_mo * ld) return;
  int m = (int)(i / ld), mu = (int)(i - (int64_t)m * ld);
  float x = mu < n_ao ? (float)C[mu + (int64_t)m * ldc] : 0.0f;
  Split<TF32>::run(x, hi[i], lo[i]);
}

// slice b of a pair-matrix source, split (TF32): S[b][nu][mu] = src(tri(mu,nu), b0 + b)
// src64: column-major (ld x ncols) FP64 pair matrix (element (r, c) at r + c*ld)
// src32: row-major FP32 pair rows (element (r, c) at c*ld + r), i.e. row c holds the slice
// Two consecutive row elements (a at o, b at o + 1; o even, so the pair is 8-byte aligned) go with one vector store
// each when both are wanted.
__device__ __forceinline__ void split_store2(float *H, float *L, int64_t o, float a, float b, bool va, bool vb) {
  if (va && vb) {
    const float ha = tf32_round(a), hb = tf32_round(b);
    *reinterpret_cast<float2 *>(H + o) = make_float2(ha, hb);
    *reinterpret_cast<float2 *>(L + o) = make_float2(tf32_round(a - ha), tf32_round(b - hb));
  } else {
    if (va) Split<true>::run(a, H[o], L[o]);
    if (vb) Split<true>::run(b, H[o + 1], L[o + 1]);
  }
}

// One block per (slice, 32x32 tile of the lower triangle): the tile is read
// with consecutive pair indices (mu <= nu) and written to both triangles, the
// upper one through a shared-memory transpose, so loads and stores are
// coalesced and every slice spreads over many SMs.  Each thread handles two
// consecutive columns (16 column pairs x 16 rows per pass).
__global__ void __launch_bounds__(256) split_slices_kernel(const double *src64, const float *src32, int64_t ld, int n,
                                                           int ld_row, int64_t b0, float *hi, float *lo) {
  __shared__ float tile[32][33];
  const int nt = (n + 31) / 32;
  const int tv = blockIdx.y / nt, tm = blockIdx.y - tv * nt;
  if (tm > tv) return;
  const int64_t b = blockIdx.x, c = b0 + b;
  float *H = hi + b * (int64_t)n * ld_row, *L = lo + b * (int64_t)n * ld_row;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  for (int y = ty; y < 32; y += 16) {
    const int nu = tv * 32 + y, mu = tm * 32 + 2 * tx;
    const bool va = nu < n && mu <= nu, vb = nu < n && mu + 1 <= nu;
    float xa = 0.0f, xb = 0.0f;
    const int64_t pr = (int64_t)nu * (nu + 1) / 2 + mu;
    if (va) xa = src64 ? (float)src64[pr + c * ld] : src32[c * ld + pr];
    if (vb) xb = src64 ? (float)src64[pr + 1 + c * ld] : src32[c * ld + pr + 1];
    split_store2(H, L, (int64_t)nu * ld_row + mu, xa, xb, va, vb);
    tile[y][2 * tx] = xa;
    tile[y][2 * tx + 1] = xb;
  }
  __syncthreads();
  for (int y = ty; y < 32; y += 16) {
    const int row = tm * 32 + y, nu = tv * 32 + 2 * tx;
    const bool va = nu < n && row < nu, vb = nu + 1 < n && row < nu + 1;
    split_store2(H, L, (int64_t)row * ld_row + nu, tile[2 * tx][y], tile[2 * tx + 1][y], va, vb);
  }
}

// full symmetric pair matrix (rows of ld) from the 8-fold packed vector, rounded to FP32 as every slice is before it is
// split: one block per
// 32x32 tile of the lower triangle (row tile >= column tile), read along
// packed rows, written to both triangles through a shared-memory transpose
__global__ void __launch_bounds__(256) expand_packed8_kernel(const double *packed, int64_t np, int64_t ld, float *full) {
  __shared__ float tile[32][33];
  const int64_t tr = blockIdx.y, tcol = blockIdx.x;
  if (tcol > tr) return;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int y = ty; y < 32; y += 8) {
    const int64_t r = tr * 32 + y, c = tcol * 32 + tx;
    float x = 0.0f;
    if (r < np && c <= r) {
      x = (float)packed[r * (r + 1) / 2 + c];
      full[r * ld + c] = x;  // element (c, r): column r, contiguous in c
    }
    tile[y][tx] = x;
  }
  __syncthreads();
  for (int y = ty; y < 32; y += 8) {
    const int64_t c = tcol * 32 + y, r = tr * 32 + tx;
    if (r < np && c < r) full[c * ld + r] = tile[tx][y];  // element (r, c): column c, contiguous in r
  }
}

// ---------------------------------------------------------------------------
// GEMM 1 for BF16 straight from the pair rows: the slices S are not written anywhere.  A CTA keeps its 128 rows of C^T
// (hi and lo, all of K: 128 KB) and takes one slice after another.  16 producer warps read the packed symmetric slice
// (FP32 rows, or a caller's FP64 pair matrix), 16 rows nu each, 32 columns mu a stage: below the diagonal along mu,
// above it along nu, two stages ahead; they split the values and write both parts as K-major
// rows of 64 bytes (64-byte swizzle).  Values, split, K order and the three products of a step are those of
// tc_gemm_kernel, so are the results.  Four warps turn an accumulator into the split U^T, 32 columns at a time through
// swizzled staging that TMA stores (rows (m, slice)), while the MMAs of the next slice fill the other accumulator.
// The pair of CTAs that shares a slice reads it through L2, where one of them prefetches it (one slice ahead): 45 GB of
// requests of 128 unaligned bytes over both halves at 256 AOs are what bounds it (without the loads 5.4 ms less, without
// the split and its stores 1.7, without the TMA stores 0.5).  256 AOs: 24.7 ms with the slices split in memory, 20.2 so,
// 18.6 with the prefetch, 17.7 with two stages of values in flight and batches of 2432 slices; 200 AOs to 160 MOs
// 10.6 -> 6.3, 128 AOs 1.84 -> 1.2, 24 AOs 0.14 -> 0.13.  In TF32 C^T takes twice the room and does not stay in shared
// memory: it keeps the other way.
namespace slices {
constexpr int KC = 32;                        // K of a stage
constexpr int PROD_WARPS = 16, EPI0 = PROD_WARPS, MMA_WARP = EPI0 + EPI_WARPS;
constexpr int THREADS = 32 * (MMA_WARP + 1);
constexpr int A_BYTES = 2 * (BN / 64) * A_TILE;  // [hi, lo][block of 64 k][128 rows]
constexpr int B_HALF = BN * KC * 2;              // 16 KB: hi or lo of a stage
constexpr int NSTAGE = 2;
constexpr int STG = 32 * KC * 2;                 // 2 KB: 32 rows x 32 columns of one part
constexpr int SMEM = A_BYTES + NSTAGE * 2 * B_HALF + EPI_WARPS * 2 * 2 * STG + 1024 + 256;
static_assert(SMEM <= 227 * 1024, "shared memory");

struct Args {
  int n, nm, m_tiles, nslices;  // slices of this launch
  int64_t ld;                   // source row length
  const void *src;              // first slice
  long long wait_cycles;
  int *err;
};

__device__ __forceinline__ void tma_store_3d(const CUtensorMap *map, uint32_t src, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(src), "r"(x), "r"(y), "r"(z)
               : "memory");
}
__device__ __forceinline__ void split2(float a, float b, uint32_t &h, uint32_t &l) {
  const __nv_bfloat162 hh = __floats2bfloat162_rn(a, b);
  const __nv_bfloat162 ll = __floats2bfloat162_rn(a - __low2float(hh), b - __high2float(hh));
  h = *reinterpret_cast<const uint32_t *>(&hh);
  l = *reinterpret_cast<const uint32_t *>(&ll);
}

// 16 rows nu0 .. of the slice and 32 columns mu0 ..; over: the whole block is above the diagonal.
// Below or on it lane = mu and v[r] = S[nu0 + r][mu]; above it lane = (half of mu, row) and v[k] = S[nu][mu of the half + k]
template <typename TS>
__device__ __forceinline__ void load16(const TS *s, int n, int nu0, int mu0, bool over, int lane, float (&v)[16]) {
  if (over) {
    const int nu = nu0 + (lane & 15), m0 = mu0 + (lane & 16);
    int o = m0 * (m0 + 1) / 2 + nu;
#pragma unroll
    for (int k = 0; k < 16; k++) {
      v[k] = m0 + k < n ? (float)s[o] : 0.0f;  // nu < m0
      o += m0 + k + 1;
    }
  } else {
    const int mu = mu0 + lane;
    const int up = mu * (mu + 1) / 2;
    int row = nu0 * (nu0 + 1) / 2;
#pragma unroll
    for (int r = 0; r < 16; r++) {
      const int nu = nu0 + r;
      v[r] = nu < n && mu < n ? (float)s[mu <= nu ? row + mu : up + nu] : 0.0f;
      row += nu + 1;
    }
  }
}
__device__ __forceinline__ void store16(unsigned char *hi, int nu0, bool over, int lane, const float (&v)[16]) {
  unsigned char *lo = hi + B_HALF;
  if (over) {
    const int r = nu0 + (lane & 15), c = (lane & 16) >> 3;  // 16-byte chunks c, c + 1 of the row
#pragma unroll
    for (int q = 0; q < 2; q++) {
      uint4 h, l;
      split2(v[8 * q], v[8 * q + 1], h.x, l.x);
      split2(v[8 * q + 2], v[8 * q + 3], h.y, l.y);
      split2(v[8 * q + 4], v[8 * q + 5], h.z, l.z);
      split2(v[8 * q + 6], v[8 * q + 7], h.w, l.w);
      const int o = r * 64 + (((c + q) ^ ((r >> 1) & 3)) << 4);
      *reinterpret_cast<uint4 *>(hi + o) = h;
      *reinterpret_cast<uint4 *>(lo + o) = l;
    }
  } else {
    // lanes exchange in pairs: the even one packs (mu, mu + 1) of row 2 k, the odd one (mu - 1, mu) of row 2 k + 1
    const int odd = lane & 1, c = lane >> 3, w = (lane >> 1) & 3;
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const float mine = odd ? v[2 * k + 1] : v[2 * k];
      const float got = __shfl_xor_sync(0xffffffffu, odd ? v[2 * k] : v[2 * k + 1], 1);
      uint32_t h, l;
      split2(odd ? got : mine, odd ? mine : got, h, l);
      const int r = nu0 + 2 * k + odd;
      const int o = r * 64 + ((c ^ ((r >> 1) & 3)) << 4) + w * 4;
      *reinterpret_cast<uint32_t *>(hi + o) = h;
      *reinterpret_cast<uint32_t *>(lo + o) = l;
    }
  }
}

template <typename TS>
__global__ void __launch_bounds__(THREADS, 1)
    slice_gemm_kernel(const __grid_constant__ CUtensorMap tmA_hi, const __grid_constant__ CUtensorMap tmA_lo,
                      const __grid_constant__ CUtensorMap tmU_hi, const __grid_constant__ CUtensorMap tmU_lo, Args g) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  unsigned char *smB = smem + A_BYTES, *smE = smB + NSTAGE * 2 * B_HALF;
  uint64_t *bars = reinterpret_cast<uint64_t *>(smE + EPI_WARPS * 2 * 2 * STG);
  uint64_t *afull = bars, *full = bars + 1, *empty = full + NSTAGE, *accf = empty + NSTAGE, *acce = accf + 2,
           *drain = acce + 2;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drain + 1);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nst = (g.n + KC - 1) / KC, cols = (g.n + 15) / 16 * 16;
  const int mt = blockIdx.x % g.m_tiles, first = blockIdx.x / g.m_tiles, step = gridDim.x / g.m_tiles;

  if (threadIdx.x == 0) {
    mbar_init(smem_u32(afull), 1);
    for (int i = 0; i < NSTAGE; i++) {
      mbar_init(smem_u32(full + i), PROD_WARPS);
      mbar_init(smem_u32(empty + i), 1);
    }
    for (int a = 0; a < 2; a++) {
      mbar_init(smem_u32(accf + a), 1);
      mbar_init(smem_u32(acce + a), EPI_WARPS);
    }
    mbar_init(smem_u32(drain), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(2 * BN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  if (warp < PROD_WARPS) {
    // ---- producers: 16 rows each, two stages of values in registers
    const int nu0 = warp * 16;
    const bool mine = nu0 < g.n;
    const TS *src = static_cast<const TS *>(g.src);
    float v0[16], v1[16];
    int lb = first, ls = 0;  // the next values to load
    auto load = [&](float (&v)[16]) {
      if (lb < g.nslices) {
        if (mine) load16(src + lb * g.ld, g.n, nu0, ls * KC, nu0 + 16 <= ls * KC, lane, v);
        if (++ls == nst) ls = 0, lb += step;
      }
    };
    // FP32 rows start at multiples of 128 bytes; a bulk prefetch takes multiples of 16
    const uint32_t pf = sizeof(TS) == 4 && threadIdx.x == 0 && mt == 0 ? (uint32_t)(g.n * (g.n + 1) / 2 * 4) & ~15u : 0u;
    int b = first, s = 0, it = 0;
    // write a stage from v, then fill v for the stage after the next: no register is waited for before it is used
    auto stage = [&](float (&v)[16]) {
      // the slice after this one into L2, once for the tiles that share it
      if (pf && s == 0 && b + step < g.nslices)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src + (b + step) * g.ld), "r"(pf) : "memory");
      const int slot = it % NSTAGE;
      const bool ok = warp_wait(smem_u32(empty + slot), (uint32_t)((it / NSTAGE) & 1) ^ 1u, g.wait_cycles);
      if (!ok || warp_aborted(abort_flag)) {
        if (!ok && lane == 0) atomicCAS(g.err, 0, ERR_TIMEOUT_MMA);
        *abort_flag = 1;
        return false;
      }
      if (mine) store16(smB + slot * 2 * B_HALF, nu0, nu0 + 16 <= s * KC, lane, v);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(full + slot));
      load(v);
      if (++s == nst) s = 0, b += step;
      it++;
      return true;
    };
    load(v0);
    load(v1);
    while (b < g.nslices && stage(v0) && b < g.nslices && stage(v1)) {
    }
  } else if (warp == MMA_WARP) {
    if (lane == 0) {
      mbar_expect_tx(smem_u32(afull), (uint32_t)(2 * ((g.n + 63) / 64) * A_TILE));
      for (int k = 0; k * 64 < g.n; k++) {
        tma_load_2d(smem_u32(smem + k * A_TILE), &tmA_hi, k * 64, mt * BM, smem_u32(afull));
        tma_load_2d(smem_u32(smem + A_BYTES / 2 + k * A_TILE), &tmA_lo, k * 64, mt * BM, smem_u32(afull));
      }
      if (!mbar_wait(smem_u32(afull), 0, g.wait_cycles)) {
        atomicCAS(g.err, 0, ERR_TIMEOUT_FULL);
        *abort_flag = 1;
      }
      const uint32_t idesc = instr_desc(1u, cols);
      int it = 0, i = 0;
      for (int b = first; b < g.nslices && !*abort_flag; b += step, i++) {
        const int a = i & 1;
        if (!mbar_wait(smem_u32(acce + a), (uint32_t)((i >> 1) & 1) ^ 1u, g.wait_cycles)) {
          atomicCAS(g.err, 0, ERR_TIMEOUT_ACC);
          *abort_flag = 1;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t d = tmem + (uint32_t)(a * BN);
        bool ok = true;
        for (int s = 0; s < nst; s++, it++) {
          const int slot = it % NSTAGE;
          if (!mbar_wait(smem_u32(full + slot), (uint32_t)((it / NSTAGE) & 1), g.wait_cycles)) {
            atomicCAS(g.err, 0, ERR_TIMEOUT_FULL);
            *abort_flag = 1;
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a_hi = smem_u32(smem + (s >> 1) * A_TILE) + (s & 1) * 64, a_lo = a_hi + A_BYTES / 2;
          const uint32_t b_hi = smem_u32(smB + slot * 2 * B_HALF), b_lo = b_hi + B_HALF;
#pragma unroll
          for (int kk = 0; kk < KC / 16; kk++) {
            const uint32_t o = kk * 32;
            mma<false>(d, smem_desc(a_hi + o), smem_desc_k64(b_hi + o), idesc, s > 0 || kk > 0);
            mma<false>(d, smem_desc(a_hi + o), smem_desc_k64(b_lo + o), idesc, 1u);
            mma<false>(d, smem_desc(a_lo + o), smem_desc_k64(b_hi + o), idesc, 1u);
          }
          mma_commit(smem_u32(empty + slot));
        }
        if (!ok) break;
        mma_commit(smem_u32(accf + a));
      }
      // no load or MMA of this CTA is in flight when it leaves
      mma_commit(smem_u32(drain));
      mbar_wait(smem_u32(drain), 0, WAIT_CYCLES);
      mbar_wait(smem_u32(afull), 0, WAIT_CYCLES);
    }
  } else {
    // ---- epilogue
    const int q = warp & 3;
    unsigned char *stg = smE + (warp - EPI0) * 2 * 2 * STG;
    const int m0 = mt * BM + q * 32;
    int i = 0, buf = 0;
    for (int b = first; b < g.nslices; b += step, i++) {
      const int a = i & 1;
      const bool ok = warp_wait(smem_u32(accf + a), (uint32_t)((i >> 1) & 1), g.wait_cycles);
      if (!ok || warp_aborted(abort_flag)) {
        if (!ok && lane == 0) atomicCAS(g.err, 0, ERR_TIMEOUT_ACC);
        *abort_flag = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (m0 < g.nm) {
        for (int c0 = 0; c0 < g.n; c0 += KC, buf ^= 1) {
          float x[32];
          tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(a * BN + c0), x);
          unsigned char *hi = stg + buf * 2 * STG, *lo = hi + STG;
          // the stores that last read this buffer are through with it
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
          __syncwarp();
#pragma unroll
          for (int c = 0; c < 4; c++) {
            uint4 h, l;
            split2(x[8 * c], x[8 * c + 1], h.x, l.x);
            split2(x[8 * c + 2], x[8 * c + 3], h.y, l.y);
            split2(x[8 * c + 4], x[8 * c + 5], h.z, l.z);
            split2(x[8 * c + 6], x[8 * c + 7], h.w, l.w);
            const int o = lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4);
            *reinterpret_cast<uint4 *>(hi + o) = h;
            *reinterpret_cast<uint4 *>(lo + o) = l;
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) {
            tma_store_3d(&tmU_hi, smem_u32(hi), c0, b, m0);
            tma_store_3d(&tmU_lo, smem_u32(lo), c0, b, m0);
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(acce + a));
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == MMA_WARP)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * BN) : "memory");
}
}  // namespace slices

}  // namespace tc

// ---------------------------------------------------------------------------
// budget of the GEMM pipeline waits; pq_debug_set_wait_budget changes it for tests of the timeout path
static long long g_gemm_wait_cycles = tcx::WAIT_CYCLES;

// 2-D tensor map over a row-major (rows x kdim) operand, box (BK x box_rows), 128-byte swizzle
static pq_status make_map(CUtensorMap *m, const void *base, bool tf32, int64_t rows, int64_t kdim, int64_t ld,
                          int box_rows) {
  auto fn = tcx::encode_fn();
  if (!fn) {
    set_error("cuTensorMapEncodeTiled is not available from the driver");
    return PQ_ERR_CUDA;
  }
  const int esz = tf32 ? 4 : 2;
  cuuint64_t dims[2] = {(cuuint64_t)kdim, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)(ld * esz)};
  cuuint32_t box[2] = {(cuuint32_t)(tc::ROW_BYTES / esz), (cuuint32_t)box_rows};
  cuuint32_t es[2] = {1, 1};
  CUresult r = fn(m, tf32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base),
                  dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed (%d): rows=%lld k=%lld ld=%lld", (int)r, (long long)rows, (long long)kdim,
              (long long)ld);
    return PQ_ERR_CUDA;
  }
  return PQ_OK;
}

struct Operand {
  const void *hi, *lo;
  int64_t rows;  // total rows in memory
  int64_t ld;    // row length in elements
};

// EPI_SPLIT: U^T of nbatch slices (A = C^T, B = the slices); EPI_PACK: M = n_mo * nbp rows of U^T times C
template <bool TF32, int EPI, typename TO>
static pq_status run_gemm(const Operand &A, const Operand &B, int M, int N, int K, int nbatch, const tc::GemmArgs &gin,
                          cudaStream_t st) {
  CUtensorMap ma_hi, ma_lo, mb_hi, mb_lo;
  PQ_TRY(make_map(&ma_hi, A.hi, TF32, A.rows, K, A.ld, tc::BM));
  PQ_TRY(make_map(&ma_lo, A.lo, TF32, A.rows, K, A.ld, tc::BM));
  PQ_TRY(make_map(&mb_hi, B.hi, TF32, B.rows, K, B.ld, tc::B_BOX));
  PQ_TRY(make_map(&mb_lo, B.lo, TF32, B.rows, K, B.ld, tc::B_BOX));
  tc::GemmArgs g = gin;
  g.M = M;
  g.N = N;
  g.K = K;
  g.m_tiles = (M + tc::BM - 1) / tc::BM;
  g.b_rows = N;
  g.nbatch = nbatch;
  g.wait_cycles = g_gemm_wait_cycles;
  auto kern = tc::tc_gemm_kernel<TF32, EPI, TO>;
  PQ_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, tc::SMEM_BYTES));
  int dev = 0, sms = 0;
  PQ_CUDA_TRY(cudaGetDevice(&dev));
  PQ_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int64_t tiles = (int64_t)nbatch * g.m_tiles;
  const int grid = (int)std::min<int64_t>(tiles, sms);  // persistent: one CTA per SM
  kern<<<grid, tc::GEMM_THREADS, tc::SMEM_BYTES, st>>>(ma_hi, ma_lo, mb_hi, mb_lo, g);
  PQ_CUDA_TRY(cudaGetLastError());
  return PQ_OK;
}

// GEMM 1 of nb slices (BF16) from their pair rows src (FP32 or FP64, ld apart)
template <typename TS>
static pq_status run_slices(const Operand &ct, void *uh, void *ul, const TS *src, int64_t ld_src, int n, int nm, int nb,
                            int nbp, int64_t ld, int *err, cudaStream_t st) {
  auto fn = tcx::encode_fn();
  CUtensorMap ma[2], mu[2];
  PQ_TRY(make_map(&ma[0], ct.hi, false, ct.rows, n, ct.ld, tc::BM));
  PQ_TRY(make_map(&ma[1], ct.lo, false, ct.rows, n, ct.ld, tc::BM));
  for (int k = 0; k < 2; k++) {
    cuuint64_t dims[3] = {(cuuint64_t)n, (cuuint64_t)nb, (cuuint64_t)nm};
    cuuint64_t strides[2] = {(cuuint64_t)(2 * ld), (cuuint64_t)(2 * ld * nbp)};
    cuuint32_t box[3] = {(cuuint32_t)tc::slices::KC, 1, 32}, es[3] = {1, 1, 1};
    CUresult r = fn(&mu[k], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, k ? ul : uh, dims, strides, box, es,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
      set_error("cuTensorMapEncodeTiled failed (%d): U^T of %d x %d, %d slices", (int)r, nm, n, nb);
      return PQ_ERR_CUDA;
    }
  }
  tc::slices::Args g{n, nm, (nm + tc::BM - 1) / tc::BM, nb, ld_src, src, g_gemm_wait_cycles, err};
  auto kern = tc::slices::slice_gemm_kernel<TS>;
  PQ_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, tc::slices::SMEM));
  int dev = 0, sms = 0;
  PQ_CUDA_TRY(cudaGetDevice(&dev));
  PQ_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int groups = std::min(nb, std::max(1, sms / g.m_tiles));
  kern<<<groups * g.m_tiles, tc::slices::THREADS, tc::slices::SMEM, st>>>(ma[0], ma[1], mu[0], mu[1], g);
  PQ_CUDA_TRY(cudaGetLastError());
  return PQ_OK;
}

// Work buffers of the split-precision transform, kept per device between calls (grow-only) so that repeated
// transforms allocate nothing; calls on one device are serialised by the mutex (they share the buffers, and
// each call synchronises its stream before it returns).  pq_ao2mo_release_workspace frees them.
struct Ao2moWorkspace {
  DevBuf full, cth, ctl, sh, sl, uh, ul, H1, err;
  Ao2moF64 f64;
  void release() {
    for (DevBuf *b : {&full, &cth, &ctl, &sh, &sl, &uh, &ul, &H1, &err}) b->release();
    f64.release();
  }
  size_t bytes() const {
    size_t n = f64.bytes();
    for (const DevBuf *b : {&full, &cth, &ctl, &sh, &sl, &uh, &ul, &H1, &err}) n += b->bytes;
    return n;
  }
};
static std::mutex g_ws_mu;
static Ao2moWorkspace g_ws[64];
static thread_local bool t_transform = false;  // this thread is inside a transform and holds the lock
struct WorkspaceLock {
  std::lock_guard<std::mutex> lock{g_ws_mu};
  cudaStream_t st;
  explicit WorkspaceLock(cudaStream_t s) : st(s) { t_transform = true; }
  ~WorkspaceLock() {
    cudaStreamSynchronize(st);  // also after an error, with kernels under way: the next call may be on another stream
    t_transform = false;
  }
};

// For an allocation that did not fit: frees this device's buffers between transforms; whether there were any.
bool ao2mo_give_back() {
  if (t_transform) return false;
  std::unique_lock<std::mutex> lock(g_ws_mu, std::try_to_lock);
  int dev = 0;
  if (!lock || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || g_ws[dev].bytes() == 0) return false;
  g_ws[dev].release();
  return true;
}

long long ao2mo_wait_cycles() { return g_gemm_wait_cycles; }

// FP64 mode through the shared workspace.  A device that is too full for it gives the buffers of earlier calls back
// and tries once more.
pq_status ao2mo_f64_shared(const double *eri_ao, int layout, int64_t n_ao_a, int64_t n_ao_b, const double *Ca, int64_t lda,
                           int64_t nmo_a, const double *Cb, int64_t ldb, int64_t nmo_b, double *eri_mo, cudaStream_t st) {
  int dev = 0;
  PQ_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) {
    set_error("pq_ao2mo: device ordinal %d out of range", dev);
    return PQ_ERR_STATE;
  }
  WorkspaceLock lock(st);
  auto run = [&] {
    return ao2mo_f64(g_ws[dev].f64, eri_ao, layout, n_ao_a, n_ao_b, Ca, lda, nmo_a, Cb, ldb, nmo_b, eri_mo, st);
  };
  pq_status s = run();
  if (s == PQ_ERR_OOM) {
    PQ_CUDA_TRY(cudaStreamSynchronize(st));
    g_ws[dev].release();
    cudaGetLastError();
    s = run();
    if (s == PQ_OK) clear_error();
  }
  return s;
}

template <bool TF32>
static pq_status ao2mo_tc_impl(const double *eri_ao, int layout, int64_t n, const double *C, int64_t ldc, int64_t nm,
                               double *eri_mo, cudaStream_t st) {
  using E = typename tc::Split<TF32>::T;
  const int64_t npa = n * (n + 1) / 2, npm = nm * (nm + 1) / 2;
  const int ld = (int)((n + 7) / 8 * 8);    // AO row length (16-byte rows for TMA)
  int dev = 0;
  PQ_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) {
    set_error("pq_ao2mo: device ordinal %d out of range", dev);
    return PQ_ERR_STATE;
  }
  WorkspaceLock lock(st);
  Ao2moWorkspace &w = g_ws[dev];
  DevBuf &full = w.full, &cth = w.cth, &ctl = w.ctl, &sh = w.sh, &sl = w.sl, &uh = w.uh, &ul = w.ul, &H1 = w.H1,
         &err = w.err;
  const double *pairs = eri_ao;
  const float *pairs32 = nullptr;
  const int64_t ld1 = (npa + 31) / 32 * 32;  // AO pairs in a row of the FP32 pair matrices
  if (layout == PQ_AO_PACKED8) {
    PQ_TRY(full.ensure(sizeof(float) * npa * ld1));
    const unsigned nt = (unsigned)((npa + 31) / 32);
    if (nt > 65535) {
      set_error("ao2mo: too many pairs for the expansion grid");
      return PQ_ERR_ARG;
    }
    tc::expand_packed8_kernel<<<dim3(nt, nt), 256, 0, st>>>(eri_ao, npa, ld1, full.as<float>());
    PQ_CUDA_TRY(cudaGetLastError());
    pairs = nullptr;
    pairs32 = full.as<float>();
  }
  PQ_TRY(err.ensure(sizeof(int)));
  PQ_CUDA_TRY(cudaMemsetAsync(err.ptr, 0, sizeof(int), st));
  // C^T split, rows = MO, row length ld (AO)
  PQ_TRY(cth.ensure(sizeof(E) * nm * ld));
  PQ_TRY(ctl.ensure(sizeof(E) * nm * ld));
  tc::split_ct_kernel<TF32><<<(unsigned)((nm * ld + 255) / 256), 256, 0, st>>>(C, ldc, (int)n, (int)nm, ld, cth.as<E>(),
                                                                               ctl.as<E>());
  PQ_CUDA_TRY(cudaGetLastError());
  // slices per batch: S (n x ld) and U^T (nm x ld) in hi/lo
  // (BF16x3, 256 AOs: 19.9 ms with 608 slices in a batch, 18.6 with 1216, 17.9 with 2432, 18.1 with 4864; 128 AOs:
  // 1.48 / 1.26 / 1.18 / 1.11; TF32x3, 200 AOs: 14.1 with 1216, 14.5 with 4096)
  const int64_t bt = std::min<int64_t>(npa, 2432), btp = (bt + 31) / 32 * 32;
  if (TF32) {
    PQ_TRY(sh.ensure(sizeof(E) * bt * n * ld));
    PQ_TRY(sl.ensure(sizeof(E) * bt * n * ld));
  }
  PQ_TRY(uh.ensure(sizeof(E) * btp * nm * ld));
  PQ_TRY(ul.ensure(sizeof(E) * btp * nm * ld));
  PQ_TRY(H1.ensure(sizeof(float) * npm * ld1));
  tc::GemmArgs g{};
  g.err = err.as<int>();
  Operand ct{cth.ptr, ctl.ptr, nm, ld};
  auto half = [&](auto *out, const double *src64, const float *src32, int64_t ld_src, int64_t nslices,
                  int64_t ld_out) -> pq_status {
    using TO = std::remove_pointer_t<decltype(out)>;
    for (int64_t b0 = 0; b0 < nslices; b0 += bt) {
      const int nb = (int)std::min(bt, nslices - b0);
      tc::GemmArgs gb = g;
      gb.nb = nb;
      gb.nbp = (nb + 31) / 32 * 32;
      // GEMM 1: U^T[b] (nm x n) = Ct (nm x n) . S[b]^T, K = n, row (m, b)
      if constexpr (!TF32) {
        if (src64) {
          PQ_TRY(run_slices(ct, uh.ptr, ul.ptr, src64 + b0 * ld_src, ld_src, (int)n, (int)nm, nb, gb.nbp, ld,
                            err.as<int>(), st));
        } else {
          PQ_TRY(run_slices(ct, uh.ptr, ul.ptr, src32 + b0 * ld_src, ld_src, (int)n, (int)nm, nb, gb.nbp, ld,
                            err.as<int>(), st));
        }
      } else {
        const unsigned ntile = (unsigned)((n + 31) / 32);
        tc::split_slices_kernel<<<dim3((unsigned)nb, ntile * ntile), 256, 0, st>>>(
            src64, src32, ld_src, (int)n, ld, b0, sh.as<float>(), sl.as<float>());
        PQ_CUDA_TRY(cudaGetLastError());
        Operand S{sh.ptr, sl.ptr, (int64_t)nb * n, ld};
        gb.out_hi = uh.as<float>();
        gb.out_lo = ul.as<float>();
        gb.ld_out = ld;
        PQ_TRY((run_gemm<TF32, tc::EPI_SPLIT, float>(ct, S, (int)nm, (int)n, (int)n, nb, gb, st)));
      }
      // GEMM 2: T (rows (m, b) x nm) = U^T . Ct^T, K = n; the pairs n <= m
      Operand U{uh.ptr, ul.ptr, nm * gb.nbp, ld};
      gb.out_pack = out + b0;
      gb.ld_pack = ld_out;
      PQ_TRY((run_gemm<TF32, tc::EPI_PACK, TO>(U, ct, (int)nm * gb.nbp, (int)nm, (int)n, 1, gb, st)));
    }
    return PQ_OK;
  };
  // half 1 over AO ket pairs: H1[ij][ket]; half 2 over its rows, MO bra pairs: eri_mo[kl][ij]
  PQ_TRY(half(H1.as<float>(), pairs, pairs32, pairs32 ? ld1 : npa, npa, ld1));
  PQ_TRY(half(eri_mo, nullptr, H1.as<float>(), ld1, npm, npm));
  int herr = 0;
  PQ_CUDA_TRY(cudaMemcpyAsync(&herr, err.ptr, sizeof(int), cudaMemcpyDeviceToHost, st));
  PQ_CUDA_TRY(cudaStreamSynchronize(st));
  if (herr) {
    set_error("ao2mo tensor-core GEMM: bounded wait gave up (code %d)", herr);
    return PQ_TIMEOUT;
  }
  return PQ_OK;
}

pq_status ao2mo_tc(const double *eri_ao, int layout, int64_t n_ao, const double *Ca, int64_t lda, int64_t nmo, int mode,
                   double *eri_mo, cudaStream_t st) {
  if (n_ao > tc::BN || nmo > tc::BN) {
    set_error("pq_ao2mo: split-precision modes support n_ao, n_mo <= %d", tc::BN);
    return PQ_ERR_ARG;
  }
  if (mode == PQ_XFORM_BF16X3) return ao2mo_tc_impl<false>(eri_ao, layout, n_ao, Ca, lda, nmo, eri_mo, st);
  return ao2mo_tc_impl<true>(eri_ao, layout, n_ao, Ca, lda, nmo, eri_mo, st);
}

}  // namespace pq

extern "C" pq_status pq_ao2mo_release_workspace(void) {
  std::lock_guard<std::mutex> lock(pq::g_ws_mu);
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    pq::set_error("pq_ao2mo_release_workspace: no current device");
    return PQ_ERR_STATE;
  }
  pq::g_ws[dev].release();
  return PQ_OK;
}

extern "C" pq_status pq_debug_set_wait_budget(long long cycles) {
  pq::g_gemm_wait_cycles = cycles > 0 ? cycles : pq::tcx::WAIT_CYCLES;
  return PQ_OK;
}
