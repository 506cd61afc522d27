// Dense FP64 products of a CI Hamiltonian by exact digit products (digits9) on the tensor cores: the GEMM of the
// same-spin terms of one species (ci_sigma64.cu) and of the pair matrices of two (ci_two64.cu).
#pragma once
#include "pq_digits.cuh"
#include "pq_internal.h"
#include "pq_tc.cuh"

namespace pq {
namespace s64 {

using namespace tcx;
namespace dg = digits9;

constexpr int KMAX = 80;                     // products of one exact sum
constexpr int BM = 128, BN = 64;             // accumulator tile of one order
constexpr int EPI_WARPS = 16, EPI = 32 * EPI_WARPS;
constexpr int THREADS = 64 + EPI;            // producer warp, MMA warp, epilogue warps
enum { ERR_WAIT = 2 };

// exponent of a plane from the high word of its largest magnitude
__device__ __forceinline__ int plane_exp(const uint32_t *hi) { return digits::exponent_of(__ldg(hi)); }

// The 11 MMAs of one K step of 16: digit i of A times digits 0 .. min(6, 7 - i) of B, which lie `bstep` bytes apart and
// form one operand of up to 256 rows; order l accumulates in columns 64 l.  FIRST: the tile's first step.  bdesc(j)
// and adesc(i) give the descriptors.
template <typename A, typename B>
__device__ __forceinline__ void mma_step(uint32_t tmem, A &&adesc, B &&bdesc, uint32_t major, bool first) {
#pragma unroll
  for (int i = 0; i < dg::N; i++) {
    const int n = (dg::ORDERS - i < dg::N ? dg::ORDERS - i : dg::N);  // digits of B
    if (i == 1 && first) {
      // order 7 begins here, the others were begun by digit 0
      mma_f16(tmem + 64, adesc(1), bdesc(0), idesc_f16(256) | major, 1u);
      mma_f16(tmem + 5 * 64, adesc(1), bdesc(4), idesc_f16(128) | major, 1u);
      mma_f16(tmem + 7 * 64, adesc(1), bdesc(6), idesc_f16(64) | major, 0u);
      continue;
    }
    const uint32_t acc = (first && i == 0) ? 0u : 1u;
    mma_f16(tmem + i * 64, adesc(i), bdesc(0), idesc_f16((n < 4 ? n : 4) * 64) | major, acc);
    if (n > 4) mma_f16(tmem + (i + 4) * 64, adesc(i), bdesc(4), idesc_f16((n - 4) * 64) | major, acc);
  }
}

constexpr int SS_A = BM * 64, SS_B = BN * 64;                  // one digit of 32 K values: 8 KB, 4 KB
constexpr int SS_STAGE = dg::N * (SS_A + SS_B);                // 84 KB
constexpr int SS_STAGES = 2;
constexpr int SS_BARS = 2 * SS_STAGES + 3;
constexpr int SS_SMEM = SS_STAGES * SS_STAGE + SS_BARS * 8 + 64 + 1024;

struct SsArgs {
  int64_t na, nb;
  int nv, m_tiles, n_tiles;   // tiles of 128 beta strings, of 64 alpha strings
  int64_t tiles;
  int win;                    // chunks per exact window
  int64_t per;                // > 0: alpha rows are (root, rest) with this many rows a root, and sigma is stored, not added to
  int ksplit;                 // parts of the K list, each with its own copy of sigma, `part` values apart
  int64_t part;
  int64_t a_plane, b_plane;   // rows of one digit of either operand
  const int32_t *kt_off, *kt_list;  // NULL: every tile has all the chunks
  int chunks;
  const uint32_t *xhi, *dhi;
  double *S;
  int64_t es, vs;
  long long wait;             // budget of the pipeline waits (the wind-down waits keep WAIT_CYCLES)
  int *gate;
};

// Y[v][Ia][Ib] += sum_Ja Ha[Ia][Ja] X[v][Ja][Ib]   (ALPHA: A = planes of C along Ib, B = rows of Ha)
//              or sum_Jb Hb[Ib][Jb] X[v][Ia][Jb]   (A = rows of Hb, B = rows (v, Ia) of C)
// The second form also multiplies the pair matrices of a two-species space (ci_two64.cu), with per > 0.
// Accumulator rows are beta strings, columns alpha strings, so sigma is read and written in whole lines.  The sums of
// a window of K chunks (at most 80 entries of a row of H) are exact; the epilogue adds windows as 96-bit integers.
template <bool ALPHA>
__global__ void __launch_bounds__(THREADS, 1)
    ss64_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, SsArgs g) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + SS_STAGES * SS_STAGE);
  uint64_t *full = bars, *empty = bars + SS_STAGES, *accf = bars + 2 * SS_STAGES, *acce = accf + 1, *drain = accf + 2;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + SS_BARS);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  // A CTA decides once for all its threads whether to start: a CTA of the same launch whose wait runs out raises the gate,
  // so threads that each read it could part ways before the barriers.  Thread 0 reads it, the barrier after the setup
  // tells the others (one of its own before the setup cost 1 us a launch).
  const int gate = threadIdx.x == 0 ? *reinterpret_cast<const volatile int *>(g.gate) : 0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < SS_STAGES; i++) {
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
  if (__syncthreads_or(gate)) {
    if (warp == 0)
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(*tmem_slot), "r"(512) : "memory");
    return;
  }
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  auto fail = [&] {
    *g.gate = ERR_WAIT;
    *abort_flag = 1;
  };
  // tile -> root (or part of the K list), beta tile, alpha tile; the alpha tile varies fastest
  auto tile_of = [&](int64_t t, int &v, int &mt, int &nt) {
    nt = (int)(t % g.n_tiles);
    t /= g.n_tiles;
    mt = (int)(t % g.m_tiles);
    v = (int)(t / g.m_tiles);
  };
  // K list positions of a tile
  auto range_of = [&](int v, int mt, int nt, int &k0, int &k1) {
    const int rt = ALPHA ? nt : mt;
    k0 = g.kt_list ? __ldg(g.kt_off + rt) : 0, k1 = g.kt_list ? __ldg(g.kt_off + rt + 1) : g.chunks;
    if (g.ksplit > 1) {
      const int n = k1 - k0;
      k1 = k0 + (int)((int64_t)n * (v + 1) / g.ksplit);
      k0 += (int)((int64_t)n * v / g.ksplit);
    }
  };
  auto chunk_of = [&](int j) { return g.kt_list ? __ldg(g.kt_list + j) : j; };
  // end of the window that starts at list position j
  auto window_end = [&](int j, int k1) {
    const int w = chunk_of(j) / g.win;
    int e = j + 1;
    while (e < k1 && chunk_of(e) / g.win == w) e++;
    return e;
  };

  if (warp == 0) {
    if (lane == 0) {
      int gs = 0;
      bool ok = true;
      for (int64_t t = blockIdx.x; t < g.tiles && ok; t += gridDim.x) {
        int v, mt, nt;
        tile_of(t, v, mt, nt);
        int k0, k1;
        range_of(v, mt, nt, k0, k1);
        for (int j = k0; j < k1; j++, gs++) {
          const int slot = gs % SS_STAGES;
          ok = mbar_wait(smem_u32(empty + slot), (uint32_t)((gs / SS_STAGES) & 1) ^ 1u, g.wait) && !*abort_flag;
          if (!ok) break;
          const uint32_t a = smem_u32(smem + slot * SS_STAGE), b = a + dg::N * SS_A, bar = smem_u32(full + slot);
          const int k = chunk_of(j) * 32;
          mbar_expect_tx(bar, SS_STAGE);
          for (int d = 0; d < dg::N; d++) {
            if (ALPHA) {
              const int y = (int)(d * g.a_plane + (int64_t)v * g.na) + k;  // rows Ja of the plane
              tma_load_2d(a + d * SS_A, &mapA, mt * BM, y, bar);
              tma_load_2d(a + d * SS_A + SS_A / 2, &mapA, mt * BM + 64, y, bar);
              tma_load_2d(b + d * SS_B, &mapB, k, (int)(d * g.b_plane) + nt * BN, bar);
            } else {
              tma_load_2d(a + d * SS_A, &mapA, k, (int)(d * g.a_plane) + mt * BM, bar);
              tma_load_2d(b + d * SS_B, &mapB, k, (int)(d * g.b_plane + (g.per ? 0 : (int64_t)v * g.na)) + nt * BN, bar);
            }
          }
        }
      }
      if (!ok) fail();
      for (int j = gs > SS_STAGES ? gs - SS_STAGES : 0; j < gs; j++)
        mbar_wait(smem_u32(full + (j % SS_STAGES)), (uint32_t)((j / SS_STAGES) & 1), WAIT_CYCLES);
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      int gs = 0, seq = 0;
      bool ok = true;
      for (int64_t t = blockIdx.x; t < g.tiles && ok; t += gridDim.x) {
        int v, mt, nt;
        tile_of(t, v, mt, nt);
        int k0, k1;
        range_of(v, mt, nt, k0, k1);
        for (int j = k0; j < k1 && ok; seq++) {
          const int e = window_end(j, k1);
          ok = mbar_wait(smem_u32(acce), (uint32_t)(seq & 1) ^ 1u, g.wait) && !*abort_flag;
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          for (int j0 = j; j < e; j++, gs++) {
            const int slot = gs % SS_STAGES;
            ok = mbar_wait(smem_u32(full + slot), (uint32_t)((gs / SS_STAGES) & 1), g.wait);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t a = smem_u32(smem + slot * SS_STAGE), b = a + dg::N * SS_A;
#pragma unroll
            for (int s = 0; s < 2; s++)
              mma_step(
                  tmem,
                  [&](int i) {
                    return ALPHA ? smem_desc_mn(a + i * SS_A + s * 2048, SS_A / 2) : smem_desc_k64(a + i * SS_A + s * 32);
                  },
                  [&](int i) { return smem_desc_k64(b + i * SS_B + s * 32); }, ALPHA ? IDESC_A_MN : 0u, j == j0 && s == 0);
            mma_commit(smem_u32(empty + slot));
          }
          if (ok) mma_commit(smem_u32(accf));
        }
      }
      if (!ok) fail();
      mma_commit(smem_u32(drain));
      mbar_wait(smem_u32(drain), 0, WAIT_CYCLES);
    }
    __syncwarp();
  } else {
    const int q4 = warp & 3, part = (warp - 2) >> 2;
    const uint32_t taddr = tmem + ((uint32_t)(q4 * 32) << 16) + 16 * part;
    int seq = 0;
    bool ok = true;
    const int ed = plane_exp(g.dhi);
    for (int64_t t = blockIdx.x; t < g.tiles && ok; t += gridDim.x) {
      int v, mt, nt;
      tile_of(t, v, mt, nt);
      int k0, k1;
      range_of(v, mt, nt, k0, k1);
      if (k0 == k1 && !g.per) continue;
      // sums of T >> 4 over the windows: 64-bit high part, 32-bit low part
      int64_t sh[16];
      uint32_t sl[16];
#pragma unroll
      for (int c = 0; c < 16; c++) sh[c] = 0, sl[c] = 0;
      for (int j = k0; j < k1; seq++) {
        j = window_end(j, k1);
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(accf), (uint32_t)(seq & 1), g.wait) && !*abort_flag);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int c0 = 0; c0 < 16; c0 += 4) {
          uint32_t a[dg::ORDERS][4];
#pragma unroll
          for (int l = 0; l < dg::ORDERS; l++) tmem_ld4(taddr + l * BN + c0, a[l]);
          tmem_wait();
#pragma unroll
          for (int c = 0; c < 4; c++) {
            float f[dg::ORDERS];
#pragma unroll
            for (int l = 0; l < dg::ORDERS; l++) f[l] = __uint_as_float(a[l][c]);
            int64_t hi, lo;
            dg::combine(f, hi, lo);
            lo >>= 4;
            const uint32_t l32 = (uint32_t)lo, s = sl[c0 + c] + l32;
            sh[c0 + c] += hi + (lo >> 32) + (s < l32);
            sl[c0 + c] = s;
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(acce));
      }
      if (!ok) break;
      const int64_t ib = (int64_t)mt * BM + q4 * 32 + lane;
      if (ib < g.nb)
#pragma unroll
        for (int c = 0; c < 16; c++) {
          const int64_t ia = (int64_t)nt * BN + 16 * part + c;
          if (ia >= g.na) break;
          const int root = g.per ? (int)(ia / g.per) : v;
          const double x = digits::to_double(sh[c], (int64_t)sl[c], plane_exp(g.xhi + root) + ed - 73);  // T counts 2^(e - 4)
          if (g.per) {
            g.S[v * g.part + ia * g.nb + ib] = x;
          } else {
            double *y = g.S + v * g.vs + (ia * g.nb + ib) * g.es;
            *y += x;
          }
        }
    }
    if (!ok && lane == 0) fail();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

static __global__ void __launch_bounds__(256) absmax_kernel(const double *x, int64_t n, uint32_t *hi) {
  uint32_t m = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    m = max(m, (uint32_t)__double2hiint(x[i]) & 0x7fffffffu);
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) atomicMax(hi, m);
}

}  // namespace s64

// FP16 matrix of `rows` rows of `cols` values, ld values apart; reads outside give zeros
inline pq_status s64_map(CUtensorMap *m, const void *base, int64_t rows, int64_t cols, int64_t ld, int box_cols,
                         int box_rows) {
  auto fn = tcx::encode_fn();
  if (!fn) {
    set_error("cuTensorMapEncodeTiled is not available from the driver");
    return PQ_ERR_CUDA;
  }
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * 2};
  cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows}, es[2] = {1, 1};
  const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(base), dims, strides, box, es,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, box_cols == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed (%d): %lld x %lld", (int)r, (long long)rows, (long long)cols);
    return PQ_ERR_CUDA;
  }
  return PQ_OK;
}

inline int64_t up64(int64_t x, int64_t m) { return (x + m - 1) / m * m; }

}  // namespace pq
