// FP64 sigma = H C of one-species full CI on the tcgen05 tensor cores.
//
// Reference: sigma_one_species_class_singleshot (src/ci/detset/direct_singleparticle.cpp:238-372) with the elements
// of slater_condon_singleparticle.cpp:4-175.  The kernel of ci_sigma.cu applies them one by one on the FP64 pipe,
// which this GPU runs at 1/64 of its FP32 rate (1.1 TFLOP/s), and is bound by it.  Here every product is a sum of 34
// exact FP16 digit products (digits9 in pq_digits.cuh), so the FP64 pipe only adds finished sums.
//
// In the full product space, with e_P = E_pq + E_qp (or E_pp) for an orbital pair P, H splits into
//   diagonal      sigma  = (E_alpha + E_beta) C                               same-spin energies of the strings
//   same spin     sigma += H_a C + C H_b^T      dense over the strings: singles (same-spin part) and doubles
//   opposite spin sigma += sum_PQ (P|Q) e_P^alpha C e_Q^beta    alpha-beta doubles, the Coulomb part of the singles
//                                                               and of the diagonal
// x64_digits_kernel splits C once, planes [digit][root][Ia][Ib], and writes the diagonal term.  ss64_kernel is a GEMM
// over those planes for either spin.  ab64_kernel forms, per alpha string Ia and tile of 128 beta strings Jb,
//   D[Jb][Q] = sum_{(Ja, P): e_P Ja = +-Ia} +-(P|Q) C(Ja, Jb)       K = singles and occupied orbitals of Ia
// with both operands fetched by TMA row gathers (rows of C's planes by Ja, signed rows of the integral digits by P),
// and adds the entries of D into sigma(Ia, Ib) along the lists of e_Q; a CTA owns the rows it adds to and their order.  The gathered rows run along Jb and Q, so both
// operands are M- and N-major and nothing is converted or transposed on the way.
//
// Errors.  A sum of digits leaves out less than 2^-64 of K max|C| max|W|.  D goes through shared memory as 64-bit
// integers with one exponent per tile, 55 bits below the tile's largest entry, and sums of its entries are exact.  An
// element-by-element FP64 sum rounds each of its terms at 2^-53 of the partial sum, which holds the diagonal (-147
// C_I at 14 orbitals).
// Against a 64-bit evaluation of the second-quantised form the 2-norm error is 7e-16 at 13 and 14 orbitals, where the
// element kernel's is 2.4e-15 and 2.8e-15.
//
// Non-finite input (or integrals), and a bounded wait that runs out, raise a device flag; the element-by-element
// kernel is launched behind with that flag as its condition and then computes the whole result, as before.
//
// Measured against the element-by-element kernel: four roots of FCI(14o, 7a7b) 51.1 / 345.6 ms (opposite spin 30, same
// spin 2 x 10, digits 0.3), one root of FCI(13o, 6a5b) 1.93 / 17.0 ms, four roots of FCI(12o, 6a6b) 2.7 / 18.2,
// FCI(11o, 5a5b) 0.68 / 2.33, FCI(10o, 5a5b) 0.20 / 0.61 ms.  Bound: the epilogue of the opposite-spin kernel, in clocks
// per tile and pass of FCI(14o): MMAs 5.6 k, which overlap the sums of the entries (4.0 k), then the drain (4.6 k: the
// integer arithmetic of eight orders), which cannot overlap MMAs because eight orders fill TMEM; the drain likewise in
// ss64_kernel.  With one gather warp a tile took 17 k (75 clocks a row gather), with three 11 k.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <numeric>
#include <utility>
#include <vector>

#include "ci_dense64.cuh"
#include "pq_bits.cuh"

namespace pq {

static long long g_sigma_wait[2] = {tcx::WAIT_CYCLES, tcx::WAIT_CYCLES};
long long sigma_wait_cycles(int kernel) { return g_sigma_wait[kernel]; }

struct Sigma64 {
  struct Side {
    unsigned short *d = nullptr;       // digits of the dense same-spin H: [digit][I][np]
    int64_t n = 0, np = 0;             // strings, row length
    int32_t *kt_off = nullptr, *kt_list = nullptr;  // K chunks of 32 with an entry, per row tile (64 rows alpha, 128 beta)
    int win = 2;                       // chunks of a window that holds at most 80 entries of a row
  };
  Side side[2];
  unsigned short *w = nullptr;         // digits of (P|Q): [digit][2 P + sign; a zero row last][pass x 64]
  int2 *klist = nullptr;               // per alpha string kp x {row of C, row of w}
  int kp = 0, npass = 1, wq = 0;
  int32_t *toff = nullptr;             // scatter lists per (pass, beta tile)
  int4 *tent = nullptr;
  uint32_t *hi = nullptr;              // high words of max|.|: same-spin H alpha, beta, integrals
  int *aux = nullptr;                  // gate; high words of max|C| per root from word 4 on
  DevBuf mem, lists, xd;               // matrices and words; the chunk and scatter lists; digits of C
  int sms = 0;
  size_t bytes() const { return mem.bytes + lists.bytes + xd.bytes; }
};
void sigma64_delete(Sigma64 *s) { delete s; }

namespace s64 {

// ---------------------------------------------------------------------------------------------- digits of C

__global__ void __launch_bounds__(256) x64_absmax_kernel(const double *C, int64_t es, int64_t vs, int64_t n, uint32_t *hi) {
  const double *c = C + (int64_t)blockIdx.y * vs;
  uint32_t m = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    m = max(m, (uint32_t)__double2hiint(c[i * es]) & 0x7fffffffu);
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) atomicMax(hi + blockIdx.y, m);
}

// planes [digit][v][Ia][nbp] of nv vectors and S = (E_alpha + E_beta - shift) C; block per (alpha string, root).
// Vector v of determinant I lies at C[I es + v vs], of sigma at S[I ses + v svs].
__global__ void __launch_bounds__(256) x64_digits_kernel(const double *C, int64_t es, int64_t vs, int64_t na, int64_t nb, int64_t nbp,
                                                        int nv, const uint32_t *xhi, const uint32_t *hi,
                                                        const double *ea, const double *eb, double shift,
                                                        unsigned short *xd, double *S, int64_t ses, int64_t svs, int *gate) {
  const int64_t ia = blockIdx.x;
  const int v = blockIdx.y;
  const int e = plane_exp(xhi + v);
  if (e == digits::BAD || plane_exp(hi) == digits::BAD || plane_exp(hi + 1) == digits::BAD || plane_exp(hi + 2) == digits::BAD) {
    if (threadIdx.x == 0) *gate = 1;
    return;
  }
  const double *c = C + v * vs + ia * nb * es;
  double *s = S + v * svs + ia * nb * ses;
  const double da = ea[ia] - shift;
  const int64_t plane = (int64_t)nv * na * nbp;
  unsigned short *row = xd + ((int64_t)v * na + ia) * nbp;
  for (int64_t b = 2 * threadIdx.x; b < nb; b += 2 * blockDim.x) {
    const double x0 = c[b * es], x1 = b + 1 < nb ? c[(b + 1) * es] : 0.0;
    unsigned short d0[dg::N], d1[dg::N];
    dg::to_half(digits::fixed_point<dg::BITS>(x0, e), d0);
    dg::to_half(digits::fixed_point<dg::BITS>(x1, e), d1);
#pragma unroll
    for (int i = 0; i < dg::N; i++) *reinterpret_cast<ushort2 *>(row + i * plane + b) = make_ushort2(d0[i], d1[i]);
    s[b * ses] = (da + eb[b]) * x0;
    if (b + 1 < nb) s[(b + 1) * ses] = (da + eb[b + 1]) * x1;
  }
}

// ---------------------------------------------------------------------------------------------- opposite spin

constexpr int A_DIGIT = BM * 16 * 2;                // 4 KB: one digit of 128 beta strings x 16 K values
constexpr int A_STAGE = dg::N * A_DIGIT;            // 28 KB
constexpr int A_STAGES = 3;
constexpr int B_BYTES = dg::N * KMAX * 128;         // 70 KB: all digits of 64 pairs x K
constexpr int LDS_D = BN + 1;                       // row length of the staged D
constexpr int D_BYTES = BM * LDS_D * 8;             // 65 KB
constexpr int AB_BARS = 2 * A_STAGES + 9;
constexpr int GATHER_WARPS = 3;                     // warp 0 and the last two
constexpr int AB_THREADS = 32 * (GATHER_WARPS + 1 + EPI_WARPS);
constexpr int AB_SMEM = A_STAGES * A_STAGE + B_BYTES + D_BYTES + GATHER_WARPS * KMAX * 8 + AB_BARS * 8 + 64 + 1024;
static_assert(AB_SMEM <= 232448, "shared memory per CTA");

struct AbArgs {
  int64_t na, nb, items;
  int nv, vsplit;            // vsplit: an item is one root of an alpha string, else all of them
  int npass, wq, kp, wrows;  // wrows: rows of one digit of w
  int m_tiles;
  const int2 *klist;
  const int32_t *toff;
  const int4 *tent;
  const uint32_t *xhi, *whi;
  double *S;
  int64_t es, vs;            // strides of sigma over determinants and roots
  long long wait;            // budget of the pipeline waits (the wind-down waits keep WAIT_CYCLES)
  int *gate;
};

// sum 2^e for an integer, rounded once or twice (outside the normal range)
__device__ __forceinline__ double pow2_scale(int e) {
  return e > -1022 && e < 1023 ? __hiloint2double((e + 1023) << 20, 0) : scalbn(1.0, e);
}

constexpr int ZERO_SLOT = BN, ZERO2 = ZERO_SLOT | ZERO_SLOT << 16;  // D[0][64], which stays zero
constexpr int NPRE = 3;  // list entries per epilogue thread loaded ahead of a tile

// Roles: warp 0 and the last two gather (their lanes share the row gathers of a stage; one warp
// issues a gather in about 75 clocks), warp 1 lane 0 issues MMAs, warps 2 .. 17 drain
// and scatter.  Per tile the epilogue finds the largest |D| from the four leading orders, so that the tile's entries
// become 56-bit integers; stages them; releases the accumulators; and sums the entries of each target.  Every wait is
// an mbarrier wait with a budget; one that runs out raises the gate and the CTA winds down.
__global__ void __launch_bounds__(AB_THREADS, 1)
    ab64_kernel(const __grid_constant__ CUtensorMap mapX, const __grid_constant__ CUtensorMap mapW, AbArgs g) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  unsigned char *sa = smem, *sb = sa + A_STAGES * A_STAGE;
  int64_t *sd = reinterpret_cast<int64_t *>(sb + B_BYTES);
  int2 *kl_all = reinterpret_cast<int2 *>(reinterpret_cast<unsigned char *>(sd) + D_BYTES);
  uint64_t *bars = reinterpret_cast<uint64_t *>(kl_all + GATHER_WARPS * KMAX);
  uint64_t *a_full = bars, *a_empty = bars + A_STAGES, *b_full = bars + 2 * A_STAGES, *b_empty = b_full + 1;
  uint64_t *acc_full = b_full + 2, *acc_empty = b_full + 3, *max_full = b_full + 4, *d_full = b_full + 5, *d_empty = b_full + 6;
  uint64_t *drain = b_full + 7;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + AB_BARS);
  uint32_t *tmax = tmem_slot + 1;  // [2]
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 3);
  volatile int *issued = abort_flag + 1;  // at the end: stages and items that each gather warp has issued
  // one decision for the CTA, as in ss64_kernel; before the setup and from every thread's word, since the kernel took 0.1 -
  // 0.9 % longer in the other forms (51.27 ms of FCI(14o) sigma, four roots, against 51.09 without an agreement)
  if (__syncthreads_count(*g.gate)) return;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < A_STAGES; i++) {
      mbar_init(smem_u32(a_full + i), GATHER_WARPS);
      mbar_init(smem_u32(a_empty + i), 1);
    }
    mbar_init(smem_u32(b_full), GATHER_WARPS);
    mbar_init(smem_u32(b_empty), 1);
    mbar_init(smem_u32(acc_full), 1);
    mbar_init(smem_u32(acc_empty), EPI_WARPS);
    mbar_init(smem_u32(max_full), EPI_WARPS);
    mbar_init(smem_u32(d_full), EPI_WARPS);
    mbar_init(smem_u32(d_empty), EPI_WARPS);
    mbar_init(smem_u32(drain), 1);
    tmax[0] = tmax[1] = 0;
    sd[ZERO_SLOT] = 0;
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
  const int steps = g.kp / 16;
  auto fail = [&] {
    *g.gate = ERR_WAIT;
    *abort_flag = 1;
  };
  // (item, pass) -> alpha string, pass, roots v0 .. v1 - 1; a CTA runs the passes of an item one after the other, so
  // that it alone adds to those rows of sigma, in a fixed order
  auto item_of = [&](int64_t it, int64_t &ia, int &p, int &v0, int &v1) {
    p = (int)(it % g.npass);
    it = blockIdx.x + (it / g.npass) * gridDim.x;
    v0 = 0, v1 = g.nv;
    if (g.vsplit) {
      v0 = (int)(it % g.nv), v1 = v0 + 1;
      it /= g.nv;
    }
    ia = it;
  };
  const int64_t mine = (int64_t)blockIdx.x < g.items ? ((g.items - 1 - blockIdx.x) / gridDim.x + 1) * g.npass : 0;

  if (warp == 0 || warp >= 2 + EPI_WARPS) {
    // ---- gather warps
    const int pw = warp == 0 ? 0 : warp - (1 + EPI_WARPS);
    int2 *kl = kl_all + pw * KMAX;  // this warp's copy of the item's K list
    int gs = 0, nit = 0;
    bool ok = true;
    // each warp announces the bytes of its own gathers: four rows of 128 bytes each
    auto share = [&](int gathers) { return (uint32_t)((gathers - pw + GATHER_WARPS - 1) / GATHER_WARPS * 512); };
    for (int64_t it = 0; it < mine && ok; it++) {
      int64_t ia;
      int p, v0, v1;
      item_of(it, ia, p, v0, v1);
      __syncwarp();
      for (int k = lane; k < g.kp; k += 32) kl[k] = __ldg(g.klist + ia * g.kp + k);
      __syncwarp();
      ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(b_empty), (uint32_t)(nit & 1) ^ 1u, g.wait)) && !*abort_flag;
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      if (lane == 0) mbar_expect_tx(smem_u32(b_full), share(dg::N * (g.kp / 4)));
      nit++;
      __syncwarp();
      for (int i = GATHER_WARPS * lane + pw; i < dg::N * (g.kp / 4); i += 32 * GATHER_WARPS) {
        const int d = i / (g.kp / 4), k = 4 * (i - d * (g.kp / 4));
        const int r = d * g.wrows;
        tma_gather4(smem_u32(sb) + d * g.kp * 128 + k * 128, &mapW, p * BN, r + kl[k].y, r + kl[k + 1].y, r + kl[k + 2].y,
                    r + kl[k + 3].y, smem_u32(b_full));
      }
      for (int v = v0; v < v1 && ok; v++)
        for (int t = 0; t < g.m_tiles && ok; t++)
          for (int s = 0; s < steps; s++, gs++) {
            const int slot = gs % A_STAGES;
            ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(a_empty + slot), (uint32_t)((gs / A_STAGES) & 1) ^ 1u, g.wait) &&
                                             !*abort_flag);
            if (!ok) break;
            if (lane == 0) mbar_expect_tx(smem_u32(a_full + slot), share(dg::N * 8));
            __syncwarp();
            // 56 gathers: digit, half of the 128 strings, group of four K values
            for (int i = GATHER_WARPS * lane + pw; i < dg::N * 8; i += 32 * GATHER_WARPS) {
              const int d = i >> 3, h = (i >> 2) & 1, k = 4 * (i & 3);
              const int2 *q = kl + 16 * s + k;
              const int y = (int)((int64_t)(d * g.nv + v) * g.na);
              tma_gather4(smem_u32(sa + slot * A_STAGE) + d * A_DIGIT + h * (A_DIGIT / 2) + k * 128, &mapX, t * BM + h * 64,
                          y + q[0].x, y + q[1].x, y + q[2].x, y + q[3].x, smem_u32(a_full + slot));
            }
          }
    }
    // The gathers in flight land before the CTA exits.  A warp that gave up first arrives, without bytes, for the
    // stages and the item that others had gone on to (at most the ring ahead of it), so that their phases complete;
    // the abort flag is up by then, and what is made of such a stage is not used.
    if (lane == 0) {
      if (!ok) fail();
      issued[2 * pw] = gs, issued[2 * pw + 1] = nit;
    }
    __syncwarp();
    asm volatile("bar.sync 1, %0;" ::"n"(32 * GATHER_WARPS) : "memory");
    if (lane == 0) {
      int gmax = 0, nmax = 0;
      for (int w = 0; w < GATHER_WARPS; w++) gmax = max(gmax, issued[2 * w]), nmax = max(nmax, issued[2 * w + 1]);
      for (int j = gs; j < gmax; j++) mbar_arrive(smem_u32(a_full + j % A_STAGES));
      for (int j = nit; j < nmax; j++) mbar_arrive(smem_u32(b_full));
      for (int j = gmax > A_STAGES ? gmax - A_STAGES : 0; j < gmax; j++)
        mbar_wait(smem_u32(a_full + (j % A_STAGES)), (uint32_t)((j / A_STAGES) & 1), WAIT_CYCLES);
      if (nmax > 0) mbar_wait(smem_u32(b_full), (uint32_t)((nmax - 1) & 1), WAIT_CYCLES);
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      int gs = 0, nit = 0, seq = 0;
      bool ok = true;
      for (int64_t it = 0; it < mine && ok; it++, nit++) {
        int64_t ia;
        int p, v0, v1;
        item_of(it, ia, p, v0, v1);
        ok = mbar_wait(smem_u32(b_full), (uint32_t)(nit & 1), g.wait) && !*abort_flag;
        for (int u = 0; u < (v1 - v0) * g.m_tiles && ok; u++, seq++) {
          ok = mbar_wait(smem_u32(acc_empty), (uint32_t)(seq & 1) ^ 1u, g.wait) && !*abort_flag;
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          for (int s = 0; s < steps; s++, gs++) {
            const int slot = gs % A_STAGES;
            ok = mbar_wait(smem_u32(a_full + slot), (uint32_t)((gs / A_STAGES) & 1), g.wait);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t a = smem_u32(sa + slot * A_STAGE), b = smem_u32(sb) + s * 2048;
            const uint32_t bstep = (uint32_t)g.kp * 128;
            mma_step(
                tmem, [&](int i) { return smem_desc_mn(a + i * A_DIGIT, A_DIGIT / 2); },
                [&](int j) { return smem_desc_mn(b + j * bstep, bstep); }, IDESC_A_MN | IDESC_B_MN, s == 0);
            mma_commit(smem_u32(a_empty + slot));
          }
          if (ok) mma_commit(smem_u32(acc_full));
        }
        if (ok) mma_commit(smem_u32(b_empty));
      }
      if (!ok) fail();
      mma_commit(smem_u32(drain));
      mbar_wait(smem_u32(drain), 0, WAIT_CYCLES);
    }
    __syncwarp();
  } else {
    // ---- epilogue
    const int q4 = warp & 3, part = (warp - 2) >> 2, te = threadIdx.x - 64;
    const uint32_t taddr = tmem + ((uint32_t)(q4 * 32) << 16);
    int64_t *drow = sd + (int64_t)(q4 * 32 + lane) * LDS_D;
    auto wait_all = [&](uint64_t *bar, int phase) {
      return __all_sync(0xffffffffu, mbar_wait(smem_u32(bar), (uint32_t)(phase & 1), g.wait) && !*abort_flag);
    };
    int seq = 0;
    bool ok = true;
    const int ew = plane_exp(g.whi);
    for (int64_t it = 0; it < mine && ok; it++) {
      int64_t ia;
      int p, v0, v1;
      item_of(it, ia, p, v0, v1);
      for (int v = v0; v < v1 && ok; v++) {
        const int ex = plane_exp(g.xhi + v);
        double *srow = g.S + v * g.vs + ia * g.nb * g.es;
        for (int t = 0; t < g.m_tiles; t++, seq++) {
          const int tl = p * g.m_tiles + t, k0 = __ldg(g.toff + tl), k1 = __ldg(g.toff + tl + 1);
          // this thread's first list entries, on their way during the MMAs
          const int4 NO_ENTRY = make_int4(0, ZERO2, ZERO2, ZERO2);
          int4 pre[NPRE];
#pragma unroll
          for (int u = 0; u < NPRE; u++) pre[u] = k0 + te + u * EPI < k1 ? __ldg(g.tent + k0 + te + u * EPI) : NO_ENTRY;
          ok = wait_all(acc_full, seq);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          // largest |D|, in units of order 3
          float m = 0.0f;
          for (int c0 = 8 * part; c0 < g.wq; c0 += 2 * EPI_WARPS) {
            uint32_t a[4][8];
#pragma unroll
            for (int l = 0; l < 4; l++) tmem_ld8(taddr + l * BN + c0, a[l]);
            tmem_wait();
#pragma unroll
            for (int c = 0; c < 8; c++) {
              float f = __uint_as_float(a[0][c]);
#pragma unroll
              for (int l = 1; l < 4; l++) f = fmaf(f, 512.0f, __uint_as_float(a[l][c]));
              m = fmaxf(m, fabsf(f));
            }
          }
          const uint32_t wm = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
          if (lane == 0) {
            atomicMax(tmax + (seq & 1), wm);
            mbar_arrive(smem_u32(max_full));
          }
          ok = wait_all(max_full, seq);
          if (!ok) break;
          // |T| < (m (1 + 2^-20) + 2^17) 2^36 with the orders behind; the entries of T >> sh are below 2^55
          const float mx = __uint_as_float(*(volatile uint32_t *)(tmax + (seq & 1))) * 1.00001f + 131072.0f;
          const int sh = max(0, (int)(__float_as_uint(mx) >> 23) - 126 + 36 - 55);
          ok = wait_all(d_empty, seq ^ 1);  // the last tile's entries have been summed
          if (!ok) break;
          if (te == 0) tmax[(seq + 1) & 1] = 0;
          // usual case: hi 2^(36 - sh) + (lo >> sh) by multiply-adds, and the constants taken off once
          const bool usual = sh >= 5 && sh <= 36;
          const uint32_t up = usual ? 1u << (36 - sh) : 0u;
          const uint64_t off = usual ? dg::HI * up + (dg::LO >> sh) : 0;
          auto group = [&](const uint32_t (&a)[dg::ORDERS][4], int c0) {
            float far = usual ? 0.0f : dg::FAR;
            uint64_t d[4];
#pragma unroll
            for (int c = 0; c < 4; c++) {
              float f[dg::ORDERS];
#pragma unroll
              for (int l = 0; l < dg::ORDERS; l++) f[l] = __uint_as_float(a[l][c]);
              uint64_t hi, lo;
              dg::combine_small(f, hi, lo, far);
              d[c] = hi * up + (lo >> sh) - off;
            }
            if (__any_sync(0xffffffffu, far >= dg::FAR)) {
#pragma unroll
              for (int c = 0; c < 4; c++) {
                float f[dg::ORDERS];
#pragma unroll
                for (int l = 0; l < dg::ORDERS; l++) f[l] = __uint_as_float(a[l][c]);
                int64_t hi, lo;
                dg::combine(f, hi, lo);
                d[c] = (uint64_t)((sh <= 36 ? hi << (36 - sh) : hi >> (sh - 36)) + (lo >> sh));
              }
            }
#pragma unroll
            for (int c = 0; c < 4; c++) drow[c0 + c] = (int64_t)d[c];
          };
          for (int c0 = 4 * part; c0 < g.wq; c0 += EPI_WARPS) {
            uint32_t a[dg::ORDERS][4];
#pragma unroll
            for (int l = 0; l < dg::ORDERS; l++) tmem_ld4(taddr + l * BN + c0, a[l]);
            tmem_wait();
            group(a, c0);
          }
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) {
            mbar_arrive(smem_u32(acc_empty));
            mbar_arrive(smem_u32(d_full));
          }
          ok = wait_all(d_full, seq);
          if (!ok) break;
          const int e = ex + ew - 77 + sh;
          // integers below 2^63: where 2^e of them stays normal the exponent is added, else multiplied in
          const bool plain = e > -1020 && e < 960;
          // the sum of an entry; a target with more than six contributions has its entries in neighbouring lanes, and
          // the first one, at place 0 of the chain, gets their total
          auto total = [&](const int4 &ent) {
            const int most = __reduce_max_sync(0xffffffffu, (ent.x >> 16) & 7);  // lists run by falling count
            const uint32_t w3[3] = {(uint32_t)ent.y, (uint32_t)ent.z, (uint32_t)ent.w};
            // entries are sign << 15 | place in D; those past the count are ZERO_SLOT.  -x is (x ^ -1) + 1
            int64_t sum = __popc(w3[0] & 0x80008000u) + __popc(w3[1] & 0x80008000u) + __popc(w3[2] & 0x80008000u);
#pragma unroll
            for (int i = 0; i < 6; i++)
              if (i < most) {
                const uint32_t w = w3[i >> 1];
                const int64_t x = sd[(i & 1) ? (w >> 16) & 0x7fffu : w & 0x7fffu];
                const int s = (i & 1) ? (int)w >> 31 : (int)(w << 16) >> 31;
                sum += x ^ (int64_t)s;
              }
            const int place = ent.x >> 19, longest = __reduce_max_sync(0xffffffffu, place);
            int64_t all = sum;
            for (int k = 1; k <= longest; k++) {
              const int64_t x = __shfl_down_sync(0xffffffffu, sum, k);
              const int q = __shfl_down_sync(0xffffffffu, place, k);
              if (place == 0 && lane + k < 32 && q == k) all += x;
            }
            return all;
          };
          auto value = [&](int64_t sum) {
            const double d = (double)sum;
            return sum == 0 ? 0.0 : plain ? __hiloint2double(__double2hiint(d) + (e << 20), __double2loint(d)) : d * pow2_scale(e);
          };
          auto head = [](const int4 &ent) { return (ent.x >> 16) != 0 && (ent.x >> 19) == 0; };
          // a target is one lane's in this tile, and tiles follow one another, so sigma is read and written plainly
          double y[NPRE];
#pragma unroll
          for (int u = 0; u < NPRE; u++) y[u] = head(pre[u]) ? srow[(int64_t)(pre[u].x & 0xffff) * g.es] : 0.0;
#pragma unroll
          for (int u = 0; u < NPRE; u++) {
            const double x = value(total(pre[u]));
            if (head(pre[u])) srow[(int64_t)(pre[u].x & 0xffff) * g.es] = y[u] + x;
          }
          for (int kb = k0 + NPRE * EPI; kb < k1; kb += EPI) {  // the same rounds for every lane
            const int4 ent = kb + te < k1 ? __ldg(g.tent + kb + te) : NO_ENTRY;
            const double x = value(total(ent));
            if (head(ent)) srow[(int64_t)(ent.x & 0xffff) * g.es] += x;
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(d_empty));
        }
      }
    }
    if (!ok && lane == 0) fail();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

// ---------------------------------------------------------------------------------------------- tables

// Row I of the dense same-spin H (digits, zeroed before): singles with their phase and doubles; flags of the
// (row tile, chunk) blocks with an entry; and the largest number of a row's entries in aligned windows of 2, 4, 8, 16
// chunks.  Shared memory: one counter per chunk.
__global__ void __launch_bounds__(128) dense_kernel(const int64_t *o1, const int32_t *J1, const int32_t *info1,
                                                   const double *F1, const int64_t *o2, const int32_t *J2,
                                                   const double *D2, int64_t n, int64_t np, const uint32_t *hi, int chunks,
                                                   int tile_rows, unsigned short *d, uint8_t *flags, int *wmax) {
  extern __shared__ int cnt[];
  const int64_t I = blockIdx.x;
  const int e = plane_exp(hi);
  for (int c = threadIdx.x; c < chunks; c += blockDim.x) cnt[c] = 0;
  __syncthreads();
  auto put = [&](int J, double x) {
    atomicAdd(cnt + J / 32, 1);
    flags[(I / tile_rows) * chunks + J / 32] = 1;
    if (!d || e == digits::BAD) return;
    unsigned short h[dg::N];
    dg::to_half(digits::fixed_point<dg::BITS>(x, e), h);
#pragma unroll
    for (int i = 0; i < dg::N; i++) d[((int64_t)i * n + I) * np + J] = h[i];
  };
  for (int64_t k = o1[I] + threadIdx.x; k < o1[I + 1]; k += blockDim.x) put(J1[k], (info1[k] & 1) ? -F1[k] : F1[k]);
  for (int64_t k = o2[I] + threadIdx.x; k < o2[I + 1]; k += blockDim.x) put(J2[k], D2[k]);
  __syncthreads();
  for (int l = 0; l < 4; l++) {
    const int L = 2 << l;
    int m = 0;
    for (int w = threadIdx.x * L; w < chunks; w += blockDim.x * L) {
      int s = 0;
      for (int c = w; c < min(w + L, chunks); c++) s += cnt[c];
      m = max(m, s);
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) atomicMax(wmax + l, m);
  }
}

// digits of (P|Q): rows 2 P and 2 P + 1 (negated) of each digit, a zero row behind; pair Q in column
// 64 (Q / wq) + Q % wq
__global__ void w_kernel(const double *eab, int npair, int wq, int ncol, const uint32_t *hi, unsigned short *w) {
  const int64_t rows = 2 * npair + 1, i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows * ncol) return;
  const int r = (int)(i / ncol), c = (int)(i - (int64_t)r * ncol);
  const int Q = (c / BN) * wq + c % BN, e = plane_exp(hi);
  int64_t t = 0;
  if (c % BN < wq && Q < npair && r < 2 * npair && e != digits::BAD)
    t = digits::fixed_point<dg::BITS>(eab[(int64_t)(r >> 1) * npair + Q], e);
  if (r & 1) t = -t;
  unsigned short h[dg::N];
  dg::to_half(t, h);
#pragma unroll
  for (int k = 0; k < dg::N; k++) w[((int64_t)k * rows + r) * ncol + c] = h[k];
}

// K list of each alpha string: its singles, its occupied orbitals, then the zero row
__global__ void klist_kernel(const int64_t *o1, const int32_t *J1, const int32_t *info1, const uint64_t *str, int64_t na,
                             int kp, int npair, int2 *kl) {
  const int64_t I = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (I >= na) return;
  int2 *o = kl + I * kp;
  int k = 0;
  for (int64_t s = o1[I]; s < o1[I + 1]; s++) o[k++] = make_int2(J1[s], info1[s]);
  for (uint64_t m = str[I]; m; m &= m - 1) {
    const int p = __ffsll((long long)m) - 1;
    o[k++] = make_int2((int)I, (p * (p + 3) / 2) << 1);
  }
  for (; k < kp; k++) o[k] = make_int2((int)I, 2 * npair);
}

}  // namespace s64

// One-species full CI of more than 32 768 determinants (below, ci_sigma_rows.cu), singles and occupied orbitals of an
// alpha string within one exact sum of 80, 16-bit beta strings in the scatter lists, dense same-spin matrices of at
// most 4 GiB of digits that are at least 2.5 % filled (a digit product of a zero costs 1/60 of an FP64 FMA), and at
// least one tile of 64 alpha strings: fewer leave most of the chip without an item and the dense product of the beta
// side with padding.  One / four roots, us, here / element kernel: 16o 1a6b (16 alpha strings) 1736 / 657, 2376 / 1870;
// 24o 1a4b (24) 3218 / 2329, 5070 / 5694; 12o 2a6b (66) 234 / 308, 331 / 952; 13o 2a6b (78) 370 / 660, 661 / 2110.
// The tables of such a handle take as long as 10 to 15 of its sigmas.
bool sigma64_applicable(const pq_ci_handle *h) {
  if (h->n_species != 1 || !h->full || h->wide || h->n_dets <= ROWS_FULL_MAX) return false;
  const SpinTablesDev &a = h->tab[0][0], &b = h->tab[0][1];
  if (a.max1 + h->desc.n_alpha[0] > s64::KMAX || a.n_str < s64::BN || b.n_str >= 65536) return false;
  for (int sp = 0; sp < 2; sp++) {
    const SpinTablesDev &t = h->tab[0][sp];
    const double n = (double)t.n_str;
    if (14.0 * n * (n + 64) > 4.3e9 || (double)(t.n1 + t.n2) < 0.025 * n * n) return false;
  }
  return 2.0 * a.n_str * 7 * 4 < 2e9;  // plane rows are 32-bit TMA coordinates
}

size_t sigma64_bytes(const pq_ci_handle *h) { return h->s64 ? h->s64->bytes() : 0; }

// Scatter lists per (pass, tile of 128 beta strings): targets, each with its contributions: the singles of the tile's
// strings by pair, and their occupied orbitals onto themselves.  An entry is {target | count << 16 | place << 19, six
// contributions}; a target takes as many neighbouring entries as it needs (at most 128 contributions of other
// strings, one pair each, and its own occupied orbitals: 25 entries, and 2^7.2 terms below 2^55).
static pq_status s64_lists(const pq_ci_handle *h, const Sigma64 &S, const std::vector<int64_t> &off,
                           const std::vector<int32_t> &J, const std::vector<int32_t> &info, std::vector<int32_t> &toff,
                           std::vector<int4> &ent) {
  using namespace s64;
  const std::vector<uint64_t> &str = h->str[0][1];
  const int64_t n = (int64_t)str.size();
  const int tiles = (int)((n + BM - 1) / BM);
  std::vector<std::vector<uint32_t>> items((size_t)S.npass * tiles);  // target << 16 | contribution
  for (int64_t b = 0; b < n; b++) {
    auto put = [&](int64_t target, int pair, int neg) {
      const int p = pair / S.wq, q = pair - p * S.wq;
      items[(size_t)p * tiles + b / BM].push_back((uint32_t)target << 16 | (uint32_t)neg << 15 |
                                                  (uint32_t)((b % BM) * LDS_D + q));
    };
    for (int64_t s = off[b]; s < off[b + 1]; s++) put(J[s], info[s] >> 1, info[s] & 1);
    for (uint64_t m = str[b]; m; m &= m - 1) {
      const int k = __builtin_ctzll(m);
      put(b, k * (k + 3) / 2, 0);
    }
  }
  toff.assign(items.size() + 1, 0);
  ent.clear();
  std::vector<uint32_t> v;
  std::vector<int32_t> at(n + 1);
  std::vector<std::pair<size_t, size_t>> runs;
  for (size_t i = 0; i < items.size(); i++) {
    // in order of target and contribution: counted by target, then sorted within each one's few
    std::fill(at.begin(), at.end(), 0);
    for (uint32_t x : items[i]) at[(x >> 16) + 1]++;
    std::partial_sum(at.begin(), at.end(), at.begin());
    v.resize(items[i].size());
    for (uint32_t x : items[i]) v[at[x >> 16]++] = x;
    runs.clear();  // ranges of one target
    for (size_t u = 0; u < v.size();) {
      const size_t w = at[v[u] >> 16];
      std::sort(v.begin() + u, v.begin() + w);
      runs.emplace_back(u, w);
      u = w;
    }
    // by falling count, so that a warp's entries take the same steps
    std::stable_sort(runs.begin(), runs.end(), [](const auto &x, const auto &y) { return x.second - x.first > y.second - y.first; });
    for (const auto &r : runs) {
      const size_t need = (r.second - r.first + 5) / 6;
      // the entries of a target stay within one group of 32
      while ((ent.size() - toff[i]) % 32 + need > 32) ent.push_back(make_int4(0, ZERO2, ZERO2, ZERO2));
      for (size_t u = r.first, place = 0; u < r.second; place++) {
        uint32_t c[6] = {ZERO_SLOT, ZERO_SLOT, ZERO_SLOT, ZERO_SLOT, ZERO_SLOT, ZERO_SLOT};
        uint32_t k = 0;
        for (; u < r.second && k < 6; u++) c[k++] = v[u] & 0xffffu;
        ent.push_back(make_int4((int)(v[r.first] >> 16 | k << 16 | (uint32_t)place << 19), (int)(c[0] | c[1] << 16),
                                (int)(c[2] | c[3] << 16), (int)(c[4] | c[5] << 16)));
      }
    }
    if (ent.size() > (size_t)INT32_MAX / 2) {
      set_error("FP64 full-CI sigma: scatter lists too large");
      return PQ_ERR_ARG;
    }
    toff[i + 1] = (int32_t)ent.size();
  }
  return PQ_OK;
}

static pq_status s64_prepare(pq_ci_handle *h) {
  using namespace s64;
  if (h->s64) return PQ_OK;
  std::unique_ptr<Sigma64, void (*)(Sigma64 *)> S(new (std::nothrow) Sigma64(), sigma64_delete);
  if (!S) {
    set_error("host allocation failed");
    return PQ_ERR_OOM;
  }
  cudaStream_t st = h->stream;
  const pq_ci_desc &d = h->desc;
  const SpinTablesDev &a = h->tab[0][0], &bt = h->tab[0][1];
  const int npair = h->npair[0];
  // identical spin lists with identical integrals share the matrix
  const bool shared = !h->selected && h->n_blocks[0] == 1 && d.n_alpha[0] == d.n_beta[0] && d.ex_level[0][0] == d.ex_level[0][1];
  S->npass = (npair + BN - 1) / BN;
  S->wq = (npair + S->npass - 1) / S->npass;
  const int ncol = S->npass * BN, wrows = 2 * npair + 1;
  S->kp = std::max<int>(16, (int)up64(a.max1 + d.n_alpha[0], 16));
  int chunks[2], tile_rows[2] = {BN, BM};
  int64_t rt[2];
  for (int sp = 0; sp < 2; sp++) {
    Sigma64::Side &z = S->side[sp];
    z.n = h->tab[0][sp].n_str;
    z.np = up64(z.n, 64);
    chunks[sp] = (int)((z.n + 31) / 32);
    rt[sp] = (z.n + tile_rows[sp] - 1) / tile_rows[sp];
  }
  uint8_t *flags = nullptr;  // both sides' flags, then 2 x 4 window maxima
  const size_t nflags = (size_t)(rt[0] * chunks[0] + rt[1] * chunks[1] + 15) / 16 * 16;
  size_t zeroed = 0;
  auto lay = [&](DevLayout &l) {
    l.take(S->hi, 4);
    l.take(S->aux, 16);
    l.take(flags, nflags + 8 * sizeof(int));
    for (int sp = 0; sp < (shared ? 1 : 2); sp++) l.take(S->side[sp].d, (size_t)dg::N * S->side[sp].n * S->side[sp].np);
    zeroed = l.used;
    l.take(S->w, (size_t)dg::N * wrows * ncol);
    l.take(S->klist, (size_t)a.n_str * S->kp);
  };
  DevLayout l;
  lay(l);
  PQ_TRY(S->mem.alloc(l.used));
  l = DevLayout{static_cast<char *>(S->mem.ptr), 0};
  lay(l);
  PQ_CUDA_TRY(cudaMemsetAsync(S->mem.ptr, 0, zeroed, st));
  int *wmax = reinterpret_cast<int *>(flags + nflags);
  for (int sp = 0; sp < 2; sp++) {
    const SpinTablesDev &t = h->tab[0][sp];
    const Sigma64::Side &z = S->side[sp];
    uint32_t *hi = S->hi + sp;
    const unsigned g1 = (unsigned)std::min<int64_t>((t.n1 + 255) / 256, 1216), g2 = (unsigned)std::min<int64_t>((t.n2 + 255) / 256, 1216);
    if (t.n1) absmax_kernel<<<g1, 256, 0, st>>>(t.s1_F64.as<double>(), t.n1, hi);
    if (t.n2) absmax_kernel<<<g2, 256, 0, st>>>(t.s2_D64.as<double>(), t.n2, hi);
    dense_kernel<<<(unsigned)z.n, 128, chunks[sp] * sizeof(int), st>>>(
        t.s1_off.as<int64_t>(), t.s1_J.as<int32_t>(), t.s1_info.as<int32_t>(), t.s1_F64.as<double>(), t.s2_off.as<int64_t>(),
        t.s2_J.as<int32_t>(), t.s2_D64.as<double>(), z.n, z.np, hi, chunks[sp], tile_rows[sp], z.d,
        flags + (sp ? rt[0] * chunks[0] : 0), wmax + 4 * sp);
    PQ_CUDA_TRY(cudaGetLastError());
  }
  absmax_kernel<<<32, 256, 0, st>>>(h->d_eab64.as<double>(), (int64_t)npair * npair, S->hi + 2);
  w_kernel<<<(unsigned)(((int64_t)wrows * ncol + 255) / 256), 256, 0, st>>>(h->d_eab64.as<double>(), npair, S->wq, ncol, S->hi + 2, S->w);
  klist_kernel<<<(unsigned)((a.n_str + 127) / 128), 128, 0, st>>>(a.s1_off.as<int64_t>(), a.s1_J.as<int32_t>(),
                                                                a.s1_info.as<int32_t>(), a.str.as<uint64_t>(), a.n_str, S->kp,
                                                                npair, S->klist);
  PQ_CUDA_TRY(cudaGetLastError());
  std::vector<uint8_t> f(nflags + 8 * sizeof(int));
  std::vector<int64_t> off(bt.n_str + 1);
  std::vector<int32_t> J(bt.n1 + 1), info(bt.n1 + 1);
  PQ_CUDA_TRY(cudaMemcpyAsync(off.data(), bt.s1_off.ptr, off.size() * 8, cudaMemcpyDeviceToHost, st));
  PQ_CUDA_TRY(cudaMemcpyAsync(J.data(), bt.s1_J.ptr, bt.n1 * 4, cudaMemcpyDeviceToHost, st));
  PQ_CUDA_TRY(cudaMemcpyAsync(info.data(), bt.s1_info.ptr, bt.n1 * 4, cudaMemcpyDeviceToHost, st));
  PQ_CUDA_TRY(cudaMemcpyAsync(f.data(), flags, f.size(), cudaMemcpyDeviceToHost, st));
  PQ_CUDA_TRY(cudaStreamSynchronize(st));
  // the lists, one upload: scatter entries, then the offsets and chunk lists
  std::vector<int32_t> toff, kto[2], ktl[2];
  std::vector<int4> ent;
  PQ_TRY(s64_lists(h, *S, off, J, info, toff, ent));
  const uint8_t *fl = f.data();
  for (int sp = 0; sp < 2; sp++) {
    int wm[4];
    memcpy(wm, f.data() + nflags + 4 * sp * sizeof(int), sizeof(wm));
    for (int k = 1; k < 4; k++)
      if (wm[k] <= KMAX) S->side[sp].win = 2 << k;
    kto[sp].assign(rt[sp] + 1, 0);
    for (int64_t r = 0; r < rt[sp]; r++) {
      for (int c = 0; c < chunks[sp]; c++)
        if (fl[r * chunks[sp] + c]) ktl[sp].push_back(c);
      kto[sp][r + 1] = (int32_t)ktl[sp].size();
    }
    fl += rt[sp] * chunks[sp];
  }
  auto lay2 = [&](DevLayout &m) {
    m.take(S->tent, ent.size() + 1);
    m.take(S->toff, toff.size());
    for (int sp = 0; sp < 2; sp++) {
      m.take(S->side[sp].kt_off, kto[sp].size());
      m.take(S->side[sp].kt_list, ktl[sp].size() + 1);
    }
  };
  DevLayout m;
  lay2(m);
  PQ_TRY(S->lists.alloc(m.used));
  std::vector<char> host(m.used);
  m = DevLayout{host.data(), 0};
  lay2(m);
  memcpy(S->tent, ent.data(), ent.size() * sizeof(int4));
  memcpy(S->toff, toff.data(), toff.size() * 4);
  for (int sp = 0; sp < 2; sp++) {
    memcpy(S->side[sp].kt_off, kto[sp].data(), kto[sp].size() * 4);
    memcpy(S->side[sp].kt_list, ktl[sp].data(), ktl[sp].size() * 4);
  }
  m = DevLayout{static_cast<char *>(S->lists.ptr), 0};
  lay2(m);
  PQ_CUDA_TRY(cudaMemcpyAsync(S->lists.ptr, host.data(), host.size(), cudaMemcpyHostToDevice, st));
  if (shared) S->side[1].d = S->side[0].d;
  int dev = 0;
  PQ_CUDA_TRY(cudaGetDevice(&dev));
  PQ_CUDA_TRY(cudaDeviceGetAttribute(&S->sms, cudaDevAttrMultiProcessorCount, dev));
  PQ_CUDA_TRY(cudaFuncSetAttribute(ab64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AB_SMEM));
  PQ_CUDA_TRY(cudaFuncSetAttribute(ss64_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SS_SMEM));
  PQ_CUDA_TRY(cudaFuncSetAttribute(ss64_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SS_SMEM));
  PQ_CUDA_TRY(cudaStreamSynchronize(st));  // the host copy of the lists ends here
  h->s64 = std::move(S);
  return PQ_OK;
}

// S = (H - shift) C for nv <= 4 vectors of device memory, vector v of determinant I at C[I es + v vs] and
// S[I ses + v svs]; C and S must not overlap, and are either columns (es = 1) or interleaved (es = nv, vs = 1)
pq_status ci_sigma64(pq_ci_handle *h, const double *C, int64_t es, int64_t vs, int nv, double shift, double *S, int64_t ses,
                     int64_t svs, bool fixed, int **gate_out) {
  using namespace s64;
  if (fixed && !h->s64) return PQ_ERR_OOM;
  PQ_TRY(s64_prepare(h));
  Sigma64 &z = *h->s64;
  cudaStream_t st = h->stream;
  const int64_t na = h->tab[0][0].n_str, nb = h->tab[0][1].n_str, n = h->n_dets, nbp = up64(nb, 64);
  const size_t xbytes = 2 * (size_t)dg::N * nv * na * nbp;
  if (fixed && z.xd.bytes < xbytes) return PQ_ERR_OOM;
  PQ_TRY(ci_grow(h, z.xd, xbytes));
  int *gate = z.aux;
  uint32_t *xhi = reinterpret_cast<uint32_t *>(z.aux) + 4, *hi = z.hi;
  PQ_CUDA_TRY(cudaMemsetAsync(z.aux, 0, 64, st));
  x64_absmax_kernel<<<dim3((unsigned)std::min<int64_t>((n + 255) / 256, 152 * 4), nv), 256, 0, st>>>(C, es, vs, n, xhi);
  x64_digits_kernel<<<dim3((unsigned)na, nv), 256, 0, st>>>(C, es, vs, na, nb, nbp, nv, xhi, hi, h->tab[0][0].e_same64.as<double>(),
                                                          h->tab[0][1].e_same64.as<double>(), shift,
                                                          z.xd.as<unsigned short>(), S, ses, svs, gate);
  PQ_CUDA_TRY(cudaGetLastError());
  const Sigma64::Side &A = z.side[0], &B = z.side[1];
  SsArgs g{};
  g.na = na, g.nb = nb, g.nv = nv;
  g.m_tiles = (int)((nb + BM - 1) / BM);
  g.n_tiles = (int)((na + BN - 1) / BN);
  g.tiles = (int64_t)nv * g.m_tiles * g.n_tiles;
  g.xhi = xhi;
  g.S = S, g.es = ses, g.vs = svs, g.gate = gate;
  g.wait = sigma_wait_cycles(0);
  const unsigned grid = (unsigned)std::min<int64_t>(g.tiles, z.sms);
  CUtensorMap ma, mb;
  const int64_t xrows = (int64_t)dg::N * nv * na;
  // alpha: strips of 64 beta strings of 32 rows Ja; rows of Ha
  PQ_TRY(s64_map(&ma, z.xd.ptr, xrows, nb, nbp, 64, 32));
  PQ_TRY(s64_map(&mb, A.d, dg::N * A.n, A.n, A.np, 32, BN));
  g.ksplit = 1;
  g.win = A.win;
  g.a_plane = (int64_t)nv * na, g.b_plane = A.n;
  g.kt_off = A.kt_off, g.kt_list = A.kt_list;
  g.dhi = hi;
  ss64_kernel<true><<<grid, THREADS, SS_SMEM, st>>>(ma, mb, g);
  // beta: rows of Hb; rows (v, Ia) of C
  PQ_TRY(s64_map(&ma, B.d, dg::N * B.n, B.n, B.np, 32, BM));
  PQ_TRY(s64_map(&mb, z.xd.ptr, xrows, nb, nbp, 32, BN));
  g.win = B.win;
  g.a_plane = B.n, g.b_plane = (int64_t)nv * na;
  g.kt_off = B.kt_off, g.kt_list = B.kt_list;
  g.dhi = hi + 1;
  ss64_kernel<false><<<grid, THREADS, SS_SMEM, st>>>(ma, mb, g);
  PQ_CUDA_TRY(cudaGetLastError());
  AbArgs x{};
  const int ncol = z.npass * BN, wrows = 2 * h->npair[0] + 1;
  PQ_TRY(s64_map(&ma, z.xd.ptr, xrows, nb, nbp, 64, 1));
  PQ_TRY(s64_map(&mb, z.w, (int64_t)dg::N * wrows, ncol, ncol, 64, 1));
  x.na = na, x.nb = nb, x.nv = nv;
  x.npass = z.npass, x.wq = z.wq, x.kp = z.kp, x.wrows = wrows;
  x.m_tiles = g.m_tiles;
  // few items: one per root, so that the last round of CTAs is short
  x.vsplit = na < 8 * z.sms;
  x.items = na * (x.vsplit ? nv : 1);
  x.klist = z.klist;
  x.toff = z.toff;
  x.tent = z.tent;
  x.xhi = xhi, x.whi = hi + 2;
  x.S = S, x.es = ses, x.vs = svs, x.gate = gate;
  x.wait = sigma_wait_cycles(1);
  ab64_kernel<<<(unsigned)std::min<int64_t>(x.items, z.sms), AB_THREADS, AB_SMEM, st>>>(ma, mb, x);
  PQ_CUDA_TRY(cudaGetLastError());
  *gate_out = gate;
  return PQ_OK;
}

}  // namespace pq

extern "C" pq_status pq_debug_set_sigma_wait_budget(long long same_spin, long long opposite_spin) {
  pq::g_sigma_wait[0] = same_spin > 0 ? same_spin : pq::tcx::WAIT_CYCLES;
  pq::g_sigma_wait[1] = opposite_spin > 0 ? opposite_spin : pq::tcx::WAIT_CYCLES;
  return PQ_OK;
}
