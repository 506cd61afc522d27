// FP64 sigma = H C of one species with one warp (or one CTA) per determinant.
//
// Reference: src/ci/detset/direct_singleparticle.cpp:238-372, the elements of
// slater_condon_singleparticle.cpp:53-175 (as ci_sigma.cu applies them).
//
// The kernel of ci_sigma.cu gives every determinant one thread of a CTA that
// covers 256 beta strings of one alpha string.  That fills the chip only when
// the beta rows are long and there are many determinants.  A truncated space
// has mostly rows of one beta string (in CISD every doubly excited alpha string
// goes with the Fermi beta string alone), so its CTAs ran one live thread
// through some 10^3 connections, and a small full space has fewer
// determinants than the chip has warps.  Here the 32 lanes of a warp share one
// determinant's connections, and a determinant with far more of them than its
// neighbours (the Fermi determinant of a truncated space has all of them) is
// shared by the 8 warps of the CTA.
//
// A truncated space keeps the pairs with level(alpha) + level(beta) <= limit.
// A single moves a string's level by -1, 0 or +1 and a double by -2 .. +2, so
// with the entries of each string grouped by that change the partners that are
// in the list are a prefix of the groups, and the alpha-beta doubles are three
// rectangles (alpha group) x (prefix of the beta groups): no entry is looked
// up in vain and no lane idles inside a rectangle.  The grouped copies hold
// the partner's row offset (alpha) or string (beta), and the opposite-spin
// Coulomb sums of the singles come from tables [string][pair].
//
// Bound: FP64 pipe and L2 gathers.  CISD of 5a5b in 24 orbitals (12 636
// determinants, 11.2 M elements), three roots: 125 us a sigma against 3914 us
// with the thread-per-determinant kernel, 0.54 TFLOP/s; full CI of water in 7
// orbitals (441 determinants), one root: 18 against 41 us.
#include <algorithm>

#include "ci_rows.cuh"

namespace pq {

void rows_delete(SigmaRows *r) { delete r; }

namespace rows {

constexpr int U = 4;  // gathers in flight per lane

// acc += c x over the entries tid, tid + nth, ... of a list of n, U of them in flight; entries past the end load
// nothing
template <int NV, typename M>
__device__ __forceinline__ void gather(const Args &p, double (&acc)[NV], int tid, int nth, int n, M &&make) {
  if (n == 0) return;
  auto entry = make(tid, nth);
  for (int t0 = 0; t0 < n; t0 += U * nth) {
    double c[U], x[U][NV];
#pragma unroll
    for (int u = 0; u < U; u++) {
      c[u] = 0.0;
#pragma unroll
      for (int v = 0; v < NV; v++) x[u][v] = 0.0;
      if (t0 + u * nth + tid < n) {
        int64_t j;
        c[u] = entry(j);
        load_x<NV>(p.X, j, x[u]);
      }
    }
#pragma unroll
    for (int u = 0; u < U; u++)
      if (t0 + u * nth < n) {  // the same for all threads that share the list
#pragma unroll
        for (int v = 0; v < NV; v++) acc[v] = fma(c[u], x[u][v], acc[v]);
      }
  }
}

// the part of thread tid of nth of determinant d's row of H times X
template <int NV>
__device__ __forceinline__ void accumulate(const Args &p, const Det &d, int tid, int nth, double (&acc)[NV]) {
  if (tid == 0) {
    double x[NV];
    load_x<NV>(p.X, d.I, x);
    const double h = p.diag[d.I] - p.shift;
#pragma unroll
    for (int v = 0; v < NV; v++) acc[v] = h * x[v];
  }
  for_lists(p, d, [&](int n, auto &&make) { gather<NV>(p, acc, tid, nth, n, make); });
}

// Sum of acc over the warp: the halving steps also halve the number of values a lane carries, so four roots take
// 6 additions instead of 20 on the FP64 pipe.  The sum of root v ends in lane root_lane(v), in acc[0].
template <int NV> __device__ __forceinline__ void warp_sum(double (&acc)[NV], int lane) {
  int w = 16;
  if constexpr (NV >= 3) {
    const bool hi = lane & 16;
    const double x3 = NV == 4 ? acc[NV - 1] : 0.0;
    const double s0 = hi ? acc[0] : acc[2], s1 = hi ? acc[1] : x3;
    const double k0 = hi ? acc[2] : acc[0], k1 = hi ? x3 : acc[1];
    acc[0] = k0 + __shfl_xor_sync(0xffffffffu, s0, 16);
    acc[1] = k1 + __shfl_xor_sync(0xffffffffu, s1, 16);
    w = 8;
  }
  if constexpr (NV >= 2) {
    const bool hi = lane & w;
    const double s = hi ? acc[0] : acc[1], k = hi ? acc[1] : acc[0];
    acc[0] = k + __shfl_xor_sync(0xffffffffu, s, w);
    w >>= 1;
  }
  for (; w; w >>= 1) acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], w);
}
template <int NV> __device__ __forceinline__ int root_of_lane(int lane) {  // -1: the lane holds no root
  if (NV == 1) return lane == 0 ? 0 : -1;
  if (NV == 2) return (lane & 15) == 0 ? lane >> 4 : -1;
  const int v = ((lane >> 4) & 1) * 2 + ((lane >> 3) & 1);
  return (lane & 7) == 0 && v < NV ? v : -1;
}

template <int NV> __global__ void __launch_bounds__(32 * WARPS, 3) sigma_rows_kernel(Args p) {
  __shared__ double part[WARPS][4];
  __shared__ int len[WARPS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t I0 = (int64_t)blockIdx.x * WARPS, I = I0 + warp;
  bool heavy = false;
#pragma unroll 1
  for (int pass = 0; pass < 2; pass++) {  // light rows, then the heavy ones that are not shared
    if (pass ? heavy && !shared_row(len, warp) : I < p.n) {
      const Det d = load_det(p, I);
      heavy = d.total > HEAVY;
      if (pass == 0 && lane == 0) len[warp] = d.total;
      if (!heavy || pass) {
        double acc[NV];
#pragma unroll
        for (int v = 0; v < NV; v++) acc[v] = 0.0;
        accumulate<NV>(p, d, lane, 32, acc);
        warp_sum<NV>(acc, lane);
        const int v = root_of_lane<NV>(lane);
        if (v >= 0) p.Y[I * NV + v] = acc[0];
      }
    } else if (pass == 0 && lane == 0) {
      len[warp] = 0;
    }
    if (pass == 0 && !__syncthreads_or(heavy)) return;
  }
  for (int k = 0; k < WARPS; k++) {
    if (!shared_row(len, k)) continue;  // the same for every thread
    const Det d = load_det(p, I0 + k);
    double acc[NV];
#pragma unroll
    for (int v = 0; v < NV; v++) acc[v] = 0.0;
    accumulate<NV>(p, d, threadIdx.x, 32 * WARPS, acc);
    warp_sum<NV>(acc, lane);
    const int v = root_of_lane<NV>(lane);
    if (v >= 0) part[warp][v] = acc[0];
    __syncthreads();
    if (threadIdx.x < NV) {
      double s = 0.0;
      for (int w = 0; w < WARPS; w++) s += part[w][threadIdx.x];
      p.Y[d.I * NV + threadIdx.x] = s;
    }
    __syncthreads();
  }
}

// Entries of each string grouped by level change, in table order inside a group: warp per string.
// key[J] is what a grouped entry stores for partner J (its row offset, or J itself when NULL).
__global__ void __launch_bounds__(128) group_kernel(int64_t n_str, const int32_t *lvl, const int64_t *key,
                                                    const int64_t *o1, const int32_t *J1, const int32_t *info1,
                                                    const double *F1, const int64_t *o2, const int32_t *J2,
                                                    const double *D2, int2 *s1, double *F, int32_t *s2, double *D,
                                                    int32_t *cum) {
  const int lane = threadIdx.x & 31;
  const int64_t I = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (I >= n_str) return;
  const int l0 = lvl[I];
  int64_t w = o1[I];
  for (int g = 0; g < 3; g++) {
    for (int64_t e0 = o1[I]; e0 < o1[I + 1]; e0 += 32) {
      const int64_t e = e0 + lane;
      const int J = e < o1[I + 1] ? J1[e] : -1;
      const bool take = J >= 0 && lvl[J] - l0 == g - 1;
      const unsigned m = __ballot_sync(0xffffffffu, take);
      if (take) {
        const int64_t o = w + __popc(m & ((1u << lane) - 1u));
        s1[o] = make_int2(key ? (int)key[J] : J, info1[e]);
        F[o] = F1[e];
      }
      w += __popc(m);
    }
    if (lane == 0) cum[8 * I + g] = (int32_t)(w - o1[I]);
  }
  w = o2[I];
  for (int g = 0; g < 5; g++) {
    for (int64_t e0 = o2[I]; e0 < o2[I + 1]; e0 += 32) {
      const int64_t e = e0 + lane;
      const int J = e < o2[I + 1] ? J2[e] : -1;
      const bool take = J >= 0 && lvl[J] - l0 == g - 2;
      const unsigned m = __ballot_sync(0xffffffffu, take);
      if (take) {
        const int64_t o = w + __popc(m & ((1u << lane) - 1u));
        s2[o] = key ? (int)key[J] : J;
        D[o] = D2[e];
      }
      w += __popc(m);
    }
    if (lane == 0) cum[8 * I + 3 + g] = (int32_t)(w - o2[I]);
  }
}

// coul[string][pair] = sum over the string's occupied orbitals k of E[pair * rs + kk * cs]
__global__ void __launch_bounds__(256) coulomb_kernel(const double *E, int npair, int64_t rs, int64_t cs,
                                                      const uint64_t *str, const uint64_t *str_hi, int64_t n_str,
                                                      double *coul) {
  const int64_t total = (int64_t)npair * n_str;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t s = i / npair;
    const int pr = (int)(i - s * npair);
    double c = 0.0;
    for_occ(str[s], hiword(str_hi, s), [&](int k) { c += E[pr * rs + (int64_t)(k * (k + 3) / 2) * cs]; });
    coul[i] = c;
  }
}

__global__ void __launch_bounds__(128) row_kernel(const int64_t *rowoff, const int32_t *rowlen, int64_t na, int32_t *row) {
  for (int64_t a = blockIdx.x; a < na; a += gridDim.x)
    for (int b = threadIdx.x; b < rowlen[a]; b += blockDim.x) row[rowoff[a] + b] = (int32_t)a;
}

}  // namespace rows

// Rules (32-bit determinant indices throughout).  Full spaces take this kernel up to ROWS_FULL_MAX determinants, where
// the other kernel has too few threads to hide the latency of its serial walk; beyond, that one's staged coefficients
// and coalesced alpha rows win.  us a sigma (whole call, four roots), this kernel / the other: 441 determinants
// 22 / 78, 4 900 55 / 126, 15 876 159 / 170, 63 504 657 / 619, 213 444 2955 / 2328.
// Truncated spaces take it unless they are large and nearly full, so that the other kernel's CTAs of 256 beta strings
// have few idle threads (`busy`, the share of threads with a determinant), and its packed registers hold the beta
// singles.  With one to four roots, us, this kernel / the other:
//   at most 32 singles  11o 5a5b, level 6 of 10 (busy 0.73): 827 / 688 ... 2224 / 1966; level 5 (0.49) 472 / 471 ...
//                       1265 / 1387; 12o 4a4b, level 7 (0.95) 1300 / 1144 ... 3448 / 2745, level 5 (0.53) 623 / 685 ...
//                       1661 / 1789; 10o 5a5b, level 7 (0.97, 62 628 determinants) 256 / 225 ... 667 / 634; 10o 4a4b,
//                       level 7 (0.82, 43 875) 178 / 188 ... 478 / 537: the other kernel from PACK32_MIN on
//   at most 64 singles  one root only: 14o 7a7b, level 8 of 14 (0.83) 113 / 98 ms, four roots 267 / 303 ms; 13o 5a5b,
//                       level 8 (0.82) 13.4 / 12.7, four 31.7 / 39.0; 14o 5a5b, level 7 (0.79) 29.5 / 28.3; 12o 6a6b,
//                       level 6 (0.59) 3.34 / 4.04, level 8 (0.88, 834 957) 5.80 / 5.82; 13o 4a4b, level 7 (0.90,
//                       495 349) 3.36 / 3.56: the other kernel from PACK64_MIN on
constexpr int64_t PACK32_MIN = 50000, PACK64_MIN = 800000;
constexpr double PACK32_BUSY = 0.7, PACK64_BUSY = 0.75;
constexpr size_t ROWS_COUL_MAX = (size_t)1 << 30;  // larger Coulomb tables are summed in the kernel instead

pq_status rows_make(pq_ci_handle *h, std::unique_ptr<SigmaRows, void (*)(SigmaRows *)> &out) {
  using namespace rows;
  const int npair = h->npair[0];
  cudaStream_t st = h->stream;
  std::unique_ptr<SigmaRows, void (*)(SigmaRows *)> r(new (std::nothrow) SigmaRows(), rows_delete);
  if (!r) {
    set_error("host allocation failed");
    return PQ_ERR_OOM;
  }
  r->lim = std::min(h->desc.ex_level[0][2], h->desc.max_collective);
  auto lay = [&](DevLayout &l) {
    for (int sp = 0; sp < 2; sp++) {
      const SpinTablesDev &t = h->tab[0][sp];
      SigmaRows::Side &s = r->side[sp];
      const size_t coul = (size_t)npair * t.n_str;
      l.take(s.lvl, t.n_str);
      l.take(s.cum, 8 * t.n_str);
      l.take(s.s1, t.n1 + 1);
      l.take(s.s1_F, t.n1 + 1);
      l.take(s.s2, t.n2 + 1);
      l.take(s.s2_D, t.n2 + 1);
      if (sizeof(double) * coul <= ROWS_COUL_MAX) l.take(s.coul, coul);
    }
    l.take(r->row, h->n_dets);
  };
  DevLayout l;
  lay(l);
  PQ_TRY(r->mem.alloc(l.used));
  l = DevLayout{static_cast<char *>(r->mem.ptr), 0};
  lay(l);
  for (int sp = 0; sp < 2; sp++) {
    const SpinTablesDev &t = h->tab[0][sp];
    SigmaRows::Side &s = r->side[sp];
    PQ_CUDA_TRY(cudaMemcpyAsync(s.lvl, h->lvl[0][sp].data(), sizeof(int32_t) * t.n_str, cudaMemcpyHostToDevice, st));
    group_kernel<<<(unsigned)((t.n_str + 3) / 4), 128, 0, st>>>(
        t.n_str, s.lvl, sp == 0 ? h->d_rowoff.as<int64_t>() : nullptr, t.s1_off.as<int64_t>(), t.s1_J.as<int32_t>(),
        t.s1_info.as<int32_t>(), t.s1_F64.as<double>(), t.s2_off.as<int64_t>(), t.s2_J.as<int32_t>(), t.s2_D64.as<double>(),
        s.s1, s.s1_F, s.s2, s.s2_D, s.cum);
    PQ_CUDA_TRY(cudaGetLastError());
    if (!s.coul) continue;
    const int64_t total = (int64_t)npair * t.n_str;
    coulomb_kernel<<<(unsigned)std::min<int64_t>((total + 255) / 256, 152 * 16), 256, 0, st>>>(
        h->d_eab64.as<double>(), npair, sp == 0 ? 1 : npair, sp == 0 ? npair : 1, t.str.as<uint64_t>(),
        t.str_hi.as<uint64_t>(), t.n_str, s.coul);
    PQ_CUDA_TRY(cudaGetLastError());
  }
  const int64_t na = h->tab[0][0].n_str;
  row_kernel<<<(unsigned)std::min<int64_t>(na, 152 * 16), 128, 0, st>>>(h->d_rowoff.as<int64_t>(),
                                                                       h->d_rowlen.as<int32_t>(), na, r->row);
  PQ_CUDA_TRY(cudaGetLastError());
  out = std::move(r);
  return PQ_OK;
}

bool ci_rows_apply(const pq_ci_handle *h, int nvp) { return h->rows && nvp >= h->rows->min_width; }

rows::Args rows_args(const pq_ci_handle *h, const SigmaRows &r) {
  rows::Args p{};
  rows::Side *out[2] = {&p.a, &p.b};
  p.npair = h->npair[0];
  for (int sp = 0; sp < 2; sp++) {
    const SpinTablesDev &t = h->tab[0][sp];
    const SigmaRows::Side &s = r.side[sp];
    // strings of one spin stand beside singles of the other: eab is [pair_alpha][pair_beta]
    *out[sp] = {t.s1_off.as<int64_t>(), t.s2_off.as<int64_t>(), s.s1, s.s1_F, s.s2, s.s2_D,
                reinterpret_cast<const int4 *>(s.cum), s.lvl, s.coul, t.str.as<uint64_t>(), t.str_hi.as<uint64_t>(),
                sp == 0 ? 1 : p.npair, sp == 0 ? p.npair : 1};
  }
  p.row = r.row;
  p.rowoff = h->d_rowoff.as<int64_t>();
  p.eab = h->d_eab64.as<double>();
  p.diag = h->d_diag.as<double>();
  p.lim = r.lim;
  p.n = h->n_dets;
  return p;
}

pq_status ci_sigma_rows_build(pq_ci_handle *h) {
  if (h->batched || h->n_species != 1 || h->n_dets <= 0 || h->n_dets > 0x7fffffffLL) return PQ_OK;
  if (h->full && h->n_dets > ROWS_FULL_MAX) return PQ_OK;
  int64_t threads = 0;
  for (int32_t len : h->rowlen) threads += (len + 255) / 256 * 256;
  const double busy = (double)h->n_dets / (double)threads;
  const int pack = h->full ? 0 : ci_sigma_pack(h);
  if (pack == 32 && h->n_dets >= PACK32_MIN && busy > PACK32_BUSY) return PQ_OK;
  const pq_status s = rows_make(h, h->rows);
  if (s == PQ_ERR_OOM) {
    clear_error();
    return PQ_OK;
  }
  PQ_TRY(s);
  h->rows->min_width = pack == 64 && h->n_dets >= PACK64_MIN && busy > PACK64_BUSY ? 2 : 1;
  return PQ_OK;
}

pq_status ci_sigma_rows(pq_ci_handle *h, const void *X, void *Y, int nvp, double shift) {
  using namespace rows;
  Args p = rows_args(h, *h->rows);
  p.shift = shift;
  p.X = (const double *)X;
  p.Y = (double *)Y;
  const unsigned grid = (unsigned)((p.n + WARPS - 1) / WARPS);
  if (nvp == 1)
    sigma_rows_kernel<1><<<grid, 32 * WARPS, 0, h->stream>>>(p);
  else if (nvp == 2)
    sigma_rows_kernel<2><<<grid, 32 * WARPS, 0, h->stream>>>(p);
  else if (nvp == 3)
    sigma_rows_kernel<3><<<grid, 32 * WARPS, 0, h->stream>>>(p);
  else if (nvp == 4)
    sigma_rows_kernel<4><<<grid, 32 * WARPS, 0, h->stream>>>(p);
  else {
    set_error("sigma: unsupported interleave width %d (widths 1 to 4)", nvp);
    return PQ_ERR_ARG;
  }
  PQ_CUDA_TRY(cudaGetLastError());
  return PQ_OK;
}

}  // namespace pq
