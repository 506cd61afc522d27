// Properties of CI vectors on the device: <S^2> of each state and species and
// the one-particle reduced density matrix of one state, species and spin.
//
// <S^2> follows POLYQUANT_DETSET::evaluate_s2 (src/ci/detset/s2.cpp:4-123):
// diagonal n_a + s_z (s_z - 1) from the open shells of each determinant
// (n_a open-shell alpha electrons, s_z = n_a - n_open / 2), and for every
// alpha single h_a -> p_a paired with the beta single p_a -> h_a (a spin
// flip) the term -phase_a phase_b C_I C_J.
// The 1-RDM follows create_1rdm (src/ci/detset/rdm1.cpp:4-72): C_I^2 on the
// occupied orbitals of the chosen spin, and phase C_I C_J on (k, l) and
// (l, k) for each single of that spin between I and an earlier J (hole k in
// I, particle l).
// One species: both properties are sums over pairs of strings that differ by
// one orbital pair, so the singles of each spin are kept once more as lists by
// orbital pair (PairLists).  The alpha 1-RDM is then a sum of dot products of
// rows of C, the beta one a sum over column pairs of rows staged in shared
// memory, and <S^2> runs, pair by pair, over alpha moves up against beta moves
// down; sums stay in registers per pair and meet in one atomic per warp or
// block.  The former kernels, thread per determinant, added every product to a
// shared-memory matrix by FP64 atomics and searched each beta partner along
// its string's list.  Four states and two 1-RDMs of FCI(12o, 6a6b): 359 us
// against 5212.
// Two species: CTA per species-0 pair, threads over its species-1 block, with
// the other species' strings held fixed, as in the reference's per-species
// loops.
#include <algorithm>
#include <new>

#include "pq_bits.cuh"
#include "pq_internal.h"

namespace pq {

constexpr int PROP_THREADS = 128;
constexpr int S2_MAXV = 8;

// ---- one species ------------------------------------------------------------
// Singles of one spin by orbital pair q = idx2(i, j), i > j: every unordered pair of strings that differ by a move
// between i and j, at the string with the larger index, in its order: {I << 1 | phase, J << 1 | (I holds i)}; for
// i = j the strings that hold i, {I << 1, I << 1}.
struct PairLists {
  struct Side {
    int64_t *off = nullptr;  // [npair + 1]
    uint2 *ent = nullptr;
    int64_t n_ent = 0;       // half of the singles, and every string's occupied orbitals
  };
  Side side[2];
  double *out = nullptr;     // sums of a call
  DevBuf mem;                // all of the above
};
void pairs_delete(PairLists *p) { delete p; }

// The lists are made in three launches for both spins, without a word from the device: a chunk of strings is counted
// by pair, the counts are summed over the chunks and then over the pairs, and each chunk's warp writes its strings'
// entries one string after the other, 32 lanes over its singles (which belong to different pairs).  The first property
// call of a handle then takes little longer than one that made no lists; with a warp per pair searching every string's
// singles, counts read back and five allocations, first calls of <S^2> took up to 1.5 ms more (14o 7a1b, 48 048
// determinants: 503 us without lists, 1974 so, 246 now; 9o 4a4b 143 / 205 / 114; CISD of 5a5b in 100 orbitals
// 175 / 89 / 9 ms).  A warp loads 128 singles at a time (CISD of 5a1b in 64 orbitals 1348 -> 1142 us).
struct PairBuild {
  const uint64_t *str[2], *str_hi[2];
  const int64_t *o1[2];
  const int32_t *J[2], *info[2];
  int64_t n[2];
  int chunks[2], per[2];  // chunks of `per` strings
  uint32_t *cnt[2];       // [chunk][pair]: entries, then those of the same pair in earlier chunks
  int64_t *off[2];
  uint2 *ent[2];
  int npair;
};
constexpr int PAIR_CHUNKS = 304;

__device__ __forceinline__ int pair_row(int q) {  // i of q = i (i + 1) / 2 + j, j <= i
  int i = (int)((sqrtf(8.0f * (float)q + 1.0f) - 1.0f) * 0.5f);
  while (i * (i + 1) / 2 > q) i--;
  while ((i + 1) * (i + 2) / 2 <= q) i++;
  return i;
}

// f(pair, string, partner, phase bit) for the entries of string I, lanes over its singles and its orbitals
template <typename F> __device__ __forceinline__ void pair_entries(const PairBuild &b, int sp, int64_t I, int lane, F &&f) {
  constexpr int U = 4;
  const int64_t end = b.o1[sp][I + 1];
  for (int64_t e = b.o1[sp][I] + lane; e < end; e += 32 * U) {
    int J[U], info[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      J[u] = e + 32 * u < end ? __ldg(b.J[sp] + e + 32 * u) : INT32_MAX;
      info[u] = e + 32 * u < end ? __ldg(b.info[sp] + e + 32 * u) : 0;
    }
#pragma unroll
    for (int u = 0; u < U; u++)
      if (J[u] < I) f(info[u] >> 1, (uint32_t)J[u], (uint32_t)(info[u] & 1));
  }
  const uint64_t m = b.str[sp][I], mh = hiword(b.str_hi[sp], I);
  for (int k = lane; k < 128; k += 32)
    if (occupied(m, mh, k)) f(k * (k + 3) / 2, (uint32_t)I, 0u);
}

__global__ void __launch_bounds__(128) pair_count_kernel(PairBuild b) {
  extern __shared__ uint32_t hist[];
  const int sp = blockIdx.y, c = blockIdx.x, lane = threadIdx.x & 31;
  if (c >= b.chunks[sp]) return;
  for (int q = threadIdx.x; q < b.npair; q += blockDim.x) hist[q] = 0;
  __syncthreads();
  const int64_t end = min(b.n[sp], (int64_t)(c + 1) * b.per[sp]);
  for (int64_t I = (int64_t)c * b.per[sp] + (threadIdx.x >> 5); I < end; I += blockDim.x >> 5)
    pair_entries(b, sp, I, lane, [&](int q, uint32_t, uint32_t) { atomicAdd(hist + q, 1u); });
  __syncthreads();
  for (int q = threadIdx.x; q < b.npair; q += blockDim.x) b.cnt[sp][(int64_t)c * b.npair + q] = hist[q];
}

// block per spin: counts to places
__global__ void __launch_bounds__(1024) pair_scan_kernel(PairBuild b) {
  __shared__ int64_t part[33];
  const int sp = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t base = 0;
  for (int q0 = 0; q0 < b.npair; q0 += blockDim.x) {
    const int q = q0 + threadIdx.x;
    int64_t total = 0;
    if (q < b.npair) {
      uint32_t *p = b.cnt[sp] + q;
      constexpr int U = 8;
      for (int c0 = 0; c0 < b.chunks[sp]; c0 += U) {
        uint32_t x[U];
#pragma unroll
        for (int u = 0; u < U; u++) x[u] = c0 + u < b.chunks[sp] ? p[(int64_t)(c0 + u) * b.npair] : 0u;
#pragma unroll
        for (int u = 0; u < U; u++) {
          if (c0 + u < b.chunks[sp]) p[(int64_t)(c0 + u) * b.npair] = (uint32_t)total;
          total += x[u];
        }
      }
    }
    int64_t inc = total;
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    __syncthreads();  // the last round's sums have been read
    if (lane == 31) part[warp + 1] = inc;
    if (threadIdx.x == 0) part[0] = 0;
    __syncthreads();
    if (threadIdx.x == 0)
      for (int w = 1; w <= 32; w++) part[w] += part[w - 1];
    __syncthreads();
    if (q < b.npair) b.off[sp][q] = base + part[warp] + inc - total;
    base += part[32];
  }
  if (threadIdx.x == 0) b.off[sp][b.npair] = base;
}

// warp per chunk
__global__ void __launch_bounds__(32) pair_fill_kernel(PairBuild b) {
  extern __shared__ int64_t next[];
  const int sp = blockIdx.y, c = blockIdx.x, lane = threadIdx.x;
  if (c >= b.chunks[sp]) return;
  for (int q = lane; q < b.npair; q += 32) next[q] = b.off[sp][q] + b.cnt[sp][(int64_t)c * b.npair + q];
  __syncwarp();
  const int64_t end = min(b.n[sp], (int64_t)(c + 1) * b.per[sp]);
  for (int64_t I = (int64_t)c * b.per[sp]; I < end; I++) {
    const uint64_t m = b.str[sp][I], mh = hiword(b.str_hi[sp], I);
    pair_entries(b, sp, I, lane, [&](int q, uint32_t J, uint32_t neg) {
      const uint32_t holds = J != (uint32_t)I && occupied(m, mh, pair_row(q));
      b.ent[sp][next[q]++] = make_uint2((uint32_t)I << 1 | neg, J << 1 | holds);
    });
    __syncwarp();
  }
}

__device__ __forceinline__ double xflip(double v, uint32_t neg) {
  return __hiloint2double(__double2hiint(v) ^ (int)(neg << 31), __double2loint(v));
}
__device__ __forceinline__ double warp_total(double x) {
  for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// pair that holds entry e of a list
__device__ __forceinline__ int pair_of(const int64_t *off, int npair, int64_t e) {
  int lo = 0, hi = npair;  // off[lo] <= e < off[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (off[mid] <= e)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

// Alpha 1-RDM: sum over the list of pair q of phase * (row I . row J), warp per ROWS_PER entries and part of the columns
constexpr int ROWS_PER = 8;
__global__ void __launch_bounds__(256) rdm_rows_kernel(const int64_t *off, const uint2 *ent, int npair, int64_t n_ent,
                                                       const int64_t *rowoff, const int32_t *rowlen, const double *C,
                                                       int width, double *out) {
  const int lane = threadIdx.x & 31, b0 = blockIdx.y * width;
  int64_t e = ((int64_t)blockIdx.x * 8 + (threadIdx.x >> 5)) * ROWS_PER;
  const int64_t e1 = min(e + ROWS_PER, n_ent);
  if (e >= e1) return;
  int q = pair_of(off, npair, e);
  while (e < e1) {
    while (off[q + 1] <= e) q++;
    double acc = 0.0;
    for (const int64_t stop = min(e1, off[q + 1]); e < stop; e++) {
      const uint2 x = __ldg(ent + e);
      const int64_t I = x.x >> 1, J = x.y >> 1;
      const double *ri = C + rowoff[I], *rj = C + rowoff[J];
      const int len = min(min(rowlen[I], rowlen[J]), b0 + width);
      double part = 0.0;
#pragma unroll 4
      for (int b = b0 + lane; b < len; b += 32) part = fma(__ldg(ri + b), __ldg(rj + b), part);
      acc += xflip(part, x.x & 1u);
    }
    acc = warp_total(acc);
    if (lane == 0 && acc != 0.0) atomicAdd(out + q, acc);
  }
}

// Beta 1-RDM: block per R rows, held in shared memory as [column][R] (R = 0: one row, read from global memory); the
// warps share the pairs.  A list is in the order of its larger column, so it ends at the longest row.
template <int R>
__global__ void __launch_bounds__(512) rdm_cols_kernel(const int64_t *off, const uint2 *ent, int npair, int64_t na,
                                                       const int64_t *rowoff, const int32_t *rowlen, const double *C,
                                                       double *out) {
  constexpr int RR = R == 0 ? 1 : R;
  extern __shared__ __align__(16) double xs[];
  const int64_t a0 = (int64_t)blockIdx.x * RR;
  int len[RR], longest = 0;
#pragma unroll
  for (int r = 0; r < RR; r++) {
    len[r] = a0 + r < na ? rowlen[a0 + r] : 0;
    longest = max(longest, len[r]);
  }
  if (R > 0) {
#pragma unroll
    for (int r = 0; r < RR; r++) {
      const double *row = C + (len[r] ? rowoff[a0 + r] : 0);
      for (int b = threadIdx.x; b < longest; b += blockDim.x) xs[b * RR + r] = b < len[r] ? row[b] : 0.0;
    }
    __syncthreads();
  }
  const double *x0 = R > 0 ? xs : C + rowoff[a0];
  const int lane = threadIdx.x & 31;
  for (int q = threadIdx.x >> 5; q < npair; q += blockDim.x >> 5) {
    double acc = 0.0;
    const int64_t e1 = off[q + 1];
    for (int64_t e = off[q]; e < e1; e += 32) {
      uint2 x = make_uint2(0u, 0u);
      bool in = e + lane < e1;
      if (in) x = __ldg(ent + e + lane);
      in = in && (int)(x.x >> 1) < longest;
      const int first = (int)(__shfl_sync(0xffffffffu, x.x, 0) >> 1);  // the smallest of the 32
      if (first >= longest) break;
      const int I = in ? (int)(x.x >> 1) : 0, J = in ? (int)(x.y >> 1) : 0;
#pragma unroll
      for (int r = 0; r < RR; r++)
        if (first < len[r]) {  // the same for the warp; a column past a shorter row reads the stored zero
          const double c = in ? xflip(x0[I * RR + r], x.x & 1u) : 0.0, d = in ? x0[J * RR + r] : 0.0;
          acc = fma(c, d, acc);
        }
    }
    acc = warp_total(acc);
    if (lane == 0 && acc != 0.0) atomicAdd(out + q, acc);
  }
}

// Beta 1-RDM with lists of a few entries: thread per entry, over the `per` rows of blockIdx.y; one atomic each
__global__ void __launch_bounds__(256) rdm_entries_kernel(const int64_t *off, const uint2 *ent, int npair, int64_t n_ent,
                                                          int64_t na, int per, const int64_t *rowoff, const int32_t *rowlen,
                                                          const double *C, double *out) {
  const int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (e >= n_ent) return;
  const uint2 x = __ldg(ent + e);
  const int I = (int)(x.x >> 1), J = (int)(x.y >> 1);  // J <= I
  const int64_t end = min(na, (int64_t)(blockIdx.y + 1) * per);
  double acc = 0.0;
#pragma unroll 4
  for (int64_t a = (int64_t)blockIdx.y * per; a < end; a++)
    if (I < __ldg(rowlen + a)) {
      const double *row = C + __ldg(rowoff + a);
      acc = fma(__ldg(row + I), __ldg(row + J), acc);
    }
  if (acc != 0.0) atomicAdd(out + pair_of(off, npair, e), xflip(acc, x.x & 1u));
}

// <S^2>, diagonal: sum of C_I^2 (s_z^2 + (n_alpha + n_beta)/2 - doubly occupied orbitals); block per alpha string
__global__ void __launch_bounds__(PROP_THREADS) s2_diag_kernel(const uint64_t *astr, const uint64_t *astr_hi,
                                                              const uint64_t *bstr, const uint64_t *bstr_hi,
                                                              const int64_t *rowoff, const int32_t *rowlen, double d0,
                                                              const double *C, int64_t ldc, int nvec, double *out) {
  __shared__ double red[PROP_THREADS / 32][S2_MAXV], dd[129];
  for (int k = threadIdx.x; k < 129; k += blockDim.x) dd[k] = d0 - k;
  __syncthreads();
  const int64_t ia = blockIdx.x, row = rowoff[ia];
  const uint64_t am = astr[ia], amh = hiword(astr_hi, ia);
  double acc[S2_MAXV];
#pragma unroll
  for (int v = 0; v < S2_MAXV; v++) acc[v] = 0.0;
  for (int b = threadIdx.x; b < rowlen[ia]; b += blockDim.x) {
    const double d = dd[popc2(am & bstr[b], amh & hiword(bstr_hi, b))];
#pragma unroll
    for (int v = 0; v < S2_MAXV; v++)
      if (v < nvec) {
        const double c = C[row + b + v * ldc];
        acc[v] = fma(c * c, d, acc[v]);
      }
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int v = 0; v < S2_MAXV; v++)
    if (v < nvec) {
      const double x = warp_total(acc[v]);
      if (lane == 0) red[w][v] = x;
    }
  __syncthreads();
  if ((int)threadIdx.x < nvec) {
    double x = 0.0;
    for (int i = 0; i < PROP_THREADS / 32; i++) x += red[i][threadIdx.x];
    if (x != 0.0) atomicAdd(out + threadIdx.x, x);
  }
}

// <S^2>, spin flips: each unordered pair of determinants (A_lo, B_hi), (A_hi, B_lo) of a pair of orbitals, where lo
// and hi are the strings that hold the lower and the higher of the two, adds -2 phase C C.  Warp per FLIP_PER alpha
// entries and part of the beta list of the same pair, lanes over that part.
constexpr int FLIP_PER = 4;
__global__ void __launch_bounds__(256) s2_flip_kernel(const int64_t *aoff, const uint2 *aent, const int64_t *boff,
                                                      const uint2 *bent, int npair, int64_t n_ent,
                                                      const int64_t *rowoff, const int32_t *rowlen, const double *C,
                                                      int64_t ldc, int nvec, double *out) {
  __shared__ double red[8][S2_MAXV];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double acc[S2_MAXV];
#pragma unroll
  for (int v = 0; v < S2_MAXV; v++) acc[v] = 0.0;
  int64_t e = ((int64_t)blockIdx.x * 8 + warp) * FLIP_PER;
  const int64_t e1 = min(e + FLIP_PER, n_ent);
  int q = e < e1 ? pair_of(aoff, npair, e) : 0;
  int i = 0;
  while ((i + 1) * (i + 2) / 2 <= q) i++;
  for (; e < e1; e++) {
    while (aoff[q + 1] <= e) {
      q++;
      if ((i + 1) * (i + 2) / 2 <= q) i++;
    }
    if (q == i * (i + 3) / 2) continue;  // i = j
    const uint2 x = __ldg(aent + e);
    const int I = (int)(x.x >> 1), J = (int)(x.y >> 1);
    const int alo = (x.y & 1u) ? J : I, ahi = (x.y & 1u) ? I : J;
    const int64_t rlo = rowoff[alo], rhi = rowoff[ahi];
    const int llo = rowlen[alo], lhi = rowlen[ahi];
    int64_t f0 = boff[q], f1 = boff[q + 1];
    if (gridDim.y > 1) {
      const int64_t width = ((f1 - f0 + gridDim.y - 1) / gridDim.y + 31) & ~31;
      f0 += blockIdx.y * width;
      f1 = min(f1, f0 + width);
    }
    for (int64_t f = f0 + lane; f < f1; f += 32) {
      const uint2 y = __ldg(bent + f);
      const int K = (int)(y.x >> 1), L = (int)(y.y >> 1);
      const int blo = (y.y & 1u) ? L : K, bhi = (y.y & 1u) ? K : L;
      if (bhi >= llo || blo >= lhi) continue;
#pragma unroll
      for (int v = 0; v < S2_MAXV; v++)
        if (v < nvec)
          acc[v] = fma(xflip(__ldg(C + rlo + bhi + v * ldc), (x.x ^ y.x) & 1u), __ldg(C + rhi + blo + v * ldc), acc[v]);
    }
  }
#pragma unroll
  for (int v = 0; v < S2_MAXV; v++)
    if (v < nvec) {
      const double s = warp_total(acc[v]);
      if (lane == 0) red[warp][v] = s;
    }
  __syncthreads();
  if ((int)threadIdx.x < nvec) {
    double s = 0.0;
    for (int w = 0; w < 8; w++) s += red[w][threadIdx.x];
    if (s != 0.0) atomicAdd(out + threadIdx.x, -2.0 * s);
  }
}

// the pair lists of a handle, made on the first property call
static pq_status pair_lists(pq_ci_handle *h) {
  if (h->pairs) return PQ_OK;
  std::unique_ptr<PairLists, void (*)(PairLists *)> p(new (std::nothrow) PairLists(), pairs_delete);
  if (!p) {
    set_error("host allocation failed");
    return PQ_ERR_OOM;
  }
  PairBuild b{};
  b.npair = h->npair[0];
  const int ne[2] = {h->desc.n_alpha[0], h->desc.n_beta[0]};
  int most = 0;
  for (int sp = 0; sp < 2; sp++) {
    const SpinTablesDev &t = h->tab[0][sp];
    b.str[sp] = t.str.as<uint64_t>(), b.str_hi[sp] = t.str_hi.as<uint64_t>();
    b.o1[sp] = t.s1_off.as<int64_t>(), b.J[sp] = t.s1_J.as<int32_t>(), b.info[sp] = t.s1_info.as<int32_t>();
    b.n[sp] = t.n_str;
    b.per[sp] = (int)std::max<int64_t>(8, (t.n_str + PAIR_CHUNKS - 1) / PAIR_CHUNKS);
    b.chunks[sp] = (int)((t.n_str + b.per[sp] - 1) / b.per[sp]);
    most = std::max(most, b.chunks[sp]);
    p->side[sp].n_ent = t.n1 / 2 + t.n_str * ne[sp];
  }
  auto lay = [&](DevLayout &l) {
    l.take(p->out, std::max(b.npair, S2_MAXV));
    for (int sp = 0; sp < 2; sp++) {
      l.take(p->side[sp].off, b.npair + 1);
      l.take(p->side[sp].ent, p->side[sp].n_ent + 1);
      l.take(b.cnt[sp], (size_t)b.chunks[sp] * b.npair);
    }
  };
  DevLayout l;
  lay(l);
  PQ_TRY(p->mem.alloc(l.used));
  l = DevLayout{static_cast<char *>(p->mem.ptr), 0};
  lay(l);
  for (int sp = 0; sp < 2; sp++) b.off[sp] = p->side[sp].off, b.ent[sp] = p->side[sp].ent;
  const size_t places = sizeof(int64_t) * b.npair;  // at most 66 KB
  if (places > 48 * 1024)
    PQ_CUDA_TRY(cudaFuncSetAttribute(pair_fill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)places));
  pair_count_kernel<<<dim3(most, 2), 128, sizeof(uint32_t) * b.npair, h->stream>>>(b);
  pair_scan_kernel<<<2, 1024, 0, h->stream>>>(b);
  pair_fill_kernel<<<dim3(most, 2), 32, places, h->stream>>>(b);
  PQ_CUDA_TRY(cudaGetLastError());
  h->pairs = std::move(p);
  return PQ_OK;
}

// Parts of the columns (or beta entries, `most` of them for an alpha entry): as many as fill the chip twice where the
// alpha entries alone leave it idle, of at least 64 columns each.  us a call, undivided / so: 16o 1a8b (136 alpha
// entries, 12 870 columns) <S^2> of four states 574 / 129, alpha 1-RDM 582 / 33; 20o 1a5b (210, 15 504) 544 / 154,
// 688 / 41; also full CI 10o 5a5b, alpha 1-RDM 41 / 28.  A part is one range: with 32 columns in turn the loops of an
// undivided call had a stride that is not known when they are compiled, and FCI(12o) took 378 us instead of 362.
static unsigned column_parts(int64_t blocks, int64_t most) {
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>((most + 63) / 64, 304 / std::max<int64_t>(blocks, 1)));
}

// <S^2> of nvec <= S2_MAXV states into device sums; lists: NULL without particles of either spin, which cannot flip
static pq_status s2_one(pq_ci_handle *h, const PairLists *lists, const double *C, int64_t ldc, int nvec, double *out) {
  const SpinTablesDev &A = h->tab[0][0], &B = h->tab[0][1];
  const int npair = h->npair[0], na = h->desc.n_alpha[0], nb = h->desc.n_beta[0];
  cudaStream_t st = h->stream;
  const double sz = 0.5 * (na - nb);
  PQ_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(double) * S2_MAXV, st));
  s2_diag_kernel<<<(unsigned)A.n_str, PROP_THREADS, 0, st>>>(
      A.str.as<uint64_t>(), A.str_hi.as<uint64_t>(), B.str.as<uint64_t>(), B.str_hi.as<uint64_t>(),
      h->d_rowoff.as<int64_t>(), h->d_rowlen.as<int32_t>(), sz * sz + 0.5 * (na + nb), C, ldc, nvec, out);
  if (lists) {
    const PairLists::Side &a = lists->side[0], &b = lists->side[1];
    const int64_t blocks = (a.n_ent + 8 * FLIP_PER - 1) / (8 * FLIP_PER);
    s2_flip_kernel<<<dim3((unsigned)blocks, column_parts(blocks, b.n_ent / npair)), 256, 0, st>>>(
        a.off, a.ent, b.off, b.ent, npair, a.n_ent, h->d_rowoff.as<int64_t>(), h->d_rowlen.as<int32_t>(), C, ldc, nvec, out);
  }
  PQ_CUDA_TRY(cudaGetLastError());
  return PQ_OK;
}

// 1-RDM sums by pair into the device sums of the lists
static pq_status rdm_one(pq_ci_handle *h, const double *C, int spin) {
  const PairLists &p = *h->pairs;
  const int npair = h->npair[0];
  cudaStream_t st = h->stream;
  double *out = p.out;
  const int64_t *ro = h->d_rowoff.as<int64_t>();
  const int32_t *rl = h->d_rowlen.as<int32_t>();
  PQ_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(double) * npair, st));
  const int64_t *off = p.side[spin].off;
  const uint2 *ent = p.side[spin].ent;
  const int64_t n_ent = p.side[spin].n_ent, na = h->tab[0][0].n_str;
  if (n_ent == 0) return PQ_OK;
  if (spin == 0) {
    const int64_t blocks = (n_ent + 8 * ROWS_PER - 1) / (8 * ROWS_PER);
    const int64_t nb = h->tab[0][1].n_str;
    const dim3 grid((unsigned)blocks, column_parts(blocks, nb));
    const int width = (int)((nb + grid.y - 1) / grid.y + 31) & ~31;
    rdm_rows_kernel<<<grid, 256, 0, st>>>(off, ent, npair, n_ent, ro, rl, C, width, out);
    PQ_CUDA_TRY(cudaGetLastError());
    return PQ_OK;
  }
  // With few entries a pair, a warp per pair idles and the blocks' sums meet in the same few atomics.  us a call, thread
  // per determinant (before there were lists) / warp per pair / thread per entry: 30o 4a1b (1 entry a pair, 465 pairs)
  // 556 / 1367 / 68; 40o 2a1b (1, 820 pairs) 109 / 229 / 48; 20o 3a1b (1) 84 / 109 / 47; 16o 8a2b (14) 1059 / 233 / 127;
  // 30o 2a2b (28) 300 / 117 / 76; CISD of 40o 2a2b (38, 820 pairs) 177 / 209 / 102; but 9o 4a4b (39, 45 pairs) 98 / 50 /
  // 59; 10o 5a5b (80) 154 / 53 / 104.
  if (n_ent < (npair >= 256 ? 64 : 32) * (int64_t)npair) {
    const int64_t blocks = (n_ent + 255) / 256;
    const int64_t chunks = std::min<int64_t>((na + 7) / 8, std::max<int64_t>(1, 1216 / blocks));
    const int per = (int)((na + chunks - 1) / chunks);
    rdm_entries_kernel<<<dim3((unsigned)blocks, (unsigned)((na + per - 1) / per)), 256, 0, st>>>(off, ent, npair, n_ent, na,
                                                                                               per, ro, rl, C, out);
    PQ_CUDA_TRY(cudaGetLastError());
    return PQ_OK;
  }
  // as many rows per block as 100 KB of shared memory hold, while the blocks still cover the chip twice
  const int64_t longest = *std::max_element(h->rowlen.begin(), h->rowlen.end());
  const size_t row = sizeof(double) * (size_t)longest;
  auto run = [&](auto kern, int R) -> pq_status {
    const size_t smem = row * R;
    if (smem > 48 * 1024) PQ_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int64_t rows = std::max(R, 1);
    kern<<<(unsigned)((na + rows - 1) / rows), 512, smem, st>>>(off, ent, npair, na, ro, rl, C, out);
    PQ_CUDA_TRY(cudaGetLastError());
    return PQ_OK;
  };
  if (8 * row <= 100 * 1024 && na >= 8 * 304) return run(rdm_cols_kernel<8>, 8);
  if (4 * row <= 100 * 1024 && na >= 4 * 304) return run(rdm_cols_kernel<4>, 4);
  if (2 * row <= 200 * 1024) return run(rdm_cols_kernel<2>, 2);
  if (row <= 200 * 1024) return run(rdm_cols_kernel<1>, 1);
  return run(rdm_cols_kernel<0>, 0);
}

// ---- two species: determinant (a0, b0, a1, b1) of the product space built
// by ci_two.cu (species-0 prefix rows x per-level species-1 blocks)
struct TwoAddr {
  const int32_t *e_a, *e_b, *elev, *rowoff0, *rowlen0, *prowoff, *prowlen, *pdet_a, *pdet_b;
  const int64_t *ebase, *pfirst, *psize;
  int npa1;
  const uint64_t *str[2][2], *str_hi[2][2];  // str_hi: orbitals 64..127 (NULL for one-word strings)
  const int64_t *s1_off[2][2];
  const int32_t *s1_J[2][2], *s1_info[2][2];
};

__device__ __forceinline__ int64_t two_lookup(const TwoAddr &t, int a0, int b0, int a1, int b1) {
  if (b0 >= t.rowlen0[a0]) return -1;
  const int ie = t.rowoff0[a0] + b0;
  const int L = t.elev[ie];
  if (L < 0) return -1;
  const int64_t r = (int64_t)L * t.npa1 + a1;
  if (b1 >= t.prowlen[r]) return -1;
  return t.ebase[ie] + t.prowoff[r] + b1;
}

// CTA per species-0 pair ie, threads over its species-1 block
__global__ void __launch_bounds__(PROP_THREADS) s2_two_kernel(TwoAddr t, int sp, const double *C, int64_t ldc,
                                                              int nvec, double *out) {
  __shared__ double red[S2_MAXV][PROP_THREADS / 32];
  const int ie = blockIdx.x;
  double acc[S2_MAXV];
#pragma unroll
  for (int v = 0; v < S2_MAXV; v++) acc[v] = 0.0;
  const int L = t.elev[ie];
  const int64_t nq = L < 0 ? 0 : t.psize[L];
  for (int64_t q = threadIdx.x; q < nq; q += blockDim.x) {
    int d[4] = {t.e_a[ie], t.e_b[ie], t.pdet_a[t.pfirst[L] + q], t.pdet_b[t.pfirst[L] + q]};
    const int64_t I = t.ebase[ie] + q;
    const int ia = d[2 * sp], ib = d[2 * sp + 1];
    const uint64_t am = t.str[sp][0][ia], bm = t.str[sp][1][ib];
    const uint64_t amh = hiword(t.str_hi[sp][0], ia), bmh = hiword(t.str_hi[sp][1], ib);
    double cI[S2_MAXV];
#pragma unroll
    for (int v = 0; v < S2_MAXV; v++) cI[v] = v < nvec ? C[I + v * ldc] : 0.0;
    const uint64_t open = am ^ bm, openh = amh ^ bmh;
    const int n_open = popc2(open, openh), n_a = popc2(open & am, openh & amh);
    const double sz = n_a - 0.5 * n_open;
    const double dg = n_a + sz * (sz - 1.0);
#pragma unroll
    for (int v = 0; v < S2_MAXV; v++) acc[v] += cI[v] * cI[v] * dg;
    const int64_t a1b = t.s1_off[sp][0][ia], b1b = t.s1_off[sp][1][ib];
    const int n1a = (int)(t.s1_off[sp][0][ia + 1] - a1b), n1b = (int)(t.s1_off[sp][1][ib + 1] - b1b);
    for (int s = 0; s < n1a; s++) {
      const int Ja = t.s1_J[sp][0][a1b + s], infa = t.s1_info[sp][0][a1b + s];
      const uint64_t jam = t.str[sp][0][Ja], jamh = hiword(t.str_hi[sp][0], Ja);
      const int ha = first_set(am & ~jam, amh & ~jamh), pa = first_set(jam & ~am, jamh & ~amh);
      if (!occupied(bm, bmh, pa) || occupied(bm, bmh, ha)) continue;
      uint64_t jbm = bm, jbmh = bmh;
      flip_orb(jbm, jbmh, pa);
      flip_orb(jbm, jbmh, ha);
      for (int q2 = 0; q2 < n1b; q2++) {
        const int Jb = t.s1_J[sp][1][b1b + q2];
        if (t.str[sp][1][Jb] != jbm || hiword(t.str_hi[sp][1], Jb) != jbmh) continue;
        int e[4] = {d[0], d[1], d[2], d[3]};
        e[2 * sp] = Ja;
        e[2 * sp + 1] = Jb;
        const int64_t J = two_lookup(t, e[0], e[1], e[2], e[3]);
        if (J >= 0) {
          const double ph = ((infa ^ t.s1_info[sp][1][b1b + q2]) & 1) ? -1.0 : 1.0;
#pragma unroll
          for (int v = 0; v < S2_MAXV; v++)
            if (v < nvec) acc[v] -= ph * cI[v] * C[J + v * ldc];
        }
        break;
      }
    }
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int v = 0; v < S2_MAXV; v++) {
    double x = acc[v];
    for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0) red[v][w] = x;
  }
  __syncthreads();
  if (threadIdx.x < nvec) {
    double x = 0.0;
    for (int i = 0; i < PROP_THREADS / 32; i++) x += red[threadIdx.x][i];
    atomicAdd(out + threadIdx.x, x);
  }
}

__global__ void __launch_bounds__(PROP_THREADS) rdm1_two_kernel(TwoAddr t, int sp, int spin, int n, const double *C,
                                                                double *rdm) {
  extern __shared__ double acc[];  // n x n
  for (int i = threadIdx.x; i < n * n; i += blockDim.x) acc[i] = 0.0;
  __syncthreads();
  const int ie = blockIdx.x;
  const int L = t.elev[ie];
  const int64_t nq = L < 0 ? 0 : t.psize[L];
  for (int64_t q = threadIdx.x; q < nq; q += blockDim.x) {
    int d[4] = {t.e_a[ie], t.e_b[ie], t.pdet_a[t.pfirst[L] + q], t.pdet_b[t.pfirst[L] + q]};
    const int64_t I = t.ebase[ie] + q;
    const double cI = C[I];
    const int si = d[2 * sp + spin];
    const uint64_t mine = t.str[sp][spin][si], mineh = hiword(t.str_hi[sp][spin], si);
    const double c2 = cI * cI;
    if (fabs(c2) > 1e-16) for_occ(mine, mineh, [&](int o) { atomicAdd(acc + o * (n + 1), c2); });
    const int64_t b = t.s1_off[sp][spin][si];
    const int ns = (int)(t.s1_off[sp][spin][si + 1] - b);
    for (int s = 0; s < ns; s++) {
      const int Js = t.s1_J[sp][spin][b + s], info = t.s1_info[sp][spin][b + s];
      int e[4] = {d[0], d[1], d[2], d[3]};
      e[2 * sp + spin] = Js;
      const int64_t J = two_lookup(t, e[0], e[1], e[2], e[3]);
      if (J < 0 || J > I) continue;  // each pair once, from the later determinant
      const double c = ((info & 1) ? -cI : cI) * C[J];
      if (fabs(c) <= 1e-16) continue;
      const uint64_t jm = t.str[sp][spin][Js], jmh = hiword(t.str_hi[sp][spin], Js);
      const int k = first_set(mine & ~jm, mineh & ~jmh), l = first_set(jm & ~mine, jmh & ~mineh);
      atomicAdd(acc + k + l * n, c);
      atomicAdd(acc + l + k * n, c);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n * n; i += blockDim.x)
    if (acc[i] != 0.0) atomicAdd(rdm + i, acc[i]);
}

static TwoAddr make_two(const pq_ci_handle *h) {
  TwoAddr t{};
  t.e_a = h->d_e_a.as<int32_t>();
  t.e_b = h->d_e_b.as<int32_t>();
  t.elev = h->d_elev.as<int32_t>();
  t.rowoff0 = h->d_rowoff.as<int32_t>();
  t.rowlen0 = h->d_rowlen.as<int32_t>();
  t.prowoff = h->d_prowoff.as<int32_t>();
  t.prowlen = h->d_prowlen.as<int32_t>();
  t.pdet_a = h->d_pdet_a.as<int32_t>();
  t.pdet_b = h->d_pdet_b.as<int32_t>();
  t.ebase = h->d_ebase.as<int64_t>();
  t.pfirst = h->d_pfirst.as<int64_t>();
  t.psize = h->d_psize.as<int64_t>();
  t.npa1 = (int)h->str[1][0].size();
  for (int s = 0; s < 2; s++)
    for (int sp = 0; sp < 2; sp++) {
      t.str[s][sp] = h->tab[s][sp].str.as<uint64_t>();
      t.str_hi[s][sp] = h->tab[s][sp].str_hi.as<uint64_t>();
      t.s1_off[s][sp] = h->tab[s][sp].s1_off.as<int64_t>();
      t.s1_J[s][sp] = h->tab[s][sp].s1_J.as<int32_t>();
      t.s1_info[s][sp] = h->tab[s][sp].s1_info.as<int32_t>();
    }
  return t;
}


}  // namespace pq

using namespace pq;

extern "C" {

pq_status pq_ci_s2(pq_ci_handle *h, const double *C, int64_t ldc, int32_t nvec, double *s2) {
  clear_error();
  if (!h || !C || !s2 || nvec < 1 || ldc < (h ? h->n_dets : 0)) {
    set_error("pq_ci_s2: bad arguments");
    return PQ_ERR_ARG;
  }
  const int ns = h->n_species;
  const bool flips = ns == 1 && h->desc.n_alpha[0] > 0 && h->desc.n_beta[0] > 0;
  DevBuf own;
  if (flips)
    PQ_TRY(with_room(h, [&] { return pair_lists(h); }));
  else
    PQ_TRY(own.alloc(sizeof(double) * S2_MAXV));
  const PairLists *lists = flips ? h->pairs.get() : nullptr;
  double *out = flips ? lists->out : own.as<double>();
  std::vector<double> part(S2_MAXV);
  for (int sp = 0; sp < ns; sp++)
    for (int v0 = 0; v0 < nvec; v0 += S2_MAXV) {
      const int c = std::min(S2_MAXV, nvec - v0);
      if (ns == 1) {
        PQ_TRY(s2_one(h, lists, C + (size_t)v0 * ldc, ldc, c, out));
      } else {
        PQ_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(double) * S2_MAXV, h->stream));
        s2_two_kernel<<<(unsigned)h->e_a.size(), PROP_THREADS, 0, h->stream>>>(make_two(h), sp, C + (size_t)v0 * ldc,
                                                                               ldc, c, out);
        PQ_CUDA_TRY(cudaGetLastError());
      }
      PQ_CUDA_TRY(cudaMemcpyAsync(part.data(), out, sizeof(double) * c, cudaMemcpyDeviceToHost, h->stream));
      PQ_CUDA_TRY(cudaStreamSynchronize(h->stream));
      for (int v = 0; v < c; v++) s2[(size_t)(v0 + v) * ns + sp] = part[v];
    }
  return PQ_OK;
}

pq_status pq_ci_rdm1(pq_ci_handle *h, const double *C, int32_t species, int32_t spin, double *rdm) {
  clear_error();
  if (!h || !C || !rdm || spin < 0 || spin > 1 || species < 0 || species >= h->n_species) {
    set_error("pq_ci_rdm1: bad arguments");
    return PQ_ERR_ARG;
  }
  const int n = h->n_orb[species];
  if (h->n_species == 1) {
    PQ_TRY(with_room(h, [&] { return pair_lists(h); }));
    PQ_TRY(rdm_one(h, C, spin));
    std::vector<double> d(h->npair[0]);
    PQ_CUDA_TRY(cudaMemcpyAsync(d.data(), h->pairs->out, sizeof(double) * d.size(), cudaMemcpyDeviceToHost, h->stream));
    PQ_CUDA_TRY(cudaStreamSynchronize(h->stream));
    for (int i = 0, q = 0; i < n; i++)
      for (int j = 0; j <= i; j++, q++) rdm[i + (size_t)j * n] = rdm[j + (size_t)i * n] = d[q];
    return PQ_OK;
  }
  DevBuf out;
  PQ_TRY(out.alloc(sizeof(double) * n * n));
  PQ_CUDA_TRY(cudaMemsetAsync(out.ptr, 0, sizeof(double) * n * n, h->stream));
  const size_t smem = sizeof(double) * n * n;
  if (smem > 48 * 1024)
    PQ_CUDA_TRY(cudaFuncSetAttribute(rdm1_two_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  rdm1_two_kernel<<<(unsigned)h->e_a.size(), PROP_THREADS, smem, h->stream>>>(make_two(h), species, spin, n, C,
                                                                             out.as<double>());
  PQ_CUDA_TRY(cudaGetLastError());
  PQ_CUDA_TRY(cudaMemcpyAsync(rdm, out.ptr, sizeof(double) * n * n, cudaMemcpyDeviceToHost, h->stream));
  PQ_CUDA_TRY(cudaStreamSynchronize(h->stream));
  return PQ_OK;
}

}  // extern "C"
