// FP64 sigma = H C of a two-species full product space with small string lists, on the tcgen05 tensor cores.
//
// Reference: sigma_two_species_class_singleshot (src/ci/detset/direct_mixedparticle.cpp:269-611), cross elements
// src/ci/detset/slater_condon_mixedparticle.cpp:4-236.  The kernel of ci_two.cu gathers every connection on the FP64
// pipe and is bound by it.  Each off-diagonal element of H moves strings of at most two of the four lists, so
//   H = diagonal + sum over pairs (x, y) of lists of H_xy (x) 1,
// where H_xy holds the moves of x alone and of y alone (their own part with one pair of each list, the Coulomb field
// of the other list with every pair) and the single x single moves of both.  With a few dozen strings in a list (one
// or two particles of either kind) H_xy is a matrix of at most 8192 rows that is mostly filled, and
//   sigma[x', y', rest] += sum_{x, y} H_xy[x' y'][x y] C[x, y, rest]
// is a dense GEMM with the strings of the other lists and the roots as columns.  It runs by exact digit products
// (ci_dense64.cuh): C is split once per pair into rows (root, rest) of K = (x, y), every pair writes its own copy of
// sigma (one per part of a split K range, so that few tiles still fill the chip), and a last pass adds the copies and
// the FP64 diagonal term in a fixed order.
//
// Non-finite input and a wait that runs out raise a device flag; the kernel of ci_two.cu is launched behind with that
// flag as its condition and then computes the whole result.
//
// Measured: positronium hydride in 60 + 40 orbitals (144 000 determinants, 8 240 connections each), three roots,
// 495 us a sigma against 7572 (one root 239 / 4485).  Bound: the drain of ss64_kernel after every 64 K values.
#include <algorithm>
#include <cstdlib>
#include <memory>
#include <new>
#include <vector>

#include "ci_dense64.cuh"
#include "pq_bits.cuh"

namespace pq {

struct Two64 {
  struct Pair {
    int x = 0, y = 1;                // lists (species-0 alpha, beta, species-1 alpha, beta)
    int64_t M = 0, np = 0;           // rows, row length
    unsigned short *d = nullptr;     // digits of H_xy
    int win = 2;
  };
  std::vector<Pair> pairs;
  uint32_t *hi = nullptr;            // high word of max|H_xy| per pair
  int *aux = nullptr;                // gate; high words of max|C| from word 4 on
  DevBuf mem, work;                  // the matrices and these words; digits and copies of a call
  int sms = 0;
  size_t bytes() const { return mem.bytes + work.bytes; }
};
void two64_delete(Two64 *t) { delete t; }

namespace two64 {

using namespace s64;

struct List {
  const int64_t *o1, *o2;
  const int32_t *J1, *info1, *J2;
  const double *F1, *D2;
  const uint64_t *str;
};

struct Shape {
  int n[4];       // strings of each list
  int64_t st[4];  // determinant index step of each list
};

// Row m' = (x', y') of a pair matrix without its diagonal.  FILL = false: largest magnitude.  FILL: digits, and the
// largest number of entries in windows of 2, 4, 8, 16 chunks.
template <bool FILL>
__global__ void __launch_bounds__(256) pair_kernel(List x, List y, int ny, bool own_x, bool own_y, const double *W, int ldw,
                                                   int64_t M, int64_t np, int chunks, uint32_t *hi, unsigned short *d, int *wmax) {
  extern __shared__ int cnt[];
  const int64_t row = blockIdx.x;
  const int xs = (int)(row / ny), ys = (int)(row - (int64_t)xs * ny);
  const int e = FILL ? plane_exp(hi) : 0;
  uint32_t top = 0;
  if (FILL) {
    for (int c = threadIdx.x; c < chunks; c += blockDim.x) cnt[c] = 0;
    __syncthreads();
  }
  auto put = [&](int xj, int yj, double v) {
    const int64_t m = (int64_t)xj * ny + yj;
    if (!FILL) {
      top = max(top, (uint32_t)__double2hiint(v) & 0x7fffffffu);
      return;
    }
    atomicAdd(cnt + m / 32, 1);
    if (e == digits::BAD) return;
    unsigned short h[dg::N];
    dg::to_half(digits::fixed_point<dg::BITS>(v, e), h);
#pragma unroll
    for (int i = 0; i < dg::N; i++) d[((int64_t)i * M + row) * np + m] = h[i];
  };
  const int64_t x0 = x.o1[xs], x1 = x.o1[xs + 1], y0 = y.o1[ys], y1 = y.o1[ys + 1];
  for (int64_t a = x0 + threadIdx.x; a < x1; a += blockDim.x) {
    double v = own_x ? x.F1[a] : 0.0;
    for_occ(y.str[ys], 0, [&](int k) { v += W[(int64_t)(x.info1[a] >> 1) * ldw + k * (k + 3) / 2]; });
    put(x.J1[a], ys, (x.info1[a] & 1) ? -v : v);
  }
  for (int64_t b = y0 + threadIdx.x; b < y1; b += blockDim.x) {
    double v = own_y ? y.F1[b] : 0.0;
    for_occ(x.str[xs], 0, [&](int k) { v += W[(int64_t)(k * (k + 3) / 2) * ldw + (y.info1[b] >> 1)]; });
    put(xs, y.J1[b], (y.info1[b] & 1) ? -v : v);
  }
  if (own_x)
    for (int64_t a = x.o2[xs] + threadIdx.x; a < x.o2[xs + 1]; a += blockDim.x) put(x.J2[a], ys, x.D2[a]);
  if (own_y)
    for (int64_t b = y.o2[ys] + threadIdx.x; b < y.o2[ys + 1]; b += blockDim.x) put(xs, y.J2[b], y.D2[b]);
  const int64_t nb = y1 - y0, n = (x1 - x0) * nb;
  for (int64_t t = threadIdx.x; t < n; t += blockDim.x) {
    const int64_t a = x0 + t / nb, b = y0 + t % nb;
    const double v = W[(int64_t)(x.info1[a] >> 1) * ldw + (y.info1[b] >> 1)];
    put(x.J1[a], y.J1[b], ((x.info1[a] ^ y.info1[b]) & 1) ? -v : v);
  }
  if (!FILL) {
    top = __reduce_max_sync(0xffffffffu, top);
    if ((threadIdx.x & 31) == 0) atomicMax(hi, top);
    return;
  }
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

__global__ void __launch_bounds__(256) absmax_vectors_kernel(const double *C, int64_t es, int64_t vs, int64_t n, uint32_t *hi) {
  const double *c = C + (int64_t)blockIdx.y * vs;
  uint32_t m = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    m = max(m, (uint32_t)__double2hiint(c[i * es]) & 0x7fffffffu);
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) atomicMax(hi + blockIdx.y, m);
}

// the strings of the two lists besides x and y, in their order
__device__ __forceinline__ void others(int x, int y, int &u, int &w) {
  u = x == 0 ? (y == 1 ? 2 : 1) : 0;
  w = y == 3 ? (x == 2 ? 1 : 2) : 3;
}

// digit rows (root v, rest r) of K = (x, y): block per row
__global__ void __launch_bounds__(256) pair_digits_kernel(const double *C, int64_t es, int64_t vs, Shape sh, int x, int y,
                                                          int64_t M, int64_t np, int64_t R, int nv, const uint32_t *xhi,
                                                          const uint32_t *hi, int npairs, unsigned short *xd, int *gate) {
  const int64_t n = blockIdx.x;
  const int v = (int)(n / R);
  const int64_t r = n - (int64_t)v * R;
  const int e = plane_exp(xhi + v);
  bool bad = e == digits::BAD;
  for (int p = 0; p < npairs; p++) bad = bad || plane_exp(hi + p) == digits::BAD;
  if (bad) {
    if (threadIdx.x == 0) *gate = 1;
    return;
  }
  int u, w;
  others(x, y, u, w);
  const double *c = C + v * vs + ((r / sh.n[w]) * sh.st[u] + (r % sh.n[w]) * sh.st[w]) * es;
  const int64_t plane = (int64_t)nv * R * np;
  for (int64_t m = threadIdx.x; m < M; m += blockDim.x) {
    const double z = c[((m / sh.n[y]) * sh.st[x] + (m % sh.n[y]) * sh.st[y]) * es];
    unsigned short h[dg::N];
    dg::to_half(digits::fixed_point<dg::BITS>(z, e), h);
#pragma unroll
    for (int i = 0; i < dg::N; i++) xd[i * plane + n * np + m] = h[i];
  }
}

struct Parts {
  const double *p[6];
  int x[6], y[6], ksplit[6];
  int64_t M[6], R[6], part[6];
  int npairs;
};

// sigma = (diagonal - shift) C + the pairs' copies
__global__ void __launch_bounds__(256) sum_kernel(const double *C, int64_t es, int64_t vs, Shape sh, Parts q, int64_t n,
                                                  const double *diag, double shift, double *S, int64_t ses, int64_t svs,
                                                  const int *gate) {
  if (*gate) return;
  const int64_t I = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int v = blockIdx.y;
  if (I >= n) return;
  int t[4];
  int64_t k = I;
#pragma unroll
  for (int s = 3; s >= 0; s--) {
    t[s] = (int)(k % sh.n[s]);
    k /= sh.n[s];
  }
  double x = (diag[I] - shift) * C[v * vs + I * es];
  for (int p = 0; p < q.npairs; p++) {
    int u, w;
    others(q.x[p], q.y[p], u, w);
    const int64_t m = (int64_t)t[q.x[p]] * sh.n[q.y[p]] + t[q.y[p]], r = (int64_t)t[u] * sh.n[w] + t[w];
    const double *o = q.p[p] + (v * q.R[p] + r) * q.M[p] + m;
    for (int z = 0; z < q.ksplit[p]; z++) x += o[z * q.part[p]];
  }
  S[v * svs + I * ses] = x;
}

static List list_of(const pq_ci_handle *h, int s) {
  const SpinTablesDev &t = h->tab[s >> 1][s & 1];
  return {t.s1_off.as<int64_t>(), t.s2_off.as<int64_t>(), t.s1_J.as<int32_t>(), t.s1_info.as<int32_t>(), t.s2_J.as<int32_t>(),
          t.s1_F64.as<double>(),  t.s2_D64.as<double>(),  t.str.as<uint64_t>()};
}

static Shape shape_of(const pq_ci_handle *h) {
  Shape s{};
  for (int i = 0; i < 4; i++) s.n[i] = (int)h->str[i >> 1][i & 1].size();
  s.st[3] = 1;
  for (int i = 2; i >= 0; i--) s.st[i] = s.st[i + 1] * s.n[i + 1];
  return s;
}

}  // namespace two64

// Full products whose lists of more than one string pair up to at most 8192 rows, up to 16 M determinants (copies and
// digits take some 150 B per determinant, root and pair).  A row of a pair matrix costs 34 digit products of one K value,
// a connection half a clock of an SM's FP64 pipe, and a pair some 25 us of launches and of a chip that is not full.
// us a sigma of three roots, this path / the element kernel: 864 determinants of 258 connections in three pairs
// 100 / 110, 4 000 of 740 146 / 301, 18 000 of 2 020 170 / 787; four lists, 82 944 of 721 (3.5 rows a connection)
// 301 / 463, but 640 / 415 with the matrices that its first call makes; 36 504 of 863 (8.1 rows a connection) 357 / 351.
// With four lists the six products are smaller, and rows that stand for few connections weigh more; one / three roots:
// 19 200 of 405 (2.3 rows a connection, 1.3e6 connections a pair) 208 / 154, 238 / 190; 22 400 of 559 (1.9, 2.1e6)
// 230 / 196, 260 / 255; 22 050 of 545 (2.3, 2.0e6) 254 / 195, 281 / 246; 12 544 of 622 (1.1, 1.3e6) 206 / 212, 229 / 258;
// 19 600 of 903 (1.1, 3.0e6) 247 / 307, 267 / 381.
bool two64_applicable(const pq_ci_handle *h) {
  if (h->n_species != 2 || !h->full2 || h->wide || h->n_dets > (16 << 20)) return false;
  double rows = 0.0, conn = 0.0;
  int npairs = 0;
  const int ne[4] = {h->desc.n_alpha[0], h->desc.n_beta[0], h->desc.n_alpha[1], h->desc.n_beta[1]};
  for (int x = 0; x < 4; x++) {
    const SpinTablesDev &a = h->tab[x >> 1][x & 1];
    if (a.n_str == 1 && ne[x] != 0) return false;  // a filled list still acts on the others
    conn += a.max1 + a.max2;
    for (int y = x + 1; y < 4; y++) {
      const SpinTablesDev &b = h->tab[y >> 1][y & 1];
      if (a.n_str < 2 || b.n_str < 2) continue;
      const int64_t M = a.n_str * b.n_str;
      if (M > 8192) return false;
      rows += (double)M;
      conn += (double)a.max1 * b.max1;
      npairs++;
    }
  }
  if (npairs == 0) return false;
  if (getenv("PQ_TWO64_ALWAYS")) return true;  // tests of small spaces, read when a handle is created
  const double least = npairs == 6 ? std::max(6e5, 1e6 * (rows / conn) * (rows / conn)) : 6e5;
  return rows <= 2.5 * conn && (double)h->n_dets * conn >= least * npairs;
}

size_t two64_bytes(const pq_ci_handle *h) { return h->two64 ? h->two64->bytes() : 0; }

static pq_status two64_prepare(pq_ci_handle *h) {
  using namespace two64;
  if (h->two64) return PQ_OK;
  std::unique_ptr<Two64, void (*)(Two64 *)> T(new (std::nothrow) Two64(), two64_delete);
  if (!T) {
    set_error("host allocation failed");
    return PQ_ERR_OOM;
  }
  cudaStream_t st = h->stream;
  const Shape sh = shape_of(h);
  for (int x = 0; x < 4; x++)
    for (int y = x + 1; y < 4; y++)
      if (sh.n[x] > 1 && sh.n[y] > 1) {
        Two64::Pair p;
        p.x = x, p.y = y;
        p.M = (int64_t)sh.n[x] * sh.n[y];
        p.np = up64(p.M, 64);
        T->pairs.push_back(p);
      }
  const int npairs = (int)T->pairs.size();
  int *wmax = nullptr;
  auto lay = [&](DevLayout &l) {
    l.take(T->hi, 8);
    l.take(T->aux, 16);
    l.take(wmax, 4 * npairs);
    for (Two64::Pair &p : T->pairs) l.take(p.d, (size_t)dg::N * p.M * p.np);
  };
  DevLayout l;
  lay(l);
  PQ_TRY(T->mem.alloc(l.used));
  l = DevLayout{static_cast<char *>(T->mem.ptr), 0};
  lay(l);
  PQ_CUDA_TRY(cudaMemsetAsync(T->mem.ptr, 0, l.used, st));
  bool owned[4] = {false, false, false, false};
  for (int i = 0; i < npairs; i++) {
    const Two64::Pair &p = T->pairs[i];
    const int x = p.x, y = p.y, ldw = h->npair[y >> 1], chunks = (int)((p.M + 31) / 32);
    const bool ox = !owned[x], oy = !owned[y];  // a list's own moves belong to one pair
    owned[x] = owned[y] = true;
    const double *W = (x >> 1) == (y >> 1) ? h->d_eabs64[x >> 1].as<double>() : h->d_epc64[x & 1][y & 1].as<double>();
    const List lx = list_of(h, x), ly = list_of(h, y);
    pair_kernel<false><<<(unsigned)p.M, 256, 0, st>>>(lx, ly, sh.n[y], ox, oy, W, ldw, p.M, p.np, chunks, T->hi + i, nullptr,
                                                    nullptr);
    pair_kernel<true><<<(unsigned)p.M, 256, chunks * sizeof(int), st>>>(lx, ly, sh.n[y], ox, oy, W, ldw, p.M, p.np, chunks,
                                                                       T->hi + i, p.d, wmax + 4 * i);
    PQ_CUDA_TRY(cudaGetLastError());
  }
  std::vector<int> wm(4 * npairs);
  PQ_CUDA_TRY(cudaMemcpyAsync(wm.data(), wmax, wm.size() * sizeof(int), cudaMemcpyDeviceToHost, st));
  PQ_CUDA_TRY(cudaStreamSynchronize(st));
  for (int i = 0; i < npairs; i++)
    for (int k = 1; k < 4; k++)
      if (wm[4 * i + k] <= KMAX) T->pairs[i].win = 2 << k;
  int dev = 0;
  PQ_CUDA_TRY(cudaGetDevice(&dev));
  PQ_CUDA_TRY(cudaDeviceGetAttribute(&T->sms, cudaDevAttrMultiProcessorCount, dev));
  PQ_CUDA_TRY(cudaFuncSetAttribute(ss64_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SS_SMEM));
  h->two64 = std::move(T);
  return PQ_OK;
}

// as ci_sigma64
pq_status ci_two64(pq_ci_handle *h, const double *C, int64_t es, int64_t vs, int nv, double shift, double *S, int64_t ses,
                   int64_t svs, bool fixed, int **gate_out) {
  using namespace two64;
  if (fixed && !h->two64) return PQ_ERR_OOM;
  PQ_TRY(two64_prepare(h));
  Two64 &T = *h->two64;
  cudaStream_t st = h->stream;
  const Shape sh = shape_of(h);
  const int64_t n = h->n_dets;
  int *gate = T.aux;
  uint32_t *xhi = reinterpret_cast<uint32_t *>(T.aux) + 4, *hi = T.hi;
  const int npairs = (int)T.pairs.size();
  Parts q{};
  q.npairs = npairs;
  unsigned short *xd[6];
  double *part[6];
  auto lay = [&](DevLayout &l) {
    for (int i = 0; i < npairs; i++) {
      l.take(xd[i], (size_t)dg::N * nv * q.R[i] * T.pairs[i].np);
      l.take(part[i], (size_t)q.ksplit[i] * q.part[i]);
    }
  };
  for (int i = 0; i < npairs; i++) {
    const Two64::Pair &p = T.pairs[i];
    const int64_t R = n / p.M, N = nv * R;
    const int64_t tiles = ((p.M + BM - 1) / BM) * ((N + BN - 1) / BN), chunks = (p.M + 31) / 32;
    // parts of the K range, of at least eight chunks, while the tiles leave SMs idle
    q.ksplit[i] = (int)std::max<int64_t>(1, std::min<int64_t>({T.sms / tiles, chunks / 8, 8}));
    q.x[i] = p.x, q.y[i] = p.y, q.M[i] = p.M, q.R[i] = R, q.part[i] = N * p.M;
  }
  DevLayout l;
  lay(l);
  if (fixed && T.work.bytes < l.used) return PQ_ERR_OOM;
  PQ_TRY(ci_grow(h, T.work, l.used));  // a full device leaves the call to the other kernel before anything is written
  l = DevLayout{static_cast<char *>(T.work.ptr), 0};
  lay(l);
  for (int i = 0; i < npairs; i++) q.p[i] = part[i];
  PQ_CUDA_TRY(cudaMemsetAsync(T.aux, 0, 64, st));
  absmax_vectors_kernel<<<dim3((unsigned)std::min<int64_t>((n + 255) / 256, 152 * 4), nv), 256, 0, st>>>(C, es, vs, n, xhi);
  for (int i = 0; i < npairs; i++) {
    const Two64::Pair &p = T.pairs[i];
    const int64_t R = q.R[i], N = nv * R;
    pair_digits_kernel<<<(unsigned)N, 256, 0, st>>>(C, es, vs, sh, p.x, p.y, p.M, p.np, R, nv, xhi, hi, npairs,
                                                  xd[i], gate);
    PQ_CUDA_TRY(cudaGetLastError());
    CUtensorMap ma, mb;
    PQ_TRY(s64_map(&ma, p.d, dg::N * p.M, p.M, p.np, 32, BM));
    PQ_TRY(s64_map(&mb, xd[i], dg::N * N, p.M, p.np, 32, BN));
    SsArgs g{};
    g.na = N, g.nb = p.M, g.nv = 1;
    g.m_tiles = (int)((p.M + BM - 1) / BM);
    g.n_tiles = (int)((N + BN - 1) / BN);
    g.ksplit = q.ksplit[i];
    g.tiles = (int64_t)g.ksplit * g.m_tiles * g.n_tiles;
    g.win = p.win;
    g.per = R;
    g.part = q.part[i];
    g.a_plane = p.M, g.b_plane = N;
    g.chunks = (int)((p.M + 31) / 32);
    g.xhi = xhi, g.dhi = hi + i;
    g.S = part[i];
    g.wait = sigma_wait_cycles(0);
    g.gate = gate;
    ss64_kernel<false><<<(unsigned)std::min<int64_t>(g.tiles, T.sms), THREADS, SS_SMEM, st>>>(ma, mb, g);
    PQ_CUDA_TRY(cudaGetLastError());
  }
  sum_kernel<<<dim3((unsigned)((n + 255) / 256), nv), 256, 0, st>>>(C, es, vs, sh, q, n, h->d_diag.as<double>(), shift, S, ses,
                                                                   svs, gate);
  PQ_CUDA_TRY(cudaGetLastError());
  *gate_out = gate;
  return PQ_OK;
}

}  // namespace pq
