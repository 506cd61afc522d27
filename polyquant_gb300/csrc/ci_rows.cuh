// Grouped excitation tables of a one-species space and one determinant's
// connection classes on them; shared by the warp-per-determinant sigma
// (ci_sigma_rows.cu), the explicit Hamiltonian and the properties.
#pragma once
#include <memory>

#include "pq_bits.cuh"
#include "pq_internal.h"

namespace pq {

// Grouped tables of one spin list and the Coulomb sums of its strings.
struct SigmaRows {
  struct Side {
    int2 *s1 = nullptr;      // {partner (row offset for alpha, string for beta), info}, grouped by level change
    double *s1_F = nullptr;  // same-spin part of the element
    int32_t *s2 = nullptr;
    double *s2_D = nullptr;
    int32_t *cum = nullptr;  // per string 8: ends of the 3 groups of singles and the 5 groups of doubles
    int32_t *lvl = nullptr;
    double *coul = nullptr;  // [string][pair]: sum over the string's orbitals k of (pair of the other spin | kk); NULL when large
  };
  Side side[2];
  int32_t *row = nullptr;    // alpha string of every determinant
  DevBuf mem;                // all of the above
  int lim = 0;
  int min_width = 1;         // sigma of fewer vectors is the other kernel's
};

namespace rows {

struct Side {
  const int64_t *o1, *o2;
  const int2 *s1;
  const double *F;
  const int32_t *s2;
  const double *D;
  const int4 *cum;
  const int32_t *lvl;
  const double *coul;
  const uint64_t *str, *str_hi;
  int64_t rs, cs;  // eab strides of a pair of the other spin and of a pair of this one
};

struct Args {
  Side a, b;
  const int32_t *row;
  const int64_t *rowoff;
  const double *eab, *diag;
  double shift;
  int npair, lim;
  int64_t n;
  const double *X;
  double *Y;
};

constexpr int WARPS = 8;     // determinants per CTA
constexpr int HEAVY = 1536;  // connections above which the CTA's warps may share a determinant

// Whether the CTA's warps share row k, the same for every thread; len: the CTA's row lengths, 0 past the last row.  A
// heavy row of more than twice the mean would keep its warp long after the others have left; rows alike are one warp's
// each, since a list split over 256 lanes leaves more of them idle and each row costs a block-wide sum.  Shared
// whenever heavy, truncated spaces of long rows took up to 3.5 times as long (12o 6a6b, level 10 of 12, four roots 49.8
// ms against 14.3; products with the explicit matrix of 30o 2a2b 7.3 against 5.3), CISD of 5a5b in 24 orbitals 146 us
// against 125, and 201 with three times the mean.
__device__ __forceinline__ bool shared_row(const int *len, int k) {
  int64_t sum = 0;
#pragma unroll
  for (int w = 0; w < WARPS; w++) sum += len[w];
  return len[k] > HEAVY && (int64_t)len[k] * WARPS > 2 * sum;
}

template <int NV> __device__ __forceinline__ void load_x(const double *X, int64_t j, double (&x)[NV]) {
  const double *p = X + j * NV;
  if constexpr (NV == 2 || NV == 4) {
#pragma unroll
    for (int v = 0; v < NV; v += 2) {
      const double2 d = __ldg(reinterpret_cast<const double2 *>(p + v));
      x[v] = d.x, x[v + 1] = d.y;
    }
  } else {
#pragma unroll
    for (int v = 0; v < NV; v++) x[v] = __ldg(p + v);
  }
}

__device__ __forceinline__ double flip(double v, int neg) {
  return __hiloint2double(__double2hiint(v) ^ (neg << 31), __double2loint(v));
}

// One determinant's connection classes: list bounds after the level limits.
struct Det {
  int64_t I, rowI, a1, a2, b1, b2;
  int ia, ib;
  int ca1[4];              // group starts of the alpha singles
  int na1, na2, nb1, nb2;  // kept singles and doubles of either spin
  int nbx[3];              // kept beta singles beside an alpha single of group g
  int total;
};

__device__ __forceinline__ Det load_det(const Args &p, int64_t I) {
  Det d;
  d.I = I;
  d.ia = p.row[I];
  d.rowI = p.rowoff[d.ia];
  d.ib = (int)(I - d.rowI);
  d.a1 = p.a.o1[d.ia], d.a2 = p.a.o2[d.ia];
  d.b1 = p.b.o1[d.ib], d.b2 = p.b.o2[d.ib];
  const int slack = min(p.lim - p.a.lvl[d.ia] - p.b.lvl[d.ib], 4);  // >= 0 for a determinant of the list
  const int4 x0 = p.a.cum[2 * d.ia], x1 = p.a.cum[2 * d.ia + 1];
  const int4 y0 = p.b.cum[2 * d.ib], y1 = p.b.cum[2 * d.ib + 1];
  d.ca1[0] = 0, d.ca1[1] = x0.x, d.ca1[2] = x0.y, d.ca1[3] = x0.z;
  // a group of change c is kept when c <= slack
  d.na1 = slack >= 1 ? x0.z : x0.y;
  d.nb1 = slack >= 1 ? y0.z : y0.y;
  d.na2 = slack >= 2 ? x1.w : (slack == 1 ? x1.z : x1.y);
  d.nb2 = slack >= 2 ? y1.w : (slack == 1 ? y1.z : y1.y);
  d.total = 1 + d.na1 + d.nb1 + d.na2 + d.nb2;
#pragma unroll
  for (int g = 0; g < 3; g++) {
    // alpha change g - 1 leaves slack - (g - 1) for the beta change
    const int s = slack - (g - 1);
    d.nbx[g] = s >= 1 ? y0.z : (s == 0 ? y0.y : (s == -1 ? y0.x : 0));
    d.total += (d.ca1[g + 1] - d.ca1[g]) * d.nbx[g];
  }
  return d;
}

// Coulomb sum beside string `s` of side `t` for a single of the other spin with pair index `pair`.
__device__ __forceinline__ double opposite(const Args &p, const Side &t, int s, int pair) {
  if (t.coul) return __ldg(t.coul + (int64_t)s * p.npair + pair);
  double c = 0.0;
  for_occ(t.str[s], hiword(t.str_hi, s), [&](int k) { c += __ldg(p.eab + pair * t.rs + (int64_t)(k * (k + 3) / 2) * t.cs); });
  return c;
}

// The off-diagonal lists of a determinant's row of H: f(count, make) is called per list.  make(t, nth) gives a
// reader that returns the element and the partner j of entry t when first called and of t + nth, t + 2 nth, ... after.
template <typename F> __device__ __forceinline__ void for_lists(const Args &p, const Det &d, F &&f) {
  f(d.na1, [&](int t, int nth) {
    return [&p, &d, t, nth](int64_t &j) mutable {
      const int2 e = __ldg(p.a.s1 + d.a1 + t);
      const double h = __ldg(p.a.F + d.a1 + t) + opposite(p, p.b, d.ib, e.y >> 1);
      t += nth;
      j = (int64_t)e.x + d.ib;
      return flip(h, e.y & 1);
    };
  });
  f(d.nb1, [&](int t, int nth) {
    return [&p, &d, t, nth](int64_t &j) mutable {
      const int2 e = __ldg(p.b.s1 + d.b1 + t);
      const double h = __ldg(p.b.F + d.b1 + t) + opposite(p, p.a, d.ia, e.y >> 1);
      t += nth;
      j = d.rowI + e.x;
      return flip(h, e.y & 1);
    };
  });
  f(d.na2, [&](int t, int nth) {
    return [&p, &d, t, nth](int64_t &j) mutable {
      j = (int64_t)__ldg(p.a.s2 + d.a2 + t) + d.ib;
      const double h = __ldg(p.a.D + d.a2 + t);
      t += nth;
      return h;
    };
  });
  f(d.nb2, [&](int t, int nth) {
    return [&p, &d, t, nth](int64_t &j) mutable {
      j = d.rowI + __ldg(p.b.s2 + d.b2 + t);
      const double h = __ldg(p.b.D + d.b2 + t);
      t += nth;
      return h;
    };
  });
#pragma unroll
  for (int g = 0; g < 3; g++) {
    const int nb = d.nbx[g], cnt = (d.ca1[g + 1] - d.ca1[g]) * nb;
    if (cnt == 0) continue;
    const int2 *la = p.a.s1 + d.a1 + d.ca1[g], *lb = p.b.s1 + d.b1;
    // entry t is (alpha single t / nb, beta single t % nb); a step of nth adds (qs, rs) with a carry
    f(cnt, [&](int t, int nth) {
      const int qs = nth / nb, rs = nth - qs * nb;
      int ea = t / nb, eb = t - ea * nb;
      return [&p, la, lb, nb, qs, rs, ea, eb](int64_t &j) mutable {
        const int2 a = __ldg(la + ea), b = __ldg(lb + eb);
        ea += qs, eb += rs;
        if (eb >= nb) eb -= nb, ea++;
        j = (int64_t)a.x + b.x;
        return flip(__ldg(p.eab + (int64_t)(a.y >> 1) * p.npair + (b.y >> 1)), (a.y ^ b.y) & 1);
      };
    });
  }
}

}  // namespace rows

// The tables of a handle's determinant list (one species, at most 2^31 - 1 determinants).
pq_status rows_make(pq_ci_handle *h, std::unique_ptr<SigmaRows, void (*)(SigmaRows *)> &out);
rows::Args rows_args(const pq_ci_handle *h, const SigmaRows &r);

}  // namespace pq
