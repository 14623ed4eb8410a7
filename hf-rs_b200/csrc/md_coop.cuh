// Block-cooperative McMurchie-Davidson machinery shared by the f-shell
// engine (eri_md.cu) and the ERI derivatives (grad.cu): one shell quartet per
// block, every table in shared memory, the class known at run time.
//
//   (ab|cd) = 2 pi^{5/2} / (p q sqrt(p+q)) sum_h E^{ab}_h sum_k (-1)^{|k|}
//             E^{cd}_k R_{h+k}(alpha, P - Q),   h = (t,u,v), alpha = pq/(p+q)
//
// * A side (ab) holds the products E^{ab}_h = E_t E_u E_v of its nonzero
//   Hermite indices only (t <= a_x + b_x and so on: 336 of the 36 x 35
//   products of (dd), 1,920 of 100 x 84 of (ff)), listed by component pair,
//   so every contraction is a sparse sum without index arithmetic.
// * R is stored in a cube of edge S, so the index of h + k is the sum of two
//   linear offsets.
// * R_{tuv} comes from three one-axis sums instead of one recursion level per
//   order: with He-type coefficients c(t,k) = t! / (2^k k! (t-2k)!),
//     R^m_{00v}  = sum_k c(v,k) z^{v-2k} R^{m+v-k}_{000},
//   and the same over y and then x, which needs 3 block barriers instead of
//   L + 1 (13 for (ff|ff)).
#pragma once
#include <cuda_runtime.h>

#include "boys.cuh"
#include "eri_md.h"

namespace hfg {
namespace coop {

constexpr int kLTot = 4 * kMDLMax;      // highest Hermite order of a quartet
constexpr int kPolyK = kLTot / 2 + 1;   // terms of one axis polynomial

// c(t,k) = t! / (2^k k! (t - 2k)!)
struct HermC {
  double c[kLTot + 1][kPolyK];
};
constexpr HermC make_herm_c() {
  HermC h{};
  for (int t = 0; t <= kLTot; ++t) {
    double c = 1.0;
    for (int k = 0; 2 * k <= t; ++k) {
      h.c[t][k] = c;
      c = c * (t - 2 * k) * (t - 2 * k - 1) / (2.0 * (k + 1));
    }
  }
  return h;
}
__device__ const HermC kHermC = make_herm_c();

// Cartesian component c of angular momentum l in hf-rs order
// (src/basis.rs:418-445: d is xx, yy, zz, xy, xz, yz; the others are
// lexicographic with x descending, then y).
__device__ __forceinline__ void component(int l, int c, int* e) {
  if (l == 2) {
    const int d[6][3] = {{2, 0, 0}, {0, 2, 0}, {0, 0, 2}, {1, 1, 0}, {1, 0, 1}, {0, 1, 1}};
    e[0] = d[c][0];
    e[1] = d[c][1];
    e[2] = d[c][2];
    return;
  }
  int k = 0;
  for (int lx = l; lx >= 0; --lx)
    for (int ly = l - lx; ly >= 0; --ly) {
      if (k == c) {
        e[0] = lx;
        e[1] = ly;
        e[2] = l - lx - ly;
        return;
      }
      ++k;
    }
}

// 1/sqrt(prod (2 l_i - 1)!!): the per-component scale of src/basis.rs:123-132
__device__ __forceinline__ double comp_scale_of(const int* e) {
  double d = 1.0;
  for (int k = 0; k < 3; ++k)
    for (int m = 2 * e[k] - 1; m > 1; m -= 2) d *= m;
  return rsqrt(d);
}

__host__ __device__ __forceinline__ int nherm(int l) { return (l + 1) * (l + 2) * (l + 3) / 6; }
__host__ __device__ __forceinline__ int ncart_of(int l) { return (l + 1) * (l + 2) / 2; }

// x / d for 0 <= x < 2^20 with inv = 1.0f / d: the float quotient of the
// shifted numerator is off by less than half a step of x / d
__device__ __forceinline__ int fast_div(int x, float inv) { return (int)(((float)x + 0.5f) * inv); }

// Nonzero (component pair, Hermite index) products of a side: the sum over
// pairs of (a_x+b_x+1)(a_y+b_y+1)(a_z+b_z+1).
__host__ __device__ inline int side_nnz(int l1, int l2) {
  int s = 0;
  for (int ax = 0; ax <= l1; ++ax)
    for (int ay = 0; ay <= l1 - ax; ++ay)
      for (int bx = 0; bx <= l2; ++bx)
        for (int by = 0; by <= l2 - bx; ++by)
          s += (ax + bx + 1) * (ay + by + 1) * (l1 - ax - ay + l2 - bx - by + 1);
  return s;
}

// One side's run-time dimensions and shared-memory tables.
struct Side {
  int l1, l2, n1, n2, nab, nh, nnz, st;  // st: stride of j in the axis table E[ax][i][j][t]
  double *E, *D;      // axis tables (D: derivatives with respect to A - B, or null)
  double* prod;       // [nnz] E^{ab}_h
  double* dprod;      // [3][nnz] its derivatives (or null)
  int* start;         // [nab + 1] products of component pair ab
  unsigned* eo;       // [nnz] packed axis-table offsets (10 bits each)
  unsigned short* lin;  // [nnz] linear offset of h in the R cube
  unsigned char* h;     // [nnz] compact index of h
  unsigned char* ab;    // [nnz] component pair
  unsigned short* hlin; // [nh] linear offset of the compact index
  double* scale;        // [nab] component scales
};

__host__ __device__ __forceinline__ int axis_size(int l1, int l2) { return 3 * (l1 + 1) * (l2 + 1) * (l1 + l2 + 1); }

// Shared memory of one side, in bytes rounded up to 8.
__host__ __device__ inline size_t side_bytes(int l1, int l2, bool deriv) {
  const size_t nnz = side_nnz(l1, l2), nab = ncart_of(l1) * ncart_of(l2), nh = nherm(l1 + l2);
  size_t b = 8 * ((size_t)axis_size(l1, l2) * (deriv ? 2 : 1) + nnz * (deriv ? 4 : 1) + nab);
  b += 4 * (nab + 1) + 4 * nnz + 2 * nnz + nnz + nnz + 2 * nh;
  return (b + 15) & ~(size_t)7;
}

__device__ inline unsigned char* side_carve(Side& s, int l1, int l2, bool deriv, unsigned char* p) {
  s.l1 = l1;
  s.l2 = l2;
  s.n1 = ncart_of(l1);
  s.n2 = ncart_of(l2);
  s.nab = s.n1 * s.n2;
  s.nh = nherm(l1 + l2);
  s.nnz = side_nnz(l1, l2);
  s.st = l1 + l2 + 1;
  unsigned char* const p0 = p;
  const int na = axis_size(l1, l2);
  s.E = (double*)p;
  p += 8 * na;
  s.D = nullptr;
  if (deriv) {
    s.D = (double*)p;
    p += 8 * na;
  }
  s.prod = (double*)p;
  p += 8 * s.nnz;
  s.dprod = nullptr;
  if (deriv) {
    s.dprod = (double*)p;
    p += 24 * s.nnz;
  }
  s.scale = (double*)p;
  p += 8 * s.nab;
  s.start = (int*)p;
  p += 4 * (s.nab + 1);
  s.eo = (unsigned*)p;
  p += 4 * s.nnz;
  s.lin = (unsigned short*)p;
  p += 2 * s.nnz;
  s.hlin = (unsigned short*)p;
  p += 2 * s.nh;
  s.h = p;
  p += s.nnz;
  s.ab = p;
  return p0 + side_bytes(l1, l2, deriv);
}

// compact index of (t,u,v) among degrees <= l: all of lower t, then of lower
// u, in the nested order t, u, v
__device__ __forceinline__ int herm_index(int l, int t, int u, int v) {
  int k = 0;
  for (int i = 0; i < t; ++i) k += (l - i + 1) * (l - i + 2) / 2;
  for (int j = 0; j < u; ++j) k += l - t - j + 1;
  return k + v;
}

__device__ __forceinline__ int axis_off(const Side& s, int ax, int i, int j, int t) {
  return ((ax * (s.l1 + 1) + i) * (s.l2 + 1) + j) * s.st + t;
}

// Index lists of a side (once per block, every thread; synchronised inside
// and by the caller after).
__device__ inline void side_setup(const Side& s, int S) {
  for (int ab = threadIdx.x; ab < s.nab; ab += blockDim.x) {
    int ea[3], eb[3];
    component(s.l1, ab / s.n2, ea);
    component(s.l2, ab % s.n2, eb);
    s.scale[ab] = comp_scale_of(ea) * comp_scale_of(eb);
    s.start[ab + 1] = (ea[0] + eb[0] + 1) * (ea[1] + eb[1] + 1) * (ea[2] + eb[2] + 1);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int sum = 0;
    s.start[0] = 0;
    for (int ab = 1; ab <= s.nab; ++ab) s.start[ab] = sum += s.start[ab];
  }
  __syncthreads();
  const int l = s.l1 + s.l2;
  for (int ab = threadIdx.x; ab < s.nab; ab += blockDim.x) {
    int ea[3], eb[3], off = s.start[ab];
    component(s.l1, ab / s.n2, ea);
    component(s.l2, ab % s.n2, eb);
    for (int t = 0; t <= ea[0] + eb[0]; ++t)
      for (int u = 0; u <= ea[1] + eb[1]; ++u) {
        const int h0 = herm_index(l, t, u, 0);
        for (int v = 0; v <= ea[2] + eb[2]; ++v, ++off) {
          s.eo[off] = (unsigned)axis_off(s, 0, ea[0], eb[0], t) | (unsigned)axis_off(s, 1, ea[1], eb[1], u) << 10 |
                      (unsigned)axis_off(s, 2, ea[2], eb[2], v) << 20;
          s.lin[off] = (unsigned short)((t * S + u) * S + v);
          s.h[off] = (unsigned char)(h0 + v);
          s.ab[off] = (unsigned char)ab;
        }
      }
  }
  for (int x = threadIdx.x; x < (l + 1) * (l + 1) * (l + 1); x += blockDim.x) {
    const int t = x / ((l + 1) * (l + 1)), u = x / (l + 1) % (l + 1), v = x % (l + 1);
    if (t + u + v <= l) s.hlin[herm_index(l, t, u, v)] = (unsigned short)((t * S + u) * S + v);
  }
}

// Axis tables of one primitive pair, by one warp: lane = 8 axis + t.  With R
// = A - B, PA = P - A = -bp R and P - B = PA + R = (1 - bp) R;
//   E^{i+1,j}_t = E^{ij}_{t-1}/(2p) + (P-A) E^{ij}_t + (t+1) E^{ij}_{t+1}
// and D = dE/dR at fixed P (the Gaussian product factor apart) follows by
// differentiating it.
__device__ inline void side_axes(const Side& s, int lane, const double* AB, const double* PA, double bp, double inv_p) {
  const int ax = lane >> 3, t = lane & 7;
  const bool on = ax < 3 && t < s.st;
  const double pa = ax == 0 ? PA[0] : (ax == 1 ? PA[1] : PA[2]);
  const double pb = pa + (ax == 0 ? AB[0] : (ax == 1 ? AB[1] : AB[2])), i2p = 0.5 * inv_p;
  for (int i = 0; i <= s.l1; ++i)
    for (int j = 0; j <= s.l2; ++j) {
      if (on) {
        double e = 0.0, d = 0.0;
        if (i + j == 0) {
          e = t == 0 ? 1.0 : 0.0;
        } else if (t <= i + j) {
          const int o = i > 0 ? axis_off(s, ax, i - 1, j, t) : axis_off(s, ax, i, j - 1, t);
          const double x = i > 0 ? pa : pb, dx = i > 0 ? -bp : 1.0 - bp;
          e = x * s.E[o];
          if (t > 0) e = fma(i2p, s.E[o - 1], e);
          if (t + 1 <= i + j - 1) e = fma((double)(t + 1), s.E[o + 1], e);
          if (s.D) {
            d = fma(x, s.D[o], dx * s.E[o]);
            if (t > 0) d = fma(i2p, s.D[o - 1], d);
            if (t + 1 <= i + j - 1) d = fma((double)(t + 1), s.D[o + 1], d);
          }
        }
        const int w = axis_off(s, ax, i, j, t);
        s.E[w] = e;
        if (s.D) s.D[w] = d;
      }
      __syncwarp();
    }
}

// Products of a side by threads [tid, nt) of the block; `pref` and the sign
// (-1)^{t+u+v} of a ket side included.
__device__ __forceinline__ void side_products(const Side& s, int tid, int nt, double pref, bool ket, int S) {
  for (int k = tid; k < s.nnz; k += nt) {
    const unsigned o = s.eo[k];
    const int ox = o & 1023, oy = (o >> 10) & 1023, oz = o >> 20;
    double f = pref;
    if (ket) {
      const int l = s.lin[k], v = l % S, u = l / S % S, t = l / (S * S);
      if ((t + u + v) & 1) f = -f;
    }
    const double ex = s.E[ox], ey = s.E[oy], ez = s.E[oz];
    s.prod[k] = f * ex * ey * ez;
    if (s.dprod) {
      s.dprod[k] = f * s.D[ox] * ey * ez;
      s.dprod[s.nnz + k] = f * ex * s.D[oy] * ez;
      s.dprod[2 * s.nnz + k] = f * ex * ey * s.D[oz];
    }
  }
}

// base[m] = (-2 alpha)^m F_m(T), m <= L <= 16, by one warp, order m on lane m:
// each order by its own Taylor row of the global grid table (kBoysCols
// columns per row; boys.cuh's expansion without its downward recursion, whose
// divisions made a chain through every order), the asymptotic form beyond
// the grid by upward recursion on each lane.
__device__ __forceinline__ void boys_base(double t, double alpha, int L, int lane, const double* __restrict__ table,
                                          double* base) {
  if (lane > L) return;
  double f;
  if (t > kBoysTMax) {
    const double r = rsqrt(t), inv2t = 0.5 * r * r, e = exp(-t);
    f = kHalfSqrtPi * r;
    for (int m = 1; m <= lane; ++m) f = ((2 * m - 1) * f - e) * inv2t;
  } else {
    const int idx = min(max(__double2int_rn(t * 20.0), 0), kBoysSmemRows - 1);
    const double x = idx * kBoysStep - t;
    const double* row = table + (size_t)idx * kBoysCols + lane;
    f = __ldg(row + 7) * (1.0 / 5040.0);
    f = fma(f, x, __ldg(row + 6) * (1.0 / 720.0));
    f = fma(f, x, __ldg(row + 5) * (1.0 / 120.0));
    f = fma(f, x, __ldg(row + 4) * (1.0 / 24.0));
    f = fma(f, x, __ldg(row + 3) * (1.0 / 6.0));
    f = fma(f, x, __ldg(row + 2) * 0.5);
    f = fma(f, x, __ldg(row + 1));
    f = fma(f, x, __ldg(row));
  }
  for (int m = 0; m < lane; ++m) f *= -2.0 * alpha;
  base[lane] = f;
}

// The R tables of one quartet: base orders, one-axis polynomials, the two
// intermediate tables and the cube of edge S.
struct RTab {
  int L, S, nall;
  double *base, *poly, *A, *B, *R;
  unsigned short* all;  // packed (t,u,v) of every Hermite index of degree <= L (5 bits each)
};

__host__ __device__ inline size_t rtab_bytes(int L) {
  const size_t e = L + 1, n = nherm(L);
  return (8 * ((L + 2) + 3 * e * kPolyK + e * e + 2 * e * e * e) + 2 * n + 15) & ~(size_t)7;
}

__device__ inline unsigned char* rtab_carve(RTab& r, int L, unsigned char* p) {
  r.L = L;
  r.S = L + 1;
  r.nall = nherm(L);
  double* d = (double*)p;
  const int e = L + 1;
  r.base = d;
  r.poly = r.base + (L + 2);
  r.A = r.poly + 3 * e * kPolyK;
  r.B = r.A + e * e;
  r.R = r.B + e * e * e;
  r.all = (unsigned short*)(r.R + e * e * e);
  return p + rtab_bytes(L);
}

__device__ inline void rtab_setup(const RTab& r) {
  const int e = r.S;
  for (int x = threadIdx.x; x < e * e * e; x += blockDim.x) {
    const int t = x / (e * e), u = x / e % e, v = x % e;
    if (t + u + v <= r.L) r.all[herm_index(r.L, t, u, v)] = (unsigned short)(t << 10 | u << 5 | v);
  }
}

// One-axis polynomials c(t,k) x^{t-2k} of the vector PQ, by one warp.
__device__ __forceinline__ void rtab_poly(const RTab& r, int lane, const double* PQ) {
  for (int x = lane; x < 3 * r.S; x += 32) {
    const int ax = x / r.S, t = x % r.S;
    const double w = PQ[ax], w2 = w * w;
    double pw = (t & 1) ? w : 1.0;
    for (int k = t / 2; k >= 0; --k) {
      r.poly[x * kPolyK + k] = kHermC.c[t][k] * pw;
      pw *= w2;
    }
  }
}

// R_{tuv} from the base orders; three passes with a block barrier after each
// (and one is expected before, once base and poly are written).
template <typename Work>
__device__ __forceinline__ void rtab_build(const RTab& r, Work&& beside) {
  const int e = r.S, tid = threadIdx.x, nt = blockDim.x;
  for (int x = tid; x < e * e; x += nt) {
    const int v = x / e, m = x % e;
    if (v + m > r.L) continue;
    const double* c = r.poly + (2 * e + v) * kPolyK;
    double s = 0.0;
    for (int k = 0; 2 * k <= v; ++k) s = fma(c[k], r.base[m + v - k], s);
    r.A[x] = s;
  }
  beside();
  __syncthreads();
  for (int x = tid; x < r.nall; x += nt) {
    const int o = r.all[x], u = o >> 10, v = (o >> 5) & 31, m = o & 31;
    const double* c = r.poly + (e + u) * kPolyK;
    const double* a = r.A + v * e + m + u;
    double s = 0.0;
    for (int k = 0; 2 * k <= u; ++k) s = fma(c[k], a[-k], s);
    r.B[(u * e + v) * e + m] = s;
  }
  __syncthreads();
  for (int x = tid; x < r.nall; x += nt) {
    const int o = r.all[x], t = o >> 10, u = (o >> 5) & 31, v = o & 31;
    const double* c = r.poly + t * kPolyK;
    const double* b = r.B + (u * e + v) * e + t;
    double s = 0.0;
    for (int k = 0; 2 * k <= t; ++k) s = fma(c[k], b[-k], s);
    r.R[(t * e + u) * e + v] = s;
  }
  __syncthreads();
}

// A launch's shell quartets, one at a time per block: unit u is ket `u % 32`
// of warp task t0 + u / 32 of the work queue.  Units are taken from the
// launch's counter in runs of `per`; the plan's own steps (up to 64 tasks)
// are far too coarse for a block per quartet on small molecules.
struct UnitQueue {
  long long t0, units;
  int per;
};
__device__ __forceinline__ UnitQueue unit_queue(const long long* chunk_start, long long nchunks) {
  UnitQueue q;
  q.t0 = chunk_start[0];
  q.units = (chunk_start[nchunks] - q.t0) * 32;
  const long long per = q.units / ((long long)gridDim.x * 16);
  q.per = (int)(per < 1 ? 1 : (per > 32 ? 32 : per));
  return q;
}

// entry of warp task w, from the last one used
__device__ __forceinline__ int entry_of(const long long* __restrict__ prefix, int nentries, long long w, int e) {
  if (prefix[e] <= w) {
    if (w < prefix[e + 1]) return e;
    if (e + 2 <= nentries && w < prefix[e + 2]) return e + 1;
  }
  int lo = 0, hi = nentries;  // largest e with prefix[e] <= w
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (prefix[mid] <= w) lo = mid; else hi = mid;
  }
  return lo;
}

}  // namespace coop
}  // namespace hfg
