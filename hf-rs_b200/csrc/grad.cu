// Nuclear derivatives of the two-electron energy (the ERI part of the HF
// gradient, hf-rs's contract_eri_derivatives, src/gradient.rs:33-69 with the
// densities of :287-301).  With G = P_ab P_cd - x (P_ac P_bd + P_ad P_bc)
// (x = 1/4 for a closed shell; per spin, x = 1/2 on the spin densities)
// the energy is E2 = 1/2 sum_abcd (ab|cd) G_abcd, so over unique quartets
//   dE2/dX = 4 sum w (d(ab|cd)/dX) G_abcd,
// w the degeneracy weight of the J/K kernels.  Everything is contracted with
// G in Hermite form: with P the bra's product centre and R_AB = A - B,
//   d/dA = (alpha/p) d/dP + d/dR_AB,  d/dB = (beta/p) d/dP - d/dR_AB,
// d/dP raises the auxiliary integrals R_{h+k} and d/dR_AB acts on the Hermite
// coefficients; centre D follows from translational invariance.
//
// Two kernels, by class:
//
// * grad_lane_kernel (la + lb + lc + ld <= 4 but (21|10)): generated straight-line code
//   (grad_gen.cuh), one primitive quartet per lane.  A shell quartet takes
//   the largest power-of-two group of lanes that its primitive quartets fill,
//   so a contracted (ss|ss) quartet of 64 x 64 primitive pairs keeps a warp
//   busy, and quartets of uncontracted shells share one.  These classes hold
//   nearly all primitive quartets.  8 warps per SM, which wait on global and
//   local loads (the generated code's stack) before FP64 results: the FP64
//   pipe is 10% busy.
// * grad_coop_kernel (the d-rich classes, 4 <= L <= 8): one quartet per
//   block on the tables of md_coop.cuh.  G is contracted with one side's
//   coefficients (W, X), those with R (V, U, over the nonzero Hermite
//   products only), and those with the derivative coefficients: about 53,000
//   multiply-adds per (dd|dd) primitive quartet (12,000 more for a bra
//   primitive's first) and 6 block barriers.
#include <cuda_runtime.h>

#include <algorithm>

#include "eri_md.h"
#include "eri_prim.cuh"
#include "grad_gen.cuh"
#include "jk_dispatch.h"
#include "md_coop.cuh"
#include "smem_limit.h"

namespace hfg {

namespace {

struct GradArgs {
  const JKEntry* entries;
  const long long* prefix;
  int nentries;
  const long long* chunk_start;
  long long nchunks;
  unsigned long long* counter;
  const PairInfo* pairs;
  KetSoA kets;
  const double* pairQ;
  double thr;
  const PrimRec64* rec;
  const double* boys;
  const double* expt;
  const double* P;   // total density, n x n
  const double* Ps;  // nspin spin densities
  int nspin, n, natom;
  const int* ao_atom;
  double* grad;  // natom x 3
};

// G_abcd of one component quadruple.
__device__ __forceinline__ double pair_density(const GradArgs& a, int I, int J, int K, int M) {
  const size_t n = a.n;
  double g = __ldg(a.P + I * n + J) * __ldg(a.P + K * n + M);
  const double xk = a.nspin == 1 ? 0.25 : 0.5;
  for (int sp = 0; sp < a.nspin; ++sp) {
    const double* D = a.Ps + sp * n * n;
    g -= xk * (__ldg(D + I * n + K) * __ldg(D + J * n + M) + __ldg(D + I * n + M) * __ldg(D + J * n + K));
  }
  return g;
}

// Primitive quartets with |k_P k_Q| below this are left out: the derivative
// of one is at most ~1e6 times its prefactor, so each stays below 1e-22.
constexpr double kPrimFloor = 1e-28;

constexpr int kLaneThreads = 128;
// lanes per quartet are at least 32 / lane_slots: the density blocks of a
// warp's quartets take at most 8 KB
__host__ __device__ constexpr int lane_slots(int nabcd) {
  int s = 32;
  while (s > 1 && s * nabcd > 1024) s /= 2;
  return s;
}
constexpr int kLaneGradAtoms = 512;  // per-atom sums held in shared memory up to this many atoms

template <int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(kLaneThreads) grad_lane_kernel(const GradArgs a) {
  using C = GradClass<LA, LB, LC, LD>;
  constexpr int NB = ncart(LB), NC = ncart(LC), ND = ncart(LD);
  constexpr int NABCD = ncart(LA) * NB * NC * ND, SLOTS = lane_slots(NABCD);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* sm = reinterpret_cast<double*>(smem_raw);
  double* gsm = sm + boys_smem_bytes<double>() / 8 + (threadIdx.x >> 5) * (NABCD * SLOTS);
  double* gacc = sm + boys_smem_bytes<double>() / 8 + (kLaneThreads / 32) * (NABCD * SLOTS);
  const bool local = a.natom <= kLaneGradAtoms;
  boys_stage<double, C::L + 1>(sm, a.boys, a.expt);
  if (local)
    for (int x = threadIdx.x; x < 3 * a.natom; x += blockDim.x) gacc[x] = 0.0;
  __syncthreads();
  double* const gout = local ? gacc : a.grad;
  const int lane = threadIdx.x & 31;
  // units: lane group `sub` of warp task t0 + u / 32; runs of `per` units
  const long long t0 = a.chunk_start[0], units = (a.chunk_start[a.nchunks] - t0) * 32;
  int per = 1;
  while (per < 32 && units > (long long)per * 2 * gridDim.x * (kLaneThreads / 32) * 8) per *= 2;
  int e = 0;
  for (;;) {
    long long u0 = 0;
    if (lane == 0) u0 = (long long)atomicAdd(a.counter, (unsigned long long)per);
    u0 = __shfl_sync(0xffffffffu, u0, 0);
    if (u0 >= units) break;
    const long long w = t0 + (u0 >> 5);
    e = coop::entry_of(a.prefix, a.nentries, w, e);
    const JKEntry ent = a.entries[e];
    const PairInfo bra = a.pairs[ent.bra];
    const int k0 = ent.k_lo + (int)(w - a.prefix[e]) * 32;
    const int nb = bra.npp, nk = __ldg(&a.kets.nn[ent.k_lo]).x;  // one pair class: equal counts
    // lanes per quartet
    int gs = 32 / SLOTS;
    while (gs < 32 && 2 * gs <= nb * nk) gs *= 2;
    const int ng = 32 / gs, slot = lane / gs, mem = lane - slot * gs;
    const double qb = __ldg(a.pairQ + ent.bra);
    double gA[3] = {0.0, 0.0, 0.0}, tP[3] = {0.0, 0.0, 0.0};
    const int sub0 = (int)(u0 & 31), sub1 = min(sub0 + per, gs);
    for (int sub = sub0; sub < sub1; ++sub) {
      const int kidx = k0 + sub * ng + slot;
      const bool active = kidx < ent.k_hi && __ldg(a.pairQ + min(kidx, ent.k_hi - 1)) * qb > a.thr;
      if (__ballot_sync(0xffffffffu, active) == 0u) continue;
      const int kx = active ? kidx : ent.k_lo;
      const double2 v0 = __ldg(a.kets.a0 + kx), v1 = __ldg(a.kets.a1 + kx), v2 = __ldg(a.kets.a2 + kx);
      const int4 ii = __ldg(a.kets.ii + kx);
      const int ksame = __ldg(a.kets.nn + kx).y;
      // 4 x degeneracy weight, zero for an idle slot
      double wt = active ? 4.0 : 0.0;
      if (bra.same) wt *= 0.5;
      if (ksame) wt *= 0.5;
      if (kidx == ent.bra) wt *= 0.5;
      // density blocks of the warp's quartets, element x of slot s at [x * ng + s]
      __syncwarp();
      for (int x = lane; x < NABCD * ng; x += 32) {
        const int s = x & (ng - 1), y = x / ng;
        const int l = y % ND, k = y / ND % NC, j = y / (ND * NC) % NB, i = y / (ND * NC * NB);
        const int kk = min(k0 + sub * ng + s, ent.k_hi - 1);
        const int4 kii = __ldg(a.kets.ii + kk);
        gsm[x] = pair_density(a, bra.ao_a + i, bra.ao_b + j, kii.x + k, kii.y + l) *
                 (comp_scale(LA, i) * comp_scale(LB, j) * comp_scale(LC, k) * comp_scale(LD, l));
      }
      __syncwarp();
      const double AC[3] = {bra.Ax - v0.x, bra.Ay - v0.y, bra.Az - v1.x};
      double sA[3] = {0.0, 0.0, 0.0}, sP[3] = {0.0, 0.0, 0.0}, sC[3] = {0.0, 0.0, 0.0};
      const int np = active ? nb * nk : 0;
      int ik = mem / nb, ib = mem - ik * nb;
      for (int x = mem; x < np; x += gs) {
        const PrimRec64 p = a.rec[bra.rec_off + (size_t)ib * bra.rec_stride];
        const PrimRec64 q = a.rec[ii.z + (size_t)ik * ii.w];
        ib += gs;
        while (ib >= nb) {
          ib -= nb;
          ++ik;
        }
        const double kpq = p.kp * q.kp;
        if (fabs(kpq) < kPrimFloor) continue;
        const double pax = -p.bp * bra.ABx, pay = -p.bp * bra.ABy, paz = -p.bp * bra.ABz;
        const double qcx = -q.bp * v1.y, qcy = -q.bp * v2.x, qcz = -q.bp * v2.y;
        const double PQx = AC[0] + pax - qcx, PQy = AC[1] + pay - qcy, PQz = AC[2] + paz - qcz;
        const double s = p.p + q.p, r = rsqrt(s), alpha = p.p * q.p * r * r;
        double F[C::L + 2];
        boys_eval<C::L + 1>(alpha * (PQx * PQx + PQy * PQy + PQz * PQz), sm, F);
        double f = kTwoPiPow25 * kpq * r;
#pragma unroll
        for (int m = 0; m <= C::L + 1; ++m) {
          F[m] *= f;
          f *= -2.0 * alpha;
        }
        double ev, gp[3], gb[3], gk[3];
        C::prim(gsm + slot, ng, F, PQx, PQy, PQz, pax, pay, paz, pax + bra.ABx, pay + bra.ABy, paz + bra.ABz,
                0.5 * p.inv_p, -p.bp, 1.0 - p.bp, qcx, qcy, qcz, qcx + v1.y, qcy + v2.x, qcz + v2.y, 0.5 * q.inv_p, -q.bp,
                1.0 - q.bp, ev, gp, gb, gk);
        const double mb = -2.0 * p.bp * (1.0 - p.bp) * p.p * ev, mk = -2.0 * q.bp * (1.0 - q.bp) * q.p * ev;
        sA[0] += (1.0 - p.bp) * gp[0] + gb[0] + mb * bra.ABx;
        sA[1] += (1.0 - p.bp) * gp[1] + gb[1] + mb * bra.ABy;
        sA[2] += (1.0 - p.bp) * gp[2] + gb[2] + mb * bra.ABz;
        sC[0] += (q.bp - 1.0) * gp[0] + gk[0] + mk * v1.y;
        sC[1] += (q.bp - 1.0) * gp[1] + gk[1] + mk * v2.x;
        sC[2] += (q.bp - 1.0) * gp[2] + gk[2] + mk * v2.y;
#pragma unroll
        for (int k = 0; k < 3; ++k) sP[k] += gp[k];
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        sA[k] *= wt;
        sP[k] *= wt;
        sC[k] *= wt;
        gA[k] += sA[k];
        tP[k] += sP[k];
        for (int off = gs >> 1; off > 0; off >>= 1) {
          sP[k] += __shfl_xor_sync(0xffffffffu, sP[k], off);
          sC[k] += __shfl_xor_sync(0xffffffffu, sC[k], off);
        }
      }
      if (active && mem == 0) {
        const int atC = __ldg(a.ao_atom + ii.x), atD = __ldg(a.ao_atom + ii.y);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          atomicAdd(gout + 3 * atC + k, sC[k]);
          atomicAdd(gout + 3 * atD + k, -sP[k] - sC[k]);
        }
      }
    }
    if (sub1 > sub0) {
      const int atA = __ldg(a.ao_atom + bra.ao_a), atB = __ldg(a.ao_atom + bra.ao_b);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        for (int off = 16; off > 0; off >>= 1) {
          gA[k] += __shfl_xor_sync(0xffffffffu, gA[k], off);
          tP[k] += __shfl_xor_sync(0xffffffffu, tP[k], off);
        }
        if (lane == 0) {
          atomicAdd(gout + 3 * atA + k, gA[k]);
          atomicAdd(gout + 3 * atB + k, tP[k] - gA[k]);
        }
      }
    }
  }
  if (local) {
    __syncthreads();
    for (int x = threadIdx.x; x < 3 * a.natom; x += blockDim.x)
      if (gacc[x] != 0.0) atomicAdd(a.grad + x, gacc[x]);
  }
}

constexpr int kCoopThreads = 128;

struct CoopLayout {
  int nab, ncd, hab, hcd, nnzb, nnzk;
  __host__ __device__ explicit CoopLayout(const MDClass& c) {
    nab = c.na * c.nb;
    ncd = c.nc * c.nd;
    hab = coop::nherm(c.lab);
    hcd = coop::nherm(c.lcd);
    nnzb = coop::side_nnz(c.la, c.lb);
    nnzk = coop::side_nnz(c.lc, c.ld);
  }
  // G, W, X, the vectors and block sums, and both sides' lists by Hermite index
  __host__ __device__ size_t own_bytes() const {
    return ((size_t)(nab * ncd + nab * hcd + ncd * hab + 16 + 9 * (kCoopThreads / 32)) * 8 +
            (size_t)(hab + hcd + 2) * 4 + (size_t)(nnzb + nnzk) * 2 + 15) & ~(size_t)7;
  }
};

size_t coop_smem(const MDClass& c) {
  return CoopLayout(c).own_bytes() + coop::side_bytes(c.la, c.lb, true) + coop::side_bytes(c.lc, c.ld, true) +
         coop::rtab_bytes(c.L + 1);
}

// products of a side listed by Hermite index
__device__ void list_by_herm(const coop::Side& s, int* start, unsigned short* list) {
  // a warp per Hermite index: 32 products a step, placed by ballot
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int h = warp; h < s.nh; h += nw) {
    int n = 0;
    for (int k0 = 0; k0 < s.nnz; k0 += 32)
      n += __popc(__ballot_sync(0xffffffffu, k0 + lane < s.nnz && s.h[k0 + lane] < h));
    if (lane == 0) start[h] = n;
    for (int k0 = 0; k0 < s.nnz; k0 += 32) {
      const bool mine = k0 + lane < s.nnz && s.h[k0 + lane] == h;
      const unsigned b = __ballot_sync(0xffffffffu, mine);
      if (mine) list[n + __popc(b & ((1u << lane) - 1u))] = (unsigned short)(k0 + lane);
      n += __popc(b);
    }
  }
  if (threadIdx.x == 0) start[s.nh] = s.nnz;
}

__global__ void __launch_bounds__(kCoopThreads) grad_coop_kernel(MDClass c, const GradArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const CoopLayout L(c);
  double* d = reinterpret_cast<double*>(smem_raw);
  double* G = d;
  double* W = G + L.nab * L.ncd;
  double* X = W + L.nab * L.hcd;
  double* S = X + L.ncd * L.hab;  // [0..2] P - Q, [3] prefactor
  double* red = S + 16;
  int* hsb = reinterpret_cast<int*>(red + 9 * (kCoopThreads / 32));
  int* hsk = hsb + L.hab + 1;
  unsigned short* hlb = reinterpret_cast<unsigned short*>(hsk + L.hcd + 1);
  unsigned short* hlk = hlb + L.nnzb;
  coop::Side B, K;
  coop::RTab R;
  unsigned char* p = smem_raw + L.own_bytes();
  p = coop::side_carve(B, c.la, c.lb, true, p);
  p = coop::side_carve(K, c.lc, c.ld, true, p);
  coop::rtab_carve(R, c.L + 1, p);
  coop::side_setup(B, R.S);
  coop::side_setup(K, R.S);
  coop::rtab_setup(R);
  __syncthreads();
  list_by_herm(B, hsb, hlb);
  list_by_herm(K, hsk, hlk);
  __shared__ long long s_unit;
  const int tid = threadIdx.x, nt = blockDim.x, warp = tid >> 5, lane = tid & 31;
  const float inv_ncd = 1.0f / L.ncd, inv_hcd = 1.0f / L.hcd, inv_hab = 1.0f / L.hab;
  const int SS = R.S * R.S, S1 = R.S;
  const coop::UnitQueue uq = coop::unit_queue(a.chunk_start, a.nchunks);
  int e = 0;
  for (;;) {
    __syncthreads();
    if (tid == 0) s_unit = (long long)atomicAdd(a.counter, (unsigned long long)uq.per);
    __syncthreads();
    const long long u0 = s_unit;
    if (u0 >= uq.units) break;
    for (long long u = u0; u < u0 + uq.per && u < uq.units; ++u) {
      const long long w = uq.t0 + (u >> 5);
      e = coop::entry_of(a.prefix, a.nentries, w, e);
      const JKEntry ent = a.entries[e];
      const int kidx = ent.k_lo + (int)(w - a.prefix[e]) * 32 + (int)(u & 31);
      if (kidx >= ent.k_hi || !(a.pairQ[kidx] * a.pairQ[ent.bra] > a.thr)) continue;
      const PairInfo bra = a.pairs[ent.bra], ket = a.pairs[kidx];
      double deg = 4.0;
      if (bra.same) deg *= 0.5;
      if (ket.same) deg *= 0.5;
      if (kidx == ent.bra) deg *= 0.5;
      __syncthreads();  // the previous quartet's tables have been read
      for (int x = tid; x < L.nab * L.ncd; x += nt) {
        const int ab = coop::fast_div(x, inv_ncd), cd = x - ab * L.ncd;
        const int i = ab / c.nb, k = cd / c.nd;
        G[x] = deg * B.scale[ab] * K.scale[cd] *
               pair_density(a, bra.ao_a + i, bra.ao_b + ab - i * c.nb, ket.ao_a + k, ket.ao_b + cd - k * c.nd);
      }
      double acc[9];
      for (int k = 0; k < 9; ++k) acc[k] = 0.0;
      const double AB[3] = {bra.ABx, bra.ABy, bra.ABz}, CD[3] = {ket.ABx, ket.ABy, ket.ABz};
      const double AC[3] = {bra.Ax - ket.Ax, bra.Ay - ket.Ay, bra.Az - ket.Az};
      const PrimRange pb = prim_range(bra.rec_off, bra.rec_stride, bra.npp, ent.slice, 0);
      const PrimRange pk = prim_range(ket.rec_off, ket.rec_stride, ket.npp, ent.slice, 16);
      for (int ib = 0; ib < pb.count; ++ib) {
        const PrimRec64 rb = a.rec[pb.off + (size_t)ib * pb.stride];
        bool fresh = true;  // this bra primitive's tables are not made yet
        for (int ik = 0; ik < pk.count; ++ik) {
          const PrimRec64 rk = a.rec[pk.off + (size_t)ik * pk.stride];
          const double kpq = rb.kp * rk.kp;
          if (fabs(kpq) < kPrimFloor) continue;  // (the same for every thread)
          __syncthreads();
          // one task per warp (4 warps)
          const double PA[3] = {-rb.bp * AB[0], -rb.bp * AB[1], -rb.bp * AB[2]};
          const double QC[3] = {-rk.bp * CD[0], -rk.bp * CD[1], -rk.bp * CD[2]};
          if (warp == 0) {
            if (fresh) coop::side_axes(B, lane, AB, PA, rb.bp, rb.inv_p);
          } else if (warp == 1) {
            coop::side_axes(K, lane, CD, QC, rk.bp, rk.inv_p);
          } else {
            const double PQ[3] = {AC[0] + PA[0] - QC[0], AC[1] + PA[1] - QC[1], AC[2] + PA[2] - QC[2]};
            if (warp == 2) {
              coop::rtab_poly(R, lane, PQ);
            } else {
              const double sum = rb.p + rk.p, r = rsqrt(sum), alpha = rb.p * rk.p * r * r;
              coop::boys_base(alpha * (PQ[0] * PQ[0] + PQ[1] * PQ[1] + PQ[2] * PQ[2]), alpha, R.L, lane, a.boys, R.base);
              if (lane == 0) S[3] = kTwoPiPow25 * kpq * r;
            }
          }
          __syncthreads();
          const double pref = S[3];
          coop::rtab_build(R, [&] {
            if (fresh) coop::side_products(B, tid, nt, 1.0, false, R.S);
            coop::side_products(K, tid, nt, pref, true, R.S);
          });
          // W[ab][k] = sum_cd G E^{cd}_k;  X[cd][h] = sum_ab G E^{ab}_h
          const int nW = L.nab * L.hcd, nX = fresh ? L.ncd * L.hab : 0;
          for (int x = tid; x < nW + nX; x += nt) {
            double v = 0.0;
            if (x < nW) {
              const int ab = coop::fast_div(x, inv_hcd), h = x - ab * L.hcd;
              const double* g = G + ab * L.ncd;
              for (int k = hsk[h]; k < hsk[h + 1]; ++k) {
                const int m = hlk[k];
                v = fma(g[K.ab[m]], K.prod[m], v);
              }
              W[x] = v;
            } else {
              const int y = x - nW, cd = coop::fast_div(y, inv_hab), h = y - cd * L.hab;
              for (int k = hsb[h]; k < hsb[h + 1]; ++k) {
                const int m = hlb[k];
                v = fma(G[B.ab[m] * L.ncd + cd], B.prod[m], v);
              }
              X[y] = v;
            }
          }
          fresh = false;
          __syncthreads();
          // V (bra products), U (ket products) and the raised sums
          double ev = 0.0, gp[3] = {0, 0, 0}, gb[3] = {0, 0, 0}, gk[3] = {0, 0, 0};
          const int nV = L.nnzb, nU = nV + L.nnzk, nZ = nU + L.hab * L.hcd;
          for (int x = tid; x < nZ; x += nt) {
            if (x < nV) {
              const double* wr = W + B.ab[x] * L.hcd;
              const double* r = R.R + B.lin[x];
              double v = 0.0;
              for (int h = 0; h < L.hcd; ++h) v = fma(wr[h], r[K.hlin[h]], v);
              ev = fma(B.prod[x], v, ev);
              for (int k = 0; k < 3; ++k) gb[k] = fma(B.dprod[k * L.nnzb + x], v, gb[k]);
            } else if (x < nU) {
              const int y = x - nV;
              const double* xr = X + K.ab[y] * L.hab;
              const double* r = R.R + K.lin[y];
              double v = 0.0;
              for (int h = 0; h < L.hab; ++h) v = fma(xr[h], r[B.hlin[h]], v);
              for (int k = 0; k < 3; ++k) gk[k] = fma(K.dprod[k * L.nnzk + y], v, gk[k]);
            } else {
              const int y = x - nU, h = coop::fast_div(y, inv_hcd), k = y - h * L.hcd;
              double z = 0.0;
              for (int m = hsb[h]; m < hsb[h + 1]; ++m) {
                const int o = hlb[m];
                z = fma(B.prod[o], W[B.ab[o] * L.hcd + k], z);
              }
              const double* r = R.R + B.hlin[h] + K.hlin[k];
              gp[0] = fma(z, r[SS], gp[0]);
              gp[1] = fma(z, r[S1], gp[1]);
              gp[2] = fma(z, r[1], gp[2]);
            }
          }
          const double mb = -2.0 * rb.bp * (1.0 - rb.bp) * rb.p * ev, mk = -2.0 * rk.bp * (1.0 - rk.bp) * rk.p * ev;
          for (int k = 0; k < 3; ++k) {
            acc[k] += (1.0 - rb.bp) * gp[k] + gb[k] + mb * AB[k];
            acc[3 + k] += gp[k];
            acc[6 + k] += (rk.bp - 1.0) * gp[k] + gk[k] + mk * CD[k];
          }
        }
      }
      // block sums of d/dA, d/dP, d/dC, then the four centres
      for (int k = 0; k < 9; ++k) {
        double v = acc[k];
        for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
        if (lane == 0) red[k * (kCoopThreads / 32) + warp] = v;
      }
      __syncthreads();
      if (tid < 12) {
        const int ax = tid % 3, centre = tid / 3;
        auto sum = [&](int k) {
          double v = 0.0;
          for (int x = 0; x < kCoopThreads / 32; ++x) v += red[k * (kCoopThreads / 32) + x];
          return v;
        };
        const double ga = sum(ax), gP = sum(3 + ax), gc = sum(6 + ax);
        const double v = centre == 0 ? ga : (centre == 1 ? gP - ga : (centre == 2 ? gc : -gP - gc));
        const int ao = centre == 0 ? bra.ao_a : (centre == 1 ? bra.ao_b : (centre == 2 ? ket.ao_a : ket.ao_b));
        atomicAdd(a.grad + 3 * a.ao_atom[ao] + ax, v);
      }
    }
  }
}

int resident_blocks(const void* kern, int threads, size_t smem) {
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
  return sms * (per_sm > 0 ? per_sm : 1);
}

template <int LA, int LB, int LC, int LD>
cudaError_t launch_lane(const GradArgs& a, long long ntasks, cudaStream_t st) {
  constexpr int NABCD = ncart(LA) * ncart(LB) * ncart(LC) * ncart(LD);
  auto kern = grad_lane_kernel<LA, LB, LC, LD>;
  const size_t smem = boys_smem_bytes<double>() + (size_t)(kLaneThreads / 32) * NABCD * lane_slots(NABCD) * 8 +
                      (a.natom <= kLaneGradAtoms ? (size_t)a.natom * 24 : 0);
  const cudaError_t err = raise_smem_limit<grad_lane_kernel<LA, LB, LC, LD>>();
  if (err != cudaSuccess) return err;
  // every task has at most 32 units of one warp each
  const long long want = (ntasks * 32 + kLaneThreads / 32 - 1) / (kLaneThreads / 32);
  const long long grid = std::min<long long>(want, resident_blocks((const void*)kern, kLaneThreads, smem));
  kern<<<(unsigned)grid, kLaneThreads, smem, st>>>(a);
  return cudaGetLastError();
}

}  // namespace

bool eri_gradient_splits(int la, int lb, int lc, int ld) {
  return la + lb + lc + ld <= 4 && !(la == 2 && lb == 1 && lc == 1 && ld == 0);
}

cudaError_t launch_eri_gradient(int la, int lb, int lc, int ld, const JKLaunchArgs& j, const int* ao_atom, int natom,
                                double* grad, cudaStream_t st) {
  if (la > kLMax || lb > kLMax || lc > kLMax || ld > kLMax) return cudaErrorInvalidValue;
  if (j.nchunks <= 0) return cudaSuccess;
  GradArgs a{};
  a.entries = j.entries;
  a.prefix = j.prefix;
  a.nentries = j.nentries;
  a.chunk_start = j.chunk_start;
  a.nchunks = j.nchunks;
  a.counter = j.counter;
  a.pairs = j.pairs;
  a.kets = j.kets;
  a.pairQ = j.pairQ;
  a.thr = j.thr;
  a.rec = j.rec64;
  a.boys = j.boys64;
  a.expt = j.expt64;
  a.P = j.Dtot;
  a.Ps = j.Dspin;
  a.nspin = j.nspin;
  a.n = j.n;
  a.natom = natom;
  a.ao_atom = ao_atom;
  a.grad = grad;
#define HFG_CASE(A, B, C, D) \
  if (la == A && lb == B && lc == C && ld == D) return launch_lane<A, B, C, D>(a, j.nwarps, st);
  HFG_CASE(0, 0, 0, 0)
  HFG_CASE(1, 0, 0, 0)
  HFG_CASE(1, 0, 1, 0)
  HFG_CASE(1, 1, 0, 0)
  HFG_CASE(1, 1, 1, 0)
  HFG_CASE(1, 1, 1, 1)
  HFG_CASE(2, 0, 0, 0)
  HFG_CASE(2, 0, 1, 0)
  HFG_CASE(2, 0, 1, 1)
  HFG_CASE(2, 0, 2, 0)
  HFG_CASE(2, 1, 0, 0)
  HFG_CASE(2, 2, 0, 0)
#undef HFG_CASE
  const MDClass c = md_class(la, lb, lc, ld);
  const size_t smem = coop_smem(c);
  const cudaError_t err = raise_smem_limit<grad_coop_kernel>();
  if (err != cudaSuccess) return err;
  const long long grid =
      std::min<long long>(j.nwarps * 32, resident_blocks((const void*)grad_coop_kernel, kCoopThreads, smem));
  grad_coop_kernel<<<(unsigned)grid, kCoopThreads, smem, st>>>(c, a);
  return cudaGetLastError();
}

}  // namespace hfg
