// Shell quartets with an f shell (l = 3): a generic McMurchie-Davidson
// engine, one thread block per shell quartet.
//
// The generated Obara-Saika kernels (eri_gen.cuh) cover s, p and d; their
// straight-line recursions grow too large to compile beyond that.  Classes
// with an f shell take this path instead, for every entry point: Schwarz
// bounds, the single-quartet block, the packed tensor and the direct J/K
// build (same work queues as the fast kernels, FP64 only).  It restates the
// scheme of hf-rs's shell engine (src/shell_integrals.rs:92-135 with
// src/integrals.rs:107-191 and :253-346) on the sparse tables of md_coop.cuh:
//
//   for every ket primitive pair Q:
//     for every bra primitive pair P:
//       the axis tables, Boys values and one-axis polynomials (a warp each),
//       the products E^{ab}_h (with the prefactor) and R,
//       G[k][ab] += sum_h E^{ab}_h R_{h+k}
//     out[ab][cd] += sum_k (-1)^{|k|} E^{cd}_k G[k][ab]     (in registers)
//
// so the second, larger contraction runs once per ket primitive pair.  The
// block is 32 to 512 threads by the size of (ab|cd), and the quartets of a
// launch are handed out one by one.  What bounds it: shared-memory loads in
// the two contractions (six for four multiply-adds) for the large classes, the
// chain of short steps with a barrier each for the small ones.
#include <cuda_runtime.h>

#include <algorithm>

#include "df_internal.h"
#include "eri_md.h"
#include "jk_dispatch.h"
#include "eri_prim.cuh"
#include "md_coop.cuh"
#include "smem_limit.h"

namespace hfg {

namespace {

constexpr int kMDThreads = 512;  // largest block
constexpr int kMDAcc = 20;       // output elements per thread, at most

// Threads by the number of items of four block elements: enough that each
// holds at most kMDAcc elements ((ff|ff): 2,500 items over 512), and no more,
// since the per-primitive steps of the small classes are shorter than a
// barrier of a wide block.
__host__ __device__ inline int md_items(const MDClass& c) { return (c.na * c.nb + 3) / 4 * c.nc * c.nd; }
__host__ __device__ inline int md_threads(const MDClass& c) {
  const int n = md_items(c);
  return n <= 32 ? 32 : (n <= 128 ? 64 : (n <= 384 ? 128 : (n <= 1024 ? 256 : 512)));
}

// Density blocks of one quartet's digestion: D[cd], D[ab], then per spin
// D[bd], D[ad], D[bc], D[ac].
__host__ __device__ inline int md_dsize(const MDClass& c) {
  return c.nc * c.nd + c.na * c.nb + 2 * (c.nb * c.nd + c.na * c.nd + c.nb * c.nc + c.na * c.nc);
}

// Shared memory of one block: scalars, G (and, once a quartet is complete,
// its block, which takes G's place and the R tables'), R tables, the sides
// and the density blocks.
struct MDShared {
  int nab, ncd, gs, os;  // gs, os: odd row strides of G[k][ab] and out[cd][ab]
  int na4;               // a thread's elements of one cd are ab, ab + na4, ab + 2 na4, ab + 3 na4
  float inv_na4;
  double *S, *G, *out, *D;
  coop::Side B, K;
  coop::RTab R;
};

__host__ __device__ inline size_t md_work_bytes(const MDClass& c) {
  const size_t nab = c.na * c.nb, ncd = c.nc * c.nd;
  const size_t g = 8 * (nab | 1) * coop::nherm(c.lcd) + coop::rtab_bytes(c.L), o = 8 * (nab | 1) * ncd;
  return g > o ? g : o;
}

size_t md_smem(const MDClass& c, bool digest) {
  return 64 + md_work_bytes(c) + coop::side_bytes(c.la, c.lb, false) + coop::side_bytes(c.lc, c.ld, false) +
         (digest ? 8 * (size_t)md_dsize(c) : 0);
}

__device__ void md_setup(const MDClass& c, unsigned char* raw, MDShared& s) {
  s.nab = c.na * c.nb;
  s.ncd = c.nc * c.nd;
  s.gs = s.os = s.nab | 1;
  s.na4 = (s.nab + 3) / 4;
  s.inv_na4 = 1.0f / s.na4;
  s.S = reinterpret_cast<double*>(raw);
  unsigned char* p = raw + 64;
  s.G = s.out = reinterpret_cast<double*>(p);
  coop::rtab_carve(s.R, c.L, p + 8 * (size_t)s.gs * coop::nherm(c.lcd));
  p += md_work_bytes(c);
  p = coop::side_carve(s.B, c.la, c.lb, false, p);
  p = coop::side_carve(s.K, c.lc, c.ld, false, p);
  s.D = reinterpret_cast<double*>(p);
  coop::side_setup(s.B, s.R.S);
  coop::side_setup(s.K, s.R.S);
  __syncthreads();
}

// One primitive pair: exponent sum, 1/p, K_p (contraction coefficients,
// Gaussian product factor and 1/p) and P - A.
struct MDPrim {
  double p, inv_p, kp, PA[3];
};

// A primitive pair from the 64-byte table (PrimPair, P - A stored).
struct PrimTable {
  const PrimPair* t;
  __device__ __forceinline__ MDPrim operator()(int k) const {
    const PrimPair& q = t[k];
    return MDPrim{q.p, q.inv_p, q.kp, {q.PAx, q.PAy, q.PAz}};
  }
  __device__ __forceinline__ float bound(int) const { return 0.f; }
};

// A primitive pair from the compact records (P - A = -(beta/p) AB).
struct PrimRecs {
  const PrimRec64* rec;
  const float* pbound;
  size_t off, stride;
  const double* AB;
  __device__ __forceinline__ MDPrim operator()(int k) const {
    const PrimRec64 r = rec[off + k * stride];
    return MDPrim{r.p, r.inv_p, r.kp, {-r.bp * AB[0], -r.bp * AB[1], -r.bp * AB[2]}};
  }
  __device__ __forceinline__ float bound(int k) const { return pbound[off + k * stride]; }
};

// The contracted block of nb x nk primitive pairs in acc, four elements
// (cd; ab, ab + na4, ...) per item cd na4 + ab of thread item % nt; primitive quartets with bound products
// below eps are skipped (eps = 0: none).  The R tables' index list is made
// here, since a finished block overwrites it.
template <int ACC, typename PB, typename PK>
__device__ __forceinline__ void md_quartet(const MDShared& s, const PB& pb, int nb, const PK& pk, int nk,
                                           const double* AB, const double* CD, const double* AC, double eps,
                                           const double* __restrict__ boys,
                                           double (&acc)[ACC]) {
  const int tid = threadIdx.x, nt = blockDim.x, warp = tid >> 5, lane = tid & 31, nw = nt >> 5;
  const int nh = s.K.nh, nq = (nh + 3) / 4;
  const float inv_nq = 1.0f / nq, feps = (float)eps;
#pragma unroll
  for (int i = 0; i < ACC; ++i) acc[i] = 0.0;
  __syncthreads();  // the previous block has been read
  coop::rtab_setup(s.R);
  for (int ik = 0; ik < nk; ++ik) {
    const MDPrim Q = pk(ik);
    const float kb = eps > 0.0 ? pk.bound(ik) : 0.f;
    bool first = true;
    for (int ib = 0; ib < nb; ++ib) {
      if (eps > 0.0 && pb.bound(ib) * kb < feps) continue;
      const MDPrim P = pb(ib);
      __syncthreads();  // the tables of the previous primitive quartet have been read
      for (int role = warp; role < 4; role += nw) {
        if (role == 0) {
          coop::side_axes(s.B, lane, AB, P.PA, 0.0, P.inv_p);
        } else if (role == 1) {
          if (first) coop::side_axes(s.K, lane, CD, Q.PA, 0.0, Q.inv_p);
        } else {
          const double PQ[3] = {AC[0] + P.PA[0] - Q.PA[0], AC[1] + P.PA[1] - Q.PA[1], AC[2] + P.PA[2] - Q.PA[2]};
          if (role == 2) {
            coop::rtab_poly(s.R, lane, PQ);
          } else {
            const double sum = P.p + Q.p, r = rsqrt(sum), alpha = P.p * Q.p * r * r;
            coop::boys_base(alpha * (PQ[0] * PQ[0] + PQ[1] * PQ[1] + PQ[2] * PQ[2]), alpha, s.R.L, lane, boys, s.R.base);
            if (lane == 0) s.S[0] = kTwoPiPow25 * P.kp * Q.kp * r;
          }
        }
      }
      __syncthreads();
      const double pref = s.S[0];
      coop::rtab_build(s.R, [&] {
        coop::side_products(s.B, tid, nt, pref, false, s.R.S);
        if (first) coop::side_products(s.K, tid, nt, 1.0, true, s.R.S);
      });
      // G[k][ab] (+)= sum_h E^{ab}_h R_{h+k}: a thread takes up to four k of
      // one ab, so that the products and their offsets are loaded once for
      // four multiply-adds; neighbouring threads share ab
      for (int x = tid; x < s.nab * nq; x += nt) {
        const int ab = coop::fast_div(x, inv_nq), h = x - ab * nq;
        const int h1 = min(h + nq, nh - 1), h2 = min(h + 2 * nq, nh - 1), h3 = min(h + 3 * nq, nh - 1);
        const double *r0 = s.R.R + s.K.hlin[h], *r1 = s.R.R + s.K.hlin[h1], *r2 = s.R.R + s.K.hlin[h2],
                     *r3 = s.R.R + s.K.hlin[h3];
        double g0 = 0.0, g1 = 0.0, g2 = 0.0, g3 = 0.0;
        const int k1 = s.B.start[ab + 1];
#pragma unroll 2
        for (int k = s.B.start[ab]; k < k1; ++k) {
          const double f = s.B.prod[k];
          const int o = s.B.lin[k];
          g0 = fma(f, r0[o], g0);
          g1 = fma(f, r1[o], g1);
          g2 = fma(f, r2[o], g2);
          g3 = fma(f, r3[o], g3);
        }
        double* o = s.G + ab;
        auto put = [&](int k, double g) { o[k * s.gs] = first ? g : o[k * s.gs] + g; };
        put(h, g0);
        if (h + nq < nh) put(h1, g1);
        if (h + 2 * nq < nh) put(h2, g2);
        if (h + 3 * nq < nh) put(h3, g3);
      }
      first = false;
    }
    if (first) continue;  // every bra primitive screened out
    __syncthreads();
    // out += sum_k E^{cd}_k G[k][ab], up to four ab of one cd per thread;
    // neighbouring threads share cd
#pragma unroll
    for (int i = 0; i < ACC / 4; ++i) {
      const int x = tid + i * nt;
      if (x < s.ncd * s.na4) {
        const int cd = coop::fast_div(x, s.inv_na4), ab = x - cd * s.na4;
        const double* g = s.G + ab;
        const int o1 = min(s.na4, s.nab - 1 - ab), o2 = min(2 * s.na4, s.nab - 1 - ab), o3 = min(3 * s.na4, s.nab - 1 - ab);
        double v0 = 0.0, v1 = 0.0, v2 = 0.0, v3 = 0.0;
        const int k1 = s.K.start[cd + 1];
#pragma unroll 2
        for (int k = s.K.start[cd]; k < k1; ++k) {
          const double f = s.K.prod[k];
          const double* r = g + s.K.h[k] * s.gs;
          v0 = fma(f, r[0], v0);
          v1 = fma(f, r[o1], v1);
          v2 = fma(f, r[o2], v2);
          v3 = fma(f, r[o3], v3);
        }
        acc[4 * i] += v0;
        acc[4 * i + 1] += v1;
        acc[4 * i + 2] += v2;
        acc[4 * i + 3] += v3;
      }
    }
  }
}

// acc scaled by f and the component scales into out[cd][ab].
template <int ACC>
__device__ __forceinline__ void md_store(const MDShared& s, const double (&acc)[ACC], double f) {
  const int nt = blockDim.x;
  __syncthreads();  // G and R have been read
#pragma unroll
  for (int i = 0; i < ACC / 4; ++i) {
    const int x = threadIdx.x + i * nt;
    if (x < s.ncd * s.na4) {
      const int cd = coop::fast_div(x, s.inv_na4), ab0 = x - cd * s.na4;
      const double fc = f * s.K.scale[cd];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int ab = ab0 + j * s.na4;
        if (ab < s.nab) s.out[cd * s.os + ab] = acc[4 * i + j] * fc * s.B.scale[ab];
      }
    }
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------
// Schwarz bounds: shell pairs (prim_mode 0) or primitive pairs (prim_mode 1)
// over persistent blocks, sqrt of the largest scaled diagonal element.
template <int ACC>
__global__ void __launch_bounds__(ACC == 8 ? 64 : kMDThreads, ACC == 8 ? 8 : 1) schwarz_md_kernel(MDClass c, const PairInfo* __restrict__ pairs,
                                                                const PrimPair* __restrict__ prims, int first,
                                                                int count, const double* __restrict__ boys,
                                                                double* __restrict__ out, int prim_mode) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  MDShared s;
  __shared__ double red[kMDThreads / 32];
  md_setup(c, smem_raw, s);
  for (int t = blockIdx.x; t < count; t += gridDim.x) {
    const int p0 = prim_mode ? first + t : pairs[first + t].pp_off;
    const int np = prim_mode ? 1 : pairs[first + t].npp;
    const PairInfo owner = prim_mode ? pairs[(int)prims[p0].pad] : pairs[first + t];
    const double AB[3] = {owner.ABx, owner.ABy, owner.ABz}, AC[3] = {0.0, 0.0, 0.0};
    double acc[ACC];
    const PrimTable tab{prims + p0};
    md_quartet<ACC>(s, tab, np, tab, np, AB, AB, AC, 0.0, boys, acc);
    md_store<ACC>(s, acc, 1.0);
    double m = 0.0;
    for (int ij = threadIdx.x; ij < s.nab; ij += blockDim.x) m = fmax(m, s.out[ij * s.os + ij]);
    for (int off = 16; off > 0; off >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, off));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
      double r = 0.0;
      for (int k = 0; k < (int)(blockDim.x >> 5); ++k) r = fmax(r, red[k]);
      out[t] = sqrt(r);
    }
  }
}

// One full scaled block (ab|cd) of bra pairs[0], ket pairs[1].
template <int ACC>
__global__ void __launch_bounds__(ACC == 8 ? 64 : kMDThreads, ACC == 8 ? 8 : 1) quartet_md_kernel(MDClass c, const PairInfo* __restrict__ pairs,
                                                                const PrimPair* __restrict__ prims,
                                                                const double* __restrict__ boys,
                                                                double* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  MDShared s;
  md_setup(c, smem_raw, s);
  const PairInfo bra = pairs[0], ket = pairs[1];
  const double AB[3] = {bra.ABx, bra.ABy, bra.ABz}, CD[3] = {ket.ABx, ket.ABy, ket.ABz};
  const double AC[3] = {bra.Ax - ket.Ax, bra.Ay - ket.Ay, bra.Az - ket.Az};
  double acc[ACC];
  md_quartet<ACC>(s, PrimTable{prims + bra.pp_off}, bra.npp, PrimTable{prims + ket.pp_off}, ket.npp, AB, CD, AC, 0.0,
                  boys, acc);
  md_store<ACC>(s, acc, 1.0);
  for (int x = threadIdx.x; x < s.nab * s.ncd; x += blockDim.x) out[x] = s.out[(x % s.ncd) * s.os + x / s.ncd];
}

__device__ __forceinline__ unsigned long long md_compound(unsigned long long i, unsigned long long j) {
  return i >= j ? i * (i + 1) / 2 + j : j * (j + 1) / 2 + i;
}

// Contracted block of (bra|ket) from the compact records.
template <int ACC>
__device__ __forceinline__ void md_quartet_rec(const MDShared& s, const PairInfo& bra, const PairInfo& ket,
                                               unsigned slice, const PrimRec64* __restrict__ rec,
                                               const float* __restrict__ pbound, double eps,
                                               const double* __restrict__ boys,
                                               double (&acc)[ACC]) {
  const double AB[3] = {bra.ABx, bra.ABy, bra.ABz}, CD[3] = {ket.ABx, ket.ABy, ket.ABz};
  const double AC[3] = {bra.Ax - ket.Ax, bra.Ay - ket.Ay, bra.Az - ket.Az};
  const PrimRange rb = prim_range(bra.rec_off, bra.rec_stride, bra.npp, slice, 0);
  const PrimRange rk = prim_range(ket.rec_off, ket.rec_stride, ket.npp, slice, 16);
  const PrimRecs pb{rec, pbound, (size_t)rb.off, (size_t)rb.stride, AB};
  const PrimRecs pk{rec, pbound, (size_t)rk.off, (size_t)rk.stride, CD};
  md_quartet<ACC>(s, pb, rb.count, pk, rk.count, AB, CD, AC, eps, boys, acc);
}

// Packed 8-fold tensor slots of the plan's quartets (the writer rules of
// eri_packed_kernel: i >= j within a same-shell pair, IJ >= KL for a pair
// with itself), over units of one ket of one warp task.
template <int ACC>
__global__ void __launch_bounds__(ACC == 8 ? 64 : kMDThreads, ACC == 8 ? 8 : 1) eri_packed_md_kernel(
    MDClass c, const JKEntry* __restrict__ entries, const long long* __restrict__ prefix, int nentries,
    long long nwarps, const PairInfo* __restrict__ pairs, const double* __restrict__ pairQ, double thr,
    const PrimRec64* __restrict__ rec, const float* __restrict__ pbound, const double* __restrict__ boys, double* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  MDShared s;
  md_setup(c, smem_raw, s);
  int e = 0;
  for (long long u = blockIdx.x; u < nwarps * 32; u += gridDim.x) {
    const long long w = u >> 5;
    e = coop::entry_of(prefix, nentries, w, e);
    const JKEntry ent = entries[e];
    const int kidx = ent.k_lo + (int)(w - prefix[e]) * 32 + (int)(u & 31);
    if (kidx >= ent.k_hi || !(pairQ[kidx] * pairQ[ent.bra] > thr)) continue;
    const PairInfo bra = pairs[ent.bra], ket = pairs[kidx];
    double acc[ACC];
    md_quartet_rec<ACC>(s, bra, ket, 0u, rec, pbound, 0.0, boys, acc);
    md_store<ACC>(s, acc, 1.0);
    const bool self = kidx == ent.bra;
    for (int x = threadIdx.x; x < s.nab * s.ncd; x += blockDim.x) {
      const int ab = x / s.ncd, cd = x % s.ncd;
      const int mu = bra.ao_a + ab / c.nb, nu = bra.ao_b + ab % c.nb;
      const int lam = ket.ao_a + cd / c.nd, sig = ket.ao_b + cd % c.nd;
      if (bra.same && mu < nu) continue;
      if (ket.same && lam < sig) continue;
      const unsigned long long IJ = md_compound(mu, nu), KL = md_compound(lam, sig);
      if (self && IJ < KL) continue;
      out[md_compound(IJ, KL)] = s.out[cd * s.os + ab];
    }
  }
}

// Direct J/K (FP64) over a launch's work queue, for the classes with an f
// shell and, of the others, the launches of few quartets in a class whose
// generated code is too long to run cold (coop_launch in ctx.cu).  A unit of
// work is one ket lane of one work-queue step; persistent blocks take units
// in runs of `per` and digest each quartet as the fast kernels do
// (jk_kernels.cuh): J'[a,b] += 4w sum D[c,d], J'[c,d] += 4w sum D[a,b],
// K'[a,c] += 2w sum D[b,d] and the three other exchange blocks, w the
// quartet's degeneracy weight.  In deterministic mode one block runs the
// queue and one thread issues every atomic of a quartet, quartet after
// quartet.  BATCH: the queues of several molecules (RHF), as jk_batch_kernel.
template <int ACC, bool BATCH>
__global__ void __launch_bounds__(ACC == 8 ? 64 : kMDThreads, ACC == 8 ? 8 : 1) jk_md_kernel(MDClass c, const JKLaunchArgs args, int per) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  MDShared s;
  __shared__ long long s_unit;
  md_setup(c, smem_raw, s);
  JKLaunchArgs a = args;
  const int NS = BATCH ? 1 : a.nspin, tid = threadIdx.x, nt = blockDim.x;
  const int na = c.na, nb = c.nb, nc = c.nc, nd = c.nd;
  double* Dcd = s.D;
  double* Dab = Dcd + nc * nd;
  double* Dk = Dab + na * nb;  // per spin: bd, ad, bc, ac
  const int nbd = nb * nd, nad = na * nd, nbc = nb * nc, nac = na * nc, nK = nbd + nad + nbc + nac;
  for (;;) {
    __syncthreads();
    if (tid == 0) s_unit = (long long)atomicAdd(args.counter, (unsigned long long)per);
    __syncthreads();
    const long long u0 = s_unit;
    if (u0 >= args.nchunks * 32) break;
    // `per` divides 32: one step, lanes [lane0, lane0 + per) of its tasks
    long long step = u0 >> 5;
    const int lane0 = (int)(u0 & 31);
    if (BATCH) {
      int lo = 0, hi = args.njobs;  // last job whose first step is <= step
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(args.job_steps + mid) <= step) lo = mid; else hi = mid;
      }
      step -= __ldg(args.job_steps + lo);
      const JKJob& jb = args.jobs[lo];
      a.entries = jb.entries;
      a.prefix = jb.prefix;
      a.chunk_start = jb.chunk_start;
      a.chunk_entry = jb.chunk_entry;
      a.pairs = jb.pairs;
      a.pairQ = jb.pairQ;
      a.rec64 = jb.rec64;
      a.pbound = jb.pbound;
      a.Dtot = a.Dspin = jb.Dtot;
      a.Jacc = jb.Jacc;
      a.Kacc = jb.Kacc;
      a.n = jb.n;
      a.thr = jb.thr;
      a.prim_eps = jb.prim_eps;
    }
    const int n = a.n;
    const long long t0 = a.chunk_start[step], tasks = a.chunk_start[step + 1] - t0;
    int e = a.chunk_entry[step];
    for (long long u = 0; u < tasks * per; ++u) {
      const long long w = t0 + u / per;
      while (a.prefix[e + 1] <= w) ++e;
      const JKEntry ent = a.entries[e];
      const int kidx = ent.k_lo + (int)(w - a.prefix[e]) * 32 + lane0 + (int)(u % per);
      if (kidx >= ent.k_hi || !(a.pairQ[kidx] * a.pairQ[ent.bra] > a.thr)) continue;
      const PairInfo bra = a.pairs[ent.bra], ket = a.pairs[kidx];
      double acc[ACC];
      md_quartet_rec<ACC>(s, bra, ket, ent.slice, a.rec64, a.pbound, a.prim_eps, args.boys64, acc);
      double deg = 1.0;
      if (bra.same) deg *= 0.5;
      if (ket.same) deg *= 0.5;
      if (kidx == ent.bra) deg *= 0.5;
      const int i0 = bra.ao_a, j0 = bra.ao_b, k0 = ket.ao_a, l0 = ket.ao_b;
      // the density blocks (the previous quartet's have been read: md_quartet
      // synchronises at its start)
      auto fetch = [&](double* dst, const double* D, int r0, int nr, int c0, int ncl) {
        for (int x = tid; x < nr * ncl; x += nt) dst[x] = __ldg(D + (size_t)(r0 + x / ncl) * n + c0 + x % ncl);
      };
      fetch(Dcd, a.Dtot, k0, nc, l0, nd);
      fetch(Dab, a.Dtot, i0, na, j0, nb);
      for (int sp = 0; sp < NS; ++sp) {
        const double* D = a.Dspin + (size_t)sp * n * n;
        double* d = Dk + sp * nK;
        fetch(d, D, j0, nb, l0, nd);
        fetch(d + nbd, D, i0, na, l0, nd);
        fetch(d + nbd + nad, D, j0, nb, k0, nc);
        fetch(d + nbd + nad + nbc, D, i0, na, k0, nc);
      }
      md_store<ACC>(s, acc, deg);
      // items: J'[ab], J'[cd], then per spin K'[ac], K'[bc], K'[ad], K'[bd];
      // they can add into the same element (J'[ab] and J'[cd] of a pair with
      // itself, K' blocks of a same-shell pair): in deterministic mode one
      // thread takes every item in order
      const int items = s.nab + s.ncd + NS * nK;
      const int x0 = a.serial ? (tid == 0 ? 0 : items) : tid, dx = a.serial ? 1 : nt;
      for (int x = x0; x < items; x += dx) {
        double v = 0.0;
        if (x < s.nab) {
          for (int cd = 0; cd < s.ncd; ++cd) v = fma(s.out[cd * s.os + x], Dcd[cd], v);
          atomicAdd(a.Jacc + (size_t)(i0 + x / nb) * n + j0 + x % nb, 4.0 * v);
          continue;
        }
        int y = x - s.nab;
        if (y < s.ncd) {
          for (int ab = 0; ab < s.nab; ++ab) v = fma(s.out[y * s.os + ab], Dab[ab], v);
          atomicAdd(a.Jacc + (size_t)(k0 + y / nd) * n + l0 + y % nd, 4.0 * v);
          continue;
        }
        y -= s.ncd;
        const int sp = y / nK;
        int r = y % nK;
        const double* d = Dk + sp * nK;
        double* K = a.Kacc + (size_t)sp * n * n;
        if (r < nac) {  // K'[a,c] from D[b,d]
          const int i = r / nc, k = r % nc;
          for (int l = 0; l < nd; ++l)
            for (int j = 0; j < nb; ++j) v = fma(s.out[(k * nd + l) * s.os + i * nb + j], d[j * nd + l], v);
          atomicAdd(K + (size_t)(i0 + i) * n + k0 + k, 2.0 * v);
          continue;
        }
        r -= nac;
        if (r < nbc) {  // K'[b,c] from D[a,d]
          const int j = r / nc, k = r % nc;
          for (int l = 0; l < nd; ++l)
            for (int i = 0; i < na; ++i) v = fma(s.out[(k * nd + l) * s.os + i * nb + j], d[nbd + i * nd + l], v);
          atomicAdd(K + (size_t)(j0 + j) * n + k0 + k, 2.0 * v);
          continue;
        }
        r -= nbc;
        if (r < nad) {  // K'[a,d] from D[b,c]
          const int i = r / nd, l = r % nd;
          for (int k = 0; k < nc; ++k)
            for (int j = 0; j < nb; ++j) v = fma(s.out[(k * nd + l) * s.os + i * nb + j], d[nbd + nad + j * nc + k], v);
          atomicAdd(K + (size_t)(i0 + i) * n + l0 + l, 2.0 * v);
          continue;
        }
        r -= nad;
        {  // K'[b,d] from D[a,c]
          const int j = r / nd, l = r % nd;
          for (int k = 0; k < nc; ++k)
            for (int i = 0; i < na; ++i)
              v = fma(s.out[(k * nd + l) * s.os + i * nb + j], d[nbd + nad + nbc + i * nc + k], v);
          atomicAdd(K + (size_t)(j0 + j) * n + l0 + l, 2.0 * v);
        }
      }
      if (a.serial) __threadfence();
    }
  }
}

// Three-centre blocks (ab|P 1) (df_kernels.cu's df3c_kernel) for launches of
// few combinations in a high class: one combination per block at a time.
template <int ACC>
__global__ void __launch_bounds__(ACC == 8 ? 64 : kMDThreads, ACC == 8 ? 8 : 1) df3c_md_kernel(MDClass c, const Df3cArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  MDShared s;
  md_setup(c, smem_raw, s);
  const long long total = (long long)a.nbra * a.nket;
  for (long long t = blockIdx.x; t < total; t += gridDim.x) {
    const int ib = (int)(t % a.nbra), ik = (int)(t / a.nbra);
    const PairInfo bra = a.bra_pairs[a.bra_idx[ib]], ket = a.ket_pairs[a.ket_idx[ik]];
    const double AB[3] = {bra.ABx, bra.ABy, bra.ABz}, CD[3] = {0.0, 0.0, 0.0};
    const double AC[3] = {bra.Ax - ket.Ax, bra.Ay - ket.Ay, bra.Az - ket.Az};
    double acc[ACC];
    md_quartet<ACC>(s, PrimTable{a.bra_prims + bra.pp_off}, bra.npp, PrimTable{a.ket_prims + ket.pp_off}, ket.npp, AB, CD,
                    AC, 0.0, a.boys, acc);
    md_store<ACC>(s, acc, 1.0);
    const long long col0 = a.bra_col[ib];
    for (int x = threadIdx.x; x < s.nab * s.ncd; x += blockDim.x) {
      const int k = x / s.nab, ab = x % s.nab, i = ab / c.nb, j = ab % c.nb;
      if (bra.same && j > i) continue;
      const long long col = bra.same ? col0 + i * (i + 1) / 2 + j : col0 + ab;
      a.out[(long long)(ket.ao_a + k) * a.ld + col] = s.out[k * s.os + ab];
    }
  }
}

int md_resident_blocks(const void* kern, int threads, size_t smem) {
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
  return sms * (per_sm > 0 ? per_sm : 1);
}

// the kernel instantiation of a class: two items per thread up to 128 items
// (md_threads), five beyond
bool md_small(const MDClass& c) { return md_items(c) <= 128; }
template <auto Small, auto Large>
auto md_kernel(const MDClass& c, cudaError_t& e) {
  e = md_small(c) ? raise_smem_limit<Small>() : raise_smem_limit<Large>();
  return md_small(c) ? Small : Large;
}

}  // namespace

MDClass md_class(int la, int lb, int lc, int ld) {
  MDClass c;
  c.la = la;
  c.lb = lb;
  c.lc = lc;
  c.ld = ld;
  c.na = ncart(la);
  c.nb = ncart(lb);
  c.nc = ncart(lc);
  c.nd = ncart(ld);
  c.lab = la + lb;
  c.lcd = lc + ld;
  c.L = c.lab + c.lcd;
  return c;
}

int md_blocks_per_sm(int la, int lb, int lc, int ld) {
  const int nt = md_threads(md_class(la, lb, lc, ld));
  return nt >= 512 ? 1 : (nt == 256 ? 2 : (nt == 128 ? 4 : 8));
}

bool md_class_ok(int la, int lb, int lc, int ld) {
  return la >= 0 && lb >= 0 && lc >= 0 && ld >= 0 && la <= kMDLMax && lb <= kMDLMax && lc <= kMDLMax &&
         ld <= kMDLMax;
}

cudaError_t launch_df3c_md(int la, int lb, int lc, const Df3cArgs& args, cudaStream_t st) {
  const long long total = (long long)args.nbra * args.nket;
  if (total <= 0) return cudaSuccess;
  const MDClass c = md_class(la, lb, lc, 0);
  const size_t smem = md_smem(c, false);
  cudaError_t e = cudaSuccess;
  auto kern = md_kernel<df3c_md_kernel<8>, df3c_md_kernel<kMDAcc>>(c, e);
  if (e != cudaSuccess) return e;
  const int nt = md_threads(c);
  kern<<<(unsigned)std::min<long long>(total, md_resident_blocks((const void*)kern, nt, smem)), nt, smem, st>>>(c, args);
  return cudaGetLastError();
}

cudaError_t launch_schwarz_md(int la, int lb, const PairInfo* pairs, const PrimPair* prims, int first, int count,
                              const double* boys, double* out, int prim_mode, cudaStream_t st) {
  if (!md_class_ok(la, lb, la, lb)) return cudaErrorInvalidValue;
  if (count <= 0) return cudaSuccess;
  const MDClass c = md_class(la, lb, la, lb);
  const size_t smem = md_smem(c, false);
  cudaError_t e = cudaSuccess;
  auto kern = md_kernel<schwarz_md_kernel<8>, schwarz_md_kernel<kMDAcc>>(c, e);
  if (e != cudaSuccess) return e;
  const int nt = md_threads(c), grid = std::min(count, md_resident_blocks((const void*)kern, nt, smem));
  kern<<<(unsigned)grid, nt, smem, st>>>(c, pairs, prims, first, count, boys, out, prim_mode);
  return cudaGetLastError();
}

cudaError_t launch_quartet_md(int la, int lb, int lc, int ld, const PairInfo* pairs, const PrimPair* prims,
                              const double* boys, double* out, cudaStream_t st) {
  if (!md_class_ok(la, lb, lc, ld)) return cudaErrorInvalidValue;
  const MDClass c = md_class(la, lb, lc, ld);
  const size_t smem = md_smem(c, false);
  cudaError_t e = cudaSuccess;
  auto kern = md_kernel<quartet_md_kernel<8>, quartet_md_kernel<kMDAcc>>(c, e);
  if (e != cudaSuccess) return e;
  kern<<<1, md_threads(c), smem, st>>>(c, pairs, prims, boys, out);
  return cudaGetLastError();
}

cudaError_t launch_eri_packed_md(int la, int lb, int lc, int ld, const JKEntry* entries, const long long* prefix,
                                 int nentries, long long nwarps, const PairInfo* pairs, const double* pairQ,
                                 double thr, const PrimRec64* rec, const float* pbound, const double* boys,
                                 double* out, cudaStream_t st) {
  if (!md_class_ok(la, lb, lc, ld)) return cudaErrorInvalidValue;
  if (nwarps <= 0) return cudaSuccess;
  if (nwarps > 0x7fffffffLL) return cudaErrorInvalidValue;
  const MDClass c = md_class(la, lb, lc, ld);
  const size_t smem = md_smem(c, false);
  cudaError_t e = cudaSuccess;
  auto kern = md_kernel<eri_packed_md_kernel<8>, eri_packed_md_kernel<kMDAcc>>(c, e);
  if (e != cudaSuccess) return e;
  const int nt = md_threads(c);
  const long long grid = std::min<long long>(nwarps * 32, md_resident_blocks((const void*)kern, nt, smem));
  kern<<<(unsigned)grid, nt, smem, st>>>(c, entries, prefix, nentries, nwarps, pairs, pairQ, thr, rec, pbound, boys, out);
  return cudaGetLastError();
}

cudaError_t launch_jk_md(int la, int lb, int lc, int ld, const JKLaunchArgs& a, cudaStream_t st) {
  if (!md_class_ok(la, lb, lc, ld)) return cudaErrorInvalidValue;
  if (a.nchunks <= 0) return cudaSuccess;
  const MDClass c = md_class(la, lb, lc, ld);
  const size_t smem = md_smem(c, true);
  cudaError_t e = cudaSuccess;
  auto kern = a.jobs ? md_kernel<jk_md_kernel<8, true>, jk_md_kernel<kMDAcc, true>>(c, e)
                     : md_kernel<jk_md_kernel<8, false>, jk_md_kernel<kMDAcc, false>>(c, e);
  if (e != cudaSuccess) return e;
  const int nt = md_threads(c);
  const long long units = a.nchunks * 32;
  const long long grid = a.serial ? 1 : std::min<long long>(units, md_resident_blocks((const void*)kern, nt, smem));
  // short runs while there are units to spare for every block
  int per = a.serial ? 32 : 1;
  while (per < 32 && units > 2LL * per * grid * 16) per *= 2;
  kern<<<(unsigned)grid, nt, smem, st>>>(c, a, per);
  return cudaGetLastError();
}

}  // namespace hfg
