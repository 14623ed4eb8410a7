// One-electron integrals S, T, V on the device (needed by the SCF driver).
//
// McMurchie-Davidson form, as hf-rs computes them (src/integrals.rs:408-535,
// :747-793; src/scf.rs:247-271).  S and T: one thread per Cartesian function
// pair mu >= nu, looping over primitive pairs; Hermite expansion coefficients
// E_t^{ij} per axis, S = E_0^x E_0^y E_0^z (pi/p)^{3/2}, T from the overlap
// recursion with lb +- 2 (instantiated for shells up to d, LM = 2, and up to
// f, LM = 3; the kinetic term needs E up to lb + 2).  V = -Z 2pi/p sum E_t E_u
// E_v R_tuv(p, P - C) over nuclei: one warp per shell pair (nuc_kernel).
#include <cuda_runtime.h>

#include "boys.cuh"
#include "eri_prim.cuh"
#include "grad_gen.cuh"
#include "hfg_ctx.h"
#include "md_coop.cuh"
#include "smem_limit.h"

namespace hfg {

// Hermite table extents for shells up to angular momentum LM
template <int LM> struct OneIntDims {
  static constexpr int EI = LM + 1;      // i index 0..LM
  static constexpr int EJ = LM + 3;      // j index 0..LM+2 (lb + 2)
  static constexpr int ET = 2 * LM + 3;  // t index
};

struct FuncInfo {
  double c[3];
  int l[3];
  int shell;
};

struct OneIntArgs {
  const FuncInfo* funcs;
  const double* exps;   // per shell primitive exponents (shell prim_off)
  const double* coefs;  // per shell contraction coefficients (component scale applied below)
  const int* sh_off;    // shell -> prim offset
  const int* sh_K;      // shell -> primitive count
  int n;
  double *S, *T;  // n x n
};

// E[i][j][t] for one axis, i <= la, j <= lb (+2 allowed), 1D MD recursion.
template <int LM>
__device__ __forceinline__ void hermite_1d(int la, int lb, double alpha, double beta, double a, double b,
                                           double E[OneIntDims<LM>::EI][OneIntDims<LM>::EJ][OneIntDims<LM>::ET]) {
  constexpr int kET = OneIntDims<LM>::ET;
  const double p = alpha + beta, inv2p = 0.5 / p;
  const double P = (alpha * a + beta * b) / p;
  const double xpa = P - a, xpb = P - b;
  const double mu = alpha * beta / p;
  for (int i = 0; i <= la; ++i)
    for (int j = 0; j <= lb; ++j)
      for (int t = 0; t < kET; ++t) E[i][j][t] = 0.0;
  E[0][0][0] = exp(-mu * (a - b) * (a - b));
  for (int i = 0; i <= la; ++i)
    for (int j = 0; j <= lb; ++j) {
      if (i == 0 && j == 0) continue;
      for (int t = 0; t <= i + j; ++t) {
        double v;
        if (i > 0) {
          v = xpa * E[i - 1][j][t];
          if (t > 0) v += inv2p * E[i - 1][j][t - 1];
          if (t + 1 <= i - 1 + j) v += (t + 1) * E[i - 1][j][t + 1];
        } else {
          v = xpb * E[i][j - 1][t];
          if (t > 0) v += inv2p * E[i][j - 1][t - 1];
          if (t + 1 <= i + j - 1) v += (t + 1) * E[i][j - 1][t + 1];
        }
        E[i][j][t] = v;
      }
    }
}

__device__ __forceinline__ double comp_norm(const int l[3]) {
  // 1/sqrt(prod (2 l_i - 1)!!)
  double d = 1.0;
  for (int k = 0; k < 3; ++k)
    for (int m = 2 * l[k] - 1; m > 1; m -= 2) d *= m;
  return rsqrt(d);
}

template <int LM>
__global__ void __launch_bounds__(128) oneint_kernel(const OneIntArgs a) {
  using Dm = OneIntDims<LM>;
  constexpr int kEI = Dm::EI, kEJ = Dm::EJ, kET = Dm::ET;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long npair = (long long)a.n * (a.n + 1) / 2;
  if (t >= npair) return;
  // t -> (mu, nu), mu >= nu
  int mu = (int)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
  while ((long long)mu * (mu + 1) / 2 > t) --mu;
  while ((long long)(mu + 1) * (mu + 2) / 2 <= t) ++mu;
  const int nu = (int)(t - (long long)mu * (mu + 1) / 2);
  const FuncInfo A = a.funcs[mu], B = a.funcs[nu];
  const double na = comp_norm(A.l), nb = comp_norm(B.l);
  const int pa = a.sh_off[A.shell], ka = a.sh_K[A.shell], pb = a.sh_off[B.shell], kb = a.sh_K[B.shell];
  double S = 0.0, Tk = 0.0;
  double Ex[kEI][kEJ][kET], Ey[kEI][kEJ][kET], Ez[kEI][kEJ][kET];
  for (int i = 0; i < ka; ++i)
    for (int j = 0; j < kb; ++j) {
      const double al = a.exps[pa + i], be = a.exps[pb + j];
      const double cc = a.coefs[pa + i] * a.coefs[pb + j] * na * nb;
      const double p = al + be, inv_p = 1.0 / p;
      hermite_1d<LM>(A.l[0], B.l[0] + 2, al, be, A.c[0], B.c[0], Ex);
      hermite_1d<LM>(A.l[1], B.l[1] + 2, al, be, A.c[1], B.c[1], Ey);
      hermite_1d<LM>(A.l[2], B.l[2] + 2, al, be, A.c[2], B.c[2], Ez);
      const double pref = 5.56832799683170784528 * inv_p * sqrt(inv_p);  // (pi/p)^{3/2}
      const double sx = Ex[A.l[0]][B.l[0]][0], sy = Ey[A.l[1]][B.l[1]][0], sz = Ez[A.l[2]][B.l[2]][0];
      S += cc * pref * sx * sy * sz;
      auto t1d = [&](int li, int lj, double E[kEI][kEJ][kET]) {
        double v = be * (2.0 * lj + 1.0) * E[li][lj][0] - 2.0 * be * be * E[li][lj + 2][0];
        if (lj >= 2) v -= 0.5 * lj * (lj - 1) * E[li][lj - 2][0];
        return v;
      };
      Tk += cc * pref * (t1d(A.l[0], B.l[0], Ex) * sy * sz + sx * t1d(A.l[1], B.l[1], Ey) * sz +
                         sx * sy * t1d(A.l[2], B.l[2], Ez));
    }
  a.S[(size_t)mu * a.n + nu] = a.S[(size_t)nu * a.n + mu] = S;
  a.T[(size_t)mu * a.n + nu] = a.T[(size_t)nu * a.n + mu] = Tk;
}

// Nuclear attraction V_ab = -sum_C Z_C (2 pi / p) sum_h E^{ab}_h R_h(p, P - C),
// one warp per shell pair.  E does not depend on the nucleus, so R is summed
// over the nuclei first: groups of nc lanes (the nuclei's, at least 4) take
// one primitive pair each, a lane walks its nuclei with R in registers, the
// group's sums meet by a butterfly and go to shared memory, and its lanes
// share the components.  (A thread per function pair, with a four-index R
// table in local memory per nucleus, took 1.5 ms for two waters in cc-pVDZ.)
// A small molecule's launches, 46 us each beside one another, wait for their
// blocks' Boys tables.
struct NucArgs {
  const PairInfo* pairs;  // of one (la, lb)
  int count;
  const PrimRec64* rec;
  const double* atoms;  // natom * 4: x, y, z, charge
  int natom, n;
  const double* boys;
  const double* expt;
  double* V;  // n x n
};

constexpr int kNucThreads = 64, kNucGroups = 8;

// index of (t, u, v) among the Hermite triples of degree <= l (nested order)
__host__ __device__ constexpr int nuc_index(int l, int t, int u, int v) {
  int k = 0;
  for (int i = 0; i < t; ++i) k += (l - i + 1) * (l - i + 2) / 2;
  for (int j = 0; j < u; ++j) k += l - t - j + 1;
  return k + v;
}

// R_tuv of degree <= L from F[m] = (-2p)^m f F_m, level by level in place
// (descending degree: a level's lower degrees are still the level before's).
template <int L>
__device__ __forceinline__ void nuc_r(const double* F, double x, double y, double z, double* R) {
  R[0] = F[L];
#pragma unroll
  for (int n = L - 1; n >= 0; --n) {
#pragma unroll
    for (int deg = L; deg >= 1; --deg)
#pragma unroll
      for (int t = 0; t <= L; ++t)
#pragma unroll
        for (int u = 0; u <= L; ++u) {
          const int v = deg - t - u;
          if (deg > L - n || v < 0) continue;
          double r;
          if (t > 0) {
            r = x * R[nuc_index(L, t - 1, u, v)];
            if (t > 1) r += (t - 1) * R[nuc_index(L, t > 1 ? t - 2 : 0, u, v)];
          } else if (u > 0) {
            r = y * R[nuc_index(L, t, u - 1, v)];
            if (u > 1) r += (u - 1) * R[nuc_index(L, t, u > 1 ? u - 2 : 0, v)];
          } else {
            r = z * R[nuc_index(L, t, u, v - 1)];
            if (v > 1) r += (v - 1) * R[nuc_index(L, t, u, v > 1 ? v - 2 : 0)];
          }
          R[nuc_index(L, t, u, v)] = r;
        }
    R[0] = F[n];
  }
}

template <int LA, int LB> struct NucDims {
  static constexpr int L = LA + LB, NH = (L + 1) * (L + 2) * (L + 3) / 6, NAB = ncart(LA) * ncart(LB);
  static constexpr int NE = 3 * (LA + 1) * (LB + 1) * (L + 1);       // E[ax][i][j][t]
  static constexpr int PER_WARP = kNucGroups * (NH + NE + NAB);      // doubles
  static constexpr size_t smem() { return boys_smem_bytes<double>() + (kNucThreads / 32) * PER_WARP * sizeof(double); }
};

template <int LA, int LB>
__global__ void __launch_bounds__(kNucThreads) nuc_kernel(const NucArgs a) {
  using D = NucDims<LA, LB>;
  constexpr int L = D::L, NH = D::NH, NB = ncart(LB), NAB = D::NAB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* sm = reinterpret_cast<double*>(smem_raw);
  double* ws = sm + boys_smem_bytes<double>() / sizeof(double) + (threadIdx.x >> 5) * D::PER_WARP;
  boys_stage<double, L>(sm, a.boys, a.expt);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  int nc = 4;
  while (nc < 32 && nc < a.natom) nc *= 2;
  const int sub = lane & (nc - 1), grp = lane / nc, groups = 32 / nc;
  double* Rs = ws + grp * NH;
  double* E = ws + kNucGroups * NH + grp * D::NE;
  double* Vg = ws + kNucGroups * (NH + D::NE);  // [group][NAB]
  auto eo = [](int ax, int i, int j, int t) { return ((ax * (LA + 1) + i) * (LB + 1) + j) * (L + 1) + t; };
  const int nw = gridDim.x * (kNucThreads / 32);
  for (int pi = blockIdx.x * (kNucThreads / 32) + (threadIdx.x >> 5); pi < a.count; pi += nw) {
    const PairInfo pr = a.pairs[pi];
    __syncwarp();
    for (int x = sub; x < NAB; x += nc) Vg[grp * NAB + x] = 0.0;
    for (int k0 = 0; k0 < pr.npp; k0 += groups) {
      const int k = k0 + grp;
      const bool on = k < pr.npp;
      const PrimRec64 r = a.rec[pr.rec_off + (size_t)(on ? k : 0) * pr.rec_stride];
      const double pa[3] = {-r.bp * pr.ABx, -r.bp * pr.ABy, -r.bp * pr.ABz};
      double acc[NH];
#pragma unroll
      for (int h = 0; h < NH; ++h) acc[h] = 0.0;
      for (int c = sub; c < a.natom && on; c += nc) {
        const double* at = a.atoms + 4 * c;
        const double x = pr.Ax + pa[0] - at[0], y = pr.Ay + pa[1] - at[1], z = pr.Az + pa[2] - at[2];
        double F[L + 1], R[NH];
        boys_eval<L>(r.p * (x * x + y * y + z * z), sm, F);
        double f = -2.0 * 3.14159265358979323846 * at[3] * r.kp;
#pragma unroll
        for (int m = 0; m <= L; ++m) {
          F[m] *= f;
          f *= -2.0 * r.p;
        }
        nuc_r<L>(F, x, y, z, R);
#pragma unroll
        for (int h = 0; h < NH; ++h) acc[h] += R[h];
      }
#pragma unroll
      for (int h = 0; h < NH; ++h) {
        for (int off = 1; off < nc; off <<= 1) acc[h] += __shfl_xor_sync(0xffffffffu, acc[h], off);
        if (sub == (h & (nc - 1))) Rs[h] = acc[h];
      }
      if (sub < 3) {
        // this axis's Hermite coefficients
        const double p = sub == 0 ? pa[0] : (sub == 1 ? pa[1] : pa[2]);
        const double q = p + (sub == 0 ? pr.ABx : (sub == 1 ? pr.ABy : pr.ABz)), i2p = 0.5 * r.inv_p;
        double e[LA + 1][LB + 1][L + 1];
#pragma unroll
        for (int i = 0; i <= LA; ++i)
#pragma unroll
          for (int j = 0; j <= LB; ++j)
#pragma unroll
            for (int t = 0; t <= L; ++t) {
              double v = 0.0;
              if (i + j == 0) {
                v = t == 0 ? 1.0 : 0.0;
              } else if (t <= i + j) {
                const int u = i > 0 ? i - 1 : 0, w = i > 0 ? j : j - 1;
                v = (i > 0 ? p : q) * e[u][w < 0 ? 0 : w][t];
                if (t > 0) v += i2p * e[u][w < 0 ? 0 : w][t > 0 ? t - 1 : 0];
                if (t < L) v += (t + 1) * e[u][w < 0 ? 0 : w][t < L ? t + 1 : t];
              }
              e[i][j][t] = v;
              E[eo(sub, i, j, t)] = v;
            }
      }
      __syncwarp();
      if (on)
        for (int x = sub; x < NAB; x += nc) {
          int ea[3], eb[3];
          coop::component(LA, x / NB, ea);
          coop::component(LB, x % NB, eb);
          double v = 0.0;
          for (int t = 0; t <= ea[0] + eb[0]; ++t)
            for (int u = 0; u <= ea[1] + eb[1]; ++u) {
              const double exy = E[eo(0, ea[0], eb[0], t)] * E[eo(1, ea[1], eb[1], u)];
              const double* rr = Rs + nuc_index(L, t, u, 0);
              for (int w = 0; w <= ea[2] + eb[2]; ++w) v = fma(exy * E[eo(2, ea[2], eb[2], w)], rr[w], v);
            }
          Vg[grp * NAB + x] += v;
        }
      __syncwarp();
    }
    for (int x = lane; x < NAB; x += 32) {
      const int i = x / NB, j = x % NB;
      if (pr.same && j > i) continue;
      int ea[3], eb[3];
      coop::component(LA, i, ea);
      coop::component(LB, j, eb);
      double v = 0.0;
      for (int g = 0; g < groups; ++g) v += Vg[g * NAB + x];
      v *= coop::comp_scale_of(ea) * coop::comp_scale_of(eb);
      const size_t mu = pr.ao_a + i, nu = pr.ao_b + j;
      a.V[mu * a.n + nu] = a.V[nu * a.n + mu] = v;
    }
  }
}

template <int LA, int LB>
static cudaError_t launch_nuc(const NucArgs& a, cudaStream_t st) {
  auto kern = nuc_kernel<LA, LB>;
  const size_t smem = NucDims<LA, LB>::smem();
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kNucThreads, smem);
  const int want = (a.count + kNucThreads / 32 - 1) / (kNucThreads / 32), fit = sms * (per_sm > 0 ? per_sm : 1);
  kern<<<(unsigned)(want < fit ? want : fit), kNucThreads, smem, st>>>(a);
  return cudaGetLastError();
}

static cudaError_t launch_nuc(int la, int lb, const NucArgs& a, cudaStream_t st) {
  if (a.count <= 0) return cudaSuccess;
#define HFG_CASE(A, B) \
  if (la == A && lb == B) return launch_nuc<A, B>(a, st);
  HFG_CASE(0, 0)
  HFG_CASE(1, 0)
  HFG_CASE(1, 1)
  HFG_CASE(2, 0)
  HFG_CASE(2, 1)
  HFG_CASE(2, 2)
  HFG_CASE(3, 0)
  HFG_CASE(3, 1)
  HFG_CASE(3, 2)
  HFG_CASE(3, 3)
#undef HFG_CASE
  return cudaErrorInvalidValue;
}

// Calls launch(la, lb, first pair, pairs, stream) for every (la, lb) of the
// pair table (its pair classes, by primitive counts, follow one another),
// over the context stream and its side streams, which are joined on every
// path.
template <typename F>
static cudaError_t for_pair_types(hfg_ctx* ctx, F&& launch) {
  cudaStream_t st = ctx->stream;
  cudaError_t e = ctx->ensure_side_streams();
  if (e == cudaSuccess) e = cudaEventRecord(ctx->ev_fork, st);
  if (e != cudaSuccess) return e;
  for (auto& x : ctx->side) cudaStreamWaitEvent(x, ctx->ev_fork, 0);
  int n = 0;
  for (size_t c = 0; c < ctx->classes.size() && e == cudaSuccess;) {
    const PairClass& k = ctx->classes[c];
    int count = 0;
    for (; c < ctx->classes.size() && ctx->classes[c].la == k.la && ctx->classes[c].lb == k.lb; ++c)
      count += ctx->classes[c].count;
    const int si = n++ % (1 + kJKSideStreams);
    e = launch(k.la, k.lb, ctx->d_pairs.p + k.first, count, si == 0 ? st : ctx->side[si - 1]);
  }
  for (int k = 0; k < kJKSideStreams; ++k) {
    cudaEventRecord(ctx->ev_join[k], ctx->side[k]);
    cudaStreamWaitEvent(st, ctx->ev_join[k], 0);
  }
  return e;
}

// One-electron part of the analytic nuclear gradient, as hf-rs's
// compute_gradient_from_density (src/gradient.rs:372-455):
//   d/dX [ sum P_ab (T_ab + V_ab) - sum W_ab S_ab ]
// over the basis centres, and the operator derivative of the nuclear
// attraction on each nucleus (by translational invariance).  One warp per
// shell pair (its functions' block of P and W in shared memory):
//
// * V: lanes over (primitive pair, nucleus).  The attraction by a point
//   charge is the (ab|00) Hermite sum with alpha = p and Q = C, so the
//   generated code of the ERI derivatives (GradClass<LA, LB, 0, 0>) gives its
//   value, d/dP (minus the force on the nucleus) and d/dR_AB.
// * S and T depend on A - B alone: lanes over primitive pairs, one-axis
//   overlaps raised by one in a and two in b.
//
// A thread per function pair with whole R tables in local memory took 1.8 ms
// for one water in cc-pVDZ.
struct OneGradArgs {
  const PairInfo* pairs;  // of one (la, lb)
  int count;
  const PrimRec64* rec;
  const double* atoms;  // natom * 4: x, y, z, charge
  const int* ao_atom;
  int natom, n;
  const double* boys;
  const double* expt;
  const double* P;  // total density
  const double* W;  // energy-weighted density
  double* grad;     // natom * 3
};

constexpr int kOneGradThreads = 128;

// power of axis ax in Cartesian component c of l <= 2 (hf-rs order)
__host__ __device__ constexpr int cart_power(int l, int c, int ax) {
  if (l == 0) return 0;
  if (l == 1) return c == ax ? 1 : 0;
  if (c < 3) return c == ax ? 2 : 0;
  return c == 3 ? (ax != 2 ? 1 : 0) : (c == 4 ? (ax != 1 ? 1 : 0) : (ax != 0 ? 1 : 0));
}

template <int LA, int LB>
__global__ void __launch_bounds__(kOneGradThreads) oneint_grad_kernel(const OneGradArgs a) {
  using C = GradClass<LA, LB, 0, 0>;
  constexpr int NA = ncart(LA), NB = ncart(LB), NAB = NA * NB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* sm = reinterpret_cast<double*>(smem_raw);
  double* gacc = sm + boys_smem_bytes<double>() / sizeof(double);  // natom * 3
  double* blk = gacc + 3 * a.natom + (threadIdx.x >> 5) * 2 * NAB;  // the pair's P block, then its W block
  boys_stage<double, C::L + 1>(sm, a.boys, a.expt);
  for (int x = threadIdx.x; x < 3 * a.natom; x += blockDim.x) gacc[x] = 0.0;
  __syncthreads();
  const int lane = threadIdx.x & 31, nw = gridDim.x * (kOneGradThreads / 32);
  int nc = 1;  // nuclei side by side in a warp; its other lanes split the primitive pairs
  while (nc < 32 && nc < a.natom) nc *= 2;
  const int sub = lane & (nc - 1), grp = lane / nc, groups = 32 / nc;
  for (int t = blockIdx.x * (kOneGradThreads / 32) + (threadIdx.x >> 5); t < a.count; t += nw) {
    const PairInfo pr = a.pairs[t];
    __syncwarp();
    for (int x = lane; x < NAB; x += 32) {
      const int i = x / NB, j = x % NB;
      // both orders of a pair of different shells
      const double w = (pr.same ? 0.5 : 1.0) * comp_scale(LA, i) * comp_scale(LB, j);
      const size_t ij = (size_t)(pr.ao_a + i) * a.n + pr.ao_b + j, ji = (size_t)(pr.ao_b + j) * a.n + pr.ao_a + i;
      blk[x] = w * (a.P[ij] + a.P[ji]);
      blk[NAB + x] = w * (a.W[ij] + a.W[ji]);
    }
    __syncwarp();
    const int atA = a.ao_atom[pr.ao_a], atB = a.ao_atom[pr.ao_b];
    const double AB[3] = {pr.ABx, pr.ABy, pr.ABz};
    double gA[3] = {0.0, 0.0, 0.0}, gB[3] = {0.0, 0.0, 0.0};
    for (int c0 = 0; c0 < a.natom; c0 += nc) {
      const bool on = c0 + sub < a.natom;
      const double* at = a.atoms + 4 * (on ? c0 + sub : c0);
      const double AC[3] = {pr.Ax - at[0], pr.Ay - at[1], pr.Az - at[2]}, Z = at[3];
      double gC[3] = {0.0, 0.0, 0.0};
      for (int k = grp; k < pr.npp && on; k += groups) {
        const PrimRec64 r = a.rec[pr.rec_off + (size_t)k * pr.rec_stride];
        if (fabs(r.kp) < 1e-28) continue;
        const double pa[3] = {-r.bp * AB[0], -r.bp * AB[1], -r.bp * AB[2]};
        const double PC[3] = {AC[0] + pa[0], AC[1] + pa[1], AC[2] + pa[2]};
        double F[C::L + 2];
        boys_eval<C::L + 1>(r.p * (PC[0] * PC[0] + PC[1] * PC[1] + PC[2] * PC[2]), sm, F);
        double f = -2.0 * 3.14159265358979323846 * Z * r.kp;
#pragma unroll
        for (int m = 0; m <= C::L + 1; ++m) {
          F[m] *= f;
          f *= -2.0 * r.p;
        }
        double ev, gp[3], gb[3], gk[3];
        C::prim(blk, 1, F, PC[0], PC[1], PC[2], pa[0], pa[1], pa[2], pa[0] + AB[0], pa[1] + AB[1], pa[2] + AB[2],
                0.5 * r.inv_p, -r.bp, 1.0 - r.bp, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, ev, gp, gb, gk);
        const double mb = -2.0 * r.bp * (1.0 - r.bp) * r.p * ev;
#pragma unroll
        for (int x = 0; x < 3; ++x) {
          const double ga = (1.0 - r.bp) * gp[x] + gb[x] + mb * AB[x];
          gA[x] += ga;
          gB[x] += gp[x] - ga;
          gC[x] -= gp[x];
        }
      }
#pragma unroll
      for (int x = 0; x < 3; ++x)
        for (int off = nc; off < 32; off <<= 1) gC[x] += __shfl_xor_sync(0xffffffffu, gC[x], off);
      if (grp == 0 && on)
        for (int x = 0; x < 3; ++x) atomicAdd(gacc + 3 * (c0 + sub) + x, gC[x]);
    }
    if (atA != atB) {
      // S and T: zero on one atom
      for (int k = lane; k < pr.npp; k += 32) {
        const PrimRec64 r = a.rec[pr.rec_off + (size_t)k * pr.rec_stride];
        const double al = (1.0 - r.bp) * r.p, be = r.bp * r.p, i2p = 0.5 * r.inv_p;
        const double pref = r.kp * 5.56832799683170784528 * rsqrt(r.p);  // (pi/p)^{3/2} p k
        double s[3][LA + 2][LB + 3];
#pragma unroll
        for (int x = 0; x < 3; ++x) {
          const double pa = -r.bp * AB[x], pb = pa + AB[x];
#pragma unroll
          for (int i = 0; i <= LA + 1; ++i)
#pragma unroll
            for (int j = 0; j <= LB + 2; ++j) {
              double v = 1.0;
              if (j > 0) {
                v = pb * s[x][i][j - 1];
                if (i > 0) v += i2p * i * s[x][i - 1][j - 1];
                if (j > 1) v += i2p * (j - 1) * s[x][i][j - 2];
              } else if (i > 0) {
                v = pa * s[x][i - 1][0];
                if (i > 1) v += i2p * (i - 1) * s[x][i - 2][0];
              }
              s[x][i][j] = v;
            }
        }
        auto kin = [&](int x, int i, int j) {
          double v = be * (2.0 * j + 1.0) * s[x][i][j] - 2.0 * be * be * s[x][i][j + 2];
          if (j >= 2) v -= 0.5 * j * (j - 1) * s[x][i][j - 2];
          return v;
        };
#pragma unroll
        for (int ci = 0; ci < NA; ++ci)
#pragma unroll
          for (int cj = 0; cj < NB; ++cj) {
            const double Pv = pref * blk[ci * NB + cj], Wv = pref * blk[NAB + ci * NB + cj];
            double sv[3], kv[3], ds[3], dk[3];
#pragma unroll
            for (int x = 0; x < 3; ++x) {
              const int i = cart_power(LA, ci, x), j = cart_power(LB, cj, x);
              sv[x] = s[x][i][j];
              kv[x] = kin(x, i, j);
              // d/dA raises with 2 alpha and lowers with the power
              ds[x] = 2.0 * al * s[x][i + 1][j] - (i > 0 ? i * s[x][i > 0 ? i - 1 : 0][j] : 0.0);
              dk[x] = 2.0 * al * kin(x, i + 1, j) - (i > 0 ? i * kin(x, i > 0 ? i - 1 : 0, j) : 0.0);
            }
#pragma unroll
            for (int x = 0; x < 3; ++x) {
              const int y = (x + 1) % 3, z = (x + 2) % 3;
              const double dT = dk[x] * sv[y] * sv[z] + ds[x] * (kv[y] * sv[z] + sv[y] * kv[z]);
              const double g = Pv * dT - Wv * ds[x] * sv[y] * sv[z];
              gA[x] += g;
              gB[x] -= g;
            }
          }
      }
    }
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      for (int off = 16; off > 0; off >>= 1) {
        gA[x] += __shfl_xor_sync(0xffffffffu, gA[x], off);
        gB[x] += __shfl_xor_sync(0xffffffffu, gB[x], off);
      }
      if (lane == 0) {
        atomicAdd(gacc + 3 * atA + x, gA[x]);
        atomicAdd(gacc + 3 * atB + x, gB[x]);
      }
    }
  }
  __syncthreads();
  for (int x = threadIdx.x; x < 3 * a.natom; x += blockDim.x)
    if (gacc[x] != 0.0) atomicAdd(a.grad + x, gacc[x]);
}

template <int LA, int LB>
static cudaError_t launch_oneint_grad(const OneGradArgs& a, cudaStream_t st) {
  if (a.count <= 0) return cudaSuccess;
  auto kern = oneint_grad_kernel<LA, LB>;
  const size_t smem = boys_smem_bytes<double>() +
                      (3 * (size_t)a.natom + 2 * ncart(LA) * ncart(LB) * (kOneGradThreads / 32)) * sizeof(double);
  const cudaError_t e = raise_smem_limit<oneint_grad_kernel<LA, LB>>();
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kOneGradThreads, smem);
  const int want = (a.count + kOneGradThreads / 32 - 1) / (kOneGradThreads / 32), fit = sms * (per_sm > 0 ? per_sm : 1);
  kern<<<(unsigned)(want < fit ? want : fit), kOneGradThreads, smem, st>>>(a);
  return cudaGetLastError();
}

// S, T, V (device, row-major n x n) of the context basis for the given nuclei.
int one_electron(hfg_ctx* ctx, int natom, const double* pos, const double* charge, double* dS, double* dT,
                 double* dV) {
  const int n = ctx->n;
  std::vector<FuncInfo> f(n);
  std::vector<int> off, K;
  for (size_t s = 0; s < ctx->shells.size(); ++s) {
    const Shell& sh = ctx->shells[s];
    off.push_back(sh.prim_off);
    K.push_back(sh.K);
    const int cnt = (sh.l + 1) * (sh.l + 2) / 2;
    int c = 0;
    // hf-rs component order (src/basis.rs:418-445)
    static const int d_order[6][3] = {{2, 0, 0}, {0, 2, 0}, {0, 0, 2}, {1, 1, 0}, {1, 0, 1}, {0, 1, 1}};
    for (int lx = sh.l; lx >= 0 && c < cnt; --lx)
      for (int ly = sh.l - lx; ly >= 0 && c < cnt; --ly) {
        FuncInfo& fi = f[sh.ao + c];
        for (int k = 0; k < 3; ++k) fi.c[k] = sh.c[k];
        if (sh.l == 2) {
          fi.l[0] = d_order[c][0];
          fi.l[1] = d_order[c][1];
          fi.l[2] = d_order[c][2];
        } else {
          fi.l[0] = lx;
          fi.l[1] = ly;
          fi.l[2] = sh.l - lx - ly;
        }
        fi.shell = (int)s;
        ++c;
      }
  }
  std::vector<double> at(4 * natom);
  for (int i = 0; i < natom; ++i) {
    for (int k = 0; k < 3; ++k) at[4 * i + k] = pos[3 * i + k];
    at[4 * i + 3] = charge[i];
  }
  DevBuf<FuncInfo> df;
  DevBuf<double> dex, dco, dat;
  DevBuf<int> doff, dK;
  int rc = HFG_OK;
  auto chk = [&](cudaError_t e, const char* w) {
    if (rc == HFG_OK) rc = cuda_check(ctx, e, w);
  };
  chk(df.alloc(n), "alloc");
  chk(dex.alloc(ctx->exps.size()), "alloc");
  chk(dco.alloc(ctx->coefs.size()), "alloc");
  chk(dat.alloc(at.size() + 1), "alloc");
  chk(doff.alloc(off.size()), "alloc");
  chk(dK.alloc(K.size()), "alloc");
  if (rc != HFG_OK) return rc;
  chk(cudaMemcpyAsync(df.p, f.data(), n * sizeof(FuncInfo), cudaMemcpyHostToDevice, ctx->stream), "copy");
  chk(cudaMemcpyAsync(dex.p, ctx->exps.data(), ctx->exps.size() * 8, cudaMemcpyHostToDevice, ctx->stream), "copy");
  chk(cudaMemcpyAsync(dco.p, ctx->coefs.data(), ctx->coefs.size() * 8, cudaMemcpyHostToDevice, ctx->stream), "copy");
  chk(cudaMemcpyAsync(dat.p, at.data(), at.size() * 8, cudaMemcpyHostToDevice, ctx->stream), "copy");
  chk(cudaMemcpyAsync(doff.p, off.data(), off.size() * 4, cudaMemcpyHostToDevice, ctx->stream), "copy");
  chk(cudaMemcpyAsync(dK.p, K.data(), K.size() * 4, cudaMemcpyHostToDevice, ctx->stream), "copy");
  OneIntArgs a{df.p, dex.p, dco.p, doff.p, dK.p, n, dS, dT};
  const long long npair = (long long)n * (n + 1) / 2;
  auto kern = ctx->lmax <= 2 ? oneint_kernel<2> : oneint_kernel<3>;
  if (npair > 0) kern<<<(unsigned)((npair + 127) / 128), 128, 0, ctx->stream>>>(a);
  chk(cudaGetLastError(), "oneint kernel");
  chk(for_pair_types(ctx,
                     [&](int la, int lb, const PairInfo* pairs, int count, cudaStream_t st) {
                       return launch_nuc(la, lb, NucArgs{pairs, count, ctx->d_rec64.p, dat.p, natom, n, ctx->d_boys64.p,
                                                         ctx->d_expt64.p, dV}, st);
                     }),
      "nuclear attraction kernel");
  chk(cudaStreamSynchronize(ctx->stream), "oneint sync");
  return rc;
}

// One-electron gradient terms (device) for nuclei (positions, charges),
// added into grad (host, natom * 3).
int one_electron_gradient(hfg_ctx* ctx, int natom, const double* pos, const double* charge, const double* P,
                          const double* W, double* grad) {
  const int n = ctx->n;
  std::vector<int> fatom(n);
  for (const Shell& sh : ctx->shells)
    for (int k = 0; k < (sh.l + 1) * (sh.l + 2) / 2; ++k) fatom[sh.ao + k] = sh.atom;
  std::vector<double> at(4 * natom);
  for (int i = 0; i < natom; ++i) {
    for (int k = 0; k < 3; ++k) at[4 * i + k] = pos[3 * i + k];
    at[4 * i + 3] = charge[i];
  }
  const size_t nn = (size_t)n * n;
  DevBuf<double> dat, dP, dW, dg;
  DevBuf<int> dfa;
  int rc = HFG_OK;
  auto chk = [&](cudaError_t e, const char* w) {
    if (rc == HFG_OK) rc = cuda_check(ctx, e, w);
  };
  chk(dat.alloc(at.size()), "alloc");
  chk(dP.alloc(nn), "alloc");
  chk(dW.alloc(nn), "alloc");
  chk(dg.alloc(3 * (size_t)natom), "alloc");
  chk(dfa.alloc(n), "alloc");
  if (rc != HFG_OK) return rc;
  cudaStream_t st = ctx->stream;
  chk(cudaMemcpyAsync(dat.p, at.data(), at.size() * 8, cudaMemcpyHostToDevice, st), "copy");
  chk(cudaMemcpyAsync(dP.p, P, nn * 8, cudaMemcpyHostToDevice, st), "copy");
  chk(cudaMemcpyAsync(dW.p, W, nn * 8, cudaMemcpyHostToDevice, st), "copy");
  chk(cudaMemcpyAsync(dfa.p, fatom.data(), n * 4, cudaMemcpyHostToDevice, st), "copy");
  chk(cudaMemsetAsync(dg.p, 0, 3 * (size_t)natom * 8, st), "memset");
  if (rc != HFG_OK) return rc;
  chk(for_pair_types(ctx,
                     [&](int la, int lb, const PairInfo* pairs, int count, cudaStream_t ls) {
                       const OneGradArgs a{pairs, count, ctx->d_rec64.p, dat.p, dfa.p, natom, n, ctx->d_boys64.p,
                                           ctx->d_expt64.p, dP.p, dW.p, dg.p};
                       if (la == 0) return launch_oneint_grad<0, 0>(a, ls);
                       if (la == 1) return lb == 0 ? launch_oneint_grad<1, 0>(a, ls) : launch_oneint_grad<1, 1>(a, ls);
                       if (la == 2 && lb == 0) return launch_oneint_grad<2, 0>(a, ls);
                       if (la == 2 && lb == 1) return launch_oneint_grad<2, 1>(a, ls);
                       return la == 2 ? launch_oneint_grad<2, 2>(a, ls) : cudaErrorInvalidValue;
                     }),
      "one-electron gradient kernel");
  std::vector<double> g(3 * (size_t)natom);
  chk(cudaMemcpyAsync(g.data(), dg.p, g.size() * 8, cudaMemcpyDeviceToHost, st), "copy");
  chk(cudaStreamSynchronize(st), "sync");
  if (rc == HFG_OK)
    for (size_t x = 0; x < g.size(); ++x) grad[x] += g[x];
  return rc;
}

}  // namespace hfg
