// Packed 8-fold ERI tensor on the device: the counterpart of hf-rs's
// compute_eri_tensor (src/scf.rs:275-333 -> compute_shell_eri_tensor,
// src/shell_integrals.rs:156-240) for small systems and for consumers that
// want stored integrals (post-HF transforms).
//
// Layout (src/scf.rs:222-235): slot eri_index(mu,nu,lam,sig) =
// c(c(mu,nu), c(lam,sig)) with c(i,j) = max(i,j)(max(i,j)+1)/2 + min(i,j),
// holding the Cartesian (mu nu|lam sig) with the per-component scale of
// src/basis.rs:123-132.  Shell quartets with Q_ab Q_cd <= threshold stay
// zero, as in the reference.  The quartets are those of the FP64 J/K plan
// (every unique Schwarz-significant shell quartet once, unsliced), all
// primitive quartets evaluated (no primitive screening).  Every slot has one
// writer: within a same-shell pair only the i >= j components are written,
// and a quartet of a pair with itself writes only IJ >= KL.
//
// A quartet takes a power-of-two group of lanes, at least 4 primitive
// quartets each: the lanes' accumulators are added by a butterfly, whose
// order is fixed and the same for every quartet of a class, so equivalent
// quartets of a symmetric molecule keep bitwise equal integrals (the pivot
// rule of the Cholesky factor depends on it).  Blocks are persistent and
// stage the Boys table once; a block per 128 quartets staged 52 KB for each,
// and one lane walked the 4,096 primitive quartets of a contracted (ss|ss).
#include "jk_dispatch.h"
#include "eri_prim.cuh"
#include "md_coop.cuh"

namespace hfg {

__device__ __forceinline__ unsigned long long compound(unsigned long long i, unsigned long long j) {
  return i >= j ? i * (i + 1) / 2 + j : j * (j + 1) / 2 + i;
}

template <int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(128) eri_packed_kernel(const JKEntry* __restrict__ entries,
                                                         const long long* __restrict__ prefix, int nentries,
                                                         long long nwarps, const PairInfo* __restrict__ pairs,
                                                         const double* __restrict__ pairQ, double thr,
                                                         const PrimRec64* __restrict__ rec,
                                                         const double* __restrict__ boys,
                                                         const double* __restrict__ expt, double* __restrict__ out) {
  using C = EriClass<LA, LB, LC, LD>;
  constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* sm = reinterpret_cast<double*>(smem_raw);
  boys_stage<double, C::L>(sm, boys, expt);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const long long units = nwarps * 32, nw = (long long)gridDim.x * (blockDim.x >> 5);
  // units: lane group `sub` of warp task u / 32, in runs of `per`
  int per = 1;
  while (per < 32 && units > 16LL * per * nw) per *= 2;
  int e = 0;
  for (long long u0 = ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * per; u0 < units; u0 += nw * per) {
    const long long warp = u0 >> 5;
    e = coop::entry_of(prefix, nentries, warp, e);
    const JKEntry ent = entries[e];
    const PairInfo bra = pairs[ent.bra];
    const int nb = bra.npp, nk = pairs[ent.k_lo].npp;  // one pair class: equal counts
    int gs = 1;
    while (gs < 32 && 8 * gs <= nb * nk) gs *= 2;
    const int ng = 32 / gs, slot = lane / gs, mem = lane - slot * gs;
    const int sub0 = (int)(u0 & 31), sub1 = min(sub0 + per, gs);
    for (int sub = sub0; sub < sub1; ++sub) {
      const int kidx = ent.k_lo + (int)(warp - prefix[e]) * 32 + sub * ng + slot;
      const bool active = kidx < ent.k_hi && pairQ[min(kidx, ent.k_hi - 1)] * pairQ[ent.bra] > thr;
      if (__ballot_sync(0xffffffffu, active) == 0u) continue;
      const PairInfo ket = pairs[active ? kidx : ent.k_lo];
      const double ACx = bra.Ax - ket.Ax, ACy = bra.Ay - ket.Ay, ACz = bra.Az - ket.Az;
      double acc[C::NACC];
#pragma unroll
      for (int x = 0; x < C::NACC; ++x) acc[x] = 0.0;
      const int np = active ? nb * nk : 0;
      int ik = mem / nb, ib = mem - ik * nb;
      for (int x = mem; x < np; x += gs) {
        const PrimRec64 Q = rec[ket.rec_off + (size_t)ik * ket.rec_stride];
        const PrimRec64 P = rec[bra.rec_off + (size_t)ib * bra.rec_stride];
        ib += gs;
        while (ib >= nb) {
          ib -= nb;
          ++ik;
        }
        prim_quartet<LA, LB, LC, LD, double>(acc, P.p, P.inv_p, P.kp, -P.bp * bra.ABx, -P.bp * bra.ABy,
                                             -P.bp * bra.ABz, Q.p, Q.inv_p, Q.kp, -Q.bp * ket.ABx, -Q.bp * ket.ABy,
                                             -Q.bp * ket.ABz, ACx, ACy, ACz, sm);
      }
      for (int off = 1; off < gs; off <<= 1) {
#pragma unroll
        for (int x = 0; x < C::NACC; ++x) acc[x] += __shfl_xor_sync(0xffffffffu, acc[x], off);
      }
      if (!active) continue;
      double blk[C::NOUT];
      C::hrr(acc, blk, bra.ABx, bra.ABy, bra.ABz, ket.ABx, ket.ABy, ket.ABz);
      const bool self = kidx == ent.bra;
#pragma unroll
      for (int i = 0; i < NA; ++i)
#pragma unroll
        for (int j = 0; j < NB; ++j) {
          const int mu = bra.ao_a + i, nu = bra.ao_b + j;
          if (bra.same && mu < nu) continue;
          const unsigned long long IJ = compound(mu, nu);
#pragma unroll
          for (int k = 0; k < NC; ++k)
#pragma unroll
            for (int l = 0; l < ND; ++l) {
              const int x = ((i * NB + j) * NC + k) * ND + l;
              const int lam = ket.ao_a + k, sig = ket.ao_b + l;
              // the group's lanes share the stores
              if ((x & (gs - 1)) != mem || (ket.same && lam < sig)) continue;
              const unsigned long long KL = compound(lam, sig);
              if (self && IJ < KL) continue;
              out[compound(IJ, KL)] =
                  blk[x] * (comp_scale(LA, i) * comp_scale(LB, j) * comp_scale(LC, k) * comp_scale(LD, l));
            }
        }
    }
  }
}

template <int LA, int LB, int LC, int LD>
static cudaError_t launch_packed_class(const JKEntry* entries, const long long* prefix, int nentries, long long nwarps,
                                       const PairInfo* pairs, const double* pairQ, double thr, const PrimRec64* rec,
                                       const double* boys, const double* expt, double* out, cudaStream_t st) {
  auto kern = eri_packed_kernel<LA, LB, LC, LD>;
  const int smem = (int)boys_smem_bytes<double>(), block = 128;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, block, smem);
  // a task has at most 32 units of one warp each
  const long long want = nwarps * 32 / (block / 32), fit = (long long)sms * (per_sm > 0 ? per_sm : 1);
  kern<<<(unsigned)(want < fit ? want : fit), block, smem, st>>>(entries, prefix, nentries, nwarps, pairs, pairQ, thr, rec,
                                                                 boys, expt, out);
  return cudaGetLastError();
}

cudaError_t launch_eri_packed(int la, int lb, int lc, int ld, const JKEntry* entries, const long long* prefix,
                              int nentries, long long nwarps, const PairInfo* pairs, const double* pairQ,
                              double thr, const PrimRec64* rec,
                              const double* boys, const double* expt, double* out, cudaStream_t st) {
  if (nwarps <= 0) return cudaSuccess;
#define HFG_CASE(A, B, C, D)                                                                                       \
  if (la == A && lb == B && lc == C && ld == D)                                                                     \
    return launch_packed_class<A, B, C, D>(entries, prefix, nentries, nwarps, pairs, pairQ, thr, rec, boys, expt, out, st);
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
  HFG_CASE(2, 1, 1, 0)
  HFG_CASE(2, 1, 1, 1)
  HFG_CASE(2, 1, 2, 0)
  HFG_CASE(2, 1, 2, 1)
  HFG_CASE(2, 2, 0, 0)
  HFG_CASE(2, 2, 1, 0)
  HFG_CASE(2, 2, 1, 1)
  HFG_CASE(2, 2, 2, 0)
  HFG_CASE(2, 2, 2, 1)
  HFG_CASE(2, 2, 2, 2)
#undef HFG_CASE
  return cudaErrorInvalidValue;
}

}  // namespace hfg
