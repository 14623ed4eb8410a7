// Pivoted Cholesky decomposition of the AO ERI supermatrix on the device.
//
// Stands in for hf-rs's pivoted_cholesky_eri (src/cholesky.rs:42-190):
// (pq|rs) ~ sum_K L_K(pq) L_K(rs), the pivot at each step being the largest
// residual diagonal (diagonals within 1e-12 relative of it are ties, taken
// by the smallest packed pair index), until the largest residual is at or
// below the threshold.  The vectors are returned as an hfg_df factor over
// every packed AO pair (compound_index order), so hfg_df_jk and hfg_scf_df
// run Cholesky-factorised RHF (run_cd_hf, src/hf_variants/cholesky_df.rs).
//
// Layout of the work: the ERI supermatrix V[pq][rs] is held on the device
// (packed 8-fold, from the J/K engine's integrals for quartets with
// Q_ab Q_cd > 1e-15, the column filter hf-rs uses), which bounds the
// system size to n_p (n_p + 1) / 2 doubles of device memory; hf-rs instead
// evaluates the pivots' columns on the fly.  All steps run in one kernel
// (chol_kernel): each block keeps a range of columns, and a step is one
// barrier over the grid.
#include <cublas_v2.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "df_handle.h"

using namespace hfg;

namespace {

__device__ __forceinline__ unsigned long long packed(unsigned long long i, unsigned long long j) {
  return i >= j ? i * (i + 1) / 2 + j : j * (j + 1) / 2 + i;
}

__global__ void chol_diag_kernel(const double* __restrict__ V, long long np, double* __restrict__ d) {
  for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < np; k += (long long)gridDim.x * blockDim.x)
    d[k] = V[packed(k, k)];
}

// The decomposition itself: one cooperative launch, each block owning the
// columns [b per, (b + 1) per).  A step:
//
//   1. the block's largest residual diagonal goes to bmax; grid barrier;
//   2. every block finds the largest M of all, and the pivot: the first
//      column with d >= M - 1e-12 |M|, which lies in the first block range
//      whose own maximum reaches that bound (hf-rs's tie rule);
//   3. for its own columns, row = (V[:, pivot] - sum_K L_K L_K[pivot]) / root
//      and diag -= row^2, with the check and clamp of src/cholesky.rs:172-178.
//
// A step costs the barrier and the pass over the vectors so far (8 rank n_p
// bytes, from L2); the earlier form, three launches, a copy of the diagonal
// and a host scan per pivot, took 52 us per pivot at n_p = 2,850 (the whole
// call 43 ms, now 5.1, with the packed tensor's kernels).
// The vectors' sum runs over 8 interleaved parts (one per warp) added in a
// fixed order, the same for every column, so equivalent pairs of a symmetric
// molecule keep equal residuals.
constexpr int kCholThreads = 256, kCholCols = 32, kCholPiv = 4096;
constexpr unsigned long long kCholWaitNs = 2000000000ull;

struct CholState {
  unsigned arrived;     // blocks that have reached the barrier, over all steps
  int bad[2];           // a residual diagonal fell below -1e-10 scale (by the step that reads it: a block may
                        // be one step ahead of another) or no pivot was found
  int status;           // 0 running, 1 done, 2 budget, 3 a bounded wait ran out
  long long rank;
  double residual;
};

struct CholArgs {
  const double* V;
  double* L;        // [cap][np]
  double* diag;     // [2][np], step r reads half r & 1 and writes the other
  double* bmax;     // [2][blocks], likewise
  CholState* st;
  long long* piv;   // [cap]
  long long np, cap, per;
  double threshold, scale, budget;
};

__device__ __forceinline__ unsigned long long chol_clock() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Barrier over the grid (all blocks resident): false when it gave up, after
// 2 s or because another block did.
__device__ __forceinline__ bool chol_barrier(CholState* st, unsigned target, int* ok) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&st->arrived, 1u);
    unsigned long long t0 = 0;
    int good = 1;
    for (unsigned i = 1; *(volatile unsigned*)&st->arrived < target; ++i) {
      if ((i & 255u) != 0) continue;  // (a read of the clock costs more than most waits)
      const unsigned long long now = chol_clock();
      if (t0 == 0) t0 = now;
      if (*(volatile int*)&st->status == 3 || now - t0 > kCholWaitNs) {
        atomicExch(&st->status, 3);
        good = 0;
        break;
      }
    }
    __threadfence();
    *ok = good;
  }
  __syncthreads();
  return *ok != 0;
}

__device__ __forceinline__ double block_max(double v, double* red) {
  for (int off = 16; off > 0; off >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, off));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  v = red[0];
  for (int k = 1; k < kCholThreads / 32; ++k) v = fmax(v, red[k]);
  return v;
}
__device__ __forceinline__ long long block_min(long long v, long long* red) {
  for (int off = 16; off > 0; off >>= 1) {
    const long long o = __shfl_xor_sync(0xffffffffu, v, off);
    v = o < v ? o : v;
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  v = red[0];
  for (int k = 1; k < kCholThreads / 32; ++k) v = red[k] < v ? red[k] : v;
  return v;
}

__global__ void __launch_bounds__(kCholThreads) chol_kernel(const CholArgs a) {
  __shared__ double redd[kCholThreads / 32];
  __shared__ long long redl[kCholThreads / 32];
  __shared__ double part[kCholThreads / 32][kCholCols];
  __shared__ double lp[kCholPiv];
  __shared__ int ok;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, G = gridDim.x;
  const long long none = 0x7fffffffffffffffLL;
  const long long c0 = blockIdx.x * a.per, c1 = min(a.np, c0 + a.per);
  unsigned target = 0;
  for (long long rank = 0;; ++rank) {
    const double* diag = a.diag + (rank & 1) * a.np;
    double* next = a.diag + ((rank + 1) & 1) * a.np;
    double m = -INFINITY;
    for (long long k = c0 + tid; k < c1; k += kCholThreads) m = fmax(m, __ldcg(diag + k));
    m = block_max(m, redd);
    double* bm = a.bmax + (rank & 1) * G;
    if (tid == 0) __stcg(bm + blockIdx.x, m);
    target += G;
    if (!chol_barrier(a.st, target, &ok)) return;
    if (*(volatile int*)&a.st->bad[rank & 1]) {
      if (blockIdx.x == 0 && tid == 0) a.st->rank = rank;
      return;
    }
    m = -INFINITY;
    for (int b = tid; b < G; b += kCholThreads) m = fmax(m, __ldcg(bm + b));
    const double largest = block_max(m, redd), bound = largest - 1e-12 * fabs(largest);
    long long first = none;
    for (int b = tid; b < G; b += kCholThreads)
      if (__ldcg(bm + b) >= bound && b < first) first = b;
    const long long owner = block_min(first, redl);
    if (owner == none) {  // an infinite diagonal: nothing compares with its bound
      if (blockIdx.x == 0 && tid == 0) a.st->bad[0] = 1;
      return;
    }
    first = none;
    const long long o1 = min(a.np, (owner + 1) * a.per);
    for (long long k = owner * a.per + tid; k < o1; k += kCholThreads)
      if (__ldcg(diag + k) >= bound) {
        first = k;
        break;
      }
    const long long pivot = block_min(first, redl);
    if (pivot == none) {  // no finite diagonal is left
      if (blockIdx.x == 0 && tid == 0) a.st->bad[0] = 1;
      return;
    }
    const double maximum = __ldcg(diag + pivot);
    const bool done = maximum <= a.threshold || rank == a.np;
    if (done || 8.0 * (double)a.np * (double)(rank + 2) > a.budget || rank >= a.cap) {
      if (blockIdx.x == 0 && tid == 0) {
        a.st->rank = rank;
        a.st->residual = fmax(maximum, 0.0);
        a.st->status = done ? 1 : 2;
      }
      return;
    }
    if (blockIdx.x == 0 && tid == 0) a.piv[rank] = pivot;
    const double root = sqrt(maximum);
    for (long long k = tid; k < rank && k < kCholPiv; k += kCholThreads) lp[k] = __ldcg(a.L + k * a.np + pivot);
    __syncthreads();
    double* row = a.L + rank * a.np;
    for (long long t = c0; t < c1; t += kCholCols) {
      const long long k = t + lane;
      double s = 0.0;
      if (k < c1) {
        const double* l = a.L + k;
        const long long r1 = rank < kCholPiv ? rank : kCholPiv;
        long long K = warp;
#pragma unroll 4
        for (; K < r1; K += kCholThreads / 32) s = fma(lp[K], l[K * a.np], s);
        for (; K < rank; K += kCholThreads / 32) s = fma(__ldcg(a.L + K * a.np + pivot), l[K * a.np], s);
      }
      part[warp][lane] = s;
      __syncthreads();
      if (warp == 0 && k < c1) {
        double v = a.V[packed(k, pivot)];
        for (int w = 0; w < kCholThreads / 32; ++w) v -= part[w][lane];
        const double r = k == pivot ? root : v / root;
        __stcg(row + k, r);
        const double d = __ldcg(diag + k) - r * r;
        if (d < -1e-10 * a.scale) a.st->bad[(rank + 1) & 1] = 1;
        __stcg(next + k, fmax(d, 0.0));
      }
      __syncthreads();
    }
  }
}

}  // namespace

extern "C" int hfg_cholesky_eri(hfg_ctx* ctx, double threshold, size_t budget, hfg_df** out, double* max_residual,
                                long long* pivots, int max_pivots, int* n_pivots) {
  if (!ctx) return HFG_ERR_INVALID_INPUT;
  if (!out) return set_error(ctx, HFG_ERR_INVALID_INPUT, "null pointer");
  *out = nullptr;
  if (!(threshold >= 0.0) || !std::isfinite(threshold))
    return set_error(ctx, HFG_ERR_INVALID_INPUT, "Cholesky requires a basis and a finite, nonnegative threshold");
  std::lock_guard<std::mutex> lk(ctx->mu);
  cudaSetDevice(ctx->device);
  AllocScope alloc_scope(ctx->stream);
  cudaStream_t st = ctx->stream;
  const long long n = ctx->n, np = n * (n + 1) / 2;
  const size_t vlen = (size_t)np * (np + 1) / 2;
  int rc = HFG_OK;
#define CK(call)                         \
  do {                                   \
    rc = cuda_check(ctx, (call), #call); \
    if (rc != HFG_OK) return rc;         \
  } while (0)
  DevBuf<double> V, diag;
  if (V.alloc(vlen) != cudaSuccess) {
    cudaGetLastError();
    return set_error(ctx, HFG_ERR_OOM, "pivoted Cholesky ERI decomposition: the ERI supermatrix does not fit");
  }
  CK(diag.alloc(2 * (size_t)np));
  rc = eri_packed_locked(ctx, 1e-15, V.p, vlen);
  if (rc != HFG_OK) return rc;
  const unsigned g = (unsigned)std::min<long long>((np + 255) / 256, 4096);
  chol_diag_kernel<<<g, 256, 0, st>>>(V.p, np, diag.p);
  CK(cudaGetLastError());
  std::vector<double> d(np);
  CK(cudaMemcpyAsync(d.data(), diag.p, np * 8, cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  double scale = 1.0;
  for (double x : d) scale = std::max(scale, x);
  for (double x : d)
    if (x < -1e-12 * scale)
      return set_error(ctx, HFG_ERR_INTEGRAL,
                       "pivoted Cholesky ERI decomposition: negative ERI diagonal; the Coulomb metric is not positive "
                       "semidefinite");
  // the vectors, row-major [rank][np]; capacity bounded by the budget
  const long long cap = std::max<long long>(1, std::min<long long>(np, (long long)(budget / (8 * (size_t)np))));
  auto df = std::make_unique<hfg_df>();
  df->ctx = ctx;
  df->n = (int)n;
  df->storage = HFG_DF_FP64;
  CK(df->B64.alloc((size_t)cap * np));
  std::vector<long long> piv;
  long long rank = 0;
  double maxres = 0.0;
  {
    DevBuf<double> bmax;
    DevBuf<CholState> state;
    DevBuf<long long> dpiv;
    int sms = 148, per_sm = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, chol_kernel, kCholThreads, 0));
    // whole tiles of columns per block, as few as blocks on every SM can
    // share, and no block without columns (n_p = 5,050: 79 blocks of two
    // tiles; every block joins the barrier of each step)
    const long long most = per_sm > 0 ? sms : 1;
    long long per = (np + most - 1) / most;
    per = (per + kCholCols - 1) / kCholCols * kCholCols;
    const int blocks = (int)((np + per - 1) / per);
    CK(bmax.alloc(2 * (size_t)blocks));
    CK(state.alloc(1));
    CK(dpiv.alloc((size_t)cap));
    CK(cudaMemsetAsync(state.p, 0, sizeof(CholState), st));
    CholArgs a{V.p, df->B64.p, diag.p, bmax.p, state.p, dpiv.p, np, cap, per, threshold, scale, (double)budget};
    void* args[] = {&a};
    CK(cudaLaunchCooperativeKernel((const void*)chol_kernel, dim3((unsigned)blocks), dim3(kCholThreads), args, 0, st));
    CholState h{};
    CK(cudaMemcpyAsync(&h, state.p, sizeof(h), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    if (h.status == 3)
      return set_error(ctx, HFG_ERR_TIMEOUT, "pivoted Cholesky ERI decomposition: a bounded wait ran out");
    if (h.status == 2)
      return set_error(ctx, HFG_ERR_INTEGRAL, "pivoted Cholesky ERI decomposition: factor storage exceeds the memory budget");
    if (h.bad[0] || h.bad[1])
      return set_error(ctx, HFG_ERR_INTEGRAL, "pivoted Cholesky ERI decomposition: nonpositive residual Coulomb diagonal");
    rank = h.rank;
    maxres = h.residual;
    piv.resize((size_t)rank);
    if (rank > 0) CK(cudaMemcpyAsync(piv.data(), dpiv.p, (size_t)rank * 8, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
  }
  if (rank == 0)
    return set_error(ctx, HFG_ERR_INTEGRAL,
                     "pivoted Cholesky ERI decomposition: threshold exceeds every ERI diagonal; no Cholesky vectors were "
                     "generated");
  // the factor over every packed AO pair, compound_index order
  std::vector<int2> colmn((size_t)np);
  for (long long p = 0; p < n; ++p)
    for (long long q = 0; q <= p; ++q) colmn[(size_t)(p * (p + 1) / 2 + q)] = make_int2((int)p, (int)q);
  CK(df->colmn.alloc(np));
  CK(cudaMemcpyAsync(df->colmn.p, colmn.data(), np * sizeof(int2), cudaMemcpyHostToDevice, st));
  CK(cudaStreamSynchronize(st));
  df->naux = df->rank = df->rank_total = (int)rank;
  df->ncol = np;
  if (max_residual) *max_residual = maxres;
  if (n_pivots) *n_pivots = (int)rank;
  if (pivots)
    for (long long k = 0; k < rank && k < max_pivots; ++k) pivots[k] = piv[k];
  *out = df.release();
#undef CK
  return HFG_OK;
}
