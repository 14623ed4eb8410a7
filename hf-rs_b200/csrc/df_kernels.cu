// Density fitting on the device: three-centre integrals (ab|P), the Coulomb
// metric (P|Q), and the unpack/convert kernels of the DF J/K contraction.
//
// hf-rs forms both with its four-centre engine and an exponent-0 unit
// partner (src/df.rs:30-78): (P|Q) = (P 1|Q 1), (P|mn) = (mn|P 1).  Here the
// same generated Obara-Saika classes EriClass<LA,LB,LC,0> evaluate them,
// with the auxiliary function and its unit partner as a one-centre "pair"
// (p = alpha_P, P = centre of P, prefactor c_P / alpha_P).
#include <cuda_bf16.h>
#include <algorithm>
#include <cuda_runtime.h>

#include "boys.cuh"
#include "df_internal.h"
#include "eri_gen.cuh"

namespace hfg {

constexpr double kTwoPiPow25df = 34.986836655249726164477;

__host__ __device__ constexpr int ncart_df(int l) { return (l + 1) * (l + 2) / 2; }

// 1/sqrt(prod (2 l_i - 1)!!) of component i of angular momentum l in hf-rs
// order (l <= 4).
__device__ __forceinline__ double comp_scale_any(int l, int i) {
  if (l < 2) return 1.0;
  int lx, ly, lz;
  if (l == 2) {
    const int t[6][3] = {{2, 0, 0}, {0, 2, 0}, {0, 0, 2}, {1, 1, 0}, {1, 0, 1}, {0, 1, 1}};
    lx = t[i][0];
    ly = t[i][1];
    lz = t[i][2];
  } else {
    int c = 0;
    lx = ly = lz = 0;
    for (int x = l; x >= 0; --x)
      for (int y = l - x; y >= 0; --y) {
        if (c == i) {
          lx = x;
          ly = y;
          lz = l - x - y;
        }
        ++c;
      }
  }
  auto df2 = [](int v) {  // (2v-1)!!
    double r = 1.0;
    for (int k = 2 * v - 1; k > 0; k -= 2) r *= k;
    return r;
  };
  return rsqrt(df2(lx) * df2(ly) * df2(lz));
}

// One block of (ab|P 1): bra pair i (orbital pair or unit-paired auxiliary
// shell), ket unit pair P, by a group of a.lanes lanes that split the bra's
// primitive pairs and add their accumulators by a butterfly.  Persistent
// blocks (the Boys table is staged once).
template <int LA, int LB, int LC>
__global__ void __launch_bounds__(128) df3c_kernel(const Df3cArgs a) {
  using C = EriClass<LA, LB, LC, 0>;
  constexpr int NA = ncart_df(LA), NB = ncart_df(LB), NC = ncart_df(LC);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* sm = reinterpret_cast<double*>(smem_raw);
  boys_stage<double, C::L>(sm, a.boys, a.expt);
  __syncthreads();
  const int gs = a.lanes, mem = threadIdx.x & (gs - 1);
  const long long total = (long long)a.nbra * a.nket, step = (long long)gridDim.x * blockDim.x / gs;
  const long long t0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / gs;
  // whole warps go round together (the butterfly needs every lane)
  for (long long base = 0; base < total; base += step) {
    const long long t = base + t0;
    const bool on = t < total;
    if (__ballot_sync(0xffffffffu, on) == 0u) break;
    const int ib = on ? (int)(t % a.nbra) : 0, ik = on ? (int)(t / a.nbra) : 0;
    const PairInfo bra = a.bra_pairs[a.bra_idx[ib]];
    const PairInfo ket = a.ket_pairs[a.ket_idx[ik]];
    double acc[C::NACC];
#pragma unroll
    for (int x = 0; x < C::NACC; ++x) acc[x] = 0.0;
    const double ACx = bra.Ax - ket.Ax, ACy = bra.Ay - ket.Ay, ACz = bra.Az - ket.Az;
    for (int q = 0; q < ket.npp; ++q) {
      const PrimPair Q = a.ket_prims[ket.pp_off + q];
      for (int p = mem; p < bra.npp; p += gs) {
        const PrimPair P = a.bra_prims[bra.pp_off + p];
        const double pp = P.p, qq = Q.p;
        const double PQx = ACx + P.PAx - Q.PAx, PQy = ACy + P.PAy - Q.PAy, PQz = ACz + P.PAz - Q.PAz;
        const double s = pp + qq, r = rsqrt(s), inv_s = r * r;
        const double tt = pp * qq * inv_s * (PQx * PQx + PQy * PQy + PQz * PQz);
        double F[C::L + 1];
        boys_eval<C::L>(tt, sm, F);
        const double pref = kTwoPiPow25df * P.kp * Q.kp * r;
#pragma unroll
        for (int m = 0; m <= C::L; ++m) F[m] *= pref;
        const double qs = qq * inv_s, ps = pp * inv_s;
        C::prim(acc, F, P.PAx, P.PAy, P.PAz, -qs * PQx, -qs * PQy, -qs * PQz, Q.PAx, Q.PAy, Q.PAz, ps * PQx,
                ps * PQy, ps * PQz, 0.5 * P.inv_p, 0.5 * Q.inv_p, 0.5 * inv_s, qs, ps);
      }
    }
    for (int off = 1; off < gs; off <<= 1) {
#pragma unroll
      for (int x = 0; x < C::NACC; ++x) acc[x] += __shfl_xor_sync(0xffffffffu, acc[x], off);
    }
    if (!on || mem != 0) continue;
    double out[C::NOUT];
    C::hrr(acc, out, bra.ABx, bra.ABy, bra.ABz, 0.0, 0.0, 0.0);
    // write: rows = ket functions (auxiliary), columns = bra components
    const long long col0 = a.bra_col[ib];
    const int kf0 = ket.ao_a;
#pragma unroll
    for (int i = 0; i < NA; ++i)
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        // unique AO pairs only: for a shell paired with itself keep i >= j
        if (bra.same && j > i) continue;
        const long long col = bra.same ? col0 + i * (i + 1) / 2 + j : col0 + i * NB + j;
        const double sab = comp_scale_any(LA, i) * comp_scale_any(LB, j);
#pragma unroll
        for (int k = 0; k < NC; ++k)
          a.out[(long long)(kf0 + k) * a.ld + col] = out[(i * NB + j) * NC + k] * sab * comp_scale_any(LC, k);
      }
  }
}

template <int LA, int LB, int LC>
static cudaError_t launch_df3c_class(const Df3cArgs& args, cudaStream_t st) {
  auto kern = df3c_kernel<LA, LB, LC>;
  const int smem = (int)boys_smem_bytes<double>();
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 128, smem);
  const long long want = ((long long)args.nbra * args.nket * args.lanes + 127) / 128,
                  fit = (long long)sms * (per_sm > 0 ? per_sm : 1);
  kern<<<(unsigned)std::min(want, fit), 128, smem, st>>>(args);
  return cudaGetLastError();
}

#define HFG_DF_CASE(A, B, Cc) \
  if (la == A && lb == B && lc == Cc) return launch_df3c_class<A, B, Cc>(args, st);
#define HFG_DF_KETS(A, B) \
  HFG_DF_CASE(A, B, 0) HFG_DF_CASE(A, B, 1) HFG_DF_CASE(A, B, 2) HFG_DF_CASE(A, B, 3) HFG_DF_CASE(A, B, 4)

cudaError_t launch_df3c(int la, int lb, int lc, Df3cArgs args, cudaStream_t st) {
  const long long total = (long long)args.nbra * args.nket;
  if (total <= 0) return cudaSuccess;
  // the high classes' straight-line code is too long to pass through for few
  // combinations (factor build and J/K in cc-pVDZ, limits of 0 / 5,000 /
  // 20,000 / 80,000 / no limit: one water 3.2 / 2.2 / 2.1 / 2.1 / 2.1 ms, (H2O)4 8.9 /
  // 8.2 / 8.2 / 8.2 / 8.2, (H2O)6 13.9 / 13.1 / 13.1 / 13.1 / 13.1; from L = 6
  // as fast as from 5, from L = 4 8% slower)
  if (la + lb + lc >= 5 && total <= 20000) return launch_df3c_md(la, lb, lc, args, st);
  // split the bra's primitive pairs over lanes while there are few
  // combinations, at least 4 per lane
  args.lanes = 1;
  while (args.lanes < 32 && 8 * args.lanes <= args.prims && total * args.lanes < 148 * 1024) args.lanes *= 2;
  HFG_DF_KETS(0, 0)
  HFG_DF_KETS(1, 0)
  HFG_DF_KETS(1, 1)
  HFG_DF_KETS(2, 0)
  HFG_DF_KETS(2, 1)
  HFG_DF_KETS(2, 2)
  HFG_DF_KETS(3, 0)
  HFG_DF_KETS(4, 0)
  return cudaErrorInvalidValue;
}

// Packed column of every (m, k) of B_Q into map (n x n, preset to -1).
__global__ void df_map_kernel(const int2* __restrict__ colmn, long long ncol, int n, int* __restrict__ map) {
  for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < ncol; c += (long long)gridDim.x * blockDim.x) {
    const int2 mn = colmn[c];
    map[(size_t)mn.x * n + mn.y] = (int)c;
    map[(size_t)mn.y * n + mn.x] = (int)c;
  }
}

cudaError_t launch_df_map(const int2* colmn, long long ncol, int n, int* map, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(map, 0xff, (size_t)n * n * 4, st);
  if (e != cudaSuccess || ncol <= 0) return e;
  df_map_kernel<<<(unsigned)std::min<long long>((ncol + 255) / 256, 148 * 8), 256, 0, st>>>(colmn, ncol, n, map);
  return cudaGetLastError();
}

// Unpack rows [q0, q0+qc) of B (rank x ncol, packed unique AO pairs) into
// the dense layout out[(m * qc + q) * n + k] = B_q[m][k] (both triangles),
// converted to the GEMM input type.  Every output element is written once,
// zeros included, in coalesced rows that gather from B_q through the map
// (a B_q row is re-read from L2); a scatter from the packed columns writes
// each pair to two far places in pieces of a sector and needs the chunk
// cleared first (J/K on the FP64 factor of (H2O)9, with this unpack and
// without: 0.81 and 1.22 ms).  The block's threads keep their map entries over
// its Q.
template <typename TO, typename TI>
__global__ void __launch_bounds__(256) df_unpack_kernel(const TI* __restrict__ B, long long ldb,
                                                        const int* __restrict__ map, int q0, int qc, int n,
                                                        TO* __restrict__ out) {
  constexpr int kRows = 4;  // rows m of one block: a shell's rows share the sectors of its pair blocks
  const int k = blockIdx.x * 64 + (threadIdx.x & 63), m = blockIdx.y * kRows + (threadIdx.x >> 6);
  if (k >= n || m >= n) return;
  const int c = __ldg(map + (size_t)m * n + k);
#pragma unroll 4
  for (int q = blockIdx.z; q < qc; q += gridDim.z) {
    TO v = (TO)0.0f;
    if (c >= 0) {
      const TI x = B[(size_t)(q0 + q) * ldb + c];
      if constexpr (sizeof(TI) == 8) v = x;
      else v = (TO)(float)x;
    }
    out[((size_t)m * qc + q) * n + k] = v;
  }
}

cudaError_t launch_df_unpack(int mode, const void* B, long long ldb, const int* map, int q0, int qc, int n, void* out,
                             cudaStream_t st) {
  if (qc <= 0) return cudaSuccess;
  // about 32 Q per block, so that the map is read once per 32 elements
  const dim3 grid((unsigned)((n + 63) / 64), (unsigned)((n + 3) / 4), (unsigned)std::min(qc, std::max(1, (qc + 31) / 32)));
  auto run = [&](auto kern, auto* src, auto* dst) {
    kern<<<grid, 256, 0, st>>>(src, ldb, map, q0, qc, n, dst);
    return cudaGetLastError();
  };
  using bf = __nv_bfloat16;
  if (mode == 0) return run(df_unpack_kernel<double, double>, (const double*)B, (double*)out);
  if (mode == 1) return run(df_unpack_kernel<float, float>, (const float*)B, (float*)out);
  if (mode == 2) return run(df_unpack_kernel<bf, bf>, (const bf*)B, (bf*)out);
  if (mode == 5) return run(df_unpack_kernel<bf, float>, (const float*)B, (bf*)out);
  if (mode == 3) return run(df_unpack_kernel<double, float>, (const float*)B, (double*)out);
  return run(df_unpack_kernel<double, bf>, (const bf*)B, (double*)out);
}

// J contractions on a stored FP32 / BF16 factor with FP64 accumulation
// (memory-bound: each reads B once): gam[q] = sum_c B[q][c] p[c], one block
// per auxiliary index; j[c] = sum_q B[q][c] gam[q], one thread per column.
template <typename TB>
__global__ void df_gamma_kernel(const TB* __restrict__ B, long long ncol, const double* __restrict__ p,
                                double* __restrict__ gam) {
  const long long row = (long long)blockIdx.x * ncol;
  double s = 0.0;
  for (long long c = threadIdx.x; c < ncol; c += blockDim.x) s += (double)(float)B[row + c] * p[c];
  for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  __shared__ double part[8];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += part[k];
    gam[blockIdx.x] = t;
  }
}

template <typename TB>
__global__ void df_jcol_kernel(const TB* __restrict__ B, long long ncol, int rank, const double* __restrict__ gam,
                               double* __restrict__ j) {
  for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < ncol; c += (long long)gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int q = 0; q < rank; ++q) s += (double)(float)B[(long long)q * ncol + c] * gam[q];
    j[c] = s;
  }
}

cudaError_t launch_df_j(int mode, const void* B, long long ncol, int rank, const double* p, double* gam, double* j,
                        cudaStream_t st) {
  if (ncol <= 0 || rank <= 0) return cudaSuccess;
  const unsigned grid = (unsigned)std::min<long long>((ncol + 255) / 256, 148 * 16);
  if (mode == 1) {
    df_gamma_kernel<float><<<rank, 256, 0, st>>>((const float*)B, ncol, p, gam);
    df_jcol_kernel<float><<<grid, 256, 0, st>>>((const float*)B, ncol, rank, gam, j);
  } else {
    df_gamma_kernel<__nv_bfloat16><<<rank, 256, 0, st>>>((const __nv_bfloat16*)B, ncol, p, gam);
    df_jcol_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>((const __nv_bfloat16*)B, ncol, rank, gam, j);
  }
  return cudaGetLastError();
}

// Packed density weights p[c] = P[m][n] (m == n) or 2 P[m][n] (m != n), so
// that gamma_Q = sum_c B[Q][c] p[c] = sum_mn B_Q[m][n] P[m][n].
__global__ void df_pack_density_kernel(const double* __restrict__ P, const int2* __restrict__ colmn, long long ncol,
                                       int n, double* __restrict__ p) {
  for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < ncol; c += (long long)gridDim.x * blockDim.x) {
    const int2 mn = colmn[c];
    const double v = P[(long long)mn.x * n + mn.y];
    p[c] = mn.x == mn.y ? v : 2.0 * v;
  }
}

// J from packed columns: J[m][n] = J[n][m] = j[c].
__global__ void df_unpack_j_kernel(const double* __restrict__ j, const int2* __restrict__ colmn, long long ncol, int n,
                                   double* __restrict__ J) {
  for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < ncol; c += (long long)gridDim.x * blockDim.x) {
    const int2 mn = colmn[c];
    J[(long long)mn.x * n + mn.y] = j[c];
    J[(long long)mn.y * n + mn.x] = j[c];
  }
}

// X[:, c] *= w[c]^{-1/2} (column-major, `rows` rows)
__global__ void whiten_kernel(double* __restrict__ X, const double* __restrict__ w, int rows, int cols) {
  const long long len = (long long)rows * cols;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (long long)gridDim.x * blockDim.x)
    X[i] *= 1.0 / sqrt(w[i / rows]);
}

cudaError_t launch_whiten(double* X, const double* w, int rows, int cols, cudaStream_t st) {
  const long long len = (long long)rows * cols;
  if (len <= 0) return cudaSuccess;
  whiten_kernel<<<(unsigned)std::min<long long>((len + 255) / 256, 148 * 32), 256, 0, st>>>(X, w, rows, cols);
  return cudaGetLastError();
}

template <typename TO>
__global__ void convert_kernel(const double* __restrict__ in, TO* __restrict__ out, long long len) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (long long)gridDim.x * blockDim.x)
    out[i] = (TO)(float)in[i];
}
template <>
__global__ void convert_kernel<double>(const double* __restrict__ in, double* __restrict__ out, long long len) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (long long)gridDim.x * blockDim.x)
    out[i] = in[i];
}

cudaError_t launch_convert(int mode, const double* in, void* out, long long len, cudaStream_t st) {
  const unsigned grid = (unsigned)std::min<long long>((len + 255) / 256, 148 * 32);
  if (len <= 0) return cudaSuccess;
  if (mode == 0) convert_kernel<double><<<grid, 256, 0, st>>>(in, (double*)out, len);
  else if (mode == 1) convert_kernel<float><<<grid, 256, 0, st>>>(in, (float*)out, len);
  else convert_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(in, (__nv_bfloat16*)out, len);
  return cudaGetLastError();
}

// out[r * ldo + c0 + j] = in[r * w + j] for r < rows, j < w (a chunk of B's
// columns, FP64 GEMM output, into the stored factor)
template <typename TO>
__global__ void convert_cols_kernel(const double* __restrict__ in, int w, long long rows, TO* __restrict__ out,
                                    long long ldo, long long c0) {
  const long long len = rows * w;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / w, j = i - r * w;
    out[r * ldo + c0 + j] = (TO)(float)in[i];
  }
}

cudaError_t launch_convert_cols(int mode, const double* in, int w, long long rows, void* out, long long ldo,
                                long long c0, cudaStream_t st) {
  const long long len = rows * w;
  if (len <= 0) return cudaSuccess;
  const unsigned grid = (unsigned)std::min<long long>((len + 255) / 256, 148 * 32);
  if (mode == 1) convert_cols_kernel<float><<<grid, 256, 0, st>>>(in, w, rows, (float*)out, ldo, c0);
  else convert_cols_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(in, w, rows, (__nv_bfloat16*)out, ldo, c0);
  return cudaGetLastError();
}

// acc (FP64) += 2 * src (FP32), n x n
__global__ void accumulate_f32_kernel(double* __restrict__ acc, const float* __restrict__ src, double scale,
                                      long long len) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (long long)gridDim.x * blockDim.x)
    acc[i] += scale * (double)src[i];
}

template <typename TO>
__global__ void convert_f32_kernel(const float* __restrict__ in, TO* __restrict__ out, long long len) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (long long)gridDim.x * blockDim.x)
    out[i] = (TO)in[i];
}

// FP32 -> FP64 (mode 0) or BF16 (mode 2)
cudaError_t launch_convert_f32(int mode, const float* in, void* out, long long len, cudaStream_t st) {
  if (len <= 0) return cudaSuccess;
  const unsigned grid = (unsigned)std::min<long long>((len + 255) / 256, 148 * 32);
  if (mode == 0) convert_f32_kernel<double><<<grid, 256, 0, st>>>(in, (double*)out, len);
  else convert_f32_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(in, (__nv_bfloat16*)out, len);
  return cudaGetLastError();
}

cudaError_t launch_pack_density(const double* P, const int2* colmn, long long ncol, int n, double* p, cudaStream_t st) {
  if (ncol <= 0) return cudaSuccess;
  const unsigned grid = (unsigned)std::min<long long>((ncol + 255) / 256, 148 * 32);
  df_pack_density_kernel<<<grid, 256, 0, st>>>(P, colmn, ncol, n, p);
  return cudaGetLastError();
}
cudaError_t launch_unpack_j(const double* j, const int2* colmn, long long ncol, int n, double* J, cudaStream_t st) {
  if (ncol <= 0) return cudaSuccess;
  const unsigned grid = (unsigned)std::min<long long>((ncol + 255) / 256, 148 * 32);
  df_unpack_j_kernel<<<grid, 256, 0, st>>>(j, colmn, ncol, n, J);
  return cudaGetLastError();
}
cudaError_t launch_accumulate_f32(double* acc, const float* src, double scale, long long len, cudaStream_t st) {
  if (len <= 0) return cudaSuccess;
  const unsigned grid = (unsigned)std::min<long long>((len + 255) / 256, 148 * 32);
  accumulate_f32_kernel<<<grid, 256, 0, st>>>(acc, src, scale, len);
  return cudaGetLastError();
}

}  // namespace hfg
