// Generic McMurchie-Davidson shell-quartet engine (eri_md.cu) for the
// angular classes with an f shell, which the generated Obara-Saika kernels
// do not cover.
#pragma once
#include <cuda_runtime.h>

#include "hfg_internal.h"

namespace hfg {

constexpr int kMDLMax = 3;  // highest shell angular momentum of the generic engine (f)

struct MDClass {
  int la, lb, lc, ld;
  int na, nb, nc, nd;  // Cartesian components per shell
  int L, lab, lcd;
};

MDClass md_class(int la, int lb, int lc, int ld);
bool md_class_ok(int la, int lb, int lc, int ld);

cudaError_t launch_schwarz_md(int la, int lb, const PairInfo* pairs, const PrimPair* prims, int first, int count,
                              const double* boys, double* out, int prim_mode, cudaStream_t st);
cudaError_t launch_quartet_md(int la, int lb, int lc, int ld, const PairInfo* pairs, const PrimPair* prims,
                              const double* boys, double* out, cudaStream_t st);
cudaError_t launch_eri_packed_md(int la, int lb, int lc, int ld, const JKEntry* entries, const long long* prefix,
                                 int nentries, long long nwarps, const PairInfo* pairs, const double* pairQ,
                                 double thr, const PrimRec64* rec, const float* pbound, const double* boys,
                                 double* out, cudaStream_t st);
// FP64 J/K over the launch's work queue (a.serial: one block, deterministic)
cudaError_t launch_jk_md(int la, int lb, int lc, int ld, const JKLaunchArgs& a, cudaStream_t st);
// Blocks of the J/K engine that an SM holds, about (by the class's block size)
int md_blocks_per_sm(int la, int lb, int lc, int ld);
// Whether the class's gradient kernel splits a quartet's primitive quartets
// over lanes by itself (the others take sliced entries)
bool eri_gradient_splits(int la, int lb, int lc, int ld);
// Nuclear derivatives of the two-electron energy over the launch's work
// queue (grad.cu; densities a.Dtot, a.Dspin; shells up to d): adds into
// grad[natom][3]
cudaError_t launch_eri_gradient(int la, int lb, int lc, int ld, const JKLaunchArgs& a, const int* ao_atom, int natom,
                                double* grad, cudaStream_t st);

}  // namespace hfg
