// Factored CUDA-core Signal: planning and launch (signal_gemm.cu).
#pragma once
#include "signal_common.cuh"

namespace fm {

// One of the two factorings of a problem: g[0] runs as columns, g[1] slabs
// (products 0: cannot apply).  Sized from the arguments alone; which one works
// is decided on the device (prep_static, prep_slab).
struct GemmPlan {
  int products;        // 1, or one per run
  int P, C;            // rows and columns of a product
  int TR, TC, nr, nc;  // threads and tiles along them
  int threads, smem, splits;
};

// Most bytes of the partial sums of a call's node splits.
constexpr int64_t kPartialBytes = 256LL << 20;

// `least`: node splits that fill the GPU by the tiles of an unfactored form.
template <typename T>
void plan_gemm(const fm_signal_args *a, const PrepDev &pr, int least, GemmPlan (&g)[2]);

template <typename T>
int launch_gemm(const fm_signal_args *a, const PrepDev &pr, const GemmPlan (&g)[2], T *out, T *partials,
                cudaStream_t st);

}  // namespace fm
