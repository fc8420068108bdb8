// wt_kernels_fast.cu — float32-arithmetic instantiations of the fused step
// (float32 and half-deviation storage), plus the force reduction. Built with
// the default multiply-add contraction.
#include "wt_internal.h"
#include "wt_pbb.cuh"
#include "wt_lean.cuh"
#include "wt_pair.cuh"

namespace wt {

void launch_step_f32_fast(const StepArgs<float>& a, dim3 grid, bool wide, cudaStream_t s) {
  if (wide) launch_pdl(k_step<float, false, long long, true>, grid, dim3(STEP_BX), s, a);
  else launch_pdl(k_step<float, false, int, true>, grid, dim3(STEP_BX), s, a);
}

void launch_step_f16_fast(const StepArgs<__half>& a, dim3 grid, bool wide, cudaStream_t s) {
  if (wide) launch_pdl(k_step<__half, false, long long, true>, grid, dim3(STEP_BX), s, a);
  else launch_pdl(k_step<__half, false, int, true>, grid, dim3(STEP_BX), s, a);
}

void launch_lean_f32(const StepArgs<float>& a, dim3 grid, bool, cudaStream_t s) {
  launch_pdl(k_step_lean<float>, grid, dim3(STEP_BX), s, a);
}

void launch_lean_f16(const StepArgs<__half>& a, dim3 grid, bool, cudaStream_t s) {
  launch_pdl(k_step_lean<__half>, grid, dim3(STEP_BX), s, a);
}

// Every step kernel (direct, lean, pair, partial bounce-back, adjoint)
// launches with programmatic dependent launch (launch_pdl): a step's blocks
// fill the slots the previous step's tail frees and start the moment it
// completes. Measured on B200: pair float32 +2.5% on 256x128x128, half
// storage +1-2%; the partial-bounce-back step on 128x64x64 +10%.
// The pair kernel's variant for a lattice, and the grid it runs on.
template <class S>
inline int pair_mode(const StepArgs<S>& a) {
  if (a.sfrac) return PAIR_PBB | (a.nx % 2 ? PAIR_ODD : 0);
  const bool rows = a.nx % (2 * PAIR_BX) == 0 && !a.zfast;
  return (a.nx % 2 ? PAIR_ODD : (rows ? PAIR_ROWS : 0)) | (a.mov ? PAIR_MOV : 0);
}

template <class S>
inline dim3 pair_grid(const StepArgs<S>& a, int mode) {
  const long long per = 2 * PAIR_BX;   // cells per block
  if (mode & PAIR_ROWS)
    return dim3((unsigned)(a.nx / per), (unsigned)a.ny, (unsigned)a.nz);
  const long long cells = (long long)row_cells(a.nx) * a.ny;
  return plane_grid((cells + per - 1) / per, a.nz, a.zfast != 0);
}

template <class S>
using PairKernel = void (*)(StepArgs<S>);

template <class S>
PairKernel<S> pair_kernel(bool sr, int mode) {
  if constexpr (sizeof(S) == 2) {
    if (sr) return mode & PAIR_ROWS ? k_step_pair<S, true, PAIR_ROWS> : k_step_pair<S, true, 0>;
    return mode & PAIR_ROWS ? k_step_pair<S, false, PAIR_ROWS> : k_step_pair<S, false, 0>;
  } else {
    switch (mode) {
      case PAIR_ODD: return k_step_pair<S, false, PAIR_ODD>;
      case PAIR_MOV: return k_step_pair<S, false, PAIR_MOV>;
      case PAIR_ODD | PAIR_MOV: return k_step_pair<S, false, PAIR_ODD | PAIR_MOV>;
      case PAIR_ROWS: return k_step_pair<S, false, PAIR_ROWS>;
      case PAIR_PBB: return k_step_pair<S, false, PAIR_PBB>;
      case PAIR_PBB | PAIR_ODD: return k_step_pair<S, false, PAIR_PBB | PAIR_ODD>;
      case PAIR_ROWS | PAIR_MOV: return k_step_pair<S, false, PAIR_ROWS | PAIR_MOV>;
      default: return k_step_pair<S, false, 0>;
    }
  }
}

// Every variant, for the preload loop below.
constexpr int kPairModes[] = {0, PAIR_ROWS, PAIR_ODD, PAIR_MOV, PAIR_ROWS | PAIR_MOV,
                              PAIR_ODD | PAIR_MOV};
template <class F>
cudaError_t each_pair_kernel(F f) {
  cudaError_t e = cudaSuccess;
  for (int m : kPairModes) {
    if (e == cudaSuccess) e = f((const void*)pair_kernel<float>(false, m));
    for (bool sr : {false, true})
      if (e == cudaSuccess && !(m & (PAIR_ODD | PAIR_MOV)))
        e = f((const void*)pair_kernel<__half>(sr, m));
  }
  return e;
}

template <class S>
void launch_pair(const StepArgs<S>& a, cudaStream_t s) {
  const int mode = pair_mode(a);
  launch_pdl(pair_kernel<S>(a.f16_sr != 0, mode), pair_grid(a, mode), dim3(PAIR_BX), s, a);
}

void launch_pair_f16(const StepArgs<__half>& a, dim3, bool, cudaStream_t s) { launch_pair(a, s); }

void launch_pair_f32(const StepArgs<float>& a, dim3, bool, cudaStream_t s) { launch_pair(a, s); }

// ---- partial bounce-back and adjoint (float32 arithmetic) -------------------------

// The float32 partial-bounce-back step runs the pair kernel (PAIR_PBB), except
// with moving walls or buffers of 2^31 bytes or more.
void launch_pbb_f32_fast(const StepArgs<float>& a, dim3 grid, bool wide, cudaStream_t s) {
  if (!a.mov && 19 * a.n * (long long)sizeof(float) < (1LL << 31)) return launch_pair(a, s);
  if (wide) launch_pdl(k_step_pbb<float, false, long long>, grid, dim3(STEP_BX), s, a);
  else launch_pdl(k_step_pbb<float, false, int>, grid, dim3(STEP_BX), s, a);
}

void launch_pbb_f16_fast(const StepArgs<__half>& a, dim3 grid, bool wide, cudaStream_t s) {
  if (wide) launch_pdl(k_step_pbb<__half, false, long long>, grid, dim3(STEP_BX), s, a);
  else launch_pdl(k_step_pbb<__half, false, int>, grid, dim3(STEP_BX), s, a);
}

void launch_adj_f32(const StepArgs<float>& a, const float* Tn, float* Tc, double* ds, double wJ,
                    int comp, cudaStream_t s) {
  launch_adjoint<float, float>(a, Tn, Tc, ds, wJ, comp, s);
}

void launch_adj_f16(const StepArgs<__half>& a, const float* Tn, float* Tc, double* ds, double wJ,
                    int comp, cudaStream_t s) {
  launch_adjoint<__half, float>(a, Tn, Tc, ds, wJ, comp, s);
}

// Marks the 32-cell segments that hold at least one near-wall cell.
__global__ void k_mark_segments(const uint8_t* __restrict__ flags, int nx, int ny, int nz,
                             uint8_t* __restrict__ mark) {
  const long long n = (long long)nx * ny * nz;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    if (flags[i] & FLAG_NEAR) {
      const int x = (int)(i % nx), y = (int)((i / nx) % ny), z = (int)(i / ((long long)nx * ny));
      mark[seg_of(x, y, z, nx, ny)] = 1;
    }
  }
}

void launch_mark_segments(const uint8_t* flags, int nx, int ny, int nz, uint8_t* mark,
                          cudaStream_t s) {
  k_mark_segments<<<148 * 16, 256, 0, s>>>(flags, nx, ny, nz, mark);
}

// One block per step; each thread sums a fixed strided subset of the warp
// partials, then a fixed-shape tree combines them. The order never depends
// on timing, so the force series is reproducible run to run.
constexpr int RED_T = 256;

__global__ void __launch_bounds__(RED_T) k_force_reduce(const double* __restrict__ part,
                                                        unsigned nblocks,
                                                        double* __restrict__ out) {
  __shared__ double sm[3][RED_T];
  const double* p = part + (size_t)blockIdx.x * nblocks * 3;
  double ax = 0, ay = 0, az = 0;
  for (unsigned b = threadIdx.x; b < nblocks; b += RED_T) {
    ax += p[3 * (size_t)b];
    ay += p[3 * (size_t)b + 1];
    az += p[3 * (size_t)b + 2];
  }
  sm[0][threadIdx.x] = ax;
  sm[1][threadIdx.x] = ay;
  sm[2][threadIdx.x] = az;
  __syncthreads();
  for (int w = RED_T / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) {
      sm[0][threadIdx.x] += sm[0][threadIdx.x + w];
      sm[1][threadIdx.x] += sm[1][threadIdx.x + w];
      sm[2][threadIdx.x] += sm[2][threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out[3 * (size_t)blockIdx.x] = sm[0][0];
    out[3 * (size_t)blockIdx.x + 1] = sm[1][0];
    out[3 * (size_t)blockIdx.x + 2] = sm[2][0];
  }
}

void launch_force_reduce(const double* part, unsigned nslots, int nsteps, double* out,
                         cudaStream_t s) {
  k_force_reduce<<<nsteps, RED_T, 0, s>>>(part, nslots, out);
}

cudaError_t configure_step_kernels(int nx, int storage) {
  // The pair kernels use no shared memory: the whole unified L1 / shared
  // array goes to L1 (measured on B200: +1.6% for half storage on
  // 256x128x128, +0.5% on 512x192x192, float32 unchanged). Only the variants a
  // lattice of this width can launch are touched.
  auto l1 = [](auto* f) {
    return cudaFuncSetAttribute((const void*)f, cudaFuncAttributePreferredSharedMemoryCarveout, 0);
  };
  const int m = nx % 2 ? PAIR_ODD : (nx % (2 * PAIR_BX) == 0 ? PAIR_ROWS : 0);
  cudaError_t e = cudaSuccess;
  if (storage == WT_STORE_F32) {
    e = l1(pair_kernel<float>(false, m));
    if (e == cudaSuccess) e = l1(pair_kernel<float>(false, m | PAIR_MOV));
  } else if (storage == WT_STORE_F16DEV && !(m & PAIR_ODD)) {
    e = l1(pair_kernel<__half>(false, m));
    if (e == cudaSuccess) e = l1(pair_kernel<__half>(true, m));
  }
  return e;
}

cudaError_t preload_step_kernels() {
  cudaFuncAttributes fa;
  const void* fns[] = {
      (const void*)k_step<float, false, int, true>, (const void*)k_step<float, false, long long, true>,
      (const void*)k_step<__half, false, int, true>, (const void*)k_step<__half, false, long long, true>,
      (const void*)k_step_lean<float>, (const void*)k_step_lean<__half>,
      (const void*)k_force_reduce};
  for (const void* f : fns) {
    const cudaError_t e = cudaFuncGetAttributes(&fa, f);
    if (e != cudaSuccess) return e;
  }
  const cudaError_t e =
      each_pair_kernel([&](const void* f) { return cudaFuncGetAttributes(&fa, f); });
  return e != cudaSuccess ? e : preload_exact_step_kernels();
}

}  // namespace wt
