// wt_lean.cuh — the fused step, one thread per cell, with lean addressing.
//
// Same semantics and per-cell rules as k_step (wt_step.cuh); the arithmetic
// is collide_x2 on one cell (scaled storage units, approximate reciprocal and
// square root, wt_x2.cuh). What differs is how the 38 population accesses of
// a cell are addressed: every thread forms one byte pointer to its cell in
// the read buffer and one in the write buffer, and each access adds a 32-bit
// byte offset that is the same for every thread of the launch (StepArgs
// srcb / dstb). A direction therefore costs one load or store plus at most
// one add, instead of a 64-bit multiply-add chain per access. Used when both
// population buffers span less than 2^31 bytes. Half storage rounds to nearest or
// stochastically (StepArgs f16_sr), as the direct kernel does.
#pragma once

#include "wt_x2.cuh"

namespace wt {

// Byte offset added to a cell pointer: zero-extended for half storage,
// sign-extended for float32 (the two measured fastest on B200 for each form;
// the offsets are non-negative either way).
template <class S>
__device__ __forceinline__ long long lean_off(uint32_t b) {
  if constexpr (sizeof(S) == 4) return (long long)(int)b;
  else return (long long)b;
}

// Resident blocks per SM the register budget is set for: float32 storage
// fits 72 registers without spills at 7 (28 warps; +3% over 64 registers
// and 8 blocks on B200), half storage is issue-bound and runs best at 8
// (32 warps, 64 registers; 7 measured -4%).
template <class S>
constexpr int lean_min_blocks() { return sizeof(S) == 4 ? 7 : 8; }

template <class S>
__global__ void __launch_bounds__(STEP_BX, lean_min_blocks<S>())
    k_step_lean(const __grid_constant__ StepArgs<S> a) {
  using T = X2<S>;
  constexpr float SC = T::SC;
  const Cell3 cell = step_cell(a);
  const int x = cell.x, y = cell.y, z = cell.z;
  const long long i = (long long)x + (long long)a.nx * y + a.nxy * z;
  const bool inside = x < a.nx - 1 && y < a.ny;
  pdl_enter();   // programmatic dependent launch (launch_pdl)
  prefetch_ahead(a, i - (long long)(threadIdx.x & 31));
  double Fx = 0, Fy = 0, Fz = 0;
  bool near_cell = false;
  if (inside) {
    // The outlet column x = nx-1 holds a copy of column nx-2 after the step
    // (js/lbm.js:504-511): the thread of cell nx-2 stores both.
    const bool dup = x == a.nx - 2;
    // The pulls of every cell that can be fluid are issued before its flags
    // byte arrives (all their sources lie inside the lattice), so a cell
    // waits for one memory latency instead of two.
    const bool inner = x >= 1 && y >= 1 && y <= a.ny - 2 && z >= 1 && z <= a.nz - 2;
    float f[Q];
    if (inner) {
      const char* Fb = reinterpret_cast<const char*>(a.F + i);
      const ShellRow row = shell_row(a, y, z);
      if (!row.any()) {
#pragma unroll
        for (int q = 0; q < Q; q++)
          f[q] = T::raw(*reinterpret_cast<const S*>(Fb + lean_off<S>(a.srcb[q])));
      } else {
#define WT_PULL(q) f[q] = T::raw(a.F[i + shell_src<q>(a, row)]);
        WT_EACH_Q(WT_PULL)
#undef WT_PULL
      }
    }
    int cat;
    uint8_t fl = 0;
    if (x == 0) {
      cat = CAT_EQ;
    } else {
      fl = a.flags[i];
      if (z == 0 || z == a.nz - 1 || y == a.ny - 1) cat = CAT_EQ;
      else if (fl & FLAG_SOLID_MASK) cat = CAT_KEEP;
      else if (y == 0) cat = CAT_EQ;
      else cat = CAT_FLUID;
    }
    char* Gb = reinterpret_cast<char*>(a.G + i);
    auto gs = [&](int q, int d = 0) -> S& {   // d = 1: the cell beside it
      return *(reinterpret_cast<S*>(Gb + lean_off<S>(a.dstb[q])) + d);
    };
    if (cat == CAT_FLUID) {   // implies inner
      const bool wall = (fl & FLAG_NEAR) != 0;
      if (wall) patch_raw<S>(a, i, f, Fx, Fy, Fz);
      near_cell = wall;
      float r, vx, vy, vz;
      collide_x2<S, float>(a, f, r, vx, vy, vz);
      if (!(r > 0.0f && r < 3.0e38f)) atomicOr(a.err, 1u);
      if (a.write_fields) {
        const float rho = r * (1.0f / SC);
        a.rho[i] = rho; a.ux[i] = vx; a.uy[i] = vy; a.uz[i] = vz;
        if (dup) { a.rho[i + 1] = rho; a.ux[i + 1] = vx; a.uy[i + 1] = vy; a.uz[i + 1] = vz; }
      }
      bool stored = false;
      if constexpr (std::is_same<S, __half>::value) {
        if (a.f16_sr) {
          // stochastic rounding, pairs converted together with the direct
          // kernel's per-cell, per-step random chain
          uint32_t h = ((uint32_t)i ^ (uint32_t)(i >> 32)) * 0x9E3779B1u ^ a.sr_seed;
          h ^= h >> 16; h *= 0x85EBCA6Bu; h ^= h >> 13; h *= 0xC2B2AE35u; h ^= h >> 16;
#pragma unroll
          for (int k = 1; k < Q; k += 2) {
            h ^= h << 13; h ^= h >> 17; h ^= h << 5;
            const __half2 p = sr_half2(f[k], f[k + 1], h);
            gs(k) = __high2half(p);
            gs(k + 1) = __low2half(p);
            if (dup) {
              gs(k, 1) = __high2half(p);
              gs(k + 1, 1) = __low2half(p);
            }
          }
          h ^= h << 13; h ^= h >> 17; h ^= h << 5;
          const __half p0 = __low2half(sr_half2(0.0f, f[0], h));
          gs(0) = p0;
          if (dup) gs(0, 1) = p0;
          stored = true;
        }
      }
      if (!stored) {
#pragma unroll
        for (int q = 0; q < Q; q++) gs(q) = T::to_s(f[q]);
        if (dup) {
#pragma unroll
          for (int q = 0; q < Q; q++) gs(q, 1) = T::to_s(f[q]);
        }
      }
    } else if (cat == CAT_EQ) {
#pragma unroll
      for (int q = 0; q < Q; q++) gs(q) = a.eq[q];
      if (dup) {
#pragma unroll
        for (int q = 0; q < Q; q++) gs(q, 1) = a.eq[q];
      }
      if (a.write_fields) {
        a.ux[i] = a.u0f; a.uy[i] = 0.0f; a.uz[i] = 0.0f; a.rho[i] = 1.0f;
        if (dup) { a.ux[i + 1] = a.u0f; a.uy[i + 1] = 0.0f; a.uz[i + 1] = 0.0f; a.rho[i + 1] = 1.0f; }
      }
    } else if (dup) {
      // outlet copy of a solid cell in column nx-2: its g is not written this step
      S v[Q];
#pragma unroll
      for (int q = 0; q < Q; q++) v[q] = gs(q);
#pragma unroll
      for (int q = 0; q < Q; q++) gs(q, 1) = v[q];
      if (a.write_fields) {
        a.ux[i + 1] = a.ux[i]; a.uy[i + 1] = a.uy[i]; a.uz[i + 1] = a.uz[i]; a.rho[i + 1] = a.rho[i];
      }
    }
    if (!near_cell) Fx = Fy = Fz = 0.0;
  }
  constexpr double inv_sc = 1.0 / (double)SC;   // a power of two: exact
  warp_force_partial(Fx * inv_sc, Fy * inv_sc, Fz * inv_sc, near_cell, a);
}

}  // namespace wt
