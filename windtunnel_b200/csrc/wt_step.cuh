// wt_step.cuh — the fused D3Q19 step: pull-stream + halfway bounce-back +
// momentum exchange + moments + equilibrium + Smagorinsky + TRT collide +
// inlet / outlet / far-field boundaries, one launch per time step.
//
// Semantics follow one reference step, js/lbm.js:285-291: stepSlab over the
// interior (js/lbm.js:303-466) followed by _boundaries (js/lbm.js:473-512).
// The boundary pass is folded into the same launch by giving every cell a
// category that reproduces the reference's write order:
//   x == 0                         inlet: equilibrium (rho=1, u=(u0,0,0))
//   z == 0 | z == nz-1 | y == ny-1 end planes / ceiling: equilibrium
//   solid                          untouched (solid cells keep stale values)
//   y == 0 (not solid)             floor: equilibrium
//   otherwise                      fluid: collide and pull-stream
// and the outlet column x = nx-1 receives a copy of whatever column nx-2
// ends up holding; the thread of cell (nx-2, y, z) writes both cells, so the
// copy needs neither a second pass nor a second computation.
#pragma once

#include <type_traits>

#include "wt_common.cuh"

namespace wt {

// Load a stored deviation as the arithmetic type M.
template <class M, class S>
__device__ __forceinline__ M ld(S v) {
  if constexpr (std::is_same<M, double>::value) return Store<S>::load_d(v);
  else return Store<S>::load_f(v);
}

// Stochastic rounding of two floats to a half pair (hi <- a, lo <- b) with
// the random bits rbits (sm_100a cvt.rs).
__device__ __forceinline__ __half2 sr_half2(float a, float b, uint32_t rbits) {
  uint32_t d;
  asm("cvt.rs.f16x2.f32 %0, %1, %2, %3;" : "=r"(d) : "f"(a), "f"(b), "r"(rbits));
  return *reinterpret_cast<__half2*>(&d);
}

// Output writer of the collision: a register array of the step's outputs.
template <class S>
struct RegOut {
  S (&o)[Q];
  __device__ __forceinline__ void put(int q, S v) { o[q] = v; }
};

enum : int { CAT_NONE = 0, CAT_EQ = 1, CAT_KEEP = 2, CAT_FLUID = 3 };

// Sum three doubles over a warp that covers one 32-cell segment, in a fixed
// order, and store them in the segment's partial slot. Exactly the segments
// that hold a near-wall cell own a slot (the table is rebuilt by voxelize),
// and each of them is written every step -- zeros when none of its links
// touches the body -- so all-fluid warps write nothing and no block-wide
// barrier is needed. Every lane of the warp must call it; `near_cell` marks a
// computed near-wall cell.
template <class S>
__device__ __forceinline__ void warp_force_partial_w(double fx, double fy, double fz,
                                                     bool near_cell, const StepArgs<S>& a,
                                                     long long seg) {
  if (__any_sync(0xffffffffu, near_cell)) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      fx += __shfl_down_sync(0xffffffffu, fx, o);
      fy += __shfl_down_sync(0xffffffffu, fy, o);
      fz += __shfl_down_sync(0xffffffffu, fz, o);
    }
    if ((threadIdx.x & 31) == 0) {
      const int slot = a.wslot[seg];
      if (slot >= 0) {
        a.part[3 * (size_t)slot] = fx;
        a.part[3 * (size_t)slot + 1] = fy;
        a.part[3 * (size_t)slot + 2] = fz;
      } else {
        atomicOr(a.err, 2u);   // slot table out of date: reported, never silently dropped
      }
    }
  }
}

// Warp partial of the one-cell-per-thread kernels: their warps cover 32-cell
// segments.
template <class S>
__device__ __forceinline__ void warp_force_partial(double fx, double fy, double fz,
                                                   bool near_cell, const StepArgs<S>& a) {
  const long long seg = plane_of(a) * segs_per_plane(a.nx, a.ny) +
                        (long long)block_of(a) * (STEP_BX / 32) + (threadIdx.x >> 5);
  warp_force_partial_w(fx, fy, fz, near_cell, a, seg);
}

// Free-slip side planes: a cell of the layer beside one (y = 1 or ny-2, z = 1
// or nz-2) pulls a direction whose source lies on the plane as the mirrored
// direction of the source reflected into the layer itself, same x - ex. Which
// directions those are depends on the row alone, so a shell row's loads take
// the mirrored offset at once instead of overwriting plain values afterwards
// (one memory latency instead of two, which the last planes of a step have
// nothing to hide behind; B200, 256x128x128 float32, free-slip against equilibrium
// sides: 98.9 against 96.3 us a step with overwriting, 96.5 against 96.4 so).
struct ShellRow {
  bool y1, yn, z1, zn;
  __device__ __forceinline__ bool any() const { return y1 || yn || z1 || zn; }
};

template <class S>
__device__ __forceinline__ ShellRow shell_row(const StepArgs<S>& a, int y, int z) {
  const bool fs = a.freeslip != 0;
  return ShellRow{fs && y == 1, fs && y == a.ny - 2, fs && z == 1, fs && z == a.nz - 2};
}

// Element offset, from a shell cell, of the value its direction q pulls.
template <int q, class S>
__device__ __forceinline__ long long shell_src(const StepArgs<S>& a, const ShellRow& r) {
  if constexpr (ey(q) == 0 && ez(q) == 0) return a.src[q];
  const bool ym = ey(q) == 1 ? r.y1 : (ey(q) == -1 ? r.yn : false);
  const bool zm = ez(q) == 1 ? r.z1 : (ez(q) == -1 ? r.zn : false);
  if (ym && zm) return mirror_z(mirror_y(q)) * a.n - ex(q);
  if (ym) return mirror_y(q) * a.n - ex(q) - (long long)ez(q) * a.nxy;
  if (zm) return mirror_z(q) * a.n - ex(q) - (long long)ey(q) * a.nx;
  return a.src[q];
}

// X(q) for every direction.
#define WT_EACH_Q(X)                                                                        \
  X(0) X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16) \
  X(17) X(18)

// Overwrite, in f (already holding the plain pulled values), the directions
// whose source is solid (bounce-back, js/lbm.js:339-359), and accumulate the
// momentum exchange of links into the body (SOLID_OBJ). The solid / body neighbours come from
// the cell's precomputed mask (one load). Two passes: the first issues every
// load of the cell (they depend only on the mask and the cell's position) and
// consumes none, so that a near-wall warp waits for one memory latency
// instead of one per link; the second forms corrections and forces (measured
// on the pair kernel, pair_patch).
// T: the type of the held values (S itself where it holds every pulled value
// exactly, else the arithmetic type M); MOV as false drops the moving-wall
// correction at compile time.
template <class S, class M, class T, bool MOV>
__device__ __forceinline__ void patch_bounce(const StepArgs<S>& a, long long i, T (&f)[Q],
                                             double& Fx, double& Fy, double& Fz) {
  const unsigned long long m = a.nmask[i];
  const unsigned sm = (unsigned)m, om = (unsigned)(m >> 32);
  const bool mov = MOV && a.mov && sm;
  const M rho_prev = (M)(mov ? a.rho[i] : 1.0f);
  M cu[MOV ? Q : 1];
  auto held = [](S v) -> T {
    if constexpr (std::is_same<T, S>::value) return v;
    else return ld<T>(v);
  };
#define WT_PATCH(q)                                                                         \
  if constexpr (MOV) cu[q] = (M)0;                                                          \
  if ((sm >> (q)) & 1u) {                                                                   \
    f[q] = held(a.F[opp(q) * a.n + i]);                                                     \
    if (MOV && mov) {                                                                       \
      const long long j = i - (ex(q) + (long long)ey(q) * a.nx + (long long)ez(q) * a.nxy); \
      cu[q] = (M)ex(q) * (M)a.uwx[j] + (M)ey(q) * (M)a.uwy[j] + (M)ez(q) * (M)a.uwz[j];     \
    }                                                                                       \
  }
  WT_EACH_Q(WT_PATCH)
#undef WT_PATCH
  if (!(om || mov)) return;
#define WT_LINK(q)                                                             \
  if (((MOV && mov ? sm : om) >> (q)) & 1u) {                                  \
    M fd, corr = (M)0;                                                         \
    if constexpr (std::is_same<T, S>::value) fd = ld<M>(f[q]);                 \
    else fd = f[q];                                                            \
    if constexpr (MOV) {                                                       \
      if (cu[q] != (M)0) corr = (M)6 * (M)wq(q) * rho_prev * cu[q];            \
      if constexpr (std::is_same<T, M>::value) f[q] = fd + corr;               \
    }                                                                          \
    if ((om >> (q)) & 1u) {                                                    \
      const M d = (M)2 * fd + corr;                                            \
      Fx -= (double)(d * (M)ex(q));                                            \
      Fy -= (double)(d * (M)ey(q));                                            \
      Fz -= (double)(d * (M)ez(q));                                            \
    }                                                                          \
  }
  WT_EACH_Q(WT_LINK)
#undef WT_LINK
}

// Hardware approximations (relative error ~2^-22) used by the float32
// collisions: one instruction each instead of a correctly rounded sequence.
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float sqrt_approx(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Float32 collision, re-associated: opposite pairs are carried as half sums
// and half differences, so moments, the equilibrium, the stress tensor of the
// Smagorinsky model and the TRT update share their partial results. The
// mathematics is that of js/lbm.js:377-460; only the rounding differs.
template <class S, class Out>
__device__ __forceinline__ void collide_fast(const StepArgs<S>& a, const float (&f)[Q],
                                             long long i, bool dup, bool near_cell, Out out) {
  // opposite pairs (a, b) in the order of js/lbm.js:443-460
  const float s1 = f[1] + f[2], d1 = f[1] - f[2];
  const float s3 = f[3] + f[4], d3 = f[3] - f[4];
  const float s5 = f[5] + f[6], d5 = f[5] - f[6];
  const float s7 = f[7] + f[8], d7 = f[7] - f[8];
  const float s9 = f[9] + f[10], d9 = f[9] - f[10];
  const float s11 = f[11] + f[12], d11 = f[11] - f[12];
  const float s13 = f[13] + f[14], d13 = f[13] - f[14];
  const float s15 = f[15] + f[16], d15 = f[15] - f[16];
  const float s17 = f[17] + f[18], d17 = f[17] - f[18];
  const float dr = ((f[0] + s1) + (s3 + s5)) + ((s7 + s9) + (s11 + s13)) + (s15 + s17);
  const float r = 1.0f + dr;
  if (!(r > 0.0f && r < 3.0e38f)) atomicOr(a.err, 1u);
  // Half storage takes the one-instruction approximations (its step is
  // issue-bound); float32 keeps the correctly rounded forms, which measured
  // faster there (the approximations' register allocation spills at 64).
  constexpr bool APPROX = std::is_same<S, __half>::value;
  const float inv = APPROX ? rcp_approx(r) : __frcp_rn(r);
  const float vx = ((d1 + d7) + (d9 + d11) + d13) * inv;
  const float vy = ((d3 + d7) - d9 + (d15 + d17)) * inv;
  const float vz = ((d5 + d11) - d13 + (d15 - d17)) * inv;
  if (a.write_fields) {
    a.rho[i] = r; a.ux[i] = vx; a.uy[i] = vy; a.uz[i] = vz;
    if (dup) { a.rho[i + 1] = r; a.ux[i + 1] = vx; a.uy[i + 1] = vy; a.uz[i + 1] = vz; }
  } else if (a.mov && near_cell) {
    a.rho[i] = r;
  }
  const float A = dr - r * 1.5f * (vx * vx + vy * vy + vz * vz);
  const float r3 = 3.0f * r, r45 = 4.5f * r;
  constexpr float WF = (float)(1.0 / 18), WE = (float)(1.0 / 36), W0 = (float)(1.0 / 3);
  // per pair: symmetric equilibrium part es = w(A + 4.5 r cu^2) and
  // antisymmetric part ea = 3 w r cu; sp = (n_a + n_b)/2, sm = (n_a - n_b)/2
  const float c1 = vx, c3 = vy, c5 = vz, c7 = vx + vy, c9 = vx - vy, c11 = vx + vz,
              c13 = vx - vz, c15 = vy + vz, c17 = vy - vz;
  const float wAF = WF * A, wAE = WE * A, w45F = WF * r45, w45E = WE * r45, w3F = WF * r3,
              w3E = WE * r3;
#define WT_PAIR(k, C)                                                          \
  const float sp##k = fmaf(0.5f, s##k, -fmaf(w45##C * c##k, c##k, wA##C));   \
  const float sm##k = fmaf(0.5f, d##k, -w3##C * c##k);
  WT_PAIR(1, F) WT_PAIR(3, F) WT_PAIR(5, F) WT_PAIR(7, E) WT_PAIR(9, E) WT_PAIR(11, E)
  WT_PAIR(13, E) WT_PAIR(15, E) WT_PAIR(17, E)
#undef WT_PAIR
  float om = a.omega0f, omm = a.omm0f;
  if (a.les) {
    // Pi_ab = sum n_q c_qa c_qb from the pair half sums (n_a + n_b = 2 sp)
    const float sxx = (sp1 + sp7) + (sp9 + sp11) + sp13;
    const float syy = (sp3 + sp7) + (sp9 + sp15) + sp17;
    const float szz = (sp5 + sp11) + (sp13 + sp15) + sp17;
    const float sxy = sp7 - sp9, sxz = sp11 - sp13, syz = sp15 - sp17;
    const float qq = sxx * sxx + syy * syy + szz * szz + 2.0f * (sxy * sxy + sxz * sxz + syz * syz);
    // SQ18 * cs2 * |Pi| / r with |Pi| = 2 sqrt(2 qq): 72 cs2 sqrt(qq) / r
    const float tau0 = a.tau0f;
    const float te =
        APPROX ? 0.5f * (tau0 + sqrt_approx(fmaf(tau0, tau0, a.les_cf * sqrt_approx(qq) * inv)))
               : 0.5f * (tau0 + sqrtf(fmaf(tau0, tau0, a.les_cf * sqrtf(qq) * inv)));
    om = APPROX ? rcp_approx(te) : __frcp_rn(te);
    if (a.trt) {
      const float t5 = te - 0.5f;
      omm = __fdividef(t5, fmaf(0.5f, t5, a.lamf));
    } else {
      omm = om;
    }
  }
  const float e0 = W0 * A;
  const float g0 = fmaf(-om, f[0] - e0, f[0]);
#define WT_OUT(k, kb)                                                   \
  const float g##k = fmaf(-omm, sm##k, fmaf(-om, sp##k, f[k]));         \
  const float g##kb = fmaf(omm, sm##k, fmaf(-om, sp##k, f[kb]));
  WT_OUT(1, 2) WT_OUT(3, 4) WT_OUT(5, 6) WT_OUT(7, 8) WT_OUT(9, 10) WT_OUT(11, 12) WT_OUT(13, 14)
  WT_OUT(15, 16) WT_OUT(17, 18)
#undef WT_OUT
  if constexpr (std::is_same<S, __half>::value) {
    if (a.f16_sr) {
      // stochastic rounding to half: each opposite pair is converted together
      // with 32 random bits from a per-cell, per-step xorshift chain
      uint32_t h = ((uint32_t)i ^ (uint32_t)(i >> 32)) * 0x9E3779B1u ^ a.sr_seed;
      h ^= h >> 16; h *= 0x85EBCA6Bu; h ^= h >> 13; h *= 0xC2B2AE35u; h ^= h >> 16;
      constexpr float SC = (float)WT_F16_SCALE;
#define WT_SR(k, kb)                                                               \
  {                                                                                \
    h ^= h << 13; h ^= h >> 17; h ^= h << 5;                                       \
    const __half2 p = sr_half2(g##k * SC, g##kb * SC, h);                          \
    out.put(k, __high2half(p));                                                    \
    out.put(kb, __low2half(p));                                                    \
  }
      WT_SR(1, 2) WT_SR(3, 4) WT_SR(5, 6) WT_SR(7, 8) WT_SR(9, 10) WT_SR(11, 12)
      WT_SR(13, 14) WT_SR(15, 16) WT_SR(17, 18)
#undef WT_SR
      h ^= h << 13; h ^= h >> 17; h ^= h << 5;
      out.put(0, __low2half(sr_half2(0.0f, g0 * SC, h)));
      return;
    }
  }
  out.put(0, Store<S>::from_f(g0));
#define WT_PUT(k, kb) out.put(k, Store<S>::from_f(g##k)); out.put(kb, Store<S>::from_f(g##kb));
  WT_PUT(1, 2) WT_PUT(3, 4) WT_PUT(5, 6) WT_PUT(7, 8) WT_PUT(9, 10) WT_PUT(11, 12) WT_PUT(13, 14)
  WT_PUT(15, 16) WT_PUT(17, 18)
#undef WT_PUT
}

// Float64 collision in the exact operation order of js/lbm.js:377-460. The
// translation unit that instantiates it is compiled with --fmad=false, so no
// multiply-add is contracted and every rounding matches the reference's
// IEEE double arithmetic; results are rounded to S only at the stores.
// Two passes over the populations, which are held as T (the storage type
// where it represents them exactly): the first adds each non-equilibrium part
// n_q = f_q - e_q into the stress sums as soon as it is formed (the sums of
// js/lbm.js:420-425 run in ascending q, so their order is kept), the second
// forms e_q and n_q again and writes each output pair. The 18 doubles n_q are
// then never live together: 30% more float64 operations for half the
// registers. `opaque` keeps the compiler from merging the passes again.
__device__ __forceinline__ void opaque(double& v) { asm volatile("" : "+d"(v)); }
__device__ __forceinline__ void opaque(float& v) { asm volatile("" : "+f"(v)); }

template <class S, class T, class Out>
__device__ __forceinline__ void collide_exact(const StepArgs<S>& a, T (&f)[Q], long long i,
                                              bool dup, bool near_cell, Out out) {
  constexpr double W0 = 1.0 / 3, WF = 1.0 / 18, WE = 1.0 / 36;
  auto fd = [&](int q) -> double { return (double)f[q]; };
  double dr, vx, vy, vz, r, inv;
  {
    const double f0 = fd(0), f1 = fd(1), f2 = fd(2), f3 = fd(3), f4 = fd(4), f5 = fd(5),
                 f6 = fd(6), f7 = fd(7), f8 = fd(8), f9 = fd(9), f10 = fd(10), f11 = fd(11),
                 f12 = fd(12), f13 = fd(13), f14 = fd(14), f15 = fd(15), f16 = fd(16),
                 f17 = fd(17), f18 = fd(18);
    dr = f0 + f1 + f2 + f3 + f4 + f5 + f6 + f7 + f8 + f9 + f10 + f11 + f12 + f13 + f14 + f15 +
         f16 + f17 + f18;
    r = 1 + dr;
    if (!(r > 0.0 && r < 1.0e300)) atomicOr(a.err, 1u);
    inv = 1 / r;
    vx = (f1 - f2 + f7 - f8 + f9 - f10 + f11 - f12 + f13 - f14) * inv;
    vy = (f3 - f4 + f7 - f8 - f9 + f10 + f15 - f16 + f17 - f18) * inv;
    vz = (f5 - f6 + f11 - f12 - f13 + f14 + f15 - f16 - f17 + f18) * inv;
  }
  if (a.write_fields) {
    const float rf = __double2float_rn(r), xf = __double2float_rn(vx),
                yf = __double2float_rn(vy), zf = __double2float_rn(vz);
    a.rho[i] = rf; a.ux[i] = xf; a.uy[i] = yf; a.uz[i] = zf;
    if (dup) { a.rho[i + 1] = rf; a.ux[i + 1] = xf; a.uy[i + 1] = yf; a.uz[i + 1] = zf; }
  } else if (a.mov && near_cell) {
    a.rho[i] = __double2float_rn(r);
  }
  double A = dr - r * 1.5 * (vx * vx + vy * vy + vz * vz);
  double r3 = 3 * r, r45 = 4.5 * r;
  // equilibria of the opposite pair (k, k+1) along b = c_k . u, weight W:
  // e_k = W (A + r3 b + h), e_{k+1} = W (A - r3 b + h), h = r45 b b
#define WT_XEQ(W, B)                                     \
  const double b_ = B, t_ = r3 * b_, h_ = r45 * b_ * b_; \
  const double ea = W * (A + t_ + h_), eb = W * (A - t_ + h_);
  const double tau0 = a.tau0;
  double om = a.omega0, tauEff = tau0;
  if (a.les) {
    double pxx, pyy, pzz, pxy, pxz, pyz;
#define WT_XN(k, W, B) WT_XEQ(W, B) const double na = fd(k) - ea, nb = fd(k + 1) - eb;
    { WT_XN(1, WF, vx) pxx = na + nb; }
    { WT_XN(3, WF, vy) pyy = na + nb; }
    { WT_XN(5, WF, vz) pzz = na + nb; }
    { WT_XN(7, WE, vx + vy) pxx = pxx + na + nb; pyy = pyy + na + nb; pxy = na + nb; }
    { WT_XN(9, WE, vx - vy) pxx = pxx + na + nb; pyy = pyy + na + nb; pxy = pxy - na - nb; }
    { WT_XN(11, WE, vx + vz) pxx = pxx + na + nb; pzz = pzz + na + nb; pxz = na + nb; }
    { WT_XN(13, WE, vx - vz) pxx = pxx + na + nb; pzz = pzz + na + nb; pxz = pxz - na - nb; }
    { WT_XN(15, WE, vy + vz) pyy = pyy + na + nb; pzz = pzz + na + nb; pyz = na + nb; }
    { WT_XN(17, WE, vy - vz) pyy = pyy + na + nb; pzz = pzz + na + nb; pyz = pyz - na - nb; }
#undef WT_XN
    const double mag = sqrt(2 * (pxx * pxx + pyy * pyy + pzz * pzz +
                                 2 * (pxy * pxy + pxz * pxz + pyz * pyz)));
    const double SQ18 = 18 * 1.4142135623730951;
    tauEff = 0.5 * (tau0 + sqrt(tau0 * tau0 + SQ18 * a.cs2 * mag * inv));
    om = 1 / tauEff;
    opaque(A); opaque(r3); opaque(r45); opaque(vx); opaque(vy); opaque(vz);
    if constexpr (!std::is_same<T, double>::value) {
#pragma unroll
      for (int q = 0; q < Q; q++) opaque(f[q]);
    }
  }
  const double omm = a.trt ? 1 / (0.5 + a.lam / (tauEff - 0.5)) : om;
  {
    const double f0 = fd(0), e0 = W0 * A;
    out.put(0, Store<S>::from_d(f0 - om * (f0 - e0)));
  }
#define WT_XOUT(k, W, B)                                      \
  {                                                           \
    WT_XEQ(W, B)                                              \
    const double fa = fd(k), fb = fd(k + 1);                  \
    const double na = fa - ea, nb = fb - eb;                  \
    const double sp = 0.5 * (na + nb), sm = 0.5 * (na - nb);  \
    out.put(k, Store<S>::from_d(fa - om * sp - omm * sm));    \
    out.put(k + 1, Store<S>::from_d(fb - om * sp + omm * sm)); \
  }
  WT_XOUT(1, WF, vx)
  WT_XOUT(3, WF, vy)
  WT_XOUT(5, WF, vz)
  WT_XOUT(7, WE, vx + vy)
  WT_XOUT(9, WE, vx - vy)
  WT_XOUT(11, WE, vx + vz)
  WT_XOUT(13, WE, vx - vz)
  WT_XOUT(15, WE, vy + vz)
  WT_XOUT(17, WE, vy - vz)
#undef WT_XOUT
#undef WT_XEQ
}

// Output writer that stores straight to the cell (and, for the thread of
// column nx-2, to the outlet cell beside it).
template <class S, class IDX>
struct CellOut {
  S* g;
  const StepArgs<S>& a;
  bool dup;
  __device__ __forceinline__ void put(int q, S v) const {
    g[(IDX)a.dst[q]] = v;
    if (dup) g[(IDX)a.dst[q] + 1] = v;
  }
};

// Resident blocks per SM the register budget is set for. The float32 step is
// capped at 64 registers so that 8 blocks of 128 threads stay resident per SM:
// it is bound by memory latency, and resident warps are what keep enough of
// the 19 load streams in flight. Exact step, measured on B200 (blocks:
// microseconds a step): float64 storage, 192x96x96: 4: 93.9, 5: 85.8, 6: 83.9;
// float32 storage, 96x44x44: 4: 11.3, 5: 10.4, 6: 10.8, 7: 11.3; with moving
// walls the held values are doubles and 4 blocks leave them in registers.
template <class S, bool EXACT, bool MOV>
constexpr int step_min_blocks() {
  return EXACT ? (MOV ? 4 : (sizeof(S) == 8 ? 6 : 5)) : 8;
}

// IDX is the type of the per-direction offsets: int when 19*n fits in 31
// bits (every practical lattice), long long otherwise.
template <class S, bool EXACT, class IDX, bool MOV>
__global__ void __launch_bounds__(STEP_BX, step_min_blocks<S, EXACT, MOV>()) k_step(const __grid_constant__ StepArgs<S> a) {
  using M = typename std::conditional<EXACT, double, float>::type;
  // held values: the storage type unless a moving-wall correction can leave it
  using T = typename std::conditional<EXACT && !MOV, S, M>::type;
  const Cell3 cell = step_cell(a);
  const int x = cell.x, y = cell.y, z = cell.z;
  const long long i = (long long)x + (long long)a.nx * y + a.nxy * z;
  double Fx = 0, Fy = 0, Fz = 0;
  bool near_cell = false;
  const bool inside = x < a.nx - 1 && y < a.ny;
  const bool inner = inside && x > 0 && y > 0 && y < a.ny - 1 && z > 0 && z < a.nz - 1;
  pdl_enter();   // programmatic dependent launch (launch_pdl)
  if (inside) {
    T f[Q];
    // the pulls of every cell that can be fluid are issued before its flags
    // byte is looked at: all their sources lie inside the lattice
    if (inner) {
      const S* Fi = a.F + i;
      auto held = [](S v) -> T {
        if constexpr (std::is_same<T, S>::value) return v;
        else return ld<T>(v);
      };
      const ShellRow row = shell_row(a, y, z);
      if (!row.any()) {
#pragma unroll
        for (int q = 0; q < Q; q++) f[q] = held(Fi[(IDX)a.src[q]]);
      } else {
#define WT_PULL(q) f[q] = held(Fi[(IDX)shell_src<q>(a, row)]);
        WT_EACH_Q(WT_PULL)
#undef WT_PULL
      }
    }
    uint8_t fl = 0;
    if (x > 0) fl = a.flags[i];
    int cat;
    const bool dup = (x == a.nx - 2);   // this thread also writes the outlet cell x+1
    if (x == 0) cat = CAT_EQ;
    else if (z == 0 || z == a.nz - 1 || y == a.ny - 1) cat = CAT_EQ;
    else if (fl & FLAG_SOLID_MASK) cat = CAT_KEEP;
    else if (y == 0) cat = CAT_EQ;
    else cat = CAT_FLUID;
    S* Gi = a.G + i;
    if (cat == CAT_FLUID) {   // implies inner
      near_cell = (fl & FLAG_NEAR) != 0;
      if (near_cell) patch_bounce<S, M, T, MOV>(a, i, f, Fx, Fy, Fz);
      if constexpr (EXACT) {
        collide_exact<S>(a, f, i, dup, near_cell, CellOut<S, IDX>{Gi, a, dup});
      } else {
        S out[Q];
        collide_fast<S>(a, f, i, dup, near_cell, RegOut<S>{out});
#pragma unroll
        for (int q = 0; q < Q; q++) Gi[(IDX)a.dst[q]] = out[q];
        if (dup) {
#pragma unroll
          for (int q = 0; q < Q; q++) Gi[(IDX)a.dst[q] + 1] = out[q];
        }
      }
    } else if (cat == CAT_EQ) {
#pragma unroll
      for (int q = 0; q < Q; q++) Gi[(IDX)a.dst[q]] = a.eq[q];
      if (dup) {
#pragma unroll
        for (int q = 0; q < Q; q++) Gi[(IDX)a.dst[q] + 1] = a.eq[q];
      }
      if (a.write_fields) {
        a.ux[i] = a.u0f; a.uy[i] = 0.0f; a.uz[i] = 0.0f; a.rho[i] = 1.0f;
        if (dup) { a.ux[i + 1] = a.u0f; a.uy[i + 1] = 0.0f; a.uz[i + 1] = 0.0f; a.rho[i + 1] = 1.0f; }
      }
    } else if (dup) {
      // outlet copy of a solid cell in column nx-2: its g is not written this step
      // (all loads before the stores, which the compiler must assume to alias)
      S v[Q];
#pragma unroll
      for (int q = 0; q < Q; q++) v[q] = Gi[(IDX)a.dst[q]];
#pragma unroll
      for (int q = 0; q < Q; q++) Gi[(IDX)a.dst[q] + 1] = v[q];
      if (a.write_fields) {
        a.ux[i + 1] = a.ux[i]; a.uy[i + 1] = a.uy[i]; a.uz[i + 1] = a.uz[i]; a.rho[i + 1] = a.rho[i];
      }
    }
  }
  warp_force_partial(Fx, Fy, Fz, near_cell, a);
}

}  // namespace wt
