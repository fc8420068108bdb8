// wt_voxel.cu — Voxel.build (js/voxel.js:32-232) on the GPU.
//
// A triangle soup (float32, nine numbers per triangle, body space) becomes the
// body-space occupancy grid the device lookup (wt_voxelize_grid) samples: the
// cells the surface passes through (a sampled rasterisation of every
// triangle) OR'd with a two-of-three vote of ray-parity fills along x, y and
// z. This translation unit is compiled without multiply-add contraction and
// every step is float64 in the reference's operation order, so the grid is
// the reference's bit for bit.
//
// Kernels, per build (the benchmark's 20000-triangle hull at 160 cells, B200: 0.17 ms
// on the device, 2.3 ms before the changes named below):
//   k_vox_shell      one warp per triangle, its lanes over the triangle's (u, v)
//                    samples; marks the shell cells
//   k_vox_count      per triangle and ray axis its bucket rectangle in the plane
//                    normal to the axis (48 x 48 buckets at most,
//                    js/voxel.js:151-171), and the buckets' counts
//   k_vox_scan       exclusive scan of the counts, one block per axis
//   k_vox_fill       every triangle into its buckets' lists
//   k_vox_order      one warp per bucket puts its list into triangle order, the
//                    reference's (a walk of all triangles per bucket, which
//                    needs no ordering, took 1.5 ms of the 2.3)
//   k_vox_rays       one warp per ray (column): the lanes test the bucket's
//                    triangles, keep the crossings (at most 512, as the
//                    reference), sort them and add a vote to the cells between
//                    alternate pairs (one thread per ray waited for every
//                    triangle in turn and sorted in global memory: 0.49 ms)
//   k_vox_combine    grid = (votes >= 2) | shell, with the solid and
//                    disagreeing-cell counts
// Bound now by host work: allocation, the copies of triangles and grid.
#include <math.h>

#include <algorithm>
#include <string>
#include <vector>

#include "wt_internal.h"

namespace {

constexpr int kBuckets = 48;
constexpr int kMaxHits = 512;
constexpr double kMaxSamples = 4096.0;

struct VoxGeom {
  int nx, ny, nz;
  double cell, inv;
  double min[3];
};

// ECMAScript ToInt32 of a finite or infinite double (js `x | 0`).
__device__ __forceinline__ int32_t to_int32(double v) {
  if (!isfinite(v)) return 0;
  if (v > -2147483649.0 && v < 2147483648.0) return (int32_t)v;
  double m = fmod(trunc(v), 4294967296.0);
  if (m < 0) m += 4294967296.0;
  return (int32_t)(uint32_t)m;
}

__global__ void k_vox_shell(const float* __restrict__ P, long long ntri, VoxGeom g,
                            uint8_t* __restrict__ shell) {
  const long long t = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (t >= ntri) return;
  const float* o = P + 9 * t;
  const double ax = o[0], ay = o[1], az = o[2], bx = o[3], by = o[4], bz = o[5];
  const double cx = o[6], cy = o[7], cz = o[8];
  const double inv = 1 / g.cell;
  const double e1 = fmax(fmax(fabs(bx - ax), fabs(by - ay)), fabs(bz - az));
  const double e2 = fmax(fmax(fabs(cx - ax), fabs(cy - ay)), fabs(cz - az));
  double n1 = ceil(e1 * inv * 2) + 1, n2 = ceil(e2 * inv * 2) + 1;
  if (n1 * n2 > kMaxSamples) {
    const double k = sqrt(kMaxSamples / (n1 * n2));
    n1 = fmax(2.0, (double)to_int32(n1 * k));
    n2 = fmax(2.0, (double)to_int32(n2 * k));
  }
  auto mark = [&](double i, double u, double j) {
    const double v = fmin(j / n2, 1 - u);
    const double x = ax + (bx - ax) * u + (cx - ax) * v;
    const double y = ay + (by - ay) * u + (cy - ay) * v;
    const double z = az + (bz - az) * u + (cz - az) * v;
    const int32_t gx = to_int32((x - g.min[0]) * inv);
    const int32_t gy = to_int32((y - g.min[1]) * inv);
    const int32_t gz = to_int32((z - g.min[2]) * inv);
    if (gx < 0 || gy < 0 || gz < 0 || gx >= g.nx || gy >= g.ny || gz >= g.nz) return;
    shell[gx + (long long)g.nx * (gy + (long long)g.ny * gz)] = 1;
  };
  if (n1 <= 255 && n2 <= 255) {
    // lanes over the samples (i, j), i in 0..n1, j in 0..n2, those with
    // j <= ceil((1 - i/n1) n2) taken
    const int w = (int)n2 + 1, all = ((int)n1 + 1) * w;
    for (int k = lane; k < all; k += 32) {
      const int ii = k / w;
      const double i = ii, j = k - ii * w, u = i / n1;
      if (j <= ceil((1 - u) * n2)) mark(i, u, j);
    }
    return;
  }
  // long thin triangles (and NaN counts, which mark nothing): lanes over i
  for (double i = lane; i <= n1; i += 32) {
    const double u = i / n1;
    const double jmax = ceil((1 - u) * n2);
    for (double j = 0; j <= jmax; j++) mark(i, u, j);
  }
}

struct AxisGeom {
  int A, B, C, nA, nB, nC, nbB, nbC;
  double minA, minB, minC, kB, kC, cell;
  long long strideA, strideB, strideC;
};
struct AllAxes {
  AxisGeom x[3];
};

constexpr int kNb = kBuckets * kBuckets;   // most buckets of an axis
struct ListBase {
  long long at[3];   // where each axis's lists begin
};

// Triangle t into its bucket rectangle for ray axis blockIdx.y, and the
// buckets' counts.
__global__ void k_vox_count(const float* __restrict__ P, long long ntri, const AllAxes ax,
                            int4* __restrict__ rects, int* __restrict__ counts) {
  const AxisGeom& x = ax.x[blockIdx.y];
  int4* rect = rects + (size_t)blockIdx.y * ntri;
  int* count = counts + blockIdx.y * kNb;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < ntri;
       t += (long long)gridDim.x * blockDim.x) {
    const float* o = P + 9 * t;
    const double b0 = o[x.B], b1 = o[3 + x.B], b2 = o[6 + x.B];
    const double c0 = o[x.C], c1 = o[3 + x.C], c2 = o[6 + x.C];
    double bl = floor((fmin(fmin(b0, b1), b2) - x.minB) * x.kB);
    double bh = floor((fmax(fmax(b0, b1), b2) - x.minB) * x.kB);
    double cl = floor((fmin(fmin(c0, c1), c2) - x.minC) * x.kC);
    double ch = floor((fmax(fmax(c0, c1), c2) - x.minC) * x.kC);
    bl = bl < 0 ? 0 : bl;
    bh = bh >= x.nbB ? x.nbB - 1 : bh;
    cl = cl < 0 ? 0 : cl;
    ch = ch >= x.nbC ? x.nbC - 1 : ch;
    // an empty rectangle (the triangle lies outside the buckets) is stored as one
    const int4 r = (bl > bh || cl > ch) ? make_int4(1, 0, 1, 0)
                                        : make_int4((int)bl, (int)bh, (int)cl, (int)ch);
    rect[t] = r;
    for (int cc = r.z; cc <= r.w; cc++)
      for (int bb = r.x; bb <= r.y; bb++)
        if (bb >= 0 && bb < x.nbB && cc >= 0 && cc < x.nbC) atomicAdd(&count[bb + x.nbB * cc], 1);
  }
}

// Exclusive scan of an axis's counts (one block per axis; at most kNb of them),
// into start[0..nb] and the fill cursors.
constexpr int SCAN_T = 768, SCAN_PER = kNb / SCAN_T;
static_assert(SCAN_T * SCAN_PER == kNb, "the scan block covers every bucket");

__global__ void __launch_bounds__(SCAN_T) k_vox_scan(const int* __restrict__ counts,
                                                     const AllAxes ax, int* __restrict__ starts,
                                                     int* __restrict__ cursors,
                                                     int* __restrict__ totals) {
  __shared__ int part[SCAN_T / 32];
  const int A = blockIdx.x, nb = ax.x[A].nbB * ax.x[A].nbC;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int v[SCAN_PER], sum = 0;
#pragma unroll
  for (int k = 0; k < SCAN_PER; k++) {
    const int b = threadIdx.x * SCAN_PER + k;
    v[k] = b < nb ? counts[A * kNb + b] : 0;
    sum += v[k];
  }
  int inc = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  if (lane == 31) part[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    int p = lane < SCAN_T / 32 ? part[lane] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, p, o);
      if (lane >= o) p += u;
    }
    if (lane < SCAN_T / 32) part[lane] = p;
  }
  __syncthreads();
  int acc = inc - sum + (warp ? part[warp - 1] : 0);
  int* start = starts + A * (kNb + 1);
#pragma unroll
  for (int k = 0; k < SCAN_PER; k++) {
    const int b = threadIdx.x * SCAN_PER + k;
    if (b < nb) {
      start[b] = acc;
      cursors[A * kNb + b] = acc;
    }
    acc += v[k];
  }
  if (threadIdx.x == SCAN_T - 1) {
    start[nb] = acc;
    totals[A] = acc;
  }
}

__global__ void k_vox_fill(const int4* __restrict__ rects, long long ntri, const AllAxes ax,
                           int* __restrict__ cursors, int* __restrict__ items, const ListBase base) {
  const int A = blockIdx.y, nbB = ax.x[A].nbB, nbC = ax.x[A].nbC;
  int* it = items + base.at[A];
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < ntri;
       t += (long long)gridDim.x * blockDim.x) {
    const int4 r = rects[(size_t)A * ntri + t];
    for (int cc = r.z; cc <= r.w; cc++)
      for (int bb = r.x; bb <= r.y; bb++)
        if (bb >= 0 && bb < nbB && cc >= 0 && cc < nbC)
          it[atomicAdd(&cursors[A * kNb + bb + nbB * cc], 1)] = (int)t;
  }
}

// A bucket's list in triangle order. Up to kSortMax items: every item's rank is
// the number of smaller ones, counted in shared memory (32 items against all per
// round). Longer lists are written again by a walk of all triangles, 32 at a
// time, whose members a ballot ranks.
constexpr int kSortMax = 1024, ORDER_WARPS = 4;

__global__ void __launch_bounds__(32 * ORDER_WARPS)
    k_vox_order(const int4* __restrict__ rects, long long ntri, const AllAxes ax,
                const int* __restrict__ starts, int* __restrict__ items, const ListBase base) {
  __shared__ int sh[ORDER_WARPS][kSortMax];
  const int A = blockIdx.y, b = blockIdx.x * ORDER_WARPS + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const int nbB = ax.x[A].nbB, nb = nbB * ax.x[A].nbC;
  if (b >= nb) return;   // whole warps leave together
  const int s = starts[A * (kNb + 1) + b], n = starts[A * (kNb + 1) + b + 1] - s;
  int* it = items + base.at[A] + s;
  if (n <= kSortMax) {
    int* v = sh[threadIdx.x >> 5];
    for (int k = lane; k < n; k += 32) v[k] = it[k];
    __syncwarp();
    for (int k = lane; k < n; k += 32) {
      const int me = v[k];
      int rank = 0;
      for (int m = 0; m < n; m++) rank += v[m] < me;
      it[rank] = me;
    }
    return;
  }
  const int bb = b % nbB, cc = b / nbB;
  int k = 0;
  for (long long t0 = 0; t0 < ntri; t0 += 32) {
    const long long t = t0 + lane;
    bool hit = false;
    if (t < ntri) {
      const int4 r = rects[(size_t)A * ntri + t];
      hit = bb >= r.x && bb <= r.y && cc >= r.z && cc <= r.w;
    }
    const unsigned m = __ballot_sync(0xffffffffu, hit);
    if (hit) it[k + __popc(m & ((1u << lane) - 1u))] = (int)t;
    k += __popc(m);
  }
}

constexpr int RAY_WARPS = 4;

__global__ void __launch_bounds__(32 * RAY_WARPS)
    k_vox_rays(const float* __restrict__ P, const int* __restrict__ start,
               const int* __restrict__ items, AxisGeom x, uint8_t* __restrict__ votes) {
  __shared__ double raw[RAY_WARPS][kMaxHits], sorted[RAY_WARPS][kMaxHits];
  const long long col = (long long)blockIdx.x * RAY_WARPS + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (col >= (long long)x.nB * x.nC) return;   // whole warps leave together
  const int ib = (int)(col % x.nB), ic = (int)(col / x.nB);
  const double pc = x.minC + (ic + 0.5003719) * x.cell;
  const int bc = (int)fmin((double)(x.nbC - 1), fmax(0.0, floor((pc - x.minC) * x.kC)));
  const double pb = x.minB + (ib + 0.4996281) * x.cell;
  const int bb = (int)fmin((double)(x.nbB - 1), fmax(0.0, floor((pb - x.minB) * x.kB)));
  const int s = start[bb + x.nbB * bc], e = start[bb + x.nbB * bc + 1];
  double* hits = raw[threadIdx.x >> 5];
  int nh = 0;
  bool nan = false;
  for (int k0 = s; k0 < e && nh < kMaxHits; k0 += 32) {
    const int k = k0 + lane;
    bool hit = false;
    double h = 0;
    if (k < e) {
      const float* o = P + 9 * (long long)items[k];
      const double b0 = o[x.B], c0 = o[x.C], b1 = o[3 + x.B], c1 = o[3 + x.C];
      const double b2 = o[6 + x.B], c2 = o[6 + x.C];
      const double d = (c1 - c2) * (b0 - b2) + (b2 - b1) * (c0 - c2);
      if (!(d == 0)) {
        const double id = 1 / d;
        const double l0 = ((c1 - c2) * (pb - b2) + (b2 - b1) * (pc - c2)) * id;
        const double l1 = ((c2 - c0) * (pb - b2) + (b0 - b2) * (pc - c2)) * id;
        const double l2 = 1 - l0 - l1;
        hit = !(l0 < 0 || l0 > 1 || l1 < 0 || l1 > 1 || l2 < 0 || l2 > 1);
        if (hit) h = l0 * (double)o[x.A] + l1 * (double)o[3 + x.A] + l2 * (double)o[6 + x.A];
      }
    }
    const unsigned m = __ballot_sync(0xffffffffu, hit);
    const int at = nh + __popc(m & ((1u << lane) - 1u));
    if (hit && at < kMaxHits) hits[at] = h;
    nan = nan || (hit && isnan(h));
    nh = min(kMaxHits, nh + __popc(m));
  }
  if (nh < 2) return;
  nan = __any_sync(0xffffffffu, nan);
  __syncwarp();
  if (nan) {
    // not an order: the reference's insertion sort, step by step
    if (lane == 0)
      for (int a = 1; a < nh; a++) {
        const double v = hits[a];
        int b = a - 1;
        while (b >= 0 && hits[b] > v) {
          hits[b + 1] = hits[b];
          b--;
        }
        hits[b + 1] = v;
      }
  } else {
    double* to = sorted[threadIdx.x >> 5];
    for (int a = lane; a < nh; a += 32) {
      const double v = hits[a];
      int rank = 0;
      for (int b = 0; b < nh; b++) rank += hits[b] < v || (hits[b] == v && b < a);
      to[rank] = v;
    }
    hits = to;
  }
  __syncwarp();
  const long long colBase = ib * x.strideB + ic * x.strideC;
  for (int k = 0; k + 1 < nh; k += 2) {
    double i0 = ceil((hits[k] - x.minA) / x.cell - 0.5);
    double i1 = floor((hits[k + 1] - x.minA) / x.cell - 0.5);
    if (i0 < 0) i0 = 0;
    if (i1 >= x.nA) i1 = x.nA - 1;
    for (double ia = i0 + lane; ia <= i1; ia += 32)
      votes[colBase + (long long)ia * x.strideA]++;
    __syncwarp();   // touching spans may add to one cell twice
  }
}

__global__ void k_vox_combine(const uint8_t* __restrict__ votes, const uint8_t* __restrict__ shell,
                              long long n, uint8_t* __restrict__ grid,
                              unsigned long long* __restrict__ counts) {
  unsigned solid = 0, disagree = 0;   // n <= 4e7
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int v = votes[i];
    const bool inside = v >= 2 || shell[i] == 1;
    solid += inside;
    disagree += (v == 1 || v == 2);
    grid[i] = inside ? 1 : 0;
  }
  __shared__ unsigned sums[2];
  if (threadIdx.x < 2) sums[threadIdx.x] = 0;
  __syncthreads();
  solid = __reduce_add_sync(0xffffffffu, solid);
  disagree = __reduce_add_sync(0xffffffffu, disagree);
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&sums[0], solid);
    atomicAdd(&sums[1], disagree);
  }
  __syncthreads();
  if (threadIdx.x < 2) atomicAdd(&counts[threadIdx.x], (unsigned long long)sums[threadIdx.x]);
}

thread_local std::string g_vox_error;

int vox_fail(int code, const std::string& msg) {
  g_vox_error = msg;
  return code;
}

// Device buffers of one build, released on every exit path.
struct VoxBuffers {
  std::vector<void*> ptrs;
  void* get(size_t n) {
    void* p = nullptr;
    if (cudaMalloc(&p, n ? n : 1) != cudaSuccess) return nullptr;
    ptrs.push_back(p);
    return p;
  }
  ~VoxBuffers() {
    for (void* p : ptrs) cudaFree(p);
  }
};

}  // namespace

extern "C" {

const char* wt_voxel_last_error(void) { return g_vox_error.c_str(); }

int wt_voxel_dims(const float* tris, int64_t ntri, int res, wt_voxel_info* info) {
  g_vox_error.clear();
  if (!info || (ntri > 0 && !tris)) return vox_fail(WT_ERR_ARG, "tris and info are required");
  if (res <= 0) res = 96;
  if (ntri <= 0) return vox_fail(WT_ERR_ARG, "Mesh has no triangles.");
  // js/voxel.js:32-42 (bounds) and :48-71
  // bounds per coordinate of a triangle (nine independent lanes, so that the
  // compiler uses packed minima), then over its three vertices; a NaN never
  // compares less or greater, as in the reference's ifs
  float lo[9], hi[9];
  for (int k = 0; k < 9; k++) {
    lo[k] = INFINITY;
    hi[k] = -INFINITY;
  }
  for (int64_t t = 0; t < ntri; t++) {
    const float* v = tris + 9 * t;
    for (int k = 0; k < 9; k++) {
      lo[k] = v[k] < lo[k] ? v[k] : lo[k];
      hi[k] = v[k] > hi[k] ? v[k] : hi[k];
    }
  }
  auto least = [&](int k) { return (double)std::min(lo[k], std::min(lo[k + 3], lo[k + 6])); };
  auto most = [&](int k) { return (double)std::max(hi[k], std::max(hi[k + 3], hi[k + 6])); };
  const double x0 = least(0), y0 = least(1), z0 = least(2);
  const double x1 = most(0), y1 = most(1), z1 = most(2);
  const double sx = x1 - x0, sy = y1 - y0, sz = z1 - z0;
  const double span = fmax(fmax(sx, sy), sz);
  if (!(span > 0)) return vox_fail(WT_ERR_ARG, "Mesh is degenerate (zero size).");
  const double cell = span / res;
  const double dx = fmax(3, ceil(sx / cell) + 4), dy = fmax(3, ceil(sy / cell) + 4),
               dz = fmax(3, ceil(sz / cell) + 4);
  if (dx * dy * dz > 40e6)
    return vox_fail(WT_ERR_ARG, "Voxel grid too large; lower the resolution.");
  memset(info, 0, sizeof(*info));
  info->nx = (int32_t)dx;
  info->ny = (int32_t)dy;
  info->nz = (int32_t)dz;
  info->tris = ntri;
  info->cell = cell;
  info->inv = 1 / cell;
  info->min[0] = x0 - (info->nx * cell - sx) * 0.5;
  info->min[1] = y0 - (info->ny * cell - sy) * 0.5;
  info->min[2] = z0 - (info->nz * cell - sz) * 0.5;
  info->ext[0] = sx * 0.5; info->ext[1] = sy * 0.5; info->ext[2] = sz * 0.5;
  info->centre[0] = (x0 + x1) * 0.5; info->centre[1] = (y0 + y1) * 0.5;
  info->centre[2] = (z0 + z1) * 0.5;
  info->bbox[0] = x0; info->bbox[1] = y0; info->bbox[2] = z0;
  info->bbox[3] = x1; info->bbox[4] = y1; info->bbox[5] = z1;
  return WT_OK;
}

int wt_voxel_build(const float* tris, int64_t ntri, int res, uint8_t* grid, size_t grid_len,
                   wt_voxel_info* info) {
  int c = wt_voxel_dims(tris, ntri, res, info);
  if (c != WT_OK) return c;
  const long long n = (long long)info->nx * info->ny * info->nz;
  if (!grid || grid_len != (size_t)n)
    return vox_fail(WT_ERR_ARG, "grid must hold nx*ny*nz = " + std::to_string(n) + " bytes");
  const int dim[3] = {info->nx, info->ny, info->nz};
  // One device block: the triangles, the three byte grids, the bucket tables and
  // room for the bucket lists of an ordinary mesh (a triangle in a few buckets).
  auto up = [](size_t v) { return (v + 255) & ~(size_t)255; };
  const size_t cap = std::max<size_t>(12 * (size_t)ntri, 1 << 14);
  const size_t sz_p = up(sizeof(float) * 9 * (size_t)ntri), sz_n = up((size_t)n),
               sz_r = up(sizeof(int4) * 3 * (size_t)ntri), sz_i = up(sizeof(int) * cap),
               sz_z = up(2 * sizeof(unsigned long long) + sizeof(int) * 3 * kNb),
               sz_s = up(sizeof(int) * (3 * (kNb + 1) + 3 * kNb + 3));
  VoxBuffers mem;
  unsigned char* block = (unsigned char*)mem.get(sz_p + 3 * sz_n + sz_r + sz_i + sz_z + sz_s);
  if (!block) return vox_fail(WT_ERR_OOM, "cannot allocate the voxel build's device buffers");
  // zeroed together: shell, votes, the two counts, the bucket counts
  uint8_t* shell = block;
  uint8_t* votes = shell + sz_n;
  unsigned long long* counts = (unsigned long long*)(votes + sz_n);
  int* bcount = (int*)(counts + 2);
  float* P = (float*)((unsigned char*)counts + sz_z);
  uint8_t* gdev = (unsigned char*)P + sz_p;
  int4* rects = (int4*)(gdev + sz_n);
  int* items = (int*)((unsigned char*)rects + sz_r);
  int* bstart = (int*)((unsigned char*)items + sz_i);
  int* cursor = bstart + 3 * (kNb + 1);
  int* total_dev = cursor + 3 * kNb;
  cudaStream_t s = nullptr;
  if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess)
    return vox_fail(WT_ERR_CUDA, "cannot create a stream");
  auto done = [&](int code, const std::string& msg) {
    cudaStreamSynchronize(s);
    cudaStreamDestroy(s);
    return code == WT_OK ? code : vox_fail(code, msg);
  };
  cudaMemcpyAsync(P, tris, sizeof(float) * 9 * (size_t)ntri, cudaMemcpyHostToDevice, s);
  cudaMemsetAsync(block, 0, 2 * sz_n + sz_z, s);
  VoxGeom g{info->nx, info->ny, info->nz, info->cell, info->inv,
            {info->min[0], info->min[1], info->min[2]}};
  k_vox_shell<<<(unsigned)((ntri * 32 + 255) / 256), 256, 0, s>>>(P, ntri, g, shell);
  AllAxes ax;
  int most = 1;
  for (int A = 0; A < 3; A++) {
    AxisGeom& x = ax.x[A];
    x.A = A; x.B = (A + 1) % 3; x.C = (A + 2) % 3;
    x.nA = dim[x.A]; x.nB = dim[x.B]; x.nC = dim[x.C];
    x.cell = info->cell;
    x.minA = info->min[x.A]; x.minB = info->min[x.B]; x.minC = info->min[x.C];
    x.nbB = x.nB < kBuckets ? x.nB : kBuckets;
    x.nbC = x.nC < kBuckets ? x.nC : kBuckets;
    x.kB = x.nbB / (x.nB * info->cell);
    x.kC = x.nbC / (x.nC * info->cell);
    auto stride = [&](int a) -> long long {
      return a == 0 ? 1 : (a == 1 ? dim[0] : (long long)dim[0] * dim[1]);
    };
    x.strideA = stride(x.A); x.strideB = stride(x.B); x.strideC = stride(x.C);
    most = std::max(most, x.nbB * x.nbC);
  }
  const dim3 tgrid((unsigned)std::min<long long>((ntri + 127) / 128, 4096), 3);
  k_vox_count<<<tgrid, 128, 0, s>>>(P, ntri, ax, rects, bcount);
  k_vox_scan<<<3, SCAN_T, 0, s>>>(bcount, ax, bstart, cursor, total_dev);
  int total[3] = {0, 0, 0};
  cudaMemcpyAsync(total, total_dev, sizeof(total), cudaMemcpyDeviceToHost, s);
  if (cudaStreamSynchronize(s) != cudaSuccess) return done(WT_ERR_CUDA, "voxel bucketing failed");
  const size_t want = (size_t)total[0] + (size_t)total[1] + (size_t)total[2];
  if (want > cap) {
    items = (int*)mem.get(sizeof(int) * want);
    if (!items) return done(WT_ERR_OOM, "cannot allocate the bucket lists");
  }
  const ListBase base{{0, total[0], (long long)total[0] + total[1]}};
  k_vox_fill<<<tgrid, 128, 0, s>>>(rects, ntri, ax, cursor, items, base);
  k_vox_order<<<dim3((most + ORDER_WARPS - 1) / ORDER_WARPS, 3), 32 * ORDER_WARPS, 0, s>>>(
      rects, ntri, ax, bstart, items, base);
  for (int A = 0; A < 3; A++) {
    const long long cols = (long long)ax.x[A].nB * ax.x[A].nC;
    k_vox_rays<<<(unsigned)((cols + RAY_WARPS - 1) / RAY_WARPS), 32 * RAY_WARPS, 0, s>>>(
        P, bstart + A * (kNb + 1), items + base.at[A], ax.x[A],
        votes);
  }
  k_vox_combine<<<(unsigned)std::min<long long>((n + 255) / 256, 148 * 4), 256, 0, s>>>(
      votes, shell, n, gdev, counts);
  unsigned long long hc[2] = {0, 0};
  cudaMemcpyAsync(hc, counts, sizeof(hc), cudaMemcpyDeviceToHost, s);
  cudaMemcpyAsync(grid, gdev, (size_t)n, cudaMemcpyDeviceToHost, s);
  if (cudaStreamSynchronize(s) != cudaSuccess || cudaGetLastError() != cudaSuccess)
    return done(WT_ERR_CUDA, "voxel build failed");
  info->solid = (int64_t)hc[0];
  info->openness = hc[0] ? (double)hc[1] / (double)hc[0] : 0.0;
  return done(WT_OK, "");
}

}  // extern "C"
