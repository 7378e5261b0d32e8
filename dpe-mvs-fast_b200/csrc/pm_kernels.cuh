// pm_kernels.cuh -- the per-view PatchMatch kernels.
//
// Kernel order and per-pixel semantics follow DPE::RunPatchMatch (DPE.cu:3130-3262).  B200
// design points: all per-call constants (cameras, relative poses, params, pointers) live in one
// argument block in device memory (one per problem of a batch); state is structure-of-arrays; view weights are packed as
// 4-bit counts (16 B per pixel instead of 32); the strong NCC's reference window is built once
// per pixel and pass and reused by every hypothesis and source view; the same-colour race of the
// edge-aware update is removed by reading candidates from a pre-pass snapshot.
#pragma once

#include "dpe_device.cuh"

namespace dpe {

__device__ __constant__ const int kDir[8][2] = {{0, -1}, {0, 1}, {-1, 0}, {1, 0}, {-1, -1}, {1, 1}, {-1, 1}, {1, -1}};

// ------------------------------------------------------------------ launch geometry
// A kernel runs either for one problem (a 2D grid over its pixels, or a 1D grid over a work list)
// or for a batch of problems in one launch (dpe_pm_run_batch): the batch's grid is the problems'
// grids laid end to end in one dimension, and each block finds its problem in a prefix table of
// block counts.
enum GridKind { kGridFull = 0, kGridHalf = 1, kGridList = 2 };
struct Launch {
  const PMArgs *args;  // [nprob] per-problem argument blocks
  const int *start;    // batched: [nprob + 1] first block of each problem; null for one problem
  int nprob;
};
// This block's problem, its coordinates in the problem's own grid, and that grid's width.
struct Blk {
  const PMArgs *a;
  int x, y, gx;
};
template <int kKind>
__device__ __forceinline__ Blk resolve(const Launch &L) {
  if (!L.start) return Blk{L.args, (int)blockIdx.x, (int)blockIdx.y, (int)gridDim.x};
  const int f = (int)blockIdx.x;
  int lo = 0, hi = L.nprob;  // the last problem whose first block is <= f
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (L.start[mid] <= f) lo = mid;
    else hi = mid;
  }
  const PMArgs *a = L.args + lo;
  const int local = f - L.start[lo];
  const int gx = kKind == kGridFull ? (a->W + 15) / 16 : kKind == kGridHalf ? (a->W + 31) / 32
                                                                            : L.start[lo + 1] - L.start[lo];
  return Blk{a, local % gx, local / gx, gx};
}

// pixel of colour `parity` ((x + y) % 2) handled by this thread of a half-height grid
__device__ __forceinline__ bool colour_pixel(const PMArgs &a, const Blk &B, int parity, int *px, int *py) {
  const int x = B.x * blockDim.x + threadIdx.x;
  const int yy = B.y * blockDim.y + threadIdx.y;
  const int y = 2 * yy + ((x + parity) & 1);
  *px = x; *py = y;
  return x < a.W && y < a.H;
}
__device__ __forceinline__ bool full_pixel(const PMArgs &a, const Blk &B, int *px, int *py) {
  *px = B.x * blockDim.x + threadIdx.x;
  *py = B.y * blockDim.y + threadIdx.y;
  return *px < a.W && *py < a.H;
}

// ------------------------------------------------------------------ setup
#ifdef DPE_CHECKED
// How the device reads the per-call block (checked builds compare it with the host's values).
__global__ void k_echo_args(const PMArgs *__restrict__ pa, long long *out) {
  out[0] = pa->W; out[1] = pa->H; out[2] = pa->N; out[3] = pa->P.strong_radius; out[4] = pa->P.strong_increment;
  out[5] = pa->P.use_edge; out[6] = pa->P.num_images; out[7] = (long long)sizeof(PMArgs);
}
#endif
__device__ __forceinline__ void pad_texel(const float *__restrict__ src, float *__restrict__ dst, int W, int H, int x, int y) {
  if (x > W || y > H) return;
  const int sx = min(max(x, 0), W - 1), sy = min(max(y, 0), H - 1);
  dst[(size_t)(y + 1) * (W + 2) + (x + 1)] = src[(size_t)sy * W + sx];
}
__global__ void k_pad_image(const float *__restrict__ src, float *__restrict__ dst, int W, int H) {
  pad_texel(src, dst, W, H, blockIdx.x * blockDim.x + threadIdx.x - 1, blockIdx.y * blockDim.y + threadIdx.y - 1);
}
// The images of a call, padded in one launch (one image per z; a launch per image was most of a small
// call's set-up).
struct PadSet {
  const float *src[kMaxImages];
  float *dst[kMaxImages];
  int W, H;
};
inline PadSet pad_set(const PMArgs &a) {
  PadSet s;
  for (int i = 0; i < kMaxImages; ++i) {
    s.src[i] = nullptr;
    s.dst[i] = i < a.N ? const_cast<float *>(a.img[i]) : nullptr;
  }
  s.W = a.W;
  s.H = a.H;
  return s;
}
__device__ __forceinline__ void pad_image_z(const PadSet &s) {
  pad_texel(s.src[blockIdx.z], s.dst[blockIdx.z], s.W, s.H, blockIdx.x * blockDim.x + threadIdx.x - 1,
            blockIdx.y * blockDim.y + threadIdx.y - 1);
}
__global__ void k_pad_images(const __grid_constant__ PadSet s) { pad_image_z(s); }

// Staged copies of the padded source images (PMArgs::quad), one image per y: word o packs the footprint
// P[o], P[o+1], P[o+pw], P[o+pw+1] as FP16 or BF16, rounded to nearest-even.  Words past the last
// footprint repeat the last texel.
template <bool kBF16>
__global__ void k_stage_quads(const float *__restrict__ pads, uint2 *__restrict__ outs, long long n, int pw) {
  const long long o = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= n) return;
  const float *pad = pads + (size_t)blockIdx.y * n;
  auto bits = [&](long long k) -> uint32_t {
    const float v = pad[k < n ? k : n - 1];
    return kBF16 ? __bfloat16_as_ushort(__float2bfloat16_rn(v)) : __half_as_ushort(__float2half_rn(v));
  };
  outs[(size_t)blockIdx.y * n + o] = make_uint2(bits(o) | bits(o + 1) << 16, bits(o + pw) | bits(o + pw + 1) << 16);
}

// Which 16-bit storage holds the n floats exactly: sets bit 0 of *flag when one is not exact in BF16 (its
// low 16 bits are not all zero; 8-bit images are exact), bit 1 when one is not in FP16 (the pyramid's
// halved levels are: averages of four 8-bit values, quarters below 256).  One atomic per block.
__global__ void k_exact16(const float *__restrict__ p, long long n, unsigned *flag) {
  unsigned b16 = 0, f16 = 0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float v = p[i];
    b16 |= __float_as_uint(v) & 0xFFFFu;
    f16 |= __float_as_uint(__half2float(__float2half_rn(v))) ^ __float_as_uint(v);
  }
  const int b = __syncthreads_or(b16 != 0 ? 1 : 0), f = __syncthreads_or(f16 != 0 ? 1 : 0);
  if ((b || f) && threadIdx.x == 0) atomicOr(flag, (b ? 1u : 0u) | (f ? 2u : 0u));
}

__global__ void k_init_state(const Launch lc, const float4 *plane_in, const uint32_t *views_in,
                             const uint8_t *weak_in, int *weak_flag) {
  const Blk B = resolve<kGridFull>(lc);
  const PMArgs &a = *B.a;
  int px, py;
  if (!full_pixel(a, B, &px, &py)) return;
  const int c = px + py * a.W;
  a.plane[c] = (a.P.state != DPE_FIRST_INIT && plane_in) ? plane_in[c] : make_float4(0, 0, 0, 0);
  a.views[c] = (a.P.state != DPE_FIRST_INIT && views_in) ? views_in[c] : 0u;
  const uint8_t wk = a.P.use_APD ? weak_in[c] : (uint8_t)DPE_STRONG;
  a.weak[c] = wk;
  weak_flag[c] = (a.P.use_APD && wk == DPE_WEAK) ? 1 : 0;
  a.rng_ctr[c] = 0u;
  a.radius[c] = a.P.strong_radius;
  a.fit_plane[c] = make_float4(0, 0, 0, 0);
  a.reliable[c] = 0;
  a.complexity[c] = 0.0f;
  a.vweight[c] = make_uint4(0, 0, 0, 0);
  a.cost[c] = 0.0f;
}

// ------------------------------------------------------------------ GenEdgeInform (DPE.cu:2487-2595)
__global__ void k_gen_edge_inform(const Launch lc) {
  const Blk B = resolve<kGridFull>(lc);
  const PMArgs &a = *B.a;
  int px, py;
  if (!full_pixel(a, B, &px, &py)) return;
  const int W = a.W, H = a.H, center = px + py * W;
  if (a.P.use_edge) {
    short2 *en = &a.edge_neigh[(size_t)center * 8];
    for (int i = 0; i < 8; ++i) {
      short2 found = make_short2(-1, -1);
      const int dx = kDir[i][0], dy = kDir[i][1];
      int nx = px + dx, ny = py + dy;
      while (nx >= 0 && nx < W && ny >= 0 && ny < H) {
        if (a.edge[nx + ny * W]) { found = make_short2(nx, ny); break; }
        nx += dx; ny += dy;
      }
      en[i] = found;
    }
    const int r = a.P.strong_radius;
    int edge_pix = 0, tot_pix = 0, bound_pix = 0;
    for (int i = -r; i <= r; ++i)
      for (int j = -r; j <= r; ++j) {
        const int nx = px + i, ny = py + j;
        if (nx < 0 || nx >= W || ny < 0 || ny >= H) continue;
        if (a.edge[ny * W + nx]) edge_pix++;
        if (a.P.use_label && a.label[ny * W + nx] == 0) bound_pix++;
        tot_pix++;
      }
    float density = 1.0f * edge_pix / tot_pix;
    if (a.P.use_label) density = cvmax(density, bound_pix / tot_pix);  // integer division (quirk Q6)
    a.complexity[center] = (float)(1.0f / (1.0f + exp(-25.0 * (density - 0.35))));
  }
  if (a.P.use_label && a.weak[center] == DPE_WEAK) {
    const int cl = a.label[center];
    if (cl > 0) {
      short2 *lb = &a.lab_bound[(size_t)a.nmap[center] * 8];
      for (int i = 0; i < 8; ++i) {
        const int dx = kDir[i][0], dy = kDir[i][1];
        int nx = px + dx, ny = py + dy, lx = -1, ly = -1;
        while (nx >= 0 && nx < W && ny >= 0 && ny < H) {
          const int nl = a.label[nx + ny * W];
          if (nl == cl) { lx = nx; ly = ny; }
          else if (nl == -1) break;
          nx += dx; ny += dy;
        }
        lb[i] = make_short2(lx, ly);
      }
    }
  }
}

// ------------------------------------------------------------------ FindNearestStrongPoint (DPE.cu:2859-2893)
__device__ __forceinline__ void find_nearest_strong_pixel(const PMArgs &a, int px, int py) {
  const int W = a.W, H = a.H, center = px + py * W;
  short2 res = make_short2(-1, -1);
  if (a.weak[center] == DPE_WEAK) {
    for (int r = 1; r <= 100; ++r) {
      bool found = false;
      for (int x = -r; x <= r && !found; ++x) {
        const int nx = px + x;
        const bool edge_col = (x == -r || x == r);
        // inner loop over y: full column on the ring's left/right edges, else only y = -r and y = r
        for (int y = -r; y <= r; y += edge_col ? 1 : 2 * r) {
          const int ny = py + y;
          if (nx < 0 || ny < 0 || nx >= W || ny >= H) continue;
          if (a.weak[nx + ny * W] == DPE_STRONG) { res = make_short2(nx, ny); found = true; break; }
        }
      }
      if (found) break;
    }
  }
  a.nearest[center] = res;
}
// One thread per pixel of a 2D grid: the tiles keep the rays of neighbouring pixels together
// (measured faster than a work list over the WEAK pixels).
__global__ void __launch_bounds__(128) k_find_nearest_strong(const Launch lc) {
  const Blk B = resolve<kGridFull>(lc);
  const PMArgs &a = *B.a;
  int px, py;
  if (!full_pixel(a, B, &px, &py)) return;
  find_nearest_strong_pixel(a, px, py);
}

// ------------------------------------------------------------------ geometry helpers for GenNeighbours
__device__ __forceinline__ uint8_t edge_at(const PMArgs &a, long idx) {
  return (idx >= 0 && idx < (long)a.W * a.H) ? a.edge[idx] : (uint8_t)0;
}

// Where the low-resolution edge map has an edge within `radius` (chessboard distance): first along the
// rows (out: 1 where none), then the columns of that.
__global__ void k_edge_clear_rows(const uint8_t *__restrict__ edge, int w, int h, int radius, uint8_t *__restrict__ out) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= w || y >= h) return;
  uint8_t clear = 1;
  for (int k = max(x - radius, 0); k <= min(x + radius, w - 1); ++k)
    if (edge[(size_t)y * w + k]) clear = 0;
  out[(size_t)y * w + x] = clear;
}
__global__ void k_edge_clear_cols(const uint8_t *__restrict__ rows, int w, int h, int radius, uint8_t *__restrict__ out) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= w || y >= h) return;
  uint8_t clear = 1;
  for (int k = max(y - radius, 0); k <= min(y + radius, h - 1); ++k)
    if (!rows[(size_t)k * w + x]) clear = 0;
  out[(size_t)y * w + x] = clear;
}

// BresenhamLine (DPE.cu:162-248); out-of-image linear indices read 0.  A point's part (its place in the
// low-resolution edge map, and whether it lies on an edge itself) is taken once per point.
struct LinePoint {  // 8 bytes: with 12, a block of GenNeighbours takes 3 KB more shared memory
  unsigned x_on;    // x in the low-resolution map << 1 | on an edge of the full-resolution map
  unsigned y_clear;  // y << 1 | no edge within max_step of it: a walk that starts here meets none
  __device__ __forceinline__ int x() const { return (int)(x_on >> 1); }
  __device__ __forceinline__ int y() const { return (int)(y_clear >> 1); }
  __device__ __forceinline__ bool on() const { return x_on & 1u; }
  __device__ __forceinline__ bool clear() const { return y_clear & 1u; }
};
struct LineMap {
  float scale_x, scale_y;
  int w, h, max_step;
};
__device__ __forceinline__ LineMap line_map(const PMArgs &a) {
  LineMap m;
  m.scale_x = 1.0f * a.lowW / (float)a.W;
  m.scale_y = 1.0f * a.lowH / (float)a.H;
  m.w = a.lowW;
  m.h = a.lowH;
  m.max_step = a.P.high_res_img ? (int)round(cvmax(m.h, m.w) / 60.0) : cvmax(m.h, m.w);
  return m;
}
__device__ __forceinline__ LinePoint line_point(const PMArgs &a, const LineMap &m, int x, int y) {
  const int lx = (int)cvmin(roundf(x * m.scale_x), (float)(m.w - 1));
  const int ly = (int)cvmin(roundf(y * m.scale_y), (float)(m.h - 1));
  const bool on = edge_at(a, (long)x + (long)y * a.W) != 0;
  // A step moves one place at most in x and in y, so max_step steps stay within that distance.  Near
  // the left and right borders a walk may pass the border by a step, where its linear index reads the
  // neighbouring row: such walks are always made.
  const bool clear = a.edge_dist && lx >= m.max_step && lx + m.max_step < m.w && a.edge_dist[lx + (size_t)ly * m.w];
  return LinePoint{(unsigned)lx << 1 | (on ? 1u : 0u), (unsigned)ly << 1 | (clear ? 1u : 0u)};
}
// One walk from (x0, y0) towards (x1, y1).  Out of line: the callers' loops stay in the instruction cache.
#ifdef __CUDA_ARCH__
__device__ __noinline__
#else
inline
#endif
bool line_walk(const uint8_t *edge_low, int w, int h, int max_step, int x0, int y0, int x1, int y1) {
  const int dx = abs(x1 - x0), sx = x0 < x1 ? 1 : -1;
  const int dy = abs(y1 - y0), sy = y0 < y1 ? 1 : -1;
  int err = (dx > dy ? dx : dy) / 2;
  int step = 0;
  bool tagx = true, tagy = true;
  const long n = (long)w * h;
  while (tagx || tagy) {
    if (x0 == x1) tagx = false;
    if (y0 == y1) tagy = false;
    const int e2 = err;
    if (e2 > -dx) { err -= dy; x0 += sx; }
    if (e2 < dy) { err += dx; y0 += sy; }
    const long idx = (long)x0 + (long)y0 * w;
    if (idx >= 0 && idx < n && edge_low[idx]) return true;
    step += 1;
    if (step >= max_step) break;
  }
  return false;
}
__device__ __forceinline__ bool line_blocked(const PMArgs &a, const LineMap &m, LinePoint A, LinePoint B) {
  if (A.on() || B.on()) return false;
  for (int pass = 0; pass < 2; ++pass) {  // from B to A, then from A to B
    const LinePoint s = pass == 0 ? B : A, t = pass == 0 ? A : B;
    if (!s.clear() && line_walk(a.edge_low, m.w, m.h, m.max_step, s.x(), s.y(), t.x(), t.y())) return true;
  }
  return false;
}
// PointinTriangle (DPE.cu:139-160)
__device__ __forceinline__ bool point_in_triangle(short2 A, short2 B, short2 C, int px, int py) {
  const float2 AB = make_float2(B.x - A.x, B.y - A.y), BC = make_float2(C.x - B.x, C.y - B.y), CA = make_float2(A.x - C.x, A.y - C.y);
  const float ab = sqrtf(AB.x * AB.x + AB.y * AB.y), bc = sqrtf(BC.x * BC.x + BC.y * BC.y), ca = sqrtf(CA.x * CA.x + CA.y * CA.y);
  if (ab <= 2 || bc <= 2 || ca <= 2) return false;
  if (!(ab + bc > ca && bc + ca > ab && ab + ca > bc)) return false;
  const float2 PA = make_float2(A.x - px, A.y - py), PB = make_float2(B.x - px, B.y - py), PC = make_float2(C.x - px, C.y - py);
  const float t1 = PA.x * PB.y - PA.y * PB.x, t2 = PB.x * PC.y - PB.y * PC.x, t3 = PC.x * PA.y - PC.y * PA.x;
  return t1 * t2 >= 0 && t1 * t3 >= 0;
}

__device__ __forceinline__ void sort_small(float *d, int n) {
  for (int i = 1; i < n; ++i) {
    const float t = d[i];
    int j;
    for (j = i; j >= 1 && t < d[j - 1]; j--) d[j] = d[j - 1];
    d[j] = t;
  }
}

// ------------------------------------------------------------------ GenNeighbours (DPE.cu:2107-2467)
// A group of kGnLanes threads works on one WEAK pixel.  The reference's thread searches 32 rays by
// random tries and then runs up to 200 RANSAC rounds, each a test of three points against up to 64;
// one thread per pixel left three quarters of a warp's lanes idle (only WEAK pixels have work) and
// kept its 2.3 KB of points in local memory.  Here the lanes split
//   * the tries of a ray: try t of a ray draws the pixel's numbers 4t..4t+3 from where the ray began
//     (the stream is counter-based), so the lanes make the next tries side by side and the first that
//     succeeds ends the ray with the counter behind it, as the sequential loop does;
//   * the label boundary's points;
//   * RANSAC rounds: round r draws numbers 3r..3r+2, and its tests (three distinct points, the triangle,
//     the edge lines, the normals, the plane) do not depend on earlier rounds; the lanes prepare the
//     next rounds side by side, which are then taken in order under the current state;
//   * the points' residuals of a round, and the ranks that replace its sorts.
// Random numbers are made ahead into shared memory, each once; lines that start where no edge is near
// are not walked (k_edge_clear_*).
// Bound by instruction issue (0.60 of the slots; about 45 k warp instructions per WEAK pixel, half of them
// the residuals, with 15 of 32 threads active).  Measured, one 1600x1200 view with 403 k WEAK pixels: 126.7 ms one thread per pixel, 43.3
// with 16 lanes, 29.1 with the numbers ahead and the walks skipped, 27.1 with points of 8 bytes; 32 lanes
// 34.4, 8 lanes do not fit the shared memory (46.8 against 43.3 before the numbers were made ahead); one 400x300
// view 2.0 -> 0.13 ms.
// Host builds of this source run it with one lane.
#ifdef __CUDA_ARCH__
#ifndef DPE_GN_LANES
#define DPE_GN_LANES 16
#endif
constexpr int kGnLanes = DPE_GN_LANES;
#else
constexpr int kGnLanes = 1;
#endif
constexpr int kGnPoints = 64;
constexpr int kGnAhead = 4 * kGnLanes;                     // numbers that one step of the group may use
constexpr int kGnDraws = 2 * kGnAhead;
struct GnGroup {
  int lane;
#ifdef __CUDA_ARCH__
  int shift;
  unsigned mask;
  __device__ __forceinline__ unsigned ballot(bool p) const {
    return (__ballot_sync(mask, p) & mask) >> shift;
  }
  template <class T> __device__ __forceinline__ T from(T v, int src) const { return __shfl_sync(mask, v, src, kGnLanes); }
  __device__ __forceinline__ void sync() const { __syncwarp(mask); }
  static __device__ __forceinline__ int first(unsigned b) { return __ffs(b) - 1; }
  static __device__ __forceinline__ int count(unsigned b) { return __popc(b); }
#else
  unsigned ballot(bool p) const { return p ? 1u : 0u; }
  template <class T> T from(T v, int) const { return v; }
  void sync() const {}
  static int first(unsigned) { return 0; }
  static int count(unsigned b) { return (int)b; }
#endif
};
// The points of one pixel.
struct GnPoints {
  union {
    short2 pts[kGnPoints];  // by ray (0-31) and label boundary (32-63), while they are found
    float res[kGnPoints];   // then the residuals of a round, or the final weights
  };
  short2 sv[kGnPoints];     // the found points in order
  float2 ray[kGnPoints];    // ((x - cx) / fx, (y - cy) / fy)
  float3 pos[kGnPoints], nrm[kGnPoints];
  LinePoint line[kGnPoints];
  uint32_t draws[kGnDraws];  // the pixel's next random numbers, number n at n % kGnDraws
};
// Per-call constants of the search.
struct GnCall {
  float cos_a, sin_a, thr;
  int shift_range;
  LineMap map;
};
__device__ __forceinline__ GnCall gn_call(const PMArgs &a) {
  GnCall k;
  const float angle = 45.0f / a.P.rotate_time;
  k.cos_a = (float)cos(angle * 3.14159265358979323846 / 180.f);
  k.sin_a = (float)sin(angle * 3.14159265358979323846 / 180.f);
  k.thr = (float)cos((angle / 2.0f) * 3.14159265358979323846 / 180.0f);
  k.shift_range = cvmax((int)(tan((angle / 2.0f) * 3.14159265358979323846 / 180.0f) * 20), 1);
  k.map = LineMap{0.f, 0.f, 0, 0, 0};
  if (a.P.use_limit) k.map = line_map(a);
  return k;
}
// Step m of a ray: 2, 4, 8, 16, 32, then 25 more each (radius = min(2 radius, radius + 25)).
__device__ __forceinline__ int gn_radius(int m) { return m < 5 ? 2 << m : 32 + 25 * (m - 4); }

// Makes the numbers ctr .. ctr + kGnAhead - 1 available in S.draws; numbers up to `end` are there.  Each is
// computed once, by one lane, however many tries turn out to be needed.
__device__ __forceinline__ void gn_fill(const PMArgs &a, const GnGroup &g, GnPoints &S, int center, uint32_t ctr,
                                        uint32_t &end) {
  if ((int)(end - ctr) >= kGnAhead) return;
  g.sync();  // the numbers being replaced have been read
#ifdef __CUDA_ARCH__
#pragma unroll 1
#endif
  for (int k = 0; k < 4; ++k) {
    const uint32_t n = end + (uint32_t)(k * kGnLanes + g.lane);
    S.draws[n % kGnDraws] = philox_word0(n, (uint32_t)center, 0x5EEDu, 0u, a.key[0], a.key[1]);
  }
  end += kGnAhead;
  g.sync();
}

__device__ __forceinline__ void gen_neighbours_pixel(const PMArgs &a, const GnCall &K, const GnGroup &g, GnPoints &S,
                                                     int px, int py) {
  const int W = a.W, H = a.H, center = px + py * W;
  const int margin = 6;
  const float depth_diff = a.P.depth_max - a.P.depth_min;
  const dpe_camera &cam = a.cam[0];
  uint32_t ctr = G(a.rng_ctr, center, (long long)W * H, 106), end = ctr;
  auto draw = [&](uint32_t n) { return S.draws[n % kGnDraws]; };
  short2 *nbs = &a.neigh[(size_t)a.nmap[center] * kNeighbours];
  for (int i = g.lane; i < kNeighbours; i += kGnLanes) nbs[i] = i == 0 ? make_short2(px, py) : make_short2(-1, -1);
  uint64_t valid = 0;
  int odi = -1, npts = 0;
  const int rt = a.P.rotate_time;
  const float ransac_thr = a.P.ransac_threshold * depth_diff;
  bool edge_limit = false;
  if (a.P.use_limit) {
    edge_limit = true;
    if (a.P.use_edge) {
      const float cv = a.complexity[center];
      gn_fill(a, g, S, center, ctr, end);
      const float rp = (float)((draw(ctr++) >> 8) + 1u) * (1.0f / 16777216.0f) - FLT_EPSILON;
      g.sync();  // every lane has read the complexity
      if (rp < cv) edge_limit = false;
      else if (g.lane == 0) a.complexity[center] = cvmax(0.99f, cv);
    }
  }
  LinePoint here{0, 0};
  if (edge_limit) here = line_point(a, K.map, px, py);
  for (int odx = -1; odx <= 1; ++odx)
    for (int ody = -1; ody <= 1; ++ody) {
      if (odx == 0 && ody == 0) continue;
      float2 od = make_float2((float)odx, (float)ody);
      normalize2(&od);
      odi++;
      for (int ri = 0; ri < rt; ++ri) {
        const int di = odi * 4 + ri;
        for (int t0 = 0;; t0 += kGnLanes) {
          gn_fill(a, g, S, center, ctr, end);
          const int t = t0 + g.lane;
          const int radius = gn_radius(t >> 2);
          const float2 tp = make_float2(px + od.x * radius, py + od.y * radius);
          const bool out = radius > 4096 || tp.x < 0 || tp.y < 0 || tp.x >= W || tp.y >= H;
          bool ok = !out;
          short2 nb = make_short2(-1, -1);
          if (ok) {
            const uint32_t c0 = ctr + 4u * (uint32_t)g.lane;
            uint32_t sgn = (draw(c0) % 2 == 0) ? 1u : 0xFFFFFFFFu;
            const int rxs = (int)((sgn * draw(c0 + 1)) % (uint32_t)K.shift_range);
            sgn = (draw(c0 + 2) % 2 == 0) ? 1u : 0xFFFFFFFFu;
            const int rys = (int)((sgn * draw(c0 + 3)) % (uint32_t)K.shift_range);
            float2 dir = make_float2(od.x * 20 + rxs, od.y * 20 + rys);
            normalize2(&dir);
            nb = make_short2((short)(int)(px + dir.x * radius), (short)(int)(py + dir.y * radius));
            ok = !(nb.x < margin || nb.y < margin || nb.x >= W - margin || nb.y >= H - margin);
            if (ok) {
              const int nbc = nb.x + nb.y * W;
              if (a.weak[nbc] != DPE_STRONG) {
                nb = a.nearest[nbc];
                ok = !(nb.x == -1 || nb.y == -1);
              }
            }
            if (ok) {
              float2 td = make_float2((float)(nb.x - px), (float)(nb.y - py));
              normalize2(&td);
              const float ca = td.x * od.x + td.y * od.y;
              ok = ca > K.thr && (!edge_limit || !line_blocked(a, K.map, here, line_point(a, K.map, nb.x, nb.y)));
            }
          }
          const unsigned hit = g.ballot(ok), over = g.ballot(out);
          if (hit) {
            const int f = g.first(hit);
            if (g.lane == f) S.pts[di] = nb;
            valid |= 1ull << di;
            npts++;
            ctr += 4u * (uint32_t)(f + 1);
            break;
          }
          if (over) {
            ctr += 4u * (uint32_t)g.first(over);
            break;
          }
          ctr += 4u * kGnLanes;
        }
        float2 rd = make_float2(od.x * K.cos_a - od.y * K.sin_a, od.x * K.sin_a + od.y * K.cos_a);
        normalize2(&rd);
        od = rd;
      }
    }
  int ext = 31;
  if (a.P.use_label && a.label[center] > 0) {
    // 2 rt points per pair of opposite directions: the first gets 2 rt - 1 steps, the second one (the
    // reference's min(1, max(2 rt - 1, ...)) is always 1: quirk Q5)
    const short2 *lb = &a.lab_bound[(size_t)a.nmap[center] * 8];
    const int total = 8 * rt;
    for (int e0 = 0; e0 < total; e0 += kGnLanes) {
      const int e = e0 + g.lane;
      bool ok = e < total;
      short2 nb = make_short2(-1, -1);
      if (ok) {
        const int k = e / (2 * rt), r = e - k * 2 * rt;
        const int i = r < 2 * rt - 1 ? 2 * k : 2 * k + 1, steps = i & 1 ? 1 : 2 * rt - 1, s = i & 1 ? 1 : r + 1;
        const short2 b = lb[i];
        float dist = 0.0f;
        if (b.x != -1 && b.y != -1) {
          const double ddx = (double)(px - b.x), ddy = (double)(py - b.y);
          dist = (float)sqrt(ddx * ddx + ddy * ddy);
          if (i >= 4) dist = (float)(dist / sqrt(2.0));
        }
        const int gap = steps + 1;
        const int step_len = cvmax(1, (int)floor(1.0 * dist / gap));
        nb = make_short2((short)(px + s * step_len * kDir[i][0]), (short)(py + s * step_len * kDir[i][1]));
        ok = !(nb.x < margin || nb.y < margin || nb.x >= W - margin || nb.y >= H - margin);
        int nbc = ok ? nb.x + nb.y * W : 0;
        if (ok && a.weak[nbc] != DPE_STRONG) {
          nb = a.nearest[nbc];
          ok = !(nb.x == -1 || nb.y == -1);
          nbc = ok ? nb.x + nb.y * W : 0;
        }
        if (ok) ok = !(a.label[nbc] != 0 && a.label[nbc] != a.label[center]);
      }
      const unsigned hit = g.ballot(ok);
      if (ok) S.pts[ext + 1 + g.count(hit & ((1u << g.lane) - 1u))] = nb;
      const int m = g.count(hit);
      for (int q = 0; q < m; ++q) valid |= 1ull << (ext + 1 + q);
      ext += m;
      npts += m;
    }
  }
  if (npts <= 3) {
    if (g.lane == 0) {
      a.reliable[center] = 0;
      a.rng_ctr[center] = ctr;
    }
    g.sync();  // the points' storage is free for the group's next pixel
    return;
  }

  // the found points in order: point i of the valid ones is lane i's, i + kGnLanes's, ...
  g.sync();
  float X[3];
  point3d(cam, px, py, a.plane[center].w, X);
  const float cwz = X[2];
  const int vc = npts;
  {
    int at = 0;
    for (int i = 0; i < kGnPoints; ++i) {
      if (!((valid >> i) & 1ull)) continue;
      if (at % kGnLanes == g.lane) {
        const short2 sp = S.pts[i];
        const float4 spl = a.plane[sp.x + sp.y * W];
        S.sv[at] = sp;
        point3d(cam, sp.x, sp.y, spl.w, X);
        S.pos[at] = make_float3(X[0], X[1], X[2]);
        const float4 n4 = normal_to_ref(cam, spl);
        S.nrm[at] = make_float3(n4.x, n4.y, n4.z);
        S.ray[at] = make_float2((sp.x - cam.K[2]) / cam.K[0], (sp.y - cam.K[5]) / cam.K[4]);
        if (edge_limit) S.line[at] = line_point(a, K.map, sp.x, sp.y);
      }
      ++at;
    }
  }
  g.sync();
  const float cfx = (px - cam.K[2]) / cam.K[0], cfy = (py - cam.K[5]) / cam.K[4];
  float4 best = make_float4(0, 0, 0, 0);
  bool has_valid = false;
  {
    int iteration = 50, max_iter = a.P.high_res_img ? 200 : 125, max_count = 3;
    float min_cost = FLT_MAX;
    float tthr = ransac_thr;
    bool has_consist = false;
    bool must_tri = (a.P.use_label && a.label[center] > 0 && edge_limit) ? false : true;
    while (iteration > 0 && max_iter > 0) {
      gn_fill(a, g, S, center, ctr, end);
      // the next rounds, one per lane: what a round's tests see, whatever the state
      bool ok = g.lane < max_iter, tri = false, nc = false, flat = true;
      float4 cr = make_float4(0, 0, 0, 0);
      if (ok) {
        const uint32_t c0 = ctr + 3u * (uint32_t)g.lane;
        const int ia = (int)(draw(c0) % (uint32_t)vc);
        const int ib = (int)(draw(c0 + 1) % (uint32_t)vc);
        const int ic = (int)(draw(c0 + 2) % (uint32_t)vc);
        ok = !(ia == ib || ib == ic || ia == ic);
        if (ok) {
          tri = point_in_triangle(S.sv[ia], S.sv[ib], S.sv[ic], px, py);
          ok = tri || !must_tri;
        }
        if (edge_limit) {
          int i = ia, j = ib;
#ifdef __CUDA_ARCH__
#pragma unroll 1
#endif
          for (int k = 0; ok && k < 3; ++k) {
            ok = !line_blocked(a, K.map, S.line[i], S.line[j]);
            i = j;
            j = k == 0 ? ic : ia;
          }
        }
        if (ok) {
          if (a.P.geom_consistency && edge_limit) {
            const float3 AN = S.nrm[ia], BN = S.nrm[ib], CN = S.nrm[ic];
            nc = !((double)(AN.x * BN.x + AN.y * BN.y + AN.z * BN.z) < 0.8660254 ||
                   (double)(AN.x * CN.x + AN.y * CN.y + AN.z * CN.z) < 0.8660254 ||
                   (double)(BN.x * CN.x + BN.y * CN.y + BN.z * CN.z) < 0.8660254);
          }
          const float3 A = S.pos[ia], B = S.pos[ib], C = S.pos[ic];
          const float3 AC = make_float3(A.x - C.x, A.y - C.y, A.z - C.z), BC = make_float3(B.x - C.x, B.y - C.y, B.z - C.z);
          cr.x = AC.y * BC.z - BC.y * AC.z;
          cr.y = -(AC.x * BC.z - BC.x * AC.z);
          cr.z = AC.x * BC.y - BC.x * AC.y;
          flat = (cr.x == 0 && cr.y == 0 && cr.z == 0) || isnan(cr.x) || isnan(cr.y) || isnan(cr.z);
          if (!flat) {
            normalize3(&cr);
            cr.w = -(cr.x * A.x + cr.y * A.y + cr.z * A.z);
          }
        }
      }
      const unsigned b_ok = g.ballot(ok), b_tri = g.ballot(tri), b_nc = g.ballot(nc), b_flat = g.ballot(flat);
      const int rounds = max_iter < kGnLanes ? max_iter : kGnLanes;
      int used = rounds;  // rounds the sequential loop runs of these
      for (unsigned todo = b_ok; todo; todo &= todo - 1) {
        const int r = g.first(todo);
        const bool r_tri = (b_tri >> r) & 1u, r_nc = (b_nc >> r) & 1u;
        if (must_tri && !r_tri) continue;
        if (a.P.geom_consistency && edge_limit && has_consist && !r_nc) continue;
        iteration--;
        const bool last = iteration == 0;
        if (last) used = r + 1;
        if (!((b_flat >> r) & 1u)) {
          const float4 pl = make_float4(g.from(cr.x, r), g.from(cr.y, r), g.from(cr.z, r), g.from(cr.w, r));
          int tcount = 0;
          bool odd = false;  // a residual that is no number
          for (int s0 = 0; s0 < vc; s0 += kGnLanes) {
            const int s = s0 + g.lane;
            bool in = false;
            if (s < vc) {
              const float fd = -pl.w / (pl.x * S.ray[s].x + pl.y * S.ray[s].y + pl.z);
              const float dist = fabsf(fd - S.pos[s].z);
              S.res[s] = dist;
              in = dist < tthr;
              if (isnan(dist)) odd = true;
            }
            tcount += g.count(g.ballot(in));
          }
          if (tcount >= 6 && tcount >= max_count) {
            const float cd = fabsf(-pl.w / (pl.x * cfx + pl.y * cfy + pl.z) - cwz);
            if (!must_tri && r_tri) must_tri = true;
            if (tcount > max_count) {
              if (!has_consist && r_nc) has_consist = true;
              best = pl; max_count = tcount; min_cost = cd; has_valid = true;
              if (tthr > (a.P.high_res_img ? 0.05 : 0.005)) {
                // the tenth smallest residual (0 with fewer than ten points)
                float r9 = 0.0f;
                g.sync();
                if (g.ballot(odd)) {  // the reference's insertion sort as it is
                  if (g.lane == 0) sort_small(S.res, vc);
                  g.sync();
                  if (vc > kNeighbours) r9 = S.res[kNeighbours];
                  if (!(tthr < r9)) {
                    tthr = (float)(r9 - 1e-6);
                    int n = 0;
                    while (n < vc && S.res[n] < tthr) ++n;
                    max_count = n;
                  }
                } else {
                  if (vc > kNeighbours)
                    for (int s0 = 0; s0 < vc; s0 += kGnLanes) {
                      const int s = s0 + g.lane;
                      int rank = -1;
                      const float v = s < vc ? S.res[s] : 0.0f;
                      if (s < vc) {
                        rank = 0;
                        for (int k = 0; k < vc; ++k) rank += S.res[k] < v || (S.res[k] == v && k < s);
                      }
                      const unsigned b = g.ballot(rank == kNeighbours);
                      if (b) r9 = g.from(v, g.first(b));
                    }
                  if (!(tthr < r9)) {
                    tthr = (float)(r9 - 1e-6);
                    max_count = 0;
                    for (int s0 = 0; s0 < vc; s0 += kGnLanes) {
                      const int s = s0 + g.lane;
                      max_count += g.count(g.ballot(s < vc && S.res[s] < tthr));
                    }
                  }
                }
                g.sync();  // the residuals are read; the next round overwrites them
              }
            } else if (cd < min_cost) {
              best = pl; min_cost = cd;
            }
          }
        }
        if (last) break;
      }
      max_iter -= used;
      ctr += 3u * (uint32_t)used;
    }
  }
  if (g.lane == 0) a.rng_ctr[center] = ctr;
  if (!has_valid) {
    if (g.lane == 0) a.reliable[center] = 0;
    g.sync();
    return;
  }
  // the points within the threshold, nearest to the plane first (equal ones in order)
  bool odd = false;
  g.sync();
  for (int s = g.lane; s < vc; s += kGnLanes) {
    const float fd = -best.w / (best.x * S.ray[s].x + best.y * S.ray[s].y + best.z);
    const float dist = fabsf(fd - S.pos[s].z);
    S.res[s] = dist >= ransac_thr ? FLT_MAX : dist;
    if (dist >= ransac_thr) S.sv[s] = make_short2(-1, -1);
    if (isnan(dist)) odd = true;
  }
  g.sync();
  if (g.ballot(odd)) {  // a weight that is no number: the reference's insertion sort as it is
    if (g.lane == 0) {
      for (int i = 1; i < vc; ++i) {
        const short2 tp = S.sv[i];
        const float tw = S.res[i];
        int j;
        for (j = i; j >= 1 && tw < S.res[j - 1]; j--) { S.sv[j] = S.sv[j - 1]; S.res[j] = S.res[j - 1]; }
        S.sv[j] = tp; S.res[j] = tw;
      }
      for (int i = 1; i < kNeighbours; ++i) nbs[i] = (i - 1 < vc) ? S.sv[i - 1] : make_short2(-1, -1);
    }
  } else {
    for (int s = g.lane; s < vc; s += kGnLanes) {
      const float v = S.res[s];
      int rank = 0;
      for (int k = 0; k < vc; ++k) rank += S.res[k] < v || (S.res[k] == v && k < s);
      if (rank < kNeighbours - 1) nbs[1 + rank] = S.sv[s];
    }
  }
  if (g.lane == 0) a.reliable[center] = 1;
  g.sync();
}
// The WEAK pixels in raster order, for k_gen_neighbours: slot nmap[c] of the list is pixel c (nmap
// counts the WEAK pixels before c).  The list lies in the buffer that the colours' lists take later.
__global__ void k_weak_list(const Launch lc) {
  const Blk B = resolve<kGridFull>(lc);
  const PMArgs &a = *B.a;
  int px, py;
  if (!full_pixel(a, B, &px, &py)) return;
  const int c = px + py * a.W;
  if (a.weak[c] == DPE_WEAK) const_cast<int *>(a.wlist[0])[a.nmap[c]] = c;
}
// On the device a grid of groups strides over the WEAK pixels' list; host builds of this source call it
// per pixel.
__global__ void __launch_bounds__(128) k_gen_neighbours(const Launch lc) {
#ifdef __CUDA_ARCH__
  const Blk B = resolve<kGridList>(lc);
  const PMArgs &a = *B.a;
  __shared__ GnPoints S[128 / kGnLanes];
  __shared__ GnCall K;
  if (threadIdx.x == 0) K = gn_call(a);
  __syncthreads();
  const int L = a.W * a.H, slot = (int)threadIdx.x / kGnLanes;
  const int count = a.nmap[L - 1] + (a.weak[L - 1] == DPE_WEAK ? 1 : 0);
  GnGroup g;
  g.lane = (int)threadIdx.x % kGnLanes;
  g.shift = ((int)threadIdx.x & 31) - g.lane;
  g.mask = (kGnLanes == 32 ? 0xFFFFFFFFu : (1u << (kGnLanes & 31)) - 1u) << g.shift;
  for (int i = B.x * (128 / kGnLanes) + slot; i < count; i += B.gx * (128 / kGnLanes)) {
    const int c = a.wlist[0][i];
    gen_neighbours_pixel(a, K, g, S[slot], c % a.W, c / a.W);
  }
#else
  const Blk B = resolve<kGridFull>(lc);
  const PMArgs &a = *B.a;
  int px, py;
  if (!full_pixel(a, B, &px, &py) || a.weak[px + py * a.W] != DPE_WEAK) return;
  GnPoints S;
  gen_neighbours_pixel(a, gn_call(a), GnGroup{0}, S, px, py);
#endif
}

__global__ void k_neighbour_update(const Launch lc) {
  const Blk B = resolve<kGridFull>(lc);
  const PMArgs &a = *B.a;
  int px, py;
  if (!full_pixel(a, B, &px, &py)) return;
  const int c = px + py * a.W;
  if (a.weak[c] == DPE_WEAK && a.reliable[c] != 1) a.weak[c] = DPE_UNKNOWN;
}

// ------------------------------------------------------------------ RandomInitialization (DPE.cu:1039-1067, 784-861)
template <int kStage>
__global__ void __launch_bounds__(128, DPE_COST_MIN_BLOCKS) k_random_init(const Launch lc) {
  const Blk B = resolve<kGridFull>(lc);
  const PMArgs &a = *B.a;
  int px, py;
  if (!full_pixel(a, B, &px, &py)) return;
  const int center = px + py * a.W;
  const dpe_camera &rc = a.cam[0];
  DPE_REF_WINDOW(rw);
  build_ref_window(a, px, py, rw, KID_RANDOM_INIT);
  const int n = a.N - 1;
  if (a.P.state == DPE_FIRST_INIT) {
    Rng rng = make_rng(a, center);
    const float depth = rng.uniform() * (a.P.depth_max - a.P.depth_min) + a.P.depth_min;
    float4 pl = random_normal(rc, px, py, rng, depth);
    pl.w = dist_to_origin(rc, px, py, depth, pl);
    a.rng_ctr[center] = rng.ctr;
    a.plane[center] = pl;
    float cv[kMaxSrc], srt[kMaxSrc];
    int valid = 0;
    ncc_all_sources<kStage, true>(a, px, py, pl, rw, cv);
    for (int i = 0; i < n; ++i) {
      const float v = cv[i];
      srt[i] = v;
      if (v < 2.0f) valid++;
    }
    sort_small(srt, n);
    uint32_t views = 0;
    float cost = 2.0f;
    const int k = min(valid, a.P.top_k);
    if (k > 0) {
      float c = 0.0f;
      for (int i = 0; i < k; ++i) c += srt[i];
      const float thr = srt[k - 1];
      for (int i = 0; i < n; ++i)
        if (cv[i] <= thr) setBit(&views, i);
      cost = c / k;
    }
    a.views[center] = views;
    a.cost[center] = cost;
  } else {
    float4 pl = normal_to_ref(rc, a.plane[center]);
    const float depth = pl.w;
    pl.w = dist_to_origin(rc, px, py, depth, pl);
    a.plane[center] = pl;
    uint32_t views = a.views[center];
    int cnt = 0;
    float cost = 0.0f;
    for (int i = 1; i < a.N; ++i) {
      if (isSet(views, i - 1)) {
        const float v = ncc_strong<kStage, true>(a, px, py, i, pl, rw);
        if (v < 2.0f) { cnt++; cost += v; }
        else unSetBit(&views, i - 1);
      }
    }
    a.views[center] = views;
    a.cost[center] = cnt == 0 ? 2.0f : cost / cnt;
  }
}

// ------------------------------------------------------------------ shared pieces of the propagation kernels
// Multi-hypothesis joint view selection (DPE.cu:1551-1619 / 1714-1783).
// cost_array: 8 candidate rows of per-source costs, `stride` floats apart.
__device__ __forceinline__ float sample_views(const PMArgs &a, Rng &rng, int iter, const float *cost_array, int stride,
                                              const float *priors, uint8_t *vw, uint32_t *temp_sel, float *probs) {
  const int n = a.N - 1;
  for (int i = 0; i < 32; ++i) vw[i] = 0;
  const float thr = (float)(0.8 * (double)dpe_expf((float)(iter * iter) / (-90.0f)));
  const float base = dpe_expf(thr * thr / (-0.32f));
  for (int i = 0; i < n; ++i) {
    float count = 0;
    int count_false = 0;
    float tmpw = 0;
    for (int j = 0; j < 8; ++j) {
      const float v = cost_array[j * stride + i];
      if (v < thr) { tmpw += dpe_expf(v * v / (-0.18f)); count++; }
      if (v > 1.2f) count_false++;
    }
    float p = 0.0f;
    if (count > 2 && count_false < 3) p = tmpw / count;
    else if (count_false < 3) p = base;
    probs[i] = p * priors[i];
  }
  float sum = 0.0f;
  for (int i = 0; i < n; ++i) sum += probs[i];
  const float inv = 1.0f / sum;
  float cum = 0.0f;
  for (int i = 0; i < n; ++i) { cum += probs[i] * inv; probs[i] = cum; }
  for (int s = 0; s < 15; ++s) {
    const float r = rng.uniform() - FLT_EPSILON;
    for (int id = 0; id < n; ++id)
      if (probs[id] > r) { vw[id] += 1; break; }
  }
  uint32_t sel = 0;
  float wn = 0;
  for (int i = 0; i < n; ++i)
    if (vw[i] > 0) { setBit(&sel, i); wn += vw[i]; }
  *temp_sel = sel;
  return wn;
}

__device__ __forceinline__ int find_min_cost_index(const float *c, int n) {
  float m = c[0];
  int idx = 0;
  for (int i = 1; i < n; ++i)
    if (c[i] <= m) { m = c[i]; idx = i; }
  return idx;
}

// ------------------------------------------------------------------ Gauss-Newton plane hypothesis
// The differentiation form's refinement step (no reference counterpart; dpe_options::gn_refine).
// Around the current plane (n, depth) it takes the cost of each sampled source j and its gradient
// (ncc_strong_adjoint) in the local parameters theta = (d depth, d a1, d a2), the normal tilted
// within its tangent plane (n' = normalize(n + a1 e1 + a2 e2)), and solves the damped normal
// equations  (J^T V J + lambda diag(J^T V J)) theta = -J^T V c  (V = the view weights).  The
// resulting plane is a hypothesis like the random ones: kept only when its cost is lower and its
// depth lies in range.  It draws no random numbers, so the rest of the update is unchanged.
struct GnFrame {
  float ray0, ray1, nr, d0;  // the pixel's ray (z = 1), n . ray, the current depth
  float e1x, e1y, e1z, e2x, e2y, e2z, e1r, e2r;  // tangent basis of n, e . ray
};
__device__ __forceinline__ GnFrame gn_frame(const dpe_camera &rc, int px, int py, float4 p, float d0) {
  GnFrame f;
  f.ray0 = ((float)px - rc.K[2]) / rc.K[0];
  f.ray1 = ((float)py - rc.K[5]) / rc.K[4];
  f.nr = p.x * f.ray0 + p.y * f.ray1 + p.z;
  f.d0 = d0;
  if (fabsf(p.x) < 0.9f) { f.e1x = 0.0f; f.e1y = p.z; f.e1z = -p.y; }  // n x (1, 0, 0)
  else { f.e1x = -p.z; f.e1y = 0.0f; f.e1z = p.x; }                    // n x (0, 1, 0)
  const float e1n = 1.0f / sqrtf(f.e1x * f.e1x + f.e1y * f.e1y + f.e1z * f.e1z);
  f.e1x *= e1n; f.e1y *= e1n; f.e1z *= e1n;
  f.e2x = p.y * f.e1z - p.z * f.e1y; f.e2y = p.z * f.e1x - p.x * f.e1z; f.e2z = p.x * f.e1y - p.y * f.e1x;
  f.e1r = f.e1x * f.ray0 + f.e1y * f.ray1 + f.e1z;
  f.e2r = f.e2x * f.ray0 + f.e2y * f.ray1 + f.e2z;
  return f;
}
// Adds source j's terms (view weight v) to the normal equations m = (A00 A01 A02 A11 A12 A22 b0 b1 b2).
template <class RW>
__device__ __forceinline__ void gn_accumulate(const PMArgs &a, int px, int py, const RW &rw, float4 p,
                                              const GnFrame &f, int j, float v, float m[9]) {
  float g[4];
  const float c = ncc_strong_adjoint(a, px, py, j + 1, p, rw, g, nullptr);
  if (!(c > 0.0f && c < 2.0f)) return;
  // w = -depth (n . ray): dC/ddepth = g_w (-(n . ray)); tilting n moves w by -depth (e . ray)
  const float jd = -g[3] * f.nr;
  const float j1 = g[0] * f.e1x + g[1] * f.e1y + g[2] * f.e1z - g[3] * f.d0 * f.e1r;
  const float j2 = g[0] * f.e2x + g[1] * f.e2y + g[2] * f.e2z - g[3] * f.d0 * f.e2r;
  m[0] += v * jd * jd; m[1] += v * jd * j1; m[2] += v * jd * j2;
  m[3] += v * j1 * j1; m[4] += v * j1 * j2; m[5] += v * j2 * j2;
  m[6] -= v * jd * c; m[7] -= v * j1 * c; m[8] -= v * j2 * c;
}
// Solves the damped normal equations m around plane p; false when singular, when the new plane
// does not face the camera, or when its depth is out of range.  *t receives the new plane.
__device__ __forceinline__ bool gn_solve(const PMArgs &a, int px, int py, float4 p, const GnFrame &f,
                                         const float m[9], float4 *t) {
  const float lambda = 0.1f;
  const float A00 = m[0] * (1.0f + lambda), A01 = m[1], A02 = m[2];
  const float A11 = m[3] * (1.0f + lambda), A12 = m[4], A22 = m[5] * (1.0f + lambda);
  const float b0 = m[6], b1 = m[7], b2 = m[8];
  const float c00 = A11 * A22 - A12 * A12, c01 = A02 * A12 - A01 * A22, c02 = A01 * A12 - A02 * A11;
  const float det = A00 * c00 + A01 * c01 + A02 * c02;
  if (!(fabsf(det) > 1e-30f) || !isfinite(det)) return false;
  const float c11 = A00 * A22 - A02 * A02, c12 = A01 * A02 - A00 * A12, c22 = A00 * A11 - A01 * A01;
  const float inv = 1.0f / det;
  const float td = (c00 * b0 + c01 * b1 + c02 * b2) * inv;
  const float t1 = (c01 * b0 + c11 * b1 + c12 * b2) * inv;
  const float t2 = (c02 * b0 + c12 * b1 + c22 * b2) * inv;
  float nx = p.x + t1 * f.e1x + t2 * f.e2x, ny = p.y + t1 * f.e1y + t2 * f.e2y, nz = p.z + t1 * f.e1z + t2 * f.e2z;
  const float nn = 1.0f / sqrtf(nx * nx + ny * ny + nz * nz);
  nx *= nn; ny *= nn; nz *= nn;
  if (!(nx * f.ray0 + ny * f.ray1 + nz < 0.0f)) return false;  // the plane must face the camera
  const float dn = f.d0 + td;
  if (!(dn >= a.P.depth_min && dn <= a.P.depth_max)) return false;
  *t = make_float4(nx, ny, nz, 0.0f);
  t->w = dist_to_origin(a.cam[0], px, py, dn, *t);
  return true;
}

// ------------------------------------------------------------------ strong update (DPE.cu:1218-1670, 1069-1122)
// Block-cooperative: a block holds kCoopPix pixels of one colour (consecutive x on one row of the
// half grid) and kCoopLanes threads per pixel.  The pixel's reference window and its candidate
// cost matrix live once in shared memory.  The four pixels of a warp put the (plane, source) pairs
// they need a cost for into one list, and the warp's 32 threads evaluate the list side by side; the
// threads of a pixel split its other work, and one thread per pixel takes every decision in the
// reference's order, so the random draws and the order of each weighted sum are those of one thread
// doing it all.  Everything a pixel needs stays within its warp, so phases end with a warp barrier; the
// block barriers around an evaluation only keep the block's warps in the same code, which they fetch
// together (without them the kernel waits on instruction fetch: 62.4 against 55.8 ms at that time).
//
// What bounds it: instruction issue and register reads of the tap loop (strong_tap2) and, with
// several inlined copies of it, instruction fetch.  Hence one evaluation loop (strong_eval) that
// every stage runs its list through, and lists without what cannot matter:
//   * candidates with the same plane share one cost row (the cost depends on the plane only), and the
//     current plane takes the row of a candidate that equals it;
//   * a refinement plane whose depth is out of range is never taken, and one whose sum over its first
//     sources already reaches the cost to beat neither: costs are not negative and rounded sums and
//     quotients of such terms are monotone, so the full sum cannot fall below it.
// Both leave every decision, and so every result bit, as it was.
// Six launches on a 1600x1200 view: first call with 10 sources 69.1 -> 50.2 ms, geometric call with 9
// and a fifth of the pixels WEAK 77.6 -> 51.0 ms; on a 801x603 level image 19.9 -> 12.1 ms.
//
// Stages (each: evaluate the list, then the work that follows from the costs and the next list):
//   start  window taps, candidate search, the list of distinct candidates x all sources
//   0      edge form's choice between the two searches; view-selection probabilities, the 15 draws,
//          the sampled sources; candidates' weighted costs; list: current plane x sampled sources
//   1      best candidate, acceptance, refinement planes; list: the planes x their heaviest sources
//   2      list: the planes still in play x their other sampled sources
//   3      refinement decisions, outputs
//   3, 4   with the Gauss-Newton hypothesis only: its normal equations (shuffle sums) and list; its
//          decision and the outputs
constexpr int kCoopPix = 16, kCoopLanes = 8, kCoopThreads = kCoopPix * kCoopLanes;
constexpr int kWarpPix = 32 / kCoopLanes;  // pixels of one warp
constexpr int kRows = 17;                  // cost rows of a pixel: 16 candidates, the current plane
constexpr int kCurRow = 16;
constexpr int kListCap = kWarpPix * 5 * 15;  // longest list: 5 planes x 15 sources per pixel

// A plane as the cost evaluation takes it (PlaneProj without the products that its normal gives).
struct HypProj {
  double iw, q;
  float nx, ny;
};

// Decision state of one pixel, in shared memory.
struct CoopPixel {
  float4 win[kWinPairs];  // the taps in pairs (win_store)
  HypProj rec[kRows];     // candidates (0-7 the first search, 8-15 the edge form's second), current
  union {
    float rc[kWinTaps];   // until the window sums: w (r - c)^2 per tap
    struct {
      float probs[kMaxSrc];
      float pad;
    };                    // view selection
    float4 hyp[5];        // from the refinement planes on
  };
  float u[16];            // the uniform draws of the view sampling; then the refinement planes' costs
  float ahead[16];        // the uniform draws after them (the refinement's)
  float fc[8];            // the candidates' weighted costs
  float4 pl_cur, pl_now, n_rand, n_pert;
  float center, inv_wsum, mean_r, var_r;
  float wn, cost_now, cost_written, depth_now, depth_rand, depth_pert;
  int pos[kCurRow];
  uint32_t views_new, temp_sel, rng_ctr;
  int cnt;                 // entries of this pixel in its warp's list
  alignas(4) uint8_t uniq[kCurRow];   // candidate h has a cost row of its own
  uint8_t dup[kRows];      // the row that holds candidate h's costs (itself, or an equal plane's)
  uint8_t row[8];          // the row of the candidate kept for direction d
  uint8_t flag[8];         // direction d has a candidate
  uint8_t valid[kCurRow];  // the search found candidate h
  uint8_t samp[16];        // the source each draw selects (255: none)
  uint8_t vw[32];
  uint8_t act[32];         // the sampled sources (source index - 1), ascending
  uint8_t alive[8];        // refinement plane h can still be taken
  uint8_t first, second;   // positions in act of the two heaviest sources
  uint8_t na, live;
};
// Shared bytes of one block: the pixels' states, the warps' lists, the n = N - 1 sources, then per pixel
// kRows cost rows of n floats.
__host__ __device__ inline size_t coop_smem_bytes(int n) {
  return sizeof(CoopPixel) * kCoopPix + sizeof(uint16_t) * kListCap * (kCoopThreads / 32) + sizeof(SrcConst) * n +
         sizeof(float) * (size_t)kCoopPix * kRows * n;
}
static_assert(sizeof(uint16_t) * kListCap * (kCoopThreads / 32) % 8 == 0, "the sources are 8-byte aligned");

// A pixel's stream whose next 16 numbers are at hand; a long rejection in random_normal goes on from the
// generator.
struct AheadRng {
  Rng next;
  const float *u;
  int used;
  __device__ __forceinline__ float uniform() {
    if (used < 16) {
      next.ctr++;
      return u[used++];
    }
    return next.uniform();
  }
};

struct CoopCtx {
  const PMArgs *a;
  int slot, lane, px, py, center, n, parity;
  bool live;  // a pixel of this colour inside the image, not WEAK
  CoopPixel *P;      // this thread's pixel
  CoopPixel *W0;     // the first pixel of this thread's warp
  float *cost;       // this pixel's rows
  float *cost0;      // the rows of the warp's first pixel
  uint16_t *list;    // the warp's list: pixel of the warp | row << 2 | source << 7
  SrcConst *src;     // the sources
};

__device__ __forceinline__ CoopCtx coop_ctx(const Launch &lc, int parity, void *smem) {
  const Blk B = resolve<kGridFull>(lc);  // kGridFull's block-row width, (W + 15) / 16, is ours too
  const PMArgs &a = *B.a;
  CoopCtx c;
  c.a = B.a;
  c.parity = parity;
  c.slot = (int)threadIdx.x / kCoopLanes;
  c.lane = (int)threadIdx.x % kCoopLanes;
  c.n = a.N - 1;
  c.px = B.x * kCoopPix + c.slot;
  c.py = 2 * B.y + ((c.px + parity) & 1);
  c.center = c.py * a.W + c.px;
  c.live = c.px < a.W && c.py < a.H;
  if (c.live) c.live = G(a.weak, c.center, (long long)a.W * a.H, 201) != DPE_WEAK;
  CoopPixel *base = static_cast<CoopPixel *>(smem);
  const int warp = (int)threadIdx.x / 32;
  c.P = base + c.slot;
  c.W0 = base + warp * kWarpPix;
  uint16_t *lists = reinterpret_cast<uint16_t *>(base + kCoopPix);
  c.list = lists + (size_t)warp * kListCap;
  c.src = reinterpret_cast<SrcConst *>(lists + (size_t)kListCap * (kCoopThreads / 32));
  float *rows = reinterpret_cast<float *>(c.src + c.n);
  c.cost = rows + (size_t)c.slot * kRows * c.n;
  c.cost0 = rows + (size_t)warp * kWarpPix * kRows * c.n;
  return c;
}
__device__ __forceinline__ void coop_rec(const CoopCtx &c, int h, float4 pl) {
  const PlaneProj p = plane_projection(*c.a, pl, c.px, c.py);
  HypProj &r = c.P->rec[h];
  r.iw = p.iw; r.q = p.q; r.nx = pl.x; r.ny = pl.y;
}
// Entries of the warp's list before this pixel's.
__device__ __forceinline__ int coop_offset(const CoopCtx &c) {
  int o = 0;
  for (int k = 0; k < kWarpPix - 1; ++k)
    if (k < (c.slot & (kWarpPix - 1))) o += c.W0[k].cnt;
  return o;
}
__device__ __forceinline__ uint16_t coop_entry(const CoopCtx &c, int row, int src) {
  return (uint16_t)((c.slot & (kWarpPix - 1)) | row << 2 | src << 7);
}

#ifdef __CUDA_ARCH__
#define DPE_WARP_BARRIER() __syncwarp()
#else
#define DPE_WARP_BARRIER() ((void)0)
#endif
// Evaluates the warp's list: costs of every entry's plane against its source, and against the ns - 1
// that follow it (stage 0: all sources), sources in the outer order so that the threads of a round
// read one source image.
template <int kStage>
__device__ __forceinline__ void strong_eval(const CoopCtx &c, int ns) {
  const PMArgs &a = *c.a;
  int T = 0;
  for (int k = 0; k < kWarpPix; ++k) T += c.W0[k].cnt;
  if (T == 0) return;
  const int px0 = c.px - (c.slot & (kWarpPix - 1)), row2 = c.py - ((c.px + c.parity) & 1);
  int r = (int)threadIdx.x & 31, j0 = 0;
  // (joining the warp for each round, as lr_eval does, costs more here than the pieces it avoids)
  while (true) {
    while (r >= T) { r -= T; ++j0; }
    if (j0 >= ns) break;
    const unsigned e = c.list[r];
    const int k = e & (kWarpPix - 1), h = (e >> 2) & 31, j = (int)(e >> 7) + j0;
    const int px = px0 + k, py = row2 + ((px + c.parity) & 1);
    const CoopPixel &Q = c.W0[k];
    const HypProj &hp = Q.rec[h];
    const PlaneProj pp{(double)hp.nx * a.dm[0], (double)hp.ny * a.dm[1], hp.iw, hp.q};
    const SmemWindow rw{Q.win, Q.center, Q.inv_wsum, Q.mean_r, Q.var_r,
                        a.counters ? a.counters + 2 * KID_STRONG_UPDATE : nullptr};
    c.cost0[((size_t)k * kRows + h) * c.n + j] = ncc_strong_proj<kStage, true>(a, px, py, c.src[j], pp, rw);
    r += 32;
  }
}

// The sources; window taps of build_ref_window, split over the lanes.
template <int kStage>
__device__ __forceinline__ void strong_taps(const CoopCtx &c) {
  load_sources<kStage>(*c.a, c.src, (int)threadIdx.x, kCoopThreads);  // read after the first block barrier
  if (!c.live) return;
  const PMArgs &a = *c.a;
  const int r = a.P.strong_radius, inc = a.P.strong_increment, side = 2 * r / inc + 1;
  const float center = texel(a, 0, c.px, c.py);
  for (int k = c.lane; k < side * side; k += kCoopLanes) {
    const int i = -r + (k / side) * inc, j = -r + (k % side) * inc;
    const float rp = texel(a, 0, c.px + i, c.py + j);
    const float w = bilateral_weight((float)i, (float)j, rp, center, a.P.sigma_spatial, a.P.sigma_color);
    const float rc = rp - center, wr = w * rc;
    win_store(c.P->win, k, w, wr);
    c.P->rc[k] = wr * rc;
  }
  if (c.lane == 0) c.P->center = center;
}

// Candidate search of the non-edge propagation (8 slots: 0 up_near, 1 up_far, 2 down_near,
// 3 down_far, 4 left_near, 5 left_far, 6 right_near, 7 right_far), slot d only.
__device__ __forceinline__ int strong_search_plain(const PMArgs &a, int px, int py, int d) {
  const int W = a.W, H = a.H;
  [[maybe_unused]] const long long L = (long long)W * H;
  const int f = d >> 1;
  const int dx = f == 2 ? -1 : f == 3 ? 1 : 0, dy = f == 0 ? -1 : f == 1 ? 1 : 0;
  // far: every second pixel from distance 3 on; near: the pixel one step away, then the pairs k to either
  // side at distance 1 + k, k = 1..3 (before the other side first).  A pixel outside the image ends the
  // far ones and skips the near one.
  const bool far = d & 1;
  float m = 0.0f;
  int mp = -1;
#ifdef __CUDA_ARCH__
#pragma unroll 1
#endif
  for (int i = 0; i < (far ? 11 : 7); ++i) {
    const int k = (i + 1) >> 1;
    const int along = far ? 3 + 2 * i : 1 + k, side = far ? 0 : i & 1 ? -k : k;
    const int x = px + dx * along + (dy != 0 ? side : 0), y = py + dy * along + (dx != 0 ? side : 0);
    const bool in = x >= 0 && x < W && y >= 0 && y < H;
    if (i == 0 && !in) return -1;
    if (!in) continue;
    const int t = y * W + x;
    const float ct = G(a.cost, t, L, 207);
    if (i == 0 || ct < m) { m = ct; mp = t; }
  }
  return mp;
}

// The edge-aware propagation's first search for direction d: steps along d up to the stored edge
// distance (DPE.cu:1262-1301).  Returns the position or -1.
__device__ __forceinline__ int strong_search_edge(const PMArgs &a, int px, int py, int center, int d, int iter) {
  const int W = a.W, H = a.H;
  [[maybe_unused]] const long long L = (long long)W * H;
  const float *cand_cost = a.cost_snap;
  const short2 e = G(a.edge_neigh, (long long)center * 8 + d, L * 8, 202);
  const float max_edge_dist = cvmax(H, W) / 30.0f;
  const int min_step = 2;
  const bool on_edge = G(a.edge, center, L, 203) != 0;
  const int dx = kDir[d][0], dy = kDir[d][1];
  const int sx = cvmax(1, 5 - 2 * iter) * dx, sy = cvmax(1, 5 - 2 * iter) * dy;
  const double ex = (double)(e.x - px), ey = (double)(e.y - py);
  float dist = (float)sqrt(ex * ex + ey * ey);
  if (d >= 4) dist = (float)(dist / sqrt(2.0));
  if (on_edge) dist = 11 * min_step;
  else if (e.x == -1 || e.y == -1 || dist > max_edge_dist) {
    dist = max_edge_dist;
    if (d >= 4) dist = (float)(dist / sqrt(2.0));
  }
  const int step_num = cvmin(cvmax(11, (int)(1.0f * dist / min_step)), 22);
  int step_len = cvmax((int)(1.0f * dist / step_num), min_step);
  if (d < 4 && step_len % 2 == 1) step_len -= 1;
  float mc = FLT_MAX;
  int mp = -1;
  int fx = 0, fy = 0;
  if (d > 4) { if (d % 2) fx = dx; else fy = dy; }
  for (int s = 0; s < step_num; ++s) {
    const int tx = px + sx + s * step_len * dx + fx, ty = py + sy + s * step_len * dy + fy;
    if (!(tx >= 0 && ty >= 0 && tx < W && ty < H)) continue;
    const int tc = tx + ty * W;
    const float cc = G(cand_cost, tc, L, 204);
    if (mc > cc) { mp = tc; mc = cc; }
  }
  return mc < FLT_MAX ? mp : -1;
}

// The edge form's second search for direction d: 11 steps of two pixels (DPE.cu:1302-1333).
__device__ __forceinline__ int strong_search_edge2(const PMArgs &a, int px, int py, int d, int iter) {
  [[maybe_unused]] const long long L = (long long)a.W * a.H;
  const int dx = kDir[d][0], dy = kDir[d][1], min_step = 2;
  const int sx = cvmax(1, 5 - 2 * iter) * dx, sy = cvmax(1, 5 - 2 * iter) * dy;
  float mc = FLT_MAX;
  int mp = -1;
  int fx = 0, fy = 0;
  if (d > 4) { if (d % 2) fx = dx; else fy = dy; }
  for (int s = 0; s < 11; ++s) {
    const int tx = px + sx + s * min_step * dx + fx, ty = py + sy + s * min_step * dy + fy;
    if (!(tx >= 0 && ty >= 0 && tx < a.W && ty < a.H)) continue;
    const int tc = tx + ty * a.W;
    const float cc = G(a.cost_snap, tc, L, 204);
    if (mc > cc) { mp = tc; mc = cc; }
  }
  return mc < FLT_MAX ? mp : -1;
}

// Candidate search (lane d: direction d) and the planes' projections; window sums in tap order, as
// build_ref_window accumulates them (lane 0).
__device__ __forceinline__ void strong_search(const CoopCtx &c, int iter) {
  if (!c.live) return;
  const PMArgs &a = *c.a;
  [[maybe_unused]] const long long L = (long long)a.W * a.H;
  CoopPixel &P = *c.P;
  const int d = c.lane;
  int pos, pos2 = -1;
  if (a.P.use_edge) {
    pos = strong_search_edge(a, c.px, c.py, c.center, d, iter);
    if (G(a.edge, c.center, L, 203) == 0) pos2 = strong_search_edge2(a, c.px, c.py, d, iter);
  } else {
    pos = strong_search_plain(a, c.px, c.py, d);
  }
  P.pos[d] = pos;
  P.pos[8 + d] = pos2;
  P.valid[d] = pos >= 0 ? 1 : 0;
  P.valid[8 + d] = pos2 >= 0 ? 1 : 0;
  const float4 *planes = a.P.use_edge ? a.plane_snap : a.plane;
  if (pos >= 0) coop_rec(c, d, G(planes, pos, L, 205));
  if (pos2 >= 0 && pos2 != pos) coop_rec(c, 8 + d, G(planes, pos2, L, 205));
  else if (pos2 >= 0) P.rec[8 + d] = P.rec[d];
  if (d == 0) {
    const float4 pl = G(a.plane, c.center, L, 212);
    P.pl_cur = pl;
    coop_rec(c, kCurRow, pl);
    const int r = a.P.strong_radius, inc = a.P.strong_increment, side = 2 * r / inc + 1;
    float sw = 0.f, swr = 0.f, swrr = 0.f;
    for (int k = 0; k < side * side; ++k) {
      const float2 t = win_tap(P.win, k);
      sw += t.x; swr += t.y; swrr += P.rc[k];
    }
    P.inv_wsum = 1.0f / sw;
    P.mean_r = swr * P.inv_wsum;
    P.var_r = swrr * P.inv_wsum - P.mean_r * P.mean_r;
  }
}

__device__ __forceinline__ bool same_rec(const HypProj &x, const HypProj &y) {
  // by value: +0 and -0 give the same costs, and a NaN plane keeps its own row
  return x.nx == y.nx && x.ny == y.ny && x.iw == y.iw && x.q == y.q;
}
// Which planes need a row of their own: lane d looks at candidates d and 8 + d, lane 0 at the current
// plane too.
__device__ __forceinline__ void strong_distinct(const CoopCtx &c) {
  CoopPixel &P = *c.P;
  if (c.lane == 0) P.live = c.live ? 1 : 0;
  if (!c.live) return;
  const int last = c.a->P.use_edge ? kCurRow : 8;
  for (int h = c.lane; h < last; h += 8) {
    int to = h;
    if (P.valid[h])
      for (int e = 0; e < h; ++e)
        if (P.valid[e] && same_rec(P.rec[e], P.rec[h])) { to = e; break; }
    P.dup[h] = (uint8_t)to;
    P.uniq[h] = P.valid[h] && to == h ? 1 : 0;
  }
  if (c.lane == kCoopLanes - 1) {
    int to = kCurRow;
    for (int e = 0; e < last; ++e)
      if (P.valid[e] && same_rec(P.rec[e], P.rec[kCurRow])) { to = e; break; }
    P.dup[kCurRow] = (uint8_t)to;
  }
}
// Sum of the bytes 0 .. h - 1 of a pixel's uniq flags.
__device__ __forceinline__ int uniq_before(const CoopPixel &P, int h) {
  int m = 0;
  for (int w = 0; w < kCurRow / 4 && 4 * w < h; ++w) {
    uint32_t v = reinterpret_cast<const uint32_t *>(P.uniq)[w];
    if (h < 4 * w + 4) v &= (1u << (8 * (h - 4 * w))) - 1u;
    m += (int)((v * 0x01010101u) >> 24);
  }
  return m;
}
__device__ __forceinline__ void strong_list(const CoopCtx &c) {
  const int last = c.a->P.use_edge ? kCurRow : 8;
  int off = 0, mine = 0;
  for (int k = 0; k < kWarpPix; ++k) {
    const int m = c.W0[k].live ? uniq_before(c.W0[k], last) : 0;
    if (k < (c.slot & (kWarpPix - 1))) off += m;
    if (k == (c.slot & (kWarpPix - 1))) mine = m;
  }
  if (c.lane == 0) c.P->cnt = mine;
  if (!c.live) return;
  const CoopPixel &P = *c.P;
  for (int h = c.lane; h < last; h += 8)
    if (P.uniq[h]) c.list[off + uniq_before(P, h)] = coop_entry(c, h, 0);
}

// The candidate kept for direction d and its cost row (lane d): the edge form takes the second search
// where it has more good sources, or as many and fewer bad ones (DPE.cu:1334-1366).  A direction
// without a candidate keeps the initial costs: 0, and 2 for the first direction's first source,
// because `= {2.0f}` initialises only the first element (quirk Q2).
__device__ __forceinline__ void strong_choose(const CoopCtx &c, int iter) {
  if (!c.live) return;
  CoopPixel &P = *c.P;
  const int n = c.n, d = c.lane;
  const bool v1 = P.valid[d] != 0, v2 = P.valid[8 + d] != 0;
  int take = d;
  if (v2) {
    take = 8 + d;
    if (v1) {
      const float good_thr = 0.8f * dpe_expf((float)(iter * iter) / (-90.0f));
      const float *r0 = c.cost + P.dup[d] * n, *r1 = c.cost + P.dup[8 + d] * n;
      int g0 = 0, g1 = 0, b0 = 0, b1 = 0;
      for (int j = 0; j < n; ++j) {
        if (r0[j] < good_thr) g0++;
        if (r0[j] > 1.2f) b0++;
        if (r1[j] < good_thr) g1++;
        if (r1[j] > 1.2f) b1++;
      }
      if (!(g1 > g0 || (g1 == g0 && b1 < b0))) take = d;
    }
  }
  P.flag[d] = v1 || v2 ? 1 : 0;
  P.row[d] = v1 || v2 ? P.dup[take] : (uint8_t)d;
  P.pos[d] = v1 || v2 ? P.pos[take] : -1;
  if (!(v1 || v2)) {
    float *row = c.cost + d * n;
    for (int j = 0; j < n; ++j) row[j] = 0.0f;
    if (d == 0) row[0] = 2.0f;
  }
}

// The view-selection probability of each source (sample_views' first loop, with the priors of
// DPE.cu:1551-1563), lane j taking sources j, j + 8, ...; and the 15 uniform draws of the sampling and the
// 16 after them (counter-based, so draw s is the pixel's counter + s), split over the lanes.
__device__ __forceinline__ void strong_probs(const CoopCtx &c, int iter) {
  if (!c.live) return;
  const PMArgs &a = *c.a;
  const int W = a.W, n = c.n, center = c.center;
  [[maybe_unused]] const long long L = (long long)W * a.H;
  CoopPixel &P = *c.P;
  const uint32_t ctr0 = G(a.rng_ctr, center, L, 106);
#ifdef __CUDA_ARCH__
#pragma unroll 1
#endif
  for (int s = c.lane; s < 15 + 16; s += kCoopLanes) {
    Rng r{a.key[0], a.key[1], (uint32_t)center, ctr0 + (uint32_t)s};
    (s < 15 ? P.u[s] : P.ahead[s - 15]) = r.uniform();
  }
  const long total = (long)W * a.H;
  const long nbr[4] = {(long)center - W, (long)center + W, (long)center - 1, (long)center + 1};
  uint32_t sv[4];
  for (int i = 0; i < 4; ++i)
    sv[i] = (P.flag[2 * i] && nbr[i] >= 0 && nbr[i] < total) ? G(a.views, nbr[i], L, 211) : 0u;
  const float thr = (float)(0.8 * (double)dpe_expf((float)(iter * iter) / (-90.0f)));
  const float base = dpe_expf(thr * thr / (-0.32f));
  for (int j = c.lane; j < n; j += kCoopLanes) {
    float prior = 0.0f;
    for (int i = 0; i < 4; ++i)
      if (P.flag[2 * i]) prior += isSet(sv[i], j) == 1 ? 0.9f : 0.1f;
    float count = 0;
    int count_false = 0;
    float tmpw = 0;
    for (int d = 0; d < 8; ++d) {
      const float v = c.cost[P.row[d] * n + j];
      if (v < thr) { tmpw += dpe_expf(v * v / (-0.18f)); count++; }
      if (v > 1.2f) count_false++;
    }
    float p = 0.0f;
    if (count > 2 && count_false < 3) p = tmpw / count;
    else if (count_false < 3) p = base;
    P.probs[j] = p * prior;
  }
  if (c.lane == 0) P.rng_ctr = ctr0 + 15;
}
// The rest of sample_views: normalised cumulative probabilities (lane 0), the source of each draw (the
// lanes split the draws), the counts per source (the lanes split the sources), the list of sampled
// sources and the weight sum (lane 0).
__device__ __forceinline__ void strong_cumulate(const CoopCtx &c) {
  if (!c.live || c.lane != 0) return;
  const int n = c.n;
  CoopPixel &P = *c.P;
  float sum = 0.0f;
  for (int i = 0; i < n; ++i) sum += P.probs[i];
  const float inv = 1.0f / sum;
  float cum = 0.0f;
  for (int i = 0; i < n; ++i) { cum += P.probs[i] * inv; P.probs[i] = cum; }
}
__device__ __forceinline__ void strong_sample(const CoopCtx &c) {
  if (!c.live) return;
  CoopPixel &P = *c.P;
  for (int s = c.lane; s < 15; s += kCoopLanes) {
    const float r = P.u[s] - FLT_EPSILON;
    int id = 0;
    while (id < c.n && !(P.probs[id] > r)) ++id;
    P.samp[s] = (uint8_t)(id < c.n ? id : 255);
  }
}
__device__ __forceinline__ void strong_weigh(const CoopCtx &c) {
  if (!c.live) return;
  CoopPixel &P = *c.P;
  for (int j = c.lane; j < 32; j += kCoopLanes) {
    int m = 0;
    if (j < c.n)
      for (int s = 0; s < 15; ++s) m += P.samp[s] == j;
    P.vw[j] = (uint8_t)m;
  }
}
__device__ __forceinline__ void strong_active(const CoopCtx &c) {
  if (c.lane != 0) return;
  CoopPixel &P = *c.P;
  if (!c.live) { P.cnt = 0; return; }
  uint32_t sel = 0;
  float wn = 0;
  int na = 0, w1 = 0, w2 = 0, f1 = 0, f2 = 0;
  for (int i = 0; i < c.n; ++i) {
    const int v = P.vw[i];
    if (v > 0) {
      setBit(&sel, i);
      wn += v;
      if (v > w1) { w2 = w1; f2 = f1; w1 = v; f1 = na; }
      else if (v > w2) { w2 = v; f2 = na; }
      P.act[na++] = (uint8_t)i;
    }
  }
  P.na = (uint8_t)na;
  P.first = (uint8_t)f1;
  P.second = (uint8_t)f2;
  P.wn = wn;
  P.temp_sel = sel;
  // the current plane is evaluated unless a candidate's row holds its costs
  P.cnt = P.dup[kCurRow] == kCurRow ? na : 0;
}
// Candidate d's cost weighted by the samples (lane d); the current plane's list.
__device__ __forceinline__ void strong_weighted(const CoopCtx &c) {
  if (!c.live) return;
  CoopPixel &P = *c.P;
  const int n = c.n, d = c.lane;
  const float *row = c.cost + P.row[d] * n;
  float fc = 0.0f;
  for (int j = 0; j < n; ++j)
    if (P.vw[j] > 0) fc += P.vw[j] * row[j];
  P.fc[d] = fc / P.wn;
  if (P.cnt > 0) {
    const int off = coop_offset(c);
    for (int q = c.lane; q < P.na; q += kCoopLanes) c.list[off + q] = coop_entry(c, kCurRow, P.act[q]);
  }
}

// The current cost, the best candidate and its acceptance, and the draws of
// PlaneHypothesisRefinementStrong (DPE.cu:1069-1122) (lane 0).
__device__ __forceinline__ void strong_accept(const CoopCtx &c) {
  if (!c.live || c.lane != 0) return;
  const PMArgs &a = *c.a;
  const dpe_camera &rc = a.cam[0];
  [[maybe_unused]] const long long L = (long long)a.W * a.H;
  CoopPixel &P = *c.P;
  const int na = P.na;
  const float *cur = c.cost + P.dup[kCurRow] * c.n;
  float cost_now = 0.0f;
  for (int q = 0; q < na; ++q) cost_now += P.vw[P.act[q]] * cur[P.act[q]];
  cost_now /= P.wn;
  P.cost_written = cost_now;
  const float4 pl_cur = P.pl_cur;
  float depth_now = depth_from_plane(rc, pl_cur, c.px, c.py);
  float4 pl_now = pl_cur;
  uint32_t views_new = G(a.views, c.center, L, 213);
  const int mi = find_min_cost_index(P.fc, 8);
  const float fcost_mi = P.fc[mi];
  if (P.flag[mi]) {
    const float4 cand = G(a.P.use_edge ? a.plane_snap : a.plane, P.pos[mi], L, 214);
    const float db = depth_from_plane(rc, cand, c.px, c.py);
    if (db >= a.P.depth_min && db <= a.P.depth_max && fcost_mi < cost_now) {
      depth_now = db; pl_now = cand; cost_now = fcost_mi;
      views_new = P.temp_sel;
    }
  }
  AheadRng rng{{a.key[0], a.key[1], (uint32_t)c.center, P.rng_ctr}, P.ahead, 0};
  const float dmin = a.P.depth_min, dmax = a.P.depth_max;
  P.depth_rand = rng.uniform() * (dmax - dmin) + dmin;
  P.n_rand = random_normal(rc, c.px, c.py, rng, depth_now);
  const float lo = (1 - 0.02f) * depth_now, hi = (1 + 0.02f) * depth_now;
  P.depth_pert = rng.uniform() * (hi - lo) + lo;
  P.n_pert = perturbed_normal(rc, c.px, c.py, pl_now, rng, (float)(0.02f * 3.14159265358979323846));
  P.pl_now = pl_now;
  P.depth_now = depth_now;
  P.cost_now = cost_now;
  P.views_new = views_new;
  P.rng_ctr = rng.next.ctr;
}
// Refinement plane h (lane h): (random depth, normal now), (depth now, random normal), both random,
// (depth now, perturbed normal), (perturbed depth, normal now).  Its first sources: the heaviest, and
// for the perturbed planes, which often win, the next one too.
__device__ __forceinline__ int refine_first(const CoopPixel &P, int h) {
  return P.na == 0 ? 0 : (h >= 3 && P.na > 1) ? 2 : 1;
}
__device__ __forceinline__ void strong_planes(const CoopCtx &c) {
  CoopPixel &P = *c.P;
  if (!c.live) return;
  const int h = c.lane;
  if (h >= 5) return;
  const PMArgs &a = *c.a;
  const dpe_camera &rc = a.cam[0];
  float4 t = h == 0 || h == 4 ? P.pl_now : h == 3 ? P.n_pert : P.n_rand;
  const float depth = h == 0 || h == 2 ? P.depth_rand : h == 4 ? P.depth_pert : P.depth_now;
  t.w = dist_to_origin(rc, c.px, c.py, depth, t);
  P.hyp[h] = t;
  coop_rec(c, h, t);
  const float db = depth_from_plane(rc, t, c.px, c.py);
  P.alive[h] = db >= a.P.depth_min && db <= a.P.depth_max && P.na > 0 ? 1 : 0;
}
__device__ __forceinline__ void strong_first_count(const CoopCtx &c) {
  CoopPixel &P = *c.P;
  if (c.lane != 0) return;
  int m = 0;
  if (c.live)
    for (int h = 0; h < 5; ++h)
      if (P.alive[h]) m += refine_first(P, h);
  P.cnt = m;
}
__device__ __forceinline__ void strong_first_list(const CoopCtx &c) {
  if (!c.live || c.lane >= 5) return;
  const CoopPixel &P = *c.P;
  const int h = c.lane;
  if (!P.alive[h]) return;
  int o = coop_offset(c);
  for (int e = 0; e < h; ++e)
    if (P.alive[e]) o += refine_first(P, e);
  c.list[o] = coop_entry(c, h, P.act[P.first]);
  if (refine_first(P, h) > 1) c.list[o + 1] = coop_entry(c, h, P.act[P.second]);
}
// A plane whose first sources' weighted sum already reaches the cost to beat is out of play (lane h).
__device__ __forceinline__ void strong_drop(const CoopCtx &c) {
  if (!c.live || c.lane >= 5) return;
  CoopPixel &P = *c.P;
  const int h = c.lane;
  if (!P.alive[h]) return;
  const float *row = c.cost + h * c.n;
  const int s0 = P.act[P.first], s1 = P.act[P.second];
  float t = 0.0f;
  if (refine_first(P, h) > 1) {  // in the order of the full sum
    t += P.vw[min(s0, s1)] * row[min(s0, s1)];
    t += P.vw[max(s0, s1)] * row[max(s0, s1)];
  } else {
    t += P.vw[s0] * row[s0];
  }
  if (!(t / P.wn < P.cost_now)) P.alive[h] = 0;
}
__device__ __forceinline__ void strong_rest_count(const CoopCtx &c) {
  CoopPixel &P = *c.P;
  if (c.lane != 0) return;
  int m = 0;
  if (c.live)
    for (int h = 0; h < 5; ++h)
      if (P.alive[h]) m += P.na - refine_first(P, h);
  P.cnt = m;
}
__device__ __forceinline__ void strong_rest_list(const CoopCtx &c) {
  if (!c.live || c.lane >= 5) return;
  const CoopPixel &P = *c.P;
  const int h = c.lane;
  if (!P.alive[h]) return;
  int o = coop_offset(c);
  for (int e = 0; e < h; ++e)
    if (P.alive[e]) o += P.na - refine_first(P, e);
  const bool two = refine_first(P, h) > 1;
  for (int q = 0; q < P.na; ++q)
    if (q != P.first && !(two && q == P.second)) c.list[o++] = coop_entry(c, h, P.act[q]);
}
// Plane h's weighted cost in list order (lane h).
__device__ __forceinline__ void strong_refine_sum(const CoopCtx &c) {
  if (!c.live || c.lane >= 5) return;
  CoopPixel &P = *c.P;
  const int h = c.lane, na = P.na;
  if (!P.alive[h]) return;
  const float *row = c.cost + h * c.n;
  float tc = 0.0f;
  for (int q = 0; q < na; ++q) tc += P.vw[P.act[q]] * row[P.act[q]];
  P.u[h] = tc / P.wn;
}

// The pixel's outputs after its last decision.
__device__ __forceinline__ void strong_write(const CoopCtx &c, float4 pl_now, float cost_now) {
  const PMArgs &a = *c.a;
  [[maybe_unused]] const long long L = (long long)a.W * a.H;
  const int center = c.center;
  CoopPixel &P = *c.P;
  G(a.rng_ctr, center, L, 215) = P.rng_ctr;
  G(a.views, center, L, 216) = P.views_new;
  store_vweight(&G(a.vweight, center, L, 217), P.vw);
  const float cost_written = P.cost_written;
  if (a.P.state == DPE_REFINE_INIT) {
    if ((double)cost_now < (double)cost_written - 0.1) { G(a.cost, center, L, 218) = cost_now; G(a.plane, center, L, 219) = pl_now; }
    else G(a.cost, center, L, 220) = cost_written;
  } else {
    G(a.cost, center, L, 221) = cost_now;
    G(a.plane, center, L, 222) = pl_now;
  }
}

// The refinement decisions in order (lane 0), then the outputs -- or, with the Gauss-Newton hypothesis,
// the state its stages continue from.
template <bool kGN>
__device__ __forceinline__ void strong_decide(const CoopCtx &c) {
  if (!c.live || c.lane != 0) return;
  const dpe_camera &rc = c.a->cam[0];
  CoopPixel &P = *c.P;
  float cost_now = P.cost_now;
  int best = -1;
  for (int h = 0; h < 5; ++h)
    if (P.alive[h] && P.u[h] < cost_now) { best = h; cost_now = P.u[h]; }
  const float4 pl_now = best >= 0 ? P.hyp[best] : P.pl_now;
  if (kGN) {
    if (best >= 0) P.depth_now = depth_from_plane(rc, pl_now, c.px, c.py);
    P.pl_now = pl_now; P.cost_now = cost_now;
    return;
  }
  strong_write(c, pl_now, cost_now);
}

#ifdef __CUDA_ARCH__
// The Gauss-Newton hypothesis split over the lanes of a pixel: lane q adds the normal equations of
// sampled sources q, q + 8, ...; the lanes' sums are added by shuffles inside each 8-lane group (a
// pixel's lanes are 8 consecutive threads of one warp, and every thread of the block takes part);
// lane 0 solves, keeps the plane in hyp[0] and lists it against the sampled sources.
__device__ __forceinline__ void strong_gn(const CoopCtx &c) {
  static_assert(kCoopLanes == 8 && kCoopThreads % 32 == 0, "lane groups must tile whole warps");
  CoopPixel &P = *c.P;
  const bool on = c.live && P.na > 0;
  float m[9] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  GnFrame f{};
  if (on) {
    const PMArgs &a = *c.a;
    f = gn_frame(a.cam[0], c.px, c.py, P.pl_now, P.depth_now);
    const SmemWindow rw{P.win, P.center, P.inv_wsum, P.mean_r, P.var_r,
                        a.counters ? a.counters + 2 * KID_STRONG_UPDATE : nullptr};
    for (int q = c.lane; q < P.na; q += kCoopLanes)
      gn_accumulate(a, c.px, c.py, rw, P.pl_now, f, P.act[q], (float)P.vw[P.act[q]], m);
  }
#pragma unroll
  for (int k = 0; k < 9; ++k)
#pragma unroll
    for (int off = 1; off < kCoopLanes; off <<= 1) m[k] += __shfl_xor_sync(0xffffffffu, m[k], off, kCoopLanes);
  if (c.lane == 0) {
    float4 t;
    const bool ok = on && gn_solve(*c.a, c.px, c.py, P.pl_now, f, m, &t);
    P.flag[0] = ok ? 1 : 0;
    if (ok) {
      P.hyp[0] = t;
      coop_rec(c, 0, t);
    }
    P.cnt = ok ? P.na : 0;
  }
}
__device__ __forceinline__ void strong_gn_list(const CoopCtx &c) {
  if (!c.live) return;
  const int off = coop_offset(c);
  for (int q = c.lane; q < c.P->cnt; q += kCoopLanes) c.list[off + q] = coop_entry(c, 0, c.P->act[q]);
}
// The weighted cost in list order, the decision, the outputs (lane 0).
__device__ __forceinline__ void strong_gn_decide(const CoopCtx &c) {
  if (!c.live || c.lane != 0) return;
  const PMArgs &a = *c.a;
  const CoopPixel &P = *c.P;
  float4 pl_now = P.pl_now;
  float cost_now = P.cost_now;
  if (P.cnt > 0) {
    float tc = 0.0f;
    for (int q = 0; q < P.na; ++q) tc += P.vw[P.act[q]] * c.cost[P.act[q]];
    tc /= P.wn;
    const float4 t = P.hyp[0];
    const float db = depth_from_plane(a.cam[0], t, c.px, c.py);
    if (db >= a.P.depth_min && db <= a.P.depth_max && tc < cost_now) { pl_now = t; cost_now = tc; }
  }
  strong_write(c, pl_now, cost_now);
}
#endif

// The phases between barriers, one thread's part of each (host builds of this source run them in
// lock-step over a block).
enum {
  kPhTaps, kPhSearch, kPhDistinct, kPhList, kPhEval0, kPhChoose, kPhProbs, kPhCumulate, kPhSample, kPhWeigh,
  kPhActive, kPhWeighted, kPhEval1, kPhAccept, kPhPlanes, kPhFirstCount, kPhFirstList, kPhEval2, kPhDrop, kPhRestCount,
  kPhRestList, kPhEval3, kPhRefineSum, kPhDecide, kStrongPhases
};
template <int kStage, bool kGN>
__device__ __forceinline__ void strong_phase(const CoopCtx &c, int phase, int iter) {
  switch (phase) {
    case kPhTaps: strong_taps<kStage>(c); break;
    case kPhSearch: strong_search(c, iter); break;
    case kPhDistinct: strong_distinct(c); break;
    case kPhList: strong_list(c); break;
    case kPhChoose: strong_choose(c, iter); break;
    case kPhProbs: strong_probs(c, iter); break;
    case kPhCumulate: strong_cumulate(c); break;
    case kPhSample: strong_sample(c); break;
    case kPhWeigh: strong_weigh(c); break;
    case kPhActive: strong_active(c); break;
    case kPhWeighted: strong_weighted(c); break;
    case kPhAccept: strong_accept(c); break;
    case kPhPlanes: strong_planes(c); break;
    case kPhFirstCount: strong_first_count(c); break;
    case kPhFirstList: strong_first_list(c); break;
    case kPhDrop: strong_drop(c); break;
    case kPhRestCount: strong_rest_count(c); break;
    case kPhRestList: strong_rest_list(c); break;
    case kPhRefineSum: strong_refine_sum(c); break;
    case kPhDecide: strong_decide<kGN>(c); break;
    case kPhEval0: strong_eval<kStage>(c, c.n); break;
    default: strong_eval<kStage>(c, 1); break;
  }
}
template <int kStage, bool kGN>
__device__ __forceinline__ void strong_update_phase(int phase, const Launch &lc, int iter, int parity, void *smem) {
  strong_phase<kStage, kGN>(coop_ctx(lc, parity, smem), phase, iter);
}

// Phases kFirst..kLast, each followed by a warp barrier.
template <int kStage, bool kGN, int kFirst, int kLast>
__device__ __forceinline__ void strong_run(const CoopCtx &c, int iter) {
  strong_phase<kStage, kGN>(c, kFirst, iter);
  DPE_WARP_BARRIER();
  if constexpr (kFirst < kLast) strong_run<kStage, kGN, kFirst + 1, kLast>(c, iter);
}

// Grid: ((W + 15) / 16, (H + 1) / 2) blocks of kCoopThreads; coop_smem_bytes(N - 1) dynamic shared
// bytes (the largest N of a batch).
template <int kStage, bool kGN>
__global__ void __launch_bounds__(kCoopThreads, DPE_STRONG_MIN_BLOCKS) k_strong_update(const Launch lc, int iter, int parity) {
  extern __shared__ float4 coop_smem[];
  const CoopCtx c = coop_ctx(lc, parity, coop_smem);
  strong_run<kStage, kGN, kPhTaps, kPhList>(c, iter);
#pragma unroll 1
  for (int stage = 0; stage < (kGN ? 5 : 4); ++stage) {
    __syncthreads();
    strong_eval<kStage>(c, stage == 0 ? c.n : 1);
    __syncthreads();
    if (stage == 0) strong_run<kStage, kGN, kPhChoose, kPhWeighted>(c, iter);
    else if (stage == 1) strong_run<kStage, kGN, kPhAccept, kPhFirstList>(c, iter);
    else if (stage == 2) strong_run<kStage, kGN, kPhDrop, kPhRestList>(c, iter);
    else if (stage == 3) {
      strong_run<kStage, kGN, kPhRefineSum, kPhDecide>(c, iter);
#ifdef __CUDA_ARCH__
      if constexpr (kGN) {
        strong_gn(c);
        DPE_WARP_BARRIER();
        strong_gn_list(c);
        DPE_WARP_BARRIER();
      }
    } else {
      if constexpr (kGN) strong_gn_decide(c);
#endif
    }
  }
}


// ------------------------------------------------------------------ RANSACToGetFitPlane (DPE.cu:2895-3128)
// A group of kGnLanes threads per WEAK pixel (only WEAK pixels read their fitted plane).  Every one of
// the 50 rounds draws three numbers, so the lanes prepare the next rounds side by side: points, tests,
// plane and its summed distance do not depend on earlier rounds; they are then taken in order under the
// current state.  Host builds of this source run it with one lane.
// 60 launches at 400x300 and 200x150: 5.4 -> 1.2 ms; three at 1600x1200 with 403 k WEAK pixels 7.7 -> 4.3 ms (one
// thread per pixel before).
struct FitPoints {
  short2 sp[kNeighbours - 1];
  float3 pos[kNeighbours - 1], nrm[kNeighbours - 1];
  float2 ray[kNeighbours - 1];
  LinePoint line[kNeighbours - 1];
};
__device__ __forceinline__ void ransac_fit_plane_pixel(const PMArgs &a, const LineMap &map, const GnGroup &g, FitPoints &S,
                                                       int px, int py) {
  const int W = a.W, center = px + py * W;
  uint32_t ctr = G(a.rng_ctr, center, (long long)W * a.H, 106);
  const dpe_camera &cam = a.cam[0];
  bool edge_limit = false;
  if (a.P.use_limit) {
    edge_limit = true;
    if (a.P.use_edge) {
      const float cv = a.complexity[center];
      Rng rng{a.key[0], a.key[1], (uint32_t)center, ctr++};
      const float rp = rng.uniform() - FLT_EPSILON;
      if (rp < cv) edge_limit = false;
    }
  }
  g.sync();  // the group's last pixel has been read
  int sc = 0;
  for (int i = 1; i < kNeighbours; ++i) {
    const short2 t = neighbour(a, center, i);
    if (t.x == -1 || t.y == -1) continue;
    if (sc % kGnLanes == g.lane) {
      S.sp[sc] = t;
      const float4 tpl = a.plane[t.x + t.y * W];
      const float d = depth_from_plane(cam, tpl, t.x, t.y);
      float X[3];
      point3d(cam, t.x, t.y, d, X);
      S.pos[sc] = make_float3(X[0], X[1], X[2]);
      S.nrm[sc] = make_float3(tpl.x, tpl.y, tpl.z);
      S.ray[sc] = make_float2((t.x - cam.K[2]) / cam.K[0], (t.y - cam.K[5]) / cam.K[4]);
      if (edge_limit) S.line[sc] = line_point(a, map, t.x, t.y);
    }
    sc++;
  }
  if (sc < 3) {
    if (g.lane == 0) {
      a.fit_plane[center] = a.plane[center];
      a.rng_ctr[center] = ctr;
    }
    return;
  }
  g.sync();
  int ua = -1, ub = -1, uc = -1;
  float min_cost = FLT_MAX;
  float4 best = make_float4(0, 0, 0, 0);
  bool has_best = false, has_strong = false;
  bool must_tri = (a.P.use_label && a.label[center] > 0 && edge_limit) ? false : true;
  for (int i0 = 0; i0 < 50; i0 += kGnLanes) {
    bool ok = i0 + g.lane < 50, tri = false, strong = false;
    int ia = 0, ib = 0, ic = 0;
    float4 cr = make_float4(0, 0, 0, 0);
    float tc = 0.0f;
    if (ok) {
      Rng rng{a.key[0], a.key[1], (uint32_t)center, ctr + 3u * (uint32_t)(i0 + g.lane)};
      ia = (int)(rng.u32() % (uint32_t)sc);
      ib = (int)(rng.u32() % (uint32_t)sc);
      ic = (int)(rng.u32() % (uint32_t)sc);
      ok = !(ia == ib || ib == ic || ia == ic);
    }
    if (ok && a.P.geom_consistency && edge_limit) {
      const float3 AN = S.nrm[ia], BN = S.nrm[ib], CN = S.nrm[ic];
      strong = !((double)(AN.x * BN.x + AN.y * BN.y + AN.z * BN.z) < 0.8660254 ||
                 (double)(AN.x * CN.x + AN.y * CN.y + AN.z * CN.z) < 0.8660254 ||
                 (double)(BN.x * CN.x + BN.y * CN.y + BN.z * CN.z) < 0.8660254);
      ok = strong || !has_strong;
    }
    if (ok) {
      tri = point_in_triangle(S.sp[ia], S.sp[ib], S.sp[ic], px, py);
      ok = tri || !must_tri;
    }
    if (edge_limit) {
      int i = ia, j = ib;
#ifdef __CUDA_ARCH__
#pragma unroll 1
#endif
      for (int k = 0; ok && k < 3; ++k) {
        ok = !line_blocked(a, map, S.line[i], S.line[j]);
        i = j;
        j = k == 0 ? ic : ia;
      }
    }
    if (ok) {
      const float3 A = S.pos[ia], B = S.pos[ib], C = S.pos[ic];
      const float3 AC = make_float3(A.x - C.x, A.y - C.y, A.z - C.z), BC = make_float3(B.x - C.x, B.y - C.y, B.z - C.z);
      cr.x = AC.y * BC.z - BC.y * AC.z;
      cr.y = -(AC.x * BC.z - BC.x * AC.z);
      cr.z = AC.x * BC.y - BC.x * AC.y;
      ok = !((cr.x == 0 && cr.y == 0 && cr.z == 0) || isnan(cr.x) || isnan(cr.y) || isnan(cr.z));
      if (ok) {
        normalize3(&cr);
        cr.w = -(cr.x * A.x + cr.y * A.y + cr.z * A.z);
        for (int s = 0; s < sc; ++s) {
          if (s == ia || s == ib || s == ic) continue;
          const float fd = -cr.w / (cr.x * S.ray[s].x + cr.y * S.ray[s].y + cr.z);
          tc += fabsf(fd - S.pos[s].z);
        }
      }
    }
    const unsigned b_tri = g.ballot(tri), b_strong = g.ballot(strong);
    for (unsigned todo = g.ballot(ok); todo; todo &= todo - 1) {
      const int r = g.first(todo);
      const bool r_tri = (b_tri >> r) & 1u, r_strong = (b_strong >> r) & 1u;
      if (a.P.geom_consistency && edge_limit && has_strong && !r_strong) continue;
      if (must_tri && !r_tri) continue;
      if (r_strong) has_strong = true;
      const float t = g.from(tc, r);
      if (t < min_cost) {
        if (r_tri) must_tri = true;
        min_cost = t;
        best = make_float4(g.from(cr.x, r), g.from(cr.y, r), g.from(cr.z, r), g.from(cr.w, r));
        has_best = true;
        ua = g.from(ia, r); ub = g.from(ib, r); uc = g.from(ic, r);
      }
    }
  }
  ctr += 150u;
  if (g.lane != 0) return;
  a.rng_ctr[center] = ctr;
  if (has_best) {
    const float depth = depth_from_plane(cam, a.plane[center], px, py);
    const float4 v = view_direction(cam, px, py, depth);
    if (best.x * v.x + best.y * v.y + best.z * v.z > 0) { best.x = -best.x; best.y = -best.y; best.z = -best.z; best.w = -best.w; }
    a.fit_plane[center] = best;
    if (a.P.use_radius) {
      if (must_tri) {
        const short2 A = S.sp[ua], B = S.sp[ub], C = S.sp[uc];
        const float la = sqrtf((float)((A.x - B.x) * (A.x - B.x) + (A.y - B.y) * (A.y - B.y)));
        const float lb = sqrtf((float)((B.x - C.x) * (B.x - C.x) + (B.y - C.y) * (B.y - C.y)));
        const float lc = sqrtf((float)((C.x - A.x) * (C.x - A.x) + (C.y - A.y) * (C.y - A.y)));
        const float p = (float)((la + lb + lc) / 2.0);
        const float S = sqrtf(p * (p - la) * (p - lb) * (p - lc));
        int radius = (int)floor(sqrtf(S) / 2.0);
        const float ad = sqrtf((float)((A.x - px) * (A.x - px) + (A.y - py) * (A.y - py)));
        const float bd = sqrtf((float)((B.x - px) * (B.x - px) + (B.y - py) * (B.y - py)));
        const float cd = sqrtf((float)((C.x - px) * (C.x - px) + (C.y - py) * (C.y - py)));
        const float md = cvmin(cvmin(ad, bd), cd);
        if (2.5 * md < radius) radius = (int)md;
        if (edge_limit) {
          if (a.P.use_edge) {
            float med = FLT_MAX;
            const short2 *en = &a.edge_neigh[(size_t)center * 8];
            for (int d = 0; d < 8; ++d) {
              const short2 e = en[d];
              if (e.x == -1 || e.y == -1) continue;
              med = cvmin(med, sqrtf((float)((e.x - px) * (e.x - px) + (e.y - py) * (e.y - py))));
            }
            if (med < radius) radius = (int)med;
          }
          if (a.P.use_label && a.label[center] > 0) {
            float mbd = FLT_MAX;
            const short2 *lb2 = &a.lab_bound[(size_t)a.nmap[center] * 8];
            for (int d = 0; d < 8; ++d) {
              const short2 bb = lb2[d];
              if (bb.x == -1 || bb.y == -1) continue;
              const double ddx = (double)(px - bb.x), ddy = (double)(py - bb.y);
              mbd = cvmin(mbd, (float)sqrt(ddx * ddx + ddy * ddy));
            }
            if (mbd < radius) radius = (int)mbd;
          }
        }
        for (int guard = 0; (radius << 1) % 5 != 0 && guard < 5; ++guard) radius--;
        if (!edge_limit) a.radius[center] = radius > a.P.strong_radius ? 0 : a.P.strong_radius;
        else a.radius[center] = radius > a.P.strong_radius ? radius : a.P.strong_radius;
      } else {
        a.radius[center] = a.P.strong_radius;
      }
    }
  } else {
    a.fit_plane[center] = make_float4(0, 0, 0, 0);
    if (a.P.use_radius) a.radius[center] = a.P.strong_radius;
  }
}
// On the device a grid of groups strides over both colours' lists; host builds call it per pixel.
__global__ void __launch_bounds__(128) k_ransac_fit_plane(const Launch lc) {
#ifdef __CUDA_ARCH__
  const Blk B = resolve<kGridList>(lc);
  const PMArgs &a = *B.a;
  __shared__ FitPoints S[128 / kGnLanes];
  const LineMap map = a.P.use_limit ? line_map(a) : LineMap{0.f, 0.f, 0, 0, 0};
  const int slot = (int)threadIdx.x / kGnLanes;
  GnGroup g;
  g.lane = (int)threadIdx.x % kGnLanes;
  g.shift = ((int)threadIdx.x & 31) - g.lane;
  g.mask = (kGnLanes == 32 ? 0xFFFFFFFFu : (1u << (kGnLanes & 31)) - 1u) << g.shift;
  const int n0 = a.wcount[0], count = n0 + a.wcount[1];
  for (int i = B.x * (128 / kGnLanes) + slot; i < count; i += B.gx * (128 / kGnLanes)) {
    const int c = i < n0 ? a.wlist[0][i] : a.wlist[1][i - n0];
    ransac_fit_plane_pixel(a, map, g, S[slot], c % a.W, c / a.W);
  }
#else
  const Blk B = resolve<kGridFull>(lc);
  const PMArgs &a = *B.a;
  int px, py;
  if (!full_pixel(a, B, &px, &py) || a.weak[px + py * a.W] != DPE_WEAK) return;
  FitPoints S;
  ransac_fit_plane_pixel(a, a.P.use_limit ? line_map(a) : LineMap{0.f, 0.f, 0, 0, 0}, GnGroup{0}, S, px, py);
#endif
}

// ------------------------------------------------------------------ weak update (DPE.cu:1672-1866, 1124-1216)
// CheckerboardPropagationWeak + PlaneHypothesisRefinementWeak for the WEAK pixels of one colour,
// split into work lists so that every lane has work:
//   k_weak_prepare      per pixel: the reference side of its nine windows (table, sums);
//   k_weak_eval<false>  per (pixel, hypothesis, source): the 8 strong-neighbour candidates, the
//                       current plane and the fitted plane;
//   k_weak_decide       per pixel: view sampling, candidate choice, fitted-plane test, and the five
//                       random refinement hypotheses (all random draws of the pixel);
//   k_weak_eval<true>   per (pixel, random hypothesis, sampled source);
//   k_weak_finish       per pixel: the random-hypothesis test, the REFINE_INIT rule, the write-back
//                       and the final strong-window re-cost.
// Each cost is the one the fused per-pixel form computes, and every sum runs in the same order.
// Pixels of one colour read only STRONG neighbours and their own state, so the order of the
// list does not matter.  Work items are strided over a grid sized for the GPU; the list lengths
// stay on the device.

// A thread per (pixel, window): the longest chain is the centre window's 36 taps (60 launches at 400x300
// and 200x150: 4.4 -> 1.5 ms against a thread per pixel).
__global__ void __launch_bounds__(128) k_weak_prepare(const Launch lc, int parity) {
  const Blk B = resolve<kGridList>(lc);
  const PMArgs &a = *B.a;
  const long long total = (long long)a.wcount[parity] * kNeighbours;
  const int *list = a.wlist[parity];
  for (long long i = (long long)B.x * blockDim.x + threadIdx.x; i < total; i += (long long)B.gx * blockDim.x) {
    const int slot = (int)(i / kNeighbours), k = (int)(i - (long long)slot * kNeighbours);
    const int center = list[slot];
    const int px = center % a.W, py = center / a.W;
    const float ref_center = texel(a, 0, px, py);
    float2 *tab = a.wtab + (size_t)slot * a.wtab_stride;
    const short2 nb = neighbour(a, center, k);
    float4 win = make_float4(0, 0, 0, 0);
    if (nb.x != -1 && nb.y != -1) {
      int radius, inc;
      weak_window_shape(a, center, k, &radius, &inc);
      int t = 0;
      float s_r = 0, s_rr = 0, s_w = 0;
      for (int x = -radius; x <= radius; x += inc) {
        float r_r = 0, r_rr = 0, r_w = 0;
        for (int y = -radius; y <= radius; y += inc) {
          const float rp = texel(a, 0, nb.x + x, nb.y + y);
          const float w = bilateral_weight((float)x, (float)y, rp, ref_center, a.P.sigma_spatial, a.P.sigma_color);
          const float rc = rp - ref_center;
          weak_store(a, tab, k, t++, w, w * rc);
          r_r += w * rc; r_rr += w * rc * rc; r_w += w;
        }
        s_r += r_r; s_rr += r_rr; s_w += r_w;
      }
      win = make_float4(s_w, s_r, s_rr, 0.0f);
    }
    a.wwin[(size_t)slot * kNeighbours + k] = win;
  }
}

// kRandom = false: hypotheses 0..7 are the candidates (the planes of the strong neighbours 1..8),
// 8 the current plane, 9 the fitted plane.  kRandom = true: the five random hypotheses, for the
// sources the pixel sampled.  Unevaluated candidates keep the fused form's initial costs (0, and 2
// for the first candidate's first source: quirk Q2).
// A warp takes one pixel: its threads split the (hypothesis, source) pairs that have a cost, the
// hypotheses of one source next to each other, so that a gather reads one image and the windows, their
// shapes and their tables are the warp's.  (A thread per pair of the whole list, sources next to each
// other, spent 72 - 84 % of L1's cycles on gathers spread over nine images, with 20 - 25 of 32
// threads active.)  Host builds of this source run it with one lane.
// Measured (12 launches; 1600x1200 geometric call / 801x603 level / 20 calls at 400x300 and 200x150): 64.6 /
// 14.9 / 7.3 -> 49.7 / 11.4 / 6.0 ms at 4 blocks (128 registers); 6 blocks 49.6 / 11.3 / 6.5, 8 blocks
// 51.2 / - / 6.8.
#ifndef DPE_WEAK_MIN_BLOCKS
#define DPE_WEAK_MIN_BLOCKS 4
#endif
#ifdef __CUDA_ARCH__
constexpr int kWeakLanes = 32;
#else
constexpr int kWeakLanes = 1;
#endif
struct WeakItems {
  float4 pl[10];
  uint8_t hyp[16], src[32];  // the hypotheses and sources that are evaluated
  int nh, ns;
};
template <bool kRandom>
__device__ __forceinline__ void weak_items(const PMArgs &a, int slot, int center, int lane, WeakItems &S) {
  const int n = a.N - 1;
  for (int h = lane; h < (kRandom ? 5 : 10); h += kWeakLanes) {
    bool on = true;
    float4 pl;
    if (kRandom) {
      pl = a.whyp[(size_t)slot * 5 + h];
    } else if (h < 8) {
      const short2 nb = neighbour(a, center, h + 1);
      on = !(nb.x == -1 || nb.y == -1 || a.weak[nb.x + nb.y * a.W] != DPE_STRONG);
      if (on) pl = a.plane[nb.x + nb.y * a.W];
    } else {
      pl = h == 8 ? a.plane[center] : a.fit_plane[center];
      if (h == 9) on = !(pl.x == 0 && pl.y == 0 && pl.z == 0);  // unused: refinement skipped
    }
    if (on) S.pl[h] = pl;
    S.hyp[h] = on ? 1 : 0;
    if (!on && h < 8)
      for (int j = 0; j < n; ++j) {
        a.wcost[((size_t)slot * 10 + h) * n + j] = (h == 0 && j == 0) ? 2.0f : 0.0f;
        a.wgeom[((size_t)slot * 10 + h) * n + j] = 0.0f;
      }
  }
}
// The lists of what is evaluated, from the flags (one thread).
template <bool kRandom>
__device__ __forceinline__ void weak_lists(const PMArgs &a, int center, WeakItems &S) {
  int m = 0;
  for (int h = 0; h < (kRandom ? 5 : 10); ++h)
    if (S.hyp[h]) S.hyp[m++] = (uint8_t)h;
  S.nh = m;
  m = 0;
  const uint4 vw = kRandom ? a.vweight[center] : make_uint4(0, 0, 0, 0);
  for (int j = 0; j < a.N - 1; ++j)
    if (!kRandom || vweight_at(vw, j) != 0) S.src[m++] = (uint8_t)j;
  S.ns = m;
}
template <bool kRandom, int kStage>
__global__ void __launch_bounds__(128, DPE_WEAK_MIN_BLOCKS) k_weak_eval(const Launch lc, int parity) {
  const Blk B = resolve<kGridList>(lc);
  const PMArgs &a = *B.a;
#ifdef __CUDA_ARCH__
  __shared__ WeakItems sh[128 / kWeakLanes];
  WeakItems &S = sh[threadIdx.x / kWeakLanes];
#else
  WeakItems S;
#endif
  const int n = a.N - 1, hyps = kRandom ? 5 : 10;
  const int count = a.wcount[parity];
  const int *list = a.wlist[parity];
  const bool geom = a.P.geom_consistency != 0;
  float *costs = kRandom ? a.wcost_r : a.wcost;
  float *geoms = kRandom ? a.wgeom_r : a.wgeom;
  const int lane = (int)threadIdx.x % kWeakLanes, per = blockDim.x / kWeakLanes;
  for (int slot = B.x * per + (int)threadIdx.x / kWeakLanes; slot < count; slot += B.gx * per) {
    const int center = list[slot];
    const int px = center % a.W, py = center / a.W;
    if (kRandom) {
      const float4 fp = a.fit_plane[center];
      if (fp.x == 0 && fp.y == 0 && fp.z == 0) continue;  // no random refinement for this pixel
    }
    DPE_WARP_BARRIER();  // the last pixel's lists have been read
    weak_items<kRandom>(a, slot, center, lane, S);
    DPE_WARP_BARRIER();
    if (lane == 0) weak_lists<kRandom>(a, center, S);
    DPE_WARP_BARRIER();
    const int total = S.nh * S.ns;
    for (int i0 = 0; i0 < total; i0 += kWeakLanes) {
      DPE_WARP_BARRIER();
      const int i = i0 + lane;
      if (i >= total) continue;
      const int jj = i / S.nh, h = S.hyp[i - jj * S.nh], j = S.src[jj];
      const float4 pl = S.pl[h];
      const size_t at = ((size_t)slot * hyps + h) * n + j;
      costs[at] = ncc_weak_tab<kStage>(a, slot, center, px, py, j + 1, pl, KID_WEAK_EVAL);
      geoms[at] = geom ? geom_cost(a, px, py, j + 1, pl) : 0.0f;
    }
  }
}

__global__ void __launch_bounds__(128) k_weak_decide(const Launch lc, int iter, int parity) {
  const Blk B = resolve<kGridList>(lc);
  const PMArgs &a = *B.a;
  const int n = a.N - 1, W = a.W;
  const int count = a.wcount[parity];
  const int *list = a.wlist[parity];
  const dpe_camera &rc = a.cam[0];
  const bool geom = a.P.geom_consistency != 0;
  const float gf = a.P.geom_factor;
  const float dmin = a.P.depth_min, dmax = a.P.depth_max;
  float priors[kMaxSrc], probs[kMaxSrc];
  uint8_t vw[32];
  float final_costs[8];
  bool flag[8];
  float4 cand[8];
  for (int slot = B.x * blockDim.x + threadIdx.x; slot < count; slot += B.gx * blockDim.x) {
    const int center = list[slot];
    const int px = center % W, py = center / W;
    const float *ca = a.wcost + (size_t)slot * 10 * n;
    const float *ga = a.wgeom + (size_t)slot * 10 * n;
    for (int i = 0; i < 8; ++i) {
      const short2 nb = neighbour(a, center, i + 1);
      flag[i] = !(nb.x == -1 || nb.y == -1 || a.weak[nb.x + nb.y * W] != DPE_STRONG);
      cand[i] = flag[i] ? a.plane[nb.x + nb.y * W] : make_float4(0, 0, 0, 0);
    }
    for (int j = 0; j < n; ++j) priors[j] = 0.0f;
    for (int i = 0; i < 8; ++i) {
      const short2 nb = neighbour(a, center, i + 1);
      if (nb.x == -1 || nb.y == -1) continue;
      const uint32_t sv = a.views[nb.x + nb.y * W];
      for (int j = 0; j < n; ++j) priors[j] += isSet(sv, j) == 1 ? 0.9f : 0.1f;
    }
    Rng rng = make_rng(a, center);
    uint32_t temp_sel = 0;
    const float wn = sample_views(a, rng, iter, ca, n, priors, vw, &temp_sel, probs);
    for (int i = 0; i < 8; ++i) {
      float fc = 0.0f;
      for (int j = 0; j < n; ++j)
        if (vw[j] > 0) {
          if (geom) fc += vw[j] * (ca[i * n + j] + gf * (flag[i] ? ga[i * n + j] : 3.0f));
          else fc += vw[j] * ca[i * n + j];
        }
      final_costs[i] = fc / wn;
    }
    const int mi = find_min_cost_index(final_costs, 8);
    const float4 pl_cur = a.plane[center];
    float cost_now = 0.0f;
    for (int i = 0; i < n; ++i) {
      if (vw[i] == 0) continue;  // 0 * (finite cost) contributes nothing
      const float c = ca[8 * n + i];
      if (geom) cost_now += vw[i] * (c + gf * ga[8 * n + i]);
      else cost_now += vw[i] * c;
    }
    cost_now /= wn;
    const float cost_written = cost_now;
    float depth_now = depth_from_plane(rc, pl_cur, px, py);
    float4 pl_now = pl_cur;
    uint32_t views_new = a.views[center];
    if (flag[mi]) {
      const float db = depth_from_plane(rc, cand[mi], px, py);
      if (db >= dmin && db <= dmax && final_costs[mi] < cost_now) {
        depth_now = db; pl_now = cand[mi]; cost_now = final_costs[mi];
        views_new = temp_sel;
      }
    }
    // PlaneHypothesisRefinementWeak: the fitted plane, then five random hypotheses.  A zero fitted
    // plane ends the refinement before the random hypotheses (DPE.cu:1146-1148).
    const float4 fp = a.fit_plane[center];
    if (!(fp.x == 0 && fp.y == 0 && fp.z == 0)) {
      float tc = 0.0f;
      for (int j = 0; j < n; ++j)
        if (vw[j] > 0) {
          const float c = ca[9 * n + j];
          if (geom) tc += vw[j] * (c + gf * ga[9 * n + j]);
          else tc += vw[j] * c;
        }
      tc /= wn;
      const float db = depth_from_plane(rc, fp, px, py);
      if (db >= dmin && db <= dmax && tc < cost_now) { depth_now = db; pl_now = fp; cost_now = tc; }
      const float depth_rand = rng.uniform() * (dmax - dmin) + dmin;
      const float4 n_rand = random_normal(rc, px, py, rng, depth_now);
      const float lo = (1 - 0.02f) * depth_now, hi = (1 + 0.02f) * depth_now;
      const float depth_pert = rng.uniform() * (hi - lo) + lo;
      const float4 n_pert = perturbed_normal(rc, px, py, pl_now, rng, (float)(0.02f * 3.14159265358979323846));
      const float depths[5] = {depth_rand, depth_now, depth_rand, depth_now, depth_pert};
      const float4 normals[5] = {pl_now, n_rand, n_rand, n_pert, pl_now};
      for (int h = 0; h < 5; ++h) {
        float4 t = normals[h];
        t.w = dist_to_origin(rc, px, py, depths[h], t);
        a.whyp[(size_t)slot * 5 + h] = t;
      }
    }
    a.rng_ctr[center] = rng.ctr;
    a.views[center] = views_new;
    store_vweight(&a.vweight[center], vw);
    a.wstate[(size_t)slot * 2] = pl_now;
    a.wstate[(size_t)slot * 2 + 1] = make_float4(depth_now, cost_now, cost_written, wn);
  }
}

// 8 threads per pixel: they split the window's taps and the sources of the final cost; the first of them
// takes the decisions (60 launches at 400x300 and 200x150: 3.8 -> 1.2 ms against a thread per pixel, whose
// chain of evaluations was the launch's length; 2.5 -> 3.2 ms for six at 1600x1200, where threads abound).
// Host builds of this source run it with one.
#ifdef __CUDA_ARCH__
constexpr int kFinishLanes = 8;
#else
constexpr int kFinishLanes = 1;
#endif
struct FinishPixel {
  float4 win[kWinPairs];
  float rc[kWinTaps];  // w (r - c)^2 per tap
  float cost[kMaxSrc];
  float4 pl;
};
template <int kStage>
__global__ void __launch_bounds__(128) k_weak_finish(const Launch lc, int parity) {
  const Blk B = resolve<kGridList>(lc);
  const PMArgs &a = *B.a;
#ifdef __CUDA_ARCH__
  __shared__ FinishPixel sh[128 / kFinishLanes];
  FinishPixel &S = sh[threadIdx.x / kFinishLanes];
#else
  FinishPixel S;
#endif
  const int n = a.N - 1, W = a.W;
  const int count = a.wcount[parity];
  const int *list = a.wlist[parity];
  const dpe_camera &rc = a.cam[0];
  const bool geom = a.P.geom_consistency != 0;
  const float gf = a.P.geom_factor;
  const float dmin = a.P.depth_min, dmax = a.P.depth_max;
  const int lane = (int)threadIdx.x % kFinishLanes, per = blockDim.x / kFinishLanes;
  const int first = B.x * per + (int)threadIdx.x / kFinishLanes;
  // every thread makes every round (the barriers are the warp's)
  for (int s0 = 0; s0 < count; s0 += B.gx * per) {
    const int slot = s0 + first;
    const bool on = slot < count;
    const int center = on ? list[slot] : 0;
    const int px = center % W, py = center / W;
    const uint4 vwp = on ? a.vweight[center] : make_uint4(0, 0, 0, 0);
    const float wn = on ? a.wstate[(size_t)slot * 2 + 1].w : 0.0f;
    DPE_WARP_BARRIER();  // the last round's shared values have been read
    float center_val = 0.0f;
    if (on) {
      // window taps of the final re-cost with the strong window (DPE.cu:1849-1865; the radius swap there
      // has no effect)
      const int r = a.P.strong_radius, inc = a.P.strong_increment, side = 2 * r / inc + 1;
      center_val = texel(a, 0, px, py);
      for (int k = lane; k < side * side; k += kFinishLanes) {
        const int i = -r + (k / side) * inc, j = -r + (k % side) * inc;
        const float rp = texel(a, 0, px + i, py + j);
        const float w = bilateral_weight((float)i, (float)j, rp, center_val, a.P.sigma_spatial, a.P.sigma_color);
        const float d = rp - center_val, wr = w * d;
        win_store(S.win, k, w, wr);
        S.rc[k] = wr * d;
      }
    }
    if (on && lane == 0) {
      float4 pl_now = a.wstate[(size_t)slot * 2];
      const float4 st = a.wstate[(size_t)slot * 2 + 1];
      float cost_now = st.y;
      const float cost_written = st.z;
      const float4 fp = a.fit_plane[center];
      if (!(fp.x == 0 && fp.y == 0 && fp.z == 0)) {
        const float *cr = a.wcost_r + (size_t)slot * 5 * n;
        const float *gr = a.wgeom_r + (size_t)slot * 5 * n;
        for (int h = 0; h < 5; ++h) {
          const float4 t = a.whyp[(size_t)slot * 5 + h];
          float tc = 0.0f;
          for (int j = 0; j < n; ++j) {
            const int v = vweight_at(vwp, j);
            if (v > 0) {
              const float c = cr[h * n + j];
              if (geom) tc += v * (c + gf * gr[h * n + j]);
              else tc += v * c;
            }
          }
          tc /= wn;
          const float db = depth_from_plane(rc, t, px, py);
          if (db >= dmin && db <= dmax && tc < cost_now) { pl_now = t; cost_now = tc; }
        }
      }
      float4 pl_final = a.plane[center];
      if (a.P.state == DPE_REFINE_INIT) {
        if ((double)cost_now < (double)cost_written - 0.1) pl_final = pl_now;
      } else {
        pl_final = pl_now;
      }
      a.plane[center] = pl_final;
      S.pl = pl_final;
    }
    DPE_WARP_BARRIER();
    if (on) {
      const int side = 2 * a.P.strong_radius / a.P.strong_increment + 1;
      float sw = 0.f, swr = 0.f, swrr = 0.f;
      for (int k = 0; k < side * side; ++k) {
        const float2 t = win_tap(S.win, k);
        sw += t.x; swr += t.y; swrr += S.rc[k];
      }
      SmemWindow rw;
      rw.t_ = S.win;
      rw.center = center_val;
      rw.inv_wsum = 1.0f / sw;
      rw.mean_r = swr * rw.inv_wsum;
      rw.var_r = swrr * rw.inv_wsum - rw.mean_r * rw.mean_r;
      rw.cnt = a.counters ? a.counters + 2 * KID_WEAK_FINISH : nullptr;
      const float4 pl = S.pl;
      for (int j = lane; j < n; j += kFinishLanes)
        if (vweight_at(vwp, j) > 0) S.cost[j] = ncc_strong<kStage, true>(a, px, py, j + 1, pl, rw);
    }
    DPE_WARP_BARRIER();
    if (on && lane == 0) {
      float tc = 0.0f;
      for (int j = 0; j < n; ++j) {
        const int v = vweight_at(vwp, j);
        if (v > 0) tc += v * S.cost[j];
      }
      a.cost[center] = tc / wn;
    }
  }
}

// ------------------------------------------------------------------ post passes
__global__ void k_get_depth_normal(const Launch lc) {
  const Blk B = resolve<kGridFull>(lc);
  const PMArgs &a = *B.a;
  int px, py;
  if (!full_pixel(a, B, &px, &py)) return;
  const int c = py * a.W + px;
  float4 pl = a.plane[c];
  pl.w = depth_from_plane(a.cam[0], pl, px, py);
  a.plane[c] = normal_to_world(a.cam[0], pl);
}

// CheckerboardFilterStrong (DPE.cu:1961-2071)
__global__ void k_filter_strong(const Launch lc, int parity) {
  const Blk B = resolve<kGridHalf>(lc);
  const PMArgs &a = *B.a;
  int px, py;
  if (!colour_pixel(a, B, parity, &px, &py)) return;
  const int W = a.W, H = a.H, center = py * W + px;
  if (a.weak[center] == DPE_WEAK) return;
  if (a.cost[center] < 0.001f) return;
  const int up = center - W, upup = center - 3 * W, dn = center + W, dndn = center + 3 * W;
  const int lf = center - 1, lflf = center - 3, rt = center + 1, rtrt = center + 3;
  const int idx[20] = {up, upup, upup - 2 * W, dn, dndn, dndn + 2 * W, lf, lflf, lflf - 2, rt, rtrt, rtrt + 2,
                       up + 2, dn + 2, up - 2, dn - 2, lf - 2 * W, rt - 2 * W, lf + 2 * W, rt + 2 * W};
  const bool ok[20] = {py > 0, py > 2, py > 4, py < H - 1, py < H - 3, py < H - 5, px > 0, px > 2, px > 4,
                       px < W - 1, px < W - 3, px < W - 5, py > 0 && px < W - 2, py < H - 1 && px < W - 2,
                       py > 0 && px > 1, py < H - 1 && px > 1, px > 0 && py > 2, px < W - 1 && py > 2,
                       px > 0 && py < H - 2, px < W - 1 && py < H - 2};
  // The median by ranks, in registers: value i's rank is the number of values before it in the stable
  // order.  (The reference's insertion sort over an indexed array lives in local memory: two launches at
  // 160x120 took 42 us, at 1600x1200 355 us; now 29 and 154 us.)
  float f[21];
  bool in[21], nan = false;
  f[0] = a.plane[center].w;
  in[0] = true;
#pragma unroll
  for (int i = 0; i < 20; ++i) {
    in[i + 1] = ok[i] && a.weak[idx[i]] == DPE_STRONG;
    f[i + 1] = in[i + 1] ? a.plane[idx[i]].w : 0.0f;
  }
  int k = 0, rank[21];
#pragma unroll
  for (int i = 0; i < 21; ++i) {
    rank[i] = 0;
    k += in[i] ? 1 : 0;
    nan = nan || (in[i] && isnan(f[i]));
  }
  const int m = k / 2;
  if (nan) {  // no order: the insertion sort as it is
    float s[21];
    int n = 0;
    for (int i = 0; i < 21; ++i)
      if (in[i]) s[n++] = f[i];
    sort_small(s, n);
    a.plane[center].w = (k % 2 == 0) ? (s[m - 1] + s[m]) / 2 : s[m];
    return;
  }
#pragma unroll
  for (int i = 0; i < 21; ++i)
#pragma unroll
    for (int j = i + 1; j < 21; ++j) {
      const bool swap = f[j] < f[i];  // j comes before i
      rank[i] += in[j] && swap ? 1 : 0;
      rank[j] += in[i] && !swap ? 1 : 0;
    }
  float lo = 0.0f, hi = 0.0f;
#pragma unroll
  for (int i = 0; i < 21; ++i) {
    if (in[i] && rank[i] == m) hi = f[i];
    if (in[i] && rank[i] == m - 1) lo = f[i];
  }
  a.plane[center].w = (k % 2 == 0) ? (lo + hi) / 2 : hi;
}

// ------------------------------------------------------------------ DepthToWeak / LocalRefine
// Block-cooperative like the strong update: a block holds kCoopPix consecutive pixels of one row
// and kCoopLanes threads per pixel.  The pixel's reference window and its per-sample costs live
// in shared memory; one lane per pixel takes the decision.
//   * DepthToWeak: the lanes split the 61 disparity samples.  (One evaluation per turn of a loop over a
//     pool of the warp's samples keeps every thread busy but no faster: its threads then read different
//     sources in a turn, 48.8 against 49.0 ms below.)
//   * LocalRefine: first the current plane against its sources.  The refinement replaces the depth only
//     when the cost falls by more than 0.1, and costs are not negative: a pixel whose cost is at most
//     0.1 is done (nearly all are on textured surfaces).  The others' samples are one pool over the
//     warp's 32 threads: first each against its heaviest source, which alone rules out most (a sample
//     counts only if its full cost, no less than that part, is 0.1 below the current one), then the
//     others against the other sources; a source's samples next to each other (they lie along one
//     line of its image).  With a negative geom_factor costs can be negative: then every sample in the
//     depth range is evaluated against every source (lr_bounds).
// LocalRefine on a 1600x1200 view: first call with 10 sources 12.7 -> 3.3 ms, geometric call with 9
// 14.4 -> 9.8 ms (13.7 without the heaviest source first); 801x603 3.9 -> 0.9 ms.
struct SweepPixel {
  float4 win[kWinPairs];
  float rc[kWinTaps];   // until the window sums: w (r - c)^2 per tap
  float4 pl;
  uint4 vw;
  float center, inv_wsum, mean_r, var_r;
  float depth, base_line, weight_normal, disp;
  float cost_now;       // LocalRefine: the current plane's cost,
  uint32_t open;        // the samples that may still replace it (bit pd + 5),
  int first;            // and the position in act of the heaviest source
  int act[kMaxSrc];
  int na, ok;           // ok: the sweep runs for this pixel
  float pc[64];         // DepthToWeak: the 61 sample costs
};
enum { kSwTaps, kSwSums, kSwEval, kSwDecide, kSwEval1, kSwDrop, kSwEval2, kSwDecide2, kSweepPhases };
// LocalRefine's shared bytes: the pixels, then per pixel 12 planes (the current one, then the 11
// samples) x n = N - 1 sources of (NCC, geometric cost).
__host__ __device__ inline size_t local_refine_smem_bytes(int n) {
  return sizeof(SweepPixel) * kCoopPix + sizeof(float2) * (size_t)kCoopPix * 12 * n;
}

struct SweepCtx {
  const PMArgs *a;
  int slot, lane, px, py, center;
  bool live;  // inside the image
  SweepPixel *P, *W0;  // this thread's pixel, and its warp's first
  float2 *items, *items0;  // LocalRefine: [12][n] (NCC, geometric cost) of this pixel, and of the warp's first
  int kid;
  __device__ __forceinline__ SmemWindow window(const SweepPixel &Q) const {
    return SmemWindow{Q.win, Q.center, Q.inv_wsum, Q.mean_r, Q.var_r, a->counters ? a->counters + 2 * kid : nullptr};
  }
};
__device__ __forceinline__ SweepCtx sweep_ctx(const Launch &lc, void *smem, int kid) {
  const Blk B = resolve<kGridFull>(lc);
  SweepCtx c;
  c.a = B.a;
  c.slot = (int)threadIdx.x / kCoopLanes;
  c.lane = (int)threadIdx.x % kCoopLanes;
  c.px = B.x * kCoopPix + c.slot;
  c.py = B.y;
  c.center = c.py * B.a->W + c.px;
  c.live = c.px < B.a->W && c.py < B.a->H;
  SweepPixel *base = static_cast<SweepPixel *>(smem);
  const int first = c.slot & ~(kWarpPix - 1);
  c.P = base + c.slot;
  c.W0 = base + first;
  float2 *items = reinterpret_cast<float2 *>(base + kCoopPix);
  c.items = items + (size_t)c.slot * 12 * (B.a->N - 1);
  c.items0 = items + (size_t)first * 12 * (B.a->N - 1);
  c.kid = kid;
  return c;
}

// The window taps, split over the lanes (as strong_taps).
__device__ __forceinline__ void sweep_taps(const SweepCtx &c) {
  if (!c.live) return;
  const PMArgs &a = *c.a;
  const int r = a.P.strong_radius, inc = a.P.strong_increment, side = 2 * r / inc + 1;
  const float center = texel(a, 0, c.px, c.py);
  for (int k = c.lane; k < side * side; k += kCoopLanes) {
    const int i = -r + (k / side) * inc, j = -r + (k % side) * inc;
    const float rp = texel(a, 0, c.px + i, c.py + j);
    const float w = bilateral_weight((float)i, (float)j, rp, center, a.P.sigma_spatial, a.P.sigma_color);
    const float rcv = rp - center, wr = w * rcv;
    win_store(c.P->win, k, w, wr);
    c.P->rc[k] = wr * rcv;
  }
  if (c.lane == 0) c.P->center = center;
}

// Window sums; the prologue's plane, baseline, weights and selected sources (DPE.cu:2619-2660,
// 2767-2806) (lane 0).  (The reference's DepthToWeak also costs the current plane here and never reads
// the result; it is not computed.)
__device__ __forceinline__ void sweep_sums(const SweepCtx &c) {
  if (c.lane != 0) return;
  SweepPixel &P = *c.P;
  P.ok = 0;
  P.na = 0;
  if (!c.live) return;
  const PMArgs &a = *c.a;
  const int r = a.P.strong_radius, inc = a.P.strong_increment, side = 2 * r / inc + 1;
  float sw = 0.f, swr = 0.f, swrr = 0.f;
  for (int k = 0; k < side * side; ++k) {
    const float2 t = win_tap(P.win, k);
    sw += t.x; swr += t.y; swrr += P.rc[k];
  }
  P.inv_wsum = 1.0f / sw;
  P.mean_r = swr * P.inv_wsum;
  P.var_r = swrr * P.inv_wsum - P.mean_r * P.mean_r;
  P.pl = normal_to_ref(a.cam[0], a.plane[c.center]);
  P.depth = P.pl.w;
  const uint32_t views = a.views[c.center];
  P.vw = a.vweight[c.center];
  float base_line = 0.0f, weight_normal = 0.0f;
  int valid = 0, na = 0;
  for (int si = 1; si < a.N; ++si) {
    const int vi = si - 1;
    if (!isSet(views, vi)) continue;
    weight_normal += vweight_at(P.vw, vi);
    const float d0 = a.cam[0].c[0] - a.cam[si].c[0], d1 = a.cam[0].c[1] - a.cam[si].c[1], d2 = a.cam[0].c[2] - a.cam[si].c[2];
    const double tv = d0 * d0 + d1 * d1 + d2 * d2;
    base_line += sqrtf((float)tv);
    valid++;
    P.act[na++] = vi;
  }
  P.na = na;
  P.ok = P.depth != 0 && valid != 0;
  P.weight_normal = weight_normal;
  if (P.ok) {
    P.base_line = base_line / valid;
    P.disp = a.cam[0].K[0] * P.base_line / P.depth;
  }
}
__device__ __forceinline__ float sweep_depth(const PMArgs &a, const SweepPixel &P, int pd) {
  return a.cam[0].K[0] * P.base_line / (P.disp + pd);
}

// DepthToWeak (DPE.cu:2597-2751): the lanes split the samples; a sample's costs over the selected sources
// are added on one lane in source order (DPE.cu:2676-2700).
template <int kStage>
__device__ __forceinline__ void d2w_eval(const SweepCtx &c) {
  SweepPixel &P = *c.P;
  if (!P.ok) return;
  const PMArgs &a = *c.a;
  const SmemWindow rw = c.window(P);
  constexpr int R = 30, NS = 61;
  for (int s = c.lane; s < NS; s += kCoopLanes) {
    const float pdep = sweep_depth(a, P, s - R);
    float v = 2.0f;
    if (!(pdep < a.P.depth_min || pdep > a.P.depth_max)) {
      float4 t = P.pl;
      t.w = dist_to_origin(a.cam[0], c.px, c.py, pdep, t);
      float cost = 0.0f;
      for (int q = 0; q < P.na; ++q) {
        const int vi = P.act[q];
        float tc = ncc_strong<kStage, true>(a, c.px, c.py, vi + 1, t, rw);
        if (a.P.geom_consistency) tc += a.P.geom_factor * geom_cost(a, c.px, c.py, vi + 1, t);
        cost += tc * vweight_at(P.vw, vi);
      }
      v = cvmin(2.0f, cost / P.weight_normal);
    }
    P.pc[s] = v;
  }
}
__device__ __forceinline__ void d2w_decide(const SweepCtx &c) {
  if (!c.live || c.lane != 0) return;
  const PMArgs &a = *c.a;
  const int W = a.W, H = a.H, margin = 6;
  const float *pc = c.P->pc;
  if (c.px < margin || c.py < margin || c.px >= W - margin || c.py >= H - margin || !c.P->ok) {
    a.weak[c.center] = DPE_UNKNOWN;
    return;
  }
  constexpr int R = 30, NS = 61;
  int peaks = 0, min_peak = 0;
  float min_cost = 2.0f;
  uint64_t peak_mask = 0;
  for (int i = 2; i < NS - 2; ++i)
    if (pc[i - 1] > pc[i] && pc[i + 1] > pc[i]) {
      peak_mask |= 1ull << i; peaks++;
      if (pc[i] < min_cost) { min_peak = i; min_cost = pc[i]; }
    }
  uint8_t res;
  if (abs(min_peak - R) > a.P.weak_peak_radius || pc[min_peak] > 0.5f) res = DPE_WEAK;
  else if (peaks == 1) res = pc[min_peak] <= 0.15f ? DPE_STRONG : DPE_WEAK;
  else {
    float var = 0.0f;
    for (int i = 2; i < NS - 2; ++i)
      if (((peak_mask >> i) & 1ull) && i != min_peak) { const float d = pc[i] - min_cost; var += d * d; }
    var = sqrtf(var);
    var /= (peaks - 1);
    res = var > 0.2f ? DPE_STRONG : DPE_WEAK;
  }
  a.weak[c.center] = res;
}
// The margin pixels take no window or sweep: every phase skips them through `live`.
__device__ __forceinline__ SweepCtx d2w_ctx(const Launch &lc, void *smem) {
  SweepCtx c = sweep_ctx(lc, smem, KID_DEPTH_TO_WEAK);
  const int margin = 6;
  if (c.live && (c.px < margin || c.py < margin || c.px >= c.a->W - margin || c.py >= c.a->H - margin)) {
    if (c.lane == 0) c.a->weak[c.center] = DPE_UNKNOWN;
    c.live = false;
  }
  return c;
}

// LocalRefine (DPE.cu:2753-2839): every (plane, selected source) pair of a stage is one item of the
// warp's pool; plane 0 is the current one, planes 1..11 the disparity samples -5..5.
//   stage 0: the current plane against the selected sources
//   stage 1: the open samples against their pixel's heaviest source
//   stage 2: the samples still open against the other sources
__device__ __forceinline__ int dpe_popc(uint32_t v) {
#ifdef __CUDA_ARCH__
  return __popc(v);
#else
  int n = 0;
  for (; v; v &= v - 1) ++n;
  return n;
#endif
}
__device__ __forceinline__ int lr_items(const SweepPixel &P, int stage) {
  return !P.ok ? 0 : stage == 0 ? P.na : dpe_popc(P.open) * (stage == 1 ? 1 : P.na - 1);
}
template <int kStage>
__device__ __forceinline__ void lr_eval(const SweepCtx &c, int stage) {
  const PMArgs &a = *c.a;
  const int n = a.N - 1, px0 = c.px - (c.slot & (kWarpPix - 1));
  const bool geom = a.P.geom_consistency != 0;
  int total = 0;
  for (int k = 0; k < kWarpPix; ++k) total += lr_items(c.W0[k], stage);
  // rounds of 32 items; the barrier joins the warp for each (a warp that has come apart evaluates piece
  // by piece: 22.0 against 13.7 ms on the geometric call)
  for (int i0 = 0; i0 < total; i0 += 32) {
    DPE_WARP_BARRIER();
    int i = i0 + ((int)threadIdx.x & 31), k = 0;
    if (i >= total) continue;
    while (i >= lr_items(c.W0[k], stage)) i -= lr_items(c.W0[k++], stage);
    const SweepPixel &P = c.W0[k];
    int q = i, h = 0;
    float pdep = P.depth;
    if (stage > 0) {
      const int m = dpe_popc(P.open);
      q = i / m;
      uint32_t left = P.open;
      for (int skip = i - q * m; skip > 0; --skip) left &= left - 1;
      int bit = 0;
      while (!((left >> bit) & 1u)) ++bit;
      h = bit + 1;
      if (stage == 1) q = P.first;
      else if (q >= P.first) ++q;
      pdep = sweep_depth(a, P, h - 6);
    }
    const int px = px0 + k, si = P.act[q] + 1;
    float4 t = P.pl;
    t.w = dist_to_origin(a.cam[0], px, c.py, pdep, t);
    const float ncc = ncc_strong<kStage, true>(a, px, c.py, si, t, c.window(P));
    c.items0[((size_t)k * 12 + h) * n + q] = make_float2(ncc, geom ? geom_cost(a, px, c.py, si, t) : 0.0f);
  }
}
// Whether a sum of a plane's costs bounds it from below: the NCC is in [0, 2], the geometric cost in [0, 3].
__device__ __forceinline__ bool lr_bounds(const PMArgs &a) {
  return !(a.P.geom_consistency && a.P.geom_factor < 0.0f);
}
// The current cost, summed in the reference's order, and the samples in the depth range; a pixel that
// no sample can change is closed.
__device__ __forceinline__ void lr_current(const SweepCtx &c) {
  if (c.lane != 0 || !c.P->ok) return;
  const PMArgs &a = *c.a;
  SweepPixel &P = *c.P;
  if (P.weight_normal == 0) { P.ok = 0; return; }
  const bool geom = a.P.geom_consistency != 0;
  float cost_now = 0.0f;
  int heaviest = -1;
  P.first = 0;
  for (int q = 0; q < P.na; ++q) {
    const float2 e = c.items[q];
    float tc = e.x;
    const int w = vweight_at(P.vw, P.act[q]);
    if (geom) tc += a.P.geom_factor * e.y;
    cost_now += tc * w;
    if (w > heaviest) { heaviest = w; P.first = q; }
  }
  cost_now /= P.weight_normal;
  P.cost_now = cost_now;
  if (lr_bounds(a) && !((double)cost_now > 0.1)) { P.ok = 0; return; }
  uint32_t open = 0;
  for (int pd = -5; pd <= 5; ++pd) {
    const float pdep = sweep_depth(a, P, pd);
    if (!(pdep < a.P.depth_min || pdep > a.P.depth_max)) open |= 1u << (pd + 5);
  }
  P.open = open;
}
// A sample's weighted cost over sources q0 .. q1 - 1 in the reference's order.
__device__ __forceinline__ float lr_cost(const SweepCtx &c, int pd, int q0, int q1) {
  const PMArgs &a = *c.a;
  const SweepPixel &P = *c.P;
  const float2 *row = c.items + (pd + 6) * (a.N - 1);
  const bool geom = a.P.geom_consistency != 0;
  float tc = 0.0f;
  for (int q = q0; q < q1; ++q) {
    const int w = vweight_at(P.vw, P.act[q]);
    tc += row[q].x * w;
    if (geom) tc += a.P.geom_factor * row[q].y * w;
  }
  return tc / P.weight_normal;
}
__device__ __forceinline__ void lr_drop(const SweepCtx &c) {
  if (c.lane != 0 || !c.P->ok || !lr_bounds(*c.a)) return;
  SweepPixel &P = *c.P;
  for (int pd = -5; pd <= 5; ++pd)
    if (((P.open >> (pd + 5)) & 1u) && !((double)(P.cost_now - lr_cost(c, pd, P.first, P.first + 1)) > 0.1))
      P.open &= ~(1u << (pd + 5));
  if (!P.open) P.ok = 0;
}
// The best open sample.  The ones that bounds dropped would not change the outcome: the depth changes only when the
// smallest cost is more than 0.1 below the current one, and a dropped sample's is not.
__device__ __forceinline__ void lr_decide(const SweepCtx &c) {
  if (c.lane != 0 || !c.P->ok) return;
  const SweepPixel &P = *c.P;
  float min_cost = 2.0f, best = P.depth;
  for (int pd = -5; pd <= 5; ++pd) {
    if (!((P.open >> (pd + 5)) & 1u)) continue;
    const float tc = lr_cost(c, pd, 0, P.na);
    if (tc < min_cost) { min_cost = tc; best = sweep_depth(*c.a, P, pd); }
  }
  if ((double)(P.cost_now - min_cost) > 0.1) c.a->plane[c.center].w = best;
}

// One phase for one thread (host builds run the phases in lock-step over a block).
template <int kStage>
__device__ __forceinline__ void depth_to_weak_phase(int phase, const Launch &lc, void *smem) {
  const SweepCtx c = d2w_ctx(lc, smem);
  switch (phase) {
    case kSwTaps: sweep_taps(c); break;
    case kSwSums: sweep_sums(c); break;
    case kSwEval: d2w_eval<kStage>(c); break;
    case kSwDecide: d2w_decide(c); break;
    default: break;
  }
}
template <int kStage>
__device__ __forceinline__ void local_refine_phase(int phase, const Launch &lc, void *smem) {
  const SweepCtx c = sweep_ctx(lc, smem, KID_LOCAL_REFINE);
  switch (phase) {
    case kSwTaps: sweep_taps(c); break;
    case kSwSums: sweep_sums(c); break;
    case kSwEval: lr_eval<kStage>(c, 0); break;
    case kSwDecide: lr_current(c); break;
    case kSwEval1: lr_eval<kStage>(c, 1); break;
    case kSwDrop: lr_drop(c); break;
    case kSwEval2: lr_eval<kStage>(c, 2); break;
    default: lr_decide(c); break;
  }
}

// Grid: ((W + 15) / 16, H) blocks of kCoopThreads.
template <int kStage>
__global__ void __launch_bounds__(kCoopThreads, DPE_SWEEP_MIN_BLOCKS) k_depth_to_weak(const Launch lc) {
  __shared__ SweepPixel sp[kCoopPix];
  const SweepCtx c = d2w_ctx(lc, sp);
  sweep_taps(c);
  __syncthreads();
  sweep_sums(c);
  __syncthreads();
  d2w_eval<kStage>(c);
  __syncthreads();
  d2w_decide(c);
}
// LocalRefine: the same grid, local_refine_smem_bytes(N - 1) dynamic shared bytes.
template <int kStage>
__global__ void __launch_bounds__(kCoopThreads, DPE_LR_MIN_BLOCKS) k_local_refine(const Launch lc) {
  extern __shared__ float4 lr_smem[];
  const SweepCtx c = sweep_ctx(lc, lr_smem, KID_LOCAL_REFINE);
  sweep_taps(c);
  __syncthreads();
  sweep_sums(c);
  __syncthreads();
#ifdef __CUDA_ARCH__
#pragma unroll 1
#endif
  for (int stage = 0; stage < 3; ++stage) {  // one copy of the evaluation
    lr_eval<kStage>(c, stage);
    __syncthreads();
    if (stage == 0) lr_current(c);
    else if (stage == 1) lr_drop(c);
    else lr_decide(c);
    // the whole block is done (a pixel's first lane has just written its ok; the others read it after this)
    if (!__syncthreads_or(c.lane == 0 && c.P->ok)) return;
  }
}

}  // namespace dpe
