// edges.cu -- the edge map of EdgeSegment (DPE.cpp:136-250, mode 0 with use_canny) on the GPU.
//
// GetProblemEdges (main.cpp:166-197) makes the edge map of a pyramid level from the level image
// converted to 8 bits: EdgeSegment takes the median of its histogram (DPE.cpp:193-216), runs
// cv::Canny with thresholds (1 - 0.67) * median and median, a 3x3 aperture and the L2 gradient
// norm (DPE.cpp:217-221), leaves the map at its size (the resize to the same size and the
// threshold at 4 change nothing on a 0 / 255 map) and clears border pixels whose inner neighbour
// is clear (DPE.cpp:239-250).
//
// Canny follows the published algorithm as OpenCV (4.x) implements it:
//   - Sobel derivatives with a replicated border; squared L2 magnitude dx^2 + dy^2 in integers,
//     compared with squared integer thresholds;
//   - non-maximum suppression along the gradient sector, chosen by the fixed-point tangent of
//     22.5 degrees (round(tan(pi/8) * 2^15)); the magnitude must exceed the neighbour before the
//     pixel and be >= the one after it (> both on the diagonals); outside the image the magnitude
//     is 0;
//   - hysteresis: a pixel that survives suppression with magnitude above the low threshold is an
//     edge when its 8-connected component of such pixels holds one above the high threshold.
// The hysteresis is a connected-components pass: union-find over the candidate pixels with
// atomicMin on the roots (the lock-free union of Playne and Hawick, "A new algorithm for
// parallel connected-component labelling on GPUs", IEEE TPDS 2018), then one flag per root.
#include <cooperative_groups.h>
#include <cub/cub.cuh>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <vector>

#include "ctx.h"

namespace {

constexpr int kTg22 = 13573;  // round(tan(22.5 deg) * 2^15)

// EdgeSegment's thresholds from the 8-bit histogram (DPE.cpp:193-219), as cv::Canny turns them
// into squared integer bounds for the L2 norm.
struct CannyBounds {
  int low, high;
};

__global__ void k_level_to_u8(const float *__restrict__ src, uint8_t *__restrict__ dst, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  // convertTo(CV_8UC1): round half to even, saturate
  const int v = __float2int_rn(src[i]);
  dst[i] = (uint8_t)(v < 0 ? 0 : v > 255 ? 255 : v);
}

__global__ void k_histogram(const uint8_t *__restrict__ img, int n, unsigned *__restrict__ hist) {
  __shared__ unsigned h[256];
  for (int i = threadIdx.x; i < 256; i += blockDim.x) h[i] = 0;
  __syncthreads();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) atomicAdd(&h[img[i]], 1u);
  __syncthreads();
  for (int i = threadIdx.x; i < 256; i += blockDim.x)
    if (h[i]) atomicAdd(&hist[i], h[i]);
}

__global__ void k_canny_bounds(const unsigned *__restrict__ hist, int n, CannyBounds *b) {
  // the first value whose cumulative count exceeds half the pixels, over 0..254; -1 if none
  const int half = n / 2;
  int median = -1, sum = 0;
  for (int i = 0; i < 255; ++i) {
    sum += (int)hist[i];
    if (sum > half) { median = i; break; }
  }
  const int t1 = (int)((1.0f - 0.67f) * (float)median);  // (1 - sigma) * median_val in float
  const int t2 = median;
  // L2 gradient: thresholds clamped to 32767 and squared when positive; the smaller is low
  int lo = t1 > 0 ? t1 * t1 : t1;
  int hi = t2 > 0 ? t2 * t2 : t2;
  if (lo > hi) { const int t = lo; lo = hi; hi = t; }
  b->low = lo;
  b->high = hi;
}

__device__ __forceinline__ int px_clamped(const uint8_t *img, int w, int h, int x, int y) {
  x = x < 0 ? 0 : x >= w ? w - 1 : x;
  y = y < 0 ? 0 : y >= h ? h - 1 : y;
  return img[y * w + x];
}

// 3x3 Sobel with a replicated border; dx, dy packed as two int16 and the squared magnitude.
__global__ void k_canny_gradient(const uint8_t *__restrict__ img, int w, int h, short2 *__restrict__ grad,
                                 int *__restrict__ mag) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= w || y >= h) return;
  const int a = px_clamped(img, w, h, x - 1, y - 1), b = px_clamped(img, w, h, x, y - 1),
            c = px_clamped(img, w, h, x + 1, y - 1);
  const int d = px_clamped(img, w, h, x - 1, y), f = px_clamped(img, w, h, x + 1, y);
  const int g = px_clamped(img, w, h, x - 1, y + 1), k = px_clamped(img, w, h, x, y + 1),
            l = px_clamped(img, w, h, x + 1, y + 1);
  const int dx = (c + 2 * f + l) - (a + 2 * d + g);
  const int dy = (g + 2 * k + l) - (a + 2 * b + c);
  grad[y * w + x] = make_short2((short)dx, (short)dy);
  mag[y * w + x] = dx * dx + dy * dy;
}

__device__ __forceinline__ int mag_at(const int *mag, int w, int h, int x, int y) {
  return (x < 0 || x >= w || y < 0 || y >= h) ? 0 : mag[y * w + x];
}

// Non-maximum suppression.  state: 0 not a candidate, 1 candidate, 2 candidate above high.
__global__ void k_canny_suppress(const short2 *__restrict__ grad, const int *__restrict__ mag, int w, int h,
                                 const CannyBounds *__restrict__ bounds, uint8_t *__restrict__ state) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= w || y >= h) return;
  const int p = y * w + x;
  const int m = mag[p];
  const CannyBounds b = *bounds;
  uint8_t st = 0;
  if (m > b.low) {
    const int xs = grad[p].x, ys = grad[p].y;
    const long long ax = xs < 0 ? -xs : xs;
    const long long ay = (long long)(ys < 0 ? -ys : ys) << 15;
    const long long tg22x = ax * kTg22;
    bool keep;
    if (ay < tg22x) {  // near horizontal gradient: compare left and right
      keep = m > mag_at(mag, w, h, x - 1, y) && m >= mag_at(mag, w, h, x + 1, y);
    } else {
      const long long tg67x = tg22x + (ax << 16);
      if (ay > tg67x) {  // near vertical: above and below
        keep = m > mag_at(mag, w, h, x, y - 1) && m >= mag_at(mag, w, h, x, y + 1);
      } else {  // diagonal: the sign of dx * dy picks the diagonal
        const int s = (xs ^ ys) < 0 ? -1 : 1;
        keep = m > mag_at(mag, w, h, x - s, y - 1) && m > mag_at(mag, w, h, x + s, y + 1);
      }
    }
    if (keep) st = m > b.high ? 2 : 1;
  }
  state[p] = st;
}

__device__ __forceinline__ int uf_find(const int *parent, int i) {
  int p = parent[i];
  while (p != i) {  // indices strictly decrease along the chain
    i = p;
    p = parent[i];
  }
  return i;
}

// Merge the two sets: the larger root is pointed at the smaller by atomicMin; a failed attempt
// (the root moved meanwhile) retries from the new value.  Every retry lowers a root index, so the
// loop ends; the bound below only guards the impossible case.
__device__ __forceinline__ void uf_union(int *parent, int a, int b, int *error) {
  for (int it = 0; it < (1 << 26); ++it) {
    a = uf_find(parent, a);
    b = uf_find(parent, b);
    if (a == b) return;
    if (a < b) { const int t = a; a = b; b = t; }  // a > b: link a under b
    const int old = atomicMin(&parent[a], b);
    if (old == a) return;
    a = old;
  }
  atomicExch(error, 1);
}

__global__ void k_cc_init(const uint8_t *__restrict__ state, int n, int *__restrict__ parent) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < n) parent[p] = state[p] ? p : -1;
}

// 8-connectivity: each candidate joins its candidate neighbours before it in raster order.
__global__ void k_cc_union(const uint8_t *__restrict__ state, int w, int h, int *parent, int *error) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= w || y >= h) return;
  const int p = y * w + x;
  if (!state[p]) return;
  if (x > 0 && state[p - 1]) uf_union(parent, p, p - 1, error);
  if (y > 0) {
    if (x > 0 && state[p - w - 1]) uf_union(parent, p, p - w - 1, error);
    if (state[p - w]) uf_union(parent, p, p - w, error);
    if (x + 1 < w && state[p - w + 1]) uf_union(parent, p, p - w + 1, error);
  }
}

__global__ void k_cc_mark(const uint8_t *__restrict__ state, int n, const int *parent, uint8_t *__restrict__ strong) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < n && state[p] == 2) strong[uf_find(parent, p)] = 1;
}

__global__ void k_cc_output(const uint8_t *__restrict__ state, int n, const int *parent,
                            const uint8_t *__restrict__ strong, uint8_t *__restrict__ edge) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  edge[p] = (state[p] && strong[uf_find(parent, p)]) ? 255 : 0;
}

// DPE.cpp:239-250: rows first (left and right columns), then columns (top and bottom rows), each
// in the reference's statement order.
__global__ void k_border_rows(uint8_t *d, int w, int h) {
  const int y = blockIdx.x * blockDim.x + threadIdx.x;
  if (y >= h || w < 2) return;
  uint8_t *r = d + (size_t)y * w;
  if (r[1] == 0) r[0] = 0;
  if (r[w - 2] == 0) r[w - 1] = 0;
}
__global__ void k_border_cols(uint8_t *d, int w, int h) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= w || h < 2) return;
  if (d[(size_t)w + x] == 0) d[x] = 0;
  if (d[(size_t)(h - 2) * w + x] == 0) d[(size_t)(h - 1) * w + x] = 0;
}


// =============================================================================================
// The label map of EdgeSegment (DPE.cpp:136-291, mode 1 without Canny), as GetProblemEdges asks
// for it (main.cpp:199-214): from the full-resolution 8-bit image, halved (high_res_img) and
// halved again, a Roberts gradient thresholded at robthr, Connect's labelling, Hough segments
// drawn across every large weak region's outer border, the map resized to the level, thresholded
// and border-ruled, labelled again, and regions up to weak_tex_num pixels marked -1.
// OpenCV's resize, HoughLinesP and line are restated in OpenCV's integer forms (the CPU
// restatement in the test oracle states each rule), so the map is OpenCV's bit for bit.
// =============================================================================================

// cv::resize INTER_LINEAR, 8-bit: source coordinate (d + 0.5) * scale - 0.5 in double rounded to
// float, 11-bit weights rounded half to even; horizontal weights and columns clamped at the
// borders, vertical weights kept and only the rows clamped; the vertical pass in OpenCV's 16-bit
// form.  Explicit roundings keep the compiler from contracting any step.
__device__ __forceinline__ void lin_coeff(int d, double scale, int ssize, bool clamp_weight, int &s0, int &s1,
                                          int &w0, int &w1) {
  float f = __double2float_rn(__dsub_rn(__dmul_rn((double)d + 0.5, scale), 0.5));
  int si = (int)floorf(f);
  f = __fsub_rn(f, (float)si);
  if (clamp_weight) {
    if (si < 0) { f = 0.f; si = 0; }
    if (si >= ssize - 1) { f = 0.f; si = ssize - 1; }
    s0 = si;
    s1 = si + 1 < ssize ? si + 1 : ssize - 1;
  } else {
    s0 = si < 0 ? 0 : si > ssize - 1 ? ssize - 1 : si;
    s1 = si + 1 < 0 ? 0 : si + 1 > ssize - 1 ? ssize - 1 : si + 1;
  }
  w0 = __float2int_rn(__fmul_rn(__fsub_rn(1.f, f), 2048.f));
  w1 = __float2int_rn(__fmul_rn(f, 2048.f));
}

__global__ void k_resize_u8(const uint8_t *__restrict__ src, int sw, int sh, uint8_t *__restrict__ dst, int dw,
                            int dh, double xscale, double yscale) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= dw || y >= dh) return;
  int xa, xb, a0, a1, ya, yb, b0, b1;
  lin_coeff(x, xscale, sw, true, xa, xb, a0, a1);
  lin_coeff(y, yscale, sh, false, ya, yb, b0, b1);
  const uint8_t *r0 = src + (size_t)ya * sw, *r1 = src + (size_t)yb * sw;
  const int h0 = r0[xa] * a0 + r0[xb] * a1, h1 = r1[xa] * a0 + r1[xb] * a1;
  const int v = (((b0 * (h0 >> 4)) >> 16) + ((b1 * (h1 >> 4)) >> 16) + 2) >> 2;
  dst[(size_t)y * dw + x] = (uint8_t)(v < 0 ? 0 : v > 255 ? 255 : v);
}

// Roberts (DPE.cpp:9-25) then cv::threshold(robthr, 255, BINARY): the magnitude is the low byte of
// the truncated root, border pixels use t1 = t2 = 50.
__global__ void k_roberts_threshold(const uint8_t *__restrict__ s, int cols, int rows, int thr, uint8_t *__restrict__ d) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y * blockDim.y + threadIdx.y;
  if (j >= cols || i >= rows) return;
  int t1 = 50, t2 = 50;
  if (i > 0 && i < rows - 1 && j > 0 && j < cols - 1) {
    t1 = s[(size_t)i * cols + j] - s[(size_t)(i + 1) * cols + j + 1];
    t2 = s[(size_t)(i + 1) * cols + j] - s[(size_t)i * cols + j + 1];
  }
  const uint8_t m = (uint8_t)(int)sqrt((double)(t1 * t1 + t2 * t2));
  d[(size_t)i * cols + j] = m > thr ? 255 : 0;
}

__global__ void k_threshold(uint8_t *d, int n, int thr) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < n) d[p] = d[p] > thr ? 255 : 0;
}

// ---- Connect (DPE.cpp:27-134) -------------------------------------------------------------
// One CTA walks the rows in order (each row's provisional labels need the previous row's).  In a
// row a pixel opens a new label when it joins neither its left nor its upper neighbour; new labels
// are numbered by a block prefix count.  Along a run of left-joined pixels the provisional label
// is the running minimum of the opening label and the upper labels where the pixel joins upwards:
// a segmented inclusive min-scan, restarted at each pixel without a left join.  A pixel joined to
// both neighbours with different labels records the join connection[larger] = smaller; the
// reference overwrites earlier joins of the same label, so only the last in raster order counts,
// kept as atomicMax of (pixel index << 32 | smaller label).
// The scan also counts the openings: within a run only its first pixel opens, so a run without an upper
// join takes the label of the last opening up to it.  Each thread takes kConnectItems neighbouring
// pixels, so a row of up to 2048 is one step of one scan; the step's length is its barriers and the
// loads behind them, not its pixels.  (With a pixel per thread and a scan each for the count and the
// minimum, a 1600x1200 map took 5.2 ms more than a 400x300 one; now 1.9 ms.)
// Both grow with the warps of the block, so a row takes the smallest block that holds it in one step.
// Label maps in all, with 512 threads for every row and with 32, 128 or 512: 0.69 -> 0.62 ms at 100x75,
// 1.03 -> 0.93 at 200x150, 1.97 -> 1.73 at 400x300, 5.16 -> 5.08 at 800x600, 16.8 -> 16.6 at 1600x1200.
constexpr int kConnectItems = 4;

struct RunScan {
  int start;  // a run starts within the scanned prefix
  int v;      // smallest upper label since
  int opens;  // openings
};
struct RunScanOp {
  __device__ __forceinline__ RunScan operator()(const RunScan &a, const RunScan &b) const {
    return RunScan{a.start | b.start, b.start ? b.v : min(a.v, b.v), a.opens + b.opens};
  }
};

template <int kThreads>
__global__ void __launch_bounds__(kThreads) k_connect_rows(const uint8_t *__restrict__ img, int cols, int rows,
                                                                 int *__restrict__ lab,
                                                                 unsigned long long *__restrict__ join, int *nlab) {
  typedef cub::BlockScan<RunScan, kThreads> Scan;
  __shared__ typename Scan::TempStorage ts;
  __shared__ int s_next, s_carry, s_last[kThreads];
  const int tid = threadIdx.x;
  if (tid == 0) {
    s_next = 1;
    s_carry = 0;
  }
  __syncthreads();
  for (int y = 0; y < rows; ++y) {
    for (int base = 0; base < cols; base += kThreads * kConnectItems) {
      const int x0 = base + tid * kConnectItems;
      const size_t p0 = (size_t)y * cols + x0;
      bool in[kConnectItems], leftj[kConnectItems], upj[kConnectItems], labelled[kConnectItems], opens[kConnectItems];
      int up[kConnectItems];
      bool left_zero = x0 > 0 && x0 <= cols && img[p0 - 1] == 0;
      RunScan agg{0, INT_MAX, 0};
#pragma unroll
      for (int i = 0; i < kConnectItems; ++i) {
        in[i] = x0 + i < cols;
        const int v = in[i] ? img[p0 + i] : 255;
        labelled[i] = in[i] && v != 255;
        const bool zero = in[i] && v == 0;
        leftj[i] = zero && left_zero;
        upj[i] = zero && y > 0 && img[p0 + i - cols] == 0;
        up[i] = upj[i] ? lab[p0 + i - cols] : INT_MAX;  // this thread wrote it
        opens[i] = labelled[i] && !leftj[i] && !upj[i];
        left_zero = zero;
        agg = RunScanOp()(agg, RunScan{leftj[i] ? 0 : 1, up[i], opens[i] ? 1 : 0});
      }
      RunScan pre, total;
      Scan(ts).ExclusiveScan(agg, pre, RunScan{0, INT_MAX, 0}, RunScanOp(), total);
      const int next = s_next, carry = s_carry;
      int run[kConnectItems], last = 0;
      RunScan o = pre;
#pragma unroll
      for (int i = 0; i < kConnectItems; ++i) {
        o = RunScanOp()(o, RunScan{leftj[i] ? 0 : 1, up[i], opens[i] ? 1 : 0});
        run[i] = !o.start ? min(carry, o.v) : o.v != INT_MAX ? o.v : next + o.opens - 1;
        if (!labelled[i]) run[i] = 0;
        if (in[i]) {
          lab[p0 + i] = run[i];
          last = run[i];
        }
      }
      s_last[tid] = last;
      __syncthreads();  // this step's last labels are written; s_next and s_carry are read
      int left = tid > 0 ? s_last[tid - 1] : carry;
#pragma unroll
      for (int i = 0; i < kConnectItems; ++i) {
        if (leftj[i] && upj[i] && left != up[i]) {
          const int big = left > up[i] ? left : up[i], small = left > up[i] ? up[i] : left;
          atomicMax(&join[big], ((unsigned long long)(p0 + i) << 32) | (unsigned)small);
        }
        left = run[i];
      }
      const int end = min(base + kThreads * kConnectItems, cols) - 1;
      if (end >= x0 && end < x0 + kConnectItems) s_carry = last;
      if (tid == 0) s_next = next + total.opens;
      __syncthreads();
    }
  }
  if (tid == 0) *nlab = s_next;
}

__global__ void k_connect_links(const unsigned long long *__restrict__ join, const int *nlab, int cap, int *conn) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= cap) return;
  conn[i] = (i < *nlab && i > 0 && join[i]) ? (int)(join[i] & 0xffffffffu) : i;
}

// chain ends by pointer doubling (every link points to a smaller label)
__global__ void k_connect_jump(const int *__restrict__ a, int *__restrict__ b, int cap) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < cap) b[i] = a[a[i]];
}

__global__ void k_connect_roots(const int *__restrict__ conn, const int *nlab, int cap, int *__restrict__ is_root) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < cap) is_root[i] = (i > 0 && i < *nlab && conn[i] == i) ? 1 : 0;
}

// final label per pixel (roots renumbered in increasing order) and the count per label
__global__ void k_connect_final(const int *__restrict__ lab, int n, const int *__restrict__ conn,
                                const int *__restrict__ rank, int *__restrict__ out, int *__restrict__ counts) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int l = lab[p];
  const int f = l == 0 ? 0 : rank[conn[l]] + 1;
  out[p] = f;
  atomicAdd(&counts[f], 1);
}

__global__ void k_mark_small(int *labels, int n, const int *__restrict__ counts, int weak_tex_num) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int l = labels[p];
  if (l != 0 && counts[l] <= weak_tex_num) labels[p] = -1;
}

// The large regions, each with a share of the border points' scratch: a region's outer border has at most
// four pixels per pixel of the region (its neighbours), and no more than the map.
struct LargeRegions {
  int n;
  unsigned long long points;
};
__global__ void k_list_large(const int *__restrict__ counts, int cap, int weak_tex_num, int *list,
                             unsigned long long *first_point, LargeRegions *large) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= 1 && k < cap && counts[k] > 0 && counts[k] >= weak_tex_num) {
    const int at = atomicAdd(&large->n, 1);
    list[at] = k;
    first_point[at] = atomicAdd(&large->points, (unsigned long long)min((long long)counts[k] * 4, (long long)cap - 1));
  }
}

// ---- HoughLinesP on one weak region's outer border, and its segments drawn --------------------
// cv::HoughLinesP(img_weak, 1, CV_PI / 180, thr, thr, thr) (DPE.cpp:185-188): OpenCV's progressive
// probabilistic Hough transform, one region per CTA or cluster of CTAs, with the results of the
// reference's sequential loop:
//   * the order of the points depends only on the generator and the number left, so a warp that has no
//     angles draws the next 32 points while the others vote;
//   * a thread owns an angle and votes for up to kVotes points at once: the counts it would see are
//     the stored ones plus its own earlier votes of the round for the same bin.  Only when some count
//     reaches the threshold does a point's argmax matter: the votes up to the first such point are
//     stored, its segment is handled, and the next round starts behind it.  Otherwise all are stored;
//   * the counts lie in shared memory, 16 bits each (kHoughMaxSide): a vote touches 180 rows, from L2 or L1 180 separate lines.  Where one CTA's shared
//     memory is too small, 2, 4 or 8 CTAs of a cluster split the angles; each keeps its own copy of the
//     mask and of the order and makes every walk, and a round exchanges only which points reached the
//     threshold and with what angle;
//   * a segment's walk looks at 16 steps of both directions at a time, and the mask is one bit per pixel.
// What bounds it is the chain of rounds of the largest border (on a 1600x1200 view 30 k points, 17 k of
// them voting, 2088 segments).  One point at a time, every load from L2, took 68 ms; rounds with the counts
// in global memory 17 ms; now 11 ms, a chain of short dependent pieces: 900 cycles of a round to vote,
// 1100 at its barrier, 2500 of a segment for its walk.
struct HoughArgs {
  const int *labels;  // first labelling, w x h
  const int *regions; // region labels, one per CTA or cluster
  const unsigned long long *first_point;  // per region: where its points start
  int w, h, threshold, line_length, line_gap, numangle, numrho;
  const float2 *tab;  // (cos, sin) / rho in float, from the host's libm as OpenCV computes it
  unsigned *mask;     // per CTA: w*h bits; null: in shared memory (it is there whenever the counts are)
  int2 *points;       // per region and CTA of its cluster: the border, point_cap in all for one CTA each
  unsigned long long point_cap;
  short *accum;       // per region: numangle*len counts; null: in shared memory
  int first, len;     // the bins that a point of the image can vote for
  int split;          // CTAs of a cluster that share a region's angles
  int4 *lines;        // per CTA: line_cap
  int line_cap;
  uint8_t *dst;       // the thresholded Roberts map the segments are drawn on
  int *error;
};

__device__ __forceinline__ int hough_bin(const HoughArgs &a, float2 t, float x, float y) {
  return __float2int_rn(__fadd_rn(__fmul_rn(x, t.x), __fmul_rn(y, t.y))) + (a.numrho - 1) / 2;
}
// A pixel of a walk in 32 bits, x below y (both fit 16 bits, kHoughMaxSide), and its coordinates as floats:
// 2^23 + k has k in its low bits, so an integer operation and an exact subtraction replace a conversion, which
// has an eighth of their rate and would run for every pixel in every angle's thread (label maps of a
// 1600x1200 image at scales 0 and 2: 17.1 and 13.1 ms with conversions from 16 bits, 16.8 and 12.8 ms so).
__device__ __forceinline__ unsigned walk_pack(int2 q) { return (unsigned)q.x | (unsigned)q.y << 16; }
__device__ __forceinline__ int hough_bin(const HoughArgs &a, float2 t, unsigned packed) {
  return hough_bin(a, t, __uint_as_float(0x4B000000u | (packed & 0xFFFFu)) - 8388608.0f,
                   __uint_as_float(0x4B000000u | packed >> 16) - 8388608.0f);
}

__device__ void draw_line8(uint8_t *img, int width, int x1, int y1, int x2, int y2) {
  int dx = x2 - x1, dy = y2 - y1;
  if (dx < 0) { int t = x1; x1 = x2; x2 = t; t = y1; y1 = y2; y2 = t; dx = -dx; dy = -dy; }
  long long step_y = width, step_x = 1;
  if (dy < 0) { dy = -dy; step_y = -step_y; }
  if (dy > dx) { int t = dx; dx = dy; dy = t; const long long u = step_x; step_x = step_y; step_y = u; }
  int err = dx - (dy + dy);
  const int plus_delta = dx + dx, minus_delta = -(dy + dy);
  long long p = (long long)y1 * width + x1;
  for (int c = 0; c <= dx; ++c) {
    img[p] = 255;
    const bool m = err < 0;
    err += minus_delta + (m ? plus_delta : 0);
    p += step_x + (m ? step_y : 0);
  }
}

constexpr int kHoughThreads = 256, kHoughVotes = 8, kHoughMaxSplit = 8;
// Shared bytes a CTA may take for the walk, the mask and the counts.
constexpr size_t kHoughShared = 200 * 1024;
inline size_t hough_walk_bytes(int w, int h) { return (size_t)2 * (std::max(w, h) + 2) * sizeof(unsigned); }
// Maps with a longer side than this are refused.  Up to it the 16-bit counts hold: a bin is a strip one
// pixel wide, which meets each row of a steep line (each column of a flat one) in at most two pixels, so a
// count stays within twice the longer side, 28890.
constexpr int kHoughMaxSide = 14445;
inline size_t hough_mask_words(size_t pixels) { return (pixels + 31) / 32; }

inline size_t hough_acc_bytes(int numangle, int split, int len) {
  return (size_t)((numangle + split - 1) / split) * len * sizeof(short);
}

template <int kVotes>
__global__ void __launch_bounds__(kHoughThreads) k_hough_region(const __grid_constant__ HoughArgs a) {
  extern __shared__ unsigned walk[];  // pixels withdrawn by one segment, both directions; then the mask, the counts
  typedef cub::BlockScan<int, kHoughThreads> ScanI;
  __shared__ typename ScanI::TempStorage ts_i;
  __shared__ int s_count, s_nwalk, s_nlines;
  __shared__ int2 s_pt[2][32];
  __shared__ float2 s_tab[kHoughThreads];
  // per round: each CTA's best (count, angle) of every point that reaches the threshold there
  // (and whether there is any)
  __shared__ unsigned s_key[3][kHoughMaxSplit][kVotes], s_any[3];
  namespace cg = cooperative_groups;
  const cg::cluster_group cluster = cg::this_cluster();
  const int split = a.split, rank = split > 1 ? (int)cluster.block_rank() : 0;
  auto barrier = [&]() {
    if (split > 1) cluster.sync();
    else __syncthreads();
  };
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kDrawWarp = kHoughThreads / 32 - 1;  // no angle is its (numangle is 180)
  const int region = a.regions[blockIdx.x / split];
  const int w = a.w, h = a.h, n = w * h;
  const int walk_cap = 2 * (max(w, h) + 2);
  unsigned *shared_mask = walk + walk_cap;
  unsigned *mask = a.mask ? a.mask + (size_t)blockIdx.x * ((n + 31) / 32) : shared_mask;
  const int per = (a.numangle + split - 1) / split;  // angles of this CTA: rank * per + 0 .. per - 1
  short *acc = a.accum ? a.accum + (size_t)blockIdx.x * a.numangle * a.len
                       : reinterpret_cast<short *>(shared_mask + (n + 31) / 32);
  auto masked = [&](int x, int y) {
    const int p = y * w + x;
    return ((mask[p >> 5] >> (p & 31)) & 1u) != 0;
  };
  int2 *pts = a.points + (size_t)rank * a.point_cap + a.first_point[blockIdx.x / split];
  int4 *lines = a.lines + (size_t)(blockIdx.x / split) * a.line_cap;
  // the region's outer border in raster order (DPE.cpp:168-182): not the region, 4-adjacent to it
  if (tid == 0) s_count = 0;
  __syncthreads();
  for (int base = 0; base < n; base += kHoughThreads) {
    const int p = base + tid;
    bool on = false;
    if (p < n && a.labels[p] != region) {
      const int x = p % w, y = p / w;
      on = (x > 0 && a.labels[p - 1] == region) || (x < w - 1 && a.labels[p + 1] == region) ||
           (y > 0 && a.labels[p - w] == region) || (y < h - 1 && a.labels[p + w] == region);
    }
    const unsigned bits = __ballot_sync(0xffffffffu, on);
    if (lane == 0 && p < n) mask[p >> 5] = bits;
    if (!__syncthreads_or(on)) continue;
    int pre, total;
    ScanI(ts_i).ExclusiveSum(on ? 1 : 0, pre, total);
    if (on) pts[s_count + pre] = make_int2(p % w, p / w);
    __syncthreads();
    if (tid == 0) s_count += total;
    __syncthreads();
  }
  for (int i = tid; i < per * a.len; i += kHoughThreads) acc[i] = 0;
  if (tid == 0) s_nlines = 0;
  for (int i = tid; i < 3 * kHoughMaxSplit * kVotes; i += kHoughThreads) (&s_key[0][0][0])[i] = 0;
  if (tid < 3) s_any[tid] = 0;
  if (tid < a.numangle) s_tab[tid] = a.tab[tid];
  barrier();  // every CTA's keys are ready for the others
  uint64_t state = ~0ull;  // cv::RNG((uint64)-1), the drawing warp only
  const int shift = 16;
  int left = s_count;  // points not drawn yet
  // The next m <= 32 points of the order (one warp): a drawn point's place is taken by the last one.
  // Lane i makes draw i.  The places drawn do not depend on the points, so the loads go out together; a
  // place that an earlier draw of the batch filled holds what that draw put there.
  auto draw = [&](int2 *out, int m) {
    uint64_t mine = 0;
    for (int i = 0; i < m; ++i) {
      state = (uint64_t)(unsigned)state * 4164903690u + (unsigned)(state >> 32);
      if (i == lane) mine = state;
    }
    const bool in = lane < m;
    const int end = left - lane - 1;
    const int idx = in ? (int)((unsigned)mine % (unsigned)(end + 1)) : -1;
    int2 at_idx = make_int2(0, 0), at_end = make_int2(0, 0);
    if (in) {
      at_idx = pts[idx];
      at_end = pts[end];
    }
    bool store = in;
    // rarely: a place drawn twice, or one of the last places drawn
    const unsigned same = __match_any_sync(0xffffffffu, in ? idx : -1 - lane);
    const bool clash = in && (__popc(same) > 1 || idx >= left - m);
    if (__any_sync(0xffffffffu, clash)) {
      for (int j = 0; j < m; ++j) {
        const int fill = __shfl_sync(0xffffffffu, idx, j);
        const int2 by = make_int2(__shfl_sync(0xffffffffu, at_end.x, j), __shfl_sync(0xffffffffu, at_end.y, j));
        if (lane > j) {
          if (idx == fill) at_idx = by;
          if (end == fill) at_end = by;
        } else if (lane < j && idx == fill) {
          store = false;  // a later draw fills this place
        }
      }
    }
    if (in) out[lane] = at_idx;
    if (store) pts[idx] = at_end;
    __syncwarp();
  };
  const int ang = rank * per + tid;
  const bool voter = tid < per && ang < a.numangle;
  const float2 angle = voter ? s_tab[ang] : make_float2(0.f, 0.f);
  short *row = acc + (size_t)(voter ? tid : 0) * a.len - a.first;
  int cur = min(left, 32), par = 0, buf = 0;
  if (warp == kDrawWarp) draw(s_pt[0], cur);
  left -= cur;
  __syncthreads();
  while (cur > 0) {
    const int ahead = min(left, 32);
    if (warp == kDrawWarp) draw(s_pt[buf ^ 1], ahead);
    left -= ahead;
    int start = 0;
    while (true) {
      // the next points of the batch that no segment has withdrawn (every warp looks for itself)
      bool on = false;
      if (lane >= start && lane < cur) on = masked(s_pt[buf][lane].x, s_pt[buf][lane].y);
      const unsigned all = __ballot_sync(0xffffffffu, on);
      if (!all) break;  // uniform: the mask is the same for every warp
      unsigned live = all;
      int bin[kVotes], val[kVotes], at[kVotes];
      unsigned hit = 0;
#pragma unroll
      for (int i = 0; i < kVotes; ++i) {
        at[i] = live ? __ffs(live) - 1 : -1;
        live &= live - 1;
        bin[i] = -1 - i;
        val[i] = 0;
        if (voter && at[i] >= 0) {
          const int2 pt = s_pt[buf][at[i]];
          bin[i] = hough_bin(a, angle, (float)pt.x, (float)pt.y);
          val[i] = row[bin[i]];
        }
      }
#pragma unroll
      for (int i = 0; i < kVotes; ++i) {
#pragma unroll
        for (int j = 0; j < i; ++j)
          if (bin[j] == bin[i]) val[i] = val[j];  // the latest earlier vote of the round for this bin
        val[i] += 1;
        if (voter && at[i] >= 0 && val[i] >= a.threshold) hit |= 1u << i;
      }
      // The first angle with the largest count, for every point that reaches the threshold: the count is
      // not negative there; the low byte prefers the smaller angle on ties.
      const unsigned whit = __reduce_or_sync(0xffffffffu, hit);
#pragma unroll
      for (int i = 0; i < kVotes; ++i) {
        if (!((whit >> i) & 1u)) continue;
        const unsigned key =
            __reduce_max_sync(0xffffffffu, ((hit >> i) & 1u) ? (unsigned)val[i] << 8 | (unsigned)(255 - ang) : 0u);
        if (lane < split) {  // to every CTA of the cluster
          unsigned *to = &s_key[par][rank][i];
          atomicMax(split > 1 ? cluster.map_shared_rank(to, lane) : to, key);
        }
      }
      if (whit && lane < split) atomicOr(split > 1 ? cluster.map_shared_rank(&s_any[par], lane) : &s_any[par], whit);
      barrier();
      const unsigned any = s_any[par];
      const int upto = any ? __ffs(any) : kVotes;  // votes of points before this one count now
      // the place in the batch of the last of these points
      unsigned rest = all;
      for (int i = min(upto, __popc(all)); i > 1; --i) rest &= rest - 1;
      const int final_pt = __ffs(rest) - 1;
      start = final_pt + 1;
      if (voter) {
#pragma unroll
        for (int i = 0; i < kVotes; ++i)
          if (at[i] >= 0 && i < upto) row[bin[i]] = (short)val[i];
      }
      unsigned best = 0;
      if (any)
        for (int c = 0; c < split; ++c) best = max(best, s_key[par][c][upto - 1]);
      // Free the slots of the round after next: their last readers are behind this round's barrier, their
      // next writers behind the next one's.
      const int old = par == 0 ? 2 : par - 1;
      if (warp == kDrawWarp) {
        for (int i = lane; i < kHoughMaxSplit * kVotes; i += 32) (&s_key[old][0][0])[i] = 0;
        if (lane == 0) s_any[old] = 0;
      }
      par = par == 2 ? 0 : par + 1;
      const int2 pt = s_pt[buf][final_pt];
      if (!any) continue;  // uniform
      if (warp == 0) {
        const int j = pt.x, i = pt.y;
        const float2 t = s_tab[255 - (int)(best & 255u)];
        const float fa = -t.y, fb = t.x;
        int x0 = j, y0 = i, dx0, dy0;
        bool xflag;
        if (fabsf(fa) > fabsf(fb)) {
          xflag = true;
          dx0 = fa > 0 ? 1 : -1;
          dy0 = __float2int_rn(__fdiv_rn(__fmul_rn(fb, (float)(1 << shift)), fabsf(fa)));
          y0 = (y0 << shift) + (1 << (shift - 1));
        } else {
          xflag = false;
          dy0 = fb > 0 ? 1 : -1;
          dx0 = __float2int_rn(__fdiv_rn(__fmul_rn(fa, (float)(1 << shift)), fabsf(fb)));
          x0 = (x0 << shift) + (1 << (shift - 1));
        }
        // step s of direction k; the major coordinate moves by one a step, so every step is another pixel
        // and a walk leaves the image for good
        auto step = [&](int k, int s) {
          const int x = x0 + (k ? -dx0 : dx0) * s, y = y0 + (k ? -dy0 : dy0) * s;
          return xflag ? make_int2(x, y >> shift) : make_int2(x >> shift, y);
        };
        // Half the warp per direction, 16 steps of each at a time.  Every mask pixel up to where a walk ends
        // is withdrawn, whether the segment counts or not, so one pass finds and clears them.
        const int k = lane >> 4, hl = lane & 15;
        int last = 0, nw = 0;  // last: the direction's last mask pixel so far
        bool open = true;
        for (int base = 0; __any_sync(0xffffffffu, open); base += 16) {
          const int2 q = step(k, base + hl);
          const bool in = open && q.x >= 0 && q.x < w && q.y >= 0 && q.y < h;
          const unsigned ins = __ballot_sync(0xffffffffu, in);
          const unsigned hits = __ballot_sync(0xffffffffu, in && masked(q.x, q.y));
          unsigned set = 0;
          if (open) {
            const unsigned out = ~(ins >> (16 * k)) & 0xffffu;
            const int inside = out ? __ffs(out) - 1 : 16;
            set = (hits >> (16 * k)) & ((1u << inside) - 1u);
            // reach: the steps within line_gap behind a set one (or behind the last of earlier steps); the
            // walk ends at the first that is not
            unsigned reach = set;
            for (int have = 0; have < min(a.line_gap, 15);) {
              const int by = min(have + 1, min(a.line_gap, 15) - have);
              reach |= reach << by;
              have += by;
            }
            const int tail = last + a.line_gap - base;  // the last step the earlier ones reach
            if (tail >= 0) reach |= tail >= 15 ? 0xffffu : (2u << tail) - 1u;
            const unsigned gap = ~reach & 0xffffu;
            const int stop = gap ? __ffs(gap) - 1 : 16;
            set &= (1u << stop) - 1u;
            if (set) last = base + 31 - __clz(set);
            if (stop < 16 || inside < 16) open = false;
            if (base > w + h + 36) {
              atomicExch(a.error, 1);
              open = false;
            }
          }
          // the second direction's first step is the first's: found and cleared there
          const bool m = ((set >> hl) & 1u) && !(k == 1 && base + hl == 0);
          const unsigned take = __ballot_sync(0xffffffffu, m);
          if (m) {
            const int to = nw + __popc(take & ((1u << lane) - 1u));
            if (to < walk_cap) walk[to] = walk_pack(q);
            const int p = q.y * w + q.x;
            atomicAnd(&mask[p >> 5], ~(1u << (p & 31)));
          }
          nw += __popc(take);
        }
        const int2 e = step(k, last);
        const int2 e0 = make_int2(__shfl_sync(0xffffffffu, e.x, 0), __shfl_sync(0xffffffffu, e.y, 0));
        const int2 e1 = make_int2(__shfl_sync(0xffffffffu, e.x, 16), __shfl_sync(0xffffffffu, e.y, 16));
        const bool good = abs(e1.x - e0.x) >= a.line_length || abs(e1.y - e0.y) >= a.line_length;
        if (lane == 0) {
          s_nwalk = good ? min(nw, walk_cap) : 0;
          if (good && s_nlines < a.line_cap) lines[s_nlines] = make_int4(e0.x, e0.y, e1.x, e1.y);
          if (good) s_nlines++;
        }
      }
      __syncthreads();
      // withdraw the segment's votes: each thread owns whole angle rows, so no two threads meet
      if (voter) {
        const int m = s_nwalk;
        int q = 0;
        for (; q + 4 <= m; q += 4) {  // four bins ahead of the counts they change
          int b4[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) b4[i] = hough_bin(a, angle, walk[q + i]);
#pragma unroll
          for (int i = 0; i < 4; ++i) row[b4[i]] -= 1;
        }
        for (; q < m; ++q) row[hough_bin(a, angle, walk[q])] -= 1;
      }
      __syncthreads();
    }
    __syncthreads();  // the next points are drawn, this batch's are read
    cur = ahead;
    buf ^= 1;
  }
  __syncthreads();
  if (split > 1) cluster.sync();  // no CTA leaves while another may write to its keys
  if (rank != 0) return;
  if (s_nlines > a.line_cap && tid == 0) atomicExch(a.error, 2);
  const int nl = min(s_nlines, a.line_cap);
  for (int q = tid; q < nl; q += kHoughThreads) draw_line8(a.dst, w, lines[q].x, lines[q].y, lines[q].z, lines[q].w);
}
}  // namespace

int dpe_edge_reserve(dpe_ctx *ctx, size_t pixels) {
  Arena &A = ctx->arena;
  A.get<uint8_t>("eg_u8", pixels);
  A.get<short2>("eg_grad", pixels);
  A.get<int>("eg_mag", pixels);
  A.get<uint8_t>("eg_state", pixels);
  A.get<int>("eg_parent", pixels);
  A.get<uint8_t>("eg_strong", pixels);
  A.get<unsigned>("eg_hist", 256);
  A.get<CannyBounds>("eg_bounds", 1);
  A.get<int>("eg_error", 1);
  return A.ok() ? DPE_OK : DPE_ERR_OUT_OF_MEMORY;
}

int dpe_edge_map_device(dpe_ctx *ctx, const float *level, const uint8_t *image, int w, int h, uint8_t *edge) {
  const int n = w * h;
  cudaStream_t s = ctx->stream;
  Arena &A = ctx->arena;
  uint8_t *u8 = A.get<uint8_t>("eg_u8", n);
  short2 *grad = A.get<short2>("eg_grad", n);
  int *mag = A.get<int>("eg_mag", n);
  uint8_t *state = A.get<uint8_t>("eg_state", n);
  int *parent = A.get<int>("eg_parent", n);
  uint8_t *strong = A.get<uint8_t>("eg_strong", n);
  unsigned *hist = A.get<unsigned>("eg_hist", 256);
  CannyBounds *bounds = A.get<CannyBounds>("eg_bounds", 1);
  int *error = A.get<int>("eg_error", 1);
  if (!A.ok()) return DPE_ERR_OUT_OF_MEMORY;
  const unsigned b1 = (unsigned)((n + 255) / 256);
  const dim3 bl(32, 8), g2((w + 31) / 32, (h + 7) / 8);
  if (level) {
    k_level_to_u8<<<b1, 256, 0, s>>>(level, u8, n);
    DPE_LAUNCHED("k_level_to_u8", s);
    image = u8;
  }
  DPE_TRY(cudaMemsetAsync(hist, 0, 256 * sizeof(unsigned), s));
  DPE_TRY(cudaMemsetAsync(strong, 0, (size_t)n, s));
  DPE_TRY(cudaMemsetAsync(error, 0, sizeof(int), s));
  DPE_TIMED(ctx, KID_EDGE_MAP, s, k_histogram<<<(unsigned)std::min(b1, 2u * (unsigned)ctx->sms), 256, 0, s>>>(image, n, hist));
  DPE_LAUNCHED("k_histogram", s);
  k_canny_bounds<<<1, 1, 0, s>>>(hist, n, bounds);
  DPE_LAUNCHED("k_canny_bounds", s);
  DPE_TIMED(ctx, KID_EDGE_MAP, s, k_canny_gradient<<<g2, bl, 0, s>>>(image, w, h, grad, mag));
  DPE_LAUNCHED("k_canny_gradient", s);
  DPE_TIMED(ctx, KID_EDGE_MAP, s, k_canny_suppress<<<g2, bl, 0, s>>>(grad, mag, w, h, bounds, state));
  DPE_LAUNCHED("k_canny_suppress", s);
  k_cc_init<<<b1, 256, 0, s>>>(state, n, parent);
  DPE_LAUNCHED("k_cc_init", s);
  DPE_TIMED(ctx, KID_EDGE_MAP, s, k_cc_union<<<g2, bl, 0, s>>>(state, w, h, parent, error));
  DPE_LAUNCHED("k_cc_union", s);
  k_cc_mark<<<b1, 256, 0, s>>>(state, n, parent, strong);
  DPE_LAUNCHED("k_cc_mark", s);
  DPE_TIMED(ctx, KID_EDGE_MAP, s, k_cc_output<<<b1, 256, 0, s>>>(state, n, parent, strong, edge));
  DPE_LAUNCHED("k_cc_output", s);
  k_border_rows<<<(unsigned)((h + 255) / 256), 256, 0, s>>>(edge, w, h);
  DPE_LAUNCHED("k_border_rows", s);
  k_border_cols<<<(unsigned)((w + 255) / 256), 256, 0, s>>>(edge, w, h);
  DPE_LAUNCHED("k_border_cols", s);
  return DPE_OK;
}

// The union loop's guard (never expected to trip): read after the caller has synchronised.
int dpe_edge_check(dpe_ctx *ctx) {
  int *error = ctx->arena.get<int>("eg_error", 1);
  int e = 0;
  DPE_TRY(cudaMemcpy(&e, error, sizeof(int), cudaMemcpyDeviceToHost));
  if (e) {
    dpe_set_last_error("k_cc_union", cudaErrorUnknown, __FILE__, __LINE__);
    return DPE_ERR_CUDA;
  }
  return DPE_OK;
}

extern "C" int dpe_edge_map(dpe_ctx *ctx, const uint8_t *image, int width, int height, int memory, uint8_t *edge_out) {
  if (!ctx || !image || !edge_out || width < 1 || height < 1) return DPE_ERR_INVALID_ARGUMENT;
  if (memory != DPE_MEM_HOST && memory != DPE_MEM_DEVICE) return DPE_ERR_INVALID_ARGUMENT;
  if ((size_t)width * height > (size_t)INT_MAX / 2) return DPE_ERR_INVALID_ARGUMENT;
  DPE_TRY(cudaSetDevice(ctx->device));
  cudaStream_t s = ctx->stream;
  const size_t n = (size_t)width * height;
  const uint8_t *img = image;
  uint8_t *out = edge_out;
  if (memory == DPE_MEM_HOST) {
    uint8_t *in_d = ctx->arena.get<uint8_t>("eg_in", n);
    uint8_t *out_d = ctx->arena.get<uint8_t>("eg_out", n);
    if (!ctx->arena.ok()) return DPE_ERR_OUT_OF_MEMORY;
    DPE_TRY(cudaMemcpyAsync(in_d, image, n, cudaMemcpyHostToDevice, s));
    img = in_d;
    out = out_d;
  }
  DPE_TRY(cudaEventRecord(ctx->ev0, s));
  int st = dpe_edge_map_device(ctx, nullptr, img, width, height, out);
  if (st != DPE_OK) return st;
  DPE_TRY(cudaEventRecord(ctx->ev1, s));
  if (memory == DPE_MEM_HOST) DPE_TRY(cudaMemcpyAsync(edge_out, out, n, cudaMemcpyDeviceToHost, s));
  DPE_TRY(cudaStreamSynchronize(s));
  ctx->collect();
  return dpe_edge_check(ctx);
}

// ---------------------------------------------------------------------------------------------
// Label maps on the device.
// ---------------------------------------------------------------------------------------------
namespace {

struct ConnectScratch {
  int *lab, *conn_a, *conn_b, *is_root, *rank, *nlab;
  unsigned long long *join;
  void *scan_tmp;
  size_t scan_bytes;
};

int connect_scratch(dpe_ctx *ctx, size_t pixels, ConnectScratch &c) {
  Arena &A = ctx->arena;
  const size_t cap = pixels + 1;
  c.lab = A.get<int>("lb_lab", pixels);
  c.conn_a = A.get<int>("lb_conn_a", cap);
  c.conn_b = A.get<int>("lb_conn_b", cap);
  c.is_root = A.get<int>("lb_is_root", cap);
  c.rank = A.get<int>("lb_rank", cap);
  c.nlab = A.get<int>("lb_nlab", 1);
  c.join = A.get<unsigned long long>("lb_join", cap);
  c.scan_bytes = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, c.scan_bytes, c.is_root, c.rank, (int)cap, ctx->stream);
  c.scan_tmp = A.get<uint8_t>("lb_scan_tmp", c.scan_bytes + 16);
  return A.ok() ? DPE_OK : DPE_ERR_OUT_OF_MEMORY;
}

// Connect (DPE.cpp:27-134) of a w x h map: final labels into `out`, pixels per label into
// `counts` (w*h + 1 entries, label 0 = the 255 pixels).
int connect_device(dpe_ctx *ctx, const uint8_t *img, int w, int h, ConnectScratch &c, int *out, int *counts) {
  cudaStream_t s = ctx->stream;
  const int n = w * h, cap = n + 1;
  const unsigned bn = (unsigned)((n + 255) / 256), bc = (unsigned)((cap + 255) / 256);
  DPE_TRY(cudaMemsetAsync(c.join, 0, (size_t)cap * sizeof(unsigned long long), s));
  auto rows = [&](auto threads) {  // the smallest block that holds a row in one step
    constexpr int kThreads = decltype(threads)::value;
    k_connect_rows<kThreads><<<1, kThreads, 0, s>>>(img, w, h, c.lab, c.join, c.nlab);
  };
  DPE_TIMED(ctx, KID_EDGE_LABELS, s,
            if (w <= 32 * kConnectItems) rows(std::integral_constant<int, 32>());
            else if (w <= 128 * kConnectItems) rows(std::integral_constant<int, 128>());
            else rows(std::integral_constant<int, 512>()));
  DPE_LAUNCHED("k_connect_rows", s);
  k_connect_links<<<bc, 256, 0, s>>>(c.join, c.nlab, cap, c.conn_a);
  DPE_LAUNCHED("k_connect_links", s);
  int *a = c.conn_a, *b = c.conn_b;
  for (int span = 1; span < 2 * cap; span *= 2) {  // ceil(log2(cap)) + 1 doublings
    k_connect_jump<<<bc, 256, 0, s>>>(a, b, cap);
    DPE_LAUNCHED("k_connect_jump", s);
    std::swap(a, b);
  }
  k_connect_roots<<<bc, 256, 0, s>>>(a, c.nlab, cap, c.is_root);
  DPE_LAUNCHED("k_connect_roots", s);
  size_t nb = c.scan_bytes;
  DPE_TRY(cub::DeviceScan::ExclusiveSum(c.scan_tmp, nb, c.is_root, c.rank, cap, s));
  DPE_TRY(cudaMemsetAsync(counts, 0, (size_t)cap * sizeof(int), s));
  k_connect_final<<<bn, 256, 0, s>>>(c.lab, n, a, c.rank, out, counts);
  DPE_LAUNCHED("k_connect_final", s);
  return DPE_OK;
}

void resize_u8_launch(cudaStream_t s, const uint8_t *src, int sw, int sh, uint8_t *dst, int dw, int dh) {
  const dim3 bl(32, 8), g((dw + 31) / 32, (dh + 7) / 8);
  k_resize_u8<<<g, bl, 0, s>>>(src, sw, sh, dst, dw, dh, 1.0 / ((double)dw / sw), 1.0 / ((double)dh / sh));
}

}  // namespace

int dpe_edge_labels_device(dpe_ctx *ctx, const uint8_t *gray, int W, int H, int scale, int high_res_img, int32_t *out,
                           int ow, int oh) {
  cudaStream_t s = ctx->stream;
  Arena &A = ctx->arena;
  const int robthr = high_res_img ? 4 : 6;
  const int weak_tex_num = (int)(1.0 * H * W / (1024 << scale << scale));
  const int c1 = high_res_img ? W / 2 : W, r1 = high_res_img ? H / 2 : H;
  const int c2 = c1 / 2, r2 = r1 / 2;
  const float factor = 1.0f / (float)(1 << scale);
  if ((int)std::round(W * factor) != ow || (int)std::round(H * factor) != oh) return DPE_ERR_INVALID_ARGUMENT;
  if (c2 < 1 || r2 < 1 || ow < 3 || oh < 3) return DPE_ERR_INVALID_ARGUMENT;
  const size_t n_full = (size_t)W * H, n2 = (size_t)c2 * r2, n_out = (size_t)ow * oh;
  uint8_t *half = high_res_img ? A.get<uint8_t>("lb_half", (size_t)c1 * r1) : nullptr;
  uint8_t *down = A.get<uint8_t>("lb_down", n2);
  uint8_t *dst = A.get<uint8_t>("lb_dst", n2);
  uint8_t *up = A.get<uint8_t>("lb_up", n_out);
  int *lab0 = A.get<int>("lb_lab0", n2);
  int *counts = A.get<int>("lb_counts", std::max(n2, n_out) + 1);
  int *regions = A.get<int>("lb_regions", n2 + 1);
  unsigned long long *first_point = A.get<unsigned long long>("lb_first_point", n2 + 1);
  LargeRegions *large = A.get<LargeRegions>("lb_large", 1);
  int *error = A.get<int>("lb_error", 1);
  if (!A.ok()) return DPE_ERR_OUT_OF_MEMORY;
  ConnectScratch cs;
  int st = connect_scratch(ctx, std::max(n2, n_out), cs);
  if (st != DPE_OK) return st;
  (void)n_full;

  // halve (high_res_img), halve again, Roberts > robthr (DPE.cpp:141-160)
  const uint8_t *s1 = gray;
  if (high_res_img) {
    resize_u8_launch(s, gray, W, H, half, c1, r1);
    DPE_LAUNCHED("k_resize_u8", s);
    s1 = half;
  }
  resize_u8_launch(s, s1, c1, r1, down, c2, r2);
  DPE_LAUNCHED("k_resize_u8", s);
  {
    const dim3 bl(32, 8), g((c2 + 31) / 32, (r2 + 7) / 8);
    k_roberts_threshold<<<g, bl, 0, s>>>(down, c2, r2, robthr, dst);
    DPE_LAUNCHED("k_roberts_threshold", s);
  }
  // first labelling and the large weak regions (DPE.cpp:162-166)
  if ((st = connect_device(ctx, dst, c2, r2, cs, lab0, counts)) != DPE_OK) return st;
  DPE_TRY(cudaMemsetAsync(large, 0, sizeof(LargeRegions), s));
  DPE_TRY(cudaMemsetAsync(error, 0, sizeof(int), s));
  k_list_large<<<(unsigned)((n2 + 1 + 255) / 256), 256, 0, s>>>(counts, (int)n2 + 1, weak_tex_num, regions, first_point,
                                                               large);
  DPE_LAUNCHED("k_list_large", s);
  LargeRegions lr{};
  DPE_TRY(cudaMemcpyAsync(&lr, large, sizeof(lr), cudaMemcpyDeviceToHost, s));
  DPE_TRY(cudaStreamSynchronize(s));
  const int nreg = lr.n;
  if (nreg > 0) {
    // Hough segments across each region's border, drawn on the Roberts map (DPE.cpp:164-190)
    if (std::max(c2, r2) > kHoughMaxSide) {
      dpe_set_last_error("k_hough_region", cudaErrorInvalidValue, __FILE__, __LINE__);
      return DPE_ERR_CUDA;
    }
    const int thr = (int)(std::min(c2, r2) / 30.0);
    const float theta = (float)(3.14159265358979323846 / 180.0);
    int numangle = (int)std::floor(3.14159265358979323846 / theta) + 1;
    if (numangle > 1 && std::fabs(3.14159265358979323846 - (numangle - 1) * (double)theta) < theta / 2) --numangle;
    if (numangle > kHoughThreads - 32) return DPE_ERR_INVALID_ARGUMENT;  // 180: an angle per thread, a warp to draw
    const int numrho = (int)std::nearbyint((double)((c2 + r2) * 2 + 1));
    std::vector<float2> tab(numangle);
    for (int k = 0; k < numangle; ++k)
      tab[k] = make_float2((float)(std::cos((double)k * theta) * 1.0f), (float)(std::sin((double)k * theta) * 1.0f));
    float2 *tab_d = A.get<float2>("lb_tab", numangle);
    const int line_cap = (int)(n2 / (size_t)std::max(1, thr)) + 16;
    HoughArgs ha;
    ha.labels = lab0;
    ha.regions = regions;
    ha.w = c2; ha.h = r2; ha.threshold = thr; ha.line_length = thr; ha.line_gap = thr;
    ha.numangle = numangle; ha.numrho = numrho;
    ha.tab = tab_d;
    // Bins a point can vote for: x cos + y sin lies in [-(c2 - 1), diagonal] (a bin more on each side for
    // the rounding).
    ha.first = (numrho - 1) / 2 - c2;
    ha.len = std::min(c2 + (int)std::ceil(std::sqrt((double)c2 * c2 + (double)r2 * r2)) + 2, numrho - ha.first);
    const size_t walk_bytes = hough_walk_bytes(c2, r2), mask_bytes = hough_mask_words(n2) * sizeof(unsigned);
    int split = 1;
    auto shared = [&](int k) { return walk_bytes + mask_bytes + hough_acc_bytes(numangle, k, ha.len); };
    while (split < kHoughMaxSplit && shared(split) > kHoughShared) split *= 2;
    const bool in_shared = shared(split) <= kHoughShared;
    if (!in_shared) split = 1;
    ha.split = split;
    ha.mask = in_shared ? nullptr : A.get<unsigned>("lb_mask", hough_mask_words(n2) * nreg);
    ha.first_point = first_point;
    ha.point_cap = lr.points;
    ha.points = A.get<int2>("lb_points", lr.points * split);
    ha.accum = in_shared ? nullptr : A.get<short>("lb_accum", (size_t)numangle * ha.len * nreg);
    ha.lines = A.get<int4>("lb_lines", (size_t)line_cap * nreg);
    ha.line_cap = line_cap;
    ha.dst = dst;
    ha.error = error;
    if (!A.ok()) return DPE_ERR_OUT_OF_MEMORY;
    DPE_TRY(cudaMemcpyAsync(tab_d, tab.data(), numangle * sizeof(float2), cudaMemcpyHostToDevice, s));
    const size_t smem = in_shared ? shared(split) : walk_bytes;
    // A first vote already makes a count of 1: at a threshold of 0 or 1 (maps up to 59 pixels on the shorter
    // side) nearly every point has a segment, and the votes of the points behind it would be made again.
    // Label maps in all, eight votes a round and one: 0.62 -> 0.55 ms at 100x75, 0.93 -> 0.83 at 200x150; at
    // 400x300, whose threshold is 2, eight are as good (1.73).
    auto *kernel = thr <= 1 ? k_hough_region<1> : k_hough_region<kHoughVotes>;
    DPE_TRY(dpe_allow_dynamic_smem((const void *)kernel, smem));
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim = {(unsigned)split, 1, 1};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(nreg * split));
    cfg.blockDim = dim3(kHoughThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaError_t launched = cudaSuccess;
    DPE_TIMED(ctx, KID_EDGE_LABELS, s, launched = cudaLaunchKernelEx(&cfg, kernel, ha));
    DPE_TRY(launched);
    DPE_LAUNCHED("k_hough_region", s);
  }
  // to the level, threshold, border rule, second labelling, small regions -1 (DPE.cpp:224-285)
  resize_u8_launch(s, dst, c2, r2, up, ow, oh);
  DPE_LAUNCHED("k_resize_u8", s);
  k_threshold<<<(unsigned)((n_out + 255) / 256), 256, 0, s>>>(up, (int)n_out, robthr);
  DPE_LAUNCHED("k_threshold", s);
  k_border_rows<<<(unsigned)((oh + 255) / 256), 256, 0, s>>>(up, ow, oh);
  DPE_LAUNCHED("k_border_rows", s);
  k_border_cols<<<(unsigned)((ow + 255) / 256), 256, 0, s>>>(up, ow, oh);
  DPE_LAUNCHED("k_border_cols", s);
  if ((st = connect_device(ctx, up, ow, oh, cs, out, counts)) != DPE_OK) return st;
  k_mark_small<<<(unsigned)((n_out + 255) / 256), 256, 0, s>>>(out, (int)n_out, counts, weak_tex_num);
  DPE_LAUNCHED("k_mark_small", s);
  return DPE_OK;
}

// The Hough guards (never expected to trip): read after the caller has synchronised.
int dpe_edge_labels_check(dpe_ctx *ctx) {
  int *error = ctx->arena.get<int>("lb_error", 1);
  int e = 0;
  DPE_TRY(cudaMemcpy(&e, error, sizeof(int), cudaMemcpyDeviceToHost));
  if (e) {
    dpe_set_last_error("k_hough_region", cudaErrorUnknown, __FILE__, __LINE__);
    return DPE_ERR_CUDA;
  }
  return DPE_OK;
}

extern "C" int dpe_edge_labels(dpe_ctx *ctx, const uint8_t *gray, int width, int height, int scale, int high_res_img,
                               int memory, int32_t *labels_out) {
  if (!ctx || !gray || !labels_out || width < 4 || height < 4 || scale < 0 || scale > 8) return DPE_ERR_INVALID_ARGUMENT;
  if (memory != DPE_MEM_HOST && memory != DPE_MEM_DEVICE) return DPE_ERR_INVALID_ARGUMENT;
  if ((size_t)width * height > (size_t)INT_MAX / 4) return DPE_ERR_INVALID_ARGUMENT;
  const float factor = 1.0f / (float)(1 << scale);
  const int ow = (int)std::round(width * factor), oh = (int)std::round(height * factor);
  DPE_TRY(cudaSetDevice(ctx->device));
  cudaStream_t s = ctx->stream;
  const size_t n = (size_t)width * height, no = (size_t)ow * oh;
  const uint8_t *img = gray;
  int32_t *out = labels_out;
  if (memory == DPE_MEM_HOST) {
    uint8_t *in_d = ctx->arena.get<uint8_t>("lb_in", n);
    int32_t *out_d = ctx->arena.get<int32_t>("lb_out", no);
    if (!ctx->arena.ok()) return DPE_ERR_OUT_OF_MEMORY;
    DPE_TRY(cudaMemcpyAsync(in_d, gray, n, cudaMemcpyHostToDevice, s));
    img = in_d;
    out = out_d;
  }
  int st = dpe_edge_labels_device(ctx, img, width, height, scale, high_res_img ? 1 : 0, out, ow, oh);
  if (st != DPE_OK) return st;
  if (memory == DPE_MEM_HOST) DPE_TRY(cudaMemcpyAsync(labels_out, out, no * sizeof(int32_t), cudaMemcpyDeviceToHost, s));
  DPE_TRY(cudaStreamSynchronize(s));
  ctx->collect();
  return dpe_edge_labels_check(ctx);
}
