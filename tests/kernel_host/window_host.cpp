// window_host.cpp -- TEST INFRASTRUCTURE: window_inside and the taps that it clears, on the host.
#include "kernel_host.cpp"

// Per projected window i: whether window_inside clears it, and the smallest and largest texel (relative to
// the padded image, so 0 .. W + 1 and 0 .. H + 1 are in it) that a clamp-free bilinear tap would touch, by the tap
// loop's own arithmetic.  wp: per window U0, V0, fu, fv, g03.xy, g14.xy, zc, h6, h7.
extern "C" void host_window_inside(int W, int H, int n, const float *wp, int *inside, int *range) {
  PMArgs a;
  memset(&a, 0, sizeof(a));
  a.W = W;
  a.H = H;
  for (int i = 0; i < n; ++i, wp += 11, range += 4) {
    WinProj w;
    w.U0 = (int)wp[0];
    w.V0 = (int)wp[1];
    w.fuv = make_float2(wp[2], wp[3]);
    w.g03 = make_float2(wp[4], wp[5]);
    w.g14 = make_float2(wp[6], wp[7]);
    w.zc = wp[8];
    w.h6 = wp[9];
    w.h7 = wp[10];
    inside[i] = window_inside(a, w, 5.0f) ? 1 : 0;
    const double big = 1e9;
    double lo[2] = {big, big}, hi[2] = {-big, -big};
    for (int dx = -5; dx <= 5; dx += 2)
      for (int dy = -5; dy <= 5; dy += 2) {
        const float cx = w.g03.x * dx, cy = w.g03.y * dx, cz = w.h6 * dx + w.zc;
        const float gx = w.g14.x * dy, gy = w.g14.y * dy, gz = w.h7 * dy;
        const float iz = tap_rcp(gz + cz);
        const float u = (gx + cx) * iz + w.fuv.x, v = (gy + cy) * iz + w.fuv.y;
        const double p[2] = {std::isfinite(u) ? std::floor((double)u) + w.U0 + 1 : -big,
                             std::isfinite(v) ? std::floor((double)v) + w.V0 + 1 : -big};
        for (int k = 0; k < 2; ++k) {
          lo[k] = std::min(lo[k], std::max(p[k], -big));
          hi[k] = std::max(hi[k], std::min(p[k] + 1, big));
        }
      }
    range[0] = (int)lo[0]; range[1] = (int)hi[0]; range[2] = (int)lo[1]; range[3] = (int)hi[1];
  }
}
