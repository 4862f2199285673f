// Host-side scan geometry for the distance-driven operators.
//
// A plan is built once per options vector (and dtype) and holds, per view:
//   * the branch (image rows are the integration lines when |cos| dominates,
//     columns otherwise) and the detector-order flip, decided exactly as the
//     reference does (src/fan_ed_kernel.cu:61-77);
//   * the D+1 detector-cell boundaries projected onto the view's axis
//     (x-axis for row lines, y-axis for column lines), evaluated in fp64 with
//     the reference's formulas (src/fan_ed_kernel.cu:78-95,
//     src/fan_ea_kernel.cu:72-84, src/para_kernel.cu:52-60), in increasing
//     order, plus the cell widths (fp64 differences);
//   * per-detector normalisation factors;
//   * an approximate inverse of the boundary map (axis coordinate -> fractional
//     cell index) used to seed the cell search in the image-side gather;
// and per (view, line) the affine map from pixel-edge index k to the axis,
// axis = alpha + sigma * k, evaluated in fp64 from the rounded source position.
#pragma once

#include <cmath>
#include <cstdint>
#include <string>
#include <vector>

namespace ctgb {

enum Scan { kFanED = 0, kFanEA = 1, kPara = 2 };

struct HostGeom {
  int V = 0, D = 0, W = 0, H = 0, L = 0, scan = 0, dtype = 0;
  // option values after rounding to the data type
  double views = 0, dets = 0, width = 0, height = 0, dImg = 0, dDet = 0, Ang0 = 0, dAng = 0, s2r = 0,
         d2r = 0, binshift = 0;
  std::vector<int32_t> flags;  // V: bit0 row lines (x-branch), bit1 flipped detector order
  std::vector<double> src;     // V*2: source x, y (fan)
  std::vector<double> db;      // V*(D+1): cell boundaries on the axis, increasing
  std::vector<double> wd;      // V*D: cell widths db[d+1]-db[d]
  std::vector<double> fq;      // V*D: A / A^T factor (fan dImg/(cbar*w), para dImg/dDet)
  std::vector<double> fbt;     // V*D: B^T factor of equal-angle fans (dImg/cbar), empty otherwise
  std::vector<double> lp;      // V*L*2: alpha, sigma (pixel edge k of a line maps to alpha + sigma*k)
  std::vector<double> inv;     // V*5: guess u = x*P0/(P1+x*P2) (atan for EA), cell = P3+P4*u
  std::vector<double> wpre;    // D: fbp detector pre-weight, applied as (y * wpre[k]) * wscale
  double wscale = 1.0;
  std::vector<double> taps;    // 2D-1: RL ramp taps (src/fan_ed_kernel.cu:926-943)
  std::vector<double> taps_lo; // 2D-1: fp64 tap minus the stored one (fp32 plans), else 0
  double dfilt = 0.0;          // tap spacing of the ramp filter (virtual bin, or dDet)
  std::vector<double> options; // the options vector the geometry was built from
  double x0 = 0, y0 = 0;       // left image edge x, bottom image edge y
  std::vector<double> slope;   // V: parallel beams, d(axis coordinate)/d(line position) of a ray
};

// A detector-cell boundary is a straight ray, so its position on the image
// lines of a view, in pixel-edge units, is linear in the line index: u(l) = u0 +
// du * l. Likewise the cell's width w(l) = w0 + dw * l in pixels.
struct RayWalk {
  double u0, du;
  double left, right;  // the (fractional) lines on which u is 0 and N; nothing if du is 0
};
inline RayWalk ray_walk(double u0, double du, int N) {
  const double r = 1 / du;
  return {u0, du, -u0 * r, (N - u0) * r};
}
struct CellWalk {
  double u0, du;  // lower boundary
  double w0, dw;  // width
  // lines first .. last of the view are the only ones on which the cell meets
  // the image (one line of margin on each side); first > last: none
  int first, last;
};

// the cell between two boundaries
inline CellWalk cell_walk(const HostGeom& g, int v, RayWalk lower, RayWalk upper) {
  const bool xb = g.flags[v] & 1;
  const int nl = xb ? g.H : g.W, N = xb ? g.W : g.H;
  CellWalk c;
  c.u0 = lower.u0;
  c.du = lower.du;
  c.w0 = upper.u0 - lower.u0;
  c.dw = upper.du - lower.du;
  double lo = 0, hi = nl - 1;
  // the lines on one side of where a boundary crosses an edge; a: its side if it runs along the lines
  auto keep = [&](double a, double s, double at) {
    if (s > 0) lo = std::fmax(lo, std::floor(at) - 1);
    else if (s < 0) hi = std::fmin(hi, std::ceil(at) + 1);
    else if (!(a > 0)) hi = -1;
  };
  keep(upper.u0, upper.du, upper.left);  // the upper boundary right of the image's left edge
  keep(N - c.u0, -c.du, lower.right);    // the lower boundary left of its right edge
  if (lo <= hi) { c.first = (int)lo; c.last = (int)hi; }
  else { c.first = 65535; c.last = 0; }
  return c;
}

// Unevaluated sums of two doubles (T. J. Dekker, "A floating-point technique for
// extending the available precision", 1971), with fused multiply-adds for the
// products' errors.
struct Pair {
  double hi, lo;
};
inline Pair fast_sum(double a, double b) {
  const double s = a + b;
  return {s, b - (s - a)};
}
inline Pair operator+(Pair a, Pair b) {
  const double s = a.hi + b.hi, t = s - a.hi;
  return fast_sum(s, (a.hi - (s - t)) + (b.hi - t) + a.lo + b.lo);
}
inline Pair operator*(Pair a, double b) {
  const double p = a.hi * b;
  return fast_sum(p, std::fma(a.hi, b, -p) + a.lo * b);
}
inline Pair operator/(Pair a, double b) {
  const double q = a.hi / b;
  return fast_sum(q, (std::fma(-q, b, a.hi) + a.lo) / b);
}

// u0 and du of a boundary at axis coordinate x as unevaluated pairs, good to about 100
// bits for x as it is stored. Both are linear in x, with a view's constants that hold
// all divisions: 2.5 ms for the 850 thousand boundaries of 1152 views of 736 bins,
// where dividing at every boundary took 16.5.
struct BoundaryWalk {
  double u0, u0_lo, du, du_lo;
};
struct ViewWalk {
  Pair a, b, c, d;  // u0 = a x + b, du = c x + d
  int N;            // pixels of a line
  BoundaryWalk at(double x) const {
    const Pair u = a * x + b, s = c * x + d;
    return {u.hi, u.lo, s.hi, s.lo};
  }
  // the same in plain double
  RayWalk ray(double x) const { return ray_walk(a.hi * x + b.hi, c.hi * x + d.hi, N); }
};
ViewWalk view_walk(const HostGeom& g, int v);

// Parse the reference's options vector and build the geometry. dtype 0 = fp32,
// 1 = fp64. Returns false and sets `err` on invalid options.
bool build_geometry(const double* options, int n_options, int dtype, HostGeom& g, std::string& err);

// fbp filter windows: the reference's Ram-Lak (RL) kernel, Shepp-Logan, and RL
// under a Hann window (its exact discrete form, [1/4, 1/2, 1/4] * RL).
enum FilterWindow { kRamLak = 0, kSheppLogan = 1, kHann = 2 };

// Ramp filter taps (2D-1, offsets -(D-1)..D-1) of `window` into g.taps /
// g.taps_lo, for the plan's dtype. ea_exact (equal-angle fans only) multiplies
// each tap by (n dDet / sin(n dDet))^2, the factor that makes the RL kernel
// exact on equiangular samples. RamLak without ea_exact reproduces the
// reference's taps; the others have no counterpart in it.
bool filter_taps(HostGeom& g, int window, bool ea_exact, std::string& err);

}  // namespace ctgb
