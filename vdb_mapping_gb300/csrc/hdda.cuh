// hdda.cuh — OpenVDB's volume ray intersector over the map's topology, for
// fast mode (castRayIntoGridFast, VDBMapping.hpp:577-602) and the raytrace
// queries (VDBMapping.hpp:675-721).
//
// The reference builds a tools::VolumeRayIntersector on the map
// (VDBMapping.hpp:1436-1449): a copy of the tree's topology, marched by a
// hierarchical DDA over the nodes below the root (4096^3 voxels), their
// children (128^3) and the leaves (8^3). What it computes, restated:
//  * setIndexRay clips the ray to the bounding box of the leaves holding an
//    active voxel (leaf granularity, max corner + 1 so a leaf spans
//    [origin, origin + 8)), by the slab method; a ray that misses the box
//    keeps its times.
//  * Each level runs DDA<Ray, log2 dim> over its cells: the start cell is
//    floor(ray(t0)) & ~(dim - 1), next[a] = t0 + (boundary - pos[a]) * invDir[a],
//    delta[a] = +-dim * invDir[a], axis = argmin of next with ties to the
//    higher axis, continue while t <= t1 (the same arithmetic as the voxel
//    DDA of castRayIntoGrid). A cell holding a node descends into it with the
//    ray's times set to [the cell's entry time, min(t1, next)].
//  * A span of the ray starts at the entry time of the first leaf cell holding
//    a leaf and ends at the entry time of the first cell, at any level, that
//    holds none (or at the end of the marched interval). Spans not longer than
//    1e-9 (math::Delta<double>) are dropped.
//  * march() returns the first span, hits() all of them.
// The map holds no tiles (values are set voxel by voxel and never pruned), so
// a node exists exactly where a leaf below it exists.
//
// The functions are templates over the topology query so that one source
// serves the kernels and a host-compiled test of the traversal.
#pragma once

#include <cstdint>
#include <cmath>
#include <cstring>

#ifdef __CUDACC__
#define VDBG_HD __host__ __device__ __forceinline__
#else
#define VDBG_HD inline
#endif

namespace vdbg {
namespace hdda {

// Exact IEEE double operations (no contraction) on both sides.
VDBG_HD double add(double a, double b)
{
#ifdef __CUDA_ARCH__
  return __dadd_rn(a, b);
#else
  return a + b;
#endif
}
VDBG_HD double sub(double a, double b)
{
#ifdef __CUDA_ARCH__
  return __dsub_rn(a, b);
#else
  return a - b;
#endif
}
VDBG_HD double mul(double a, double b)
{
#ifdef __CUDA_ARCH__
  return __dmul_rn(a, b);
#else
  return a * b;
#endif
}
VDBG_HD double dvd(double a, double b)
{
#ifdef __CUDA_ARCH__
  return __ddiv_rn(a, b);
#else
  return a / b;
#endif
}
VDBG_HD double root(double a)
{
#ifdef __CUDA_ARCH__
  return __dsqrt_rn(a);
#else
  return std::sqrt(a);
#endif
}
// (int)floor(a) for |a| < 2^31, in one conversion with rounding down.
VDBG_HD int flr_int(double a)
{
#ifdef __CUDA_ARCH__
  return __double2int_rd(a);
#else
  return static_cast<int>(std::floor(a));
#endif
}

constexpr double kDblMax   = 1.7976931348623157e308;  // std::numeric_limits<double>::max()
constexpr double kSpanEps  = 1e-9;                    // math::Delta<double>::value()
// Index coordinates a traversal may start from: |c| < 2^30 keeps every cell
// coordinate of every level inside int32.
constexpr double kCoordLimit = 1073741824.0;
// Upper bound on the cells one ray may step through, summed over the levels:
// a ray inside the +-2^30 box crosses at most 1.6M cells of 4096^3 and, inside
// the map's +-2^21 box, at most 3 * 2^22 voxels, far below; reaching it is an
// error.
constexpr uint32_t kStepLimit = 1u << 26;

struct Ray
{
  double eye[3], dir[3], inv[3];
  double t0, t1;
};

// math::Ray(eye, dir, t0, t1): invDir = 1 / dir per component.
VDBG_HD Ray make_ray(const double eye[3], const double dir[3], double t0, double t1)
{
  Ray r;
  for (int a = 0; a < 3; ++a)
  {
    r.eye[a] = eye[a];
    r.dir[a] = dir[a];
    r.inv[a] = dvd(1.0, dir[a]);
  }
  r.t0 = t0;
  r.t1 = t1;
  return r;
}

VDBG_HD long long dbits(double x)
{
#ifdef __CUDA_ARCH__
  return __double_as_longlong(x);
#else
  long long b;
  std::memcpy(&b, &x, sizeof(b));
  return b;
#endif
}
VDBG_HD double bits_double(long long b)
{
#ifdef __CUDA_ARCH__
  return __longlong_as_double(b);
#else
  double x;
  std::memcpy(&x, &b, sizeof(x));
  return x;
#endif
}

// The tests DDA::init makes of an axis, on the bit patterns (integer
// compares, off the narrow FP64 pipe): dir == 0.0 (either zero), and
// inv > 0.0 (sign clear, not zero, not NaN).
VDBG_HD bool is_zero(double x) { return (dbits(x) & 0x7fffffffffffffffll) == 0; }
VDBG_HD bool is_positive(double x)
{
  const long long b = dbits(x);
  return b > 0 && b <= 0x7ff0000000000000ll;
}

// step * inv for step = +-2^log2 of inv's sign: |inv| * 2^log2, which is
// exact, formed on the exponent field (off the narrow FP64 pipe) when |inv|
// is a normal number that stays finite; otherwise the product itself.
VDBG_HD double pow2_delta(double inv, int step, int log2)
{
  const long long b = dbits(inv) & 0x7fffffffffffffffll;
  const long long e = b >> 52;
  if (e > 0 && e + log2 < 2047) return bits_double(b + (static_cast<long long>(log2) << 52));
  return mul(static_cast<double>(step), inv);
}

struct Span
{
  double t0, t1;
};

VDBG_HD bool span_valid(const Span& s, double eps) { return sub(s.t1, s.t0) > eps; }

// Ray::clip(CoordBBox) as VolumeRayIntersector::setIndexRay uses it: lo and
// hi_excl are the box's min and (max + 1). Returns false (times unchanged)
// when the ray misses the box.
VDBG_HD bool clip(Ray& r, const int lo[3], const int hi_excl[3])
{
  double t0 = r.t0, t1 = r.t1;
  for (int a = 0; a < 3; ++a)
  {
    double x = mul(sub(static_cast<double>(lo[a]), r.eye[a]), r.inv[a]);
    double y = mul(sub(static_cast<double>(hi_excl[a]), r.eye[a]), r.inv[a]);
    if (x > y)
    {
      const double s = x;
      x              = y;
      y              = s;
    }
    if (x > t0) t0 = x;
    if (y < t1) t1 = y;
    if (t0 > t1) return false;
  }
  r.t0 = t0;
  r.t1 = t1;
  return true;
}

// math::DDA<Ray, log2> over cells of 2^log2 voxels.
struct Dda
{
  int voxel[3];
  int step[3];
  double next[3], delta[3];
  double t0, t1;
};

// Order key of a DDA time. Every time a walk compares is >= 0 (the clipped
// ray starts at t0 >= 0, each cell's exit time is at least its entry time,
// the steps are positive) or DBL_MAX, never negative or NaN; for such values
// the bit pattern read as an integer orders as the doubles do, once -0.0 is
// folded onto +0.0 (they compare equal). Integer compares keep the walks off
// the FP64 pipe, which is narrow on this GPU; the results are those of the
// double compares. Only a ray's t1 can be -0.0 (a product of its clip): t0 starts
// at +0.0, and a sum t0 + x with t0 = +0.0 is never -0.0.
VDBG_HD long long tkey(double t)
{
  const long long b = dbits(t);
  return b == static_cast<long long>(0x8000000000000000ull) ? 0ll : b;
}

// DDA::init(ray, t0, t1). The caller guarantees |ray(t0)| < 2^30 per axis.
VDBG_HD void dda_init(Dda& d, const Ray& r, double t0, double t1, int log2)
{
  const int dim = 1 << log2;
  d.t0          = t0;
  d.t1          = t1;
  double pos[3];
  for (int a = 0; a < 3; ++a)
  {
    pos[a]     = add(r.eye[a], mul(r.dir[a], t0));
    d.voxel[a] = flr_int(pos[a]) & ~(dim - 1);
  }
  for (int a = 0; a < 3; ++a)
  {
    if (is_zero(r.dir[a]))
    {
      d.step[a]  = 0;
      d.next[a]  = kDblMax;
      d.delta[a] = kDblMax;
    }
    else if (is_positive(r.inv[a]))
    {
      d.step[a]  = dim;
      d.next[a]  = add(t0, mul(sub(static_cast<double>(d.voxel[a] + dim), pos[a]), r.inv[a]));
      d.delta[a] = pow2_delta(r.inv[a], d.step[a], log2);
    }
    else
    {
      d.step[a]  = -dim;
      d.next[a]  = add(t0, mul(sub(static_cast<double>(d.voxel[a]), pos[a]), r.inv[a]));
      d.delta[a] = pow2_delta(r.inv[a], d.step[a], log2);
    }
  }
}

// DDA::step(): enter the next cell; false once its entry time passes t1. The
// axis is the smallest time's, ties to the higher index (math::MinIndex). Without
// branches: the lanes of a warp step different axes, and three branches cost
// three FP64 additions a step.
VDBG_HD bool dda_step(Dda& d)
{
  const long long n0 = dbits(d.next[0]), n1 = dbits(d.next[1]), n2 = dbits(d.next[2]);
  const bool ax      = n0 < n1 && n0 < n2;
  const bool ay      = !ax && n1 < n2;
  const bool az      = !ax && !ay;
  d.t0               = ax ? d.next[0] : (ay ? d.next[1] : d.next[2]);
  const double t     = add(d.t0, ax ? d.delta[0] : (ay ? d.delta[1] : d.delta[2]));
  d.next[0]          = ax ? t : d.next[0];
  d.next[1]          = ay ? t : d.next[1];
  d.next[2]          = az ? t : d.next[2];
  d.voxel[0] += ax ? d.step[0] : 0;
  d.voxel[1] += ay ? d.step[1] : 0;
  d.voxel[2] += az ? d.step[2] : 0;
  return dbits(d.t0) <= tkey(d.t1);
}

// A voxel-level DDA (log2 = 0) continued on integer-keyed state: the times
// held as their bit patterns, the argmin with ties to the higher axis,
// and the FP64 tMax += tDelta; fine_step enters the next voxel exactly as
// dda_step does, with fewer instructions per step.
struct FineDda
{
  int voxel[3];
  int step[3];
  long long next[3];  // bits of the times
  double delta[3];
  long long t1;
};

VDBG_HD FineDda fine_from(const Dda& d)
{
  FineDda f;
  for (int a = 0; a < 3; ++a)
  {
    f.voxel[a] = d.voxel[a];
    f.step[a]  = d.step[a];
    f.next[a]  = dbits(d.next[a]);
    f.delta[a] = d.delta[a];
  }
  f.t1 = tkey(d.t1);
  return f;
}

VDBG_HD bool fine_step(FineDda& f)
{
  const bool ax      = (f.next[0] < f.next[1]) && (f.next[0] < f.next[2]);
  const bool ay      = !ax && (f.next[1] < f.next[2]);
  const long long t0 = ax ? f.next[0] : (ay ? f.next[1] : f.next[2]);
  const double d     = ax ? f.delta[0] : (ay ? f.delta[1] : f.delta[2]);
  const long long tn = dbits(add(bits_double(t0), d));
  f.next[0]          = ax ? tn : f.next[0];
  f.next[1]          = ay ? tn : f.next[1];
  f.next[2]          = (!ax && !ay) ? tn : f.next[2];
  f.voxel[0] += ax ? f.step[0] : 0;
  f.voxel[1] += ay ? f.step[1] : 0;
  f.voxel[2] += (!ax && !ay) ? f.step[2] : 0;
  return t0 <= f.t1;
}

// DDA::next(): the time the current cell is left, at most t1.
VDBG_HD double dda_exit(const Dda& d)
{
  double m = d.t1;
  for (int a = 0; a < 3; ++a)
    if (dbits(d.next[a]) < tkey(m)) m = d.next[a];
  return m;
}

// True when eye + dir * t lies inside the +-2^30 index box (NaN fails).
VDBG_HD bool point_ok(const double eye[3], const double dir[3], double t)
{
  for (int a = 0; a < 3; ++a)
  {
    const double p = add(eye[a], mul(dir[a], t));
    if (!(p > -kCoordLimit && p < kCoordLimit)) return false;
  }
  return true;
}

enum Walk : int
{
  kWalkDone  = 0,  // traversal finished
  kWalkFirst = 1,  // march: the first span is complete
  kWalkBound = 2,  // the step bound was reached
};

// Where a span's voxel walk can meet an active voxel: windows of time (lo, hi]
// around the leaf cells with an active voxel, so that the walk can jump from one
// to the next. The cells are those of the hierarchical walk; the voxel walk is a
// DDA of its own, and each puts a leaf boundary of an axis at a time of its own.
// The two differ by less than
//   2^-50 (|eye| + |dir| + 1) |1 / dir|   (the rounding of the start position)
//   + 2^-31 t                             (of at most 2^22 additions per axis)
// = e. So at any time t the voxel walk is in a leaf cell that the hierarchical
// walk visits within e of t, unless that walk crosses two axes within 2 e of
// one another around t, in either order. Such a pair is told by the upper words
// of the two times (at least 2^-21 t apart when they differ by two) once t is
// past 2^23 times the first term, before which every crossing is taken for one
// (`floor_hi`), and gets a window by itself. A ray whose first term reaches
// 2^-26 (nearly parallel to a boundary, or starting far outside the map) is one
// window from end to end.
// A window is wider than its cells by three voxel steps of the ray (they come
// |dir|_1 to a unit of time) and 2^-21 > 3 e (and the times' single precision):
// at least one voxel boundary lies between its start and the cells, so that the
// voxel the walk stands on at its start need not be looked at either.
// `sink`: open(t0) at a span's first cell; window(lo, hi) in ascending order, without
// overlap (the last one's hi may lie past the span's end).
// A window that starts within gap_voxels of the last one's end joins it: walking
// the gap costs less than the jump over it, or a piece of its own. (Infinite: a span
// has one window, from its first active leaf to its last.)
template <class Sink>
struct RunTrack
{
  static constexpr float kGapVoxels = 24.0f;
  Sink& sink;
  float gap_voxels = kGapVoxels;
  float margin = 0.0f, gap = 0.0f, lo = 0.0f, hi = 0.0f;
  int floor_hi = 0;
  bool all = false, has = false, running = false, near = false;
  VDBG_HD explicit RunTrack(Sink& s) : sink(s) {}
  VDBG_HD void set_ray(const Ray& r)
  {
    constexpr float k2m50 = 9.3132257e-10f * 9.5367432e-7f;
    float e = k2m50, l1 = 0.0f;
    for (int a = 0; a < 3; ++a)
    {
      if (is_zero(r.dir[a])) continue;
      const float d = fabsf(static_cast<float>(r.dir[a]));
      const float w = (fabsf(static_cast<float>(r.eye[a])) + d + 1.0f) * fabsf(static_cast<float>(r.inv[a])) * k2m50;
      e             = w > e || w != w ? w : e;
      l1 += d;
    }
    all    = !(e < 1.4901161e-8f);  // 2^-26
    margin = 3.0f / l1 + 4.7683716e-7f;
    gap    = gap_voxels / l1;
    // Upper word of 2^23 e as a double, rounded up.
    const float f = all ? 2.0f : e * 8388608.0f;
    int b;
#ifdef __CUDA_ARCH__
    b = __float_as_int(f);
#else
    std::memcpy(&b, &f, sizeof(b));
#endif
    floor_hi = (b >> 3) + ((1023 - 127) << 20) + 1;
  }
  static VDBG_HD int upper(double t) { return static_cast<int>(dbits(t) >> 32); }
  // Before a step of a DDA at any level: are its two next crossings too close?
  VDBG_HD void crossing(const double next[3])
  {
    const int a = upper(next[0]), b = upper(next[1]), c = upper(next[2]);
    const int low = a < b ? a : b, high = a < b ? b : a;
    const int first = low < c ? low : c, rest = low < c ? c : low, second = rest < high ? rest : high;
    near = near || second - first < 2 || first < floor_hi;
  }
  VDBG_HD void add_time(double t)
  {
    const float f = static_cast<float>(t);
    if (has && (running || f - margin <= hi + gap))
    {
      hi = f + margin;
      return;
    }
    if (has && !all) sink.window(lo, hi);
    lo  = f - margin;
    hi  = f + margin;
    has = true;
  }
  // The span opens in the leaf cell `cell` of a ray at time t.
  VDBG_HD void open(const Ray& r, double t, const int cell[3])
  {
    sink.open(t);
    has     = false;
    running = false;
    near    = false;
    for (int a = 0; a < 3; ++a)
      near = near || (flr_int(add(r.eye[a], mul(r.dir[a], t))) & ~7) != cell[a];
  }
  VDBG_HD void enter(double t, bool active)
  {
    if (near || running || active) add_time(t);
    running = active;
    near    = false;
  }
  VDBG_HD void close(double t)
  {
    if (near || running) add_time(t);
    if (all)
      sink.window(-1.0f, 2.0f);
    else if (has)
      sink.window(lo, hi);
    has     = false;
    running = false;
    near    = false;
  }
};

// The windows of one span, kept (further ones are joined to the last).
struct Runs
{
  static constexpr int kMax = 4;
  float lo[kMax], hi[kMax];
  int n = 0;
  VDBG_HD void open(double) { n = 0; }
  VDBG_HD void window(float a, float b)
  {
    for (int k = 0; k < kMax; ++k)  // (constant indices: the state stays in registers)
    {
      if (k == n) lo[k] = a;
      if (k == n || (k == kMax - 1 && n == kMax)) hi[k] = b;
    }
    n += n < kMax ? 1 : 0;
  }
};

// (a walk that needs no runs)
struct NoTrack
{
  VDBG_HD void set_ray(const Ray&) {}
  VDBG_HD void crossing(const double*) {}
  VDBG_HD void open(const Ray&, double, const int*) {}
  VDBG_HD void enter(double, bool) {}
  VDBG_HD void close(double) {}
};

// Active bit of the leaf cell that has0 found, for a walk that asks for it.
template <class Topo, class Sink>
VDBG_HD bool cell_active(const Topo& topo, const RunTrack<Sink>&)
{
  return topo.active0();
}
template <class Topo>
VDBG_HD bool cell_active(const Topo&, const NoTrack&)
{
  return false;
}

// VolumeHDDA<Tree, Ray, 2>::march / ::hits over `topo` (has2/has1/has0 of a
// cell origin at that level). For every complete span, `on_span(span)` is
// called; with `first_only` the walk stops at the first one (march). The open
// span at the end (t1 = the end of the marched interval) is left in `t`, as
// the reference leaves it for its caller. `steps` counts cells stepped.
// `track` (RunTrack) reports a span's windows before on_span reports the span.
template <class Topo, class OnSpan, class Track>
VDBG_HD int walk(Ray r, const Topo& topo, bool first_only, Span& t, uint32_t& steps, OnSpan&& on_span, Track& track)
{
  // `open`: a span has started (t.t0 holds its start; closed spans are reset
  // to t = {-1, -1}). A span ends at a cell without a node: report it (march
  // stops there).
  bool open = t.t0 >= 0.0;
  track.set_ray(r);
#define VDBG_HDDA_CLOSE(time)                       \
  do                                                \
  {                                                 \
    t.t1 = (time);                                  \
    track.close(t.t1);                              \
    if (span_valid(t, kSpanEps))                    \
    {                                               \
      on_span(t);                                   \
      if (first_only) return kWalkFirst;            \
    }                                               \
    t.t0 = -1.0;                                    \
    t.t1 = -1.0;                                    \
    open = false;                                   \
  } while (0)
#define VDBG_HDDA_STEP(d) (track.crossing((d).next), dda_step(d))

  Dda d2;
  dda_init(d2, r, r.t0, r.t1, 12);
  do
  {
    if (++steps > kStepLimit) return kWalkBound;
    if (topo.has2(d2.voxel))
    {
      r.t0 = d2.t0;
      r.t1 = dda_exit(d2);
      Dda d1;
      dda_init(d1, r, r.t0, r.t1, 7);
      do
      {
        if (++steps > kStepLimit) return kWalkBound;
        if (topo.has1(d1.voxel))
        {
          r.t0 = d1.t0;
          r.t1 = dda_exit(d1);
          Dda d0;
          dda_init(d0, r, r.t0, r.t1, 3);
          do
          {
            if (++steps > kStepLimit) return kWalkBound;
            if (topo.has0(d0.voxel))
            {
              if (!open)
              {
                t.t0 = d0.t0;
                open = true;
                track.open(r, d0.t0, d0.voxel);
              }
              track.enter(d0.t0, cell_active(topo, track));
            }
            else if (open)
            {
              VDBG_HDDA_CLOSE(d0.t0);
            }
          } while (VDBG_HDDA_STEP(d0));
          if (open) t.t1 = d0.t1;
        }
        else if (open)
        {
          VDBG_HDDA_CLOSE(d1.t0);
        }
      } while (VDBG_HDDA_STEP(d1));
      if (open) t.t1 = d1.t1;
    }
    else if (open)
    {
      VDBG_HDDA_CLOSE(d2.t0);
    }
  } while (VDBG_HDDA_STEP(d2));
  if (open)
  {
    t.t1 = d2.t1;
    track.close(t.t1);
  }
  return kWalkDone;
#undef VDBG_HDDA_CLOSE
#undef VDBG_HDDA_STEP
}

// VolumeRayIntersector::march(t0, t1) after setIndexRay: the first span, valid
// when longer than 0. `r` is the ray after the bounding-box clip.
template <class Topo, class Track>
VDBG_HD int march_first(const Ray& r, const Topo& topo, Span& out, bool& found, uint32_t& steps, Track& track)
{
  Span t{-1.0, -1.0};
  found = false;
  if (!(sub(r.t1, r.t0) > kSpanEps)) return kWalkDone;  // VolumeHDDA::march: ray.valid()
  const int w = walk(r, topo, true, t, steps, [&](const Span&) {}, track);
  if (w == kWalkBound) return w;
  out   = t;
  found = span_valid(t, 0.0);
  return kWalkDone;
}
template <class Topo>
VDBG_HD int march_first(const Ray& r, const Topo& topo, Span& out, bool& found, uint32_t& steps)
{
  NoTrack none;
  return march_first(r, topo, out, found, steps, none);
}

// VolumeRayIntersector::hits after setIndexRay: every span, the last open one
// included when valid.
template <class Topo, class OnSpan, class Track>
VDBG_HD int all_spans(const Ray& r, const Topo& topo, uint32_t& steps, OnSpan&& on_span, Track& track)
{
  Span t{-1.0, -1.0};
  const int w = walk(r, topo, false, t, steps, on_span, track);
  if (w == kWalkBound) return w;
  if (span_valid(t, kSpanEps)) on_span(t);
  return kWalkDone;
}
template <class Topo, class OnSpan>
VDBG_HD int all_spans(const Ray& r, const Topo& topo, uint32_t& steps, OnSpan&& on_span)
{
  NoTrack none;
  return all_spans(r, topo, steps, on_span, none);
}

// One axis of a voxel walk from its next time t on: the first time >= tau, and
// how many times lie before it. FP64 addition is linear within a binade (from
// the second time on, see march.cuh), so a binade takes three additions.
VDBG_HD uint32_t jump_axis(long long& t, double d, long long tau)
{
  constexpr long long kBinade = 1ll << 52;
  uint32_t k                  = 0;
  while (t < tau)
  {
    const long long top = (t & ~(kBinade - 1)) + kBinade;  // the next binade
    const long long lim = tau < top ? tau : top;
    const long long t2  = dbits(add(bits_double(t), d));
    k += 1;
    t = t2;
    if (t2 >= lim) continue;
    const long long t3 = dbits(add(bits_double(t2), d));
    k += 1;
    t = t3;
    if (t3 >= lim) continue;
    // `more` further times stay below lim; the next addition is made.
    const long long step = t3 - t2, room = lim - 1 - t3;
    uint32_t more        = static_cast<uint32_t>(static_cast<float>(room) / static_cast<float>(step));
    while (static_cast<long long>(more) * step > room) --more;
    while (static_cast<long long>(more + 1u) * step <= room) ++more;
    k += more + 1u;
    t = dbits(add(bits_double(t3 + static_cast<long long>(more) * step), d));
  }
  return k;
}

// Steps f past every time < tau.
VDBG_HD void jump(FineDda& f, long long tau)
{
  for (int a = 0; a < 3; ++a) f.voxel[a] += f.step[a] * static_cast<int>(jump_axis(f.next[a], f.delta[a], tau));
}

// Walks f over the voxels entered at times in (lo, hi], `visit(voxel)` for each
// until it returns false (then false). f stands at the span's start t0 or after
// an earlier window; hi <= the span's end.
template <class Visit>
VDBG_HD bool walk_window(FineDda& f, double t0, double lo, long long hi, Visit&& visit)
{
  if (lo > t0) jump(f, tkey(lo) + 1);
  for (;;)
  {
    const long long m = f.next[1] < f.next[2] ? f.next[1] : f.next[2];
    if ((f.next[0] < m ? f.next[0] : m) > hi) return true;
    fine_step(f);
    if (!visit(f.voxel)) return false;
  }
}

// Bounding box of the intersector (leaves holding an active voxel): lo and
// hi_excl = max + 1; with no such leaf, lo = INT_MAX and hi_excl = INT_MIN + 1.
struct Box
{
  int lo[3];
  int hi_excl[3];
};

enum TraceStatus : int
{
  kTraceOk    = 0,
  kTraceRange = 1,  // a query's start or end leaves the +-2^30 index box, or is NaN
  kTraceBound = 2,  // the step bound was reached
};

// One raytrace query (VDBMapping.hpp:686-719): the direction is normalised
// (Vec3d::normalize: scaled by 1/length unless the length is within 1e-7 of
// 0) and scaled to `len`; origin and direction go to index space by the
// linear map (x * (1/res)); the ray [0, 1] is clipped by the box; if march
// finds a span, the voxel DDA from its start steps until it enters an active
// voxel or passes the span's end (the start voxel is not tested), and the
// end point is that voxel in world space; otherwise the ray's end.
// In three parts, so that a caller can run them apart (the device finds all
// queries' spans first, then walks them): trace_ray, trace_span, trace_walk.

// The query's ray in index space, origin oi and direction di (t in [0, 1]);
// false when its start or end leaves the +-2^30 index box (or is NaN).
VDBG_HD bool trace_ray(const double o[3], const double dir[3], double len, double inv_res, double oi[3],
                       double di[3])
{
  double d[3]     = {dir[0], dir[1], dir[2]};
  const double ln = root(add(add(mul(d[0], d[0]), mul(d[1], d[1])), mul(d[2], d[2])));
  if ((ln < 0.0 ? -ln : ln) > 1e-7)
  {
    const double s = dvd(1.0, ln);
    for (int a = 0; a < 3; ++a) d[a] = mul(d[a], s);
  }
  for (int a = 0; a < 3; ++a)
  {
    d[a]  = mul(d[a], len);
    oi[a] = mul(o[a], inv_res);
    di[a] = mul(d[a], inv_res);
  }
  return point_ok(oi, di, 0.0) && point_ok(oi, di, 1.0);
}

// The first span of the query's ray clipped by the box (march).
template <class Topo, class Track>
VDBG_HD int trace_span(const double oi[3], const double di[3], const Box& box, const Topo& topo, Span& sp,
                       bool& found, uint32_t& steps, Track& track)
{
  Ray r = make_ray(oi, di, 0.0, 1.0);
  clip(r, box.lo, box.hi_excl);
  sp    = Span{-1.0, -1.0};
  found = false;
  if (march_first(r, topo, sp, found, steps, track) == kWalkBound) return kTraceBound;
  return kTraceOk;
}
template <class Topo>
VDBG_HD int trace_span(const double oi[3], const double di[3], const Box& box, const Topo& topo, Span& sp,
                       bool& found, uint32_t& steps)
{
  NoTrack none;
  return trace_span(oi, di, box, topo, sp, found, steps, none);
}

// The voxel walk over span `sp`: end = the first active voxel after the
// start voxel, or the voxel just past the span, in world space.
template <class Active>
VDBG_HD int trace_walk(const double oi[3], const double di[3], const Span& sp, double res, Active&& active,
                       double end[3], uint32_t& steps)
{
  const Ray fine = make_ray(oi, di, sp.t0, sp.t1);
  Dda dda;
  dda_init(dda, fine, sp.t0, sp.t1, 0);
  FineDda f = fine_from(dda);
  while (fine_step(f) && !active(f.voxel))
  {
    if (++steps > kStepLimit) return kTraceBound;
  }
  for (int a = 0; a < 3; ++a) end[a] = mul(static_cast<double>(f.voxel[a]), res);
  return kTraceOk;
}

// The same from the span's windows (RunTrack); `fine` is the query's ray (make_ray).
template <class Active>
VDBG_HD void trace_walk_runs(const Ray& fine, const Span& sp, const float* lo, const float* hi, int n, double res,
                             Active&& active, double end[3])
{
  Dda dda;
  dda_init(dda, fine, sp.t0, sp.t1, 0);
  FineDda f = fine_from(dda);
  bool hit  = false;
  for (int i = 0; i < n && !hit; ++i)
  {
    const long long stop = tkey(static_cast<double>(hi[i]));
    hit = !walk_window(f, sp.t0, static_cast<double>(lo[i]), stop < f.t1 ? stop : f.t1,
                       [&](const int v[3]) { return !active(v); });
  }
  if (!hit)
  {
    // Past the last time <= t1, and one step more.
    jump(f, f.t1 + 1);
    fine_step(f);
  }
  for (int a = 0; a < 3; ++a) end[a] = mul(static_cast<double>(f.voxel[a]), res);
}

// castRayIntoGridFast's voxel walk (VDBMapping.hpp:593-600) of the span from t0,
// as far as the voxels entered at times in (lo, hi], and the span's first voxel
// when lo <= t0.
template <class Visit>
VDBG_HD void fast_walk_window(const double eye[3], const double dir[3], double t0, double lo, double hi, Visit&& visit)
{
  const Ray fine = make_ray(eye, dir, t0, hi);
  Dda dda;
  dda_init(dda, fine, t0, hi, 0);
  FineDda f = fine_from(dda);
  if (!(lo > t0)) visit(f.voxel);
  walk_window(f, t0, lo, tkey(hi), [&](const int v[3]) {
    visit(v);
    return true;
  });
}

// The pieces of a window (lo, hi] of fast mode's walk, about kPieceVoxels voxel
// steps each (l1 = |dir|_1): `item(lo, hi)` for each, in order and adjoining; the
// first one of a span starts at -1. hi <= the span's end.
constexpr float kPieceVoxels = 48.0f;
template <class Item>
VDBG_HD void window_pieces(double t0, float lo, double hi, float l1, Item&& item)
{
  const float a = lo > static_cast<float>(t0) ? lo : static_cast<float>(t0);
  const float b = static_cast<float>(hi);
  const float k = (b - a) * l1 * (1.0f / kPieceVoxels);
  const int n   = k > 1.5f ? static_cast<int>(k + 0.5f < 1.0e6f ? k + 0.5f : 1.0e6f) : 1;
  const float w = (b - a) / static_cast<float>(n);
  double from   = static_cast<double>(lo) > t0 ? static_cast<double>(lo) : -1.0;
  for (int i = 1; i <= n; ++i)
  {
    const double to = i < n ? static_cast<double>(a + w * static_cast<float>(i)) : hi;
    item(from, to);
    from = to;
  }
}

// The end point of a query without a span: the ray's end.
VDBG_HD void trace_miss(const double oi[3], const double di[3], double res, double end[3])
{
  for (int a = 0; a < 3; ++a) end[a] = mul(add(oi[a], di[a]), res);
}

template <class Topo, class Active>
VDBG_HD int raytrace_one(const double o[3], const double dir[3], double len, double res, double inv_res,
                         const Box& box, const Topo& topo, Active&& active, bool& success, double end[3],
                         uint32_t& steps)
{
  double oi[3], di[3];
  if (!trace_ray(o, dir, len, inv_res, oi, di)) return kTraceRange;
  Span sp{-1.0, -1.0};
  bool found = false;
  if (trace_span(oi, di, box, topo, sp, found, steps) == kTraceBound) return kTraceBound;
  if (found)
  {
    if (trace_walk(oi, di, sp, res, active, end, steps) == kTraceBound) return kTraceBound;
    success = true;
  }
  else
  {
    trace_miss(oi, di, res, end);
    success = false;
  }
  return kTraceOk;
}

// castRayIntoGridFast (VDBMapping.hpp:577-602) from voxel o to voxel e: the
// ray of castRayIntoGrid (eye o + 0.5, direction e - o, [0, 1]) clipped by
// the box, every span of it walked by the voxel DDA, `mark(v)` for each voxel
// the DDA enters (the span's start voxel included) that is active in the map.
template <class Topo, class Active, class Mark>
VDBG_HD int fast_cast_one(const int o[3], const int e[3], const Box& box, const Topo& topo, Active&& active,
                          Mark&& mark, uint32_t& steps)
{
  double eye[3], dir[3];
  for (int a = 0; a < 3; ++a)
  {
    eye[a] = add(static_cast<double>(o[a]), 0.5);
    dir[a] = sub(static_cast<double>(e[a]), static_cast<double>(o[a]));
  }
  Ray r = make_ray(eye, dir, 0.0, 1.0);
  clip(r, box.lo, box.hi_excl);
  bool bound = false;
  const int w = all_spans(r, topo, steps, [&](const Span& sp) {
    if (bound) return;
    const Ray fine = make_ray(eye, dir, sp.t0, sp.t1);
    Dda dda;
    dda_init(dda, fine, sp.t0, sp.t1, 0);
    do
    {
      if (++steps > kStepLimit)
      {
        bound = true;
        return;
      }
      if (active(dda.voxel)) mark(dda.voxel);
    } while (dda_step(dda));
  });
  return (w == kWalkBound || bound) ? kTraceBound : kTraceOk;
}

} // namespace hdda
} // namespace vdbg
