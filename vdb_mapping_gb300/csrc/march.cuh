// march.cuh — castRayIntoGrid's voxel DDA (VDBMapping.hpp:550-566, OpenVDB's
// DDA<Ray<double>,0>) in chunks that can be walked in any order, in parallel.
//
// The DDA of a ray from the sensor voxel o to the end voxel e (eye = o + 0.5,
// dir = e - o, t in [0, 1]) merges three sequences of crossing times, one per
// axis: with n = |dir| and d = fl(1 / n), the axis steps at
//   t_0 = d / 2 (exact: half a voxel times 1 / dir),  t_k = fl(t_{k-1} + d),
// an axis with n = 0 never. The walk takes the smallest time, ties to the
// higher axis, while it is <= 1. The three sequences do not depend on one
// another, so the state of the walk at a threshold T (every step at a time
// below T taken) is, per axis, the number of its times below T. That lets a
// walk start at any threshold, provided the exact t_k there is known without
// adding k times.
//
// It is known because FP64 addition is linear within a binade. For t and
// t + d in [2^e, 2^(e+1)) the sum is rounded to the same spacing u, so t grows
// by round(d / u) units each time: a constant D on the bit pattern. The one
// exception is a tie (d an odd multiple of u / 2): it rounds to even, so the
// first sum of the binade may take the other neighbour; its result is even and
// from there on the increment is constant again. A sequence is therefore
// described, per binade, by its first time t1 (index k1) in it, the first
// increment D + df (df in {-1, 0, 1}) and the increment D of all later ones.
//
// [0, 1] is cut at multiples of 2^-p, p the smallest with L1 * 2^-p <= 2^clog.
// Chunk i >= 1 lies inside one binade, so it is walked with integer additions
// of bit patterns alone; chunk 0 holds the small binades and is walked with
// the FP64 additions themselves. Ideal
// times are (k + 1/2) / n; the index a threshold falls at is computed from
// them and corrected by at most one against the exact times.
//
// A DADD of a warp occupies this GPU's FP64 pipe for about 19 cycles, so a walk
// of one DADD per step is bound by it; and a whole ray per lane makes a warp
// wait for its longest ray, and a scan for the longest of all (10,000 voxels).
// Chunks are equally long and carry no FP64.
#pragma once

#include "hdda.cuh"

namespace vdbg {
namespace march {

// Chunks of up to 32, 64 or 128 steps (the caller's choice by the size of its
// scan: `clog`), more precisely below L1 * 2^-p + 3 (each axis at most
// n * 2^-p + 1).
constexpr int kMinChunkLog2 = 5;
constexpr int kMaxChunkLog2 = 7;
constexpr uint32_t kMaxSteps = (1u << kMaxChunkLog2) + 3u;

constexpr uint64_t kOneBits  = 0x3ff0000000000000ull;  // 1.0
constexpr uint64_t kNever    = 0x7fefffffffffffffull;  // DBL_MAX, the time of an axis that never steps
constexpr uint64_t kMantissa = (1ull << 52) - 1ull;

VDBG_HD int log2_floor(uint32_t x)
{
#ifdef __CUDA_ARCH__
  return 31 - __clz(static_cast<int>(x));
#else
  return 31 - __builtin_clz(x);
#endif
}

// p of a ray of L1 length l1: the walk has 2^p chunks.
VDBG_HD int chunk_log2(uint32_t l1, int clog) { return l1 <= (1u << clog) ? 0 : log2_floor((l1 - 1u) >> clog) + 1; }

VDBG_HD uint64_t bits_of(double x) { return static_cast<uint64_t>(hdda::dbits(x)); }
VDBG_HD double double_of(uint64_t b) { return hdda::bits_double(static_cast<long long>(b)); }
VDBG_HD uint64_t pow2_bits(int e) { return static_cast<uint64_t>(1023 + e) << 52; }

// Bits of i * 2^-p (1 <= i < 2^31).
VDBG_HD uint64_t threshold_bits(uint32_t i, int p)
{
  const int e = log2_floor(i);
  return pow2_bits(e - p) + ((static_cast<uint64_t>(i) << (52 - e)) & kMantissa);
}

// One axis' times in the binade [2^-(j+1), 2^-j): see above. An axis without
// a time in it has its first later time as t1.
struct Axis
{
  uint64_t t1;  // bits of the first time >= 2^-(j+1)
  uint64_t d;   // increment on the bits, after the first
  uint32_t k1;  // index of t1
  int32_t df;   // the first increment is d + df
};

VDBG_HD double axis_delta(uint32_t n) { return hdda::dvd(1.0, static_cast<double>(n)); }

// The entry of an axis of n > 0 voxels for binade j, binade by binade from t_0
// on. Both branches of a binade with at most two times take the additions
// themselves.
VDBG_HD Axis axis_entry(uint32_t n, int j)
{
  const double d     = axis_delta(n);
  const uint64_t lo  = pow2_bits(-(j + 1));
  double t           = hdda::mul(d, 0.5);
  uint32_t k         = 0;
  while (bits_of(t) < lo)
  {
    const uint64_t top = (bits_of(t) & ~kMantissa) + (1ull << 52);  // the next binade
    const double t2    = hdda::add(t, d);
    if (bits_of(t2) >= top)
    {
      t = t2;
      k += 1;
      continue;
    }
    const double t3 = hdda::add(t2, d);
    if (bits_of(t3) >= top)
    {
      t = t3;
      k += 2;
      continue;
    }
    const uint64_t step = bits_of(t3) - bits_of(t2);
    const uint64_t more = (top - 1ull - bits_of(t3)) / step;  // further times in the binade
    t                   = hdda::add(double_of(bits_of(t3) + more * step), d);
    k += 3u + static_cast<uint32_t>(more);
  }
  Axis a;
  const uint64_t top = lo + (1ull << 52);
  const uint64_t b1 = bits_of(t), b2 = bits_of(hdda::add(t, d));
  const uint64_t b3 = bits_of(hdda::add(double_of(b2), d));
  const uint64_t f  = b2 - b1;
  a.t1              = b1;
  a.k1              = k;
  a.d               = f;
  if (b2 < top)
  {
    // (past the binade any increment that leaves it does)
    if (b3 < top)
      a.d = b3 - b2;
    else if (b2 + f < top)
      a.d = f + 1ull;
  }
  a.df = static_cast<int32_t>(static_cast<int64_t>(f - a.d));
  return a;
}

VDBG_HD Axis axis_never() { return Axis{kNever, 0ull, 0u, 0}; }

// The walk's state. Voxels are held relative to the chunk: `pos` has 9 bits
// per axis (x lowest), the in-leaf coordinate of the chunk's first voxel plus
// kPosBias, so that the steps of a chunk (up to 2^clog + 1 on one axis, and
// three more of step_free) stay inside 1..511; a leaf or plane crossing is then
// one test of kCrossing, and a step one addition. The five bits left are the
// caller's (k_march: the lane).
constexpr int kPosBits       = 9;
constexpr int kPosBias       = 136;  // 17 leaves
constexpr uint32_t kPosMask  = (1u << kPosBits) - 1u;
constexpr uint32_t kCrossing = (kPosMask << (2 * kPosBits)) | ((kPosMask - 7u) << kPosBits) | (kPosMask - 7u);
static_assert((1 << kMaxChunkLog2) + 4 < kPosBias && (1 << kMaxChunkLog2) + 4 + 7 + kPosBias <= int(kPosMask),
              "positions of a chunk");

struct Walk
{
  uint64_t tx, ty, tz;  // next times (bits)
  uint64_t dx, dy, dz;  // increments: of the bits, or (chunk 0) the FP64 deltas' bits
  uint32_t end;         // the walk stops at times whose upper word is >= end
  uint32_t pos;
  int px, py, pz;       // position steps
  uint32_t one;         // 1 (see step)
};

// One step: nothing changes once the next time has reached `end`.
template <bool kFp64>
VDBG_HD void step(Walk& w)
{
#ifdef __CUDA_ARCH__
  if (!kFp64)
  {
    // Predicated additions on 32-bit halves: no branch, no select of what is
    // added. The walk is bound by the ALU pipe (a warp instruction every two
    // cycles): compares, selects and additions; the position's additions are
    // written as multiply-adds by a register that holds 1, which go to the
    // FMA pipe.
    asm("{\n\t"
        ".reg .pred yz, ax, go, nx, gx, gy, gz;\n\t"
        ".reg .b64 m;\n\t"
        ".reg .b32 lo, mh, th, xl, xh, yl, yh, zl, zh, al, ah;\n\t"
        "mov.b64 {xl, xh}, %0;\n\t"
        "mov.b64 {yl, yh}, %1;\n\t"
        "mov.b64 {zl, zh}, %2;\n\t"
        "setp.lt.u64 yz, %1, %2;\n\t"
        "selp.b64 m, %1, %2, yz;\n\t"
        "setp.lt.u64 ax, %0, m;\n\t"
        "mov.b64 {lo, mh}, m;\n\t"
        "selp.b32 th, xh, mh, ax;\n\t"
        "setp.lt.u32 go, th, %10;\n\t"
        "and.pred gx, go, ax;\n\t"
        "not.pred nx, ax;\n\t"
        "and.pred go, go, nx;\n\t"
        "and.pred gy, go, yz;\n\t"
        "not.pred nx, yz;\n\t"
        "and.pred gz, go, nx;\n\t"
        "mov.b64 {al, ah}, %4;\n\t"
        "@gx add.cc.u32 xl, xl, al;\n\t"
        "@gx addc.u32 xh, xh, ah;\n\t"
        "mov.b64 {al, ah}, %5;\n\t"
        "@gy add.cc.u32 yl, yl, al;\n\t"
        "@gy addc.u32 yh, yh, ah;\n\t"
        "mov.b64 {al, ah}, %6;\n\t"
        "@gz add.cc.u32 zl, zl, al;\n\t"
        "@gz addc.u32 zh, zh, ah;\n\t"
        "@gx mad.lo.u32 %3, %7, %11, %3;\n\t"
        "@gy mad.lo.u32 %3, %8, %11, %3;\n\t"
        "@gz mad.lo.u32 %3, %9, %11, %3;\n\t"
        "mov.b64 %0, {xl, xh};\n\t"
        "mov.b64 %1, {yl, yh};\n\t"
        "mov.b64 %2, {zl, zh};\n\t"
        "}"
        : "+l"(w.tx), "+l"(w.ty), "+l"(w.tz), "+r"(w.pos)
        : "l"(w.dx), "l"(w.dy), "l"(w.dz), "r"(w.px), "r"(w.py), "r"(w.pz), "r"(w.end), "r"(w.one));
    return;
  }
#endif
  const bool yz     = w.ty < w.tz;
  const uint64_t m  = yz ? w.ty : w.tz;
  const bool ax     = w.tx < m;
  const uint64_t t0 = ax ? w.tx : m;
  const bool go     = static_cast<uint32_t>(t0 >> 32) < w.end;
  const bool gx = go && ax, gy = go && !ax && yz, gz = go && !ax && !yz;
  // (one addition for all three axes: the FP64 pipe is narrow)
  const uint64_t d  = ax ? w.dx : (yz ? w.dy : w.dz);
  const uint64_t tn = kFp64 ? bits_of(hdda::add(double_of(t0), double_of(d))) : t0 + d;
  w.tx              = gx ? tn : w.tx;
  w.ty              = gy ? tn : w.ty;
  w.tz              = gz ? tn : w.tz;
  w.pos += static_cast<uint32_t>(go ? (ax ? w.px : (yz ? w.py : w.pz)) : 0);
}

// One step of a chunk whose upper threshold is not a binade's (and without
// cuts), whatever `end` is: up to three steps past it stay in the binade, on
// voxels of the next chunk, which marks them as well. A quarter fewer ALU
// instructions than step.
VDBG_HD void step_free(Walk& w)
{
#ifdef __CUDA_ARCH__
  asm("{\n\t"
      ".reg .pred yz, ax, nyz, nax, gy, gz;\n\t"
      ".reg .b64 m;\n\t"
      ".reg .b32 al, ah, xl, xh;\n\t"
      "setp.lt.u64 yz|nyz, %1, %2;\n\t"
      "selp.b64 m, %1, %2, yz;\n\t"
      "setp.lt.u64 ax|nax, %0, m;\n\t"
      "and.pred gy, nax, yz;\n\t"
      "and.pred gz, nax, nyz;\n\t"
      "mov.b64 {al, ah}, %4;\n\t"
      "mov.b64 {xl, xh}, %0;\n\t"
      "@ax add.cc.u32 xl, xl, al;\n\t"
      "@ax addc.u32 xh, xh, ah;\n\t"
      "mov.b64 %0, {xl, xh};\n\t"
      "mov.b64 {al, ah}, %5;\n\t"
      "mov.b64 {xl, xh}, %1;\n\t"
      "@gy add.cc.u32 xl, xl, al;\n\t"
      "@gy addc.u32 xh, xh, ah;\n\t"
      "mov.b64 %1, {xl, xh};\n\t"
      "mov.b64 {al, ah}, %6;\n\t"
      "mov.b64 {xl, xh}, %2;\n\t"
      "@gz add.cc.u32 xl, xl, al;\n\t"
      "@gz addc.u32 xh, xh, ah;\n\t"
      "mov.b64 %2, {xl, xh};\n\t"
      "@ax mad.lo.u32 %3, %7, %10, %3;\n\t"
      "@gy mad.lo.u32 %3, %8, %10, %3;\n\t"
      "@gz mad.lo.u32 %3, %9, %10, %3;\n\t"
      "}"
      : "+l"(w.tx), "+l"(w.ty), "+l"(w.tz), "+r"(w.pos)
      : "l"(w.dx), "l"(w.dy), "l"(w.dz), "r"(w.px), "r"(w.py), "r"(w.pz), "r"(w.one));
#else
  if (w.tx < w.ty && w.tx < w.tz)
    w.tx += w.dx, w.pos += static_cast<uint32_t>(w.px);
  else if (w.ty < w.tz)
    w.ty += w.dy, w.pos += static_cast<uint32_t>(w.py);
  else
    w.tz += w.dz, w.pos += static_cast<uint32_t>(w.pz);
#endif
}

// Whether chunk i (not cut) may be walked with step_free.
VDBG_HD bool chunk_is_free(uint32_t i) { return i != 0u && (i & (i + 1u)) != 0u; }

// Whether the next step would change anything.
VDBG_HD bool has_step(const Walk& w)
{
  const uint32_t x = static_cast<uint32_t>(w.tx >> 32), y = static_cast<uint32_t>(w.ty >> 32),
                 z = static_cast<uint32_t>(w.tz >> 32);
  const uint32_t m = y < z ? y : z;
  return (x < m ? x : m) < w.end;
}

VDBG_HD uint32_t pos_field(uint32_t pos, int a) { return (pos >> (a * kPosBits)) & kPosMask; }

// Bit of the position's voxel in its z-plane word, and the plane.
VDBG_HD int plane_bit(uint32_t pos) { return static_cast<int>((pos & 7u) | ((pos >> (kPosBits - 3)) & 0x38u)); }
VDBG_HD int plane_of(uint32_t pos) { return static_cast<int>((pos >> (2 * kPosBits)) & 7u); }

// Where a chunk starts on one axis: the first index k whose time is >= the
// threshold i * 2^-p (bits tau), from the entry of the threshold's binade.
struct Start
{
  uint64_t t;   // the time
  uint64_t d;   // increment after it
  uint32_t k;
  int32_t df;   // non-zero: d holds the first increment, the later ones are d - df
};

VDBG_HD Start start_axis(const Axis& a, uint32_t n, uint32_t i, int p, uint64_t tau)
{
  // Ideal index: the k with (k + 1/2) / n < i * 2^-p, counted.
  uint32_t k = static_cast<uint32_t>((2ull * n * i + (1ull << p) - 1ull) >> (p + 1));
  if (k < a.k1) k = a.k1;
  const uint32_t r = k - a.k1;
  uint64_t t       = a.t1 + static_cast<uint64_t>(r) * a.d + static_cast<uint64_t>(static_cast<int64_t>(r ? a.df : 0));
  const uint64_t in  = a.d + static_cast<uint64_t>(static_cast<int64_t>(r ? 0 : a.df));  // from k on
  const uint64_t out = a.d + static_cast<uint64_t>(static_cast<int64_t>(r == 1u ? a.df : 0));  // up to k
  if (t < tau)
  {
    t += in;
    k += 1u;
  }
  else if (r && t - out >= tau)
  {
    t -= out;
    k -= 1u;
  }
  Start s;
  s.t  = t;
  s.k  = k;
  s.df = k == a.k1 ? a.df : 0;
  s.d  = a.d + static_cast<uint64_t>(static_cast<int64_t>(s.df));
  return s;
}

// A chunk whose axis a is at its binade's first time with df != 0 must not
// take two more steps of it with the same increment: its walk is cut at that
// axis' second time (at its upper word, so a little before it at most, and
// after the first) and resumed with the later increment. `first` is the
// position the chunk began at (an axis that has stepped is past its first
// time), f[] the axes' df.
struct Cuts
{
  int8_t f[3];
};

VDBG_HD uint32_t upper(uint64_t t) { return static_cast<uint32_t>(t >> 32); }

VDBG_HD void cut_end(Walk& w, const Cuts& c, uint32_t end)
{
  w.end = end;
  if (c.f[0] && upper(w.tx + w.dx) < w.end) w.end = upper(w.tx + w.dx);
  if (c.f[1] && upper(w.ty + w.dy) < w.end) w.end = upper(w.ty + w.dy);
  if (c.f[2] && upper(w.tz + w.dz) < w.end) w.end = upper(w.tz + w.dz);
}

VDBG_HD void resume(Walk& w, Cuts& c, uint32_t first, uint32_t end)
{
  const uint32_t moved = w.pos ^ first;
  if (c.f[0] && pos_field(moved, 0))
  {
    w.dx -= static_cast<uint64_t>(static_cast<int64_t>(c.f[0]));
    c.f[0] = 0;
  }
  if (c.f[1] && pos_field(moved, 1))
  {
    w.dy -= static_cast<uint64_t>(static_cast<int64_t>(c.f[1]));
    c.f[1] = 0;
  }
  if (c.f[2] && pos_field(moved, 2))
  {
    w.dz -= static_cast<uint64_t>(static_cast<int64_t>(c.f[2]));
    c.f[2] = 0;
  }
  cut_end(w, c, end);
}

// The end of chunk i of 2^p, as an upper word (thresholds i * 2^-p with i < 2^20
// have no lower bits; p <= 19: L1 < 3 * 2^22 in chunks of 32). The walk goes on while t <= 1, and no time
// equals 1: the nearest ideal times are 1 -+ 1 / (2 n), n < 2^23, and the sums
// are off by at most n * 2^-53.
VDBG_HD uint32_t chunk_end(uint32_t i, int p) { return upper(threshold_bits(i + 1u, p)); }

// Position and origin leaf of a chunk that begins at voxel v: pos as above,
// leaf coordinate = base + (field >> 3).
VDBG_HD uint32_t first_pos(int x, int y, int z)
{
  return static_cast<uint32_t>((x & 7) + kPosBias) | (static_cast<uint32_t>((y & 7) + kPosBias) << kPosBits) |
         (static_cast<uint32_t>((z & 7) + kPosBias) << (2 * kPosBits));
}
VDBG_HD int base_leaf(int v) { return (v >> 3) - kPosBias / 8; }

// Chunk 0 (walked with step<true>): it visits the sensor voxel itself first.
VDBG_HD void begin_head(Walk& w, double ddx, double ddy, double ddz, int p)
{
  w.dx  = bits_of(ddx);
  w.dy  = bits_of(ddy);
  w.dz  = bits_of(ddz);
  w.tx  = bits_of(hdda::mul(ddx, 0.5));
  w.ty  = bits_of(hdda::mul(ddy, 0.5));
  w.tz  = bits_of(hdda::mul(ddz, 0.5));
  w.end = chunk_end(0u, p);
}

} // namespace march
} // namespace vdbg
