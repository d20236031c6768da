// Host build of the chunked voxel walk the insertion kernel runs
// (vdb_mapping_gb300/csrc/march.cuh), compared step by step with the plain
// sequential DDA of castRayIntoGrid in doubles: every ray's chunks, walked one
// after the other, must give the same voxels in the same order. Rays cover
// ties (equal, doubled and small-ratio components), powers of two, single
// axes, all lengths up to the index range's. Prints one line per mismatch and
// "ok <rays> <steps>" at the end; exit status 1 on any mismatch.
#include "../../vdb_mapping_gb300/csrc/march.cuh"

#include <cstdio>
#include <cstdlib>
#include <random>

namespace M = vdbg::march;

namespace {

struct Sequential
{
  long v[3];
  int s[3];
  double t[3], d[3];
  explicit Sequential(const long o[3], const long e[3])
  {
    for (int a = 0; a < 3; ++a)
    {
      v[a]             = o[a];
      const double dir = static_cast<double>(e[a]) - static_cast<double>(o[a]);
      const double pos = static_cast<double>(o[a]) + 0.5;
      if (dir == 0.0)
      {
        s[a] = 0;
        t[a] = d[a] = 1.7976931348623157e308;
        continue;
      }
      const double inv = 1.0 / dir;
      s[a]             = inv > 0 ? 1 : -1;
      t[a]             = 0.0 + (static_cast<double>(o[a] + (inv > 0 ? 1 : 0)) - pos) * inv;
      d[a]             = s[a] * inv;
    }
  }
  // false: the walk ended before another voxel.
  bool next()
  {
    const int a    = t[0] < t[1] ? (t[0] < t[2] ? 0 : 2) : (t[1] < t[2] ? 1 : 2);
    const double c = t[a];
    if (c > 1.0) return false;
    t[a] += d[a];
    v[a] += s[a];
    return true;
  }
};

long long steps_total = 0;

// All chunks of a ray (of up to 2^clog steps) against the sequential walk. A
// chunk that may be walked without end checks is also walked three steps on,
// which must be the sequential walk's next voxels.
bool check(const long o[3], const long e[3], int clog)
{
  uint32_t n[3];
  int sgn[3];
  uint32_t l1 = 0;
  for (int a = 0; a < 3; ++a)
  {
    n[a]   = static_cast<uint32_t>(std::labs(e[a] - o[a]));
    sgn[a] = e[a] > o[a] ? 1 : e[a] < o[a] ? -1 : 0;
    l1 += n[a];
  }
  if (l1 == 0) return true;
  const int p = M::chunk_log2(l1, clog);
  Sequential seq(o, e);
  M::Axis ax[3];
  int bin = -1;
  for (uint32_t i = 0; i < (1u << p); ++i)
  {
    M::Walk w;
    M::Cuts c{{0, 0, 0}};
    long at[3];
    const uint32_t end = M::chunk_end(i, p);
    if (i == 0)
    {
      double dd[3];
      for (int a = 0; a < 3; ++a)
      {
        dd[a] = n[a] ? M::axis_delta(n[a]) : 1.7976931348623157e308;
        at[a] = o[a];
      }
      M::begin_head(w, dd[0], dd[1], dd[2], p);
    }
    else
    {
      const uint64_t tau = M::threshold_bits(i, p);
      const int j        = p - 1 - M::log2_floor(i);
      if (j != bin)
        for (int a = 0; a < 3; ++a) ax[a] = n[a] ? M::axis_entry(n[a], j) : M::axis_never();
      bin = j;
      M::Start s[3];
      for (int a = 0; a < 3; ++a)
      {
        s[a]   = M::start_axis(ax[a], n[a], i, p, tau);
        at[a]  = o[a] + sgn[a] * static_cast<long>(s[a].k);
        c.f[a] = static_cast<int8_t>(s[a].df);
        if (s[a].df < -1 || s[a].df > 1) { std::printf("df %d\n", s[a].df); return false; }
      }
      w.tx = s[0].t, w.ty = s[1].t, w.tz = s[2].t;
      w.dx = s[0].d, w.dy = s[1].d, w.dz = s[2].d;
      M::cut_end(w, c, end);
    }
    w.px  = sgn[0];
    w.py  = sgn[1] * (1 << M::kPosBits);
    w.pz  = sgn[2] * (1 << (2 * M::kPosBits));
    w.pos = M::first_pos(static_cast<int>(at[0]), static_cast<int>(at[1]), static_cast<int>(at[2]));
    const uint32_t first = w.pos;
    long base[3];
    for (int a = 0; a < 3; ++a) base[a] = 8l * M::base_leaf(static_cast<int>(at[a]));
    // The sequential walk stands where the chunk begins.
    for (int a = 0; a < 3; ++a)
      if (at[a] != seq.v[a])
      {
        std::printf("start n=(%u,%u,%u) chunk %u axis %d: %ld, not %ld\n", n[0], n[1], n[2], i, a, at[a], seq.v[a]);
        return false;
      }
    uint32_t steps = 0;
    for (;;)
    {
      if (!M::has_step(w))
      {
        if (i != 0 && w.end != end)
        {
          M::resume(w, c, first, end);
          continue;
        }
        break;
      }
      if (i == 0)
        M::step<true>(w);
      else
        M::step<false>(w);
      if (++steps > M::kMaxSteps) { std::printf("too many steps\n"); return false; }
      const bool more = seq.next();
      const long x = base[0] + M::pos_field(w.pos, 0), y = base[1] + M::pos_field(w.pos, 1), z = base[2] + M::pos_field(w.pos, 2);
      if (!more || x != seq.v[0] || y != seq.v[1] || z != seq.v[2])
      {
        std::printf("step n=(%u,%u,%u) chunk %u step %u\n", n[0], n[1], n[2], i, steps);
        return false;
      }
      const int bit = M::plane_bit(w.pos);
      if (bit != static_cast<int>(((y & 7) << 3) | (x & 7)) || M::plane_of(w.pos) != static_cast<int>(z & 7))
      {
        std::printf("bit\n");
        return false;
      }
    }
    steps_total += steps;
    if (M::chunk_is_free(i) && w.end == end)
    {
      Sequential ahead = seq;
      for (int k = 0; k < 3; ++k)
      {
        M::step_free(w);
        const bool more = ahead.next();
        for (int a = 0; a < 3; ++a)
          if (!more || base[a] + static_cast<long>(M::pos_field(w.pos, a)) != ahead.v[a])
          {
            std::printf("past the end n=(%u,%u,%u) chunk %u\n", n[0], n[1], n[2], i);
            return false;
          }
      }
    }
  }
  if (seq.next())
  {
    std::printf("end n=(%u,%u,%u)\n", n[0], n[1], n[2]);
    return false;
  }
  return true;
}

} // namespace

int main(int argc, char** argv)
{
  const long scale = argc > 1 ? std::atol(argv[1]) : 1;
  std::mt19937_64 rng(20240611);
  auto uni = [&](long lo, long hi) { return std::uniform_int_distribution<long>(lo, hi)(rng); };
  auto logu = [&](double hi) {
    return static_cast<long>(std::exp(std::uniform_real_distribution<double>(0.0, std::log(hi))(rng)));
  };
  long rays = 0;
  int bad   = 0;
  auto run = [&](long x, long y, long z) {
    long o[3] = {uni(-100000, 100000), uni(-100000, 100000), uni(-3000, 3000)};
    long e[3] = {o[0] + (uni(0, 1) ? x : -x), o[1] + (uni(0, 1) ? y : -y), o[2] + (uni(0, 1) ? z : -z)};
    ++rays;
    if (!check(o, e, M::kMinChunkLog2 + static_cast<int>(rays % 3))) ++bad;
  };
  // Structured: single axes, equal and small-ratio components, powers of two.
  const long pat[][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}, {1, 1, 0}, {1, 0, 1}, {0, 1, 1}, {1, 1, 1}, {1, 2, 0}, {2, 1, 1},
                         {1, 3, 0}, {3, 5, 0}, {1, 3, 5}, {2, 6, 0}, {1, 1, 2}, {2, 2, 1}, {1, 7, 49}, {4, 1, 16}, {3, 6, 12}};
  for (const auto& q : pat)
    for (long k = 1; k <= 600; k += 1 + k / 40) run(q[0] * k, q[1] * k, q[2] * k);
  for (int b = 0; b < 14; ++b)
    for (int c = 0; c < 14; ++c)
      for (long off = -1; off <= 1; ++off) run((1l << b) + off, 1l << c, uni(0, 40));
  for (long n = 0; n < 300; ++n)
    for (long m = 0; m < 300; m += 7) run(n, m, uni(0, 20));
  // Random, over the lengths of depth cameras, LiDARs and the precision-stress rays.
  for (long k = 0; k < 6000 * scale; ++k) run(uni(0, 400), uni(0, 400), uni(0, 60));
  for (long k = 0; k < 2000 * scale; ++k) run(logu(10000), logu(10000), logu(10000));
  for (long k = 0; k < 1000 * scale; ++k) run(uni(0, 1400), uni(0, 1400), uni(0, 200));
  // Beyond the table of the kernel, up to the index range.
  for (long k = 0; k < 6; ++k) run(logu(4194303), logu(4194303), logu(4194303));
  run(4194303, 4194303, 4194303);
  run(4194303, 1, 0);
  run(4194304 / 3, 4194304 / 7, 5);
  if (bad)
  {
    std::printf("%d of %ld rays differ\n", bad, rays);
    return 1;
  }
  std::printf("ok %ld %lld\n", rays, steps_total);
  return 0;
}
