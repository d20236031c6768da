// Host build of the walks over a span's windows (vdb_mapping_gb300/csrc/hdda.cuh:
// RunTrack, walk_window), compared with the walks over every voxel of the span:
// raytrace end points and the active voxels fast mode meets, bit for bit.
// Leaves over several 128^3 nodes, most without an active voxel; rays along
// lattice diagonals (tied crossings), nearly parallel to an axis, from far
// outside, long and short, and maps far from the origin. Prints one line per
// mismatch and "ok <cases>" at the end; exit status 1 on any mismatch.
#include "../../vdb_mapping_gb300/csrc/hdda.cuh"

#include <algorithm>
#include <cstdio>
#include <random>
#include <vector>

namespace H = vdbg::hdda;

namespace {

constexpr int kLeaves = 48;  // leaf cells per axis

struct World
{
  int base[3];                 // voxel of the first cell
  std::vector<uint8_t> state;  // per leaf cell: 0 none, 1 no active voxel, 2 active ones
  std::vector<uint64_t> on;    // [cells][8], word z, bit y * 8 + x
  H::Box box;
  int cell(const int v[3]) const
  {
    int c[3];
    for (int a = 0; a < 3; ++a)
    {
      const long long d = static_cast<long long>(v[a]) - base[a];
      if (d < 0 || d >= kLeaves * 8) return -1;
      c[a] = static_cast<int>(d >> 3);
    }
    return (c[0] * kLeaves + c[1]) * kLeaves + c[2];
  }
  bool active(const int v[3]) const
  {
    const int c = cell(v);
    return c >= 0 && state[c] == 2 && ((on[8 * static_cast<size_t>(c) + (v[2] & 7)] >> (((v[1] & 7) << 3) | (v[0] & 7))) & 1u);
  }
};

struct Topo
{
  const World& w;
  mutable bool act = false;
  bool node(const int v[3], int dim) const
  {
    for (int a = 0; a < 3; ++a)
      if (static_cast<long long>(v[a]) + dim <= w.base[a] || v[a] >= w.base[a] + kLeaves * 8) return false;
    return true;
  }
  bool has2(const int v[3]) const { return node(v, 4096); }
  bool has1(const int v[3]) const { return node(v, 128); }
  bool has0(const int v[3]) const
  {
    const int c = w.cell(v);
    act         = c >= 0 && w.state[c] == 2;
    return c >= 0 && w.state[c] != 0;
  }
  bool active0() const { return act; }
};

void build(World& w, std::mt19937_64& rng, const int base[3], int active_pct, bool full)
{
  std::uniform_int_distribution<int> pct(0, 99), bit(0, 63), word(0, 7);
  const size_t cells = static_cast<size_t>(kLeaves) * kLeaves * kLeaves;
  w.state.assign(cells, 0);
  w.on.assign(cells * 8, 0);
  for (int a = 0; a < 3; ++a)
  {
    w.base[a]        = base[a];
    w.box.lo[a]      = base[a];
    w.box.hi_excl[a] = base[a] + kLeaves * 8;
  }
  for (size_t c = 0; c < cells; ++c)
  {
    if (pct(rng) < 3) continue;
    w.state[c] = 1;
    if (pct(rng) >= active_pct) continue;
    w.state[c] = 2;
    if (full)
      for (int k = 0; k < 8; ++k) w.on[c * 8 + k] = ~0ull;  // a leaf entered one voxel too early or late shows
    else
      for (int k = pct(rng) % 30; k >= 0; --k) w.on[c * 8 + word(rng)] |= 1ull << bit(rng);
  }
}

} // namespace

int main()
{
  std::mt19937_64 rng(77);
  const int bases[5][3] = {{-192, -192, -192}, {0, 0, 0}, {1 << 20, -(1 << 20), 64}, {(1 << 21) - 384, -(1 << 21), 0}, {-200, 72, -4096}};
  int bad = 0, cases = 0, hits = 0, runs0 = 0, runs1 = 0, runs_many = 0, whole = 0;
  long long marks = 0, pieces = 0;
  for (int m = 0; m < 15; ++m)
  {
    World w;
    build(w, rng, bases[m % 5], m % 3 == 0 ? 1 : (m % 3 == 1 ? 5 : 30), (m & 1) != 0);
    std::uniform_real_distribution<double> u(-1.0, 1.0);
    std::uniform_int_distribution<int> small(-4, 4), at(-40, kLeaves * 8 + 40);
    for (int q = 0; q < 6000; ++q, ++cases)
    {
      double eye[3], dir[3];
      const int kind = q % 12;
      for (int a = 0; a < 3; ++a)
      {
        const int o = w.base[a] + at(rng), e = w.base[a] + at(rng);
        eye[a] = o + 0.5;
        dir[a] = e - o;
      }
      if (kind == 1 || kind == 2)
      {
        // lattice diagonals, from voxel centres, corners and leaf corners
        for (int a = 0; a < 3; ++a)
        {
          dir[a] = small(rng) * (kind == 1 ? 64.0 : 37.0);
          if (q & 16) eye[a] = static_cast<double>(w.base[a] + (at(rng) & ~7));
        }
      }
      else if (kind == 3)
      {
        for (int a = 0; a < 3; ++a) dir[a] *= a == q / 12 % 3 ? 1.0 : 1e-3 * u(rng);
      }
      else if (kind == 4)
      {
        for (int a = 0; a < 3; ++a) dir[a] *= a == q / 12 % 3 ? 1.0 : std::ldexp(u(rng), -(q / 36 % 60));
      }
      else if (kind == 5)
      {
        for (int a = 0; a < 3; ++a)
        {
          eye[a] += u(rng);
          dir[a] += u(rng);
        }
      }
      else if (kind == 6)
      {
        // from far outside, through the map
        const double back = std::ldexp(1.0, 8 + q / 12 % 20);
        for (int a = 0; a < 3; ++a)
        {
          const double to = eye[a] + 0.3 * u(rng), way = u(rng);
          eye[a]          = to - way * back;
          dir[a]          = 2.0 * way * back;
        }
      }
      else if (kind == 7)
      {
        for (int a = 0; a < 3; ++a) dir[a] = a == q / 12 % 3 ? dir[a] * 4.0 : 0.0;
      }
      else if (kind == 8)
      {
        for (int a = 0; a < 3; ++a) dir[a] *= 0.02;
      }
      else if (kind == 9)
      {
        for (int a = 0; a < 3; ++a) dir[a] *= 2000.0;
      }
      else if (kind == 10)
      {
        // |dx| = |dy| but for a few ulps: crossings that rounding may swap
        dir[1] = dir[0] * (1.0 + 2.2e-16 * small(rng));
        eye[1] = w.base[1] + (eye[0] - w.base[0]);
      }
      if (!H::point_ok(eye, dir, 0.0) || !H::point_ok(eye, dir, 1.0)) continue;
      const Topo topo{w};
      auto active = [&](const int v[3]) { return w.active(v); };
      // raytrace
      {
        H::Span sp, st;
        bool found, ft;
        uint32_t steps = 0;
        H::Runs runs;
        H::RunTrack<H::Runs> track(runs);
        H::trace_span(eye, dir, w.box, topo, sp, found, steps);
        steps = 0;
        H::trace_span(eye, dir, w.box, topo, st, ft, steps, track);
        if (found != ft || std::memcmp(&sp, &st, sizeof(sp)) != 0)
        {
          if (bad++ < 20) std::printf("span case %d kind %d\n", cases, kind);
          continue;
        }
        if (found)
        {
          double e0[3], e1[3];
          H::trace_walk(eye, dir, sp, 0.05, active, e0, steps);
          H::trace_walk_runs(H::make_ray(eye, dir, sp.t0, sp.t1), sp, runs.lo, runs.hi, runs.n, 0.05, active, e1);
          if (std::memcmp(e0, e1, sizeof(e0)) != 0 && bad++ < 20) std::printf("trace case %d kind %d\n", cases, kind);
          ++hits;
          runs0 += runs.n == 0;
          runs1 += runs.n == 1 && !track.all;
          runs_many += runs.n > 1;
          whole += track.all;
        }
      }
      // fast mode's spans
      {
        H::Ray r = H::make_ray(eye, dir, 0.0, 1.0);
        H::clip(r, w.box.lo, w.box.hi_excl);
        uint32_t steps = 0;
        H::Runs runs;
        H::RunTrack<H::Runs> track(runs);
        const float l1 = static_cast<float>(std::fabs(dir[0]) + std::fabs(dir[1]) + std::fabs(dir[2]));
        H::all_spans(r, topo, steps, [&](const H::Span& sp) {
          std::vector<int> a, b;
          const H::Ray fine = H::make_ray(eye, dir, sp.t0, sp.t1);
          H::Dda dda;
          H::dda_init(dda, fine, sp.t0, sp.t1, 0);
          do
          {
            if (w.active(dda.voxel)) a.insert(a.end(), dda.voxel, dda.voxel + 3);
          } while (H::dda_step(dda));
          for (int k = 0; k < runs.n; ++k)
            H::window_pieces(sp.t0, runs.lo[k], std::min(static_cast<double>(runs.hi[k]), sp.t1), l1, [&](double lo, double hi) {
              ++pieces;
              H::fast_walk_window(eye, dir, sp.t0, lo, hi, [&](const int v[3]) {
                if (w.active(v)) b.insert(b.end(), v, v + 3);
              });
            });
          if (a != b && bad++ < 20) std::printf("fast case %d kind %d\n", cases, kind);
          marks += static_cast<long long>(a.size() / 3);
        }, track);
      }
    }
  }
  std::printf("coverage hits %d runs 0: %d 1: %d more: %d whole: %d marks %lld pieces %lld\n", hits, runs0, runs1, runs_many,
              whole, marks, pieces);
  if (bad)
  {
    std::printf("FAILED %d of %d\n", bad, cases);
    return 1;
  }
  if (runs0 < 500 || runs1 < 500 || runs_many < 500 || whole < 100 || marks < 100000)
  {
    std::printf("FAILED coverage\n");
    return 1;
  }
  std::printf("ok %d\n", cases);
  return 0;
}
