// kernels.cuh — the scan-insertion kernels.
//
//   k_prep     VDBMapping.hpp:499-519   NaN skip, FP64 length + max-range clip,
//                                       worldToIndex of the endpoint, L1 length,
//                                       direction-bin histogram
//   k_scan     (none)                   exclusive scan of the bin histogram
//   k_scatter  (none)                   counting-sort scatter of ray ids (rays
//                                       grouped by direction)
//   k_march    VDBMapping.hpp:550-566   DDA from the sensor voxel to the endpoint
//                                       voxel, in chunks; ORs the visited voxels
//                                       into the per-leaf update masks
//   k_mark_hits VDBMapping.hpp:533-536  hit bits of unclipped endpoints
//   k_compact  (none)                   touched blocks -> flat touched-leaf list
//                                       (a dropped marking)
//   k_sweep    VDBMapping.hpp:731-792 + finds the touched leaves; per leaf the FP32
//              OccupancyVDBMapping.hpp:92-117  log-odds update, thresholds, clamp,
//                                       active mask; clears the update masks
//   k_change_* VDBMapping.hpp:733-781   the change set in order
//   k_section_* VDBMapping.hpp:883-1085 map sections out of and into the map
//   k_rehash   (none)                   rebuilds the block hash after growth
//   k_topo_build VDBMapping.hpp:1436-1449  the volume ray intersector's view of
//                                       the map: node sets and active-leaf box
//   k_fast_spans, k_fast_walk VDBMapping.hpp:577-602  fast mode: the
//                                       intersector's spans of each ray, then
//                                       the active map voxels along each span
//   k_trace_*  VDBMapping.hpp:675-721   raytrace queries: their order, the first
//                                       spans, then the voxel walks
//   k_morph_*  VDBMapping.hpp:1094-1147 dilation / erosion of section leaves
//   k_wall_voxels VDBMapping.hpp:1210-1236  artificial walls, castRayIntoGrid per layer
//   k_artificial_restore VDBMapping.hpp:1153-1166  restoreMapIntegrity
#pragma once

#include "device_common.cuh"
#include "hdda.cuh"
#include "march.cuh"
#include "morph.cuh"

namespace vdbg {

// Length classes of the sort, longest first: rays of 2^9 chunks and more
// (march.cuh), one class per number of chunks down to two, and those of one
// chunk by halves of a chunk. The rays of a class have the same number of
// chunks (the first class up to the scan's longest ray), so the lanes of a
// ray group walk equally far.
__device__ __forceinline__ int ray_class(uint32_t l1, int clog)
{
  const int p = march::chunk_log2(l1, clog);
  return p > 0 ? max(9 - p, 0) : (l1 > (1u << (clog - 1)) ? 9 : 10);
}
// log2 of the chunks of class k's rays, at most.
__device__ __forceinline__ int class_log2(int k, uint32_t max_l1, int clog)
{
  return k == 0 ? max(9, march::chunk_log2(max_l1, clog)) : max(9 - k, 0);
}
static_assert(kLenClasses == 11, "length classes");

// Sort bucket of a ray of scan s (voxel offset d from the sensor voxel, L1
// length l1): its length class, then the scan, then the cube-map face of the
// dominant axis and a 13 x 13 cell on it (6 * 169 = 1014 direction cells).
// Rays of one bucket are angular neighbours of similar length in one map; a
// warp walks 32 consecutive rays of this order, so its lanes go through the
// same leaves and their runs merge. Order only; the map does not depend on it.
__device__ __forceinline__ int ray_bucket(int dx, int dy, int dz, uint32_t l1, int s, const ScanTable& t)
{
  const int n_scans = t.n;
  const int ax = abs(dx), ay = abs(dy), az = abs(dz);
  int face, u, v, mx;
  if (ax >= ay && ax >= az)
  {
    face = dx >= 0 ? 0 : 1;
    u    = dy;
    v    = dz;
    mx   = ax;
  }
  else if (ay >= az)
  {
    face = dy >= 0 ? 2 : 3;
    u    = dx;
    v    = dz;
    mx   = ay;
  }
  else
  {
    face = dz >= 0 ? 4 : 5;
    u    = dx;
    v    = dy;
    mx   = az;
  }
  const int cls  = ray_class(l1, t.clog);
  const int base = (cls * n_scans + s) * kDirCells;
  if (mx == 0) return base;
  const int iu = static_cast<int>((static_cast<long long>(u + mx) * 13) / (2 * mx + 1));
  const int iv = static_cast<int>((static_cast<long long>(v + mx) * 13) / (2 * mx + 1));
  return base + face * 169 + iv * 13 + iu;
}
static_assert(6 * 169 == kDirCells, "direction cells");

// Points of the call: a table of several scans holds its total in
// first[n] (so a captured step may launch for the scratch capacity `n`).
__device__ __forceinline__ int64_t points_of(const ScanTable& t, int64_t n)
{
  return t.n > 1 ? min(n, static_cast<int64_t>(__ldg(t.first + t.n))) : n;
}

// One thread per point. rays[i] = (end voxel xyz, meta). Every lane of a
// warp stays to the end so the warp-wide reductions see a full mask.
// `pts_ref` (a captured step): the points' address is read there instead.
// Blocks of 64: a small scan's points spread over the SMs, whose FP64 pipe bounds
// this kernel (2,048 points 8.2 us, in blocks of 256 10.4; larger scans the same).
constexpr int kPrepThreads = 64;

__global__ void __launch_bounds__(kPrepThreads) k_prep(const char* __restrict__ pts, const char* const* pts_ref, int64_t n,
                                              int64_t stride, ScanTable t, int4* __restrict__ rays,
                                              uint16_t* __restrict__ ray_scan, uint32_t* __restrict__ hist,
                                              DevStatus* st)
{
  if (pts_ref) pts = *pts_ref;
  const int64_t i     = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const bool in_range = i < points_of(t, n);
  uint32_t meta       = 0;
  int ex = 0, ey = 0, ez = 0;
  unsigned long long visits = 0, hit = 0, valid = 0, nonfinite = 0;
  const int sc       = in_range ? scan_of_point(t, static_cast<uint32_t>(i)) : 0;
  const ScanGeom& g  = scan_geom(t, sc);
  if (in_range)
  {
    if (t.n > 1) ray_scan[i] = static_cast<uint16_t>(sc);
    const float* p = reinterpret_cast<const float*>(pts + i * stride);
    const float px = p[0], py = p[1], pz = p[2];
    if (g.map < 0)
    {
      // A scan of the batch that is not cast (no points to cast, NaN origin).
    }
    else if (isnan(px) || isnan(py) || isnan(pz))
    {
      // VDBMapping.hpp:505-510: skipped.
    }
    else if (isinf(px) || isinf(py) || isinf(pz))
    {
      // Undefined in the reference (the quantiser floors a NaN); skipped here.
      nonfinite = 1;
    }
    else
    {
      double wx = static_cast<double>(px), wy = static_cast<double>(py), wz = static_cast<double>(pz);
      const double dx = __dsub_rn(wx, g.ox), dy = __dsub_rn(wy, g.oy), dz = __dsub_rn(wz, g.oz);
      const double len =
        __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)));
      bool clipped = false;
      if (g.range > 0.0 && len > g.range)
      {
        // origin + (d / |d|) * range, component-wise (Vec3d::unit divides).
        wx      = __dadd_rn(g.ox, __dmul_rn(__ddiv_rn(dx, len), g.range));
        wy      = __dadd_rn(g.oy, __dmul_rn(__ddiv_rn(dy, len), g.range));
        wz      = __dadd_rn(g.oz, __dmul_rn(__ddiv_rn(dz, len), g.range));
        clipped = true;
      }
      const bool okx = world_to_index_axis(wx, g, ex);
      const bool oky = world_to_index_axis(wy, g, ey);
      const bool okz = world_to_index_axis(wz, g, ez);
      if (!(okx && oky && okz))
      {
        atomicOr(&st->error, kErrCoordRange);
        ex = ey = ez = 0;
      }
      else
      {
        const uint32_t l1 =
          static_cast<uint32_t>(abs(ex - g.ovx) + abs(ey - g.ovy) + abs(ez - g.ovz));
        meta   = kMetaValid | (clipped ? kMetaClipped : 0u) | (l1 & kMetaL1Mask);
        valid  = 1;
        visits = (l1 > 0 ? l1 + 1ull : 0ull) + (clipped ? 0ull : 1ull);
        hit    = clipped ? 0ull : 1ull;
      }
    }
    rays[i] = make_int4(ex, ey, ez, static_cast<int>(meta));
  }

  // Warp-aggregated counters and histogram (full warp: blockDim % 32 == 0).
  unsigned long long sv = visits, sh = hit, sr = valid, sn = nonfinite;
  for (int off = 16; off > 0; off >>= 1)
  {
    sv += __shfl_xor_sync(0xffffffffu, sv, off);
    sh += __shfl_xor_sync(0xffffffffu, sh, off);
    sr += __shfl_xor_sync(0xffffffffu, sr, off);
    sn += __shfl_xor_sync(0xffffffffu, sn, off);
  }
  const uint32_t longest = __reduce_max_sync(0xffffffffu, meta & kMetaL1Mask);
  if ((threadIdx.x & 31) == 0)
  {
    // (only the first length class needs the longest ray's length)
    if (ray_class(longest, t.clog) == 0) atomicMax(&st->max_l1, longest);
    if (sv) atomicAdd(&st->visits, sv);
    if (sh) atomicAdd(&st->hits, sh);
    if (sr) atomicAdd(&st->rays, sr);
    if (sn) atomicAdd(&st->nonfinite, sn);
  }
  const int b =
    valid ? ray_bucket(ex - g.ovx, ey - g.ovy, ez - g.ovz, meta & kMetaL1Mask, sc, t) : -1;
  const unsigned peers = __match_any_sync(0xffffffffu, b);
  if (valid && (__ffs(peers) - 1) == static_cast<int>(threadIdx.x & 31))
  {
    atomicAdd(hist + b, static_cast<uint32_t>(__popc(peers)));
  }
}

// Single block of 1024 threads: exclusive scan of the nb <= 4 * kScanTile bucket
// counts into cursor[], total into st->n_valid; clears the histogram for the next
// call. Four tiles of 4096 buckets, 4 a thread. One SM moves 135 kB, so the
// accesses are 16 bytes wide where the arrays are aligned, and all loads are made
// at once; the tiles' scans run side by side over one barrier. (Preparation, scan
// and scatter of 2,048 points 24 us, 32 with a tile after the other.)
__global__ void __launch_bounds__(1024) k_scan(uint32_t* __restrict__ hist, uint32_t* __restrict__ cursor,
                                               uint32_t nb, DevStatus* st)
{
  constexpr int kPer = 4, kTiles = 4;
  const bool wide = ((reinterpret_cast<uintptr_t>(hist) | reinterpret_cast<uintptr_t>(cursor)) & 15u) == 0u;
  __shared__ uint32_t sums[kTiles][32];
  const int t    = threadIdx.x;
  const int lane = t & 31, warp = t >> 5;
  uint32_t v[kTiles][kPer], local[kTiles], inc[kTiles], top[kTiles];
#pragma unroll
  for (int q = 0; q < kTiles; ++q)
  {
    const uint32_t i0 = static_cast<uint32_t>((q * 1024 + t) * kPer);
    if (wide && i0 + kPer <= nb)
    {
      const uint4 w = *reinterpret_cast<const uint4*>(hist + i0);
      v[q][0] = w.x, v[q][1] = w.y, v[q][2] = w.z, v[q][3] = w.w;
    }
    else
    {
#pragma unroll
      for (int k = 0; k < kPer; ++k) v[q][k] = i0 + k < nb ? hist[i0 + k] : 0u;
    }
    local[q] = v[q][0] + v[q][1] + v[q][2] + v[q][3];
  }
#pragma unroll
  for (int q = 0; q < kTiles; ++q) inc[q] = local[q];
#pragma unroll
  for (int off = 1; off < 32; off <<= 1)
#pragma unroll
    for (int q = 0; q < kTiles; ++q)
    {
      const uint32_t y = __shfl_up_sync(0xffffffffu, inc[q], off);
      if (lane >= off) inc[q] += y;
    }
#pragma unroll
  for (int q = 0; q < kTiles; ++q)
    if (lane == 31) sums[q][warp] = inc[q];
  __syncthreads();
  // Every warp scans the warps' sums of all tiles.
#pragma unroll
  for (int q = 0; q < kTiles; ++q) top[q] = sums[q][lane];
#pragma unroll
  for (int off = 1; off < 32; off <<= 1)
#pragma unroll
    for (int q = 0; q < kTiles; ++q)
    {
      const uint32_t y = __shfl_up_sync(0xffffffffu, top[q], off);
      if (lane >= off) top[q] += y;
    }
  uint32_t carry = 0;
#pragma unroll
  for (int q = 0; q < kTiles; ++q)
  {
    const uint32_t before = __shfl_sync(0xffffffffu, top[q], warp > 0 ? warp - 1 : 0);
    uint32_t base         = carry + (warp > 0 ? before : 0u) + inc[q] - local[q];
    const uint32_t i0     = static_cast<uint32_t>((q * 1024 + t) * kPer);
    if (wide && i0 + kPer <= nb)
    {
      *reinterpret_cast<uint4*>(cursor + i0) =
        make_uint4(base, base + v[q][0], base + v[q][0] + v[q][1], base + v[q][0] + v[q][1] + v[q][2]);
      *reinterpret_cast<uint4*>(hist + i0) = make_uint4(0u, 0u, 0u, 0u);
    }
    else
    {
#pragma unroll
      for (int k = 0; k < kPer; ++k)
      {
        if (i0 + k < nb)
        {
          cursor[i0 + k] = base;
          hist[i0 + k]   = 0u;
        }
        base += v[q][k];
      }
    }
    carry += __shfl_sync(0xffffffffu, top[q], 31);
  }
  if (t == 0) st->n_valid = carry;
}

// Multi-block form of k_scan for large bucket counts (batches of many
// maps): per-tile sums, a scan of the tile sums, then each tile's own scan
// from its offset. A tile is kScanTile buckets of a 1024-thread block.
constexpr uint32_t kScanTile     = 4096;
constexpr uint32_t kScanMaxTiles = 1024;

// Exclusive scan of one value per thread over a 1024-thread block; *total
// receives the block's sum.
__device__ __forceinline__ uint32_t block_scan_exclusive(uint32_t v, uint32_t* total)
{
  __shared__ uint32_t ws[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t inc   = v;
  for (int off = 1; off < 32; off <<= 1)
  {
    const uint32_t y = __shfl_up_sync(0xffffffffu, inc, off);
    if (lane >= off) inc += y;
  }
  if (lane == 31) ws[warp] = inc;
  __syncthreads();
  if (warp == 0)
  {
    uint32_t w = ws[lane];
    for (int off = 1; off < 32; off <<= 1)
    {
      const uint32_t y = __shfl_up_sync(0xffffffffu, w, off);
      if (lane >= off) w += y;
    }
    ws[lane] = w;
  }
  __syncthreads();
  const uint32_t excl = (warp > 0 ? ws[warp - 1] : 0u) + inc - v;
  *total              = ws[31];
  __syncthreads();
  return excl;
}

__global__ void __launch_bounds__(1024) k_scan_sums(const uint32_t* __restrict__ hist, uint32_t nb,
                                                    uint32_t* __restrict__ sums)
{
  const uint32_t i0 = blockIdx.x * kScanTile + threadIdx.x * 4u;
  uint32_t v        = 0;
#pragma unroll
  for (uint32_t k = 0; k < 4; ++k) v += (i0 + k < nb) ? hist[i0 + k] : 0u;
  uint32_t total = 0;
  block_scan_exclusive(v, &total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// Tile sums -> tile offsets (one block, at most kScanMaxTiles tiles); the
// grand total is the number of rays in the order.
__global__ void __launch_bounds__(1024) k_scan_tops(uint32_t* __restrict__ sums, uint32_t tiles, DevStatus* st)
{
  const uint32_t v = threadIdx.x < tiles ? sums[threadIdx.x] : 0u;
  uint32_t total   = 0;
  const uint32_t e = block_scan_exclusive(v, &total);
  if (threadIdx.x < tiles) sums[threadIdx.x] = e;
  if (threadIdx.x == 0) st->n_valid = total;
}

__global__ void __launch_bounds__(1024) k_scan_tiles(uint32_t* __restrict__ hist, uint32_t* __restrict__ cursor,
                                                     uint32_t nb, const uint32_t* __restrict__ sums)
{
  const uint32_t i0 = blockIdx.x * kScanTile + threadIdx.x * 4u;
  uint32_t v[4], local = 0;
#pragma unroll
  for (uint32_t k = 0; k < 4; ++k)
  {
    v[k] = (i0 + k < nb) ? hist[i0 + k] : 0u;
    local += v[k];
  }
  uint32_t total = 0;
  uint32_t base  = sums[blockIdx.x] + block_scan_exclusive(local, &total);
#pragma unroll
  for (uint32_t k = 0; k < 4; ++k)
  {
    if (i0 + k < nb)
    {
      cursor[i0 + k] = base;
      hist[i0 + k]   = 0u;
    }
    base += v[k];
  }
}

__global__ void __launch_bounds__(256) k_scatter(const int4* __restrict__ rays, int64_t n, ScanTable t,
                                                 uint32_t* __restrict__ cursor, int* __restrict__ order)
{
  const int64_t i      = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int4 r         = i < points_of(t, n) ? rays[i] : make_int4(0, 0, 0, 0);
  const uint32_t meta  = static_cast<uint32_t>(r.w);
  const bool valid     = (meta & kMetaValid) != 0;
  const int sc         = valid ? scan_of_ray(t, static_cast<uint32_t>(i)) : 0;
  const ScanGeom& g    = scan_geom(t, sc);
  const int b =
    valid ? ray_bucket(r.x - g.ovx, r.y - g.ovy, r.z - g.ovz, meta & kMetaL1Mask, sc, t) : -1;
  const unsigned peers = __match_any_sync(0xffffffffu, b);
  const int lane       = static_cast<int>(threadIdx.x & 31);
  const int leader     = __ffs(peers) - 1;
  uint32_t base        = 0;
  if (valid && lane == leader) base = atomicAdd(cursor + b, static_cast<uint32_t>(__popc(peers)));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (!valid) return;
  const int rank     = __popc(peers & ((1u << lane) - 1u));
  order[base + rank] = static_cast<int>(i);
}

__device__ __forceinline__ uint32_t lanemask_lt()
{
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// A slot of `count` for each active thread, one atomic for them together.
__device__ __forceinline__ uint32_t take_slot(uint32_t* count)
{
  const unsigned mask = __activemask();
  const int leader    = __ffs(mask) - 1;
  uint32_t base       = 0;
  if (static_cast<int>(threadIdx.x & 31) == leader) base = atomicAdd(count, static_cast<uint32_t>(__popc(mask)));
  return __shfl_sync(mask, base, leader) + static_cast<uint32_t>(__popc(mask & lanemask_lt()));
}

// ---------------------------------------------------------------------------
// k_march: castRayIntoGrid for every ray (VDBMapping.hpp:550-566) into the
// update grid's visited masks.
//
// The rays are walked in chunks of 32 to 128 voxel steps (march.cuh). A work
// item is chunk i of 32 rays that follow one another in the sorted order; they
// share a length class, so all of them have 2^p chunks of similar length and
// the lanes of a warp finish together (8-24% of the step slots are idle). Items are numbered class by class,
// ray group by ray group, chunk by chunk, and persistent warps take short runs
// of them from a device cursor: neither a long ray nor a small scan leaves
// most of the device waiting, and the lanes of an item walk neighbouring rays
// through the same leaves.
//
// A ray is monotone in every axis, so it visits each z-plane of each 8^3 leaf
// (64 voxels, one mask word) in a single contiguous run. A lane keeps the bits
// of its current run in a register; a run that ends is appended to the warp's
// record list in shared memory, ranked among the warp's lanes by one ballot.
// Records are applied 32 at a time, with every lane busy: a lane finds its
// run's leaf through the block index (allocating leaves and blocks as needed),
// marks it touched and ORs the run into the leaf's mask word.
//
// A leaf or block pool that runs out sets the error word; the walk goes on, so the
// allocation counters tell the whole demand (a full block hash, which cannot
// count, ends it), and the host grows the pools and runs the marking again
// (the ORs are idempotent).
//
// It is bound by the ALU pipe and instruction issue: a step of a warp takes
// about 51 instructions, more than half of them on the ALU pipe, which takes one every
// two cycles; applying 32 runs takes about 120. Measured on one GB300 against one
// FP64 walk per ray with a run buffer and a merging kernel behind it (marking
// alone, hits included): 262,144-point street scan 0.55 ms (1.10), 307,200-point
// depth image 0.45 (0.78), 65,536-point room scan 0.097 (0.23), 16,381 random
// rays of 2,490 steps 0.62 (4.0), 2,048 points 0.027 (0.10).
// Merging the runs per leaf in shared memory before they reach L2 was slower
// (0.66-0.73 ms on the street scan): neighbouring rays share too few leaves for
// the 150 instructions a merge of 32 runs takes, and the tables cost warps.
// ---------------------------------------------------------------------------
constexpr int kMarchWarps          = 2;    // per block (each works by itself)
constexpr int kMarchBlocks         = 14;   // per SM (72 registers; 12 and 16 were 1-4% slower)
constexpr int kMarchSteps          = 4;    // steps between looks at the ends and the record list
constexpr uint32_t kMarchRecords   = 32u * (kMarchSteps + 2);  // a remainder below 32, kMarchSteps steps, the last runs
constexpr uint32_t kMarchMaxRounds = 96;   // far above a chunk's rounds (one more per cut)

// The axis entries of march.cuh for all n below kAxisTableN in the binades
// [2^-(j + 1), 2^-j), j < kAxisTableJ, n fastest: with chunks of 64 steps all
// that rays with L1 up to 65,536 need. Other entries are computed when a chunk
// begins, and all of them for a map whose budget has no room for the table.
constexpr uint32_t kAxisTableN   = 16384;
constexpr int kAxisTableJ        = 10;
constexpr size_t kAxisTableBytes = size_t(kAxisTableN) * kAxisTableJ * (sizeof(ulonglong2) + sizeof(int2)) +
                                   size_t(kAxisTableN) * sizeof(double);

struct AxisTable
{
  ulonglong2* td;  // [kAxisTableJ][kAxisTableN] t1, d
  int2* kf;        // [kAxisTableJ][kAxisTableN] k1, df
  double* delta;   // [kAxisTableN] 1 / n (DBL_MAX for 0)
  uint32_t n;      // kAxisTableN, or 0: no table
};

__device__ __noinline__ march::Axis axis_entry_far(uint32_t n, int j) { return march::axis_entry(n, j); }

__device__ __forceinline__ march::Axis axis_at(const AxisTable& at, uint32_t n, int j)
{
  if (n < at.n && j < kAxisTableJ)
  {
    const ulonglong2 td = __ldg(at.td + static_cast<size_t>(j) * kAxisTableN + n);
    const int2 kf       = __ldg(at.kf + static_cast<size_t>(j) * kAxisTableN + n);
    return march::Axis{td.x, td.y, static_cast<uint32_t>(kf.x), kf.y};
  }
  return n == 0u ? march::axis_never() : axis_entry_far(n, j);
}

__device__ __forceinline__ double axis_delta_at(const AxisTable& at, uint32_t n)
{
  if (n < at.n) return __ldg(at.delta + n);
  return n == 0u ? hdda::kDblMax : march::axis_delta(n);
}

// One thread per entry.
__global__ void __launch_bounds__(256) k_axis_table(AxisTable at)
{
  const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= kAxisTableN * kAxisTableJ) return;
  const uint32_t n    = x % kAxisTableN;
  const int j         = static_cast<int>(x / kAxisTableN);
  const march::Axis a = n == 0u ? march::axis_never() : march::axis_entry(n, j);
  at.td[x]            = make_ulonglong2(a.t1, a.d);
  at.kf[x]            = make_int2(static_cast<int>(a.k1), a.df);
  if (j == 0) at.delta[n] = n == 0u ? hdda::kDblMax : march::axis_delta(n);
}

// A ray as the walk takes it: origin voxel, signed voxel counts, p (its 2^p
// chunks; negative: nothing to walk) and map.
struct MarchRay
{
  int ox, oy, oz;
  int nx, ny, nz;
  int p;
  int map;
};

__device__ __forceinline__ int sign_of(int x) { return (x > 0) - (x < 0); }

// Begins chunk i of ray r: the walk (its `end` possibly cut, see march::Cuts)
// and the origin leaf (bx, by, bz) its positions are relative to. Returns the
// chunk's end.
__device__ __forceinline__ uint32_t march_begin(const AxisTable& at, const MarchRay& r, uint32_t i, march::Walk& w,
                                                march::Cuts& cuts, int& bx, int& by, int& bz)
{
  const uint32_t nx = static_cast<uint32_t>(abs(r.nx)), ny = static_cast<uint32_t>(abs(r.ny)),
                 nz = static_cast<uint32_t>(abs(r.nz));
  const int sx = sign_of(r.nx), sy = sign_of(r.ny), sz = sign_of(r.nz);
  w.px         = sx;
  w.py         = sy * (1 << march::kPosBits);
  w.pz         = sz * (1 << (2 * march::kPosBits));
  int vx = r.ox, vy = r.oy, vz = r.oz;
  cuts.f[0] = cuts.f[1] = cuts.f[2] = 0;
  const uint32_t end = march::chunk_end(i, r.p);
  if (i == 0u)
  {
    march::begin_head(w, axis_delta_at(at, nx), axis_delta_at(at, ny), axis_delta_at(at, nz), r.p);
  }
  else
  {
    const uint64_t tau   = march::threshold_bits(i, r.p);
    const int j          = r.p - 1 - march::log2_floor(i);
    const march::Axis ax = axis_at(at, nx, j), ay = axis_at(at, ny, j), az = axis_at(at, nz, j);
    const march::Start x = march::start_axis(ax, nx, i, r.p, tau);
    const march::Start y = march::start_axis(ay, ny, i, r.p, tau);
    const march::Start z = march::start_axis(az, nz, i, r.p, tau);
    w.tx = x.t;
    w.ty = y.t;
    w.tz = z.t;
    w.dx = x.d;
    w.dy = y.d;
    w.dz = z.d;
    vx += sx * static_cast<int>(x.k);
    vy += sy * static_cast<int>(y.k);
    vz += sz * static_cast<int>(z.k);
    cuts.f[0] = static_cast<int8_t>(x.df);
    cuts.f[1] = static_cast<int8_t>(y.df);
    cuts.f[2] = static_cast<int8_t>(z.df);
    march::cut_end(w, cuts, end);
  }
  w.pos = march::first_pos(vx, vy, vz);
  bx    = march::base_leaf(vx);
  by    = march::base_leaf(vy);
  bz    = march::base_leaf(vz);
  return end;
}

__device__ __forceinline__ MarchRay march_ray(const int4& r, const ScanGeom& g, int clog)
{
  MarchRay q;
  q.ox              = g.ovx;
  q.oy              = g.ovy;
  q.oz              = g.ovz;
  q.nx              = r.x - g.ovx;
  q.ny              = r.y - g.ovy;
  q.nz              = r.z - g.ovz;
  const uint32_t l1 = static_cast<uint32_t>(r.w) & kMetaL1Mask;
  // (an endpoint in the sensor voxel is only a hit; k_mark_hits does it)
  q.p   = l1 == 0u ? -1 : march::chunk_log2(l1, clog);
  q.map = g.map;
  return q;
}

// Sets the position's voxel in the run: its bit is the low six bits of
// (pos & 7) | (pos >> 6 & ~7).
__device__ __forceinline__ void march_mark(uint32_t pos, uint32_t& lo, uint32_t& hi)
{
  const uint32_t s = (pos & 7u) | ((pos >> (march::kPosBits - 3)) & ~7u);
  asm("{\n\t"
      ".reg .pred p;\n\t"
      ".reg .b32 b, t;\n\t"
      "shf.l.wrap.b32 b, 0, 1, %2;\n\t"
      "and.b32 t, %2, 32;\n\t"
      "setp.ne.u32 p, t, 0;\n\t"
      "@p or.b32 %1, %1, b;\n\t"
      "@!p or.b32 %0, %0, b;\n\t"
      "}"
      : "+r"(lo), "+r"(hi)
      : "r"(s));
}

struct MarchWarp
{
  unsigned long long bits[kMarchRecords];  // a run: its visited voxels,
  uint32_t pos[kMarchRecords];             // its position (march::Walk), the lane above it
};

// ORs records [at, at + n) (n <= 32) into the update masks, one lane per run.
// Finding the word (block and leaf exist) costs three dependent loads: the
// hash bucket of the block with its slots, the leaf cell, the word itself.
// Anything else takes the general find-or-insert paths. A word that already
// holds the bits is left alone: the leaves around the sensor lie on every ray,
// and their words would otherwise take an atomic from each (an SM's own
// atomics drop the line from its L1, so a set bit is seen by the next load; a
// stale line only costs another atomic). A word without a bit may be its
// leaf's first of the window, which marks the leaf touched in its block.
__device__ __forceinline__ void march_apply(const MarchWarp& q, uint32_t at, uint32_t n, int bx, int by, int bz, int map,
                                            const MapView& m, const ChannelView& c, int lane)
{
  const bool have     = static_cast<uint32_t>(lane) < n;
  const uint32_t pos  = have ? q.pos[at + lane] : 0u;
  const int src       = static_cast<int>(pos >> (3 * march::kPosBits));
  constexpr int kLeaf = static_cast<int>(march::kPosMask >> 3);
  const int lx = __shfl_sync(0xffffffffu, bx, src) + (static_cast<int>(pos >> 3) & kLeaf);
  const int ly = __shfl_sync(0xffffffffu, by, src) + (static_cast<int>(pos >> (march::kPosBits + 3)) & kLeaf);
  const int lz = __shfl_sync(0xffffffffu, bz, src) + (static_cast<int>(pos >> (2 * march::kPosBits + 3)) & kLeaf);
  const int mp = __shfl_sync(0xffffffffu, map, src);
  if (!have) return;
  const unsigned long long bits = q.bits[at + lane];
  const unsigned long long bkey = pack_leaf_key(mp, lx >> 3, ly >> 3, lz >> 3);
  const uint32_t h              = block_home(bkey, m.bhmask);
  const ulonglong2 k2           = ld_ca_u64x2(m.bkeys + h);
  const int2 s2                 = ld_ca_s32x2(m.bslots + h);
  int b                         = k2.x == bkey ? s2.x : k2.y == bkey ? s2.y : -1;
  if (b < 0) b = find_or_insert_block(m, mp, lx >> 3, ly >> 3, lz >> 3);
  if (b < 0) return;
  const int cell = ((lx & 7) << 6) | ((ly & 7) << 3) | (lz & 7);
  int slot       = ld_ca_s32(m.bleaf + static_cast<size_t>(b) * 512 + cell);
  if (slot < 0) slot = find_or_insert_leaf(m, b, cell, mp, lx, ly, lz);
  if (slot < 0) return;
  unsigned long long* const u  = c.upd + static_cast<size_t>(slot) * 16 + march::plane_of(pos);
  const unsigned long long old = ld_ca_u64(u);
  if (bits & ~old) atomicOr(u, bits);
  if (old == 0ull)
  {
    touch_block(c, b);
    atomicOr(c.btouched + static_cast<size_t>(b) * 8 + (cell >> 6), 1ull << (cell & 63));
  }
}

// How a chunk is walked: chunk 0 with FP64 additions, the others with integer
// ones, with or without a look at the chunk's end at every step.
enum MarchMode : int
{
  kMarchFp64,
  kMarchChecked,
  kMarchFree,
};

// kMarchSteps steps: marks every voxel in the open run (lo, hi) before it is
// left, and appends the runs that end to the list. Returns whether the last
// step moved.
template <int kMode>
__device__ __forceinline__ bool march_steps(MarchWarp& q, march::Walk& w, uint32_t& lo, uint32_t& hi, uint32_t& n,
                                            uint32_t lt)
{
  uint32_t before = 0u;
#pragma unroll
  for (int s = 0; s < kMarchSteps; ++s)
  {
    march_mark(w.pos, lo, hi);
    before = w.pos;
    if (kMode == kMarchFp64)
      march::step<true>(w);
    else if (kMode == kMarchChecked)
      march::step<false>(w);
    else
      march::step_free(w);
    // The run ends when the voxel leaves its plane or leaf.
    const bool ends   = ((w.pos ^ before) & march::kCrossing) != 0u;
    const unsigned em = __ballot_sync(0xffffffffu, ends);
    if (ends)
    {
      const uint32_t p = n + static_cast<uint32_t>(__popc(em & lt));
      q.bits[p]        = (static_cast<unsigned long long>(hi) << 32) | lo;
      q.pos[p]         = before;
      lo = hi = 0u;
    }
    n += static_cast<uint32_t>(__popc(em));
  }
  return w.pos != before;
}

// Walks one chunk on every `live` lane and applies its runs. The chunk's first
// voxel is marked too: it is the sensor voxel, or the last of the chunk before.
// Returns the number of runs.
__device__ __forceinline__ uint32_t march_chunk(MarchWarp& q, int mode, march::Walk& w, march::Cuts& cuts, uint32_t end,
                                                bool live, int bx, int by, int bz, int map, const MapView& m,
                                                const ChannelView& c, int lane, uint32_t lt)
{
  const uint32_t first = w.pos;
  uint32_t n = 0, runs = 0;  // records in the list; all of the chunk's
  uint32_t lo = 0, hi = 0;   // the open run
  unsigned walking = 0xffffffffu;
  for (uint32_t round = 0;; ++round)
  {
    bool go;
    if (mode == kMarchFree)
    {
      march_steps<kMarchFree>(q, w, lo, hi, n, lt);
      go                   = march::has_step(w);
      const unsigned going = __ballot_sync(0xffffffffu, go);
      if (going != walking)
      {
        // (a lane that has passed its end stays where it is)
        walking = going;
        if (!go)
        {
          w.dx = w.dy = w.dz = 0ull;
          w.px = w.py = w.pz = 0;
        }
      }
    }
    else if (mode == kMarchChecked)
    {
      go = march_steps<kMarchChecked>(q, w, lo, hi, n, lt);
      if (!go && w.end != end)
      {
        march::resume(w, cuts, first, end);
        go = true;
      }
    }
    else
    {
      go = march_steps<kMarchFp64>(q, w, lo, hi, n, lt);
    }
    bool more = __any_sync(0xffffffffu, go);
    if (more && round >= kMarchMaxRounds)
    {
      // More than L1 + 1 visits: cannot happen for integer rays.
      if (lane == 0) atomicOr(&m.st->error, kErrStepBound);
      more = false;
    }
    if (!more)
    {
      march_mark(w.pos, lo, hi);
      const unsigned em = __ballot_sync(0xffffffffu, live);
      if (live)
      {
        const uint32_t p = n + static_cast<uint32_t>(__popc(em & lt));
        q.bits[p]        = (static_cast<unsigned long long>(hi) << 32) | lo;
        q.pos[p]         = w.pos;
      }
      n += static_cast<uint32_t>(__popc(em));
    }
    __syncwarp();
    while (n >= 32u || (!more && n > 0u))
    {
      const uint32_t take = min(n, 32u);
      n -= take;
      runs += take;
      march_apply(q, n, take, bx, by, bz, map, m, c, lane);
    }
    if (!more) break;
  }
  return runs;
}

// `cursor`: the sort's bucket cursors after k_scatter (each holds its
// bucket's end). `max_take`: items a warp takes at a time, at most. `one`: 1, as
// a value the compiler does not know (march::step).
__global__ void __launch_bounds__(kMarchWarps * 32, kMarchBlocks)
  k_march(const int4* __restrict__ rays, const int* __restrict__ order, const uint32_t* __restrict__ cursor,
          ScanTable t, MapView m, ChannelView c, AxisTable at, uint32_t max_take, uint32_t one)
{
  __shared__ MarchWarp warps[kMarchWarps];
  __shared__ uint32_t s_end[kLenClasses];             // rays of the classes up to each
  __shared__ unsigned long long s_items[kLenClasses];  // items of the classes up to each
  __shared__ int s_log2[kLenClasses];                  // log2 of a group's items, by class
  __shared__ uint32_t s_error;
  const int lane    = static_cast<int>(threadIdx.x & 31);
  const uint32_t lt = lanemask_lt();
  MarchWarp& q      = warps[threadIdx.x >> 5];
  c.cur_epoch       = *c.epoch;
  if (threadIdx.x < kLenClasses)
    s_end[threadIdx.x] = cursor[(threadIdx.x + 1u) * static_cast<uint32_t>(t.n) * kDirCells - 1u];
  __syncthreads();
  if (threadIdx.x == 0)
  {
    unsigned long long items = 0ull;
    uint32_t from            = 0u;
    for (int k = 0; k < kLenClasses; ++k)
    {
      const int l = class_log2(k, m.st->max_l1, t.clog);
      items += static_cast<unsigned long long>((s_end[k] - from + 31u) >> 5) << l;
      from       = s_end[k];
      s_items[k] = items;
      s_log2[k]  = l;
    }
    // A scan with a voxel index out of range is not cast at all (the prep
    // stage flagged it). Other errors of this call do not stop the walk.
    s_error = ld_relaxed_u32(&m.st->error) & kErrCoordRange;
  }
  __syncthreads();
  if (s_error != 0u) return;
  const unsigned long long total = s_items[kLenClasses - 1];
  // Several items at a time (their chunks follow one another and share
  // leaves), but no fewer than four turns for every warp.
  const unsigned long long share = total / (static_cast<unsigned long long>(gridDim.x) * kMarchWarps * 4ull);
  const uint32_t take = share < 1ull ? 1u : share > max_take ? max_take : static_cast<uint32_t>(share);

  unsigned long long it = 0ull, it_end = 0ull, runs = 0ull;
  uint32_t loaded = 0xffffffffu;  // first ray of the group held in `r`
  MarchRay r{0, 0, 0, 0, 0, 0, -1, 0};
  for (;;)
  {
    if (it == it_end)
    {
      // (a full block hash can count no demand: the walk ends, the host grows
      // it and marks again)
      if (lane == 0)
        it = (ld_relaxed_u32(&m.st->error) & kErrHashFull)
               ? total
               : atomicAdd(&m.st->item_cursor, static_cast<unsigned long long>(take));
      it = __shfl_sync(0xffffffffu, it, 0);
      if (it >= total) break;
      it_end = min(it + take, total);
    }
    int k = 0;
    while (it >= s_items[k]) ++k;
    const unsigned long long local = it - (k ? s_items[k - 1] : 0ull);
    const int l                    = s_log2[k];
    const uint32_t i               = static_cast<uint32_t>(local) & ((1u << l) - 1u);
    const uint32_t ray0            = (k ? s_end[k - 1] : 0u) + (static_cast<uint32_t>(local >> l) << 5);
    ++it;
    if (ray0 != loaded)
    {
      loaded             = ray0;
      const uint32_t idx = ray0 + static_cast<uint32_t>(lane);
      r.p                = -1;
      if (idx < s_end[k])
      {
        const int ri = order[idx];
        r            = march_ray(rays[ri], scan_geom(t, scan_of_ray(t, static_cast<uint32_t>(ri))), t.clog);
      }
    }
    const bool live = r.p >= 0 && (i >> r.p) == 0u;
    if (!__any_sync(0xffffffffu, live)) continue;
    march::Walk w{march::kNever, march::kNever, march::kNever, 0ull, 0ull, 0ull, 0u, 0u, 0, 0, 0, one};
    march::Cuts cuts{{0, 0, 0}};
    int bx = 0, by = 0, bz = 0;
    uint32_t end = 0u;
    if (live) end = march_begin(at, r, i, w, cuts, bx, by, bz);
    w.pos |= static_cast<uint32_t>(lane) << (3 * march::kPosBits);
    const bool cut = live && w.end != end;
    const int mode = i == 0u                                                            ? kMarchFp64
                     : march::chunk_is_free(i) && !__any_sync(0xffffffffu, cut) ? kMarchFree
                                                                                        : kMarchChecked;
    runs += march_chunk(q, mode, w, cuts, end, live, bx, by, bz, r.map, m, c, lane, lt);
  }
  if (lane == 0 && runs) atomicAdd(&m.st->runs, runs);
}

// Endpoint hits (setValueOn(end, true), VDBMapping.hpp:533-536): one thread
// per unclipped ray ORs the hit bit of its end voxel, creating the leaf when
// the DDA did not visit it (an endpoint in the sensor voxel).
__global__ void __launch_bounds__(256) k_mark_hits(const int4* __restrict__ rays, const int* __restrict__ order,
                                                   ScanTable t, MapView m, ChannelView c)
{
  if (ld_relaxed_u32(&m.st->error) != 0u) return;
  c.cur_epoch = *c.epoch;
  const uint32_t nv = m.st->n_valid;
  const uint32_t j  = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= nv) return;
  const int ri        = order[j];
  const int4 r        = rays[ri];
  const uint32_t meta = static_cast<uint32_t>(r.w);
  if (meta & kMetaClipped) return;
  const int mp = scan_geom(t, scan_of_ray(t, static_cast<uint32_t>(ri))).map;
  const int lx = r.x >> 3, ly = r.y >> 3, lz = r.z >> 3;
  const int b  = find_or_insert_block(m, mp, lx >> 3, ly >> 3, lz >> 3);
  if (b < 0) return;
  touch_block(c, b);
  const int cell = ((lx & 7) << 6) | ((ly & 7) << 3) | (lz & 7);
  const int slot = find_or_insert_leaf(m, b, cell, mp, lx, ly, lz);
  if (slot < 0) return;
  unsigned long long* bt = c.btouched + static_cast<size_t>(b) * 8 + (cell >> 6);
  if (!((*bt >> (cell & 63)) & 1ull)) atomicOr(bt, 1ull << (cell & 63));
  const uint32_t off = (static_cast<uint32_t>(r.z & 7) << 6) | (static_cast<uint32_t>(r.y & 7) << 3) |
                       static_cast<uint32_t>(r.x & 7);
  atomicOr(c.upd + static_cast<size_t>(slot) * 16 + 8 + (off >> 6), 1ull << (off & 63));
}

// Persistent sweep over the window's touched leaves (VDBMapping.hpp:731-792,
// OccupancyVDBMapping.hpp:92-117), each warp by itself, in three stages.
// Leaves: a lane takes a byte of a block's touched cells (eight cells), which
// gives leaf slots; neighbouring bytes go to different warps, and to as many
// as there are, because the blocks around the sensor are full and most others
// are not. Planes: up to eight leaves at a time, two
// planes per lane; a leaf's update and active words are read side by side, its
// update words cleared, and every 16-byte group of values (four voxels) with
// an update bit goes to the warp's list. Values: one lane per group, four
// groups per lane loaded before the first is used; the log-odds rules, the
// store, and an atomic on the active word where a voxel's state flipped (few
// do). So every lane has a group whatever the planes hold, and neighbouring
// lanes take neighbouring groups of a plane.
//
// It is bound by its 32-byte sectors at random places (2.6 times the bytes of the
// updated voxels on a street scan): its warps wait for their loads, and neither more
// groups ahead nor more leaves a batch make it faster. Measured on one GB300 against a
// compaction kernel and a sweep of one plane per lane (eight lanes per plane for
// batches): street scan, 1.48M leaves with 42 updates each, 0.44 ms (0.53); 32 maps,
// 6.3M leaves with 51, 1.8 ms (2.8); random long rays, 4.5M leaves with 9, 1.22 ms
// (1.46); 2,048 points, 3,400 leaves, 0.012 ms (0.030).
//
// kPerMap: the pool holds a batch of maps, each leaf takes its map's log-odds
// constants. kChanges: record the change set (every touched word, and the
// leaves with a flip).
constexpr int kSweepWarps  = 4;                // per block
constexpr int kSweepBlocks = 7;                // per SM (70 registers; 6 and 8 were 0-4% slower)
constexpr int kSweepLeaves = 8;                // leaves whose planes are handled together
constexpr int kSweepQueue  = 32 * 8 + kSweepLeaves;
constexpr int kSweepAhead  = 4;                // groups a lane loads ahead (2: 1% slower, 8: 15%)

struct SweepWarp
{
  unsigned long long act[kSweepLeaves * 8];  // visited-or-hit bits of a plane
  unsigned long long hit[kSweepLeaves * 8];
  unsigned long long on[kSweepLeaves * 8];   // active word before the sweep
  int leaves[kSweepQueue];                   // leaf slots found
  int slot[kSweepLeaves];                    // the leaves in hand
  int map[kSweepLeaves];
  unsigned short groups[kSweepLeaves * 128];  // plane << 4 | quad
};

// Exclusive scan over the warp; *total receives the sum.
__device__ __forceinline__ uint32_t warp_scan_exclusive(uint32_t v, int lane, uint32_t* total)
{
  uint32_t inc = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1)
  {
    const uint32_t y = __shfl_up_sync(0xffffffffu, inc, off);
    if (lane >= off) inc += y;
  }
  *total = __shfl_sync(0xffffffffu, inc, 31);
  return inc - v;
}

// The four bits of group `quad` in a plane's word held in shared memory.
__device__ __forceinline__ uint32_t group_bits(const unsigned long long* word, int quad)
{
  const uint32_t half = reinterpret_cast<const uint32_t*>(word)[quad >> 3];
  return (half >> (4 * (quad & 7))) & 0xfu;
}

// The log-odds node update (OccupancyVDBMapping.hpp:92-117) without branches:
// FP32 add, clamp only past the threshold; a hit never deactivates, a miss
// never activates. A value is clamped when it passes both the threshold and
// the limit: `past_max` / `past_min` are the outer of the two.
struct SweepOdds
{
  LogOdds lo;
  float past_max, past_min;
};

__device__ __forceinline__ SweepOdds sweep_odds(const LogOdds& lo)
{
  // (a threshold that is NaN is never passed)
  return SweepOdds{lo, lo.thres_max <= lo.max ? lo.max : lo.thres_max, lo.thres_min >= lo.min ? lo.min : lo.thres_min};
}

// One voxel: `act`, `hit` its update bits, `bit` its place in the group's
// states `on`.
__device__ __forceinline__ float update_voxel(float v, uint32_t act, uint32_t hit, uint32_t bit, const SweepOdds& o,
                                              uint32_t& on)
{
  const float x = __fadd_rn(v, hit ? o.lo.hit : o.lo.miss);
  if (act && (hit ? x > o.lo.thres_max : x < o.lo.thres_min)) on = hit ? on | bit : on & ~bit;
  const bool clip = hit ? x > o.past_max : x < o.past_min;
  return act ? (clip ? (hit ? o.lo.max : o.lo.min) : x) : v;
}

// The same for a miss.
__device__ __forceinline__ float update_missed(float v, uint32_t act, uint32_t bit, const SweepOdds& o, uint32_t& on)
{
  const float x = __fadd_rn(v, o.lo.miss);
  if (act && x < o.lo.thres_min) on &= ~bit;
  return act ? (x < o.past_min ? o.lo.min : x) : v;
}

// Bit q set where nibble q of x holds a bit.
__device__ __forceinline__ uint32_t nibbles(unsigned long long x)
{
  auto half = [](uint32_t y) {
    y |= y >> 1;
    y |= y >> 2;
    y &= 0x11111111u;        // bits 0, 4, .., 28
    y = (y | (y >> 3)) & 0x03030303u;
    y = (y | (y >> 6)) & 0x000f000fu;
    return (y | (y >> 12)) & 0xffu;
  };
  return half(static_cast<uint32_t>(x)) | (half(static_cast<uint32_t>(x >> 32)) << 8);
}

template <bool kPerMap, bool kChanges>
__global__ void __launch_bounds__(kSweepWarps * 32, kSweepBlocks)
  k_sweep(MapView m, ChannelView c, float* __restrict__ values, unsigned long long* __restrict__ active,
          uint32_t* __restrict__ flags, LogOddsTable lt, int n_maps, ChangeView ch, DevStatus* st, int gated)
{
  if (gated ? !marking_complete(st) : ld_relaxed_u32(&st->error) != 0u) return;
  __shared__ SweepWarp warps[kSweepWarps];
  __shared__ SweepOdds odds[kPerMap ? kMaxMaps : 1];
  SweepWarp& q        = warps[threadIdx.x >> 5];
  const int lane      = static_cast<int>(threadIdx.x & 31);
  const int w         = lane & 7;
  const uint32_t grp  = static_cast<uint32_t>(lane >> 3);
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw   = (gridDim.x * blockDim.x) >> 5;
  if (kPerMap)
  {
    for (int i = static_cast<int>(threadIdx.x); i < n_maps; i += kSweepWarps * 32) odds[i] = sweep_odds(lt.table[i]);
    __syncthreads();
  }
  const SweepOdds odds0 = sweep_odds(lt.lo0);
  // Byte i of the window's touched cells goes to warp i % nw; a warp looks at
  // `lanes` of its bytes at a time.
  const uint64_t bytes = *c.n_blist * 64ull;
  const uint32_t lanes = bytes >= 32ull * nw ? 32u : max(static_cast<uint32_t>(bytes) / nw, 1u);
  uint64_t next        = warp;
  uint32_t n = 0, head = 0;  // leaves found, and handled, of q.leaves
  uint32_t n_touched = 0;
  unsigned long long n_upd = 0;
  // The words of the batch that follows the one in hand, loaded ahead of its
  // values so that the two latencies overlap (lane: planes w of leaves grp and
  // grp + 4).
  unsigned long long vis[2], hit[2], on[2];
  int slot[2], map[2];
  uint32_t flag[2], take = 0;
  auto load_batch = [&]() {
    // ---- leaves ------------------------------------------------------------
    while (n - head < static_cast<uint32_t>(kSweepLeaves) && next < bytes)
    {
      if (head > 0)
      {
        // (fewer than eight are left: to the front)
        const int keep = head + lane < n ? q.leaves[head + lane] : -1;
        __syncwarp();
        if (keep >= 0) q.leaves[lane] = keep;
        n -= head;
        head = 0;
      }
      const uint64_t t = next + static_cast<uint64_t>(lane) * nw;
      next += static_cast<uint64_t>(lanes) * nw;
      uint32_t bits = 0;
      int4 s0{}, s1{};
      if (static_cast<uint32_t>(lane) < lanes && t < bytes)
      {
        const int b         = c.blist[t >> 6];
        const uint32_t i    = static_cast<uint32_t>(t) & 63u;  // cells 8i .. 8i + 7
        unsigned char* mark = reinterpret_cast<unsigned char*>(c.btouched + static_cast<size_t>(b) * 8) + i;
        bits                = *mark;
        if (bits)
        {
          *mark             = 0;
          const int4* cells = reinterpret_cast<const int4*>(m.bleaf + static_cast<size_t>(b) * 512 + i * 8u);
          s0                = cells[0];
          s1                = cells[1];
        }
      }
      uint32_t found = 0;
      uint32_t at    = n + warp_scan_exclusive(static_cast<uint32_t>(__popc(bits)), lane, &found);
      const int s[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if ((bits >> k) & 1u) q.leaves[at++] = s[k];
      n += found;
      n_touched += found;
      __syncwarp();
    }
    take = min(n - head, static_cast<uint32_t>(kSweepLeaves));
#pragma unroll
    for (int k = 0; k < 2; ++k)
    {
      const uint32_t i = static_cast<uint32_t>(k) * 4u + grp;
      vis[k] = hit[k] = on[k] = 0ull;
      slot[k]                 = -1;
      if (i < take)
      {
        slot[k]                     = q.leaves[head + i];
        const unsigned long long* u = c.upd + static_cast<size_t>(slot[k]) * 16;
        vis[k]                      = u[w];
        hit[k]                      = u[8 + w];
        on[k]                       = active[static_cast<size_t>(slot[k]) * 8 + w];
        if (w == 0)
        {
          flag[k] = flags[slot[k]];
          if (kPerMap) map[k] = m.origin[slot[k]].w;
        }
      }
    }
    head += take;
  };
  load_batch();
  while (take)
  {
    // ---- planes ------------------------------------------------------------
    uint32_t held = 0;  // groups with an update bit: 16 bits per plane
#pragma unroll
    for (int k = 0; k < 2; ++k)
    {
      const uint32_t i             = static_cast<uint32_t>(k) * 4u + grp;
      const uint32_t p             = i * 8u + static_cast<uint32_t>(w);
      const unsigned long long act = vis[k] | hit[k];
      if (slot[k] >= 0)
      {
        unsigned long long* u = c.upd + static_cast<size_t>(slot[k]) * 16;
        q.act[p]              = act;
        q.hit[p]              = hit[k];
        q.on[p]               = on[k];
        if (vis[k]) u[w] = 0ull;
        if (hit[k]) u[8 + w] = 0ull;
        if (kChanges)
        {
          ch.words[static_cast<size_t>(slot[k]) * 16 + w]     = 0ull;
          ch.words[static_cast<size_t>(slot[k]) * 16 + 8 + w] = 0ull;
        }
        if (w == 0)
        {
          q.slot[i] = slot[k];
          if (kPerMap) q.map[i] = map[k];
          // Part of the map from the first time it is swept on (every touched
          // leaf carries at least one update bit).
          if (flag[k] == 0u) flags[slot[k]] = 1u;
        }
      }
      n_upd += static_cast<uint32_t>(__popcll(act));
      held |= nibbles(act) << (16 * k);
    }
    uint32_t n_groups = 0;
    uint32_t at       = warp_scan_exclusive(static_cast<uint32_t>(__popc(held)), lane, &n_groups);
    // (bit 16k + q of `held` is group q of plane 32k + lane)
    for (uint32_t z = held; z; z &= z - 1u)
    {
      const uint32_t f = static_cast<uint32_t>(__ffs(static_cast<int>(z)) - 1);
      q.groups[at++]   = static_cast<unsigned short>(((f & 16u) << 5) | (static_cast<uint32_t>(lane) << 4) | (f & 15u));
    }
    __syncwarp();
    load_batch();
    // ---- values ------------------------------------------------------------
    for (uint32_t g0 = 0; g0 < n_groups; g0 += 32u * kSweepAhead)
    {
      float4 v[kSweepAhead];
      uint32_t e[kSweepAhead];
      auto at_group = [&](uint32_t x) {
        const uint32_t p = x >> 4;
        return reinterpret_cast<float4*>(values + static_cast<size_t>(q.slot[p >> 3]) * 512 + (p & 7u) * 64u) +
               plane_quad(static_cast<int>(x & 15u));
      };
#pragma unroll
      for (int k = 0; k < kSweepAhead; ++k)
      {
        const uint32_t g = g0 + static_cast<uint32_t>(k) * 32u + static_cast<uint32_t>(lane);
        e[k]             = g < n_groups ? q.groups[g] : 0xffffffffu;
        if (e[k] != 0xffffffffu) v[k] = *at_group(e[k]);
      }
#pragma unroll
      for (int k = 0; k < kSweepAhead; ++k)
      {
        if (e[k] == 0xffffffffu) continue;
        const uint32_t p  = e[k] >> 4;
        const int quad    = static_cast<int>(e[k] & 15u);
        const SweepOdds& o = kPerMap ? odds[q.map[p >> 3]] : odds0;
        const uint32_t a4 = group_bits(&q.act[p], quad), h4 = group_bits(&q.hit[p], quad), o4 = group_bits(&q.on[p], quad);
        uint32_t n4       = o4;
        if (h4)
        {
          v[k].x = update_voxel(v[k].x, a4 & 1u, h4 & 1u, 1u, o, n4);
          v[k].y = update_voxel(v[k].y, a4 & 2u, h4 & 2u, 2u, o, n4);
          v[k].z = update_voxel(v[k].z, a4 & 4u, h4 & 4u, 4u, o, n4);
          v[k].w = update_voxel(v[k].w, a4 & 8u, h4 & 8u, 8u, o, n4);
        }
        else
        {
          v[k].x = update_missed(v[k].x, a4 & 1u, 1u, o, n4);
          v[k].y = update_missed(v[k].y, a4 & 2u, 2u, o, n4);
          v[k].z = update_missed(v[k].z, a4 & 4u, 4u, o, n4);
          v[k].w = update_missed(v[k].w, a4 & 8u, 8u, o, n4);
        }
        *at_group(e[k])   = v[k];
        const uint32_t flip = n4 ^ o4;
        if (flip)
        {
          const int leaf = q.slot[p >> 3];
          atomicXor(active + static_cast<size_t>(leaf) * 8 + (p & 7u), static_cast<unsigned long long>(flip) << (4 * quad));
          if (kChanges)
          {
            // A hit only turns voxels on and a miss only off, so the flipped
            // bits that are now on are the hits of VDBMapping.hpp:768-772.
            unsigned long long* cw = ch.words + static_cast<size_t>(leaf) * 16 + (p & 7u);
            atomicOr(cw, static_cast<unsigned long long>(flip) << (4 * quad));
            if (flip & n4) atomicOr(cw + 8, static_cast<unsigned long long>(flip & n4) << (4 * quad));
            if (atomicExch(ch.epoch + leaf, ch.cur) != ch.cur) ch.list[atomicAdd(ch.count, 1u)] = leaf;
          }
        }
      }
    }
    __syncwarp();
  }
  for (int off = 16; off > 0; off >>= 1) n_upd += __shfl_xor_sync(0xffffffffu, n_upd, off);
  if (lane == 0 && n_upd) atomicAdd(&st->updates, n_upd);
  if (lane == 0 && n_touched) atomicAdd(&st->touched, n_touched);
  if (gated)
  {
    // The last block closes the window.
    __syncthreads();
    if (threadIdx.x == 0)
    {
      __threadfence();
      if (atomicAdd(&st->sweep_blocks, 1u) == gridDim.x - 1u)
      {
        st->sweep_blocks = 0u;
        finish_window(c, st);
      }
    }
  }
}

// Word of the plane of x (`a`, 0-7) of a leaf in OpenVDB's order, bit
// (y << 3) | z, from the z-plane words (bit (y << 3) | x): an 8 x 8 x 8
// transposition of x and z, the same both ways.
template <class Word>
__device__ __forceinline__ unsigned long long swap_mask_word(Word&& word, int a)
{
  unsigned long long out = 0ull;
#pragma unroll
  for (int b = 0; b < 8; ++b) out |= ((word(b) >> a) & 0x0101010101010101ull) << b;
  return out;
}

// A short change list in the order of its origins, in two kernels. Keys first: the
// leaves of map `map` (-1: all) as their origins' order, with the map's own order
// after it; head[0] counts them (0 at the start), head[1] is the length of the
// list (above `rows` nothing is done).
__global__ void __launch_bounds__(256) k_change_keys(ChangeView ch, const int4* __restrict__ origin, int map,
                                                     uint32_t rows, ulonglong2* __restrict__ keys,
                                                     uint32_t* __restrict__ head)
{
  const uint32_t n = *ch.count;
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k == 0u) head[1] = n;
  if (n > rows || k >= n) return;
  const int slot = ch.list[k];
  const int4 o   = origin[slot];
  if (map >= 0 && o.w != map) return;
  constexpr int kBias = 1 << 22;
  const unsigned long long x = static_cast<unsigned long long>((o.x + kBias) >> 3),
                           y = static_cast<unsigned long long>((o.y + kBias) >> 3),
                           z = static_cast<unsigned long long>((o.z + kBias) >> 3);
  keys[atomicAdd(head, 1u)] = make_ulonglong2((x << 42) | (y << 21) | z, static_cast<unsigned long long>(slot));
}

// One warp per leaf: its place is the number of smaller keys (equal origins, of
// different maps, by slot); its origin and its words in OpenVDB's order go to row
// `place` of pinned memory. Quadratic, but of 2,000 leaves a warp compares 63 keys
// a lane. An export of 2,110 leaves takes 54 us, of 10,079 236 (gathered, fetched
// and sorted on the host 560 and 2,100).
__global__ void __launch_bounds__(256) k_change_rows(ChangeView ch, const ulonglong2* __restrict__ keys,
                                                     const uint32_t* __restrict__ head, uint32_t rows,
                                                     int* __restrict__ out_o, unsigned long long* __restrict__ out_a,
                                                     unsigned long long* __restrict__ out_v, uint32_t* __restrict__ out_n)
{
  const uint32_t listed = head[1], n = head[0];
  if (blockIdx.x == 0u && threadIdx.x == 0u)
  {
    out_n[0] = n;
    out_n[1] = listed;
  }
  const uint32_t j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane   = static_cast<int>(threadIdx.x & 31);
  if (listed > rows || j >= n) return;
  const ulonglong2 mine = keys[j];
  uint32_t place        = 0;
  for (uint32_t k = static_cast<uint32_t>(lane); k < n; k += 32u)
  {
    const ulonglong2 other = keys[k];
    place += other.x < mine.x || (other.x == mine.x && other.y < mine.y) ? 1u : 0u;
  }
  place = __reduce_add_sync(0xffffffffu, place);
  // Lanes 0-7 hold the words flipped, 8-15 those flipped on.
  const unsigned long long w = lane < 16 ? ch.words[mine.y * 16ull + static_cast<unsigned long long>(lane)] : 0ull;
  const unsigned long long v = swap_mask_word([&](int b) { return __shfl_sync(0xffffffffu, w, (lane & 8) | b); }, lane & 7);
  if (lane < 8) out_a[static_cast<size_t>(place) * 8 + lane] = v;
  if (lane >= 8 && lane < 16) out_v[static_cast<size_t>(place) * 8 + (lane & 7)] = v;
  if (lane >= 16 && lane < 19)
  {
    const int shift = lane == 16 ? 42 : lane == 17 ? 21 : 0;
    out_o[static_cast<size_t>(place) * 3 + (lane - 16)] =
      static_cast<int>(((mine.x >> shift) & 0x1fffffull) << 3) - (1 << 22);
  }
}

// Gathers the listed change leaves of map `map` (-1: all): origin and the 16
// change words per leaf, one thread per word; out_n counts what was kept.
__global__ void k_gather_changes(ChangeView ch, const int4* __restrict__ origin, int map, int4* __restrict__ out_o,
                                 unsigned long long* __restrict__ out_w, uint32_t* __restrict__ out_n)
{
  const uint32_t n = *ch.count;
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int slot = ch.list[k];
  const int4 o   = origin[slot];
  if (map >= 0 && o.w != map) return;
  const uint32_t j = atomicAdd(out_n, 1u);
  out_o[j]         = o;
  for (int w = 0; w < 16; ++w) out_w[static_cast<size_t>(j) * 16 + w] = ch.words[static_cast<size_t>(slot) * 16 + w];
}

// Turns the touched-block list of a window into the flat list of its touched
// leaves, clearing the blocks' touched bits (a marking that is dropped: the
// sweep finds its leaves itself). One warp per block, one lane per 64-cell
// word.
__global__ void __launch_bounds__(256) k_compact(MapView m, ChannelView c)
{
  const uint32_t nb   = *c.n_blist;
  const int lane      = static_cast<int>(threadIdx.x & 31);
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw   = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t i = warp; i < nb; i += nw)
  {
    const int b                 = c.blist[i];
    unsigned long long* tw      = c.btouched + static_cast<size_t>(b) * 8;
    const unsigned long long w  = lane < 8 ? tw[lane] : 0ull;
    uint32_t total              = 0;
    uint32_t at                 = warp_scan_exclusive(static_cast<uint32_t>(__popcll(w)), lane, &total);
    uint32_t base               = 0;
    if (lane == 0) base = atomicAdd(c.n_touched, total);
    at += __shfl_sync(0xffffffffu, base, 0);
    if (w)
    {
      const int* cells = m.bleaf + static_cast<size_t>(b) * 512 + lane * 64;
      for (unsigned long long z = w; z; z &= z - 1) c.touched[at++] = cells[__ffsll(z) - 1];
      tw[lane] = 0ull;
    }
  }
}

// Test hook for the bounded waits: the empty cell of leaf (lx, ly, lz) of
// `map` is left pending, as if a thread had claimed it and never published
// its slot. *out: 0 planted, 1 the cell was not empty, 2 no block.
__global__ void k_test_stall_leaf(MapView m, int map, int lx, int ly, int lz, int* out)
{
  const int b = find_or_insert_block(m, map, lx >> 3, ly >> 3, lz >> 3);
  if (b < 0)
  {
    *out = 2;
    return;
  }
  const int cell = ((lx & 7) << 6) | ((ly & 7) << 3) | (lz & 7);
  const int prev = atomicCAS(m.bleaf + static_cast<size_t>(b) * 512 + cell, kLeafEmpty, kLeafPending);
  *out           = prev == kLeafEmpty ? 0 : 1;
}

// Starts a channel's first window: empty lists, epoch 1.
__global__ void k_window_init(ChannelView c)
{
  c.n_touched[0] = 0u;
  c.n_touched[2] = 1u;
  *c.n_blist     = 0u;
}

// A step whose rays were prepared ahead on another stream into their own
// status block: its counters and the quantiser's error bit join the call's
// status before the marking reads them.
__global__ void k_absorb_prep(DevStatus* st, const DevStatus* __restrict__ prep)
{
  st->rays += prep->rays;
  st->visits += prep->visits;
  st->hits += prep->hits;
  st->nonfinite += prep->nonfinite;
  st->n_valid = prep->n_valid;
  st->max_l1  = prep->max_l1;
  st->error |= prep->error;
}

// After a sweep that does not end its window itself, or a dropped marking.
__global__ void k_finish_window(ChannelView c, DevStatus* st) { finish_window(c, st); }

// Inserts blocks [0, n) of the block pool into an empty block hash.
__global__ void k_rehash(MapView m, uint32_t n)
{
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const int4 o                 = m.borigin[s];
  const unsigned long long key = pack_leaf_key(o.w, o.x, o.y, o.z);
  uint32_t h                   = block_home(key, m.bhmask);
  for (uint32_t probe = 0; probe <= m.bhmask; ++probe)
  {
    if (atomicCAS(m.bkeys + h, kEmptyKey, key) == kEmptyKey)
    {
      m.bslots[h] = static_cast<int>(s);
      return;
    }
    h = (h + 1) & m.bhmask;
  }
  atomicOr(&m.st->error, kErrHashFull);
}

// Zeroes the update words of the leaves on a channel's touched list (when a
// marking has to give up and its partial update grid is dropped).
__global__ void k_clear_touched(ChannelView c)
{
  const size_t words = static_cast<size_t>(*c.n_touched) * 16;
  for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < words;
       i += static_cast<size_t>(gridDim.x) * blockDim.x)
  {
    c.upd[static_cast<size_t>(c.touched[i >> 4]) * 16 + (i & 15u)] = 0ull;
  }
}

// Releases leaf slots [from, to) (allocated by a call whose marking was
// dropped): their cells in blocks below `keep_blocks` become empty again (the
// tables of younger blocks are cleared whole by the host). Their values,
// masks and flags were never written. The block hash must still hold the
// blocks (it is rebuilt afterwards).
__global__ void k_release_leaves(MapView m, uint32_t from, uint32_t to, uint32_t keep_blocks)
{
  const uint32_t slot = from + blockIdx.x * blockDim.x + threadIdx.x;
  if (slot >= to || slot >= m.capacity) return;
  const int4 o = m.origin[slot];
  const int lx = o.x >> 3, ly = o.y >> 3, lz = o.z >> 3;
  const unsigned long long key = pack_leaf_key(o.w, lx >> 3, ly >> 3, lz >> 3);
  uint32_t h = block_home(key, m.bhmask);
  for (uint32_t probe = 0; probe <= m.bhmask; ++probe)
  {
    const unsigned long long k = m.bkeys[h];
    if (k == kEmptyKey) return;
    if (k == key)
    {
      const int b = m.bslots[h];
      if (b >= 0 && static_cast<uint32_t>(b) < keep_blocks)
      {
        int* e = m.bleaf + static_cast<size_t>(b) * 512 + (((lx & 7) << 6) | ((ly & 7) << 3) | (lz & 7));
        if (*e == static_cast<int>(slot)) *e = kLeafEmpty;
      }
      return;
    }
    h = (h + 1) & m.bhmask;
  }
}

// After a pool growth: leaf cells whose allocation failed become empty again.
__global__ void k_reset_failed_leaves(int* __restrict__ bleaf, size_t cells)
{
  for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < cells;
       i += static_cast<size_t>(gridDim.x) * blockDim.x)
  {
    if (bleaf[i] == kLeafFailed) bleaf[i] = kLeafEmpty;
  }
}

// ---------------------------------------------------------------------------
// Map sections (VDBMapping.hpp:922-1085): the voxels of an index box taken
// out of the map, and sections written back, in OpenVDB's leaf order on the
// outside (x outermost, where the pool has z-planes).
//
// A section's candidates are leaf slots in the order of the leaf origins (-1:
// no leaf). The box itself gives that order, with one look-up per cell through
// the block index however many leaves the map holds; the kernels keep, number and
// write the leaves, and the copies go straight into the caller's arrays. Boxes of
// many cells for the leaves in them, and those of more than kSectionCells, list the
// map's leaves and sort them on the host (the rule is at section_candidates).
// Measured on one GB300 through getMapSection, a box of 936 cells: 0.06 ms (0.73-1.1
// ms with the list, per-call allocations, a counting call and the conversion and sort
// on the host), in a map of 4.2M leaves as much (1.5 ms).
// ---------------------------------------------------------------------------

// Slot of the existing leaf (lx, ly, lz) of map `map`, or -1 (no insertion;
// nothing may insert concurrently).
__device__ __forceinline__ int find_leaf(const MapView& m, int map, int lx, int ly, int lz)
{
  const unsigned long long bkey = pack_leaf_key(map, lx >> 3, ly >> 3, lz >> 3);
  uint32_t h                    = block_home(bkey, m.bhmask);
  for (uint32_t probe = 0; probe < kMaxProbes; ++probe)
  {
    const unsigned long long k = m.bkeys[h];
    if (k == kEmptyKey) return -1;
    if (k == bkey)
    {
      const int b = m.bslots[h];
      if (b < 0) return -1;
      const int s = m.bleaf[static_cast<size_t>(b) * 512 + (((lx & 7) << 6) | ((ly & 7) << 3) | (lz & 7))];
      return s >= 0 ? s : -1;
    }
    h = (h + 1) & m.bhmask;
  }
  return -1;
}

// Bits of z-plane word `w` of the leaf at `o` whose voxels lie inside [lo, hi].
__device__ __forceinline__ unsigned long long box_plane_mask(const int4& o, int w, int3 lo, int3 hi)
{
  const int z = o.z + w;
  if (z < lo.z || z > hi.z) return 0ull;
  const int x0 = max(lo.x - o.x, 0), x1 = min(hi.x - o.x, 7);
  const int y0 = max(lo.y - o.y, 0), y1 = min(hi.y - o.y, 7);
  if (x0 > x1 || y0 > y1) return 0ull;
  const unsigned long long row = ((1ull << (x1 - x0 + 1)) - 1ull) << x0;
  unsigned long long mask      = 0ull;
  for (int y = y0; y <= y1; ++y) mask |= row << (8 * y);
  return mask;
}

// Leaves of map `map` in the map (flags set) whose 8^3 box overlaps [lo, hi]
// (CoordBBox::hasOverlap): their slots into list, their number into *count (more than
// `room`: the rest is counted only).
__global__ void k_section_leaves(const int4* __restrict__ origin, const uint32_t* __restrict__ flags, uint32_t n,
                                 int map, int3 lo, int3 hi, uint32_t* __restrict__ list, uint32_t room,
                                 uint32_t* count)
{
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || flags[i] == 0u) return;
  const int4 o = origin[i];
  if (o.w != map) return;
  if (o.x > hi.x || o.x + 7 < lo.x || o.y > hi.y || o.y + 7 < lo.y || o.z > hi.z || o.z + 7 < lo.z) return;
  const uint32_t at = take_slot(count);
  if (at < room) list[at] = i;
}

// Candidates of the leaf cells first + [0, dims): one thread per cell, in the
// order of the origins.
__global__ void __launch_bounds__(256) k_section_cells(MapView m, int map, const uint32_t* __restrict__ flags, int3 first,
                                                       int3 dims, uint32_t n, int* __restrict__ cand)
{
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t z = i % static_cast<uint32_t>(dims.z), xy = i / static_cast<uint32_t>(dims.z);
  const int lx = first.x + static_cast<int>(xy / static_cast<uint32_t>(dims.y)),
            ly = first.y + static_cast<int>(xy % static_cast<uint32_t>(dims.y)), lz = first.z + static_cast<int>(z);
  const int slot = find_leaf(m, map, lx, ly, lz);
  cand[i]        = slot >= 0 && flags[slot] != 0u ? slot : -1;
}

// Origins of listed leaves (for the host's sort of a large box's list).
__global__ void k_section_origins(const uint32_t* __restrict__ list, uint32_t n, const int4* __restrict__ origin,
                                  int4* __restrict__ out)
{
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = origin[list[i]];
}

// Does a plane (w) of leaf `slot` hold a voxel of the section (getMapSection: an
// inside voxel is active or, full, holds a value other than the background 0)?
__device__ __forceinline__ bool section_plane(int slot, int w, const int4* __restrict__ origin,
                                              const float* __restrict__ values,
                                              const unsigned long long* __restrict__ active, int3 lo, int3 hi, int full)
{
  const unsigned long long inbox = box_plane_mask(origin[slot], w, lo, hi);
  bool any                       = (active[static_cast<size_t>(slot) * 8 + w] & inbox) != 0ull;
  if (full && !any && inbox)
  {
    const float4* vp = reinterpret_cast<const float4*>(values + static_cast<size_t>(slot) * 512 + w * 64);
    for (int q0 = 0; q0 < 16 && !any; q0 += 4)
#pragma unroll
      for (int k = 0; k < 4; ++k)
      {
        const int qd      = q0 + k;
        const uint32_t in = static_cast<uint32_t>(inbox >> (4 * qd)) & 0xfu;
        const float4 v    = vp[plane_quad(qd)];
        any = any || ((in & 1u) && v.x != 0.0f) || ((in & 2u) && v.y != 0.0f) || ((in & 4u) && v.z != 0.0f) ||
              ((in & 8u) && v.w != 0.0f);
      }
  }
  return any;
}

// Candidates of the leaf cells first + [0, dims) in the order of their origins
// (k_section_cells) and which of them give a leaf of the section, eight lanes per
// cell.
__global__ void __launch_bounds__(256) k_section_find(MapView m, int map, const uint32_t* __restrict__ flags, int3 first,
                                                      int3 dims, uint32_t n, const float* __restrict__ values,
                                                      const unsigned long long* __restrict__ active, int3 lo, int3 hi,
                                                      int full, int* __restrict__ cand, uint32_t* __restrict__ keep)
{
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t i = t >> 3;
  const int w      = static_cast<int>(t & 7u);
  int slot         = -1;
  if (w == 0 && i < n)
  {
    const uint32_t z = i % static_cast<uint32_t>(dims.z), xy = i / static_cast<uint32_t>(dims.z);
    const int lx = first.x + static_cast<int>(xy / static_cast<uint32_t>(dims.y)),
              ly = first.y + static_cast<int>(xy % static_cast<uint32_t>(dims.y)), lz = first.z + static_cast<int>(z);
    slot = find_leaf(m, map, lx, ly, lz);
    if (slot >= 0 && flags[slot] == 0u) slot = -1;
  }
  slot                 = __shfl_sync(0xffffffffu, slot, static_cast<int>(threadIdx.x & 24u));
  const bool any       = slot >= 0 && section_plane(slot, w, m.origin, values, active, lo, hi, full);
  const unsigned votes = __ballot_sync(0xffffffffu, any);
  if (w != 0 || i >= n) return;
  cand[i] = slot;
  keep[i] = ((votes >> (threadIdx.x & 24u)) & 0xffu) ? 1u : 0u;
}

// Which candidates give a leaf of the section, eight lanes per candidate, one
// z-plane each.
__global__ void __launch_bounds__(256) k_section_keep(const int* __restrict__ cand, uint32_t n,
                                                      const int4* __restrict__ origin,
                                                      const float* __restrict__ values,
                                                      const unsigned long long* __restrict__ active, int3 lo, int3 hi,
                                                      int full, uint32_t* __restrict__ keep)
{
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t j = t >> 3;
  const int w      = static_cast<int>(t & 7u);
  const int slot   = j < n ? cand[j] : -1;
  const bool any   = slot >= 0 && section_plane(slot, w, origin, values, active, lo, hi, full);
  const unsigned votes = __ballot_sync(0xffffffffu, any);
  if (w == 0 && j < n) keep[j] = ((votes >> (threadIdx.x & 24u)) & 0xffu) ? 1u : 0u;
}

// Positions of the kept candidates (exclusive scan) and their number; one
// block of 1024 threads.
__global__ void __launch_bounds__(1024) k_section_scan(const uint32_t* __restrict__ keep, uint32_t n,
                                                       uint32_t* __restrict__ pos, uint32_t* __restrict__ total)
{
  constexpr uint32_t kPer = 8;
  uint32_t carry          = 0;
  for (uint32_t tile = 0; tile < n; tile += 1024u * kPer)
  {
    const uint32_t i0 = tile + threadIdx.x * kPer;
    uint32_t v[kPer], local = 0;
#pragma unroll
    for (uint32_t k = 0; k < kPer; ++k)
    {
      v[k] = i0 + k < n ? keep[i0 + k] : 0u;
      local += v[k];
    }
    uint32_t sum = 0;
    uint32_t at  = carry + block_scan_exclusive(local, &sum);
#pragma unroll
    for (uint32_t k = 0; k < kPer; ++k)
    {
      if (i0 + k < n) pos[i0 + k] = at;
      at += v[k];
    }
    carry += sum;
  }
  if (threadIdx.x == 0) *total = carry;
}

// getMapSection of the kept candidates, one warp each: the voxels inside the
// box keep their state and value (full, extractFullLeaf VDBMapping.hpp:972-990)
// or value 1 where active (extractSparseLeaf :1001-1012), the others are
// background.
__global__ void __launch_bounds__(256) k_section_write(const int* __restrict__ cand, uint32_t n,
                                                       const uint32_t* __restrict__ keep,
                                                       const uint32_t* __restrict__ pos,
                                                       const int4* __restrict__ origin,
                                                       const float* __restrict__ values,
                                                       const unsigned long long* __restrict__ active, int3 lo, int3 hi,
                                                       int full, int* __restrict__ out_o, float* __restrict__ out_v,
                                                       unsigned long long* __restrict__ out_m)
{
  const uint32_t j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane   = static_cast<int>(threadIdx.x & 31);
  if (j >= n || !keep[j]) return;
  const int slot  = cand[j];
  const size_t at = pos[j];
  const int4 o    = origin[slot];
  if (lane < 3) out_o[at * 3 + lane] = lane == 0 ? o.x : lane == 1 ? o.y : o.z;
  // Lane b (0-7) holds the z-plane b of the states inside the box.
  unsigned long long in = 0ull, on = 0ull;
  if (lane < 8)
  {
    in = box_plane_mask(o, lane, lo, hi);
    on = active[static_cast<size_t>(slot) * 8 + lane] & in;
  }
  const unsigned long long mword =
    swap_mask_word([&](int b) { return __shfl_sync(0xffffffffu, on, b); }, lane & 7);
  const unsigned long long inword =
    swap_mask_word([&](int b) { return __shfl_sync(0xffffffffu, in, b); }, lane & 7);
  if (out_m && lane < 8) out_m[at * 8 + lane] = mword;
  if (!out_v) return;
#pragma unroll
  for (int k = 0; k < 16; ++k)
  {
    const int off                  = k * 32 + lane;  // x << 6 | y << 3 | z
    const unsigned long long isw   = __shfl_sync(0xffffffffu, inword, k >> 1);
    const unsigned long long onw   = __shfl_sync(0xffffffffu, mword, k >> 1);
    const bool inside              = (isw >> (off & 63)) & 1ull;
    float v                        = ((onw >> (off & 63)) & 1ull) ? 1.0f : 0.0f;
    if (full)
      v = inside ? values[static_cast<size_t>(slot) * 512 + leaf_float(((off & 7) << 6) | (off & 0x38) | (off >> 6))]
                 : 0.0f;
    out_v[at * 512 + off] = v;
  }
}

// applyMapSectionUpdateGrid, first loop (VDBMapping.hpp:1071-1077): the
// candidates lose their active voxels inside the box. One thread per
// (candidate, plane).
__global__ void k_section_clear(const int* __restrict__ cand, uint32_t n, const int4* __restrict__ origin,
                                unsigned long long* __restrict__ active, int3 lo, int3 hi)
{
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * 8u) return;
  const int slot = cand[t >> 3];
  if (slot < 0) return;
  const int w                    = static_cast<int>(t & 7u);
  const unsigned long long inbox = box_plane_mask(origin[slot], w, lo, hi);
  if (inbox) active[static_cast<size_t>(slot) * 8 + w] &= ~inbox;
}

// applyMapSectionUpdateGrid, second loop (:1078-1081): each section leaf's
// active voxels are set active in the map, creating the leaf (values at the
// background 0) where needed. One thread per section leaf. kVdb: the masks are
// in OpenVDB's order (else the pool's).
template <bool kVdb>
__global__ void k_section_set_states(MapView m, const int4* __restrict__ sec_o,
                                     const unsigned long long* __restrict__ sec_m, uint32_t n, int map,
                                     uint32_t* __restrict__ flags, unsigned long long* __restrict__ active)
{
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  unsigned long long word[8], any = 0ull;
#pragma unroll
  for (int w = 0; w < 8; ++w) any |= word[w] = sec_m[static_cast<size_t>(i) * 8 + w];
  if (!any) return;
  const int4 o = sec_o[i];
  const int lx = o.x >> 3, ly = o.y >> 3, lz = o.z >> 3;
  const int b  = find_or_insert_block(m, map, lx >> 3, ly >> 3, lz >> 3);
  if (b < 0) return;
  const int slot = find_or_insert_leaf(m, b, ((lx & 7) << 6) | ((ly & 7) << 3) | (lz & 7), map, lx, ly, lz);
  if (slot < 0) return;
  if (flags[slot] == 0u) flags[slot] = 1u;
#pragma unroll
  for (int w = 0; w < 8; ++w)
  {
    const unsigned long long bits = kVdb ? swap_mask_word([&](int k) { return word[k]; }, w) : word[w];
    if (bits) atomicOr(active + static_cast<size_t>(slot) * 8 + w, bits);
  }
}

// applyMapSectionGrid for the section's leaves (VDBMapping.hpp:1031-1046), one
// warp per section leaf: the map leaf takes all 512 values and states; it is
// created when `create[i]` (a voxel is active or not background), otherwise
// only an existing map leaf is overwritten.
__global__ void k_section_set_values(MapView m, const int4* __restrict__ sec_o, const float* __restrict__ sec_v,
                                     const unsigned long long* __restrict__ sec_m,
                                     const uint32_t* __restrict__ create, uint32_t n, int map,
                                     uint32_t* __restrict__ flags, float* __restrict__ values,
                                     unsigned long long* __restrict__ active)
{
  const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane   = static_cast<int>(threadIdx.x & 31);
  if (i >= n) return;
  int slot = -1;
  if (lane == 0)
  {
    const int4 o = sec_o[i];
    const int lx = o.x >> 3, ly = o.y >> 3, lz = o.z >> 3;
    if (create[i])
    {
      const int b = find_or_insert_block(m, map, lx >> 3, ly >> 3, lz >> 3);
      if (b >= 0) slot = find_or_insert_leaf(m, b, ((lx & 7) << 6) | ((ly & 7) << 3) | (lz & 7), map, lx, ly, lz);
    }
    else
    {
      slot = find_leaf(m, map, lx, ly, lz);
      if (slot >= 0 && flags[slot] == 0u) slot = -1;
    }
    if (slot >= 0 && flags[slot] == 0u) flags[slot] = 1u;
  }
  slot = __shfl_sync(0xffffffffu, slot, 0);
  if (slot < 0) return;
  for (int k = 0; k < 16; ++k)
    values[static_cast<size_t>(slot) * 512 + leaf_float(k * 32 + lane)] =
      sec_v[static_cast<size_t>(i) * 512 + k * 32 + lane];
  if (lane < 8) active[static_cast<size_t>(slot) * 8 + lane] = sec_m[static_cast<size_t>(i) * 8 + lane];
}

// The section tree's tiles (VDBMapping.hpp:1035 visits them as values): the map
// voxel at each point becomes the inactive background where a map leaf holds
// it. One thread per point.
__global__ void k_section_clear_voxels(MapView m, const int4* __restrict__ pts, uint32_t n, int map,
                                       const uint32_t* __restrict__ flags, float* __restrict__ values,
                                       unsigned long long* __restrict__ active)
{
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int4 p   = pts[i];
  const int slot = find_leaf(m, map, p.x >> 3, p.y >> 3, p.z >> 3);
  if (slot < 0 || flags[slot] == 0u) return;
  const int off = ((p.z & 7) << 6) | ((p.y & 7) << 3) | (p.x & 7);
  values[static_cast<size_t>(slot) * 512 + leaf_float(off)] = 0.0f;
  atomicAnd(active + static_cast<size_t>(slot) * 8 + (off >> 6), ~(1ull << (off & 63)));
}

// ---------------------------------------------------------------------------
// Fast mode and raytrace queries: the volume ray intersector
// (VDBMapping.hpp:1436-1449) over the map's leaves as they are at the call
// (the integrated ones, flags set). Nodes of 128^3 and 4096^3 voxels hold a
// leaf exactly when one of the map's leaves lies in them; they go to two
// open-addressing key sets built per call, leaf cells are looked up in the
// map's own block hash.
// ---------------------------------------------------------------------------
constexpr uint32_t kErrTopoFull = 128u;  // a node set ran out of probes (set size >= 2x the leaves)

struct TopoView
{
  unsigned long long* key1;  // 128^3-voxel nodes: pack_leaf_key(map, v >> 7)
  unsigned long long* key2;  // 4096^3-voxel nodes: pack_leaf_key(map, v >> 12)
  uint32_t mask;             // set capacity - 1 (both sets; >= 2x the map's blocks)
  int* box;                  // [6] min xyz, max xyz (inclusive) of the leaves with an active voxel
  uint32_t* count;           // [0] nonzero when the map has a leaf, [1] when an insert failed
  int map;
  // [blocks][8][2]: of word w, bit `cell & 63` of the first part is set when the
  // leaf in that cell of the block (cell >> 6 = w) is in the map; of the second
  // part, when it also holds an active voxel.
  unsigned long long* leafbits;
};

__device__ __forceinline__ bool topo_insert(unsigned long long* keys, uint32_t mask, unsigned long long key)
{
  uint32_t h = static_cast<uint32_t>(mix64(key)) & mask;
  for (uint32_t probe = 0; probe < kMaxProbes; ++probe)
  {
    const unsigned long long k = keys[h];
    if (k == key) return true;
    if (k == kEmptyKey)
    {
      const unsigned long long prev = atomicCAS(keys + h, kEmptyKey, key);
      if (prev == kEmptyKey || prev == key) return true;
    }
    h = (h + 1) & mask;
  }
  return false;
}

__device__ __forceinline__ bool topo_find(const unsigned long long* keys, uint32_t mask, unsigned long long key)
{
  uint32_t h = static_cast<uint32_t>(mix64(key)) & mask;
  for (uint32_t probe = 0; probe < kMaxProbes; ++probe)
  {
    const unsigned long long k = __ldg(keys + h);
    if (k == key) return true;
    if (k == kEmptyKey) return false;
    h = (h + 1) & mask;
  }
  return false;
}

// box = (INT_MAX x3, INT_MIN x3), counts 0: the empty CoordBBox of an
// intersector on a map without active voxels.
__global__ void k_topo_init(TopoView tv)
{
  if (threadIdx.x < 3) tv.box[threadIdx.x] = 0x7fffffff;
  if (threadIdx.x >= 3 && threadIdx.x < 6) tv.box[threadIdx.x] = static_cast<int>(0x80000000u);
  if (threadIdx.x < 2) tv.count[threadIdx.x] = 0u;
}

// One warp per block of 8^3 leaf cells: the bitmaps of its integrated leaves and
// of those with an active voxel; the block's nodes enter the node sets, and its
// active leaves widen the box. The bitmaps are written whole (no clearing, no
// atomics), a node is looked up once per block instead of once per leaf, and
// the box and the count take an atomic only from a warp that still changes
// them. Bound by the reads of every leaf's flag and active words: 70 us for a map of 3.3M leaves (150 us
// with a thread, two node lookups and up to three atomics per leaf, and 128 MB of
// node keys to clear).
constexpr int kTopoWarps = 8;

__global__ void __launch_bounds__(kTopoWarps * 32) k_topo_build(const uint32_t* __restrict__ flags,
                                                                const unsigned long long* __restrict__ active,
                                                                uint32_t blocks, MapView m, TopoView tv)
{
  const int lane   = static_cast<int>(threadIdx.x & 31);
  const uint32_t b = blockIdx.x * kTopoWarps + (threadIdx.x >> 5);
  if (b >= blocks) return;
  const int4 o = m.borigin[b];
  if (o.w != tv.map) return;  // (another map's block is never looked up)
  const int* cells = m.bleaf + static_cast<size_t>(b) * 512;
  unsigned long long mine_in = 0ull, mine_act = 0ull;  // lane w < 8: word w
  uint32_t xs = 0u, ys = 0u, zs = 0u;  // leaf coordinates of the block with an active leaf
#pragma unroll
  for (int half = 0; half < 2; ++half)
  {
    int slot[8];
    uint32_t in[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) slot[k] = __ldg(cells + half * 256 + k * 32 + lane);
#pragma unroll
    for (int k = 0; k < 8; ++k) in[k] = slot[k] >= 0 ? __ldg(flags + slot[k]) : 0u;
#pragma unroll
    for (int k = 0; k < 8; ++k)
    {
      unsigned long long any = 0ull;
      if (in[k])
      {
        const ulonglong2* a = reinterpret_cast<const ulonglong2*>(active + static_cast<size_t>(slot[k]) * 8);
        const ulonglong2 a0 = __ldg(a), a1 = __ldg(a + 1), a2 = __ldg(a + 2), a3 = __ldg(a + 3);
        any = a0.x | a0.y | a1.x | a1.y | a2.x | a2.y | a3.x | a3.y;
      }
      const unsigned iw = __ballot_sync(0xffffffffu, in[k] != 0u);
      const unsigned aw = __ballot_sync(0xffffffffu, any != 0ull);
      // cell = x * 64 + y * 8 + z: lanes 0-31 of step k hold x = word, y = (k & 1) * 4 + lane / 8
      const int word = half * 4 + (k >> 1);
      if (lane == word)
      {
        mine_in |= static_cast<unsigned long long>(iw) << (32 * (k & 1));
        mine_act |= static_cast<unsigned long long>(aw) << (32 * (k & 1));
      }
      if (aw) xs |= 1u << word;
      for (int q = 0; q < 4; ++q)
      {
        const uint32_t row = (aw >> (8 * q)) & 0xffu;
        zs |= row;
        if (row) ys |= 1u << ((k & 1) * 4 + q);
      }
    }
  }
  if (lane < 8) reinterpret_cast<ulonglong2*>(tv.leafbits)[static_cast<size_t>(b) * 8 + lane] = make_ulonglong2(mine_in, mine_act);
  const bool present = __any_sync(0xffffffffu, mine_in != 0ull);
  if (!present || lane != 0) return;
  if (*reinterpret_cast<volatile uint32_t*>(tv.count) == 0u) atomicOr(tv.count, 1u);
  const bool ok = topo_insert(tv.key1, tv.mask, pack_leaf_key(tv.map, o.x >> 1, o.y >> 1, o.z >> 1)) &&
                  topo_insert(tv.key2, tv.mask, pack_leaf_key(tv.map, o.x >> 6, o.y >> 6, o.z >> 6));
  if (!ok) atomicOr(tv.count + 1, 1u);
  if (!xs) return;
  const int lo[3] = {o.x * 64 + 8 * (__ffs(xs) - 1), o.y * 64 + 8 * (__ffs(ys) - 1), o.z * 64 + 8 * (__ffs(zs) - 1)};
  const int hi[3] = {o.x * 64 + 8 * (31 - __clz(xs)) + 7, o.y * 64 + 8 * (31 - __clz(ys)) + 7,
                     o.z * 64 + 8 * (31 - __clz(zs)) + 7};
  for (int a = 0; a < 3; ++a)
  {
    if (lo[a] < *reinterpret_cast<volatile int*>(tv.box + a)) atomicMin(tv.box + a, lo[a]);
    if (hi[a] > *reinterpret_cast<volatile int*>(tv.box + 3 + a)) atomicMax(tv.box + 3 + a, hi[a]);
  }
}

__device__ __forceinline__ bool voxel_in_map_range(const int v[3])
{
  return v[0] >= static_cast<int>(kVoxelMin) && v[0] < static_cast<int>(kVoxelMaxExcl) &&
         v[1] >= static_cast<int>(kVoxelMin) && v[1] < static_cast<int>(kVoxelMaxExcl) &&
         v[2] >= static_cast<int>(kVoxelMin) && v[2] < static_cast<int>(kVoxelMaxExcl);
}

// Block index of (bx, by, bz) of `map`, or -1 (read only).
__device__ __forceinline__ int find_block(const MapView& m, int map, int bx, int by, int bz)
{
  const unsigned long long bkey = pack_leaf_key(map, bx, by, bz);
  uint32_t h                    = block_home(bkey, m.bhmask);
  for (uint32_t probe = 0; probe < kMaxProbes; ++probe)
  {
    const unsigned long long k = m.bkeys[h];
    if (k == kEmptyKey) return -1;
    if (k == bkey)
    {
      const int b = m.bslots[h];
      return b >= 0 ? b : -1;
    }
    h = (h + 1) & m.bhmask;
  }
  return -1;
}

// The intersector's topology queries for hdda::walk (cell origins at each
// level; outside the map's coordinate range nothing exists). Leaf cells
// remember the last 64^3 block looked up: consecutive leaf cells of a ray
// mostly share one.
struct DevTopo
{
  TopoView tv;
  MapView m;
  mutable int cbx, cby, cbz, cb;  // last block coordinate and its index (-1: none)
  mutable int cw = -1;            // word of cb's leaf bitmap held in `bits` (-1: none)
  mutable ulonglong2 bits = {0ull, 0ull};
  mutable int at = 0;             // bit of the last cell found
  __device__ __forceinline__ bool has2(const int v[3]) const
  {
    return voxel_in_map_range(v) && topo_find(tv.key2, tv.mask, pack_leaf_key(tv.map, v[0] >> 12, v[1] >> 12, v[2] >> 12));
  }
  __device__ __forceinline__ bool has1(const int v[3]) const
  {
    return voxel_in_map_range(v) && topo_find(tv.key1, tv.mask, pack_leaf_key(tv.map, v[0] >> 7, v[1] >> 7, v[2] >> 7));
  }
  __device__ __forceinline__ bool has0(const int v[3]) const
  {
    const int bx = v[0] >> 6, by = v[1] >> 6, bz = v[2] >> 6;
    if (bx != cbx || by != cby || bz != cbz)
    {
      cbx = bx;
      cby = by;
      cbz = bz;
      cb  = voxel_in_map_range(v) ? find_block(m, tv.map, bx, by, bz) : -1;
      cw  = -1;
    }
    if (cb < 0) return false;
    const int cell = (((v[0] >> 3) & 7) << 6) | (((v[1] >> 3) & 7) << 3) | ((v[2] >> 3) & 7);
    if ((cell >> 6) != cw)
    {
      cw   = cell >> 6;
      bits = __ldg(reinterpret_cast<const ulonglong2*>(tv.leafbits) + static_cast<size_t>(cb) * 8 + cw);
    }
    at = cell & 63;
    return (bits.x >> at) & 1ull;
  }
  // The leaf has0 has just found holds an active voxel.
  __device__ __forceinline__ bool active0() const { return (bits.y >> at) & 1ull; }
};

// isValueOn of the map for voxels along one ray, remembering the last leaf
// (its block and slot, -1 when absent) and the active word of the z-plane
// last read (a near-horizontal ray stays in one plane of a leaf for many
// voxels). A leaf without an active voxel is known from the intersector's
// bitmaps (`bits`, TopoView leafbits), and its slot and active words are not
// read.
struct ActiveCache
{
  const MapView* m;
  const unsigned long long* active;
  int map;
  int lx, ly, lz;
  int b, slot;
  int wz;                   // plane (z & 7) held in `word`, -1 none
  unsigned long long word;  // active bits of plane wz of leaf `slot`
  int bx = 0x7fffffff, by = 0, bz = 0;  // block coordinate `b` was found for
  const unsigned long long* bits = nullptr;  // TopoView leafbits
  int aw = -1;                               // word of b's active-leaf bitmap held in `abits`
  unsigned long long abits = 0ull;
  __device__ __forceinline__ bool operator()(const int v[3])
  {
    const int x = v[0] >> 3, y = v[1] >> 3, z = v[2] >> 3;
    if (x != lx || y != ly || z != lz)
    {
      lx = x;
      ly = y;
      lz = z;
      // A ray crosses several leaves of a block (8^3 leaves) in a row: probe
      // the block hash only when the block changes.
      if ((x >> 3) != bx || (y >> 3) != by || (z >> 3) != bz)
      {
        bx = x >> 3;
        by = y >> 3;
        bz = z >> 3;
        b  = voxel_in_map_range(v) ? find_block(*m, map, bx, by, bz) : -1;
        aw = -1;
      }
      const int cell = ((x & 7) << 6) | ((y & 7) << 3) | (z & 7);
      bool maybe     = b >= 0;
      if (maybe)
      {
        if ((cell >> 6) != aw)
        {
          aw    = cell >> 6;
          abits = __ldg(bits + static_cast<size_t>(b) * 16 + 2 * aw + 1);
        }
        maybe = (abits >> (cell & 63)) & 1ull;
      }
      slot = maybe ? m->bleaf[static_cast<size_t>(b) * 512 + cell] : -1;
      if (slot < 0) slot = -1;
      wz = -1;
    }
    if (slot < 0) return false;
    const int pz = v[2] & 7;
    if (pz != wz)
    {
      word = active[static_cast<size_t>(slot) * 8 + pz];
      wz   = pz;
    }
    return (word >> (((v[1] & 7) << 3) | (v[0] & 7))) & 1ull;
  }
};

__device__ __forceinline__ hdda::Box topo_box(const TopoView& tv)
{
  hdda::Box b;
  for (int a = 0; a < 3; ++a)
  {
    b.lo[a]      = tv.box[a];
    b.hi_excl[a] = tv.box[3 + a] + 1;  // mBBox.max().offset(1)
  }
  return b;
}

// Fast mode (castRayIntoGridFast, VDBMapping.hpp:577-602, called by
// raycastPointCloud VDBMapping.hpp:520-526 when the map is not empty): the
// voxels of the intersector's spans that are active in the map are marked
// visited in the update grid. Those voxels' leaves exist, so nothing is
// allocated. The prep stage counted the castRayIntoGrid visits of the rays;
// they are replaced by the marks made here (k_fast_visits).
// Two phases, so that the lanes of a warp run the same loop: k_fast_spans
// walks the intersector's three coarse levels for every ray and writes the
// windows of its spans in which the voxel walk can meet an active voxel
// (hdda::RunTrack), in pieces of about hdda::kPieceVoxels voxel steps;
// k_fast_walk then walks the voxel DDA over one piece per thread. The spans and
// their marks are those of hdda::fast_cast_one. The span walk is bound by
// the FP64 pipe (74% busy; most of it the DDA start in each 128^3 node), the voxel
// walk by the latency of its loads: 262144 rays of 60 m at 0.05 m take 0.50 +
// 0.15 ms, where a walk of every voxel of every span took 0.61 after the span walk
// of 0.38 (the windows cost that one a quarter), its longest thread 841 voxels.
struct alignas(16) FastPiece
{
  double t0;      // the span's start, where its voxel walk starts
  double lo, hi;  // the piece: voxels entered in (lo, hi] (and the first one, lo <= t0)
  int ray;        // index into the ray records
  int pad;
};
// One span of a raytrace query, with the windows in which it can meet an active
// voxel.
struct alignas(16) SpanRec
{
  double t0, t1;
  int ray;  // the query
  int n;    // windows
  float lo[hdda::Runs::kMax], hi[hdda::Runs::kMax];
  int cls;  // length class: floor(log2) of the voxel steps over the windows, estimated
  int pad;
};
constexpr int kSpanClasses = 32;

// Item of a thread when each warp takes `lanes` of the items (threads past them
// take none: the value is >= n).
__device__ __forceinline__ uint32_t lane_item(uint32_t lanes, uint32_t n)
{
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  return lane < lanes ? warp * lanes + lane : n;
}

// Records written by a span kernel. `Count`: 64 bits for pieces, of which a ray may have
// any number.
template <class Rec, class Count>
struct SpanBuf
{
  Rec* rec;
  uint32_t cap;
  Count* count;                    // written (may exceed cap: the host grows and repeats)
  unsigned long long* dda_visits;  // castRayIntoGrid visits the prep counted for these rays
};
using PieceBuf = SpanBuf<FastPiece, unsigned long long>;
using TraceBuf = SpanBuf<SpanRec, uint32_t>;

// A ray's windows during its coarse walk, in shared memory (thread's column of a
// block's arrays): those of all its spans are written out as pieces when the ray
// is done, the warp's lanes together. Written where a span ends, at a different
// step in each lane, the records took longer than the walk.
constexpr int kSpanThreads = 32;  // (blocks of one warp: the rays of a block take very different times)
constexpr int kFastWindows = 12;
struct FastWindows
{
  double t0[kFastWindows][kSpanThreads], hi[kFastWindows][kSpanThreads];
  float lo[kFastWindows][kSpanThreads];
};

// All 32 lanes: the pieces of each lane's n windows, one atomic for the warp.
__device__ __forceinline__ void write_pieces(const FastWindows& w, int n, float l1, int ray,
                                             const PieceBuf& sb)
{
  const int x   = static_cast<int>(threadIdx.x);
  uint32_t mine = 0u;
  for (int k = 0; k < n; ++k)
    hdda::window_pieces(w.t0[k][x], w.lo[k][x], w.hi[k][x], l1, [&](double, double) { ++mine; });
  uint32_t total = 0u;
  uint32_t slot  = warp_scan_exclusive(mine, static_cast<int>(threadIdx.x & 31u), &total);
  unsigned long long base = 0ull;
  if ((threadIdx.x & 31u) == 0u && total) base = atomicAdd(sb.count, static_cast<unsigned long long>(total));
  base                = __shfl_sync(0xffffffffu, base, 0);
  const uint32_t room = base < sb.cap ? sb.cap - static_cast<uint32_t>(base) : 0u;
  FastPiece* rec      = sb.rec + base;
  for (int k = 0; k < n; ++k)
  {
    const double t0 = w.t0[k][x];
    hdda::window_pieces(t0, w.lo[k][x], w.hi[k][x], l1, [&](double from, double to) {
      if (slot < room) rec[slot] = FastPiece{t0, from, to, ray, 0};
      ++slot;
    });
  }
}

// Sink of hdda::RunTrack: [0, base) belong to spans that ended, [base, n) to the
// open one. Further windows join the open span's last; a span that finds no room
// writes the last window before it, whole.
struct FastSink
{
  FastWindows& w;
  const PieceBuf& sb;
  int ray = 0;
  int n = 0, base = 0;
  double t0 = 0.0;
  __device__ __forceinline__ void open(double t)
  {
    t0 = t;
    n  = base;
  }
  __device__ __forceinline__ void window(float lo, float hi)
  {
    const int x = static_cast<int>(threadIdx.x);
    if (base == kFastWindows)
    {
      n = --base;
      const double at = w.t0[n][x], from = w.lo[n][x];
      const unsigned long long slot = atomicAdd(sb.count, 1ull);
      if (slot < sb.cap) sb.rec[slot] = FastPiece{at, from > at ? from : -1.0, w.hi[n][x], ray, 0};
    }
    if (n < kFastWindows)
    {
      w.t0[n][x] = t0;
      w.lo[n][x] = lo;
      ++n;
    }
    w.hi[n - 1][x] = static_cast<double>(hi);
  }
  // The span ends (its last window may lie past its end).
  __device__ __forceinline__ void span(const hdda::Span& sp)
  {
    const int x = static_cast<int>(threadIdx.x);
    if (n > base) w.hi[n - 1][x] = fmin(w.hi[n - 1][x], sp.t1);
    base = n;
  }
};

__device__ __forceinline__ void fast_ray(const int4& r, const ScanGeom& g, double eye[3], double dir[3])
{
  const int o[3] = {g.ovx, g.ovy, g.ovz};
  const int e[3] = {r.x, r.y, r.z};
  for (int a = 0; a < 3; ++a)
  {
    eye[a] = hdda::add(static_cast<double>(o[a]), 0.5);
    dir[a] = hdda::sub(static_cast<double>(e[a]), static_cast<double>(o[a]));
  }
}

// `coarse`: one piece a span, for when there is no room for more.
// (12 warps an SM: 16, with 128 registers, spilled and took 16% longer)
__global__ void __launch_bounds__(kSpanThreads, 12) k_fast_spans(const int4* __restrict__ rays,
                                                                 const int* __restrict__ order, ScanTable t,
                                                                 MapView m, TopoView tv, PieceBuf sb,
                                                                 uint32_t lanes, int coarse)
{
  __shared__ FastWindows windows;
  // (read once per warp: the warp reduces below)
  const int lane = static_cast<int>(threadIdx.x & 31);
  if (__shfl_sync(0xffffffffu, lane == 0 ? ld_relaxed_u32(&m.st->error) : 0u, 0) != 0u) return;
  const uint32_t nv = m.st->n_valid;
  const uint32_t j  = lane_item(lanes, nv);
  unsigned long long dv = 0;
  double eye[3], dir[3];
  hdda::Ray ray;
  float l1f = 0.0f;
  int ri    = 0;
  bool todo = false;
  if (j < nv && tv.count[1] == 0u)
  {
    ri                = order[j];
    const int4 r      = rays[ri];
    const uint32_t l1 = static_cast<uint32_t>(r.w) & kMetaL1Mask;
    dv                = l1 > 0u ? l1 + 1ull : 0ull;
    todo              = tv.count[0] != 0u;
    const ScanGeom& g = scan_geom(t, scan_of_ray(t, static_cast<uint32_t>(ri)));
    fast_ray(r, g, eye, dir);
    l1f = static_cast<float>(fabs(dir[0]) + fabs(dir[1]) + fabs(dir[2]));
    ray = hdda::make_ray(eye, dir, 0.0, 1.0);
    hdda::clip(ray, topo_box(tv).lo, topo_box(tv).hi_excl);
  }
  else if (j < nv)
  {
    atomicOr(&m.st->error, kErrTopoFull);
  }
  FastSink sink{windows, sb, ri};
  if (todo)
  {
    DevTopo topo{tv, m, 0x7fffffff, 0, 0, -1};
    uint32_t steps = 0;
    hdda::RunTrack<FastSink> track(sink);
    if (coarse)
    {
      track.gap_voxels = INFINITY;
      l1f              = 0.0f;
    }
    const int w = hdda::all_spans(ray, topo, steps, [&](const hdda::Span& sp) { sink.span(sp); }, track);
    if (w == hdda::kWalkBound) atomicOr(&m.st->error, kErrStepBound);
  }
  __syncwarp();
  write_pieces(windows, sink.base, l1f, ri, sb);
  for (int off = 16; off > 0; off >>= 1) dv += __shfl_xor_sync(0xffffffffu, dv, off);
  if ((threadIdx.x & 31) == 0 && dv) atomicAdd(sb.dda_visits, dv);
}

__global__ void __launch_bounds__(128) k_fast_walk(const int4* __restrict__ rays, ScanTable t, MapView m,
                                                   ChannelView c, TopoView tv,
                                                   const unsigned long long* __restrict__ active,
                                                   PieceBuf sb)
{
  const int lane = static_cast<int>(threadIdx.x & 31);
  if (__shfl_sync(0xffffffffu, lane == 0 ? ld_relaxed_u32(&m.st->error) : 0u, 0) != 0u) return;
  c.cur_epoch      = *c.epoch;
  const unsigned long long pieces = *sb.count;
  if (pieces > sb.cap) return;  // (the host repeats the spans with more room)
  const uint32_t n = static_cast<uint32_t>(pieces);
  unsigned long long marks = 0ull;
  ActiveCache act{&m, active, tv.map, 0x7fffffff, 0, 0, -1, -1, -1, 0ull};
  act.bits = tv.leafbits;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
  {
    const FastPiece p = sb.rec[i];
    const int4 r      = rays[p.ray];
    const ScanGeom& g = scan_geom(t, scan_of_ray(t, static_cast<uint32_t>(p.ray)));
    double eye[3], dir[3];
    fast_ray(r, g, eye, dir);
    hdda::fast_walk_window(eye, dir, p.t0, p.lo, p.hi, [&](const int v[3]) {
      if (!act(v)) return;
      // act holds the voxel's leaf: mark it visited in the update grid.
      const int b    = act.b;
      const int cell = ((act.lx & 7) << 6) | ((act.ly & 7) << 3) | (act.lz & 7);
      touch_block(c, b);
      unsigned long long* bt = c.btouched + static_cast<size_t>(b) * 8 + (cell >> 6);
      if (!((*bt >> (cell & 63)) & 1ull)) atomicOr(bt, 1ull << (cell & 63));
      const int off = ((v[2] & 7) << 6) | ((v[1] & 7) << 3) | (v[0] & 7);
      atomicOr(c.upd + static_cast<size_t>(act.slot) * 16 + (off >> 6), 1ull << (off & 63));
      ++marks;
    });
  }
  for (int off = 16; off > 0; off >>= 1) marks += __shfl_xor_sync(0xffffffffu, marks, off);
  if ((threadIdx.x & 31) == 0 && marks) atomicAdd(&m.st->visits, marks);
}

// Span records by length class, longest first (a counting sort, so that the
// spans a warp walks together take about as many steps each).
__global__ void __launch_bounds__(256) k_span_hist(const SpanRec* __restrict__ rec, const uint32_t* __restrict__ count,
                                                   uint32_t* __restrict__ hist)
{
  const uint32_t n = *count;
  __shared__ uint32_t h[kSpanClasses];
  if (threadIdx.x < kSpanClasses) h[threadIdx.x] = 0u;
  __syncthreads();
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    atomicAdd(h + rec[i].cls, 1u);
  __syncthreads();
  if (threadIdx.x < kSpanClasses && h[threadIdx.x]) atomicAdd(hist + threadIdx.x, h[threadIdx.x]);
}

// One warp: hist[c] becomes the first position of class c, classes in
// descending order.
__global__ void k_span_offsets(uint32_t* hist)
{
  const int lane   = static_cast<int>(threadIdx.x);
  const int c      = kSpanClasses - 1 - lane;  // lane 0: the longest class
  const uint32_t v = hist[c];
  uint32_t incl    = v;
  for (int off = 1; off < 32; off <<= 1)
  {
    const uint32_t o = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += o;
  }
  hist[c] = incl - v;
}

__global__ void __launch_bounds__(256) k_span_scatter(const SpanRec* __restrict__ rec,
                                                      const uint32_t* __restrict__ count,
                                                      uint32_t* __restrict__ cursor, uint32_t* __restrict__ out)
{
  const uint32_t n = *count;
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool in    = i < n;
  const int cls    = in ? rec[i].cls : -1;
  // one atomic per class present in the warp, ranks within it by lane order
  const unsigned peers = __match_any_sync(0xffffffffu, cls);
  const int leader     = __ffs(peers) - 1;
  uint32_t base        = 0;
  if (in && static_cast<int>(threadIdx.x & 31) == leader) base = atomicAdd(cursor + cls, static_cast<uint32_t>(__popc(peers)));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (in) out[base + static_cast<uint32_t>(__popc(peers & lanemask_lt()))] = i;
}

// The fast marking's visits replace the castRayIntoGrid visits the prep
// counted (one thread).
__global__ void k_fast_visits(DevStatus* st, PieceBuf sb)
{
  if (*sb.count <= sb.cap) st->visits -= *sb.dda_visits;
}

// raytrace (VDBMapping.hpp:675-721) in two phases, as fast mode walks its
// spans: k_trace_spans finds every query's first span (hdda::trace_span) and
// answers the queries without one; the spans are sorted by length (longest
// first, k_span_hist / k_span_scatter), and k_trace_walk walks one span per
// thread to its first active voxel, in the windows that can hold one
// (hdda::trace_walk_runs): 0.53 ms for a million spans of 420 voxels, where
// every voxel of them took 2.0. (In clutter they save little and the windows cost
// more: 200,000 queries among points scattered through 20% of the leaves take 1.82 ms
// in both walks, 1.22 without windows; which it is only the device could tell.) The
// coarse walk needs
// many registers and the voxel walk few, so apart each runs at its own
// occupancy, and the walks of a warp take about as many steps each. q holds
// the origins [n][3], then the directions [n][3], then the lengths [n]; ok[n]
// and end[n][3] receive success and end point. A query outside the +-2^30
// index box sets kErrCoordRange.
__device__ __forceinline__ void trace_query(const double* __restrict__ q, uint32_t n, uint32_t i, double o[3],
                                            double d[3], double& len)
{
  const double* dq = q + 3 * static_cast<size_t>(n);
  for (int a = 0; a < 3; ++a)
  {
    o[a] = q[3 * static_cast<size_t>(i) + a];
    d[a] = dq[3 * static_cast<size_t>(i) + a];
  }
  len = q[6 * static_cast<size_t>(n) + i];
}

__device__ __forceinline__ void trace_answer(unsigned char* ok, double* end, uint32_t i, bool success,
                                             const double e[3])
{
  ok[i] = success ? 1 : 0;
  for (int a = 0; a < 3; ++a) end[3 * static_cast<size_t>(i) + a] = e[a];
}

// The queries' order for the span phase: by a coarse origin region and the
// direction cell of ray_bucket's cube map (face, 13 x 13), so that the lanes
// of a warp walk neighbouring rays through the same nodes, and take about as
// many steps (the answers do not depend on the order). A counting sort over a few
// blocks, each with a run of the queries and its own histogram in shared memory:
// the blocks' counts of a bin become its blocks' first positions, so no count is
// shared between blocks (one histogram in global memory took 0.16 ms for a
// million queries, and as long again for the scatter; the four kernels here 0.06).
constexpr int kTraceRegions = 8;
constexpr int kTraceBins    = kTraceRegions * kDirCells;

__device__ __forceinline__ int trace_bin(const double* __restrict__ q, uint32_t n, uint32_t i, double inv_res)
{
  const double* dq = q + 3 * static_cast<size_t>(n);
  const float dx = static_cast<float>(dq[3 * static_cast<size_t>(i)]);
  const float dy = static_cast<float>(dq[3 * static_cast<size_t>(i) + 1]);
  const float dz = static_cast<float>(dq[3 * static_cast<size_t>(i) + 2]);
  const float ax = fabsf(dx), ay = fabsf(dy), az = fabsf(dz);
  int face;
  float u, v, mx;
  if (ax >= ay && ax >= az)
  {
    face = dx >= 0.f ? 0 : 1;
    u    = dy;
    v    = dz;
    mx   = ax;
  }
  else if (ay >= az)
  {
    face = dy >= 0.f ? 2 : 3;
    u    = dx;
    v    = dz;
    mx   = ay;
  }
  else
  {
    face = dz >= 0.f ? 4 : 5;
    u    = dx;
    v    = dy;
    mx   = az;
  }
  int cell = 0;
  if (mx > 0.f)  // (a zero or NaN direction takes cell 0)
  {
    const int iu = min(12, max(0, static_cast<int>((u / mx + 1.f) * 6.5f)));
    const int iv = min(12, max(0, static_cast<int>((v / mx + 1.f) * 6.5f)));
    cell         = face * 169 + iv * 13 + iu;
  }
  // origin region: 256-voxel cells, hashed (single precision: an ordering key only)
  int c[3];
  const float inv = static_cast<float>(inv_res) * (1.f / 256.f);
  for (int a = 0; a < 3; ++a)
  {
    const float x = static_cast<float>(q[3 * static_cast<size_t>(i) + a]) * inv;
    c[a]          = (x > -1e9f && x < 1e9f) ? __float2int_rd(x) : 0;
  }
  const unsigned long long h = mix64(static_cast<unsigned long long>(static_cast<unsigned>(c[0])) * 73856093ull ^
                                     static_cast<unsigned long long>(static_cast<unsigned>(c[1])) * 19349663ull ^
                                     static_cast<unsigned long long>(static_cast<unsigned>(c[2])) * 83492791ull);
  return static_cast<int>(h % kTraceRegions) * kDirCells + cell;
}

constexpr int kTraceSortThreads = 1024;

// Queries [b * per, (b + 1) * per) of block b: their bins, and its counts[b][].
__global__ void __launch_bounds__(kTraceSortThreads) k_trace_bin(const double* __restrict__ q, uint32_t n, uint32_t per,
                                                                 double inv_res, unsigned short* __restrict__ bin,
                                                                 uint32_t* __restrict__ counts)
{
  __shared__ uint32_t h[kTraceBins];
  for (int k = static_cast<int>(threadIdx.x); k < kTraceBins; k += kTraceSortThreads) h[k] = 0u;
  __syncthreads();
  const uint32_t from = blockIdx.x * per, to = min(n, from + per);
  for (uint32_t i = from + threadIdx.x; i < to; i += kTraceSortThreads)
  {
    const int b = trace_bin(q, n, i, inv_res);
    bin[i]      = static_cast<unsigned short>(b);
    atomicAdd(h + b, 1u);
  }
  __syncthreads();
  uint32_t* mine = counts + static_cast<size_t>(blockIdx.x) * kTraceBins;
  for (int k = static_cast<int>(threadIdx.x); k < kTraceBins; k += kTraceSortThreads) mine[k] = h[k];
}

// One thread per bin: its counts become the sums of the blocks before, its total
// goes to `total`.
__global__ void __launch_bounds__(64) k_trace_sums(uint32_t* __restrict__ counts, uint32_t blocks,
                                                    uint32_t* __restrict__ total)
{
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= static_cast<uint32_t>(kTraceBins)) return;
  uint32_t sum = 0;
  for (uint32_t k = 0; k < blocks; k += 32u)
  {
    uint32_t v[32];
#pragma unroll
    for (uint32_t j = 0; j < 32u; ++j) v[j] = k + j < blocks ? counts[static_cast<size_t>(k + j) * kTraceBins + b] : 0u;
#pragma unroll
    for (uint32_t j = 0; j < 32u; ++j)
    {
      if (k + j < blocks) counts[static_cast<size_t>(k + j) * kTraceBins + b] = sum;
      sum += v[j];
    }
  }
  total[b] = sum;
}

// One block of 1024 threads: total[] (kTraceBins) becomes the first position of each bin.
__global__ void __launch_bounds__(1024) k_trace_offsets(uint32_t* __restrict__ total)
{
  constexpr uint32_t kPer = (kTraceBins + 1023) / 1024;
  const uint32_t i0       = threadIdx.x * kPer;
  uint32_t v[kPer], local = 0;
#pragma unroll
  for (uint32_t k = 0; k < kPer; ++k)
  {
    v[k] = i0 + k < static_cast<uint32_t>(kTraceBins) ? total[i0 + k] : 0u;
    local += v[k];
  }
  uint32_t sum = 0;
  uint32_t at  = block_scan_exclusive(local, &sum);
#pragma unroll
  for (uint32_t k = 0; k < kPer; ++k)
  {
    if (i0 + k < static_cast<uint32_t>(kTraceBins)) total[i0 + k] = at;
    at += v[k];
  }
}

__global__ void __launch_bounds__(kTraceSortThreads) k_trace_scatter(const unsigned short* __restrict__ bin, uint32_t n,
                                                                     uint32_t per, const uint32_t* __restrict__ counts,
                                                                     const uint32_t* __restrict__ first,
                                                                     uint32_t* __restrict__ order)
{
  __shared__ uint32_t at[kTraceBins];
  const uint32_t* mine = counts + static_cast<size_t>(blockIdx.x) * kTraceBins;
  for (int k = static_cast<int>(threadIdx.x); k < kTraceBins; k += kTraceSortThreads) at[k] = first[k] + mine[k];
  __syncthreads();
  const uint32_t from = blockIdx.x * per, to = min(n, from + per);
  for (uint32_t i = from + threadIdx.x; i < to; i += kTraceSortThreads) order[atomicAdd(at + bin[i], 1u)] = i;
}

// (20 warps an SM, which costs some spills: 16 took 3% longer, 12 without spills as much)
__global__ void __launch_bounds__(kSpanThreads, 20) k_trace_spans(double* q, uint32_t n, double res,
                                                     double inv_res, MapView m, TopoView tv,
                                                     const uint32_t* __restrict__ order,
                                                     unsigned char* __restrict__ ok, double* __restrict__ end,
                                                     TraceBuf sb, uint32_t lanes)
{
  const uint32_t j = lane_item(lanes, n);
  if (j >= n) return;
  const uint32_t i = order ? order[j] : j;
  if (tv.count[1] != 0u)
  {
    atomicOr(&m.st->error, kErrTopoFull);
    return;
  }
  double o[3], d[3], len;
  trace_query(q, n, i, o, d, len);
  const double zero[3] = {0.0, 0.0, 0.0};
  double oi[3], di[3];
  if (!hdda::trace_ray(o, d, len, inv_res, oi, di))
  {
    atomicOr(&m.st->error, kErrCoordRange);
    trace_answer(ok, end, i, false, zero);
    return;
  }
  DevTopo topo{tv, m, 0x7fffffff, 0, 0, -1};
  hdda::Span sp{-1.0, -1.0};
  bool found     = false;
  uint32_t steps = 0;
  hdda::Runs runs;
  hdda::RunTrack<hdda::Runs> track(runs);
  if (hdda::trace_span(oi, di, topo_box(tv), topo, sp, found, steps, track) == hdda::kTraceBound)
  {
    atomicOr(&m.st->error, kErrStepBound);
    trace_answer(ok, end, i, false, zero);
    return;
  }
  if (!found)
  {
    double e[3];
    hdda::trace_miss(oi, di, res, e);
    trace_answer(ok, end, i, false, e);
    return;
  }
  SpanRec r;
  r.t0        = sp.t0;
  r.t1        = sp.t1;
  r.ray       = static_cast<int>(i);
  r.n         = runs.n;
  float total = 0.0f;
  for (int k = 0; k < hdda::Runs::kMax; ++k)
  {
    const bool in = k < runs.n;
    r.lo[k]       = in ? runs.lo[k] : 0.0f;
    r.hi[k]       = in ? runs.hi[k] : 0.0f;
    total += r.hi[k] - r.lo[k];
  }
  const float l1 = fabsf(static_cast<float>(di[0])) + fabsf(static_cast<float>(di[1])) + fabsf(static_cast<float>(di[2]));
  r.cls          = 31 - __clz(static_cast<int>(fminf(total * l1 + 1.0f, 1.0e9f)));  // (for ordering only)
  r.pad          = 0;
  // The walk takes the ray from here: its direction in the query's place, its
  // inverse where the end point will be. (A root and four divisions it would make
  // again: a million queries' walks 571 to 528 us, the spans 20 more.)
  double* dq = q + 3 * static_cast<size_t>(n);
  for (int a = 0; a < 3; ++a)
  {
    dq[3 * static_cast<size_t>(i) + a]  = di[a];
    end[3 * static_cast<size_t>(i) + a] = hdda::dvd(1.0, di[a]);
  }
  const uint32_t k = take_slot(sb.count);
  if (k < sb.cap) sb.rec[k] = r;
}

__global__ void __launch_bounds__(128) k_trace_walk(const double* __restrict__ q, uint32_t n, double res,
                                                    double inv_res, MapView m, TopoView tv,
                                                    const unsigned long long* __restrict__ active,
                                                    unsigned char* __restrict__ ok, double* __restrict__ end,
                                                    const SpanRec* __restrict__ rec,
                                                    const uint32_t* __restrict__ by_class,
                                                    const uint32_t* __restrict__ count, uint32_t lanes)
{
  const uint32_t n_spans = *count;
  const uint32_t j       = lane_item(lanes, n_spans);
  if (j >= n_spans) return;
  const SpanRec& r = rec[by_class ? by_class[j] : j];
  const uint32_t i = static_cast<uint32_t>(r.ray);
  // (k_trace_spans left the direction and its inverse)
  const double* dq = q + 3 * static_cast<size_t>(n);
  hdda::Ray ray;
  for (int a = 0; a < 3; ++a)
  {
    ray.eye[a] = hdda::mul(q[3 * static_cast<size_t>(i) + a], inv_res);
    ray.dir[a] = dq[3 * static_cast<size_t>(i) + a];
    ray.inv[a] = end[3 * static_cast<size_t>(i) + a];
  }
  ray.t0 = r.t0;
  ray.t1 = r.t1;
  ActiveCache act{&m, active, tv.map, 0x7fffffff, 0, 0, -1, -1, -1, 0ull};
  act.bits = tv.leafbits;
  double e[3];
  hdda::trace_walk_runs(ray, hdda::Span{r.t0, r.t1}, r.lo, r.hi, r.n, res, act, e);
  trace_answer(ok, end, i, true, e);
}

// ---------------------------------------------------------------------------
// Morphology of section leaves (VDBMapping.hpp:1094-1147): one dilation or
// erosion step with the 26-neighbourhood over a set of leaves (origins and
// OpenVDB-order masks), per vdbg::morph. A set carries an open-addressing
// hash from leaf key to index, so the 27 neighbours of a leaf are found by
// lookup. A dilation step's leaves are the input leaves' neighbours that
// receive bits (morph::feeds), an erosion step's are the input leaves; the
// steps' empty leaves are dropped by a compaction.
// ---------------------------------------------------------------------------
constexpr uint32_t kMorphHashFull = 1u;  // MorphSet::flags: a hash insert ran out of probes
constexpr uint32_t kMorphSetFull  = 2u;  //                  more leaves than the set holds

struct MorphSet
{
  int4* origin;               // [cap] leaf origins (.w unused)
  unsigned long long* mask;   // [cap][8]
  uint32_t* count;            // device scalar
  uint32_t cap;
  unsigned long long* keys;   // [hmask + 1] leaf keys, kEmptyKey when free
  int* vals;                  // [hmask + 1] leaf index of the key
  uint32_t hmask;
  uint32_t* flags;            // device scalar, kMorph* bits
};

__device__ __forceinline__ unsigned long long morph_key(int x, int y, int z)
{
  return pack_leaf_key(0, x >> 3, y >> 3, z >> 3);
}

__device__ __forceinline__ int morph_find(const MorphSet& s, unsigned long long key)
{
  uint32_t h = static_cast<uint32_t>(mix64(key)) & s.hmask;
  for (uint32_t probe = 0; probe < kMaxProbes; ++probe)
  {
    const unsigned long long k = s.keys[h];
    if (k == key) return s.vals[h];
    if (k == kEmptyKey) return -1;
    h = (h + 1) & s.hmask;
  }
  return -1;
}

// Inserts `key`; the thread that adds it takes the next index of the set,
// writes the origin and publishes the index (read by later kernels only).
// Returns false when the hash or the set is full (flag set).
__device__ __forceinline__ bool morph_insert(const MorphSet& s, unsigned long long key, int4 o)
{
  uint32_t h = static_cast<uint32_t>(mix64(key)) & s.hmask;
  for (uint32_t probe = 0; probe < kMaxProbes; ++probe)
  {
    const unsigned long long k = s.keys[h];
    if (k == key) return true;
    if (k == kEmptyKey)
    {
      const unsigned long long prev = atomicCAS(s.keys + h, kEmptyKey, key);
      if (prev == kEmptyKey)
      {
        const uint32_t i = atomicAdd(s.count, 1u);
        if (i >= s.cap)
        {
          atomicOr(s.flags, kMorphSetFull);
          s.vals[h] = -1;
          return false;
        }
        s.origin[i] = o;
        s.vals[h]   = static_cast<int>(i);
        return true;
      }
      if (prev == key) return true;
    }
    h = (h + 1) & s.hmask;
  }
  atomicOr(s.flags, kMorphHashFull);
  return false;
}

// The leaves of `in` (n of them, with their masks) into the empty set `out`
// (hash and origins; the masks are copied by index).
__global__ void k_morph_load(const int4* __restrict__ origin, const unsigned long long* __restrict__ mask, uint32_t n,
                             MorphSet out)
{
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int4 o = origin[i];
  if (!morph_insert(out, morph_key(o.x, o.y, o.z), o)) return;
  const int j = morph_find(out, morph_key(o.x, o.y, o.z));
  if (j < 0) return;
  for (int w = 0; w < 8; ++w) out.mask[static_cast<size_t>(j) * 8 + w] = mask[static_cast<size_t>(i) * 8 + w];
}

// The same over a dense grid of leaf cells, for a set whose cells (with room for
// what its dilations reach) are few: no hash, no list between the steps, and the
// cells' order is that of the origins. Bound by its launches (a word reads 27
// words that its neighbours read too, from L1): reading a section of about 5400
// leaves, closing it by two voxels, applying it and reading the result take
// 0.44 ms together, where the hashed sets, with their allocations and counts
// between the steps, took 2.2. A scattered set, of more than 2^18 cells, keeps
// those: the grid's time and memory are those of its cells.
struct MorphGrid
{
  int3 first, dims;            // leaf coordinate of the first cell; cells x, y, z (z fastest)
  uint32_t cells;
  unsigned char* present;      // [cells] a leaf of the kept topology
};

__device__ __forceinline__ void morph_cell(const MorphGrid& g, uint32_t i, int& x, int& y, int& z)
{
  const uint32_t xy = i / static_cast<uint32_t>(g.dims.z);
  z                 = static_cast<int>(i - xy * static_cast<uint32_t>(g.dims.z));
  x                 = static_cast<int>(xy / static_cast<uint32_t>(g.dims.y));
  y                 = static_cast<int>(xy - static_cast<uint32_t>(x) * static_cast<uint32_t>(g.dims.y));
}

// One thread per (leaf, word) of the input; a repeated origin's masks merge.
__global__ void __launch_bounds__(256) k_morph_place(MorphGrid g, const int* __restrict__ origin,
                                                     const unsigned long long* __restrict__ mask, uint32_t n,
                                                     unsigned long long* __restrict__ out)
{
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t i = t >> 3;
  if (i >= n) return;
  const int x = (origin[3 * static_cast<size_t>(i)] >> 3) - g.first.x,
            y = (origin[3 * static_cast<size_t>(i) + 1] >> 3) - g.first.y,
            z = (origin[3 * static_cast<size_t>(i) + 2] >> 3) - g.first.z;
  const uint32_t c = (static_cast<uint32_t>(x) * static_cast<uint32_t>(g.dims.y) + static_cast<uint32_t>(y)) *
                       static_cast<uint32_t>(g.dims.z) + static_cast<uint32_t>(z);
  const unsigned long long m = mask[t];
  if (m) atomicOr(out + static_cast<size_t>(c) * 8 + (t & 7u), m);
  if ((t & 7u) == 0u) g.present[c] = 1;
}

// The 27 neighbour cells of a cell (none outside the grid).
struct MorphCells
{
  const unsigned long long* in;
  const MorphGrid* g;
  int x, y, z;
  __device__ __forceinline__ const uint64_t* operator()(int d) const
  {
    const int nx = x + d / 9 - 1, ny = y + (d / 3) % 3 - 1, nz = z + d % 3 - 1;
    if (nx < 0 || ny < 0 || nz < 0 || nx >= g->dims.x || ny >= g->dims.y || nz >= g->dims.z) return nullptr;
    return reinterpret_cast<const uint64_t*>(
      in + (static_cast<size_t>(nx * g->dims.y + ny) * static_cast<size_t>(g->dims.z) + static_cast<size_t>(nz)) * 8);
  }
};

// One step, one thread per (cell, word). A leaf that a dilation reaches (its word
// is not empty) joins the kept topology.
__global__ void __launch_bounds__(256) k_morph_step(MorphGrid g, const unsigned long long* __restrict__ in,
                                                    unsigned long long* __restrict__ out, int dilate)
{
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t i = t >> 3;
  if (i >= g.cells) return;
  const int a = static_cast<int>(t & 7u);
  unsigned long long w = 0ull;
  if (dilate || in[t])  // (an erosion leaves nothing where nothing was)
  {
    MorphCells nb{in, &g, 0, 0, 0};
    morph_cell(g, i, nb.x, nb.y, nb.z);
    w = dilate ? morph::dilate_word(nb, a) : morph::erode_word(nb, a);
  }
  out[t] = w;
  if (dilate && w) g.present[i] = 1;
}

// Which cells are leaves of the result.
__global__ void __launch_bounds__(256) k_morph_keep(MorphGrid g, const unsigned long long* __restrict__ in, int keep,
                                                    uint32_t* __restrict__ out)
{
  const uint32_t t     = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t i     = t >> 3;
  const bool any       = i < g.cells && in[t] != 0ull;
  const unsigned votes = __ballot_sync(0xffffffffu, any);
  if (i >= g.cells || (t & 7u) != 0u) return;
  out[i] = ((votes >> (threadIdx.x & 24u)) & 0xffu) != 0u || (keep && g.present[i]) ? 1u : 0u;
}

__global__ void __launch_bounds__(256) k_morph_write(MorphGrid g, const unsigned long long* __restrict__ in,
                                                     const uint32_t* __restrict__ keep,
                                                     const uint32_t* __restrict__ pos, int* __restrict__ out_o,
                                                     unsigned long long* __restrict__ out_m)
{
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t i = t >> 3, a = t & 7u;
  if (i >= g.cells || !keep[i]) return;
  const size_t at    = pos[i];
  out_m[at * 8 + a] = in[t];
  if (a < 3u)
  {
    int x, y, z;
    morph_cell(g, i, x, y, z);
    out_o[at * 3 + a] = 8 * (a == 0u ? g.first.x + x : a == 1u ? g.first.y + y : g.first.z + z);
  }
}

// Dilation: one thread per (leaf of `in`, direction); the neighbours that
// receive bits become the leaves of `out` (deduplicated by its hash).
// Erosion (dilate == 0): the leaves of `in` themselves. `keep`: every leaf of
// `in` is also a leaf of `out`, empty or not (the topology is never pruned).
__global__ void k_morph_candidates(MorphSet in, uint32_t n_in, MorphSet out, int dilate, int keep)
{
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n_in * 27u) return;
  const uint32_t i = t / 27u;
  const int d      = static_cast<int>(t % 27u);
  const int dx = d / 9 - 1, dy = (d / 3) % 3 - 1, dz = d % 3 - 1;
  if (!dilate && d != 13) return;
  if (dilate && !(keep && d == 13) &&
      !morph::feeds(reinterpret_cast<const uint64_t*>(in.mask + static_cast<size_t>(i) * 8), dx, dy, dz))
    return;
  const int4 o = in.origin[i];
  const int4 c = make_int4(o.x + 8 * dx, o.y + 8 * dy, o.z + 8 * dz, 0);
  morph_insert(out, morph_key(c.x, c.y, c.z), c);
}

// The 27 neighbour leaves of one leaf of a step's output, looked up in the
// step's input set.
struct MorphNeighbours
{
  const MorphSet* in;
  int cx, cy, cz;
  __device__ __forceinline__ const uint64_t* operator()(int d) const
  {
    const int j = morph_find(*in, morph_key(cx + 8 * (d / 9 - 1), cy + 8 * ((d / 3) % 3 - 1), cz + 8 * (d % 3 - 1)));
    return j < 0 ? nullptr : reinterpret_cast<const uint64_t*>(in->mask + static_cast<size_t>(j) * 8);
  }
};

// One thread per (leaf of `out`, word): the word after the step.
__global__ void k_morph_words(MorphSet in, MorphSet out, uint32_t n_out, int dilate)
{
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n_out * 8u) return;
  const uint32_t j = t >> 3;
  const int a      = static_cast<int>(t & 7u);
  const int4 o     = out.origin[j];
  const MorphNeighbours nb{&in, o.x, o.y, o.z};
  out.mask[static_cast<size_t>(j) * 8 + a] = dilate ? morph::dilate_word(nb, a) : morph::erode_word(nb, a);
}

// The leaves of `in` with an active voxel (`keep`: all of them), into the
// empty set `out`.
__global__ void k_morph_compact(MorphSet in, uint32_t n_in, MorphSet out, int keep)
{
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_in) return;
  unsigned long long any = keep ? 1ull : 0ull;
  for (int w = 0; w < 8; ++w) any |= in.mask[static_cast<size_t>(i) * 8 + w];
  if (!any) return;
  const int4 o = in.origin[i];
  if (!morph_insert(out, morph_key(o.x, o.y, o.z), o)) return;
  const int j = morph_find(out, morph_key(o.x, o.y, o.z));
  if (j < 0) return;
  for (int w = 0; w < 8; ++w) out.mask[static_cast<size_t>(j) * 8 + w] = in.mask[static_cast<size_t>(i) * 8 + w];
}

// ---------------------------------------------------------------------------
// Artificial areas (VDBMapping.hpp:1152-1236). Their voxels are re-activated
// after every update of the map by k_section_set_states (VDBMapping.hpp:
// 785-789 does setActiveState(v, true)); walls are rasterised here and the
// states restored when the areas are replaced.
// ---------------------------------------------------------------------------

// addArtificialWall (VDBMapping.hpp:1210-1236): layer i is castRayIntoGrid
// (VDBMapping.hpp:550-566) from voxel a[i] to b[i]: the voxel DDA of the ray
// a + 0.5 -> b + 0.5 over t in [0, 1], nothing when a == b. Its 1 + L1
// voxels go to out[first[i], first[i + 1]); a count that disagrees sets *bad.
__global__ void k_wall_voxels(const int4* __restrict__ a, const int4* __restrict__ b,
                              const uint32_t* __restrict__ first, uint32_t n, int4* __restrict__ out,
                              uint32_t* bad)
{
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t base = first[i], cnt = first[i + 1] - base;
  if (cnt == 0u) return;
  const int4 s = a[i], e = b[i];
  const double eye[3] = {hdda::add(static_cast<double>(s.x), 0.5), hdda::add(static_cast<double>(s.y), 0.5),
                         hdda::add(static_cast<double>(s.z), 0.5)};
  const double dir[3] = {hdda::sub(static_cast<double>(e.x), static_cast<double>(s.x)),
                         hdda::sub(static_cast<double>(e.y), static_cast<double>(s.y)),
                         hdda::sub(static_cast<double>(e.z), static_cast<double>(s.z))};
  const hdda::Ray r = hdda::make_ray(eye, dir, 0.0, 1.0);
  hdda::Dda d;
  hdda::dda_init(d, r, 0.0, 1.0, 0);
  uint32_t k = 0;
  do
  {
    if (k >= cnt)
    {
      atomicOr(bad, 1u);
      return;
    }
    out[base + k] = make_int4(d.voxel[0], d.voxel[1], d.voxel[2], 0);
    ++k;
  } while (hdda::dda_step(d));
  if (k != cnt) atomicOr(bad, 1u);
}

// restoreMapIntegrity (VDBMapping.hpp:1153-1166) on the integrated map
// leaves holding artificial voxels: each such voxel's state becomes
// value > thres_max (setNodeState, OccupancyVDBMapping.hpp:130-134). One
// thread per (artificial leaf, plane word); the leaves are distinct, so no
// word has two writers.
__global__ void k_artificial_restore(MapView m, const int4* __restrict__ art_o,
                                     const unsigned long long* __restrict__ art_m, uint32_t n,
                                     const uint32_t* __restrict__ flags, const float* __restrict__ values,
                                     unsigned long long* __restrict__ active, float thres_max)
{
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * 8u) return;
  const uint32_t i              = t >> 3;
  const int w                   = static_cast<int>(t & 7u);
  const unsigned long long bits = art_m[static_cast<size_t>(i) * 8 + w];
  if (!bits) return;
  const int4 o   = art_o[i];
  const int slot = find_leaf(m, o.w, o.x >> 3, o.y >> 3, o.z >> 3);
  if (slot < 0 || flags[slot] == 0u) return;
  unsigned long long on = 0ull;
  for (unsigned long long z = bits; z; z &= z - 1ull)
  {
    const int k = __ffsll(static_cast<long long>(z)) - 1;
    if (values[static_cast<size_t>(slot) * 512 + w * 64 + plane_float(k)] > thres_max) on |= 1ull << k;
  }
  unsigned long long* a = active + static_cast<size_t>(slot) * 8 + w;
  *a                    = (*a & ~bits) | on;
}

// ---------------------------------------------------------------------------
// Digests for verification at sizes where exporting a map is impractical.
// Both are restated in the oracle (oracle_capi.cpp), which computes the same
// numbers from its own traversal and map.
//   voxel key  k(x,y,z) = u32(x)*0x9E3779B97F4A7C15 ^ u32(y)*0xC2B2AE3D27D4EB4F
//                         ^ u32(z)*0x165667B19E3779F9
//   ray digest: h = 0x243F6A8885A308D3, then h = mix64(h ^ k(v)) for every
//               voxel castRayIntoGrid visits, in order; finally
//               h = mix64(h ^ k(end) ^ 0x5851F42D4C957F2D)
//               word 0: visits | clipped << 40 | valid << 41; word 1: h
//   map digest: over the map's leaves, sums (mod 2^64) of mix64(k(origin))
//               and, over its voxels whose value bits are non-zero or that
//               are active, of mix64(k(x,y,z) ^ (bits << 1 | active) *
//               0xD6E8FEB86659FD93); plus the counts of both.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long digest_key(int x, int y, int z)
{
  return static_cast<unsigned long long>(static_cast<uint32_t>(x)) * 0x9E3779B97F4A7C15ull ^
         static_cast<unsigned long long>(static_cast<uint32_t>(y)) * 0xC2B2AE3D27D4EB4Full ^
         static_cast<unsigned long long>(static_cast<uint32_t>(z)) * 0x165667B19E3779F9ull;
}

// One thread per ray record (k_prep's output, point order): the walk of
// k_march (march_begin, march::step), chunk after chunk, hashed as above.
__global__ void __launch_bounds__(256) k_ray_digest(const int4* __restrict__ rays, int64_t n, ScanTable t,
                                                    AxisTable at, unsigned long long* __restrict__ out, DevStatus* st)
{
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int4 rec          = rays[i];
  const uint32_t meta     = static_cast<uint32_t>(rec.w);
  const bool valid        = (meta & kMetaValid) != 0u;
  const bool clipped      = (meta & kMetaClipped) != 0u;
  unsigned long long h    = 0x243F6A8885A308D3ull;
  unsigned long long cnt  = 0;
  const MarchRay r = march_ray(valid ? rec : make_int4(0, 0, 0, 0), scan_geom(t, scan_of_point(t, static_cast<uint32_t>(i))),
                               t.clog);
  for (uint32_t k = 0; valid && r.p >= 0 && (k >> r.p) == 0u; ++k)
  {
    march::Walk w;
    w.one = 1u;
    march::Cuts cuts;
    int bx, by, bz;
    const uint32_t end   = march_begin(at, r, k, w, cuts, bx, by, bz);
    const uint32_t first = w.pos;
    auto visit = [&]() {
      h = mix64(h ^ digest_key(bx * 8 + static_cast<int>(march::pos_field(w.pos, 0)),
                               by * 8 + static_cast<int>(march::pos_field(w.pos, 1)),
                               bz * 8 + static_cast<int>(march::pos_field(w.pos, 2))));
      ++cnt;
    };
    if (k == 0u) visit();
    uint32_t steps = 0;
    for (;;)
    {
      if (march::has_step(w))
      {
        if (k == 0u)
          march::step<true>(w);
        else
          march::step<false>(w);
        visit();
        if (++steps <= march::kMaxSteps) continue;
        atomicOr(&st->error, kErrStepBound);
        break;
      }
      if (k == 0u || w.end == end) break;
      march::resume(w, cuts, first, end);
    }
  }
  if (valid) h = mix64(h ^ digest_key(rec.x, rec.y, rec.z) ^ 0x5851F42D4C957F2Dull);
  out[2 * i]     = cnt | (clipped ? 1ull << 40 : 0ull) | (valid ? 1ull << 41 : 0ull);
  out[2 * i + 1] = valid ? h : 0ull;
}

// One warp per leaf slot below `n`: the map digest of map `map` (-1: all),
// added into out[4] = {leaves, voxels, leaf sum, voxel sum}.
__global__ void __launch_bounds__(256) k_map_digest(const int4* __restrict__ origin,
                                                    const uint32_t* __restrict__ flags,
                                                    const float* __restrict__ values,
                                                    const unsigned long long* __restrict__ active, uint32_t n,
                                                    int map, unsigned long long* __restrict__ out)
{
  const uint32_t slot = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane      = static_cast<int>(threadIdx.x & 31);
  if (slot >= n) return;  // (whole warps)
  const int4 o = origin[slot];
  if (flags[slot] == 0u || (map >= 0 && o.w != map)) return;
  unsigned long long cnt = 0, sum = 0;
  for (int k = lane; k < 512; k += 32)
  {
    // device leaf order: offset = z << 6 | y << 3 | x, mask word = z
    const int z = k >> 6, y = (k >> 3) & 7, x = k & 7;
    const uint32_t bits = __float_as_uint(values[static_cast<size_t>(slot) * 512 + leaf_float(k)]);
    const uint32_t on   = static_cast<uint32_t>((active[static_cast<size_t>(slot) * 8 + z] >> (k & 63)) & 1ull);
    if (bits != 0u || on)
    {
      ++cnt;
      sum += mix64(digest_key(o.x + x, o.y + y, o.z + z) ^
                   ((static_cast<unsigned long long>(bits) << 1) | on) * 0xD6E8FEB86659FD93ull);
    }
  }
  for (int off = 16; off > 0; off >>= 1)
  {
    cnt += __shfl_xor_sync(0xffffffffu, cnt, off);
    sum += __shfl_xor_sync(0xffffffffu, sum, off);
  }
  if (lane == 0)
  {
    atomicAdd(out + 0, 1ull);
    atomicAdd(out + 1, cnt);
    atomicAdd(out + 2, mix64(digest_key(o.x, o.y, o.z)));
    atomicAdd(out + 3, sum);
  }
}

// ---------------------------------------------------------------------------
// L2 atomic throughput probe (the atomic half of the roofline): every thread
// issues `iters` 64-bit ORs whose results are unused (RED) to words of an
// L2-resident buffer of mask + 1 words. pattern 0: each warp ORs 32
// consecutive words (one 256-byte request, as the apply's leaf-mask ORs
// are); pattern 1: every lane a pseudo-random word (as the endpoint hits
// are).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_atomic_probe(unsigned long long* __restrict__ buf, uint32_t mask,
                                                      uint32_t iters, int pattern)
{
  const uint32_t tid  = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t x          = tid * 2654435761u + 12345u;
  uint32_t base       = (tid >> 5) * 32u * 97u;
  for (uint32_t i = 0; i < iters; ++i)
  {
    uint32_t idx;
    if (pattern == 0)
    {
      base += 32u * 131u;
      idx = (base + lane) & mask;
    }
    else
    {
      x ^= x << 13;
      x ^= x >> 17;
      x ^= x << 5;
      idx = x & mask;
    }
    atomicOr(buf + idx, 1ull << (i & 63u));
  }
}

} // namespace vdbg
