// Execution of the Radiating (radial scan) and Spreading (flow accumulation)
// skeletons; their kernels are generated in codegen.cpp (gen_radial, gen_spread).
//
// Radiating (runtime/skeleton/RadiatingSkeleton.cpp:32-323): a cell's scan value is
// op(LIT(prev front at d1, prev front at d1-1), in) when `in` is finite; the start
// cell holds the neutral value. The octants are cut into tiles of fronts and cells
// that CTAs claim in strip order (codegen.cpp radial_tiles_source,
// skeleton/scan.cuh radial_tiles): the chain of a strip's fronts runs in one warp's
// registers, everything else of a cell beside it, and a strip waits only for the
// last front of the one above. 4096^2 viewshed: 217 us, against 4161 us for one
// front at a time with a cluster barrier between fronts; 8 B per cell would take 21
// us of HBM: the 2250 fronts' chain (about 65 ns each with the exchange between
// strips) and the issue of two IEEE divisions and square roots per cell bound it.
// A scan whose scratch (an eighth of the raster's bytes, up to four times them for
// rasters one cell wide) cannot be had is swept front by front, which needs none: one CTA per octant,
// a front's cells spread over the CTA's threads, the previous and current fronts in
// shared memory when both fit (radial_front_smem, up to 200 KiB); for rasters at
// least kRadialClusterDim cells across, the octant runs on a cluster of
// kRadialCluster CTAs, each holding one segment of both fronts in its shared
// memory and reading the value left of its segment from its neighbour's
// (distributed shared memory). Fronts too long for either are read back from the
// scan's own output raster (written by this CTA one step earlier; cells on an
// octant boundary are written by both adjacent octants with identical values).
// The group's local nodes before the scan are evaluated per cell to produce
// `in`; those after it are evaluated right after the cell's scan value.
//
// Spreading (runtime/skeleton/SpreadingSkeleton.cpp:288-393): the reference
// relaxes "pending spread" one neighbour per iteration, block by block, until
// stable; the fixed point is, for every cell, the sum of the water of all
// strictly-upstream cells. Here the same fixed point is reached without
// iterating to convergence. 32-bit integer accumulations run over tiles in three
// passes (skeleton/flow.cuh). Other types, and plain launches (the reference's
// granularity), count in-degrees by pulling from the 8 neighbours; then either one
// CTA sweeps frontier by frontier (topological order; rasters up to
// kSpreadKahnCells = 64 K cells) or, for larger rasters, a thread per source walks
// down its flow path pushing (accumulation + water) with atomic adds and continues
// into a cell only when its push was the cell's last pending one, so each cell is
// completed exactly once after all its upstream cells. Integer sums are exact and
// order-independent.
#include "codegen.hpp"
#include "cuda_env.hpp"
#include "executor.hpp"
#include "stream_memory.hpp"

#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <unordered_map>

namespace mapb {

// Walked flow accumulations of at most this many cells run as one CTA's frontier sweep;
// larger ones as the two grid-wide passes (in-degrees, then downstream walks),
// which spread over every SM (measured at 1024²: 1.7 ms against 5.6 ms for one
// CTA). Serving runs one CTA per window instead, many windows side by side.
constexpr size_t kSpreadKahnCells = (size_t)1 << 16;
// Integer flow accumulations of more cells than kSpreadKahnCells and at most this
// many run as pointer jumping over the Euler tour of the D8 forest (a fixed
// number of rounds, independent of the longest flow path; O(N log N) work).
// Whole rasters on an otherwise idle GPU walk faster (measured 0.21 against
// 0.43 ms at 1024^2, 0.61 against 1.82 ms at 2048^2), so the default is 0
// (never); serving windows, which run beside other requests, jump (server.cpp).
// ma_setFlowJumpCells, or MAP_B200_SPREAD_PJ for the default, sets the limit.
size_t spread_pj_cells() {
  static const size_t dflt = [] {
    const char *e = std::getenv("MAP_B200_SPREAD_PJ");
    return e ? (size_t)std::strtoull(e, nullptr, 10) : (size_t)0;
  }();
  const long long v = Runtime::get().flow_jump_cells;
  return v < 0 ? dflt : (size_t)v;
}
// rounds of pointer jumping for N cells: 2^rounds exceeds 2N, the longest tour
int spread_pj_rounds(size_t N) {
  int r = 1;
  while (((size_t)1 << r) <= 2 * N) r++;
  return r;
}
bool spread_pj_type(int dt) { return dt == S32 || dt == U32 || dt == S64 || dt == U64; }
size_t spread_pj_scratch(size_t N, int dt) { return 4 * N * (sizeof(int32_t) + dt_size(dt)); }
bool spread_tile_type(int dt) { return dt == S32 || dt == U32; }
// radial scans of rasters at least this wide or tall use CTA clusters per octant
constexpr int kRadialClusterDim = 2048;
constexpr int kRadialCluster = 8;

size_t radial_front_smem(int W, int H, int dtype) {
  const size_t b = 2 * (size_t)std::max(W, H) * dt_size(dtype);   // previous and current front
  return b <= (size_t)200 * 1024 ? b : 0;                          // larger: fronts re-read from the output
}

// The most scratch that the tiles of one scan may take: MAP_B200_SCAN_SCRATCH bytes,
// read at each scan, or whatever the pool has. A scan whose tiles cannot have theirs
// runs in the form that needs none (radial: front by front) or, thin, less (flow: walks).
static bool tile_scratch(StreamMemory &work, size_t bytes) {
  const char *e = std::getenv("MAP_B200_SCAN_SCRATCH");
  if (e && bytes > std::strtoull(e, nullptr, 10)) return false;
  const cudaError_t r = work.alloc(bytes);
  if (r == cudaErrorMemoryAllocation) return false;
  cuda_check(r, "allocation of a scan's scratch");
  return true;
}

size_t radial_tile_smem(int dtype) {
  // the arguments of a tile's fronts, rows padded by four cells
  return (size_t)kRadialT * (kRadialB + kRadialT + 4) * dt_size(dtype);
}
RadialScratch radial_tile_scratch(int W, int H, int sx, int sy, long long lim, int dtype) {
  constexpr int b = kRadialB, t = kRadialT;
  // the octants' extents along and across their axis: each pair of a side in x and a side in y twice
  const int ex[2] = {sx, W - 1 - sx}, ey[2] = {sy, H - 1 - sy};
  RadialScratch R;
  size_t slots = 0;
  auto octant = [&](int ep, int eq) {
    const int dmax = lim >= 0 && lim < ep ? (int)lim : ep;
    const int strips = (dmax + t - 1) / t;
    slots += (size_t)strips * (eq / b + 1);
    for (int s = 0; s < strips; s++) R.tiles += std::min(std::min(s * t + t, dmax), eq) / b + 1;
  };
  for (int i = 0; i < 2; i++)
    for (int j = 0; j < 2; j++) {
      octant(ex[i], ey[j]);
      octant(ey[j], ex[i]);
    }
  R.bytes = 64 + slots * b * 2 * dt_size(dtype);
  return R;
}

void run_scan_group(const Group &g, const KernelPlan &P, std::unordered_map<Node *, DevRaster> &bufs,
                    const std::function<DevRaster &(Node *)> &get, const std::function<DevRaster(Node *)> &alloc_out) {
  CudaEnv &env = CudaEnv::get();
  cudaStream_t st = (cudaStream_t)env.stream();
  Node *scan = P.core;
  StreamMemory work(st);
  RadialScratch R;
  long long lim = -1;
  bool tiled = false;
  if (scan->kind == K_RADIALSCAN) {
    if (scan->radius > 0) lim = (long long)scan->radius;
    R = radial_tile_scratch(g.W, g.H, scan->coord.arr[0], scan->coord.arr[1], lim, scan->meta.dtype);
    tiled = tile_scratch(work, R.bytes);
  }
  for (Node *o : P.out_rasters) {
    if (bufs.count(o)) continue;
    if (o == scan && g.scan_private && tiled) {
      DevRaster none;   // the tiled form keeps no raster that only the group itself reads
      none.dtype = o->meta.dtype;
      none.W = g.W;
      none.H = g.H;
      bufs[o] = none;
    } else {
      bufs[o] = alloc_out(o);
    }
  }
  if (scan->kind == K_RADIALSCAN) {
    if (lim >= 0)
      for (Node *o : P.out_rasters) {
        DevRaster &r = bufs.at(o);
        if (r.ptr) cuda_check(cudaMemset2DAsync(r.ptr, r.pitch, 0xFF, (size_t)r.W * dt_size(r.dtype), r.H, st), "memset");
      }
    uint64_t aux[4] = {(uint64_t)scan->coord.arr[0], (uint64_t)scan->coord.arr[1], (uint64_t)lim, 0};
    if (tiled) {
      cuda_check(cudaMemsetAsync(work.ptr(), 0, R.bytes, st), "memset");
      KernelHandle kt = env.kernel(P.source, P.kname + "_tiles", P.smem_bytes);
      const long long cap = (long long)env.sm_count() * std::max(1, env.occupancy(kt, kRadialThreads, P.smem_bytes));
      aux[3] = (uint64_t)(uintptr_t)work.ptr();
      auto at = pack_args(g, P, get, bufs, 0, 0, g.W, g.H, aux);
      env.launch(kt, (int)std::max<long long>(1, std::min(cap, R.tiles)), kRadialThreads, P.smem_bytes, (CUstream_st *)st, at.data(),
                 at.size());
      return;
    }
    auto a = pack_args(g, P, get, bufs, 0, 0, g.W, g.H, aux);
    // long fronts: a cluster of kRadialCluster CTAs per octant, each holding a
    // segment of the fronts in shared memory
    const int maxdim = std::max(g.W, g.H);
    const size_t seg = ((size_t)maxdim + kRadialCluster - 1) / kRadialCluster;
    const size_t csmem = 2 * seg * dt_size(scan->meta.dtype);
    if (maxdim >= kRadialClusterDim && csmem <= (size_t)200 * 1024) {
      KernelHandle kc = env.kernel(P.source, P.kname + "_cl", csmem);
      env.launch_cluster(kc, 8 * kRadialCluster, 512, kRadialCluster, csmem, (CUstream_st *)st, a.data());
      return;
    }
    const size_t smem = radial_front_smem(g.W, g.H, scan->meta.dtype);
    env.launch(env.kernel(P.source, P.kname, smem), 8, 512, smem, (CUstream_st *)st, a.data(), a.size());
    return;
  }
  KernelHandle kh = env.kernel(P.source, P.kname, 0);
  const size_t N = (size_t)g.W * g.H;
  if (N >= (size_t)1 << 31) throw MapError("spreadScan: raster too large");
  if (N > kSpreadKahnCells && N <= spread_pj_cells() && spread_pj_type(scan->meta.dtype)) {
    cuda_check(work.alloc(spread_pj_scratch(N, scan->meta.dtype)), "allocation of the flow accumulation's scratch");
    const int rounds = spread_pj_rounds(N);
    const int grid = (int)std::max<size_t>(1, std::min<size_t>((2 * N + 255) / 256, (size_t)env.sm_count() * 8));
    uint64_t aux[4] = {(uint64_t)(uintptr_t)work.ptr(), 0, 0, 0};
    auto a = pack_args(g, P, get, bufs, 0, 0, g.W, g.H, aux);
    env.launch(env.kernel(P.source, P.kname + "_pj_init", 0), grid, 256, 0, (CUstream_st *)st, a.data(), a.size());
    KernelHandle ks = env.kernel(P.source, P.kname + "_pj_step", 0);
    for (int r = 0; r < rounds; r++) {
      aux[1] = (uint64_t)r;
      auto ar = pack_args(g, P, get, bufs, 0, 0, g.W, g.H, aux);
      env.launch(ks, grid, 256, 0, (CUstream_st *)st, ar.data(), ar.size());
    }
    aux[1] = (uint64_t)rounds;
    auto af = pack_args(g, P, get, bufs, 0, 0, g.W, g.H, aux);
    env.launch(env.kernel(P.source, P.kname + "_pj_final", 0), grid, 256, 0, (CUstream_st *)st, af.data(), af.size());
    return;
  }
  // Over tiles at every size: 64^2 33 us against 42 of the one-CTA sweep, 256^2 38
  // against 365, 700 x 500 50 against 98 of the walks, 2048^2 103 against 500-544,
  // 8000^2 1.1 ms against 7.4 (directions included). The walks are ahead only where next
  // to nothing flows, which no size tells: no code set, 700^2, 28 us against 15; rasters
  // 4 cells wide, whose paths soon end, 47 against 23 (along them, 1 ms against 59).
  // Rasters too thin for the slots' numbers walk.
  if (spread_tile_type(scan->meta.dtype) && spread_tiles_fit(g.W, g.H) && Runtime::get().exec_mode == EXEC_FUSED &&
      tile_scratch(work, spread_tile_scratch(g.W, g.H))) {
    uint64_t aux[4] = {(uint64_t)(uintptr_t)work.ptr(), 0, 0, 0};
    auto a = pack_args(g, P, get, bufs, 0, 0, g.W, g.H, aux);
    for (const char *pass : {"_flow_a", "_flow_b", "_flow_c"})
      env.launch(env.kernel(P.source, P.kname + pass, 0), (int)spread_tiles(g.W, g.H), kFlowThreads, 0, (CUstream_st *)st, a.data(),
                 a.size());
    return;
  }
  cuda_check(work.alloc(6 * N * sizeof(int32_t)), "allocation of the flow accumulation's scratch");
  int32_t *const w = (int32_t *)work.ptr();
  uint64_t aux[4] = {(uint64_t)(uintptr_t)w, (uint64_t)(uintptr_t)(w + 2 * N), (uint64_t)(uintptr_t)(w + 4 * N), (uint64_t)(N + 1)};
  auto a = pack_args(g, P, get, bufs, 0, 0, g.W, g.H, aux);
  if (N <= kSpreadKahnCells) {
    // one CTA, frontier by frontier: the lowest latency up to 64 K cells
    env.launch(env.kernel(P.source, P.kname + "_kahn", 0), 1, 1024, 0, (CUstream_st *)st, a.data(), a.size());
  } else {
    const int grid = (int)std::max<size_t>(1, std::min<size_t>((N + 255) / 256, (size_t)env.sm_count() * 8));
    KernelHandle ki = env.kernel(P.source, P.kname + "_init", 0);
    env.launch(ki, grid, 256, 0, (CUstream_st *)st, a.data(), a.size());
    env.launch(kh, grid, 256, 0, (CUstream_st *)st, a.data(), a.size());
  }
}

}  // namespace mapb
