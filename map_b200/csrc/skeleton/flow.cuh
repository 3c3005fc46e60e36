// Device building blocks of flow accumulation over tiles (32-bit integer water).
// The D8 forest is cut at the edges of 64 x 64 tiles and summed in three passes:
//   A. every tile sums its own cells in shared memory, and finds for every cell of
//      its rim that takes water from outside the rim cell where that water leaves
//      again (or that it stays);
//   B. the rim cells where water leaves form a much smaller forest (a hop crosses a
//      tile); each gets the water of all tiles above it by downstream walks, as the
//      whole-raster walks do cell by cell;
//   C. every tile adds the water that enters at its rim to the sums of pass A (kept
//      in the output) down the paths it takes, and takes each cell's own water off.
// Integer sums are exact in any order, modulo the type's width, so the result is the
// whole-raster walks' bit for bit. Cells on a cycle of codes never complete and hold
// zero, as there; a cell has one code, so no path leaves a cycle and all other cells
// complete. Cycles inside a tile are found by pass A's pointers and marked in the
// scratch, those that cross tiles by the slots that pass B leaves pending.
//
// 2048^2 (fBm, 4.2 M cells): 42 + 7 + 38 us for the passes, against 46 + 540 us for
// counting and walking the whole raster, whose longest path of one L2 atomic per cell
// bounds it. The tiles' passes are bound by shared-memory latency at five CTAs per SM
// (launch bounds; passes on terrain of 2048^2 / 3000^2: four 78.7 / 97.1 us, five 76.3 /
// 91.0, six 76.6 / 90.4 and random codes slower, none given 78.7 / 94.0). Tried for the
// tiles: walks with counts 200 us a pass (a thread's longest walk sets the tile's time), doubling in
// pass C too 56 us. Random codes, full of cycles, at 2048^2: 124 us, against 279 of the
// whole-raster walks and 642 when tiles with a cycle took walks with counts.
#pragma once
#include "map_scan.cuh"

#define FLOW_T 64                      // cells per tile side
#define FLOW_NT 256
#define FLOW_RIM 256                   // rim slots per tile
#define FLOW_SOURCE 0x80000000u        // pending count of a cell nothing flows into
#define FLOW_DONE 0x8000               // a path's pointer that has reached its end
#define FLOW_CYCLE (-2)                // the enter slot that marks a tile with a cycle of codes
#define FLOW_EXIT 0x4000               // the end is a rim cell whose water leaves the tile

// Scratch at aux[0] (host: spread_tile_scratch): per rim slot the water that leaves
// there and its pending pushes (u64), the slot it enters by in the next tile (s32), and
// for a slot where water enters the one where it leaves again (s32, -1: it stays); per
// tile with a cycle of codes a bit per cell, set for the cycles' cells.
struct FlowScratch {
  u64 *pk;
  s32 *enter, *leave;
  u32 *loop;
  int tx, ty;
};
template <class ARGS> __device__ __forceinline__ FlowScratch flow_scratch(const ARGS &a) {
  FlowScratch f;
  f.tx = (a.g.W + FLOW_T - 1) / FLOW_T;
  f.ty = (a.g.H + FLOW_T - 1) / FLOW_T;
  const s64 n = (s64)f.tx * f.ty * FLOW_RIM;
  f.pk = (u64 *)a.aux[0];
  f.enter = (s32 *)(f.pk + n);
  f.leave = f.enter + n;
  f.loop = (u32 *)(f.leave + n);
  return f;
}
// Rim slot of cell (lx, ly) of a w x h tile: top row, bottom row, left and right column.
__device__ __forceinline__ int flow_rim(int lx, int ly, int w, int h) {
  return ly == 0 ? lx : ly == h - 1 ? FLOW_T + lx : lx == 0 ? 2 * FLOW_T + ly : 3 * FLOW_T + ly;
}
// Slot of raster cell (x, y), which lies on its tile's rim.
__device__ __forceinline__ int flow_slot(const FlowScratch &f, int W, int H, int x, int y) {
  const int cx = x / FLOW_T, cy = y / FLOW_T;
  return (cy * f.tx + cx) * FLOW_RIM +
         flow_rim(x - cx * FLOW_T, y - cy * FLOW_T, min(FLOW_T, W - cx * FLOW_T), min(FLOW_T, H - cy * FLOW_T));
}

// Sums a tile by doubling: in round r every cell adds what it holds to the cell 2^r
// steps down its path, if the path is that long, and takes over that cell's pointer;
// afterwards sum[c] is the water of c and of all cells above it (c on no cycle of
// codes), and next[c] names the end of its path. Cells of a thread are independent, so
// a round's shared-memory latencies overlap. False when a path has not ended after
// rounds for twice the longest: its pointer is then a cell of the cycle that it runs
// into, and the cycle's own cells' pointers are all of its cells.
template <int PER> __device__ __forceinline__ bool flow_double(u32 *sum, u16 *next, int tid) {
  u32 s[PER];
  u16 n[PER];
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    s[k] = sum[tid + k * FLOW_NT];
    n[k] = next[tid + k * FLOW_NT];
  }
  for (int r = 0; r <= 12; ++r) {
    bool more = false;
#pragma unroll
    for (int k = 0; k < PER; ++k) more |= !(n[k] & FLOW_DONE);
    if (!__syncthreads_or(more)) return true;
#pragma unroll
    for (int k = 0; k < PER; ++k)
      if (!(n[k] & FLOW_DONE)) {
        atomicAdd(&sum[n[k]], s[k]);
        n[k] = next[n[k]];
      }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      s[k] = sum[tid + k * FLOW_NT];
      next[tid + k * FLOW_NT] = n[k];
    }
  }
  return false;
}

template <class OPS, bool FINAL, class ARGS>
__device__ __forceinline__ void flow_tile(const ARGS &a, const RasterArg &D, const RasterArg &O, int tile) {
  constexpr int CW = FLOW_T + 32, PAD = 16, CELLS = FLOW_T * FLOW_T, PER = CELLS / FLOW_NT;
  __shared__ __align__(16) u8 code[CW * (FLOW_T + 2)];   // rows y0 - 1 .. y0 + 64, columns x0 - 16 .. x0 + 79
  __shared__ u32 sum[CELLS], loop[CELLS / 32];   // loop: bits of the cells on cycles
  __shared__ u16 next[CELLS];
  __shared__ u32 pending[FLOW_RIM];
  const FlowScratch f = flow_scratch(a);
  const int W = a.g.W, H = a.g.H, tid = (int)threadIdx.x;
  const int x0 = tile % f.tx * FLOW_T, y0 = tile / f.tx * FLOW_T;
  const int w = min(FLOW_T, W - x0), h = min(FLOW_T, H - y0);
  const bool aligned = ((D.p | (u64)D.pitch) & 15) == 0;
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const int i = tid + s * FLOW_NT, row = i / (CW / 16), x = x0 - PAD + 16 * (i % (CW / 16)), y = y0 - 1 + row;
    if (row >= FLOW_T + 2) break;
    uint4 q = make_uint4(0u, 0u, 0u, 0u);
    if (y >= 0 && y < H) {
      const u8 *const p = row_ptr<u8>(D, y) + x;
      if (aligned && x >= 0 && x + 16 <= W) {
        q = __ldg((const uint4 *)p);
      } else {
        u32 v[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int b = 0; b < 16; ++b)
          if (x + b >= 0 && x + b < W) v[b / 4] |= (u32)__ldg(p + b) << (8 * (b % 4));
        q = make_uint4(v[0], v[1], v[2], v[3]);
      }
    }
    *(uint4 *)(code + 16 * i) = q;
  }
  static_assert((FLOW_T + 2) * (CW / 16) <= 2 * FLOW_NT, "two pieces of 16 codes per thread");
  pending[tid] = 0u;
  __syncthreads();
  // every cell's water, and the next cell of its path or the end of it (itself)
  auto step = [&](int c, int lx, int ly) -> u16 {
    const int d = d8_index(code[(ly + 1) * CW + lx + PAD]);
    if (lx >= w || ly >= h || d < 0) return (u16)(c | FLOW_DONE);
    const int nx = lx + d8_dx(d), ny = ly + d8_dy(d);
    if ((unsigned)nx < (unsigned)w && (unsigned)ny < (unsigned)h) return (u16)(ny * FLOW_T + nx);
    return (unsigned)(x0 + nx) < (unsigned)W && (unsigned)(y0 + ny) < (unsigned)H ? (u16)(c | FLOW_DONE | FLOW_EXIT)
                                                                                   : (u16)(c | FLOW_DONE);
  };
#pragma unroll 4
  for (int k = 0; k < PER; ++k) {
    const int c = tid + k * FLOW_NT, lx = c % FLOW_T, ly = c / FLOW_T;
    sum[c] = lx < w && ly < h ? (FINAL ? *cell_ptr<u32>(O, x0 + lx, y0 + ly) : OPS::water(a, x0 + lx, y0 + ly)) : 0u;
    next[c] = step(c, lx, ly);
  }
  // thread tid's rim cell, and what enters there from other tiles: the number of
  // cells (pass A), their water (pass C); blocked: cells that never completed
  int lx = tid % FLOW_T, ly = 0;
  const int side = tid / FLOW_T;
  bool rim = lx < w;
  if (side == 1) {
    ly = h - 1;
    rim = lx < w && h > 1;
  } else if (side > 1) {
    ly = tid % FLOW_T;
    lx = side == 2 ? 0 : w - 1;
    rim = ly > 0 && ly < h - 1 && (side == 2 || w > 1);
  }
  const int slot = tile * FLOW_RIM + tid, cell = ly * FLOW_T + lx;
  // the neighbours (bit j) outside the tile whose code leads to the rim cell
  u32 enter = 0u;
  if (rim) {
    const u8 *const p = code + (ly + 1) * CW + lx + PAD;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int nx = lx - d8_dx(j), ny = ly - d8_dy(j);
      const bool in = (unsigned)nx < (unsigned)w && (unsigned)ny < (unsigned)h;
      if (p[-d8_dx(j) - CW * d8_dy(j)] == (u8)(1 << j) && !in) enter |= 1u << j;
    }
  }
  auto mark = [&](int c) { atomicOr(&loop[c >> 5], 1u << (c & 31)); };
  auto marked = [&](int c) { return (*(volatile u32 *)&loop[c >> 5] >> (c & 31) & 1u) != 0u; };
  if (tid < CELLS / 32) loop[tid] = 0u;
  if (!FINAL) {
    __syncthreads();
    const bool cyclic = !flow_double<PER>(sum, next, tid);
    if (cyclic) {
      for (int k = 0; k < PER; ++k) {
        const u16 n = next[tid + k * FLOW_NT];
        if (!(n & FLOW_DONE)) mark(n);
      }
      __syncthreads();
      if (tid < CELLS / 32) f.loop[(s64)tile * (CELLS / 32) + tid] = loop[tid];
    }
    // where water that enters at a rim cell leaves the tile
    if (enter) {
      const u16 end = next[cell];
      if ((end & FLOW_DONE) && (end & FLOW_EXIT)) {
        const int at = end & (CELLS - 1), r = flow_rim(at % FLOW_T, at / FLOW_T, w, h);
        atomicAdd(&pending[r], (u32)__popc(enter));
        f.leave[slot] = tile * FLOW_RIM + r;
      } else {
        f.leave[slot] = -1;
      }
    }
    __syncthreads();
    s32 into = -1;
    if (rim && next[cell] == (u16)(cell | FLOW_DONE | FLOW_EXIT)) {
      const int d = d8_index(code[(ly + 1) * CW + lx + PAD]);
      into = flow_slot(f, W, H, x0 + lx + d8_dx(d), y0 + ly + d8_dy(d));
      f.pk[slot] = (u64)sum[cell] << 32 | (pending[tid] ? pending[tid] : FLOW_SOURCE);
    }
    // (the last slot is no cell's: the tile's cycle mark)
    f.enter[slot] = cyclic && tid == FLOW_RIM - 1 ? FLOW_CYCLE : into;
#pragma unroll 4
    for (int k = 0; k < PER; ++k) {
      const int i = tid + k * FLOW_NT, cx = i % FLOW_T, cy = i / FLOW_T;
      if (cx < w && cy < h) *cell_ptr<u32>(O, x0 + cx, y0 + cy) = sum[i];
    }
  } else {
    // the water that enters at the rim cell; slots still pending lie on a cycle, and
    // so do the cells down the path from where they enter
    u32 inflow = 0u;
    bool blocked = false;
    for (u32 m = enter; m; m &= m - 1) {
      const int j = __ffs((int)m) - 1;
      const u64 v = f.pk[flow_slot(f, W, H, x0 + lx - d8_dx(j), y0 + ly - d8_dy(j))];
      if ((u32)v == 0u || (u32)v == FLOW_SOURCE) inflow += (u32)(v >> 32);
      else blocked = true;
    }
    const bool cyclic = f.enter[tile * FLOW_RIM + FLOW_RIM - 1] == FLOW_CYCLE;
    const bool cycles = __syncthreads_or(blocked || cyclic);
    if (cyclic) {
      if (tid < CELLS / 32) loop[tid] = f.loop[(s64)tile * (CELLS / 32) + tid];
      __syncthreads();
    }
    if (!cycles) {
      if (inflow)
        for (int c = cell;; c = next[c]) {
          atomicAdd(&sum[c], inflow);
          if (next[c] & FLOW_DONE) break;
        }
    } else if (inflow || blocked) {
      // (apart: with the marks in them the usual walks took up to a third longer)
      int c = cell;
      for (int n = 0; n < CELLS; ++n) {
        if (cyclic && marked(c)) break;
        atomicAdd(&sum[c], inflow);
        if (blocked) mark(c);
        const u16 to = next[c];
        if (to & FLOW_DONE) break;
        c = to;
      }
    }
    __syncthreads();
    // (the cycles' cells, which hold no other tile's water, first: zero)
    if (cycles) {
      for (int k = 0; k < PER; ++k) {
        const int i = tid + k * FLOW_NT, cx = i % FLOW_T, cy = i / FLOW_T;
        if (cx < w && cy < h && marked(i)) sum[i] = OPS::water(a, x0 + cx, y0 + cy);
      }
    }
#pragma unroll 4
    for (int k = 0; k < PER; ++k) {
      const int i = tid + k * FLOW_NT, cx = i % FLOW_T, cy = i / FLOW_T;
      if (cx < w && cy < h) *cell_ptr<u32>(O, x0 + cx, y0 + cy) = sum[i] - OPS::water(a, x0 + cx, y0 + cy);
    }
  }
}

// Pass B: slot i of a raster.
template <class ARGS> __device__ __forceinline__ void flow_slots(const ARGS &a, s64 i) {
  const FlowScratch f = flow_scratch(a);
  const s64 n = (s64)f.tx * f.ty * FLOW_RIM;
  if (i >= n) return;
  s32 in = f.enter[i];
  if (in < 0) return;
  const u64 own = f.pk[i];
  if ((u32)own != FLOW_SOURCE) return;
  u32 carry = (u32)(own >> 32);
  for (s64 it = 0;; ++it) {
    if (it > n) {
      skel_fail(a.err, ERR_ITER_LIMIT);
      break;
    }
    const s32 to = f.leave[in];
    if (to < 0) break;
    in = f.enter[to];
    const u64 old = atomicAdd((unsigned long long *)&f.pk[to], ((u64)carry << 32) - 1ull);
    if ((u32)old != 1u) break;
    carry += (u32)(old >> 32);
  }
}
