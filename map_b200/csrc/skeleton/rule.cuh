// Device building blocks of chained generations of a binary neighbourhood rule: a
// focal step on a byte raster that maps windows of zeros and ones to zero or one
// by the centre cell and the count of its eight neighbours (Life and its kin; the
// generator finds such steps by evaluating all 512 windows). Several generations
// run per launch on a tile held as bits, 32 cells of a row per word.
//
// 100 Life generations at 4096^2: 224 us, against 1600 us for a launch per
// generation on bytes (16 us each: reading and writing the grid through L2 and 20
// instructions per cell). A launch of 15 generations takes 35 us on 130 CTAs, one
// per SM; the integer pipe bounds it (about 24 instructions per word and
// generation at half rate). Measured beside it: 8 warps of 24 rows 340 us (too few
// warps, and the unrolled rows' code misses the instruction cache), loads and stores
// of a warp's own rows instead of 16 cells per thread step 427 us, the border
// tests inside the row loop 738 us.
#pragma once
#include "map_common.cuh"

// A tile is 32 words (one per lane) by NW warps of R rows each. Every generation
// invalidates one more ring of the tile, so a launch of K generations keeps the
// rows K .. NW R - K and all columns but the RULE_PAD outer ones on either side.
// K is at most RULE_PAD = 16: tiles then start 16 bytes into a word's 32 cells, on
// 16-byte boundaries of the raster's rows.
#define RULE_PAD 16
#define RULE_COLS (1024 - 2 * RULE_PAD)

// 32 bytes of zeros and ones as one word: the products' terms of four bytes land on
// distinct bits, the four of interest on bits 28 .. 31
__device__ __forceinline__ u32 rule_pack4(u32 w) { return (w * 0x10204080u) >> 28; }
__device__ __forceinline__ u32 rule_unpack4(u32 n) { return (n * 0x00204081u) & 0x01010101u; }

// Left and right neighbours of a row's cells; the words' outer neighbours come from
// the lanes beside. At the raster's first and last column (bit masks P, Q) the
// neighbour outside is `sub`'s cell in that column (a mirror), or nothing (sub = 0).
template <bool COL> __device__ __forceinline__ void rule_lr(u32 w, u32 sub, u32 P, u32 Q, u32 &l, u32 &r) {
  const u32 pw = __shfl_up_sync(0xffffffffu, w, 1), nw = __shfl_down_sync(0xffffffffu, w, 1);
  l = __funnelshift_l(pw, w, 1);
  r = __funnelshift_r(w, nw, 1);
  if (COL) {
    l = (l & ~P) | (sub & P);
    r = (r & ~Q) | (sub & Q);
  }
}
// Sum of the left neighbour, own and right cells (two bits), and of the left and
// right ones alone.
struct RuleRow { u32 s0, s1, m0, m1; };
__device__ __forceinline__ RuleRow rule_sum(u32 l, u32 c, u32 r) {
  RuleRow s;
  s.m0 = l ^ r;
  s.m1 = l & r;
  s.s0 = s.m0 ^ c;
  s.s1 = s.m1 | (s.m0 & c);
  return s;
}
// count of the eight neighbours in four bits, and the rule's next cells
template <class RULE> __device__ __forceinline__ u32 rule_next(const RuleRow &u, const RuleRow &m, const RuleRow &d, u32 c) {
  const u32 x = u.s0 ^ d.s0, s0 = x ^ m.m0, c0 = (u.s0 & d.s0) | (x & m.m0);
  const u32 y = u.s1 ^ d.s1, z = y ^ m.m1, w = (u.s1 & d.s1) | (y & m.m1);
  const u32 s1 = z ^ c0, c1 = z & c0;
  return RULE::next(s0, s1, w ^ c1, w & c1, c);
}

struct RuleEdge {
  u32 P, Q;       // this lane's bits of the raster's first and last column
  u32 F, L;       // its first and last columns of a block (block mirror), with P and Q
  u32 mirror;     // all ones under a mirror border, zero under the dead one
};

// One generation of a warp's R rows; `above` and `below` are the rows beside them.
// COL: the tile holds the raster's first or last column.
template <class RULE, int R, bool COL>
__device__ __forceinline__ void rule_step(u32 (&w)[R], u32 above, u32 below, const RuleEdge &e) {
  auto row = [&](u32 c) {
    u32 l, r;
    rule_lr<COL>(c, c & e.mirror, e.P, e.Q, l, r);
    return rule_sum(l, c, r);
  };
  RuleRow up = row(above), me = row(w[0]);
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const RuleRow down = row(i + 1 < R ? w[i + 1 < R ? i + 1 : 0] : below);
    w[i] = rule_next<RULE>(up, me, down, w[i]);
    up = me;
    me = down;
  }
}

// The next cells of a row y whose windows the border rule bends: the raster's first
// or last row, whose outer row is its own cells, reflected at its blocks' columns;
// or a block's first or last row at the raster's first or last column, where the
// window reads its own row. p, c, n: the old rows y - 1, y, y + 1.
template <class RULE>
__device__ __forceinline__ u32 rule_bent(u32 p, u32 c, u32 n, int y, const Geom &g, const RuleEdge &e) {
  auto row = [&](u32 v, u32 sub) {
    u32 l, r;
    rule_lr<true>(v, sub & e.mirror, e.P, e.Q, l, r);
    return rule_sum(l, v, r);
  };
  auto outside = [&]() {
    u32 l, r;
    rule_lr<true>(c, c, e.P, e.Q, l, r);
    RuleRow s = rule_sum((l & ~e.F) | (c & e.F), c, (r & ~e.L) | (c & e.L));
    s.s0 &= e.mirror;
    s.s1 &= e.mirror;
    return s;
  };
  const bool block = g.border == 0;
  const RuleRow up = y == 0 ? outside() : row(p, block && y % g.BS1 == 0 ? c : p);
  const RuleRow down = y == g.H - 1 ? outside() : row(n, block && y % g.BS1 == g.BS1 - 1 ? c : n);
  return rule_next<RULE>(up, row(c, c), down, c);
}

// The rule on bytes of any value, for tiles that hold others than zero and one:
// RULE_SX x RULE_SY cells with a ring of RULE_PAD in shared memory, one cell per
// thread step, two buffers in turn.
#define RULE_SX 256
#define RULE_SY 128
#define RULE_BX (RULE_SX + 2 * RULE_PAD)
#define RULE_BY (RULE_SY + 2 * RULE_PAD)
#define RULE_SMEM (2 * RULE_BX * RULE_BY)
struct RuleTap {
  const u8 *s;
  const Geom *g;
  int x0, y0;
  __device__ __forceinline__ u8 tap(int x, int y, int, int, int dx, int dy) const {
    int sx, sy;
    return focal_src(*g, x, y, dx, dy, sx, sy) ? s[(sy - y0) * RULE_BX + (sx - x0)] : (u8)0;
  }
};

// K generations of the rows [ya, yb) and columns [xa, xb) of the raster
template <class RULE, class ARGS>
__device__ __forceinline__ void rule_bytes(const ARGS &a, int K, int xa, int ya, int xb, int yb, unsigned char *smem) {
  const Geom &g = a.g;
  for (int by = ya; by < yb; by += RULE_SY)
    for (int bx = xa; bx < xb; bx += RULE_SX) {
      const int x0 = bx - K, y0 = by - K, ex = min(xb, bx + RULE_SX), ey = min(yb, by + RULE_SY);
      u8 *src = smem, *dst = smem + RULE_BX * RULE_BY;
      __syncthreads();
      for (int m = 0; m <= K; ++m) {
        // generation m of the cells within K - m of the sub-tile (m = 0: the loads)
        const int cx = max(0, x0 + m), cy = max(0, y0 + m), dx = min(g.W, ex + K - m), dy = min(g.H, ey + K - m);
        const int w = dx - cx, n = w * (dy - cy);
        const RuleTap f{src, &g, x0, y0};
        for (int i = (int)threadIdx.x; i < n; i += (int)blockDim.x) {
          const int x = cx + i % w, y = cy + i / w, at = (y - y0) * RULE_BX + (x - x0);
          const u8 v = m == 0 ? ldr<u8>(a.in[0], x, y) : RULE::cell(a, f, x, y);
          if (m == K) str<u8>(a.out[0], x, y, v);
          else if (m == 0) src[at] = v;
          else dst[at] = v;
        }
        __syncthreads();
        if (m > 0) {
          u8 *t = src;
          src = dst;
          dst = t;
        }
      }
    }
}

// One tile: aux[0] generations. Whole 16-byte pieces of a row inside the raster
// are read and written as such, others byte by byte.
template <class RULE, int R, int NW, class ARGS> __device__ __forceinline__ void rule_tile(const ARGS &a) {
  extern __shared__ __align__(16) unsigned char rule_smem[];
  const Geom &g = a.g;
  const int K = (int)a.aux[0], lane = (int)threadIdx.x & 31, warp = (int)threadIdx.x >> 5;
  const int rows = NW * R - 2 * K;
  const int xa = (int)blockIdx.x * RULE_COLS, ya = (int)blockIdx.y * rows;
  const int xb = min(g.W, xa + RULE_COLS), yb = min(g.H, ya + rows);
  const int x = xa - RULE_PAD + 32 * lane, y0 = ya - K + warp * R;
  u32 *const old = (u32 *)rule_smem;   // [generation parity][row of the tile][lane]
  // the tile's bytes as bits, 16 cells of a row per thread step; steps outside the
  // raster read its first cells and count for nothing
  u32 odd = 0u;
  constexpr int NT = 32 * NW, STEPS = NW * R * 64 / NT, BATCH = 8;
  static_assert(STEPS % BATCH == 0, "whole batches");
  for (int s = 0; s < STEPS; s += BATCH) {
    uint4 q[BATCH];
    bool in[BATCH];
#pragma unroll
    for (int u = 0; u < BATCH; ++u) {
      const int c = (int)threadIdx.x + (s + u) * NT, y = ya - K + (c >> 6), xs = xa - RULE_PAD + 16 * (c & 63);
      in[u] = y >= 0 && y < g.H && xs >= 0 && xs + 16 <= g.W;
      q[u] = make_uint4(0u, 0u, 0u, 0u);
      if (in[u]) q[u] = __ldg((const uint4 *)(row_ptr<u8>(a.in[0], y) + xs));
    }
#pragma unroll
    for (int u = 0; u < BATCH; ++u) {
      const int c = (int)threadIdx.x + (s + u) * NT;
      odd |= q[u].x | q[u].y | q[u].z | q[u].w;
      ((u16 *)old)[c] = (u16)(rule_pack4(q[u].x) | rule_pack4(q[u].y) << 4 | rule_pack4(q[u].z) << 8 | rule_pack4(q[u].w) << 12);
    }
  }
  // the 16 cells of every row that the raster's end cuts
  const int cut = g.W & ~15;
  if (cut != g.W && cut >= xa - RULE_PAD && cut < xa - RULE_PAD + 1024) {
    __syncthreads();
    for (int i = (int)threadIdx.x; i < NW * R; i += NT) {
      const int y = ya - K + i;
      if (y < 0 || y >= g.H) continue;
      const u8 *const p = row_ptr<u8>(a.in[0], y);
      u32 b = 0u;
      for (int j = cut; j < g.W; ++j) {
        const u32 v = p[j];
        odd |= v;
        b |= (v & 1u) << (j - cut);
      }
      ((u16 *)old)[i * 64 + (cut - xa + RULE_PAD) / 16] = (u16)b;
    }
  }
  if (__syncthreads_or((odd & 0xfefefefeu) != 0u)) {
    rule_bytes<RULE>(a, K, xa, ya, xb, yb, rule_smem);
    return;
  }
  u32 w[R];
#pragma unroll
  for (int i = 0; i < R; ++i) w[i] = old[(warp * R + i) * 32 + lane];
  RuleEdge e;
  e.P = x <= 0 && x + 31 >= 0 ? 1u << (-x & 31) : 0u;
  e.Q = x <= g.W - 1 && x + 31 >= g.W - 1 ? 1u << ((g.W - 1 - x) & 31) : 0u;
  e.F = e.P;
  e.L = e.Q;
  e.mirror = g.border != 2 ? 0xffffffffu : 0u;
  const bool col = xa == 0 || xb + RULE_PAD >= g.W, block = g.border == 0;
  // the warp's rows whose windows the border rule bends
  u32 bent = 0u;
  for (int i = 0; i < R; ++i) {
    const int y = y0 + i;
    if (y == 0 || y == g.H - 1 || (block && col && y > 0 && y < g.H && (y % g.BS1 == 0 || y % g.BS1 == g.BS1 - 1))) bent |= 1u << i;
  }
  if (block && (ya < K || yb + K >= g.H))
    for (int j = 0; j < 32; ++j)
      if (x + j >= 0 && x + j < g.W) {
        const int bx = (x + j) % g.BS0;
        if (bx == 0) e.F |= 1u << j;
        if (bx == g.BS0 - 1) e.L |= 1u << j;
      }
  // Tiles with such rows keep every row of the generation before in shared memory,
  // others only each warp's first and last.
  const bool keep = __syncthreads_or(bent != 0u);
  for (int n = 0; n < K; ++n) {
    u32 *const o = old + ((n & 1) * NW * R + warp * R) * 32 + lane;
    if (keep) {
#pragma unroll
      for (int i = 0; i < R; ++i) o[32 * i] = w[i];
    } else {
      o[0] = w[0];
      o[32 * (R - 1)] = w[R - 1];
    }
    __syncthreads();
    const u32 above = warp > 0 ? o[-32] : 0u, below = warp + 1 < NW ? o[32 * R] : 0u;
    if (col) rule_step<RULE, R, true>(w, above, below, e);
    else rule_step<RULE, R, false>(w, above, below, e);
    for (u32 m = bent; m; m &= m - 1) {
      const int k = __ffs((int)m) - 1;
      const u32 v = rule_bent<RULE>(k > 0 ? o[32 * (k - 1)] : above, o[32 * k], k + 1 < R ? o[32 * (k + 1)] : below, y0 + k, g, e);
#pragma unroll
      for (int i = 0; i < R; ++i)
        if (i == k) w[i] = v;
    }
  }
  // The next launch may take its place from here: earlier, its tiles would crowd
  // the SMs this one leaves free instead of spreading over all (49 against 35 us).
  griddep_launch();
  // back to bytes: the columns and rows the tile keeps
  u32 *const fin = old + (K & 1) * NW * R * 32;
#pragma unroll
  for (int i = 0; i < R; ++i) fin[(warp * R + i) * 32 + lane] = w[i];
  __syncthreads();
#pragma unroll 4
  for (int s = 0; s < STEPS; ++s) {
    const int c = (int)threadIdx.x + s * NT, y = ya - K + (c >> 6), xs = xa - RULE_PAD + 16 * (c & 63);
    if (y < ya || y >= yb || xs < xa || xs >= xb) continue;
    const u32 b = ((const u16 *)fin)[c];
    u8 *const p = (u8 *)(a.out[0].p + (u64)(s64)y * (u64)a.out[0].pitch) + xs;
    if (xs + 16 <= g.W) {
      *(uint4 *)p = make_uint4(rule_unpack4(b & 15u), rule_unpack4((b >> 4) & 15u), rule_unpack4((b >> 8) & 15u), rule_unpack4(b >> 12));
    } else {
      for (int j = 0; j < 16; ++j)
        if (xs + j < g.W) p[j] = (u8)((b >> j) & 1u);
    }
  }
}
