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

// Tiles that hold other bytes than zero and one run the rule on bytes, four cells of a
// row as 16-bit lanes (Q4), until every cell is zero or one: after the first generation
// for rules that only yield these. A tile's two buffers in turn lie in scratch memory
// that stays in L2: row i holds raster row ya - K + i, its 1024 cells RULE_PAD bytes in.
// Cells outside the raster hold what the border rule reads there: zero, or their mirror
// image. 4096^2 cells of 0 and 255: 10 generations 69 us, 50 155 us, of noise 67 and 199
// (one byte at a time, ring and border rule in every tap, 2488 and 3324; a launch per
// generation 162 and 800); one odd byte in 10 generations of Life 50 (2383; 162). Two
// generations take 37 us against 31 of two launches, three 39 against 48: the four passes
// over the tile's bytes are behind for two only. A generation is bound by its 65
// instructions per four cells on the CTA's 16 warps.
#define RULE_BW (1024 + 2 * RULE_PAD)
// Scratch at aux[1] (host: rule_scratch): RULE_SLOTS lock words, zero between launches,
// then aux[2] slots of RULE_BYTES. A tile takes a slot while it runs on bytes; there are
// as many as CTAs can be resident (up to two per SM, beyond which they wait).
#define RULE_SLOTS 2048
#define RULE_BYTES(rows) (2 * (rows) * RULE_BW)
#define RULE_TRIES (1u << 22)
template <class ARGS> __device__ __forceinline__ int rule_take_slot(const ARGS &a) {
  u32 *const lock = (u32 *)a.aux[1];
  const u32 n = (u32)a.aux[2];
  u32 i = (blockIdx.y * gridDim.x + blockIdx.x) % n;
  for (u32 t = 0; t < RULE_TRIES; ++t) {
    if (atomicCAS(&lock[i], 0u, 1u) == 0u) {
      __threadfence();
      return (int)i;
    }
    if (++i == n) i = 0u;
    if (t >= n) __nanosleep(100);
  }
  skel_fail(a.err, ERR_SPIN_LIMIT);
  return -1;
}
struct RuleTap {
  const u8 *s;   // the cell (x0, y0)
  const Geom *g;
  int x0, y0;
  __device__ __forceinline__ u8 tap(int x, int y, int, int, int dx, int dy) const {
    int sx, sy;
    return focal_src(*g, x, y, dx, dy, sx, sy) ? s[(sy - y0) * RULE_BW + (sx - x0)] : (u8)0;
  }
};
// The words left of, at and right of a quad, in the rows above, of and below a batch
// (the taps as SmemTap::tap4 takes them from staged rows).
template <int RB> struct RuleQuads {
  u32 w[RB + 2][3];
  __device__ __forceinline__ void load(int r, const u8 *p) {
#pragma unroll
    for (int m = 0; m < 3; ++m) w[r][m] = *(const u32 *)(p + 4 * (m - 1));
  }
  __device__ __forceinline__ Q4 tap4(int, int ly, int dx, int dy) const {
    const u32 *const c = w[ly + 1 + dy];
    if (dx == 0) return q4_bytes(c[1]);
    if (dx < 0) return Q4{__byte_perm(c[0], q4_odd(c[1]), 0x5453), q4_even(c[1])};
    return Q4{q4_odd(c[1]), __byte_perm(q4_even(c[1]), c[2], 0x1412)};
  }
};

// Up to K generations of a tile; returns how many were run, with the cells of the last
// in `cells` (column 0 of row 0): K, or fewer when all are zero or one.
template <class RULE, int ROWS, int NT, class ARGS>
__device__ __forceinline__ int rule_bytes(const ARGS &a, int K, int xa, int ya, u8 *buf, const u8 *&cells) {
  constexpr int RB = 4, PIECES = RULE_BW / 16;
  static_assert(NT % 256 == 0, "256 quads a row");
  const Geom &g = a.g;
  const int tid = (int)threadIdx.x, x0 = xa - RULE_PAD, y0 = ya - K;
  u8 *src = buf + RULE_PAD, *dst = src + ROWS * RULE_BW;
  const bool mirror = g.border != 2;
  // the tile's cells, zero outside the raster; there the other buffer is zero too
  constexpr int BATCH = 4;
  for (int c0 = tid; c0 < ROWS * PIECES; c0 += BATCH * NT) {
    uint4 v[BATCH];
    bool whole[BATCH];
#pragma unroll
    for (int u = 0; u < BATCH; ++u) {
      const int c = c0 + u * NT, i = c / PIECES, p = c % PIECES - 1, x = x0 + 16 * p, y = y0 + i;
      whole[u] = i < ROWS && y >= 0 && y < g.H && p >= 0 && p < 64 && x >= 0 && x + 16 <= g.W;
      v[u] = make_uint4(0u, 0u, 0u, 0u);
      if (whole[u]) v[u] = __ldg((const uint4 *)(row_ptr<u8>(a.in[0], y) + x));
    }
#pragma unroll
    for (int u = 0; u < BATCH; ++u) {
      const int c = c0 + u * NT, i = c / PIECES, at = i * RULE_BW + 16 * (c % PIECES - 1);
      if (i < ROWS) *(uint4 *)(src + at) = v[u];
      if (i < ROWS && !whole[u]) *(uint4 *)(dst + at) = v[u];
    }
  }
  // the cells of every row that the raster's end cuts
  const int cut = g.W & ~15;
  if (cut != g.W && cut >= x0 && cut < x0 + 1024) {
    __syncthreads();
    for (int i = max(0, -y0) + tid; i < min(ROWS, g.H - y0); i += NT)
      for (int x = cut; x < g.W; ++x) src[i * RULE_BW + x - x0] = row_ptr<u8>(a.in[0], y0 + i)[x];
  }
  __syncthreads();
  // the cells beside the raster's edges, from the edges' own
  auto ring = [&](u8 *s) {
    auto put = [&](int x, int y) {
      s[(y - y0) * RULE_BW + x - x0] = s[(min(max(y, 0), g.H - 1) - y0) * RULE_BW + min(max(x, 0), g.W - 1) - x0];
    };
#pragma unroll 1
    for (int side = 0; side < 2; ++side) {
      const int y = side ? g.H : -1, x = side ? g.W : -1;
      const int yc = side ? g.H - 1 : 0, xc = side ? g.W - 1 : 0;
      if (y >= y0 && y < y0 + ROWS && yc >= y0 && yc < y0 + ROWS)
        for (int c = tid; c < 1024; c += NT)
          if (x0 + c >= -1 && x0 + c <= g.W && min(max(x0 + c, 0), g.W - 1) >= x0) put(x0 + c, y);
      if (x >= x0 && x < x0 + 1024 && xc >= x0)
        for (int i = tid; i < ROWS; i += NT)
          if (y0 + i >= 0 && y0 + i < g.H) put(x, y0 + i);
    }
  };
  if (mirror) {
    ring(src);
    __syncthreads();
  }
  const int q = tid & 255, xq = x0 + 4 * q;
  const bool quad = xq >= 0 && xq < g.W;
  const u32 mask = xq + 4 <= g.W ? 0xffffffffu : 0xffffffffu >> (8 * (xq + 4 - g.W) & 31);
  const bool edge = g.border == 0 && (x0 <= 0 || x0 + 1024 >= g.W || y0 <= 0 || y0 + ROWS >= g.H);
  for (int m = 1;; ++m) {
    const int ia = max(m, -y0), ib = min(ROWS - m, g.H - y0), per = (ib - ia + NT / 256 - 1) / (NT / 256);
    const int ra = ia + (tid >> 8) * per, rb = min(ib, ra + per);
    u32 odd = 0u;
    if (quad && ra < rb) {
      const u8 *s = src + (ra - 1) * RULE_BW + 4 * q;
      u8 *d = dst + ra * RULE_BW + 4 * q;
      RuleQuads<RB> f;
      f.load(0, s);
      f.load(1, s + RULE_BW);
      for (int i = ra; i < rb; i += RB, s += RB * RULE_BW, d += RB * RULE_BW) {
#pragma unroll
        for (int r = 0; r < RB; ++r)
          if (i + r < rb) f.load(r + 2, s + (r + 2) * RULE_BW);
#pragma unroll
        for (int r = 0; r < RB; ++r)
          if (i + r < rb) {
            const u32 v = RULE::cell4(a, f, r) & mask;
            odd |= v;
            *(u32 *)(d + r * RULE_BW) = v;
          }
#pragma unroll
        for (int n = 0; n < 3; ++n) {
          f.w[0][n] = f.w[RB][n];
          f.w[1][n] = f.w[RB + 1][n];
        }
      }
    }
    if (edge) {
      // the cells whose windows the block mirror reflects inside their block
      __syncthreads();
      const RuleTap f{src, &g, x0, y0};
      auto cell = [&](int x, int y) {
        const u8 v = RULE::cell(a, f, x, y);
        odd |= v;
        dst[(y - y0) * RULE_BW + x - x0] = v;
      };
#pragma unroll 1
      for (int side = 0; side < 2; ++side) {
        const int y = side ? g.H - 1 : 0, x = side ? g.W - 1 : 0;
        if (y - y0 >= ia && y - y0 < ib)
          for (int c = tid + 1; c < 1023; c += NT) {
            const int cx = x0 + c, b = cx % g.BS0;
            if (cx >= 0 && cx < g.W && (b == 0 || b == g.BS0 - 1 || cx == g.W - 1)) cell(cx, y);
          }
        if (x > x0 && x < x0 + 1023)
          for (int i = ia + tid; i < ib; i += NT) {
            const int b = (y0 + i) % g.BS1;
            if (b == 0 || b == g.BS1 - 1 || y0 + i == g.H - 1) cell(x, y0 + i);
          }
      }
    }
    const bool more = __syncthreads_or((odd & 0xfefefefeu) != 0u);
    cells = dst;
    if (m == K || !more) return m;
    if (mirror) {
      ring(dst);
      __syncthreads();
    }
    u8 *t = src;
    src = dst;
    dst = t;
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
  int done = 0;   // generations run on bytes
  if (__syncthreads_or((odd & 0xfefefefeu) != 0u)) {
    if (threadIdx.x == 0) old[0] = (u32)rule_take_slot(a);   // (the tile's bits are not needed)
    __syncthreads();
    const int slot = (int)old[0];
    if (slot < 0) return;
    const u8 *cells;
    u8 *const buf = (u8 *)a.aux[1] + 4 * RULE_SLOTS + (s64)slot * RULE_BYTES(NW * R);
    done = rule_bytes<RULE, NW * R, NT>(a, K, xa, ya, buf, cells);
#pragma unroll 4
    for (int s = 0; s < STEPS; ++s) {
      const int c = (int)threadIdx.x + s * NT, i = c >> 6, xs = xa - RULE_PAD + 16 * (c & 63), y = ya - K + i;
      const uint4 v = *(const uint4 *)(cells + i * RULE_BW + 16 * (c & 63));
      if (done < K) {
        ((u16 *)old)[c] = (u16)(rule_pack4(v.x & 0x01010101u) | rule_pack4(v.y & 0x01010101u) << 4 |
                                rule_pack4(v.z & 0x01010101u) << 8 | rule_pack4(v.w & 0x01010101u) << 12);
      } else if (y >= ya && y < yb && xs >= xa && xs < xb) {
        u8 *const p = (u8 *)(a.out[0].p + (u64)(s64)y * (u64)a.out[0].pitch) + xs;
        if (xs + 16 <= g.W) {
          *(uint4 *)p = v;
        } else {
          for (int j = 0; xs + j < g.W; ++j) p[j] = cells[i * RULE_BW + 16 * (c & 63) + j];
        }
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      atomicExch((u32 *)a.aux[1] + slot, 0u);
    }
    if (done == K) return;
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
  for (int n = done; n < K; ++n) {
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
