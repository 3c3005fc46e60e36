// Device building blocks of the Radiating (radial scan) and Spreading (flow
// accumulation) skeletons.
#pragma once
#include "map_common.cuh"

// Octants of a radial scan: primary unit (p0,p1) and secondary unit (q0,q1).
// A cell at (d0, d1) from the start, 0 <= d1 <= d0, lies at start + d0*p + d1*q
// (the reference's eight RadialCase pairs, runtime/Direction.hpp:71-164).
__device__ __forceinline__ void octant_units(int o, int &p0, int &p1, int &q0, int &q1) {
  const int P[8][4] = {{0, -1, 1, 0}, {1, 0, 0, -1}, {1, 0, 0, 1}, {0, 1, 1, 0},
                       {0, 1, -1, 0}, {-1, 0, 0, 1}, {-1, 0, 0, -1}, {0, -1, -1, 0}};
  p0 = P[o][0]; p1 = P[o][1]; q0 = P[o][2]; q1 = P[o][3];
}

// Linear interpolation of the two previous cells along the ray
// (runtime/skeleton/util.cpp:564): a at (d0-1, d1), b at (d0-1, d1-1).
template <class T> __device__ __forceinline__ T radial_lit(T a, T b, int d0, int d1) {
  if (d1 == 0) return a;
  if (d0 == d1) return b;
  T w = (T)d1 / (T)d0 * ((T)d0 - (T)1.0f) - ((T)d1 - (T)1.0f);
  return a * w + b * ((T)1.0f - w);
}

// The weight of radial_lit's first operand (cells off the octant's two edges),
// given the correctly rounded reciprocal rc of d0. QUOT (float32, fronts below
// 2^20): the quotient d1 / d0 is the product d1 * rc with one residual correction
// (Markstein's method: P. Markstein, IBM J. Res. Dev. 34(1), 1990). The corrected
// value differs from the true quotient by less than 2^-47 of it before its one
// rounding, and no quotient of integers below 2^20 lies closer than 2^-46 of
// itself to a midpoint of two floats (its numerator would need 25 bits), so it is
// the correctly rounded quotient, the division's own result.
template <bool QUOT, class T> __device__ __forceinline__ T radial_weight(T d0, T d1, T rc) {
  T q;
  if constexpr (QUOT) {
    q = d1 * rc;
    q = __fmaf_rn(__fmaf_rn(-q, d0, d1), rc, q);
  } else {
    q = d1 / d0;
  }
  return q * (d0 - (T)1.0f) - (d1 - (T)1.0f);
}
template <class T> constexpr bool radial_has_quot = sizeof(T) == 4;
template <class T> __device__ __forceinline__ bool radial_quot(int last) { return radial_has_quot<T> && last < (1 << 20); }

__device__ __forceinline__ bool is_finite(float v) { return (__float_as_uint(v) & 0x7fffffffu) < 0x7f800000u; }
__device__ __forceinline__ bool is_finite(double v) { return isfinite(v); }
__device__ __forceinline__ u64 ld_relaxed_u64(const u64 *p) {
  u64 v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_u64(u64 *p, u64 v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// A cell handed to another CTA: every 32-bit word of its value travels with its
// own ready mark in one 64-bit word (zero before), so a reader that sees the mark
// has the value and no fence is needed.
#define RADIAL_WORDS(T) (sizeof(T) / 4)
__device__ __forceinline__ void radial_put(u64 *p, int i, float v) {
  st_relaxed_u64(p + i, (u64)1 << 32 | __float_as_uint(v));
}
__device__ __forceinline__ bool radial_get(const u64 *p, int i, float &v) {
  const u64 w = ld_relaxed_u64(p + i);
  v = __uint_as_float((u32)w);
  return (w >> 32) != 0;
}
__device__ __forceinline__ void radial_put(u64 *p, int i, double v) {
  const u64 b = (u64)__double_as_longlong(v);
  st_relaxed_u64(p + 2 * (s64)i, (u64)1 << 32 | (u32)b);
  st_relaxed_u64(p + 2 * (s64)i + 1, (u64)1 << 32 | (u32)(b >> 32));
}
__device__ __forceinline__ bool radial_get(const u64 *p, int i, double &v) {
  const u64 a = ld_relaxed_u64(p + 2 * (s64)i), b = ld_relaxed_u64(p + 2 * (s64)i + 1);
  v = __longlong_as_double((long long)((u64)(u32)b << 32 | (u32)a));
  return (a >> 32) != 0 && (b >> 32) != 0;
}

// Tiles of a radial scan: RADIAL_B own cells by RADIAL_T fronts, RADIAL_NT threads,
// the cell visits unrolled RADIAL_U times, RADIAL_G fronts per step of the sweep.
// Measured on the viewshed of a 4096^2 raster (217 us): 64 x 64 tiles of 128
// threads 225-232 us (longer strips between exchanges, but a tile evaluates the
// scan's argument 1.5 times per own cell over 64 cells at once, so the last strips
// leave SMs idle), 256 threads 242 us, G = 4 within 3% of 8.
#define RADIAL_B 32
#define RADIAL_T 32
#define RADIAL_NT 64
#define RADIAL_U 4
#define RADIAL_G 8
// Polls of the cells of the strip above before a tile gives up (about a second),
// and the pause between two polls in ns: 40 to 200 measured alike, none 15% slower
// (the polls of waiting tiles take the L2's time from the others').
#define RADIAL_POLLS (1u << 20)
#define RADIAL_PAUSE 100

// V consecutive cells of a shared-memory row, as 16-byte words where they fill them
template <int V> struct radial_row {
  static __device__ __forceinline__ void load(float (&x)[V], const float *p) {
    if constexpr (V % 4 == 0) {
#pragma unroll
      for (int r = 0; r < V; r += 4) {
        const float4 q = *(const float4 *)(p + r);
        x[r] = q.x; x[r + 1] = q.y; x[r + 2] = q.z; x[r + 3] = q.w;
      }
    } else {
#pragma unroll
      for (int r = 0; r < V; ++r) x[r] = p[r];
    }
  }
  static __device__ __forceinline__ void store(float *p, const float (&x)[V]) {
    if constexpr (V % 4 == 0) {
#pragma unroll
      for (int r = 0; r < V; r += 4) *(float4 *)(p + r) = make_float4(x[r], x[r + 1], x[r + 2], x[r + 3]);
    } else {
#pragma unroll
      for (int r = 0; r < V; ++r) p[r] = x[r];
    }
  }
  static __device__ __forceinline__ void load(double (&x)[V], const double *p) {
#pragma unroll
    for (int r = 0; r < V; r += 2) {
      const double2 q = *(const double2 *)(p + r);
      x[r] = q.x; x[r + 1] = q.y;
    }
  }
  static __device__ __forceinline__ void store(double *p, const double (&x)[V]) {
#pragma unroll
    for (int r = 0; r < V; r += 2) *(double2 *)(p + r) = make_double2(x[r], x[r + 1]);
  }
};

// Warp 0's sweep of G fronts from d0 = f on over the S region cells of a tile: a
// lane holds V consecutive cells, so one shuffle a front hands on the neighbour of
// its first. `row`: the lane's cells of the first front in shared memory; rc: the
// lane's share of the reciprocals of 32 fronts, of which the sweep's start at `at`.
// The arguments and weights do not depend on the sweep: only the two products, the
// sum and the fold of a cell are in its chain.
template <class OPS, class T, int S, int G, bool EDGE, bool QUOT>
__device__ __forceinline__ void radial_fronts(T *row, T (&val)[S / 32], const T (&d1f)[S / 32], T rc, int at, int f, int lo, int lane) {
  constexpr int V = S / 32, RS = S + 4;
  T x[G][V], rct[G];
#pragma unroll
  for (int t = 0; t < G; ++t) {
    rct[t] = __shfl_sync(0xffffffffu, rc, at + t);
    radial_row<V>::load(x[t], row + t * RS);
  }
#pragma unroll
  for (int t = 0; t < G; ++t) {
    const T d0f = (T)(f + t), left = __shfl_up_sync(0xffffffffu, val[V - 1], 1);
#pragma unroll
    for (int r = V - 1; r >= 0; --r) {
      const T b = r > 0 ? val[r > 0 ? r - 1 : 0] : left;
      const T w = radial_weight<QUOT, T>(d0f, d1f[r], rct[t]);
      T lit = val[r] * w + b * ((T)1.0f - w);
      if (EDGE) {
        const int d1 = lo + V * lane + r;
        if (f + t == d1) lit = b;
        if (d1 == 0) lit = val[r];
      }
      val[r] = OPS::fold(lit, x[t][r]);
    }
    radial_row<V>::store(row + t * RS, val);
  }
}

// Warp 0's sweep of a strip's nt fronts.
template <class OPS, class T, int S, int TT, bool EDGE, bool QUOT>
__device__ __forceinline__ void radial_sweep(T *s_in, T (&val)[S / 32], int f0, int nt, int lo, int lane) {
  constexpr int V = S / 32, RS = S + 4, G = RADIAL_G;
  T d1f[V];
#pragma unroll
  for (int r = 0; r < V; ++r) d1f[r] = (T)(lo + V * lane + r);
  for (int h = 0; h < nt; h += 32) {
    const T rc = (T)1 / (T)(f0 + 1 + h + lane);
    const int m = min(32, nt - h);
    int g = 0;
    for (; g + G <= m; g += G)
      radial_fronts<OPS, T, S, G, EDGE, QUOT>(s_in + (h + g) * RS + V * lane, val, d1f, rc, g, f0 + 1 + h + g, lo, lane);
    for (; g < m; ++g)
      radial_fronts<OPS, T, S, 1, EDGE, QUOT>(s_in + (h + g) * RS + V * lane, val, d1f, rc, g, f0 + 1 + h + g, lo, lane);
  }
}

// Visits the cells of a strip of nt fronts from f0 + 1 on and N cells from d1 = l0
// on that lie in the octant (and, above = 1, right of the tile's left edge, i > t),
// each by one thread of NT: `load` for U cells, then `use` for each with its place
// in a shared-memory row of the region. Threads run along x: along a front where
// fronts are rows, along the fronts where they are columns. A thread keeps one
// coordinate and steps the other over the range that the conditions leave.
template <int NT, int N, int TT, int U, class IN, class LOAD, class USE>
__device__ __forceinline__ void radial_visit(int n0, int n1, int i, int t, int di, int dt, int x, int y, int dx, int dy, int rs,
                                             LOAD load, USE use) {
  i += n0 * di;
  t += n0 * dt;
  x += n0 * dx;
  y += n0 * dy;
  int at = t * rs + i;
  const int da = dt * rs + di;
  for (int n = n0; n < n1; n += U) {
    IN in[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (n + u < n1) load(in[u], x + u * dx, y + u * dy);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (n + u < n1) use(in[u], x + u * dx, y + u * dy, at + u * da);
    x += U * dx;
    y += U * dy;
    at += U * da;
  }
}
template <int NT, int N, int TT, int U, class IN, class LOAD, class USE>
__device__ __forceinline__ void radial_cells(bool along_x, int f0, int nt, int l0, int above, int eq, int p0, int p1, int q0,
                                             int q1, int sx, int sy, int rs, LOAD load, USE use) {
  const int tid = (int)threadIdx.x;
  int i0, t0, di, dt, n0, n1;
  if (along_x) {
    i0 = tid % N;
    t0 = tid / N;
    di = 0;
    dt = NT / N;
    const int d1 = l0 + i0;
    const int ta = max(0, d1 - f0 - 1);                                        // first front that holds d1
    const int tb = d1 >= 0 && d1 <= eq ? (above ? min(nt, i0) : nt) : 0;       // end of the fronts
    n0 = ta > t0 ? (ta - t0 + dt - 1) / dt : 0;
    n1 = tb > t0 ? (tb - t0 + dt - 1) / dt : 0;
  } else {
    i0 = tid / TT;
    t0 = tid % TT;
    di = NT / TT;
    dt = 0;
    const int ia = max(above ? t0 + 1 : 0, -l0);
    const int ib = t0 < nt ? min(N, min(eq, f0 + 1 + t0) - l0 + 1) : 0;
    n0 = ia > i0 ? (ia - i0 + di - 1) / di : 0;
    n1 = ib > i0 ? (ib - i0 + di - 1) / di : 0;
  }
  const int d0 = f0 + 1 + t0, d1 = l0 + i0;
  radial_visit<NT, N, TT, U, IN>(n0, n1, i0, t0, di, dt, sx + p0 * d0 + q0 * d1, sy + p1 * d0 + q1 * d1, p0 * dt + q0 * di,
                                 p1 * dt + q1 * di, rs, load, use);
}

// The tiles of one radial scan (see the generator's radial_tiles_source). The
// scratch area at aux[3] (host: radial_tile_scratch), zero at the start: u32
// ticket, u64 abort at byte 8, and from byte 64 the last fronts' cells (radial_put),
// B per tile of every octant, strip and tile column. CTA 0 of the scan writes the
// observer's cell.
template <class OPS, class T, int B, int TT, class ARGS> __device__ __forceinline__ void radial_tiles(const ARGS &a, int cta) {
  constexpr int S = B + TT, V = S / 32, RS = S + 4, NT = RADIAL_NT, U = RADIAL_U;
  static_assert(S % 32 == 0 && TT % 32 == 0 && TT <= B && NT % S == 0 && NT % B == 0 && NT % TT == 0, "tile shape");
  static_assert(S * TT % (NT * U) == 0 && B * TT % (NT * U) == 0, "whole unrolled steps");
  extern __shared__ __align__(16) unsigned char radial_smem[];
  T *const s_in = (T *)radial_smem;
  __shared__ int s_dmax[8], s_eq[8], s_slot[9], s_job[4];
  const int tid = (int)threadIdx.x, lane = tid & 31;
  const int sx = (int)a.aux[0], sy = (int)a.aux[1], W = a.g.W, H = a.g.H;
  const long long lim = (long long)a.aux[2];
  u32 *const head = (u32 *)a.aux[3];
  if (tid < 8) {
    int p0, p1, q0, q1;
    octant_units(tid, p0, p1, q0, q1);
    const int ep = p0 > 0 ? W - 1 - sx : p0 < 0 ? sx : p1 > 0 ? H - 1 - sy : sy;
    s_eq[tid] = q0 > 0 ? W - 1 - sx : q0 < 0 ? sx : q1 > 0 ? H - 1 - sy : sy;
    s_dmax[tid] = (lim >= 0 && lim < ep) ? (int)lim : ep;
  }
  __syncthreads();
  if (tid == 0) {
    int at = 0;
    for (int o = 0; o < 8; ++o) {
      s_slot[o] = at;
      at += (s_dmax[o] + TT - 1) / TT * (s_eq[o] / B + 1);
    }
    s_slot[8] = at;
    if (cta == 0) {
      typename OPS::Cell in0;
      OPS::load(a, in0, sx, sy);
      OPS::post(a, in0, sx, sy, OPS::neutral());
    }
  }
  __syncthreads();
  u64 *const fronts = (u64 *)(head + 16);
  int strip = 0, before = 0;   // warp 0: the strip of the last claimed tile, the tiles of the strips above it
  for (;;) {
    if (tid < 32) {
      int ticket = 0;
      if (lane == 0) ticket = (int)atomicAdd(head, 1u);
      ticket = __shfl_sync(0xffffffffu, ticket, 0);
      int job = -1, k = 0;
      for (;;) {
        const int d0 = strip * TT;
        int n = 0, more = 0;
        if (lane < 8 && d0 < s_dmax[lane]) {
          const int dl = min(d0 + TT, s_dmax[lane]);
          n = min(dl, s_eq[lane]) / B + 1;
          more = 1;
        }
        if (!__any_sync(0xffffffffu, more)) break;
        int upto = n;
        for (int off = 1; off < 8; off <<= 1) {
          const int u = __shfl_up_sync(0xffffffffu, upto, off);
          if (lane >= off) upto += u;
        }
        const int total = __shfl_sync(0xffffffffu, upto, 7);
        if (ticket < before + total) {
          const u32 m = __ballot_sync(0xffffffffu, lane < 8 && ticket < before + upto);
          job = __ffs((int)m) - 1;
          k = ticket - before - __shfl_sync(0xffffffffu, upto - n, job);
          break;
        }
        before += total;
        ++strip;
      }
      if (lane == 0) {
        s_job[0] = job;
        s_job[1] = strip;
        s_job[2] = k;
        s_job[3] = 0;
      }
    }
    __syncthreads();
    const int o = s_job[0];
    if (o < 0) return;
    const int st = s_job[1], k = s_job[2];
    int p0, p1, q0, q1;
    octant_units(o, p0, p1, q0, q1);
    const int dmax = s_dmax[o], eq = s_eq[o], nk = eq / B + 1;
    const int f0 = st * TT;                      // the front before the strip's first
    const int nt = min(TT, dmax - f0);           // fronts of this strip
    const int lo = k * B - TT;                   // d1 of region cell 0
    // 1. arguments; region cell i of front f0 + 1 + t is needed from i = t + 1 on
    const bool along_x = q0 != 0;
    radial_cells<NT, S, TT, U, typename OPS::Cell>(
        along_x, f0, nt, lo, 1, eq, p0, p1, q0, q1, sx, sy, RS,
        [&](typename OPS::Cell &in, int x, int y) { OPS::load(a, in, x, y); },
        [&](const typename OPS::Cell &in, int x, int y, int at) { s_in[at] = OPS::arg(a, in, x, y); });
    __syncthreads();
    // 2. warp 0 sweeps the fronts
    if (tid < 32) {
      // the last front of the strip above, published cell by cell (radial_put): the
      // whole warp polls the cells it needs and stays converged for the sweep
      T val[V];
      const u64 *const above = fronts + (s64)(s_slot[o] + (st - 1) * nk) * B * RADIAL_WORDS(T);
      bool fail = false;
      if (st == 0) {
#pragma unroll
        for (int r = 0; r < V; ++r) val[r] = lo + V * lane + r == 0 ? OPS::neutral() : (T)0;
      } else {
        for (u32 n = 1;; ++n) {
          bool ok = true;
#pragma unroll
          for (int r = 0; r < V; ++r) {
            const int d1 = lo + V * lane + r;
            val[r] = (T)0;
            if (d1 >= 0 && d1 <= f0 && d1 <= eq) ok &= radial_get(above, d1, val[r]);
          }
          if (__all_sync(0xffffffffu, ok)) break;
          __nanosleep(RADIAL_PAUSE);
          if ((n & 255u) == 0 && __any_sync(0xffffffffu, n > RADIAL_POLLS || ld_relaxed_u64((const u64 *)(head + 2)) != 0)) {
            fail = true;
            break;
          }
        }
      }
      if (fail) {
        if (lane == 0) {
          st_relaxed_u64((u64 *)(head + 2), 1ull);
          skel_fail(a.err, ERR_SPIN_LIMIT);
          s_job[3] = 1;
        }
      } else {
        // cells with d1 = 0 (only a tile's own) or d1 = d0 read one neighbour: tiles
        // that hold none run without the two tests
        if (!radial_quot<T>(f0 + TT))
          radial_sweep<OPS, T, S, TT, true, false>(s_in, val, f0, nt, lo, lane);
        else if (k == 0 || (f0 + nt >= lo && f0 + 1 <= lo + S - 1))
          radial_sweep<OPS, T, S, TT, true, radial_has_quot<T>>(s_in, val, f0, nt, lo, lane);
        else
          radial_sweep<OPS, T, S, TT, false, radial_has_quot<T>>(s_in, val, f0, nt, lo, lane);
        const int last = min(f0 + nt, eq);
#pragma unroll
        for (int r = 0; r < V; ++r) {
          const int i = V * lane + r, d1 = lo + i;
          if (i >= TT && d1 <= last) radial_put(fronts + (s64)(s_slot[o] + st * nk) * B * RADIAL_WORDS(T), d1, val[r]);
        }
      }
    }
    __syncthreads();
    if (s_job[3]) return;
    // 3. the nodes after the scan, and the stores
    radial_cells<NT, B, TT, U, typename OPS::Cell>(
        along_x, f0, nt, lo + TT, 0, eq, p0, p1, q0, q1, sx, sy, RS,
        [&](typename OPS::Cell &in, int x, int y) { OPS::load(a, in, x, y); },
        [&](const typename OPS::Cell &in, int x, int y, int at) { OPS::post(a, in, x, y, s_in[at + TT]); });
    __syncthreads();
  }
}

// D8 code -> direction index (E, SE, S, SW, W, NW, N, NE), -1 when the code is
// not a single direction.
__device__ __forceinline__ int d8_index(u8 c) {
  if (c == 0 || (c & (c - 1)) != 0) return -1;
  return __ffs((int)c) - 1;
}
// x and y step of direction d, from two bits each (no table in memory)
__device__ __forceinline__ int d8_dx(int d) { return (int)((0x901Au >> (2 * d)) & 3u) - 1; }   // 1 1 0 -1 -1 -1 0 1
__device__ __forceinline__ int d8_dy(int d) { return (int)((0x01A9u >> (2 * d)) & 3u) - 1; }   // 0 1 1 1 0 -1 -1 -1

// Downstream cell of (x, y) along its D8 code, or -1.
__device__ __forceinline__ s64 d8_down(const RasterArg &dir, int W, int H, int x, int y) {
  int d = d8_index(ldr<u8>(dir, x, y));
  if (d < 0) return -1;
  int nx = x + d8_dx(d), ny = y + d8_dy(d);
  if (nx < 0 || ny < 0 || nx >= W || ny >= H) return -1;
  return (s64)ny * W + nx;
}

template <class T> __device__ __forceinline__ T ld_coherent(const RasterArg &r, int x, int y) {
  return __ldcg(row_ptr<T>(r, y) + x);
}
template <class T> __device__ __forceinline__ T *cell_ptr(const RasterArg &r, int x, int y) {
  return (T *)(r.p + (u64)(s64)y * (u64)r.pitch) + x;
}
// Decrements *p with acquire-release ordering at device scope (the caller's earlier
// writes are visible to whoever sees the result, and later reads see theirs);
// returns the previous value.
__device__ __forceinline__ s32 atomic_dec_acq_rel(s32 *p) {
  s32 old;
  asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], -1;" : "=r"(old) : "l"(p) : "memory");
  return old;
}
__device__ __forceinline__ void atomic_add_any(s32 *p, s32 v) { atomicAdd(p, v); }
__device__ __forceinline__ void atomic_add_any(u32 *p, u32 v) { atomicAdd(p, v); }
__device__ __forceinline__ void atomic_add_any(float *p, float v) { atomicAdd(p, v); }
__device__ __forceinline__ void atomic_add_any(double *p, double v) { atomicAdd(p, v); }
__device__ __forceinline__ void atomic_add_any(s64 *p, s64 v) { atomicAdd((unsigned long long *)p, (unsigned long long)v); }
__device__ __forceinline__ void atomic_add_any(u64 *p, u64 v) { atomicAdd((unsigned long long *)p, (unsigned long long)v); }
