// hashgrid.cu -- multi-resolution hash encoding (forward, deterministic backward).
//
// Replaces the tiny-cuda-nn HashGrid encoding the reference consumes at
// models/complex_inr.py:130-145 (called at :279 and :294): 2-D coordinates
// in [0,1] -> n_levels x F features.  Level l has scale
// s_l = base * per_level_scale^l - 1 and r_l = ceil(s_l) + 1 vertices per
// axis; a coordinate maps to x * s_l + 0.5, whose floor is the cell corner and
// whose fraction gives the bilinear weights.  A level whose r_l^2 (rounded up
// to a multiple of 8) fits in T = 2^log2_hashmap_size entries is indexed
// densely (ix + iy * r_l), otherwise by (ix * 1) ^ (iy * 2654435761) mod T.
// Level l's entries start at the sum of the previous levels' entry counts;
// each entry holds F = 2 floats (the table is [entries][2] float32).
//
// Backward: the coordinates of an INR are fixed, so the (entry, coordinate,
// weight) contributions are static.  ptycho_hashgrid_contrib emits them; the
// caller sorts them by entry once (stable) and passes the CSR to
// ptycho_hashgrid_backward, which gathers each entry's contributions in that
// fixed order -- a deterministic table-gradient "scatter" without atomics.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "common.cuh"

namespace pty {

constexpr int kMaxLevels = 32;
constexpr uint32_t kPrimeY = 2654435761u;

struct LevelTable {
  float scale[kMaxLevels];
  int res[kMaxLevels];
  int n[kMaxLevels];       // entries in the level
  int offset[kMaxLevels];  // first entry of the level
  int dense[kMaxLevels];
  int levels;
  int total;  // total entries
  int ndense; // levels 0 .. ndense - 1 are dense, the rest hashed (n = 2^log2_hashmap_size)
  int whole;  // every scale is below 2^20
};

static int make_levels(int n_levels, int log2_T, int base_res, float per_level_scale, LevelTable* L) {
  if (n_levels < 1 || n_levels > kMaxLevels || log2_T < 4 || log2_T > 26 || base_res < 1 ||
      !(per_level_scale >= 1.0f))
    return PTYCHO_ERR_INVALID_ARG;
  const long long T = 1ll << log2_T;
  long long off = 0;
  L->ndense = 0;
  L->whole = 1;
  for (int l = 0; l < n_levels; ++l) {
    const double scale = double(base_res) * pow(double(per_level_scale), double(l)) - 1.0;
    const long long res = (long long)ceil(scale) + 1;
    long long dn = res * res;
    dn = (dn + 7) / 8 * 8;
    const long long n = dn < T ? dn : T;
    L->scale[l] = (float)scale;
    L->res[l] = (int)res;
    L->n[l] = (int)n;
    L->offset[l] = (int)off;
    L->dense[l] = dn <= T;
    if (dn <= T) L->ndense = l + 1;  // res never falls with l
    if (!(scale < 1048576.0)) L->whole = 0;
    off += n;
  }
  L->levels = n_levels;
  L->total = (int)off;
  return off < (1ll << 31) ? PTYCHO_OK : PTYCHO_ERR_INVALID_ARG;
}

// entry of corner (cx, cy) of level l: index mod n_l.  A hashed level has
// n_l = 2^log2_hashmap_size (a mask); a dense level's index cx + cy*r is below
// n_l except for corners on the far edge, which take the modulo.
PTY_DEVI int corner_entry(const LevelTable& L, int l, int cx, int cy) {
  const uint32_t n = uint32_t(L.n[l]);
  uint32_t e;
  if (L.dense[l]) {
    e = uint32_t(cx) + uint32_t(cy) * uint32_t(L.res[l]);
    if (e >= n) e %= n;
  } else {
    e = uint32_t(cx) ^ (uint32_t(cy) * kPrimeY);
    e = (n & (n - 1)) == 0 ? (e & (n - 1)) : (e % n);
  }
  return L.offset[l] + int(e);
}

// the bilinear value from the four corners
PTY_DEVI float2 bilinear(float2 t00, float2 t10, float2 t01, float2 t11, float fx, float fy) {
  const float w00 = (1.f - fx) * (1.f - fy), w10 = fx * (1.f - fy), w01 = (1.f - fx) * fy, w11 = fx * fy;
  return make_float2(fmaf(w11, t11.x, fmaf(w01, t01.x, fmaf(w10, t10.x, w00 * t00.x))),
                     fmaf(w11, t11.y, fmaf(w01, t01.y, fmaf(w10, t10.y, w00 * t00.y))));
}

// floor and fraction of 0 <= p < 2^22 in two adds: p + 1.5 * 2^23 rounded down
// holds floor(p) in its last bits (floorf and the conversion to int would both
// run at a quarter of the rate)
PTY_DEVI int cell_of(float p, float& f) {
  const float t = __fadd_rd(p, 12582912.f);
  f = p - (t - 12582912.f);
  return __float_as_int(t) - 0x4B400000;
}

// Forward: one thread per coordinate, all levels, so the coordinate is read once
// and the corner gathers of a warp (adjacent coordinates) fall on neighbouring
// cells.  PLANAR writes features [2L][N] (every store coalesced), else [N][2L]
// (a thread's features contiguous).  Bound by instructions: with the floors by
// adds, the dense and hashed levels in loops of their own (one compare covers a
// dense cell's four corners, the modulo only where the last is past the level's
// end), 1024^2 coordinates and 16 levels take 51 us
// (57 with floorf and corner_entry; 134 MB of features, 2.6 TB/s; two or four
// coordinates per thread measured 3 and 15 us more).  The short loops hold for
// coordinates in [0, 1] and scales below 2^20; any other coordinate takes the
// general one, bitwise the same where both apply.
template <bool PLANAR>
__global__ void __launch_bounds__(256) k_hash_fwd(const float2* __restrict__ coords, int N,
                                                  const float2* __restrict__ table, const LevelTable L,
                                                  float* __restrict__ feat) {
  const int n = blockIdx.x * 256 + threadIdx.x;
  if (n >= N) return;
  const float2 x = __ldg(coords + n);
  float* out = PLANAR ? feat + n : feat + (size_t)n * (2 * L.levels);
  const size_t plane = size_t(N);
  auto put = [&](float2 o) {
    if constexpr (PLANAR) {
      out[0] = o.x;
      out[plane] = o.y;
      out += 2 * plane;
    } else {
      *reinterpret_cast<float2*>(out) = o;
      out += 2;
    }
  };
  if (L.whole && x.x >= 0.f && x.x <= 1.f && x.y >= 0.f && x.y <= 1.f) {
    int l = 0;
#pragma unroll 4
    for (; l < L.ndense; ++l) {
      const float s = L.scale[l];
      float fx, fy;
      const int ix = cell_of(fmaf(x.x, s, 0.5f), fx), iy = cell_of(fmaf(x.y, s, 0.5f), fy);
      const uint32_t n_l = uint32_t(L.n[l]), r = uint32_t(L.res[l]);
      uint32_t e00 = uint32_t(ix) + uint32_t(iy) * r, e10 = e00 + 1, e01 = e00 + r, e11 = e01 + 1;
      if (e11 >= n_l) {
        e00 %= n_l;
        e10 %= n_l;
        e01 %= n_l;
        e11 %= n_l;
      }
      const float2* T = table + L.offset[l];
      put(bilinear(__ldg(T + e00), __ldg(T + e10), __ldg(T + e01), __ldg(T + e11), fx, fy));
    }
#pragma unroll 4
    for (; l < L.levels; ++l) {
      const float s = L.scale[l];
      float fx, fy;
      const int ix = cell_of(fmaf(x.x, s, 0.5f), fx), iy = cell_of(fmaf(x.y, s, 0.5f), fy);
      const uint32_t m = uint32_t(L.n[l]) - 1, h0 = uint32_t(iy) * kPrimeY, h1 = h0 + kPrimeY;
      const uint32_t c0 = uint32_t(ix), c1 = c0 + 1;
      const float2* T = table + L.offset[l];
      put(bilinear(__ldg(T + ((c0 ^ h0) & m)), __ldg(T + ((c1 ^ h0) & m)), __ldg(T + ((c0 ^ h1) & m)),
                   __ldg(T + ((c1 ^ h1) & m)), fx, fy));
    }
    return;
  }
  for (int l = 0; l < L.levels; ++l) {
    const float s = L.scale[l];
    const float px = fmaf(x.x, s, 0.5f), py = fmaf(x.y, s, 0.5f);
    const float gx = floorf(px), gy = floorf(py);
    const int ix = int(gx), iy = int(gy);
    put(bilinear(__ldg(table + corner_entry(L, l, ix, iy)), __ldg(table + corner_entry(L, l, ix + 1, iy)),
                 __ldg(table + corner_entry(L, l, ix, iy + 1)), __ldg(table + corner_entry(L, l, ix + 1, iy + 1)),
                 px - gx, py - gy));
  }
}

// contributions: for coordinate n, level l, corner k -> key = entry,
// item = n * levels + l (feature pair index), weight
__global__ void __launch_bounds__(256) k_hash_contrib(const float2* __restrict__ coords, int N, const LevelTable L,
                                                      int* __restrict__ key, int* __restrict__ item,
                                                      float* __restrict__ weight) {
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= (long long)N * L.levels) return;
  const int n = int(i / L.levels), l = int(i - (long long)n * L.levels);
  const float2 x = __ldg(coords + n);
  const float s = L.scale[l];
  const float px = fmaf(x.x, s, 0.5f), py = fmaf(x.y, s, 0.5f);
  const float gx = floorf(px), gy = floorf(py);
  const float fx = px - gx, fy = py - gy;
  const int ix = int(gx), iy = int(gy);
  const long long base = i * 4;
  const int it = n * L.levels + l;
  key[base + 0] = corner_entry(L, l, ix, iy);
  key[base + 1] = corner_entry(L, l, ix + 1, iy);
  key[base + 2] = corner_entry(L, l, ix, iy + 1);
  key[base + 3] = corner_entry(L, l, ix + 1, iy + 1);
  weight[base + 0] = (1.f - fx) * (1.f - fy);
  weight[base + 1] = fx * (1.f - fy);
  weight[base + 2] = (1.f - fx) * fy;
  weight[base + 3] = fx * fy;
#pragma unroll
  for (int k = 0; k < 4; ++k) item[base + k] = it;
}

// segment starts from sorted keys: start[e] = first position with key >= e
__global__ void __launch_bounds__(256) k_seg_starts(const int* __restrict__ skey, long long K, int E,
                                                    int* __restrict__ start) {
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i > K) return;
  const int prev = i == 0 ? -1 : skey[i - 1];
  const int cur = i == K ? E : skey[i];
  for (int e = prev + 1; e <= cur; ++e) start[e] = int(i);
}

// feature gradient of a contribution: PLANAR = false -> item = n*L + l into
// [N][L] float2; PLANAR = true -> item = 2*l*N + n into feature-major [2L][N]
// floats (real part at item, imaginary part N further), which makes the
// gathers of one entry's spatially adjacent coordinates coalesced
template <bool PLANAR>
PTY_DEVI float2 dfeat_at(const float* __restrict__ dfeat, int item, int N) {
  if constexpr (PLANAR) return make_float2(__ldg(dfeat + item), __ldg(dfeat + item + N));
  else return __ldg(reinterpret_cast<const float2*>(dfeat) + item);
}

// long segments (coarse levels): a group of G lanes per entry (G = 32: one warp;
// G = 8: four entries per warp, for hashed levels' segments of 16 to 31), lanes stride the
// segment in order, fixed xor tree within the group.  Entries [e0, e1).
template <bool PLANAR, int G>
__global__ void __launch_bounds__(256) k_hash_bwd_warp(const int* __restrict__ start, const int* __restrict__ item,
                                                       const float* __restrict__ weight,
                                                       const float* __restrict__ dfeat, int N, int e0, int e1,
                                                       float2* __restrict__ dtable, int accumulate) {
  static_assert(G == 8 || G == 16 || G == 32, "lane group");
  const int lane = threadIdx.x & 31, gl = lane % G;
  const int e = e0 + (blockIdx.x * 8 + (threadIdx.x >> 5)) * (32 / G) + lane / G;
  const bool in = e < e1;  // every lane stays for the shuffles
  const int s0 = in ? start[e] : 0, s1 = in ? start[e + 1] : 0;
  float ax = 0.f, ay = 0.f;
  int j = s0 + gl;
  // four strides' loads in flight, then the adds in the same order as one at a time
  for (; j + 3 * G < s1; j += 4 * G) {
    float w[4];
    float2 g[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      w[k] = __ldg(weight + j + G * k);
      g[k] = dfeat_at<PLANAR>(dfeat, __ldg(item + j + G * k), N);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      ax = fmaf(w[k], g[k].x, ax);
      ay = fmaf(w[k], g[k].y, ay);
    }
  }
  for (; j < s1; j += G) {
    const float w = __ldg(weight + j);
    const float2 g = dfeat_at<PLANAR>(dfeat, __ldg(item + j), N);
    ax = fmaf(w, g.x, ax);
    ay = fmaf(w, g.y, ay);
  }
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
    ax += __shfl_xor_sync(0xffffffffu, ax, o);
    ay += __shfl_xor_sync(0xffffffffu, ay, o);
  }
  if (in && gl == 0) {
    float2 r = make_float2(ax, ay);
    if (accumulate) {
      const float2 old = dtable[e];
      r = make_float2(old.x + r.x, old.y + r.y);
    }
    dtable[e] = r;
  }
}

// short segments (fine levels): one thread per entry, sequential in order
template <bool PLANAR>
__global__ void __launch_bounds__(256) k_hash_bwd_thread(const int* __restrict__ start, const int* __restrict__ item,
                                                         const float* __restrict__ weight,
                                                         const float* __restrict__ dfeat, int N, int e0, int E,
                                                         float2* __restrict__ dtable, int accumulate) {
  const int e = e0 + blockIdx.x * 256 + threadIdx.x;
  if (e >= E) return;
  const int s0 = start[e], s1 = start[e + 1];
  float ax = 0.f, ay = 0.f;
  int j = s0;
  for (; j + 3 < s1; j += 4) {  // four items' loads in flight, adds in order
    float w[4];
    float2 g[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      w[k] = __ldg(weight + j + k);
      g[k] = dfeat_at<PLANAR>(dfeat, __ldg(item + j + k), N);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      ax = fmaf(w[k], g[k].x, ax);
      ay = fmaf(w[k], g[k].y, ay);
    }
  }
  for (; j < s1; ++j) {
    const float w = __ldg(weight + j);
    const float2 g = dfeat_at<PLANAR>(dfeat, __ldg(item + j), N);
    ax = fmaf(w, g.x, ax);
    ay = fmaf(w, g.y, ay);
  }
  float2 r = make_float2(ax, ay);
  if (accumulate) {
    const float2 old = dtable[e];
    r = make_float2(old.x + r.x, old.y + r.y);
  }
  dtable[e] = r;
}

// ---------------------------------------------------------------------------
// Grid backward.  When the coordinates are a tensor-product grid (coordinate
// n = i * Bj + j at (ax0[j], ax1[i]), both axes non-decreasing -- an INR's
// pixel centres), the contributors of one level's vertex (cx, cy) are the
// rectangle of coordinates with ix0[j] in {cx - 1, cx} and iy1[i] in
// {cy - 1, cy}: j in [lo0[cx - 1], lo0[cx + 1]), i in [lo1[cy - 1],
// lo1[cy + 1]).  Phase 1 sums each vertex's rectangle with the forward's
// bilinear weights (wx * wy, wx = 1 - fx on the cell's own corner, fx on the
// next) into G[vertex]; phase 2 sums, per table entry, the G of the vertices
// mapping to it (a hashed level's collisions, a dense level's far-edge
// aliases) in the order of the vertex list sorted by entry.  Both phases have
// fixed orders: deterministic, no atomics, and the only per-step state is
// the per-axis tables and one list entry per vertex (the host builds them,
// hashgrid.py GridPlan).
// ---------------------------------------------------------------------------
struct GridArgs {
  const int* iy1;
  const int* lo0;
  const int* lo1;
  const int* vstart;
  const int* vorder;
  const float* fx0;
  const float* fy1;
  const float* dfeat;
  int planar;
  int N, A, Bj, L;
  int E0[kMaxLevels], E1[kMaxLevels];
  int cw0[kMaxLevels], cw1[kMaxLevels];  // most axis values in one cell
  int lo0off[kMaxLevels], lo1off[kMaxLevels];
  long long voff[kMaxLevels + 1];
  float2* G;
  // the coarse levels (k = 0 .. nsep-1): level, columns of a block, cells of a
  // row slot, column blocks, lanes of the row pass, offset of the level's columns
  // in H0 / H1, first block of each pass
  int nsep;
  int sep_l[kMaxLevels], sep_cb[kMaxLevels], sep_kc[kMaxLevels], sep_nx[kMaxLevels], sep_g[kMaxLevels];
  long long sep_h[kMaxLevels];
  int sep_b1[kMaxLevels + 1], sep_b2[kMaxLevels + 1];
  // the fine levels: level, vertex columns of a tile, tiles per row, first block
  int nfine;
  int fine_l[kMaxLevels], fine_kx[kMaxLevels], fine_gx[kMaxLevels];
  int fine_b[kMaxLevels + 1];
  float2 *H0, *H1;  // column sums of the coarse levels, [cells][Bj] per level
};

// gradient value n of a level: re and im planes of [2L][N], or a pair of [N][2L]
struct LevelGrad {
  const float* p;
  size_t im;  // imaginary part's distance
  size_t es;  // element stride
};
PTY_DEVI LevelGrad level_grad(const GridArgs& g, int l) {
  LevelGrad r;
  r.p = g.dfeat + (g.planar ? size_t(2 * l) * g.N : size_t(2 * l));
  r.im = g.planar ? size_t(g.N) : 1;
  r.es = g.planar ? 1 : size_t(2 * g.L);
  return r;
}

// the slot of block b among levels whose blocks start at `first`
PTY_DEVI int level_slot(int n, const int* first, int b) {
  int k = 0;
  while (k + 1 < n && b >= first[k + 1]) ++k;
  return k;
}

// Both kinds of level sum along the columns first: a thread owns a column j of
// the grid and runs down the rows of a cell, C0 = sum (1 - fy) g and C1 = sum
// fy g (a term's weight is wx(j, cx) * wy(i, cy)), so adjacent threads read
// adjacent values, every value is read once and costs two loads and four FMAs.
// Bound by instructions and load latency.  (Rows first, with lanes sharing a cell,
// took 116 instructions per value, and a sum per vertex from a staged rectangle 240;
// these take about 50 and 80: the backward of 1024^2 coordinates and 16 levels 118 ->
// 80 us.)

// C0 and C1 of one column
struct ColumnSum {
  float2 c0 = make_float2(0.f, 0.f), c1 = make_float2(0.f, 0.f);
  PTY_DEVI void add(float w, float re, float im) {
    const float v = 1.f - w;
    c0.x = fmaf(v, re, c0.x);
    c0.y = fmaf(v, im, c0.y);
    c1.x = fmaf(w, re, c1.x);
    c1.y = fmaf(w, im, c1.y);
  }
};

// R rows of a column from row i, the loads in flight together; then use(row, re,
// im) in row order.  Fewer than R where the rows end at i1.
template <int R, bool ALL, class F>
PTY_DEVI void column_batch(const float*& p, size_t im_off, size_t rs, int i, int i1, F& use) {
  float re[R], im[R];
#pragma unroll
  for (int u = 0; u < R; ++u) {
    re[u] = im[u] = 0.f;
    if (ALL || i + u < i1) {
      re[u] = __ldg(p);
      im[u] = __ldg(p + im_off);
    }
    p += rs;
  }
#pragma unroll
  for (int u = 0; u < R; ++u)
    if (ALL || i + u < i1) use(i + u, re[u], im[u]);
}

// rows [i, i1) of a column
template <class F>
PTY_DEVI void column_rows(const float* p, size_t im_off, size_t rs, int i, int i1, F use) {
  for (; i + 8 <= i1; i += 8) column_batch<8, true>(p, im_off, rs, i, i1, use);
  if (i + 4 <= i1) {
    column_batch<4, true>(p, im_off, rs, i, i1, use);
    i += 4;
  }
  if (i < i1) column_batch<3, false>(p, im_off, rs, i, i1, use);
}

// Coarse levels, column pass: C0 and C1 of every (cell row, column) into H0, H1.
// A block holds CB columns (a power of two) x 256 / CB row slots.  Cells shorter
// than kShared rows: a slot runs down kc cells.  Longer ones: the slots share one
// cell and are added by a fixed tree.  Empty cells are neither written nor
// read; where there are more cells than rows, an occupied cell's row in H0 and H1
// is the number of its first grid row, so that they never outgrow the grid.
constexpr int kShared = 32;

PTY_DEVI size_t sep_row(const GridArgs& g, int l, int c, int first_row) {
  return size_t(g.E1[l] > g.A ? first_row : c) * g.Bj;
}

__global__ void __launch_bounds__(256) k_gsep_cols(const GridArgs g) {
  __shared__ float4 part[256];
  const int b = blockIdx.x;
  const int k = level_slot(g.nsep, g.sep_b1, b);
  const int l = g.sep_l[k], CB = g.sep_cb[k], RS = 256 / CB;
  const int bl = b - g.sep_b1[k], nx = g.sep_nx[k], by = bl / nx, bx = bl - by * nx;
  const int t = threadIdx.x, r = t / CB, j = bx * CB + (t & (CB - 1));
  const bool in = j < g.Bj;
  const int* lo1 = g.lo1 + g.lo1off[l];
  const float* fy = g.fy1 + size_t(l) * g.A;
  const LevelGrad d = level_grad(g, l);
  const size_t rs = size_t(g.Bj) * d.es;
  float2* h0 = g.H0 + g.sep_h[k] + j;
  float2* h1 = g.H1 + g.sep_h[k] + j;
  ColumnSum s;
  if (g.cw1[l] < kShared) {
    int c = (by * RS + r) * g.sep_kc[k];
    const int c_end = min(c + g.sep_kc[k], g.E1[l]);
    if (!in || c >= c_end) return;
    const int i0 = lo1[c];
    int first = i0, next = lo1[c + 1];  // cell c's rows
    auto close = [&]() {
      if (first < next) {
        const size_t h = sep_row(g, l, c, first);
        h0[h] = s.c0;
        h1[h] = s.c1;
        s = ColumnSum();
      }
      first = next;
      if (++c < c_end) next = lo1[c + 1];
    };
    column_rows(d.p + (size_t(i0) * g.Bj + j) * d.es, d.im, rs, i0, lo1[c_end], [&](int i, float re, float im) {
      while (i >= next) close();  // i < lo1[c_end], so c stays below c_end
      s.add(__ldg(fy + i), re, im);
    });
    while (c < c_end) close();
    return;
  }
  const int c = by, i0 = lo1[c], n = lo1[c + 1] - i0, m = (n + RS - 1) / RS;
  const int ia = i0 + min(r * m, n), ib = i0 + min((r + 1) * m, n);
  if (in)
    column_rows(d.p + (size_t(ia) * g.Bj + j) * d.es, d.im, rs, ia, ib,
                [&](int i, float re, float im) { s.add(__ldg(fy + i), re, im); });
  part[t] = make_float4(s.c0.x, s.c0.y, s.c1.x, s.c1.y);
  __syncthreads();
  for (int o = 128; o >= CB; o >>= 1) {
    if (t < o) {
      const float4 a = part[t], q = part[t + o];
      part[t] = make_float4(a.x + q.x, a.y + q.y, a.z + q.z, a.w + q.w);
    }
    __syncthreads();
  }
  if (in && r == 0 && n > 0) {
    const float4 a = part[t];
    const size_t h = sep_row(g, l, c, i0);
    h0[h] = make_float2(a.x, a.y);
    h1[h] = make_float2(a.z, a.w);
  }
}

// Coarse levels, row pass: G[cy][cx] = sum over the columns of cells cx - 1 and
// cx of wx (C1 of cell row cy - 1 + C0 of cell row cy); lanes share a vertex.
__global__ void __launch_bounds__(256) k_gsep_rows(const GridArgs g) {
  const int b = blockIdx.x;
  const int k = level_slot(g.nsep, g.sep_b2, b);
  const int l = g.sep_l[k], G = g.sep_g[k];
  const int t = threadIdx.x, gl = t & (G - 1);
  // 32-bit index math (vertices < 2^31; G is a power of two)
  const unsigned item = unsigned(b - g.sep_b2[k]) * unsigned(256 / G) + (unsigned(t) >> (__ffs(G) - 1));
  const int E0 = g.E0[l], E1 = g.E1[l];
  const bool in = item < unsigned(E0) * unsigned(E1);
  float ax = 0.f, ay = 0.f;
  if (in) {
    const int cy = int(item / unsigned(E0)), cx = int(item - unsigned(cy) * unsigned(E0));
    const int* lo0 = g.lo0 + g.lo0off[l];
    const int j1 = lo0[cx + 1];
    const float* fx0 = g.fx0 + size_t(l) * g.Bj;
    const int jm = lo0[cx];  // first column of cell cx: weight fx before it, 1 - fx from it
    const int* lo1 = g.lo1 + g.lo1off[l];
    const int ra = lo1[max(cy - 1, 0)], rb = lo1[cy];
    const bool own = rb < lo1[cy + 1], above = ra < rb;  // cells cy and cy - 1 hold rows
    const float2* h0 = g.H0 + g.sep_h[k] + (own ? sep_row(g, l, cy, rb) : 0);
    const float2* h1 = g.H1 + g.sep_h[k] + (above ? sep_row(g, l, cy - 1, ra) : 0);
    const float2 none = make_float2(0.f, 0.f);
    int j = lo0[max(cx - 1, 0)] + gl;
    for (; j + 3 * G < j1; j += 4 * G) {
      float w[4];
      float2 a[4], q[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float f = __ldg(fx0 + j + u * G);
        w[u] = j + u * G < jm ? f : 1.f - f;
        a[u] = own ? h0[j + u * G] : none;
        q[u] = above ? h1[j + u * G] : none;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        ax = fmaf(w[u], q[u].x + a[u].x, ax);
        ay = fmaf(w[u], q[u].y + a[u].y, ay);
      }
    }
    for (; j < j1; j += G) {
      const float f = __ldg(fx0 + j), w = j < jm ? f : 1.f - f;
      const float2 a = own ? h0[j] : none, q = above ? h1[j] : none;
      ax = fmaf(w, q.x + a.x, ax);
      ay = fmaf(w, q.y + a.y, ay);
    }
  }
  for (int o = G >> 1; o > 0; o >>= 1) {
    ax += __shfl_xor_sync(0xffffffffu, ax, o);
    ay += __shfl_xor_sync(0xffffffffu, ay, o);
  }
  if (in && gl == 0) g.G[g.voff[l] + item] = make_float2(ax, ay);
}

// lanes for a sum of about n terms: the power of two nearest n / 4 in 1 .. 32
static int lanes_for_terms(double n) {
  int G = 1;
  while (G < 32 && 8.0 * G <= n) G *= 2;
  return G;
}

// Fine levels: one block per kx x kFY vertices, all such levels in one launch
// (blocks by level).  The block's threads own the columns that its vertices
// touch and run down the rows of cells cy0 - 1 .. cy0 + kFY - 1; a finished cell
// gives vertex row cy its column sums V = C1(cy - 1) + C0(cy) in shared memory.
// Then a thread per vertex column sums wx V for all kFY rows.  The halo is one
// cell row per kFY and one cell column per tile.
constexpr int kFY = 8;
constexpr int kFineCell = 32;  // most axis values in a fine level's cell

__global__ void __launch_bounds__(256) k_gfine(const GridArgs g) {
  __shared__ float2 V[kFY][256];
  __shared__ float sfx[256];
  __shared__ float2 sy[(kFY + 1) * kFineCell];  // a row's cell (as bits) and fraction
  const int b = blockIdx.x;
  const int k = level_slot(g.nfine, g.fine_b, b);
  const int l = g.fine_l[k], kx = g.fine_kx[k];
  const int bl = b - g.fine_b[k], by = bl / g.fine_gx[k], bx = bl - by * g.fine_gx[k];
  const int E0 = g.E0[l], E1 = g.E1[l];
  const int cx0 = bx * kx, cy0 = by * kFY, cx1 = min(cx0 + kx, E0), cy1 = min(cy0 + kFY, E1);
  const int* lo0 = g.lo0 + g.lo0off[l];
  const int* lo1 = g.lo1 + g.lo1off[l];
  const int j_lo = lo0[max(cx0 - 1, 0)], nc = min(lo0[cx1] - j_lo, 256);
  const int i_lo = lo1[max(cy0 - 1, 0)], nr = min(lo1[cy1] - i_lo, (kFY + 1) * kFineCell);
  const int t = threadIdx.x;
  for (int q = t; q < nr; q += 256) {
    sy[q] = make_float2(__int_as_float(__ldg(g.iy1 + size_t(l) * g.A + i_lo + q)),
                        __ldg(g.fy1 + size_t(l) * g.A + i_lo + q));
  }
  if (t < nc) sfx[t] = __ldg(g.fx0 + size_t(l) * g.Bj + j_lo + t);
  __syncthreads();
  if (t < nc) {
    const LevelGrad d = level_grad(g, l);
    const float* p = d.p + (size_t(i_lo) * g.Bj + j_lo + t) * d.es;
    const size_t rs = size_t(g.Bj) * d.es;
    ColumnSum s;
    float2 up = make_float2(0.f, 0.f);
    int c = max(cy0 - 1, 0);
    auto close = [&]() {  // cell row c is complete
      if (c >= cy0) V[c - cy0][t] = make_float2(up.x + s.c0.x, up.y + s.c0.y);
      up = s.c1;
      s = ColumnSum();
      ++c;
    };
    column_rows(p, d.im, rs, 0, nr, [&](int i, float re, float im) {
      const float2 y = sy[i];
      const int ci = min(__float_as_int(y.x), cy1 - 1);
      while (c < ci) close();
      s.add(y.y, re, im);
    });
    while (c < cy1) close();
  }
  __syncthreads();
  const int cx = cx0 + t;
  if (cx >= cx1) return;
  float2 a[kFY];
#pragma unroll
  for (int q = 0; q < kFY; ++q) a[q] = make_float2(0.f, 0.f);
  const int jm = lo0[cx] - j_lo, j1 = min(lo0[cx + 1] - j_lo, nc);
  for (int j = lo0[max(cx - 1, 0)] - j_lo; j < j1; ++j) {
    const float f = sfx[j], w = j < jm ? f : 1.f - f;
#pragma unroll
    for (int q = 0; q < kFY; ++q) {
      const float2 v = V[q][j];
      a[q].x = fmaf(w, v.x, a[q].x);
      a[q].y = fmaf(w, v.y, a[q].y);
    }
  }
  float2* G = g.G + g.voff[l] + (long long)cy0 * E0 + cx;
#pragma unroll
  for (int q = 0; q < kFY; ++q)
    if (cy0 + q < cy1) G[(long long)q * E0] = a[q];
}

// A level takes the two passes when its cells hold at least kSepTerms values or
// are too long for a fine tile's tables.  1024^2 coordinates, 16 levels, forward and
// backward: 140, 135.5 and 135.4 us with the line at 16, 36 and 64 values; 900 x 1000:
// 124, 119 and 121
constexpr int kSepTerms = 36;
constexpr int kSepRows = 16;  // rows of a row slot in the coarse levels' column pass
static bool separable_level(const int32_t* extents, int l) {
  const int32_t cw0 = extents[4 * l + 2], cw1 = extents[4 * l + 3];
  return cw0 > kFineCell || cw1 > kFineCell || cw0 * cw1 >= kSepTerms;
}

// per table entry: the G of its vertices, in vertex-list order (four entries per
// thread: 18.7 against 14.3 us, fewer warps for the gathers)
__global__ void __launch_bounds__(256) k_gentry(const int* __restrict__ vstart, const int* __restrict__ vorder,
                                                const float2* __restrict__ G, int E, float2* __restrict__ dtable,
                                                int accumulate) {
  const int e = blockIdx.x * 256 + threadIdx.x;
  if (e >= E) return;
  const int s0 = __ldg(vstart + e), s1 = __ldg(vstart + e + 1);
  float2 r = make_float2(0.f, 0.f);
  for (int k = s0; k < s1; ++k) r = c_add(r, G[__ldg(vorder + k)]);
  if (accumulate) r = c_add(dtable[e], r);
  dtable[e] = r;
}

}  // namespace pty

using namespace pty;

extern "C" {

int ptycho_hashgrid_entries(int n_levels, int log2_hashmap_size, int base_resolution, float per_level_scale) {
  LevelTable L;
  if (make_levels(n_levels, log2_hashmap_size, base_resolution, per_level_scale, &L)) return -1;
  return L.total;
}

int ptycho_hashgrid_forward(const float* coords, int N, const float* table, int n_levels,
                            int log2_hashmap_size, int base_resolution, float per_level_scale,
                            float* features, ptycho_stream_t stream) {
  LevelTable L;
  int st = make_levels(n_levels, log2_hashmap_size, base_resolution, per_level_scale, &L);
  if (st) return st;
  if (N < 0 || (N > 0 && (!coords || !table || !features))) return PTYCHO_ERR_INVALID_ARG;
  if (!pty_aligned(coords, 8) || !pty_aligned(table, 8) || !pty_aligned(features, 8))
    return PTYCHO_ERR_MISALIGNED;
  if (N == 0) return PTYCHO_OK;
  k_hash_fwd<false><<<(unsigned)((N + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const float2*>(coords), N, reinterpret_cast<const float2*>(table), L, features);
  return cudaGetLastError() == cudaSuccess ? PTYCHO_OK : PTYCHO_ERR_LAUNCH;
}

int ptycho_hashgrid_forward_planar(const float* coords, int N, const float* table, int n_levels,
                                   int log2_hashmap_size, int base_resolution, float per_level_scale,
                                   float* features_planar, ptycho_stream_t stream) {
  LevelTable L;
  int st = make_levels(n_levels, log2_hashmap_size, base_resolution, per_level_scale, &L);
  if (st) return st;
  if (N < 0 || (N > 0 && (!coords || !table || !features_planar))) return PTYCHO_ERR_INVALID_ARG;
  if (!pty_aligned(coords, 8) || !pty_aligned(table, 8) || !pty_aligned(features_planar, 4))
    return PTYCHO_ERR_MISALIGNED;
  if (N == 0) return PTYCHO_OK;
  k_hash_fwd<true><<<(unsigned)((N + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const float2*>(coords), N, reinterpret_cast<const float2*>(table), L, features_planar);
  return cudaGetLastError() == cudaSuccess ? PTYCHO_OK : PTYCHO_ERR_LAUNCH;
}

int ptycho_hashgrid_contrib(const float* coords, int N, int n_levels, int log2_hashmap_size,
                            int base_resolution, float per_level_scale, int32_t* key, int32_t* item,
                            float* weight, ptycho_stream_t stream) {
  LevelTable L;
  int st = make_levels(n_levels, log2_hashmap_size, base_resolution, per_level_scale, &L);
  if (st) return st;
  if (N < 0 || (N > 0 && (!coords || !key || !item || !weight))) return PTYCHO_ERR_INVALID_ARG;
  if ((long long)N * n_levels * 4 >= (1ll << 31)) return PTYCHO_ERR_UNSUPPORTED_SIZE;
  if (N == 0) return PTYCHO_OK;
  const long long work = (long long)N * n_levels;
  k_hash_contrib<<<(unsigned)((work + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const float2*>(coords), N, L, key, item, weight);
  return cudaGetLastError() == cudaSuccess ? PTYCHO_OK : PTYCHO_ERR_LAUNCH;
}

int ptycho_hashgrid_segments(const int32_t* sorted_key, long long K, int n_entries, int32_t* start,
                             ptycho_stream_t stream) {
  if (K < 0 || n_entries < 1 || !start || (K > 0 && !sorted_key)) return PTYCHO_ERR_INVALID_ARG;
  k_seg_starts<<<(unsigned)((K + 1 + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      sorted_key, K, n_entries, start);
  return cudaGetLastError() == cudaSuccess ? PTYCHO_OK : PTYCHO_ERR_LAUNCH;
}

static int hash_backward(bool planar, const int32_t* start, const int32_t* item, const float* weight,
                         const float* dfeatures, int N, int n_levels, int log2_hashmap_size, int base_resolution,
                         float per_level_scale, float* dtable, int accumulate, ptycho_stream_t stream) {
  LevelTable L;
  int st = make_levels(n_levels, log2_hashmap_size, base_resolution, per_level_scale, &L);
  if (st) return st;
  if (N < 0 || !start || !item || !weight || !dfeatures || !dtable) return PTYCHO_ERR_INVALID_ARG;
  if (!pty_aligned(dfeatures, planar ? 4 : 8) || !pty_aligned(dtable, 8)) return PTYCHO_ERR_MISALIGNED;
  // by average segment length 4N / n_l (levels run coarse to fine, so each rule
  // holds for a prefix): >= 32, or >= 16 on a dense level, a warp per entry;
  // >= 16 on a hashed level eight lanes per entry; shorter a thread per entry
  // (measured: eight lanes gained on 2^20-entry hashed levels with segments of
  // 16 and lost on dense levels with segments of 16 to 31)
  int split32 = 0, split = 0;
  for (int l = 0; l < L.levels; ++l) {
    const long long seg4 = (long long)N * 4;
    if (seg4 >= 32ll * L.n[l] || (L.dense[l] && seg4 >= 16ll * L.n[l])) split32 = L.offset[l] + L.n[l];
    if ((long long)N * 4 >= 16ll * L.n[l]) split = L.offset[l] + L.n[l];
  }
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  float2* dt = reinterpret_cast<float2*>(dtable);
  if (split32 > 0) {
    const unsigned g = unsigned((split32 + 7) / 8);
    if (planar)
      k_hash_bwd_warp<true, 32><<<g, 256, 0, s>>>(start, item, weight, dfeatures, N, 0, split32, dt, accumulate);
    else
      k_hash_bwd_warp<false, 32><<<g, 256, 0, s>>>(start, item, weight, dfeatures, N, 0, split32, dt, accumulate);
  }
  if (split > split32) {
    const unsigned g = unsigned((split - split32 + 31) / 32);  // 8 warps x 4 entries per block
    if (planar)
      k_hash_bwd_warp<true, 8><<<g, 256, 0, s>>>(start, item, weight, dfeatures, N, split32, split, dt, accumulate);
    else
      k_hash_bwd_warp<false, 8><<<g, 256, 0, s>>>(start, item, weight, dfeatures, N, split32, split, dt, accumulate);
  }
  if (L.total > split) {
    const unsigned g = (L.total - split + 255) / 256;
    if (planar)
      k_hash_bwd_thread<true><<<g, 256, 0, s>>>(start, item, weight, dfeatures, N, split, L.total, dt, accumulate);
    else
      k_hash_bwd_thread<false><<<g, 256, 0, s>>>(start, item, weight, dfeatures, N, split, L.total, dt, accumulate);
  }
  return cudaGetLastError() == cudaSuccess ? PTYCHO_OK : PTYCHO_ERR_LAUNCH;
}

int ptycho_hashgrid_backward(const int32_t* start, const int32_t* item, const float* weight,
                             const float* dfeatures, int N, int n_levels, int log2_hashmap_size,
                             int base_resolution, float per_level_scale, float* dtable, int accumulate,
                             ptycho_stream_t stream) {
  return hash_backward(false, start, item, weight, dfeatures, N, n_levels, log2_hashmap_size, base_resolution,
                       per_level_scale, dtable, accumulate, stream);
}

int ptycho_hashgrid_backward_planar(const int32_t* start, const int32_t* item_planar, const float* weight,
                                    const float* dfeatures_planar, int N, int n_levels, int log2_hashmap_size,
                                    int base_resolution, float per_level_scale, float* dtable, int accumulate,
                                    ptycho_stream_t stream) {
  if ((long long)2 * n_levels * N > 0x7fffffffll) return PTYCHO_ERR_UNSUPPORTED_SIZE;
  return hash_backward(true, start, item_planar, weight, dfeatures_planar, N, n_levels, log2_hashmap_size,
                       base_resolution, per_level_scale, dtable, accumulate, stream);
}

size_t ptycho_hashgrid_grid_scratch_size(const int32_t* extents, int n_levels, int A, int Bj) {
  if (!extents || n_levels < 1 || n_levels > kMaxLevels || A < 1 || Bj < 1) return 0;
  size_t n = 0, h = 0;
  for (int l = 0; l < n_levels; ++l) {
    if (extents[4 * l] < 1 || extents[4 * l + 1] < 1 || extents[4 * l + 2] < 1 || extents[4 * l + 3] < 1) return 0;
    n += size_t(extents[4 * l]) * size_t(extents[4 * l + 1]);
    if (separable_level(extents, l)) h += size_t(Bj) * size_t(extents[4 * l + 1] < A ? extents[4 * l + 1] : A);
  }
  // vertex sums, then every coarse level's column sums C0 and C1
  return (n + 2 * h) * sizeof(float2);
}

int ptycho_hashgrid_backward_grid(const int32_t* grid_int, const float* grid_frac, const int32_t* extents, int A,
                                  int Bj, const float* dfeatures, int planar, int n_levels, int log2_hashmap_size,
                                  int base_resolution, float per_level_scale, float* dtable, int accumulate,
                                  void* scratch, size_t scratch_bytes, ptycho_stream_t stream) {
  LevelTable L;
  int st = make_levels(n_levels, log2_hashmap_size, base_resolution, per_level_scale, &L);
  if (st) return st;
  if (!grid_int || !grid_frac || !extents || !dfeatures || !dtable || A < 1 || Bj < 1) return PTYCHO_ERR_INVALID_ARG;
  const long long N = (long long)A * Bj;
  if (N * 4 >= (1ll << 31) || (planar && 2ll * n_levels * N >= (1ll << 31))) return PTYCHO_ERR_UNSUPPORTED_SIZE;
  const size_t need = ptycho_hashgrid_grid_scratch_size(extents, n_levels, A, Bj);
  if (need == 0) return PTYCHO_ERR_INVALID_ARG;
  if (!scratch || scratch_bytes < need) return PTYCHO_ERR_WORKSPACE;
  if (!pty_aligned(dfeatures, planar ? 4 : 8) || !pty_aligned(dtable, 8) || !pty_aligned(scratch, 8) ||
      !pty_aligned(grid_int, 4) || !pty_aligned(grid_frac, 4))
    return PTYCHO_ERR_MISALIGNED;
  GridArgs g{};
  g.dfeat = dfeatures;
  g.planar = planar ? 1 : 0;
  g.N = int(N);
  g.A = A;
  g.Bj = Bj;
  g.L = n_levels;
  // layout of grid_int: ix0 [L][Bj], iy1 [L][A], lo0 [sum (E0 + 1)], lo1 [sum (E1 + 1)],
  // vstart [entries + 1], vorder [vertices]; grid_frac: fx0 [L][Bj], fy1 [L][A]
  size_t off = 0;
  off += size_t(n_levels) * Bj;  // (ix0: no kernel reads it)
  g.iy1 = grid_int + off;
  off += size_t(n_levels) * A;
  g.lo0 = grid_int + off;
  int o0 = 0, o1 = 0;
  long long nv = 0;
  for (int l = 0; l < n_levels; ++l) {
    g.E0[l] = extents[4 * l];
    g.E1[l] = extents[4 * l + 1];
    g.cw0[l] = extents[4 * l + 2];
    g.cw1[l] = extents[4 * l + 3];
    g.lo0off[l] = o0;
    g.lo1off[l] = o1;
    o0 += g.E0[l] + 1;
    o1 += g.E1[l] + 1;
    g.voff[l] = nv;
    nv += (long long)g.E0[l] * g.E1[l];
  }
  g.voff[n_levels] = nv;
  off += size_t(o0);
  g.lo1 = grid_int + off;
  off += size_t(o1);
  g.vstart = grid_int + off;
  off += size_t(L.total) + 1;
  g.vorder = grid_int + off;
  g.fx0 = grid_frac;
  g.fy1 = grid_frac + size_t(n_levels) * Bj;
  g.G = static_cast<float2*>(scratch);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  // plan the levels: the coarse ones take two launches for all of them, the fine
  // ones one
  long long hoff = 0, b1 = 0, b2 = 0, tb = 0;
  for (int l = 0; l < n_levels; ++l) {
    const int cw0 = g.cw0[l], cw1 = g.cw1[l];
    if (separable_level(extents, l)) {
      const int k = g.nsep++;
      g.sep_l[k] = l;
      // columns of a block: the grid's, at most 256, and fewer where the slots share
      // a cell, so that a thread adds about 16 rows
      int CB = 256;
      while (CB > 1 && (CB / 2 >= Bj || (CB > 32 && cw1 >= kShared && cw1 >= 32 * (256 / CB)))) CB /= 2;
      const int RS = 256 / CB;
      g.sep_cb[k] = CB;
      g.sep_kc[k] = cw1 >= kShared ? 1 : (kSepRows + cw1 - 1) / cw1;
      const int cells = cw1 >= kShared ? 1 : g.sep_kc[k] * RS;  // of a block
      g.sep_nx[k] = (Bj + CB - 1) / CB;
      g.sep_g[k] = lanes_for_terms(2.0 * Bj / g.E0[l]);
      g.sep_h[k] = hoff;
      hoff += (long long)(g.E1[l] < A ? g.E1[l] : A) * Bj;
      g.sep_b1[k] = int(b1);
      b1 += (long long)g.sep_nx[k] * ((g.E1[l] + cells - 1) / cells);
      g.sep_b2[k] = int(b2);
      b2 += ((long long)g.E0[l] * g.E1[l] * g.sep_g[k] + 255) / 256;
    } else {
      const int k = g.nfine++;
      const int most = 256 / cw0 - 1;  // kx + 1 cells' columns fit the block
      g.fine_l[k] = l;
      g.fine_gx[k] = (g.E0[l] + most - 1) / most;
      g.fine_kx[k] = (g.E0[l] + g.fine_gx[k] - 1) / g.fine_gx[k];
      g.fine_b[k] = int(tb);
      tb += (long long)g.fine_gx[k] * ((g.E1[l] + kFY - 1) / kFY);
    }
  }
  g.H0 = g.G + g.voff[n_levels];
  g.H1 = g.H0 + hoff;
  if (b1 >= (1ll << 31) || b2 >= (1ll << 31) || tb >= (1ll << 31)) return PTYCHO_ERR_UNSUPPORTED_SIZE;
  if (g.nsep) {
    k_gsep_cols<<<unsigned(b1), 256, 0, s>>>(g);
    k_gsep_rows<<<unsigned(b2), 256, 0, s>>>(g);
  }
  if (g.nfine) k_gfine<<<unsigned(tb), 256, 0, s>>>(g);
  k_gentry<<<unsigned((L.total + 255) / 256), 256, 0, s>>>(g.vstart, g.vorder, g.G, L.total,
                                                           reinterpret_cast<float2*>(dtable), accumulate);
  return cudaGetLastError() == cudaSuccess ? PTYCHO_OK : PTYCHO_ERR_LAUNCH;
}

}  // extern "C"
