// lines.cuh -- batched DFTs of any length along lines held in shared memory.
//
// Smooth lengths run as Stockham passes of register butterflies, radix 2 to 16
// (dft_small.cuh), planned on the host for the fewest passes: 192 = 16 x 12, 1500 =
// 15 x 10 x 10.  A length with a larger prime factor runs as Bluestein's
// convolution of smooth length m >= 2n - 1 (two transforms of length m and three
// diagonals; a 317-point line costs about two 640-point ones, where a direct sum
// over the factor 317 costs 317 terms a value), or, when its tables do not fit
// shared memory (n beyond about 2500), with direct-sum passes for the large primes.
//
// A CTA holds `lines` lines in two ping-pong buffers; the inverse transform is
// conj(DFT(conj)), so only forward passes exist.  Twiddles are
// tables in shared memory built per CTA, in FP64 and rounded once (cis_ratio below;
// with sincospi they took a third of the short kernels).  Index
// divisions are multiplications by reciprocals from the plan.
#pragma once
#include "common.cuh"
#include "dft_small.cuh"

namespace pty {
namespace ln {

constexpr int kMaxPasses = 8;
constexpr int kMaxLen = 8192;
constexpr size_t kSmemCap = 200 * 1024;

struct Pass {
  int R, NS, bpl, tws;   // radix, product of the radices before, butterflies per line, twiddle stride
  unsigned m_bpl, m_ns;  // reciprocals of bpl and NS
};
struct Plan {
  int n;             // line length
  int m;             // transform length: n, or Bluestein's convolution length
  int blue;
  int np;
  unsigned m_n;      // reciprocal of n
  Pass p[kMaxPasses];
};

// x / d for x d < 2^32; d = 1 has no 32-bit reciprocal (m = 0)
inline unsigned reciprocal(int d) { return d == 1 ? 0u : unsigned((1ull << 32) / unsigned(d)) + 1u; }
PTY_DEVI int fdiv(int x, unsigned m) { return m ? int(__umulhi(unsigned(x), m)) : x; }

// fewest passes of radix 2 .. 16 whose product is L (0: none); radices into r
inline int factor_smooth(int L, int* r, int limit) {
  if (L == 1) return 0;
  if (limit <= 0) return -1;
  int best = -1, tmp[kMaxPasses];
  for (int f = 16; f >= 2; --f) {
    if (f == 14 || L % f) continue;
    const int k = factor_smooth(L / f, tmp, (best < 0 ? limit : best - 1) - 1);
    if (k < 0) continue;
    best = k + 1;
    r[0] = f;
    for (int i = 0; i < k; ++i) r[i + 1] = tmp[i];
    if (best == 1 || (L > 16 && best == 2)) break;
  }
  return best;
}

inline bool set_passes(Plan* p, int m, const int* r, int np) {
  p->m = m;
  p->np = np;
  int ns = 1;
  for (int i = 0; i < np; ++i) {
    Pass& q = p->p[i];
    q.R = r[i];
    q.NS = ns;
    q.bpl = m / r[i];
    q.tws = m / (ns * r[i]);
    q.m_bpl = reciprocal(q.bpl);
    q.m_ns = reciprocal(ns);
    ns *= r[i];
  }
  return true;
}

// shared memory of a CTA with `lines` lines
inline int line_stride(int m) { return (m - 1) + ((m - 1) >> 4) + 1; }
inline size_t smem_bytes(const Plan& p, int lines, int extra_tables) {
  size_t n = size_t(2) * lines * line_stride(p.m) + p.m;
  if (p.blue) n += size_t(p.m) + p.n;
  return (n + size_t(extra_tables) * p.n) * sizeof(float2);
}

// extra_tables: further tables of n float2 that the caller keeps
inline bool make_plan(int n, int extra_tables, Plan* p) {
  if (n < 1 || n > kMaxLen) return false;
  p->n = n;
  p->blue = 0;
  p->m_n = reciprocal(n);
  int r[kMaxPasses];
  const int k = factor_smooth(n, r, kMaxPasses);
  if (k >= 0) return set_passes(p, n, r, k);
  for (int m = 2 * n - 1; m <= 2 * kMaxLen; ++m) {  // the next length of no more passes than its size needs
    const int want = m <= 256 ? 2 : (m <= 4096 ? 3 : 4);
    const int q = factor_smooth(m, r, want);
    if (q < 0) continue;
    p->blue = 1;
    set_passes(p, m, r, q);
    if (smem_bytes(*p, 1, extra_tables) <= kSmemCap) return true;
    break;
  }
  p->blue = 0;  // direct-sum passes for the primes above 13
  int np = 0, rest = n;
  for (int f = 17; f <= rest; f += 2)
    while (rest % f == 0 && np < kMaxPasses) {
      bool prime = true;
      for (int d = 3; d * d <= f; d += 2) prime = prime && f % d;
      if (!prime) break;
      r[np++] = f;
      rest /= f;
    }
  const int q = factor_smooth(rest, r + np, kMaxPasses - np);
  if (q < 0) return false;
  return set_passes(p, n, r, np + q);
}

// exp(-2 pi i num / den), 0 <= num < den, rounded once: the angle is taken to a
// quarter turn's half, [-pi/4, pi/4], in whole numbers, then cos and sin are their
// Taylor sums in FP64 (to 1e-10; about twenty instructions)
PTY_DEVI float2 cis_ratio(int num, int den) {
  const double inv = 1.57079632679489662 / double(den);  // one division per loop
  const int q = __float2int_rn(4.0f * float(num) / float(den));
  const double x = double(4 * num - q * den) * inv, y = x * x;
  double c = -1.0 / 3628800.0, s = -1.0 / 39916800.0;
  c = fma(c, y, 1.0 / 40320.0);
  s = fma(s, y, 1.0 / 362880.0);
  c = fma(c, y, -1.0 / 720.0);
  s = fma(s, y, -1.0 / 5040.0);
  c = fma(c, y, 1.0 / 24.0);
  s = fma(s, y, 1.0 / 120.0);
  c = fma(c, y, -0.5);
  s = fma(s, y, -1.0 / 6.0);
  c = fma(c, y, 1.0);
  s = fma(s * y, x, x);
  const float fc = float(c), fs = float(s);
  const float u = q & 1 ? fs : fc, v = q & 1 ? fc : fs;   // q quarter turns further
  return make_float2((q + 1) & 2 ? -u : u, q & 2 ? v : -v);
}

// where value i of line l lives: LINES = 0: whole lines, one float2 of padding
// every 16; LINES > 0: lines interleaved (LINES adjacent columns)
template <int LINES>
PTY_DEVI int slot(int l, int i, int ls) {
  if constexpr (LINES == 0) return l * ls + i + (i >> 4);
  else if constexpr (LINES >= 16) return i * LINES + l;
  else return (i + (i >> 4)) * LINES + l;
}

template <int LINES, int NT, int R>
PTY_DEVI void pass_r(const Pass& ps, const float2* __restrict__ src, float2* __restrict__ dst,
                     const float2* __restrict__ tw, int lines, int ls, int t) {
  const int nb = lines * ps.bpl;
  for (int b = t; b < nb; b += NT) {
    int l, j;
    if constexpr (LINES == 0) {
      l = fdiv(b, ps.m_bpl);
      j = b - l * ps.bpl;
    } else {
      l = b % LINES;
      j = b / LINES;
    }
    const int k = j - fdiv(j, ps.m_ns) * ps.NS;
    float2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = src[slot<LINES>(l, j + r * ps.bpl, ls)];
    if (ps.NS > 1) {
      const float2* w = tw;
#pragma unroll
      for (int r = 1; r < R; ++r) {
        w += k * ps.tws;
        v[r] = c_mul(v[r], *w);
      }
    }
    dft_any<R>(v);
    const int o = (j - k) * R + k;
#pragma unroll
    for (int r = 0; r < R; ++r) dst[slot<LINES>(l, o + r * ps.NS, ls)] = v[r];
  }
}

// direct sum for a prime radix p: output o = (j / NS) NS p + k + r NS gets
// sum_m x[j + m L/p] exp(-2 pi i m (k + r NS) / (NS p))
template <int LINES, int NT>
PTY_DEVI void pass_direct(const Pass& ps, int len, const float2* __restrict__ src, float2* __restrict__ dst,
                          const float2* __restrict__ tw, int lines, int ls, int t) {
  const int p = ps.R, blk = ps.NS * p;
  for (int e = t; e < lines * len; e += NT) {
    const int l = LINES == 0 ? e / len : e % lines, o = LINES == 0 ? e - l * len : e / lines;
    const int ob = o / blk, rem = o - ob * blk;
    const int r = rem / ps.NS, k = rem - r * ps.NS;
    const int j = ob * ps.NS + k;
    const int q = (k + r * ps.NS) * ps.tws;  // < len
    float2 acc = make_float2(0.f, 0.f);
    int idx = 0;
    for (int m = 0; m < p; ++m) {
      const float2 w = tw[idx], x = src[slot<LINES>(l, j + m * ps.bpl, ls)];
      acc.x = fmaf(x.x, w.x, fmaf(-x.y, w.y, acc.x));
      acc.y = fmaf(x.x, w.y, fmaf(x.y, w.x, acc.y));
      idx += q;
      if (idx >= len) idx -= len;
    }
    dst[slot<LINES>(l, o, ls)] = acc;
  }
}

// The lines and tables of a CTA of NT threads.  Use: put() every value of every
// line, pad(), run(), then get() every value; put() may follow a get() of the same
// place.  (Passes that read from and write to global memory directly would save a
// trip through shared memory, but every radix then compiles once per caller:
// ptxas took a quarter of an hour.)
template <int LINES, int NT>
struct Lines {
  float2 *cur, *alt, *tw, *bf, *ch;
  int lines, ls, t;

  // lays out shared memory and builds the tables; returns the first free float2
  PTY_DEVI float2* init(const Plan& p, float2* smem, int nlines, int tid) {
    lines = nlines;
    ls = (p.m - 1) + ((p.m - 1) >> 4) + 1;
    t = tid;
    cur = smem;
    alt = cur + lines * ls;
    tw = alt + lines * ls;
    bf = tw + p.m;
    ch = bf + (p.blue ? p.m : 0);
    for (int i = t; i < p.m; i += NT) tw[i] = cis_ratio(i, p.m);
    if (p.blue) {
      // chirp c_j = exp(-pi i j^2 / n) and the transform of its conjugate, / m; the
      // one-line transform uses whole-line addressing in the two buffers
      for (int i = t; i < p.n; i += NT) ch[i] = cis_ratio(int((long long)i * i % (2 * p.n)), 2 * p.n);
      __syncthreads();
      Lines<0, NT> one{cur, alt, tw, bf, ch, 1, ls, t};
      const float inv = 1.0f / float(p.m);
      for (int i = t; i < p.m; i += NT) {
        const int j = i < p.n ? i : p.m - i;
        const float2 c = j < p.n ? ch[j] : make_float2(0.f, 0.f);
        one.cur[slot<0>(0, i, ls)] = make_float2(c.x * inv, -c.y * inv);
      }
      one.passes(p);
      for (int i = t; i < p.m; i += NT) bf[i] = one.cur[slot<0>(0, i, ls)];
      __syncthreads();
    }
    return ch + (p.blue ? p.n : 0);
  }

  PTY_DEVI void put(const Plan& p, int l, int i, float2 v) {
    cur[slot<LINES>(l, i, ls)] = p.blue ? c_mul(v, ch[i]) : v;
  }
  // Bluestein: zeros after the line (call after the puts, before run)
  PTY_DEVI void pad(const Plan& p) {
    if (!p.blue) return;
    const int z = p.m - p.n;
    for (int e = t; e < lines * z; e += NT) {
      const int l = LINES == 0 ? e / z : e % lines, i = LINES == 0 ? e - l * z : e / lines;
      cur[slot<LINES>(l, p.n + i, ls)] = make_float2(0.f, 0.f);
    }
  }
  PTY_DEVI float2 get(const Plan& p, int l, int i) const {
    const float2 v = cur[slot<LINES>(l, i, ls)];
    return p.blue ? c_mulc(ch[i], v) : v;
  }

  PTY_DEVI void passes(const Plan& p) {
    __syncthreads();
    for (int i = 0; i < p.np; ++i) {
      const Pass& ps = p.p[i];
      switch (ps.R) {
#define PTY_LN(R) \
  case R: pass_r<LINES, NT, R>(ps, cur, alt, tw, lines, ls, t); break;
        PTY_LN(2) PTY_LN(3) PTY_LN(4) PTY_LN(5) PTY_LN(6) PTY_LN(7) PTY_LN(8) PTY_LN(9) PTY_LN(10) PTY_LN(11)
        PTY_LN(12) PTY_LN(13) PTY_LN(15) PTY_LN(16)
#undef PTY_LN
        default: pass_direct<LINES, NT>(ps, p.m, cur, alt, tw, lines, ls, t); break;
      }
      __syncthreads();
      float2* c = cur;
      cur = alt;
      alt = c;
    }
  }

  // DFT of every line (barriers on both sides)
  PTY_DEVI void run(const Plan& p) {
    passes(p);
    if (!p.blue) return;
    for (int e = t; e < lines * p.m; e += NT) {
      const int l = LINES == 0 ? e / p.m : e % lines, i = LINES == 0 ? e - l * p.m : e / lines;
      float2& v = cur[slot<LINES>(l, i, ls)];
      v = c_conj(c_mul(v, bf[i]));
    }
    passes(p);  // conj of the inverse transform; get() undoes the conj
  }
};

}  // namespace ln
}  // namespace pty
