// lines.cuh -- batched DFTs of any length along lines held in shared memory.
//
// Smooth lengths run as Stockham passes of register butterflies, radix 2 to 16
// (dft_small.cuh), planned on the host for the fewest passes: 192 = 16 x 12, 1500 =
// 15 x 10 x 10.  Larger primes up to kDirectPrime are passes of their own, summed in
// pairs (pass_prime).  A length with a prime factor beyond that runs as Bluestein's
// convolution of smooth length m >= 2n - 1 (two transforms of length m and three
// diagonals; a 317-point line costs about two 640-point ones), or, when its tables do
// not fit shared memory (n beyond about 2500), with the pair sums too.
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
// Largest prime that is summed directly.  The pair sums are closer to 64 bits than a
// plain direct sum (0.46 to 0.81 of its error for any prime).  Bluestein's chirp transform
// adds an error of its own: 1.2 to 2.1 times the plain sum's for most lengths with a prime
// of 17 to 47, 0.5 to 1.5 for 53 to 97, and 0.4 to 0.9 beyond (149 alone 0.8 to 1.25,
// by loss).  Steps on B200, pairs : Bluestein: 64 patterns 119^2 86 : 133 us, 148^2 131 :
// 209, 194^2 297 : 470, 226^2 393 : 469, 127^2 165 : 135, 149^2 248 : 213, 251^2 812 : 530;
// 100 patterns 101^2 160 : 154, 113^2 203 : 193, 127^2 264 : 176, 151^2 409 : 307; 4 of
// 226^2 82 : 72, 254^2 92 : 70, 302^2 121 : 98.
constexpr int kDirectPrime = 113;

struct Pass {
  int R, NS, bpl, tws;   // radix, product of the radices before, butterflies per line, twiddle stride
  unsigned m_bpl, m_ns;  // reciprocals of bpl and NS
};
struct Plan {
  int n;             // line length
  int m;             // transform length: n, or Bluestein's convolution length
  int blue;
  int ls;            // distance of whole lines in shared memory
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
  p->ls = (m - 1) + ((m - 1) >> 4) + 1;
  if (np && r[0] > 16) p->ls |= 1;  // pass_prime's neighbouring threads: lines on other banks
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
inline size_t smem_bytes(const Plan& p, int lines, int extra_tables) {
  size_t n = size_t(2) * lines * p.ls + p.m;
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
  int big = n;  // the largest prime factor
  for (int f = 2; f * f <= big; ++f)
    while (big > f && big % f == 0) big /= f;
  for (int m = 2 * n - 1; big > kDirectPrime && m <= 2 * kMaxLen; ++m) {  // the next length of no more passes than its size needs
    const int want = m <= 256 ? 2 : (m <= 4096 ? 3 : 4);
    const int q = factor_smooth(m, r, want);
    if (q < 0) continue;
    p->blue = 1;
    set_passes(p, m, r, q);
    if (smem_bytes(*p, 1, extra_tables) <= kSmemCap) return true;
    break;
  }
  p->blue = 0;  // pair sums for the primes above 13
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

// butterfly b of the CTA -> its line and place
template <int LINES>
PTY_DEVI void line_place(const Pass& ps, int b, int& l, int& j) {
  if constexpr (LINES == 0) {
    l = fdiv(b, ps.m_bpl);
    j = b - l * ps.bpl;
  } else {
    l = b % LINES;
    j = b / LINES;
  }
}

template <int LINES, int NT, int R>
PTY_DEVI void pass_r(const Pass& ps, const float2* __restrict__ src, float2* __restrict__ dst,
                     const float2* __restrict__ tw, int lines, int ls, int t) {
  const int nb = lines * ps.bpl;
  for (int b = t; b < nb; b += NT) {
    int l, j;
    line_place<LINES>(ps, b, l, j);
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

// A prime radix p beyond the register butterflies, in the symmetric pair form at run
// time: twiddled inputs m and p - m become their sum and difference, in place, and
// outputs r and p - r are sum_m (sum_m cos +- i diff_m sin).  A thread sums R
// such r, so that a pair is read once for 4 R products; R of 2 to 4 by the rounds that
// the CTA needs (a round of R costs about 2 + 8 R for each pair).
template <int LINES, int NT, int R>
PTY_DEVI void prime_sums(const Pass& ps, int len, const float2* __restrict__ src, float2* __restrict__ dst,
                         const float2* __restrict__ tw, int lines, int ls, int t) {
  const int p = ps.R, h = (p - 1) / 2, nb = lines * ps.bpl;
  for (int e = t; e < nb * ((h + R) / R); e += NT) {
    const int r0 = e / nb * R;  // r0 .. r0 + R - 1, of 0 .. h
    const int b = e - e / nb * nb;
    int l, j;
    line_place<LINES>(ps, b, l, j);
    const float2 x0 = src[slot<LINES>(l, j, ls)];
    float2 a[R], d[R];  // sums by cos, differences by -sin
    int idx[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      a[i] = x0;
      d[i] = make_float2(0.f, 0.f);
      idx[i] = 0;
    }
#pragma unroll 1
    for (int m = 1; m <= h; ++m) {
      const float2 u = src[slot<LINES>(l, j + m * ps.bpl, ls)], v = src[slot<LINES>(l, j + (p - m) * ps.bpl, ls)];
#pragma unroll
      for (int i = 0; i < R; ++i) {
        idx[i] += (r0 + i) * ps.bpl;
        if (idx[i] >= len) idx[i] -= len;
        const float2 w = tw[idx[i]];
        a[i] = make_float2(fmaf(u.x, w.x, a[i].x), fmaf(u.y, w.x, a[i].y));
        d[i] = make_float2(fmaf(v.x, w.y, d[i].x), fmaf(v.y, w.y, d[i].y));
      }
    }
    const int k = j - fdiv(j, ps.m_ns) * ps.NS, o = (j - k) * p + k;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int r = r0 + i;
      if (r > h) break;
      dst[slot<LINES>(l, o + r * ps.NS, ls)] = make_float2(a[i].x - d[i].y, a[i].y + d[i].x);
      if (r > 0) dst[slot<LINES>(l, o + (p - r) * ps.NS, ls)] = make_float2(a[i].x + d[i].y, a[i].y - d[i].x);
    }
  }
}

template <int LINES, int NT>
PTY_DEVI void pass_prime(const Pass& ps, int len, float2* __restrict__ src, float2* __restrict__ dst,
                         const float2* __restrict__ tw, int lines, int ls, int t) {
  const int p = ps.R, h = (p - 1) / 2, nb = lines * ps.bpl;
  int l, j;
#pragma unroll 1
  for (int e = t; e < nb * h; e += NT) {
    const int m = e / nb + 1;
    line_place<LINES>(ps, e - (m - 1) * nb, l, j);
    float2 &u = src[slot<LINES>(l, j + m * ps.bpl, ls)], &v = src[slot<LINES>(l, j + (p - m) * ps.bpl, ls)];
    float2 x = u, y = v;
    if (ps.NS > 1) {
      const int k = j - fdiv(j, ps.m_ns) * ps.NS;
      x = c_mul(x, tw[m * k * ps.tws]);
      y = c_mul(y, tw[(p - m) * k * ps.tws]);
    }
    u = c_add(x, y);
    v = c_sub(x, y);
  }
  __syncthreads();
  const auto cost = [&](int R) { return (nb * ((h + R) / R) + NT - 1) / NT * (2 + 8 * R); };
  const int c2 = cost(2), c3 = cost(3), c4 = cost(4);
  if (c2 <= c3 && c2 <= c4) prime_sums<LINES, NT, 2>(ps, len, src, dst, tw, lines, ls, t);
  else if (c3 <= c4) prime_sums<LINES, NT, 3>(ps, len, src, dst, tw, lines, ls, t);
  else prime_sums<LINES, NT, 4>(ps, len, src, dst, tw, lines, ls, t);
}

// All passes of the lines in a, with b the other buffer; the result is in b after an odd
// number of them.  The butterflies of fourteen radices are most of a kernel's code, so
// they are inlined once: with a copy each for the loss's second transform, Bluestein's
// way back and its filter, the first step of a process on 192^2 took 4.6 ms (2.8 here)
// and every later one, 64 patterns, 110 us (106).  As one function for all kernels the
// first takes 2.4 ms, but its callers spill: 117 us.
template <int LINES, int NT>
PTY_DEVI void run_passes(const Pass* passes, int np, int m, float2* a, float2* b, const float2* tw, int lines, int ls,
                         int t) {
  __syncthreads();
#pragma unroll 1
  for (int i = 0; i < np; ++i) {
    const Pass& ps = passes[i];
    switch (ps.R) {
#define PTY_LN(R) \
  case R: pass_r<LINES, NT, R>(ps, a, b, tw, lines, ls, t); break;
      PTY_LN(2) PTY_LN(3) PTY_LN(4) PTY_LN(5) PTY_LN(6) PTY_LN(7) PTY_LN(8) PTY_LN(9) PTY_LN(10) PTY_LN(11)
      PTY_LN(12) PTY_LN(13) PTY_LN(15) PTY_LN(16)
#undef PTY_LN
      default: pass_prime<LINES, NT>(ps, m, a, b, tw, lines, ls, t); break;
    }
    __syncthreads();
    float2* c = a;
    a = b;
    b = c;
  }
}
// the same for Bluestein's filter, once per CTA: a function of its own
template <int NT>
__device__ __noinline__ void one_line(const Pass* passes, int np, int m, float2* a, float2* b, const float2* tw, int ls) {
  run_passes<0, NT>(passes, np, m, a, b, tw, 1, ls, threadIdx.x);
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
    ls = p.ls;
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
      const float inv = 1.0f / float(p.m);
      for (int i = t; i < p.m; i += NT) {
        const int j = i < p.n ? i : p.m - i;
        const float2 c = j < p.n ? ch[j] : make_float2(0.f, 0.f);
        cur[slot<0>(0, i, ls)] = make_float2(c.x * inv, -c.y * inv);
      }
      __shared__ Pass sp[kMaxPasses];
      if (t < p.np) sp[t] = p.p[t];
      __syncthreads();
      one_line<NT>(sp, p.np, p.m, cur, alt, tw, ls);
      const float2* f = p.np & 1 ? alt : cur;
      for (int i = t; i < p.m; i += NT) bf[i] = f[slot<0>(0, i, ls)];
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
    run_passes<LINES, NT>(p.p, p.np, p.m, cur, alt, tw, lines, ls, t);
    if (p.np & 1) {
      float2* c = cur;
      cur = alt;
      alt = c;
    }
  }

  // DFT of every line (barriers on both sides)
  PTY_DEVI void run(const Plan& p) {
#pragma unroll 1
    for (int back = 0;; ++back) {  // the passes' code once
      passes(p);
      if (back == p.blue) return;  // Bluestein: conj of the inverse transform; get() undoes the conj
      for (int e = t; e < lines * p.m; e += NT) {
        const int l = LINES == 0 ? e / p.m : e % lines, i = LINES == 0 ? e - l * p.m : e / lines;
        float2& v = cur[slot<LINES>(l, i, ls)];
        v = c_conj(c_mul(v, bf[i]));
      }
    }
  }
};

}  // namespace ln
}  // namespace pty
