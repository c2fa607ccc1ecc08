// resample.cu -- Fourier (band-limited) upsampling of the object and its adjoint.
//
// Replaces models/complex_inr.py:252-271 (called at :287):
//   y = ifft2( ifftshift( zero_pad( fftshift( fft2(x) ) ) ) ) * s^2,
// x [h][w] -> y [h*s][w*s] complex64, and the gradient of that map (torch's
// complex convention, the conjugate-transpose operator).  The map is
// separable: per axis, y = (s / N) F_N^-1 P F_n x, where F is the
// unnormalised DFT and P places frequency f in [-n/2, n/2) of the length-n
// spectrum at f mod N of the length-N one (for even n and N this is what the
// shift / centred pad / inverse shift of the reference does).  Its adjoint is
// (s / N) F_n^-1 P^T F_N.  Neither forms the long spectrum: the s interleaved
// phases of the long line are length-n transforms (below).
//   row pass    -- lines are rows (contiguous), written as rows;
//   column pass -- lines are a few adjacent columns.
// Upsampling: column pass x -> t [h s][w], row pass t -> y.  Adjoint: row pass
// g -> t [h s][w], column pass t -> x-gradient.  Both column passes move the
// narrow side, in pieces of a few columns; the wide side moves as whole rows.
// Twiddles of the power-of-two kernels come from the correctly rounded build-time
// table kTw4096 (twiddle4096.cuh).
// A NaN or infinity anywhere reaches every output of its line, hence of the plane, as
// it does through the transforms of the reference, also where phase 0 is copied.
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "dft_regs.cuh"
#include "lines.cuh"
#include "twiddle4096.cuh"

namespace pty {

// x, not finite where z is not
PTY_DEVI float2 c_taint(float2 x, float2 z) { return make_float2(fmaf(0.f, z.x, x.x), fmaf(0.f, z.y, x.y)); }

namespace sh {

// ---------------------------------------------------------------------------
// Power-of-two lines of 256 to 2048 points, upsampled by s = 2 or 4.
//
// Interleaving the s phases of the long line, y[s m + p] is the inverse length-n
// transform of X_k exp(2 pi i k p / N): phase 0 is x itself, and every other
// phase is one forward and one inverse length-n transform with a diagonal
// between -- for s = 2 a third of the arithmetic and half the shared memory of
// padding the spectrum to length N, and a quarter of the samples are copies.  The
// adjoint is the same with the conjugate diagonal, summed over the phases.
//
// n = 16 * 16 * C: a line is held by n / 16 threads, 16 values each.  Forward,
// decimation in frequency: thread q has x[q + 16 C e]; DFT16 over e -> digit a,
// twiddle W_n^(q a); exchange; thread (a, q0) has q = q0 + C e; DFT16 -> digit b,
// twiddle W_16C^(q0 b); exchange; DFT_C -> digit c, frequency a + 16 b + 256 c.
// The diagonal is applied in that order and the inverse walks back, so nothing is
// reordered: four exchanges in all (the padded form moved the line through
// shared memory seven times).  The diagonal of frequency a + 16 b + 256 c is a
// product of three factors: that of c is applied where c is in registers, those of
// a and b are part of the inverse's twiddles.  An exchange writes value (a, q) at a P + q or
// (a, q0, b) at a P + 17 q0 + b, P = 17 C: conflict free both ways for 8-byte
// accesses of a half-warp (P = C, 17 = 1 mod 16).
// Measured on B200, 2048^2 to 4096^2 and back: 279 us for the four passes (48 + 72
// up, 79 + 66 down) against 668 us by padded spectra; bound by latency (issue 35 to
// 40 %, four to seven barriers between loads and stores), 336 MB would take 51 us.
// Columns: COLS adjacent columns per CTA, interleaved in shared memory the same
// way, so global accesses are pieces of 8 COLS bytes.
// ---------------------------------------------------------------------------
template <int N, bool COL>
struct Cfg {
  static constexpr int C = N / 256;           // last radix
  static constexpr int T = N / 16;            // threads per line
  static constexpr int COLS = COL ? (512 / T) : 1;
  static constexpr int LINES = 512 / T;       // lines per CTA
  static constexpr int NT = 512;
  static constexpr int P = 17 * C;
  static constexpr int PLANE = 16 * P;        // float2 per line
  static constexpr size_t SMEM = size_t(LINES * PLANE + 2 * N + 32 * C + 16) * sizeof(float2);
  static constexpr int MINB = 2;              // CTAs per SM: 64 registers
  static_assert(C == 1 || C == 2 || C == 4 || C == 8, "line length");
};

struct Args {
  const float2* in;
  float2* out;
  int nlines;
  long long ld_in, ld_out;  // elements between rows
  int s;
  int vec;  // rows: the long line's pairs (s = 2) are 16-byte aligned
};

// bring the lines from l0 on towards L2 (a line's loads start its chain)
template <int N, bool COL, bool ADJ>
PTY_DEVI void prefetch_line(const Args& g, int l0, int t) {
  using F = Cfg<N, COL>;
  const int len = ADJ ? N * g.s : N;  // input length
  if constexpr (COL) {
    if (l0 < g.nlines)
      for (int i = t; i < len; i += F::NT) asm volatile("prefetch.global.L2 [%0];" ::"l"(g.in + i * g.ld_in + l0));
  } else {
    for (int i = t * 16; i < F::LINES * len; i += F::NT * 16) {  // 128-byte pieces
      const int l = l0 + i / len;
      if (l < g.nlines) asm volatile("prefetch.global.L2 [%0];" ::"l"(g.in + l * g.ld_in + i % len));
    }
  }
}

template <int N, bool COL, bool ADJ>
__global__ void __launch_bounds__(Cfg<N, COL>::NT, Cfg<N, COL>::MINB) k_shift(const Args g) {
  using F = Cfg<N, COL>;
  constexpr int C = F::C, T = F::T, P = F::P, LINES = F::LINES, ST = COL ? F::COLS : 1;
  extern __shared__ __align__(16) unsigned char smem[];
  float2* buf = reinterpret_cast<float2*>(smem);
  float2* twa = buf + LINES * F::PLANE;  // W_N^(q a) at a T + q
  float2* twi = twa + N;                 // its conjugate times the diagonal's factor of a, / N
  float2* twb = twi + N;                 // W_16C^(q0 b) at b C + q0
  float2* twj = twb + 16 * C;            // its conjugate times the factor of b
  float2* dg = twj + 16 * C;             // the factor of c (C = 1: of b)
  const int t = threadIdx.x;
  const int line = COL ? t % LINES : t / T, q = COL ? t / LINES : t % T;
  float2* lb = buf + (COL ? line : line * F::PLANE);  // this line's value i at lb[i * ST]
  const int a = q / C, q0 = q % C;                    // stage B: digit a, residue q0; stage C: b = q0 + C g
  const int s = g.s;
  const int unit = 4096 / (s * N);  // exp(2 pi i j / (s N)) is the conjugate of entry j unit
  for (int i = t; i < N; i += F::NT) twa[i] = __ldg(&kTw4096[((i / T) * (i % T) * s * unit) & 4095]);
  for (int i = t; i < 16 * C; i += F::NT) twb[i] = __ldg(&kTw4096[((i / C) * (i % C) * (256 / C)) & 4095]);
  // upsampling: a CTA has one phase; adjoint: it sums over all of them
  const int p0 = ADJ ? 1 : blockIdx.y + 1, p1 = ADJ ? s : p0 + 1;
  for (int p = p0; p < p1; ++p) {
    const int sp = ADJ ? -p : p;  // the adjoint's diagonal is the conjugate
    if (p > p0) __syncthreads();  // the last phase's tables are no longer read
    for (int i = t; i < N; i += F::NT) {
      const float2 w = __ldg(&kTw4096[(-(i / T) * ((i % T) * s + sp) * unit) & 4095]);
      twi[i] = make_float2(w.x * (1.0f / float(N)), w.y * (1.0f / float(N)));
    }
    for (int i = t; i < 16 * C; i += F::NT)
      twj[i] = __ldg(&kTw4096[(-16 * (i / C) * ((i % C) * s + sp) * unit) & 4095]);
    if (t < 16) {  // frequencies from N / 2 on are negative
      const int f = C > 1 ? 256 * (t < C / 2 ? t : t - C) : 16 * (t < 8 ? t : t - 16);
      dg[t] = __ldg(&kTw4096[(-f * sp * unit) & 4095]);
    }
    for (int l0 = blockIdx.x * LINES; l0 < g.nlines; l0 += gridDim.x * LINES) {
      const int l = l0 + line;
      const bool ok = l < g.nlines;
      // element i of this line (short side: x or gx; long side: y or gy)
      auto at = [&](auto* base, long long ld, int i) { return COL ? base + i * ld + l : base + l * ld + i; };
      float2 v[16];
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const int m = q + T * e;
        v[e] = make_float2(0.f, 0.f);
        if (ok) v[e] = ADJ ? __ldg(at(g.in, g.ld_in, s * m + p)) : __ldg(at(g.in, g.ld_in, m));
        if (ADJ && ok && p == 1) v[e] = c_taint(v[e], __ldg(at(g.in, g.ld_in, s * m)));
        if (COL && !ADJ && ok && p == 1) *at(g.out, g.ld_out, s * m) = v[e];  // phase 0
      }
      prefetch_line<N, COL, ADJ>(g, l0 + gridDim.x * LINES, t);
      __syncthreads();  // the tables are in place; earlier readers of the exchange are done
      dft16<false, 1>(v);
#pragma unroll
      for (int k = 1; k < 16; ++k) v[k] = c_mul(v[k], twa[k * T + q]);
#pragma unroll
      for (int k = 0; k < 16; ++k) lb[(k * P + q) * ST] = v[k];
      __syncthreads();
#pragma unroll
      for (int e = 0; e < 16; ++e) v[e] = lb[(a * P + q0 + C * e) * ST];
      dft16<false, 1>(v);
      if constexpr (C > 1) {
#pragma unroll
        for (int b = 1; b < 16; ++b) v[b] = c_mul(v[b], twb[b * C + q0]);
        __syncthreads();
#pragma unroll
        for (int b = 0; b < 16; ++b) lb[(a * P + 17 * q0 + b) * ST] = v[b];
        __syncthreads();
#pragma unroll
        for (int gg = 0; gg < 16 / C; ++gg)
#pragma unroll
          for (int k = 0; k < C; ++k) v[gg * C + k] = lb[(a * P + 17 * k + q0 + C * gg) * ST];
#pragma unroll
        for (int gg = 0; gg < 16 / C; ++gg) dft<C, false, 1>(v + gg * C);
      }
#pragma unroll
      for (int j = 1; j < 16; ++j)
        if (C == 1 || j % C > 0) v[j] = c_mul(v[j], dg[C > 1 ? j % C : j]);
      if constexpr (C > 1) {
#pragma unroll
        for (int gg = 0; gg < 16 / C; ++gg) dft<C, true, 1>(v + gg * C);
        __syncthreads();
#pragma unroll
        for (int gg = 0; gg < 16 / C; ++gg)
#pragma unroll
          for (int k = 0; k < C; ++k) lb[(a * P + 17 * k + q0 + C * gg) * ST] = v[gg * C + k];
        __syncthreads();
#pragma unroll
        for (int b = 0; b < 16; ++b) v[b] = lb[(a * P + 17 * q0 + b) * ST];
#pragma unroll
        for (int b = 1; b < 16; ++b) v[b] = c_mul(v[b], twj[b * C + q0]);
      }
      dft16<true, 1>(v);
      __syncthreads();
#pragma unroll
      for (int e = 0; e < 16; ++e) lb[(a * P + q0 + C * e) * ST] = v[e];
      __syncthreads();
#pragma unroll
      for (int k = 0; k < 16; ++k) v[k] = lb[(k * P + q) * ST];
      v[0] = c_scale(v[0], 1.0f / float(N));
#pragma unroll
      for (int k = 1; k < 16; ++k) v[k] = c_mul(v[k], twi[k * T + q]);
      dft16<true, 1>(v);
      if (!ok) continue;
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const int m = q + T * e;
        if constexpr (ADJ) {
          float2* o = at(g.out, g.ld_out, m);
          *o = c_add(p == 1 ? __ldg(at(g.in, g.ld_in, s * m)) : *o, v[e]);
        } else if (!COL && s == 2 && g.vec) {
          const float2 x = c_taint(__ldg(at(g.in, g.ld_in, m)), v[e]);
          *reinterpret_cast<float4*>(at(g.out, g.ld_out, 2 * m)) = make_float4(x.x, x.y, v[e].x, v[e].y);
        } else {
          if (!COL && p == 1) *at(g.out, g.ld_out, s * m) = c_taint(__ldg(at(g.in, g.ld_in, m)), v[e]);
          if (COL && p == 1 && !(isfinite(v[e].x) && isfinite(v[e].y))) *at(g.out, g.ld_out, s * m) = v[e];
          *at(g.out, g.ld_out, s * m + p) = v[e];
        }
      }
    }
  }
}

template <int N, bool COL, bool ADJ>
static int launch(const Args& g, cudaStream_t st) {
  using F = Cfg<N, COL>;
  auto kern = k_shift<N, COL, ADJ>;
  static PtyDevCache slots_cache;  // resident CTAs, with the shared-memory attribute set
  int dev = 0;
  for (int attempt = 0; attempt < 2; ++attempt) {
    int slots = slots_cache.get(&dev);
    if (dev < 0) return PTYCHO_ERR_LAUNCH;
    if (slots == 0) {
      int nsm = 148, per_sm = 1;
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(F::SMEM)) != cudaSuccess)
        return PTYCHO_ERR_LAUNCH;
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, F::NT, F::SMEM) != cudaSuccess || per_sm < 1)
        per_sm = 1;
      slots = nsm * per_sm;
      slots_cache.put(dev, slots);
    }
    const int need = (g.nlines + F::LINES - 1) / F::LINES;
    kern<<<dim3(need < slots ? need : slots, ADJ ? 1 : g.s - 1), F::NT, F::SMEM, st>>>(g);
    if (cudaGetLastError() == cudaSuccess) return PTYCHO_OK;
    slots_cache.put(dev, 0);
  }
  return PTYCHO_ERR_LAUNCH;
}

static bool supported(int n, int s) {
  return (n == 256 || n == 512 || n == 1024 || n == 2048) && (s == 2 || s == 4) && n * s <= 4096;
}

// one axis of the upsampling (ADJ: of its adjoint) on every line of a pass
template <bool COL, bool ADJ>
static int dispatch(int n, const Args& g, cudaStream_t st) {
  switch (n) {
    case 256: return launch<256, COL, ADJ>(g, st);
    case 512: return launch<512, COL, ADJ>(g, st);
    case 1024: return launch<1024, COL, ADJ>(g, st);
    default: return launch<2048, COL, ADJ>(g, st);
  }
}

}  // namespace sh

// ---------------------------------------------------------------------------
// Any other line length (the canvases Recovery.py builds are multiples of 6, so
// object grids are multiples of 3 and can hold large prime factors: 498 =
// 2 * 3 * 83) and any scale, by the same phases on the transforms of lines.cuh.
// For odd n the reference's fftshift / centred pad / ifftshift puts the band's bin k
// at (k + d) mod N, d = floor(n/2) + floor((N-n)/2) - floor(N/2): d = 0 for even n,
// or odd n and odd N; d = -1 for odd n and even N (the reference's half-bin
// asymmetry, kept): every sample j of the long line is turned by exp(2 pi i d j / N).
// Measured on B200: 1500^2 to 3000^2 61 + 113 us against 213 + 141 by padded spectra
// with run-time radix loops; 498^2 to 996^2 and back 118 against 675 us (factor 83).
// ---------------------------------------------------------------------------
namespace rsg {

using ln::Plan;

struct Args {
  const float2* in;
  float2* out;
  int nlines;
  long long ld_in, ld_out;
  int s, d;     // scale; band offset (0 or -1)
  int lines;    // lines per CTA
  int tables;   // tables of n values: the diagonals, and the turns when d != 0
  int acc;      // keeps a sum of spectra (adjoint, s > 2)
  int ngroups;
  int vec;      // rows: the long line's pairs (s = 2) are 16-byte aligned
  Plan plan;    // length n, the short side
};

// LINES = 0: rows; else LINES adjacent columns per CTA
template <int LINES, int NT, bool ADJ>
__global__ void __launch_bounds__(NT, LINES == 16 || LINES == 0 ? 4 : 1) k_resample_any(const Args g) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr bool COL = LINES > 0;
  const int t = threadIdx.x, n = g.plan.n, N = n * g.s, s = g.s;
  ln::Lines<LINES, NT> ln;
  float2* ph = ln.init(g.plan, reinterpret_cast<float2*>(smem), COL ? LINES : g.lines, t);
  auto at = [&](auto* base, long long ld, int l, int i) { return COL ? base + i * ld + l : base + l * ld + i; };
  // upsampling: a CTA has one phase, whose diagonal is ph; adjoint: it sums all phases'
  // spectra (s > 2: in acc) before the one inverse transform, with a diagonal each
  const int p0 = ADJ ? 1 : blockIdx.y + 1, p1 = ADJ ? s : p0 + 1;
  // odd n, even N: sample s k + p of the long line is turned into (ADJ: out of) the
  // band's place by exp(-2 pi i (s k + p) / N)
  const bool turned = g.d != 0;
  float2* turn_k = ph + (p1 - p0) * n;
  float2* acc = turn_k + (turned ? n : 0);
  for (int e = t; e < (p1 - p0) * n; e += NT) {
    const int p = p0 + e / n, k = e % n;
    const int f = k < (n + 1) / 2 ? k : k - n;  // signed frequency
    int j = int((long long)(ADJ ? f : -f) * p % N);
    if (j < 0) j += N;
    ph[e] = c_scale(ln::cis_ratio(j, N), 1.0f / float(n));
  }
  if (turned)
    for (int k = t; k < n; k += NT) turn_k[k] = ln::cis_ratio(s * k, N);
  __syncthreads();
  auto turn = [&](float2 v, int k, float2 wp) {
    if (!turned) return v;
    const float2 w = c_mul(turn_k[k], wp);
    return ADJ ? c_mulc(v, w) : c_mul(v, w);
  };
  const float2 one = make_float2(1.f, 0.f);
  // element e of a group -> its line and place
  auto split = [&](int e, int& l, int& k) {
    if constexpr (COL) {
      l = e % LINES;
      k = e / LINES;
    } else {
      l = ln::fdiv(e, g.plan.m_n);
      k = e - l * n;
    }
  };
  const int per = (COL ? LINES : g.lines) * n;
  for (int grp = blockIdx.x; grp < g.ngroups; grp += gridDim.x) {
    const int l0 = grp * (COL ? LINES : g.lines);
    int l, k;
    for (int p = p0; p < p1; ++p) {
      const float2 wp = turned ? ln::cis_ratio(p, N) : one;
      const float2* d = ph + (p - p0) * n;
#pragma unroll 4
      for (int e = t; e < per; e += NT) {
        split(e, l, k);
        float2 v = make_float2(0.f, 0.f);
        if (l0 + l < g.nlines)
          v = ADJ ? turn(__ldg(at(g.in, g.ld_in, l0 + l, s * k + p)), k, wp) : __ldg(at(g.in, g.ld_in, l0 + l, k));
        if (ADJ && p == 1 && l0 + l < g.nlines) v = c_taint(v, __ldg(at(g.in, g.ld_in, l0 + l, s * k)));
        ln.put(g.plan, l, k, v);
      }
      ln.pad(g.plan);
      ln.run(g.plan);
      for (int e = t; e < per; e += NT) {
        split(e, l, k);
        float2 v = c_mul(ln.get(g.plan, l, k), d[k]);
        if (ADJ && s > 2) {  // this thread's own place of acc
          if (p > 1) v = c_add(acc[e], v);
          if (p + 1 < s) {
            acc[e] = v;
            continue;
          }
        }
        ln.put(g.plan, l, k, c_conj(v));
      }
      if (p + 1 < p1) __syncthreads();  // the spectrum is read before the next phase's line overwrites it
    }
    ln.pad(g.plan);
    ln.run(g.plan);
    const float2 wp = turned ? ln::cis_ratio(p0, N) : one;
#pragma unroll 4
    for (int e = t; e < per; e += NT) {
      split(e, l, k);
      if (l0 + l >= g.nlines) continue;
      const float2 v = c_conj(ln.get(g.plan, l, k));
      if constexpr (ADJ) {
        *at(g.out, g.ld_out, l0 + l, k) = c_add(turn(__ldg(at(g.in, g.ld_in, l0 + l, s * k)), k, one), v);
      } else {
        const float2 z = turn(v, k, wp);
        float2 x = make_float2(0.f, 0.f);
        if (p0 == 1) x = c_taint(turn(__ldg(at(g.in, g.ld_in, l0 + l, k)), k, one), z);
        if (!COL && s == 2 && g.vec) {
          *reinterpret_cast<float4*>(at(g.out, g.ld_out, l0 + l, 2 * k)) = make_float4(x.x, x.y, z.x, z.y);
        } else {
          if (p0 == 1) *at(g.out, g.ld_out, l0 + l, s * k) = x;
          *at(g.out, g.ld_out, l0 + l, s * k + p0) = z;
        }
      }
    }
    __syncthreads();  // the buffers are free for the next group
  }
}

static size_t smem_of(const Args& g, int lines) {
  return ln::smem_bytes(g.plan, lines, g.tables + (g.acc ? lines : 0));
}

template <int LINES, int NT, bool ADJ>
static int launch_k(const Args& g, cudaStream_t st) {
  auto kern = k_resample_any<LINES, NT, ADJ>;
  const size_t smem = smem_of(g, LINES > 0 ? LINES : g.lines);
  static PtyDevCache attr;
  int dev = 0;
  for (int attempt = 0; attempt < 2; ++attempt) {
    int nsm = attr.get(&dev);
    if (dev < 0) return PTYCHO_ERR_LAUNCH;
    if (!nsm) {
      nsm = 148;
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(ln::kSmemCap)) != cudaSuccess)
        return PTYCHO_ERR_LAUNCH;
      attr.put(dev, nsm);
    }
    const int per_sm = int(233472 / (smem + 1024 + 192));
    const int slots = nsm * (per_sm < 1 ? 1 : (per_sm > 4 ? 4 : per_sm));
    kern<<<dim3(g.ngroups < slots ? g.ngroups : slots, ADJ ? 1 : g.s - 1), NT, smem, st>>>(g);
    if (cudaGetLastError() == cudaSuccess) return PTYCHO_OK;
    attr.put(dev, 0);
  }
  return PTYCHO_ERR_LAUNCH;
}

// one axis of length n upsampled by s (ADJ: its adjoint) on every line of a pass
template <bool COL, bool ADJ>
static int launch(int n, int s, const float2* in, float2* out, int nlines, long long ld_in, long long ld_out,
                  cudaStream_t st) {
  Args g{};
  const int N = n * s;
  g.d = n / 2 + (N - n) / 2 - N / 2;
  g.acc = ADJ && s > 2;
  g.tables = (ADJ ? s - 1 : 1) + (g.d ? 1 : 0);
  if (!ln::make_plan(n, g.tables + g.acc, &g.plan)) return PTYCHO_ERR_UNSUPPORTED_SIZE;
  g.in = in;
  g.out = out;
  g.nlines = nlines;
  g.ld_in = ld_in;
  g.ld_out = ld_out;
  g.s = s;
  g.vec = ld_out % 2 == 0 && pty_aligned(out, 16) ? 1 : 0;
  auto groups = [&](int lines) {
    g.lines = lines;
    g.ngroups = (nlines + lines - 1) / lines;
  };
  if constexpr (COL) {
    // 16 adjacent columns (128-byte pieces) while two CTAs fit an SM, else 4 or 1; four
    // long columns leave room for one CTA, so it has 1024 threads (1500^2 by 2, up and
    // down: 419 us with 512, 403 with 768, 395 with 1024)
    // lines with a large prime compute for long: four columns per CTA while 16 would leave
    // SMs idle (249^2 by 2 133 -> 83-99 us, 255^2 107 -> 75, 222 x 333 by 3 123 -> 97)
    const bool few = g.plan.np && g.plan.p[0].R > 16 && (nlines + 15) / 16 * (ADJ ? 1 : s - 1) < 148;
    if (smem_of(g, 16) <= 112 * 1024 && !few) {
      groups(16);
      return launch_k<16, 256, ADJ>(g, st);
    }
    if (smem_of(g, 4) <= ln::kSmemCap) {
      groups(4);
      return launch_k<4, 1024, ADJ>(g, st);
    }
    groups(1);
    return launch_k<1, 512, ADJ>(g, st);
  } else {
    // about 1536 values per CTA: four CTAs of a long line fit an SM (1500^2 by 2: 419
    // -> 396 us, 500^2 by 3 126 -> 115, 999 x 1500 463 -> 435 against 3072 values)
    int lines = 1536 / g.plan.m;
    lines = lines < 1 ? 1 : lines;
    while (lines > 1 && smem_of(g, lines) > ln::kSmemCap) --lines;
    groups(lines);
    return launch_k<0, 256, ADJ>(g, st);
  }
}

}  // namespace rsg
}  // namespace pty

using namespace pty;

namespace {

// one axis of the upsampling by s (ADJ: of its adjoint) on every line of a pass:
// n is the short side
template <bool COL, bool ADJ>
int axis_pass(int n, int s, const float2* in, float2* out, int nlines, long long ld_in, long long ld_out,
              cudaStream_t st) {
  if (sh::supported(n, s)) {
    sh::Args g{in, out, nlines, ld_in, ld_out, s, pty_aligned(ADJ ? in : out, 16) ? 1 : 0};
    return sh::dispatch<COL, ADJ>(n, g, st);
  }
  return rsg::launch<COL, ADJ>(n, s, in, out, nlines, ld_in, ld_out, st);
}

// s = 1: the operator is the identity, and NaN throughout where any input is not
// finite: every block says whether its share is, then every block copies
constexpr int kCopyBlocks = 148 * 4;
__global__ void __launch_bounds__(256) k_nonfinite(const float* __restrict__ in, size_t n, int* __restrict__ bad) {
  int b = 0;
  for (size_t i = size_t(blockIdx.x) * 256 + threadIdx.x; i < n; i += size_t(gridDim.x) * 256) b |= !isfinite(in[i]);
  b = __syncthreads_or(b);
  if (threadIdx.x == 0) bad[blockIdx.x] = b;
}
__global__ void __launch_bounds__(256) k_copy(const float* in, float* out, size_t n, const int* __restrict__ bad) {
  int b = 0;
  for (int i = threadIdx.x; i < gridDim.x; i += 256) b |= bad[i];
  b = __syncthreads_or(b);
  for (size_t i = size_t(blockIdx.x) * 256 + threadIdx.x; i < n; i += size_t(gridDim.x) * 256)
    out[i] = b ? __int_as_float(0x7fc00000) : in[i];
}
int copy_plane(const float* in, float* out, size_t n, void* workspace, cudaStream_t st) {
  n *= 2;  // floats
  const size_t need = (n + 255) / 256;  // blocks; their flags (n / 64 bytes) fit the workspace (4 n bytes)
  const unsigned grid = unsigned(need < kCopyBlocks ? need : kCopyBlocks);
  k_nonfinite<<<grid, 256, 0, st>>>(in, n, static_cast<int*>(workspace));
  k_copy<<<grid, 256, 0, st>>>(in, out, n, static_cast<const int*>(workspace));
  return cudaGetLastError() == cudaSuccess ? PTYCHO_OK : PTYCHO_ERR_LAUNCH;
}

bool supported_upsample(int h, int w, int s) {
  if (h <= 0 || w <= 0 || s <= 0) return false;
  if (h > ln::kMaxLen / s || w > ln::kMaxLen / s) return false;
  return true;
}

}  // namespace

extern "C" {

size_t ptycho_fourier_upsample_workspace_size(int h, int w, int s) {
  if (h <= 0 || w <= 0 || s <= 0) return 0;
  return size_t(h) * size_t(w) * size_t(s) * sizeof(float2);
}

int ptycho_fourier_upsample(const float* x, int h, int w, int s, float* y, void* workspace,
                            size_t workspace_bytes, ptycho_stream_t stream) {
  if (!x || !y || h <= 0 || w <= 0 || s <= 0) return PTYCHO_ERR_INVALID_ARG;
  if (!supported_upsample(h, w, s)) return PTYCHO_ERR_UNSUPPORTED_SIZE;
  if (!workspace || workspace_bytes < ptycho_fourier_upsample_workspace_size(h, w, s))
    return PTYCHO_ERR_WORKSPACE;
  if (!pty_aligned(x, 8) || !pty_aligned(y, 8) || !pty_aligned(workspace, 8)) return PTYCHO_ERR_MISALIGNED;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int W = w * s, H = h * s;
  if (s == 1) return copy_plane(x, y, size_t(h) * w, workspace, st);
  float2* tmp = static_cast<float2*>(workspace);  // [H][w]: the column pass moves the narrow side
  int rc = axis_pass<true, false>(h, s, reinterpret_cast<const float2*>(x), tmp, w, w, w, st);  // columns
  if (rc) return rc;
  return axis_pass<false, false>(w, s, tmp, reinterpret_cast<float2*>(y), H, w, W, st);          // rows
}

int ptycho_fourier_upsample_adjoint(const float* gy, int h, int w, int s, float* gx, void* workspace,
                                    size_t workspace_bytes, ptycho_stream_t stream) {
  if (!gy || !gx || h <= 0 || w <= 0 || s <= 0) return PTYCHO_ERR_INVALID_ARG;
  if (!supported_upsample(h, w, s)) return PTYCHO_ERR_UNSUPPORTED_SIZE;
  if (!workspace || workspace_bytes < ptycho_fourier_upsample_workspace_size(h, w, s))
    return PTYCHO_ERR_WORKSPACE;
  if (!pty_aligned(gy, 8) || !pty_aligned(gx, 8) || !pty_aligned(workspace, 8)) return PTYCHO_ERR_MISALIGNED;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int W = w * s, H = h * s;
  if (s == 1) return copy_plane(gy, gx, size_t(h) * w, workspace, st);
  float2* tmp = static_cast<float2*>(workspace);  // [H][w]
  int rc = axis_pass<false, true>(w, s, reinterpret_cast<const float2*>(gy), tmp, H, W, w, st);  // rows
  if (rc) return rc;
  return axis_pass<true, true>(h, s, tmp, reinterpret_cast<float2*>(gx), w, w, w, st);            // columns
}

}  // extern "C"
