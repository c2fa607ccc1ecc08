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
// (s / N) F_n^-1 P^T F_N.  Both are "forward FFT of length L1, spectrum remap,
// inverse FFT of length L2, scale 1 / min(L1, L2)", so one kernel does all
// four line transforms:
//   row pass    -- lines are rows (contiguous), written as rows;
//   column pass -- lines are LINES adjacent columns (32-byte or wider
//                  segments per row), written the same way.
// Upsampling: column pass x -> t [h s][w], row pass t -> y.  Adjoint: row pass
// g -> t [h s][w], column pass t -> x-gradient.  Both column passes move the
// narrow side, in pieces of a few columns; the wide side moves as whole rows.
//
// Each CTA loads LINES lines into two shared-memory planes (re, im; one float
// of padding every 32), runs radix-8 or radix-16 Stockham passes (8- or
// 16-value register slots; lines up to 1024 points use 8 for more threads) --
// natural order in and out, each thread holding one or two slots in
// registers, in place between barriers -- remaps the spectrum, runs the
// inverse passes and writes the lines back.  Twiddles come from the
// correctly rounded build-time table kTw4096 (twiddle4096.cuh, read through
// the L1 cache with stride 4096 / L), so no CTA spends time building one.
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "dft_regs.cuh"
#include "line_fft.cuh"
#include "twiddle4096.cuh"

namespace pty {
namespace rs {

constexpr int cmax(int a, int b) { return a > b ? a : b; }
constexpr int cmin(int a, int b) { return a < b ? a : b; }

template <int L1, int L2, bool COL>
struct Cfg {
  static constexpr int LMAX = cmax(L1, L2);
  // row pass: 2048 values per CTA (>= 1 line); column pass: >= 4 lines
  // (32-byte segments) and 4096 values per CTA when lines are short (2 lines
  // of 4096, which would fit three CTAs per SM, ran slower: 16-byte pieces)
  static constexpr int LINES = COL ? cmax(4, 4096 / LMAX) : cmax(1, 2048 / LMAX);
  static constexpr int N = LINES * LMAX;            // values held by the CTA
  // values per register slot: 8 (radix-8 passes) for lines up to 1024 points,
  // which doubles the threads of these small, latency-bound transforms
  static constexpr int VPT = LMAX <= 1024 ? 8 : 16;
  static constexpr int NT = cmin(512, N / VPT);     // threads: one slot each, or two
  static constexpr int SPT = N / VPT / NT;          // slots per thread (1 or 2)
  static constexpr int PLANE = N + N / 32;          // padded plane length (floats)
  static constexpr size_t SMEM = size_t(2) * PLANE * 4;
  static_assert(SPT == 1 || SPT == 2, "slot count");
  static_assert(L1 >= 64 && L2 >= 64 && LMAX <= 4096, "supported line lengths");
};

PTY_DEVI int pad(int i) { return i + (i >> 5); }

// One Stockham pass of radix R over every line of length L: butterfly j of a
// line reads j + r L/R, applies exp(-+2 pi i (j mod NS) r / (NS R)) and the
// radix-R DFT, and writes (j / NS) NS R + (j mod NS) + r NS.  Twiddles are
// read from the 4096-entry table kTw4096 (global memory, L1-cached).
template <int L, int R, int NS, bool INV, int LINES, int NT, int SPT, int LMAX, int VPT>
PTY_DEVI void stockham(float* re, float* im, int t) {
  constexpr int BPL = L / R;              // butterflies per line
  constexpr int NB = LINES * BPL;         // butterflies in the CTA
  constexpr int PER = VPT / R;            // butterflies per VPT-value slot
  constexpr int NSLOT = NB / PER;         // slots in use (<= SPT * NT)
  constexpr int TWS = 4096 / (NS * R);    // twiddle table stride
  float2 v[SPT][VPT];
  int jj[SPT][PER], base[SPT][PER];
#pragma unroll
  for (int q = 0; q < SPT; ++q) {
    const int s = t + q * NT;
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      const int b = s + p * NSLOT;  // consecutive lanes -> consecutive j
      const int line = b / BPL, j = b - line * BPL;
      jj[q][p] = j;
      base[q][p] = line * LMAX;
      if (s < NSLOT) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int i = pad(base[q][p] + j + r * BPL);
          v[q][p * R + r] = make_float2(re[i], im[i]);
        }
      }
    }
  }
  __syncthreads();  // every value is read before any is overwritten
#pragma unroll
  for (int q = 0; q < SPT; ++q) {
    const int s = t + q * NT;
    if (s < NSLOT) {
#pragma unroll
      for (int p = 0; p < PER; ++p) {
        const int j = jj[q][p];
        const int k = j % NS;
        if constexpr (NS > 1) {
#pragma unroll
          for (int r = 1; r < R; ++r) {
            float2 w = __ldg(&kTw4096[k * r * TWS]);
            if constexpr (INV) w.y = -w.y;
            v[q][p * R + r] = c_mul(v[q][p * R + r], w);
          }
        }
        dft<R, INV, 1>(&v[q][p * R]);
        const int o = base[q][p] + (j / NS) * NS * R + k;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int i = pad(o + r * NS);
          re[i] = v[q][p * R + r].x;
          im[i] = v[q][p * R + r].y;
        }
      }
    }
  }
  __syncthreads();
}

// all passes of a length-L transform: radix VPT while it divides the rest, then smaller
template <int L, bool INV, int LINES, int NT, int SPT, int LMAX, int VPT, int NS = 1>
PTY_DEVI void fft_lines(float* re, float* im, int t) {
  if constexpr (NS < L) {
    constexpr int REST = L / NS;
    constexpr int R = REST >= VPT ? VPT : REST;
    stockham<L, R, NS, INV, LINES, NT, SPT, LMAX, VPT>(re, im, t);
    fft_lines<L, INV, LINES, NT, SPT, LMAX, VPT, NS * R>(re, im, t);
  }
}

template <int L1, int L2, bool COL>
__global__ void __launch_bounds__(Cfg<L1, L2, COL>::NT) k_resample(const float2* __restrict__ in,
                                                                   float2* __restrict__ out, int nlines,
                                                                   long long ld_in, long long ld_out,
                                                                   float scale) {
  using C = Cfg<L1, L2, COL>;
  constexpr int LINES = C::LINES, NT = C::NT, LMAX = C::LMAX;
  extern __shared__ __align__(16) unsigned char smem[];
  float* re = reinterpret_cast<float*>(smem);
  float* im = re + C::PLANE;
  const int t = threadIdx.x;
  const int l0 = blockIdx.x * LINES;
  // load LINES lines of length L1 (lines past the end read as zero)
  for (int idx = t; idx < LINES * L1; idx += NT) {
    int l, k;
    if constexpr (COL) {
      l = idx % LINES;
      k = idx / LINES;
    } else {
      l = idx / L1;
      k = idx - l * L1;
    }
    float2 x = make_float2(0.f, 0.f);
    if (l0 + l < nlines)
      x = COL ? __ldg(in + k * ld_in + (l0 + l)) : __ldg(in + (l0 + l) * ld_in + k);
    const int i = pad(l * LMAX + k);
    re[i] = x.x;
    im[i] = x.y;
  }
  __syncthreads();
  fft_lines<L1, false, LINES, NT, C::SPT, LMAX, C::VPT>(re, im, t);
  // spectrum remap: frequency f in [-n/2, n/2), n = min(L1, L2), from f mod L1 to f mod L2
  if constexpr (L2 > L1) {
    for (int idx = t; idx < LINES * (L1 / 2); idx += NT) {  // negative frequencies move up
      const int l = idx / (L1 / 2), k = L1 / 2 + (idx - l * (L1 / 2));
      const int a = pad(l * LMAX + k), b = pad(l * LMAX + k + (L2 - L1));
      re[b] = re[a];
      im[b] = im[a];
    }
    __syncthreads();
    for (int idx = t; idx < LINES * (L2 - L1); idx += NT) {  // the new band is empty
      const int l = idx / (L2 - L1), k = L1 / 2 + (idx - l * (L2 - L1));
      const int a = pad(l * LMAX + k);
      re[a] = 0.f;
      im[a] = 0.f;
    }
    __syncthreads();
  } else if constexpr (L2 < L1) {
    for (int idx = t; idx < LINES * (L2 / 2); idx += NT) {  // negative frequencies move down
      const int l = idx / (L2 / 2), k = L2 / 2 + (idx - l * (L2 / 2));
      const int a = pad(l * LMAX + k + (L1 - L2)), b = pad(l * LMAX + k);
      re[b] = re[a];
      im[b] = im[a];
    }
    __syncthreads();
  }
  fft_lines<L2, true, LINES, NT, C::SPT, LMAX, C::VPT>(re, im, t);
  for (int idx = t; idx < LINES * L2; idx += NT) {
    int l, k;
    if constexpr (COL) {
      l = idx % LINES;
      k = idx / LINES;
    } else {
      l = idx / L2;
      k = idx - l * L2;
    }
    if (l0 + l < nlines) {
      const int i = pad(l * LMAX + k);
      const float2 y = make_float2(re[i] * scale, im[i] * scale);
      if constexpr (COL)
        out[k * ld_out + (l0 + l)] = y;
      else
        out[(l0 + l) * ld_out + k] = y;
    }
  }
}

template <int L1, int L2, bool COL>
int launch(const float2* in, float2* out, int nlines, long long ld_in, long long ld_out, cudaStream_t s) {
  using C = Cfg<L1, L2, COL>;
  auto kern = k_resample<L1, L2, COL>;
  if (C::SMEM > 48 * 1024 &&
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(C::SMEM)) != cudaSuccess)
    return PTYCHO_ERR_LAUNCH;
  const int grid = (nlines + C::LINES - 1) / C::LINES;
  kern<<<grid, C::NT, C::SMEM, s>>>(in, out, nlines, ld_in, ld_out, 1.0f / float(L1 < L2 ? L1 : L2));
  return cudaGetLastError() == cudaSuccess ? PTYCHO_OK : PTYCHO_ERR_LAUNCH;
}

// short power-of-two lines: 64 and 128 points, s = 2 or 4
template <bool COL>
int dispatch(int l1, int l2, const float2* in, float2* out, int nlines, long long ld_in, long long ld_out,
             cudaStream_t s) {
#define PTY_RS(A, B)                                                                                \
  if (l1 == A && l2 == B) return launch<A, B, COL>(in, out, nlines, ld_in, ld_out, s);               \
  if (l1 == B && l2 == A) return launch<B, A, COL>(in, out, nlines, ld_in, ld_out, s);
  PTY_RS(64, 128) PTY_RS(64, 256) PTY_RS(128, 256) PTY_RS(128, 512)
#undef PTY_RS
  return PTYCHO_ERR_UNSUPPORTED_SIZE;
}

bool supported(int n, int N) {
  const int lo = n < N ? n : N, r = n < N ? N / n : n / N;
  return (lo == 64 || lo == 128) && lo * r == (n < N ? N : n) && (r == 2 || r == 4);
}

}  // namespace rs

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
// Measured on B200, 2048^2 to 4096^2 and back: 286 us for the four passes (49 + 77
// up, 93 + 64 down) against 668 us by padded spectra; bound by latency (issue 35 to
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
  for (int p = 1; p < s; ++p) {
    const int sp = ADJ ? -p : p;  // the adjoint's diagonal is the conjugate
    if (p > 1) __syncthreads();   // the last phase's tables are no longer read
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
          const float2 x = __ldg(at(g.in, g.ld_in, m));
          *reinterpret_cast<float4*>(at(g.out, g.ld_out, 2 * m)) = make_float4(x.x, x.y, v[e].x, v[e].y);
        } else {
          if (!COL && p == 1) *at(g.out, g.ld_out, s * m) = __ldg(at(g.in, g.ld_in, m));
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
    kern<<<need < slots ? need : slots, F::NT, F::SMEM, st>>>(g);
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
// Any line length (the canvases Recovery.py builds are multiples of 6, so
// object grids are multiples of 3 and can hold large prime factors: 498 =
// 2 * 3 * 83).  Per line: forward DFT of length L1, band remap, inverse DFT
// of length L2, scale -- the same per-axis operator as above, with the remap
// written for odd lengths too.  With n = min(L1, L2), N = max(L1, L2) and the
// band k in [lo, lo + n), lo = -floor(n/2), the reference's fftshift /
// centred pad / ifftshift puts bin k of the length-n spectrum at bin
// (k + d) mod N of the length-N one, d = floor(n/2) + floor((N-n)/2) -
// floor(N/2): d = 0 for even n, or odd n and odd N; d = -1 for odd n and even
// N (the reference's half-bin asymmetry, kept).  The adjoint gathers back.
//
// Transforms are Stockham passes with a run-time plan: radix 16, 8, 4, 2, 3,
// 5, 7 as register butterflies (dft_regs.cuh), any other prime factor p as a
// direct p-term sum per output with table twiddles.  Passes ping-pong between
// two shared-memory buffers of float2 (one float2 of padding every 16 breaks
// the stride-2^k bank conflicts of the first passes).  Twiddles:
// exp(-2 pi i j / LMAX), LMAX = max(L1, L2) = s * min(L1, L2), rounded from
// double-precision sincospi; a length-L pass reads it with stride LMAX / L.
// ---------------------------------------------------------------------------
namespace rsg {

using lfft::LinePlan;
using lfft::make_plan;
using lfft::kMaxLen;
using lfft::pad16;
using lfft::transform;
constexpr int kNT = lfft::kLineNT;
constexpr size_t kSmemCap = 200 * 1024;

struct Args {
  const float2* in;
  float2* out;
  int nlines;
  long long ld_in, ld_out;
  LinePlan f1, f2;  // forward transform (length L1), inverse transform (length L2)
  int lmax;         // max(L1, L2): twiddle table length
  int lines;        // lines per CTA
  int ls;           // padded line stride in float2
  int d, lo;        // band remap offset and lowest band frequency
  float scale;
};

template <bool COL>
__global__ void __launch_bounds__(kNT) k_resample_any(const Args g) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lines = g.lines, ls = g.ls, lmax = g.lmax;
  float2* bufA = reinterpret_cast<float2*>(smem);
  float2* bufB = bufA + size_t(lines) * ls;
  float2* tw = bufB + size_t(lines) * ls;
  const int t = threadIdx.x;
  const int l0 = blockIdx.x * lines;
  const int L1 = g.f1.L, L2 = g.f2.L;
  for (int k = t; k < lmax; k += kNT) {
    double sn, cs;
    sincospi(-2.0 * double(k) / double(lmax), &sn, &cs);
    tw[k] = make_float2(float(cs), float(sn));
  }
  for (int idx = t; idx < lines * L1; idx += kNT) {
    int l, k;
    if (COL) {
      l = idx % lines;
      k = idx / lines;
    } else {
      l = idx / L1;
      k = idx - l * L1;
    }
    float2 x = make_float2(0.f, 0.f);
    if (l0 + l < g.nlines) x = COL ? __ldg(g.in + k * g.ld_in + (l0 + l)) : __ldg(g.in + (l0 + l) * g.ld_in + k);
    bufA[l * ls + pad16(k)] = x;
  }
  __syncthreads();
  float2* spec = transform<false>(g.f1, bufA, bufB, tw, lines, ls, lmax, t);
  float2* rem = spec == bufA ? bufB : bufA;
  // band remap into the other buffer
  const int n = L1 < L2 ? L1 : L2;
  for (int idx = t; idx < lines * L2; idx += kNT) {
    const int l = idx / L2, j = idx - l * L2;
    float2 v = make_float2(0.f, 0.f);
    if (L2 >= L1) {  // pad: bin j of the long spectrum holds band frequency k, or nothing
      int k = (j - g.d - g.lo) % L2;
      if (k < 0) k += L2;
      k += g.lo;
      if (k < g.lo + n) {
        int src = k % L1;
        if (src < 0) src += L1;
        v = spec[l * ls + pad16(src)];
      }
    } else {  // crop: bin j of the short spectrum is band frequency k of the long one
      int k = (j - g.lo) % n;
      if (k < 0) k += n;
      k += g.lo;
      int src = (k + g.d) % L1;
      if (src < 0) src += L1;
      v = spec[l * ls + pad16(src)];
    }
    rem[l * ls + pad16(j)] = v;
  }
  __syncthreads();
  float2* other = rem == bufA ? bufB : bufA;
  float2* res = transform<true>(g.f2, rem, other, tw, lines, ls, lmax, t);
  for (int idx = t; idx < lines * L2; idx += kNT) {
    int l, k;
    if (COL) {
      l = idx % lines;
      k = idx / lines;
    } else {
      l = idx / L2;
      k = idx - l * L2;
    }
    if (l0 + l < g.nlines) {
      const float2 y = res[l * ls + pad16(k)];
      const float2 o = make_float2(y.x * g.scale, y.y * g.scale);
      if (COL)
        g.out[k * g.ld_out + (l0 + l)] = o;
      else
        g.out[(l0 + l) * g.ld_out + k] = o;
    }
  }
}

static size_t smem_bytes(int lines, int ls, int lmax) {
  return (size_t(2) * lines * ls + size_t(lmax)) * sizeof(float2);
}

// true when the pair of line lengths is handled (one a whole multiple of the other)
static bool supported_pair(int l1, int l2) {
  if (l1 < 1 || l2 < 1 || l1 > kMaxLen || l2 > kMaxLen) return false;
  const int lo = l1 < l2 ? l1 : l2, hi = l1 < l2 ? l2 : l1;
  return hi % lo == 0;
}

// lines of length l1 -> lines of length l2: forward DFT, band remap, inverse DFT, scale 1 / min(l1, l2)
template <bool COL>
static int launch(int l1, int l2, const float2* in, float2* out, int nlines, long long ld_in, long long ld_out,
                  cudaStream_t s) {
  if (!supported_pair(l1, l2)) return PTYCHO_ERR_UNSUPPORTED_SIZE;
  Args g{};
  if (!make_plan(l1, &g.f1) || !make_plan(l2, &g.f2)) return PTYCHO_ERR_UNSUPPORTED_SIZE;
  g.in = in;
  g.out = out;
  g.nlines = nlines;
  g.ld_in = ld_in;
  g.ld_out = ld_out;
  const int n = l1 < l2 ? l1 : l2, N = l1 < l2 ? l2 : l1;
  g.lmax = N;
  g.lo = -(n / 2);
  g.d = n / 2 + (N - n) / 2 - N / 2;
  g.scale = 1.0f / float(n);
  g.ls = pad16(N - 1) + 1;
  // lines per CTA: ~8192 values, at least 4 adjacent columns (32-byte
  // segments) in the column pass, within the shared-memory cap
  int lines = N >= 8192 ? 1 : 8192 / N;
  if (COL && lines < 4) lines = 4;
  while (lines > 1 && smem_bytes(lines, g.ls, N) > kSmemCap) --lines;
  g.lines = lines;
  const size_t smem = smem_bytes(lines, g.ls, N);
  auto kern = k_resample_any<COL>;
  static PtyDevCache attr_set;
  int dev = 0;
  for (int attempt = 0; attempt < 2; ++attempt) {
    if (!attr_set.get(&dev)) {
      if (dev < 0) return PTYCHO_ERR_LAUNCH;
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemCap)) != cudaSuccess)
        return PTYCHO_ERR_LAUNCH;
      attr_set.put(dev, 1);
    }
    kern<<<(nlines + lines - 1) / lines, kNT, smem, s>>>(g);
    if (cudaGetLastError() == cudaSuccess) return PTYCHO_OK;
    attr_set.put(dev, 0);
  }
  return PTYCHO_ERR_LAUNCH;
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
  const int l1 = ADJ ? n * s : n, l2 = ADJ ? n : n * s;
  if (rs::supported(l1, l2)) return rs::dispatch<COL>(l1, l2, in, out, nlines, ld_in, ld_out, st);
  return rsg::launch<COL>(l1, l2, in, out, nlines, ld_in, ld_out, st);
}

// s = 1: the operator is the identity
int copy_plane(const float* in, float* out, size_t n, cudaStream_t st) {
  return cudaMemcpyAsync(out, in, n * sizeof(float2), cudaMemcpyDeviceToDevice, st) == cudaSuccess
             ? PTYCHO_OK
             : PTYCHO_ERR_LAUNCH;
}

bool supported_upsample(int h, int w, int s) {
  if (h <= 0 || w <= 0 || s <= 0) return false;
  if (h > rsg::kMaxLen / s || w > rsg::kMaxLen / s) return false;
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
  if (s == 1) return copy_plane(x, y, size_t(h) * w, st);
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
  if (s == 1) return copy_plane(gy, gx, size_t(h) * w, st);
  float2* tmp = static_cast<float2*>(workspace);  // [H][w]
  int rc = axis_pass<false, true>(w, s, reinterpret_cast<const float2*>(gy), tmp, H, W, w, st);  // rows
  if (rc) return rc;
  return axis_pass<true, true>(h, s, tmp, reinterpret_cast<float2*>(gx), w, w, w, st);            // columns
}

}  // extern "C"
