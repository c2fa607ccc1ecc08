// general.cu -- forward model, losses and adjoint for probes of any M x N.
//
// The fused kernels cover square 64, 128 and 256 probes.  Recovery.py takes
// the probe shape from the data (Recovery.py:290, utils/optics.py:102-112:
// any M x N window), so every other shape runs here, as three passes over a
// workspace X [B][M][N] complex64 (lines.cuh transforms of any length):
//   rows      gather P * O[window_b] and the DFT of length N along every row
//   columns   DFT of length M -> spectrum F_b; I = |F|^2 against Imeas at the
//             fftshifted index ((p + M/2) mod M, (q + N/2) mod N), the loss terms
//             of Recovery.py:294-305, and the inverse DFT of 2 dL/dI F_b, all on
//             the columns in shared memory; one FP64 loss partial per CTA
//   rows      inverse (unnormalised) DFT -> E_b = dL/dpsi_b; the pattern's loss
//             from the partials in order
// followed by the assembly of dO and dP (assemble.cu, without the (-1)^(x+y)
// factor the fused kernels fold in for even M).  The FD loss needs its
// neighbours on the shifted grid, so its columns end at F and dW, one CTA per
// pattern forms the stencil through three float planes of the workspace, and a
// second column pass starts from the gradient.  Every reduction has a fixed
// order: results are bitwise deterministic.
// Measured on B200 (batch 64 of 192^2, smooth L1, a step with its assembly): 106 us
// against 241 as seven passes with run-time radix loops (gather 9, lines 31 + 43 +
// 43 + 32, one CTA per pattern for the loss 43).  251^2, batch 32: 285 against 1815 us
// (prime length).  Bound by issue and latency: about 110 instructions a value and
// transform.
#include <cuda_runtime.h>
#include <stdint.h>

#include "assemble.cuh"
#include "fused.cuh"
#include "general.cuh"
#include "lines.cuh"

namespace pty {
namespace gen {

using ln::Plan;
constexpr int kNT = 256;
template <int LINES>
using Lines = ln::Lines<LINES, kNT>;

enum { COLS_LOSS = 0, COLS_GRAD = 1, COLS_FD = 2, COLS_FD_INV = 3, COLS_INTENSITY = 4 };

struct Args {
  FusedArgs f;
  int M, N;
  float2* X;
  int2* tlb;      // resolved windows (null: intensity only)
  float* scr;     // FD: dW, ax, ay planes [B][3][M][N]
  double* lpart;  // [B][nblk] loss partials
  int nblk;
  int loss, mode;
  int lines, gpp;  // lines per CTA, groups per pattern
  int ngroups;
  Plan plan;
};

// frame id and window of pattern b; false: skipped
PTY_DEVI bool window(const Args& g, int b, int& f, int2& c) {
  const FusedArgs& a = g.f;
  f = a.batch ? __ldg(a.batch + b) : b;
  c = make_int2(-1, -1);
  if (f < 0 || f >= a.F) return false;
  c = __ldg(a.tl + f);
  return c.x >= 0 && c.y >= 0 && c.x <= a.H - g.M && c.y <= a.W - g.N;
}

// shifted (measurement) index of spectrum element (p, q)
PTY_DEVI int shifted(int p, int q, int M, int N) {
  int u = p + M / 2, v = q + N / 2;
  if (u >= M) u -= M;
  if (v >= N) v -= N;
  return u * N + v;
}

// FP64 block sum in a fixed order (result valid in thread 0; barriers on both sides)
template <int NT>
PTY_DEVI double block_sum_nt(double x, double* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
    for (int i = 0; i < NT / 32; ++i) s += red[i];
  return s;
}

// a pattern's loss from its column blocks' partials, by one warp in a fixed order
PTY_DEVI void pattern_loss(const Args& g, int b, bool ok, int lane) {
  double s = 0.0;
  for (int i = lane; i < g.nblk; i += 32) s += g.lpart[size_t(b) * g.nblk + i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) g.f.loss_pat[b] = ok ? s / double(g.M * g.N) : (double)__int_as_float(0x7fc00000);
}

// rows: CTAs loop over groups of g.lines rows of one pattern.  Forward: gather and
// DFT.  Inverse: X -> E in place, and the losses.
template <bool INV>
__global__ void __launch_bounds__(kNT, 4) k_rows(const Args g) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int t = threadIdx.x, M = g.M, N = g.N;
  Lines<0> ln;
  ln.init(g.plan, reinterpret_cast<float2*>(smem), g.lines, t);
  const FusedArgs& a = g.f;
  for (int grp = blockIdx.x; grp < g.ngroups; grp += gridDim.x) {
    const int b = grp / g.gpp, y0 = (grp - b * g.gpp) * g.lines;
    const int rows = min(g.lines, M - y0);
    int f;
    int2 c;
    const bool ok = window(g, b, f, c);
    if (y0 == 0 && t < 32) {
      if (!INV && t == 0) {
        if (g.tlb) g.tlb[b] = ok ? c : make_int2(-1, -1);
        if (!ok) pty_raise(a.status, PTYCHO_ERR_WINDOW);
      }
      if (INV && a.loss_pat && g.lpart) pattern_loss(g, b, ok, t);
    }
    if (!ok) continue;  // uniform over the CTA
    float2* Xb = g.X + size_t(b) * M * N + size_t(y0) * N;
    const float2* Pb = a.P + y0 * N;
    const float2* Ob = a.O + size_t(c.x + y0) * a.W + c.y;
    const int n = rows * N;
#pragma unroll 4
    for (int e = t; e < n; e += kNT) {
      const int l = ln::fdiv(e, g.plan.m_n), x = e - l * N;
      float2 v;
      if constexpr (INV) v = c_conj(Xb[e]);
      else v = c_mul(__ldg(Pb + e), __ldg(Ob + size_t(l) * a.W + x));
      ln.put(g.plan, l, x, v);
    }
    ln.pad(g.plan);
    ln.run(g.plan);
#pragma unroll 4
    for (int e = t; e < n; e += kNT) {
      const int l = ln::fdiv(e, g.plan.m_n), x = e - l * N;
      const float2 v = ln.get(g.plan, l, x);
      Xb[e] = INV ? c_conj(v) : v;
    }
    __syncthreads();  // the buffers are free for the next group
  }
}

// dL/dI (without the 1/MN of the mean) and the loss term of one pixel
PTY_DEVI float pixel_loss(int loss, float I, float meas, float inv_mn, float mn, float& term) {
  if (loss == PTYCHO_LOSS_INTENSITY_GRAD) {
    term = I * meas * mn;
    return meas;
  }
  if (loss == PTYCHO_LOSS_SMOOTH_L1) {
    const float dd = I - meas, ad = fabsf(dd);
    term = ad < 1.0f ? 0.5f * dd * dd : ad - 0.5f;
    return (ad < 1.0f ? dd : copysignf(1.0f, dd)) * inv_mn;
  }
  const float Ie = I + kEps;
  term = fmaf(-meas, __logf(Ie), I);
  return (1.0f - __fdividef(meas, Ie)) * inv_mn;
}

// columns: CTAs loop over groups of LINES adjacent columns of one pattern
template <int LINES>
__global__ void __launch_bounds__(kNT, LINES == 16 ? 4 : 2) k_cols(const Args g) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double red[kNT / 32];
  const int t = threadIdx.x, M = g.M, N = g.N, MN = M * N;
  Lines<LINES> ln;
  ln.init(g.plan, reinterpret_cast<float2*>(smem), LINES, t);
  const FusedArgs& a = g.f;
  const float inv_mn = 1.0f / float(MN);
  const int cl = t % LINES;  // this thread's column of the group
  for (int grp = blockIdx.x; grp < g.ngroups; grp += gridDim.x) {
    const int b = grp / g.gpp, blk = grp - b * g.gpp;
    const int q = blk * LINES + cl;
    const bool in = q < N;
    int f;
    int2 c;
    const bool ok = window(g, b, f, c);
    float2* Xb = g.X + size_t(b) * MN + q;
    if (!ok) {  // uniform; the other outputs of a skipped pattern are written elsewhere
      if (g.mode == COLS_INTENSITY && in)
        for (int p = t / LINES; p < M; p += kNT / LINES)
          a.I_out[size_t(b) * MN + size_t(p) * N + q] = __int_as_float(0x7fc00000);
      continue;
    }
    const float* Im = a.Imeas + size_t(f) * MN;
    float* dW = g.scr + size_t(b) * 3 * MN;
#pragma unroll 4
    for (int p = t / LINES; p < M; p += kNT / LINES) {
      float2 v = in ? Xb[size_t(p) * N] : make_float2(0.f, 0.f);
      if (g.mode == COLS_FD_INV && in) {  // the stencil's adjoint on the shifted grid
        const float *ax = dW + MN, *ay = ax + MN;
        const int s = shifted(p, q, M, N), w = s % N, u = s / N;
        const float dl =
            (ax[w == 0 ? s + N - 1 : s - 1] - ax[s] + ay[u == 0 ? s + MN - N : s - N] - ay[s]) * inv_mn;
        const float I = fmaf(v.x, v.x, v.y * v.y);
        v = c_conj(c_scale(v, 2.0f * (dl * (-0.5f / sqrtf(I + kEps)))));
      }
      ln.put(g.plan, cl, p, v);
    }
    // forward (COLS_FD_INV: inverse); COLS_GRAD comes back with the gradient's columns
    // for a second transform (a loop, so that the passes' code is there once)
#pragma unroll 1
    for (int back = 0;; ++back) {
      ln.pad(g.plan);
      ln.run(g.plan);
      if (back || (g.mode != COLS_LOSS && g.mode != COLS_GRAD)) break;
      double acc = 0.0;
#pragma unroll 4
      for (int p = t / LINES; p < M; p += kNT / LINES) {
        const float2 v = ln.get(g.plan, cl, p);
        float2 w = make_float2(0.f, 0.f);
        if (in) {
          const float meas = __ldg(Im + shifted(p, q, M, N));
          const float I = fmaf(v.x, v.x, v.y * v.y);
          float term;
          const float d = pixel_loss(g.loss, I, meas, inv_mn, float(MN), term);
          acc += (double)term;
          w = c_conj(c_scale(v, 2.0f * d));
        }
        if (g.mode == COLS_GRAD) ln.put(g.plan, cl, p, w);
      }
      const double tot = block_sum_nt<kNT>(acc, red);
      if (t == 0) g.lpart[size_t(b) * g.nblk + blk] = tot;
      if (g.mode == COLS_LOSS) break;
    }
    if (g.mode != COLS_LOSS && in)
      for (int p = t / LINES; p < M; p += kNT / LINES) {
        const float2 v = ln.get(g.plan, cl, p);
        if (g.mode == COLS_GRAD || g.mode == COLS_FD_INV) {
          Xb[size_t(p) * N] = c_conj(v);
          continue;
        }
        const float I = fmaf(v.x, v.x, v.y * v.y);
        const int s = shifted(p, q, M, N);
        if (g.mode == COLS_INTENSITY) {
          a.I_out[size_t(b) * MN + s] = I;
        } else {
          Xb[size_t(p) * N] = v;
          dW[s] = sqrtf(__ldg(Im + s) + kEps) - sqrtf(I + kEps);
        }
      }
    __syncthreads();  // the buffers are free for the next group
  }
}

// FD loss of one pattern per CTA on the shifted grid: dW -> ax = Rx / G, ay = Ry / G
constexpr int kStencilNT = 1024;
__global__ void __launch_bounds__(kStencilNT) k_stencil(const Args g, int grad) {
  __shared__ double red[kStencilNT / 32];
  const int b = blockIdx.x, M = g.M, N = g.N, MN = M * N;
  int f;
  int2 c;
  const bool ok = window(g, b, f, c);
  if (!ok) {  // uniform
    if (threadIdx.x == 0 && g.f.loss_pat) g.f.loss_pat[b] = (double)__int_as_float(0x7fc00000);
    return;
  }
  float* dW = g.scr + size_t(b) * 3 * MN;
  float *ax = dW + MN, *ay = ax + MN;
  double acc = 0.0;
  for (int s = threadIdx.x; s < MN; s += kStencilNT) {
    const int u = s / N, v = s - u * N;
    const float d = dW[s];
    const float rx = dW[v + 1 == N ? s + 1 - N : s + 1] - d;
    const float ry = dW[u + 1 == M ? v : s + N] - d;
    const float G = sqrtf(fmaf(rx, rx, fmaf(ry, ry, kEps)));
    acc += (double)G;
    if (grad) {
      ax[s] = rx / G;
      ay[s] = ry / G;
    }
  }
  const double tot = block_sum_nt<kStencilNT>(acc, red);
  if (threadIdx.x == 0 && g.f.loss_pat) g.f.loss_pat[b] = tot / double(MN);
}

// losses without gradients: one warp per pattern
__global__ void __launch_bounds__(32) k_pattern_loss(const Args g) {
  int f;
  int2 c;
  const bool ok = window(g, blockIdx.x, f, c);
  pattern_loss(g, blockIdx.x, ok, threadIdx.x);
}

// persistent launch: one CTA per resident slot at most
template <typename K>
static int launch(K kern, PtyDevCache& attr, const Args& g, size_t smem, cudaStream_t s) {
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
    const int per_sm = int(233472 / (smem + 1024 + 256));
    const int slots = nsm * (per_sm < 1 ? 1 : (per_sm > 4 ? 4 : per_sm));
    kern<<<g.ngroups < slots ? g.ngroups : slots, kNT, smem, s>>>(g);
    if (cudaGetLastError() == cudaSuccess) return PTYCHO_OK;
    attr.put(dev, 0);  // e.g. the attribute was lost with a device reset: set up again once
  }
  return PTYCHO_ERR_LAUNCH;
}

static void set_groups(Args* g, int per_pattern_lines) {
  g->gpp = (per_pattern_lines + g->lines - 1) / g->lines;
  g->ngroups = g->gpp * g->f.B;
}

template <bool INV>
static int run_rows(Args g, cudaStream_t s) {
  if (!ln::make_plan(g.N, 0, &g.plan)) return PTYCHO_ERR_UNSUPPORTED_SIZE;
  // about 3072 values per CTA (four CTAs per SM), never more rows than there are; half
  // of that where the batch would not fill the slots (148 x 4): steps of 1 x 150^2 47.6 ->
  // 43.5 us, 32 x 100 x 120 51.7 -> 47.7, 64 x 96^2 60.0 -> 58.1.  On full grids the
  // larger CTA is better: 40 x 320^2 171 against 183, 64 x 192^2 91 against 96
  int lines = 0;
  for (int values = 3072; values >= 1536; values /= 2) {
    lines = values / g.plan.m;
    lines = lines < 1 ? 1 : (lines > g.M ? g.M : lines);
    while (lines > 1 && ln::smem_bytes(g.plan, lines, 0) > ln::kSmemCap) --lines;
    g.lines = lines;
    set_groups(&g, g.M);
    if (g.ngroups >= 148 * 4) break;
  }
  static PtyDevCache attr;
  return launch(k_rows<INV>, attr, g, ln::smem_bytes(g.plan, lines, 0), s);
}

// columns per CTA: 16 (128-byte pieces), 4 for long lines, 1 for the longest; a
// function of the probe shape alone, so the loss partials' count is too
static int col_lines(const Plan& p) {
  if (ln::smem_bytes(p, 16, 0) <= 100 * 1024) return 16;
  return ln::smem_bytes(p, 4, 0) <= ln::kSmemCap ? 4 : 1;
}

static int run_cols(Args g, int mode, cudaStream_t s) {
  if (!ln::make_plan(g.M, 0, &g.plan)) return PTYCHO_ERR_UNSUPPORTED_SIZE;
  g.mode = mode;
  g.lines = col_lines(g.plan);
  set_groups(&g, g.N);
  const size_t smem = ln::smem_bytes(g.plan, g.lines, 0);
  static PtyDevCache a16, a4, a1;
  if (g.lines == 16) return launch(k_cols<16>, a16, g, smem, s);
  if (g.lines == 4) return launch(k_cols<4>, a4, g, smem, s);
  return launch(k_cols<1>, a1, g, smem, s);
}

static bool make_args(Args* g, const FusedArgs& a, int M, int N, float2* X) {
  *g = Args{};
  g->f = a;
  g->M = M;
  g->N = N;
  g->X = X;
  Plan p;
  if (!ln::make_plan(M, 0, &p)) return false;
  const int l = col_lines(p);
  g->nblk = (N + l - 1) / l;
  return true;
}

}  // namespace gen

bool general_supported(int M, int N) { return M >= 1 && N >= 1 && M <= kGeneralMaxDim && N <= kGeneralMaxDim; }

int general_forward_intensity(const FusedArgs& a, int M, int N, float2* X, cudaStream_t s) {
  using namespace gen;
  Args g;
  if (!make_args(&g, a, M, N, X)) return PTYCHO_ERR_UNSUPPORTED_SIZE;
  const int st = run_rows<false>(g, s);
  return st ? st : run_cols(g, COLS_INTENSITY, s);
}

int general_fwd_adj(const FusedArgs& a, int M, int N, int loss, bool grad, float2* X, float* scr, int2* tlb,
                    cudaStream_t s) {
  using namespace gen;
  Args g;
  if (!make_args(&g, a, M, N, X)) return PTYCHO_ERR_UNSUPPORTED_SIZE;
  g.tlb = tlb;
  g.loss = loss;
  g.scr = scr;
  const bool fd = loss == PTYCHO_LOSS_FD;
  if (!fd) g.lpart = reinterpret_cast<double*>(scr);  // the FD planes' place, unused by the other losses
  int st = run_rows<false>(g, s);
  if (!st) st = run_cols(g, fd ? COLS_FD : (grad ? COLS_GRAD : COLS_LOSS), s);
  if (st) return st;
  if (fd) {
    k_stencil<<<a.B, kStencilNT, 0, s>>>(g, grad ? 1 : 0);
    if (cudaGetLastError() != cudaSuccess) return PTYCHO_ERR_LAUNCH;
    if (grad) st = run_cols(g, COLS_FD_INV, s);
  } else if (!grad && a.loss_pat) {
    k_pattern_loss<<<a.B, 32, 0, s>>>(g);
    if (cudaGetLastError() != cudaSuccess) return PTYCHO_ERR_LAUNCH;
  }
  if (st || !grad) return st;
  return run_rows<true>(g, s);
}

}  // namespace pty
