// cluster_small.cuh -- forward / loss / adjoint with one pattern per thread-block
// cluster of CL = M / 16 CTAs (M = 64, 128, 256: 4, 8, 16 CTAs): small batches, the
// FD loss at M = 256, and M = 256 intensities without a workspace.
//
// Same contract as the fused kernels (fused.cuh).  Those hold a pattern of M = 64 or
// 128 in one SM, so a batch of ten leaves the rest of the chip idle and its step
// is one pattern's serial latency.  Here a CTA holds RW = M / CL rows, then as many
// columns, a thread 16 values:
//   rows      (-1)^(x+y) P O[window], DFT along x in registers (16 x M/16)
//   exchange  value (y, fx) to the CTA of column fx / RW, through distributed shared
//             memory, between two cluster barriers
//   columns   DFT along y, loss, 2 dL/dI F, inverse DFT along y
//   exchange  back to the CTA of row y / RW
//   rows      inverse DFT along x -> E'
// The per-pattern FP64 loss is the CTAs' partials in rank order.  The FD loss takes
// its neighbour columns' dW and Rx / G from the CTAs on either side (two more
// cluster barriers).  Every sum has a fixed order: results are bitwise
// deterministic.
// Bound by latency: two global round trips, four line transforms and two (FD: four)
// cluster barriers.  Whole captured steps on B200 against a pattern per SM: 10 patterns
// of 128^2 33.2 -> 23.0 us, FD 49.8 -> 27.1; 10 of 256^2, FD, 78.4 -> 33.5 (a cluster of
// four, 32 values a thread); an eager call of that takes 86 us of host time either way.  small_batch_max (fused.cuh) says which batches come here.
// Sixteen CTAs are more than the portable eight: a partition of the chip may not hold
// them together.  M = 256 runs eight CTAs of 32 rows there (large_clusters, fused.cuh):
// on a whole B200 10 FD patterns 30.8 us against 26.9, 200 355 : 343, intensities
// without scratch 512 frames 271 : 246, 10 equal.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "dft_regs.cuh"
#include "fused.cuh"
#include "launch_retry.cuh"

namespace pty {
namespace csm {

template <int M, int CL>
struct Cfg {
  static constexpr int C = M / 16;     // last radix of a line, lanes of a row
  static constexpr int RW = M / CL;    // rows, then columns, of a CTA
  static constexpr int NT = RW * C;
  static constexpr int G = 16 / C;     // radix-C groups per thread
  static constexpr int K = RW / 16;
  static_assert(RW % 16 == 0, "rows of a CTA");
  // row transposes: value (a, q) of a row at a (C + 1) + q, rows PR apart, so that a
  // half-warp's 8-byte accesses are free of conflicts both ways
  static constexpr int PR = C == 4 ? 84 : (C == 8 ? 152 : 272);
  static constexpr int PC = M + C;     // row pitch of the returned rows
  static constexpr int TW = 0;         // float2 offsets in shared memory
  static constexpr int A = TW + M;                                  // columns, [y][RW]
  static constexpr int B = A + M * RW;                              // transposes
  static constexpr int R = B + (RW * PR > M * RW ? RW * PR : M * RW);  // returned rows, [RW][PC]
  static constexpr int HALO = R + RW * PC;                          // FD: two columns of floats
  static constexpr int RED = HALO + M;                              // doubles: warp sums, then CTA partials
  static constexpr size_t SMEM = size_t(RED + NT / 32 + CL) * sizeof(float2);
  static_assert(SMEM <= 232448, "shared memory");
};

PTY_DEVI uint32_t mapa(uint32_t saddr, uint32_t rank) {
  uint32_t out;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(saddr), "r"(rank));
  return out;
}
PTY_DEVI void st_remote(uint32_t addr, float2 v) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(v.x), "f"(v.y) : "memory");
}
PTY_DEVI void st_remote(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
PTY_DEVI void st_remote(uint32_t addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
PTY_DEVI void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
PTY_DEVI void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// DFT of one line: in, thread q holds x[q + C e] in v[e]; out, value g C + k is
// frequency (q + C g) + 16 k.  xchg(v): the line's transpose from v[a] = (a, q) to
// v[g C + k] = (a = q + C g, k).
template <int C, class X>
PTY_DEVI void line_fwd(float2 (&v)[16], int q, const float2* tw, X xchg) {
  dft16<false, 1>(v);
#pragma unroll
  for (int a = 1; a < 16; ++a) v[a] = c_mul(v[a], tw[a * C + q]);
  xchg(v);
#pragma unroll
  for (int g = 0; g < 16 / C; ++g) dft<C, false, 1>(v + g * C);
}
// the way back (unnormalised inverse); xchg the other way
template <int C, class X>
PTY_DEVI void line_inv(float2 (&v)[16], int q, const float2* tw, X xchg) {
#pragma unroll
  for (int g = 0; g < 16 / C; ++g) dft<C, true, 1>(v + g * C);
  xchg(v);
#pragma unroll
  for (int a = 1; a < 16; ++a) v[a] = c_mul(v[a], c_conj(tw[a * C + q]));
  dft16<true, 1>(v);
}

template <int M, int CL, int MODE, int LOSS>
__global__ void __launch_bounds__(Cfg<M, CL>::NT) k_small(const FusedArgs a) {
  using F = Cfg<M, CL>;
  constexpr bool ADJ = MODE == MODE_ADJ;
  constexpr int C = F::C, NT = F::NT, RW = F::RW, K = F::K;
  extern __shared__ __align__(16) float2 sm[];
  float2 *tw = sm + F::TW, *bufA = sm + F::A, *bufB = sm + F::B, *bufR = sm + F::R;
  float* halo_p = reinterpret_cast<float*>(sm + F::HALO);  // column 16's dW
  float* halo_m = halo_p + M;                              // column -1's Rx / G
  double* red = reinterpret_cast<double*>(sm + F::RED);
  double* parts = red + NT / 32;  // rank 0: the CTAs' loss partials
  const int t = threadIdx.x, b = blockIdx.x / CL, rank = blockIdx.x % CL;  // clusters of CL adjacent CTAs
  if (a.done && b == 0)
    for (int i = rank * NT + t; i < a.ndone; i += CL * NT) a.done[i] = 0u;
  const int f = a.batch ? __ldg(a.batch + b) : b;
  int2 w = make_int2(-1, -1);
  bool ok = f >= 0 && f < a.F;
  if (ok) {
    w = __ldg(a.tl + f);
    ok = w.x >= 0 && w.y >= 0 && w.x <= a.H - M && w.y <= a.W - M;
  }
  if (rank == 0 && t == 0) {
    if (ADJ) a.tlb[b] = ok ? w : make_int2(-1, -1);
    if (!ok) {
      pty_raise(a.status, PTYCHO_ERR_WINDOW);
      if (MODE != MODE_INTENSITY && a.loss_pat) a.loss_pat[b] = (double)__int_as_float(0x7fc00000);
    }
  }
  if (!ok) {  // uniform over the cluster, before any of its barriers
    if (MODE == MODE_INTENSITY)
      for (int i = t; i < RW * M; i += NT)
        a.I_out[size_t(b) * M * M + size_t(rank) * RW * M + i] = __int_as_float(0x7fc00000);
    return;
  }
  cluster_arrive();  // waited for below: no remote store before every CTA runs

  // ---- rows: thread (r, q) --------------------------------------------------------
  float2 v[16];
  {
    const int r = t / C, q = t % C, y = RW * rank + r;
    const float2* Or = a.O + size_t(w.x + y) * a.W + w.y + q;
    const float2* Pr = a.P + y * M + q;
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      const unsigned sg = unsigned((q + C * e + y) & 1) << 31;
      float2 p = __ldg(Pr + C * e);
      p.x = __uint_as_float(__float_as_uint(p.x) ^ sg);
      p.y = __uint_as_float(__float_as_uint(p.y) ^ sg);
      v[e] = c_mul(p, __ldg(Or + C * e));
    }
    if (t < M) {  // W_M^(q a) at a C + q
      float s, c;
      sincospif(-float((t / C) * (t % C)) * (2.0f / float(M)), &s, &c);
      tw[t] = make_float2(c, s);
    }
    __syncthreads();
    float2* row = bufB + r * F::PR;
    line_fwd<C>(v, q, tw, [&](float2(&x)[16]) {
#pragma unroll
      for (int k = 0; k < 16; ++k) row[k * (C + 1) + q] = x[k];
      __syncwarp();
#pragma unroll
      for (int g = 0; g < F::G; ++g)
#pragma unroll
        for (int k = 0; k < C; ++k) x[g * C + k] = row[(q + C * g) * (C + 1) + k];
    });
    cluster_wait();
    // frequency (q + C g) + 16 k goes to CTA k / K, column 16 (k % K) + q + C g, row y
    const uint32_t base = smem_u32(bufA + y * RW + q);
#pragma unroll
    for (int k = 0; k < C; ++k) {
      const uint32_t dst = mapa(base, k / K) + 16 * (k % K) * 8;
#pragma unroll
      for (int g = 0; g < F::G; ++g) st_remote(dst + C * g * 8, v[g * C + k]);
    }
  }
  // ---- columns: thread (q, col); value g C + k is row frequency (q + C g) + 16 k ---------
  const int col = t % RW, q = t / RW, fx = RW * rank + col;
  auto fy = [&](int i) { return q + C * (i / C) + 16 * (i % C); };
  float meas[16];
  if constexpr (MODE != MODE_INTENSITY) {  // on its way during the exchange and the transform
    const float* Im = a.Imeas + size_t(f) * M * M + fx;
#pragma unroll
    for (int i = 0; i < 16; ++i) meas[i] = __ldg(Im + fy(i) * M);
  }
  cluster_arrive();
  cluster_wait();
#pragma unroll
  for (int e = 0; e < 16; ++e) v[e] = bufA[(q + C * e) * RW + col];
  line_fwd<C>(v, q, tw, [&](float2(&x)[16]) {
#pragma unroll
    for (int k = 0; k < 16; ++k) bufB[(k * C + q) * RW + col] = x[k];
    __syncthreads();
#pragma unroll
    for (int g = 0; g < F::G; ++g)
#pragma unroll
      for (int k = 0; k < C; ++k) x[g * C + k] = bufB[((q + C * g) * C + k) * RW + col];
  });
  if constexpr (MODE == MODE_INTENSITY) {  // no remote access is left after the barrier above
    float* Io = a.I_out + size_t(b) * M * M + fx;
#pragma unroll
    for (int i = 0; i < 16; ++i) Io[fy(i) * M] = fmaf(v[i].x, v[i].x, v[i].y * v[i].y);
    return;
  }
  constexpr float inv_mn = 1.0f / float(M * M);
  float part[16];
  if constexpr (LOSS != PTYCHO_LOSS_FD) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float I = fmaf(v[i].x, v[i].x, v[i].y * v[i].y);
      float gq;
      if constexpr (LOSS == PTYCHO_LOSS_INTENSITY_GRAD) {
        part[i] = I * meas[i] * float(M * M);
        v[i] = c_scale(v[i], 2.0f * meas[i]);
      } else {
        if constexpr (LOSS == PTYCHO_LOSS_SMOOTH_L1) {
          const float dd = I - meas[i];
          const float ad = fabsf(dd);
          part[i] = ad < 1.0f ? 0.5f * dd * dd : ad - 0.5f;
          gq = ad < 1.0f ? dd : copysignf(1.0f, dd);
        } else {
          const float Ie = I + kEps;
          part[i] = fmaf(-meas[i], __logf(Ie), I);
          gq = 1.0f - __fdividef(meas[i], Ie);
        }
        v[i] = c_scale(v[i], 2.0f * gq * inv_mn);
      }
    }
  } else {
    // 5-point circular stencil on the natural frequency grid.  dW: [M][RW] in bufR
    // (free until the rows return, which is after these barriers); Rx / G and Ry / G
    // in bufA, whose columns have been read
    float* dW = reinterpret_cast<float*>(bufR);
    float *ax = reinterpret_cast<float*>(bufA), *ay = ax + M * RW;
    const int up = rank == 0 ? CL - 1 : rank - 1, dn = rank == CL - 1 ? 0 : rank + 1;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float I = fmaf(v[i].x, v[i].x, v[i].y * v[i].y);
      const float d = sqrtf(meas[i] + kEps) - sqrtf(I + kEps);
      dW[fy(i) * RW + col] = d;
      if (col == 0) st_remote(mapa(smem_u32(halo_p + fy(i)), up), d);
    }
    cluster_arrive();
    cluster_wait();
    float gy[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int y = fy(i);
      const float d = dW[y * RW + col];
      const float rx = (col == RW - 1 ? halo_p[y] : dW[y * RW + col + 1]) - d;
      const float ry = dW[((y + 1) & (M - 1)) * RW + col] - d;
      const float G = sqrtf(fmaf(rx, rx, fmaf(ry, ry, kEps)));
      part[i] = G;
      if constexpr (ADJ) {
        const float qx = rx / G;
        gy[i] = ry / G;
        ax[y * RW + col] = qx;
        ay[y * RW + col] = gy[i];
        if (col == RW - 1) st_remote(mapa(smem_u32(halo_m + y), dn), qx);
      }
    }
    if constexpr (ADJ) {
      cluster_arrive();
      cluster_wait();
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int y = fy(i);
        const float left = col == 0 ? halo_m[y] : ax[y * RW + col - 1];
        const float dl = ((left - ax[y * RW + col]) + ay[((y - 1) & (M - 1)) * RW + col] - gy[i]) * inv_mn;
        const float I = fmaf(v[i].x, v[i].x, v[i].y * v[i].y);
        v[i] = c_scale(v[i], 2.0f * (dl * (-0.5f / sqrtf(I + kEps))));
      }
    }
  }
#pragma unroll
  for (int s = 1; s < 16; s <<= 1)
#pragma unroll
    for (int i = 0; i < 16; i += 2 * s) part[i] += part[i + s];
  const double tot = block_sum<NT>((double)part[0], red);
  if (t == 0) st_remote(mapa(smem_u32(parts + rank), 0), tot);
  if constexpr (ADJ) {
    line_inv<C>(v, q, tw, [&](float2(&x)[16]) {
      // (block_sum's barriers: every thread has read its column of bufB)
#pragma unroll
      for (int g = 0; g < F::G; ++g)
#pragma unroll
        for (int k = 0; k < C; ++k) bufB[((q + C * g) * C + k) * RW + col] = x[g * C + k];
      __syncthreads();
#pragma unroll
      for (int k = 0; k < 16; ++k) x[k] = bufB[(k * C + q) * RW + col];
    });
    // row y = q + C e goes to CTA y / RW, frequency fx
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      const int y = q + C * e;
      st_remote(mapa(smem_u32(bufR + (y % RW) * F::PC + fx), y / RW), v[e]);
    }
  }
  cluster_arrive();
  cluster_wait();
  if (rank == 0 && t == 0 && a.loss_pat) {
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < CL; ++i) s += parts[i];
    a.loss_pat[b] = s / double(M * M);
  }
  // ---- rows back: thread (r, q) ----------------------------------------------------
  if constexpr (ADJ) {
    const int r = t / C, qr = t % C;
    const float2* in = bufR + r * F::PC;
#pragma unroll
    for (int g = 0; g < F::G; ++g)
#pragma unroll
      for (int k = 0; k < C; ++k) v[g * C + k] = in[qr + C * g + 16 * k];
    float2* row = bufB + r * F::PR;
    line_inv<C>(v, qr, tw, [&](float2(&x)[16]) {
#pragma unroll
      for (int g = 0; g < F::G; ++g)
#pragma unroll
        for (int k = 0; k < C; ++k) row[(qr + C * g) * (C + 1) + k] = x[g * C + k];
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 16; ++k) x[k] = row[k * (C + 1) + qr];
    });
    float2* Er = a.Eout + size_t(b) * M * M + (RW * rank + r) * M + qr;
#pragma unroll
    for (int e = 0; e < 16; ++e) Er[C * e] = v[e];
  }
}

// launch configuration of b patterns; `at` is its one attribute
template <int M, int CL>
static cudaLaunchConfig_t config(int b, cudaLaunchAttribute* at, cudaStream_t s) {
  using F = Cfg<M, CL>;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(CL) * unsigned(b));
  cfg.blockDim = dim3(F::NT);
  cfg.dynamicSmemBytes = F::SMEM;
  cfg.stream = s;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = CL;
  at->val.clusterDim.y = 1;
  at->val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

template <int M, int CL, int MODE, int LOSS>
static bool set_attributes() {
  auto kern = k_small<M, CL, MODE, LOSS>;
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(Cfg<M, CL>::SMEM)) == cudaSuccess &&
         (CL <= 8 || cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess);
}

// whether the current device can hold a cluster of this kernel
template <int M, int CL, int MODE, int LOSS>
static bool fits() {
  cudaLaunchAttribute at{};
  const cudaLaunchConfig_t cfg = config<M, CL>(1, &at, nullptr);
  int n = 0;
  const bool ok = set_attributes<M, CL, MODE, LOSS>() &&
                  cudaOccupancyMaxActiveClusters(&n, k_small<M, CL, MODE, LOSS>, &cfg) == cudaSuccess;
  if (!ok) cudaGetLastError();
  return ok && n > 0;
}

template <int M, int CL, int MODE, int LOSS>
static int launch(const FusedArgs& a, cudaStream_t s) {
  cudaLaunchAttribute at{};
  const cudaLaunchConfig_t cfg = config<M, CL>(a.B, &at, s);
  static PtyDevCache attr;  // attributes set
  int dev = 0;
  const bool ok = launch_retry(
      [&](bool again) {
        if (!again && attr.get(&dev)) return true;
        if (dev < 0 || !set_attributes<M, CL, MODE, LOSS>()) return false;
        attr.put(dev, 1);
        return true;
      },
      [&] { return int(cudaLaunchKernelEx(&cfg, k_small<M, CL, MODE, LOSS>, a)); },
      [] { return int(cudaGetLastError()); });
  return ok ? PTYCHO_OK : PTYCHO_ERR_LAUNCH;
}

}  // namespace csm
}  // namespace pty
