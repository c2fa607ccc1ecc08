// dft_small.cuh -- DFTs of 2 to 16 values in registers, natural order, forward.
//
// Powers of two, 3, 5 and 7 are those of dft_regs.cuh; 11 and 13 use its symmetric
// pair form; 6, 10, 12 and 15 split into coprime factors without twiddles
// (Good-Thomas: n = R2 n1 + R1 n2 mod R in, k by the Chinese remainder theorem out);
// 9 is 3 x 3 Cooley-Tukey.
#pragma once
#include "dft_regs.cuh"

namespace pty {

template <int R1, int R2>
PTY_DEVI void dft_coprime(float2* a) {
  constexpr int R = R1 * R2;
  float2 t[R];
#pragma unroll
  for (int n2 = 0; n2 < R2; ++n2)
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) t[n2 * R1 + n1] = a[(R2 * n1 + R1 * n2) % R];
#pragma unroll
  for (int n2 = 0; n2 < R2; ++n2) dft<R1, false, 1>(t + n2 * R1);
#pragma unroll
  for (int k1 = 0; k1 < R1; ++k1) dft<R2, false, R1>(t + k1);
#pragma unroll
  for (int k = 0; k < R; ++k) a[k] = t[(k % R2) * R1 + k % R1];
}

PTY_DEVI void dft9(float2* a) {
  constexpr CosSinTable<9> w = cos_sin_table<9>();
  float2 t[9];
#pragma unroll
  for (int n2 = 0; n2 < 3; ++n2)
#pragma unroll
    for (int n1 = 0; n1 < 3; ++n1) t[n2 * 3 + n1] = a[3 * n1 + n2];
#pragma unroll
  for (int n2 = 0; n2 < 3; ++n2) dft<3, false, 1>(t + n2 * 3);  // k1 at t[n2 * 3 + k1]
#pragma unroll
  for (int n2 = 1; n2 < 3; ++n2)
#pragma unroll
    for (int k1 = 1; k1 < 3; ++k1)
      t[n2 * 3 + k1] = c_mul(t[n2 * 3 + k1], make_float2(w.c[n2 * k1], -w.s[n2 * k1]));
#pragma unroll
  for (int k1 = 0; k1 < 3; ++k1) dft<3, false, 3>(t + k1);  // k2 at t[k2 * 3 + k1]
#pragma unroll
  for (int k1 = 0; k1 < 3; ++k1)
#pragma unroll
    for (int k2 = 0; k2 < 3; ++k2) a[k1 + 3 * k2] = t[k2 * 3 + k1];
}

template <int R>
PTY_DEVI void dft_any(float2* a) {
  if constexpr (R == 6) dft_coprime<2, 3>(a);
  else if constexpr (R == 9) dft9(a);
  else if constexpr (R == 10) dft_coprime<2, 5>(a);
  else if constexpr (R == 11 || R == 13) dft_odd<R, false, 1>(a);
  else if constexpr (R == 12) dft_coprime<4, 3>(a);
  else if constexpr (R == 15) dft_coprime<3, 5>(a);
  else dft<R, false, 1>(a);
}

}  // namespace pty
