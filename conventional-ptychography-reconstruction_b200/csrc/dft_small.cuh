// dft_small.cuh -- DFTs of 2 to 16 values in registers, natural order, forward.
//
// Powers of two, 3, 5 and 7 are those of dft_regs.cuh; 11 and 13 use its symmetric
// pair form; 6, 10, 12 and 15 split into coprime factors without twiddles
// (Good-Thomas: n = R2 n1 + R1 n2 mod R in, k by the Chinese remainder theorem out);
// 9 is 3 x 3 Cooley-Tukey.
#pragma once
#include "dft_regs.cuh"

namespace pty {

// cos and sin of 2 pi j / n at compile time: the angle is brought to [0, pi/4] by
// symmetry, then summed as a Taylor series in double
struct CosSin {
  double c, s;
};
__host__ __device__ constexpr CosSin cos_sin_2pi(int j, int n) {
  j %= n;
  const int oct = 8 * j / n;  // octant
  // angle = oct pi/4 + rest, rest = 2 pi (8 j - oct n) / (8 n); odd octants run backwards
  const double step = 0.78539816339744830962 * double(8 * j - oct * n) / double(n);
  const double x = (oct & 1) ? 0.78539816339744830962 - step : step;
  double c = 1.0, s = x, tc = 1.0, ts = x;
  for (int k = 1; k < 12; ++k) {
    tc *= -x * x / double((2 * k - 1) * (2 * k));
    ts *= -x * x / double((2 * k) * (2 * k + 1));
    c += tc;
    s += ts;
  }
  const bool swap = (((oct + 1) / 2) & 1) != 0;  // octants 1, 2, 5, 6
  const double u = swap ? s : c, v = swap ? c : s;
  return {(oct >= 2 && oct < 6) ? -u : u, oct >= 4 ? -v : v};
}

// cos, sin(2 pi j / n) rounded to float, as a table that unrolled code indexes
template <int N>
struct CosSinTable {
  float c[N], s[N];
};
template <int N>
__host__ __device__ constexpr CosSinTable<N> cos_sin_table() {
  CosSinTable<N> t{};
  for (int j = 0; j < N; ++j) {
    const CosSin w = cos_sin_2pi(j, N);
    t.c[j] = float(w.c);
    t.s[j] = float(w.s);
  }
  return t;
}

template <int P>
PTY_DEVI void dft_prime(float2* a) {
  constexpr int h = (P - 1) / 2;
  constexpr CosSinTable<P> w = cos_sin_table<P>();
  float2 sp[h], sm[h];
  const float2 x0 = a[0];
  float2 sum = a[0];
#pragma unroll
  for (int m = 1; m <= h; ++m) {
    sp[m - 1] = c_add(a[m], a[P - m]);
    sm[m - 1] = c_sub(a[m], a[P - m]);
    sum = c_add(sum, sp[m - 1]);
  }
#pragma unroll
  for (int r = 1; r <= h; ++r) {
    float2 A = x0, B = make_float2(0.f, 0.f);
#pragma unroll
    for (int m = 1; m <= h; ++m) {
      const float c = w.c[m * r % P], s = w.s[m * r % P];
      A = make_float2(fmaf(sp[m - 1].x, c, A.x), fmaf(sp[m - 1].y, c, A.y));
      B = make_float2(fmaf(sm[m - 1].x, s, B.x), fmaf(sm[m - 1].y, s, B.y));
    }
    a[r] = make_float2(A.x + B.y, A.y - B.x);
    a[P - r] = make_float2(A.x - B.y, A.y + B.x);
  }
  a[0] = sum;
}

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
  else if constexpr (R == 11 || R == 13) dft_prime<R>(a);
  else if constexpr (R == 12) dft_coprime<4, 3>(a);
  else if constexpr (R == 15) dft_coprime<3, 5>(a);
  else dft<R, false, 1>(a);
}

}  // namespace pty
