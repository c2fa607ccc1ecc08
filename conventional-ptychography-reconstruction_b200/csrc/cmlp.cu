// cmlp.cu -- complex-exponential MLP on the 5th-generation tensor cores (tcgen05).
//
// Replaces ComplexMLP.net of models/complex_inr.py:6-82 (as called through
// _get_complex_output, :308-314) for the configuration every reference config
// uses: 32 input features (16 hash levels x 2), hidden_features 64 (32
// complex units), hidden_layers 2, one complex output:
//   z1 = W1 x + b1 (real 32x32),          h1 = exp(i w1 z1)
//   z2 = W2 h1 + b2 (complex 32x32),      h2 = exp(i w2 z2)
//   z3 = W3 h2 + b3,                      h3 = exp(i w3 z3)
//   y  = Wo h3 + bo (complex 1x32).
// A complex layer acts on [Re h; Im h] as the real 64x64 block [[A,-B],[B,A]]
// (W = A + iB).  Operands are BF16 in shared memory, accumulators FP32 in
// tensor memory; the hidden activations entering layer 2, layer 3 and the
// output layer are split into bf16(h) + bf16(h - bf16(h)), two MMAs into one
// accumulator (with h rounded once to BF16, training on 1e3-photon Poisson data
// stalled at about 3x the residual an FP32 MLP reached).
//
// A tile of 128 coordinates is a chain of dependent MMA -> elementwise steps, so
// the SM is kept busy by several tiles in flight, and the chain is kept short:
//  * the output layer's MMA runs with the next tile's first one; G_h3 = Wo_r^T G_y
//    comes with z3;
//  * sin, cos and exp run at 16 results a clock, and rintf and the conversion of a
//    single float to BF16 share their unit: the range reduction rounds by adding
//    1.5 2^23 and conversions are done in pairs, off that unit;
//  * the arithmetic between is packed two floats to an instruction.
// One CTA per SM with several slots of 256 threads, each with a tile, buffers,
// TMEM columns and a barrier of its own.  Forward (k_cmlp_fwd): four slots, three
// MMA steps a tile.  Backward (k_cmlp_bwd): two slots, six MMA steps a tile:
//   z1 | z2 | z3, G_h3 -> G_z3 | G_h2 -> G_z2 | G_h1 -> G_z1 | G_x
//   G_z = conj(i w h) G_h (complex layers), G_z1 = Re(conj(G_h1) i w1 h1),
//   G_h(prev) = W_r^T G_z, G_x = W1^T G_z1,
// with the weight gradients
//   sum_c [G_z3 | G_z2]_c^T [h2 | h1 | 1]_c,   sum_c G_z1_c^T [x | 1]_c,
//   sum_c G_y_c^T [h3 | 1]_c
// accumulated in TMEM across all the CTA's tiles in tile order (the appended
// ones column yields the bias gradients).  In a tile's 256 threads, warp w
// reads TMEM lane quarter w & 3 (tile rows 32 (w & 3) .. +31) and does the
// elementwise work of half w >> 2 of each layer's complex units.
// Measured on B200, 4,194,304 coordinates: forward 523 us (820 as four serial
// steps, two CTAs per SM, rintf and single conversions), backward 1322 us (1905
// as nine serial steps, one tile in flight).  The forward is bound by its 256
// sin / cos / exp results per coordinate (236 us) and issue (65 %); the backward
// by latency with two tiles in flight (issue 39 %), which is all that shared
// memory (100 KB a tile) and TMEM (256 accumulator columns + 128 a tile) hold.
//
// Each CTA writes its raw accumulators once; k_cmlp_reduce sums the CTA
// partials in a fixed order and folds the real-form blocks back into complex
// gradients (G_W = (P+S) + i(R-Q) for [[P,Q],[R,S]]) -- deterministic, no
// atomics.  Gradients follow torch's complex convention.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "async_copy.cuh"
#include "common.cuh"
#include "tc_umma.cuh"

namespace pty {
namespace cm {

constexpr int GRP = 2048;  // one group of 8 bf16 features x 128 rows

// ---- packed operand blob (bytes) ---------------------------------------------
constexpr int S_W1 = 0;             // W1  [32 out][32 in]   K-major, LBO 512
constexpr int S_W2 = S_W1 + 2048;   // Wr2 [64][64]          LBO 1024
constexpr int S_W3 = S_W2 + 8192;   // Wr3 [64][64]
constexpr int S_WO = S_W3 + 8192;   // Wor [16][64] (rows 0,1 used), LBO 256
constexpr int kWBytes = S_WO + 2048;  // 20480

// ---- fp32 parameter block (floats) ------------------------------------------
constexpr int P_B1 = 0, P_B2R = 32, P_B2I = 64, P_B3R = 96, P_B3I = 128, P_BOR = 160, P_BOI = 161,
              P_W1 = 162, P_W2 = 163, P_W3 = 164, kParFloats = 168;
constexpr int kPackedBytes = kWBytes + kParFloats * 4;  // 21152
// the kernels' copy of it: the parameters, then Re and Im of the BF16 output weights
constexpr int P_WOR = kParFloats, P_WOI = P_WOR + 32, kParSmem = P_WOI + 32;

// ---- raw per-CTA gradient partials (floats) ----------------------------------
constexpr int R_W3 = 0, R_B3 = 4096, R_W2 = 4160, R_B2 = 8256, R_W1 = 8320, R_B1 = 9344, R_WO = 9376,
              R_BO = 9504, R_OM = 9506, kPartFloats = 9512;
// ---- final gradient blob (floats; complex entries interleaved re, im) --------
constexpr int G_W1 = 0, G_B1 = 1024, G_OM1 = 1056, G_W2 = 1058, G_B2 = 3106, G_OM2 = 3170, G_W3 = 3172,
              G_B3 = 5220, G_OM3 = 5284, G_WO = 5286, G_BO = 5350, kGradFloats = 5352;

// byte offset of (row c, feature f) in an activation buffer
PTY_DEVI int cm_off(int c, int f) { return (f >> 3) * GRP + (c >> 3) * 128 + (c & 7) * 16 + (f & 7) * 2; }
// byte offset of (n, k) in a weight matrix with nout rows (K-major view)
__host__ __device__ constexpr int wm_off(int n, int k, int nout) {
  return (k >> 3) * (nout * 16) + (n >> 3) * 128 + (n & 7) * 16 + (k & 7) * 2;
}

PTY_DEVI uint32_t pack_bf16x2(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
// Two floats in one 64-bit register pair: add, multiply and fused multiply-add of
// both in one issue slot (same results as the scalar instructions)
typedef unsigned long long u64;
PTY_DEVI u64 pk(float a, float b) {
  u64 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
  return d;
}
PTY_DEVI u64 pk(float a) { return pk(a, a); }
PTY_DEVI void upk(u64 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
PTY_DEVI u64 add2(u64 a, u64 b) {
  u64 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
PTY_DEVI u64 mul2(u64 a, u64 b) {
  u64 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
PTY_DEVI u64 fma2(u64 a, u64 b, u64 c) {
  u64 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
// a - b (the product with -1 is exact)
PTY_DEVI u64 sub2(u64 a, u64 b) { return fma2(b, pk(-1.f), a); }

// store 8 consecutive features [f0, f0+8) of row c (f0 % 8 == 0)
PTY_DEVI void st8(unsigned char* base, int c, int f0, const u64 (&v)[4]) {
  uint32_t q[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float a, b;
    upk(v[j], a, b);
    q[j] = pack_bf16x2(a, b);
  }
  *reinterpret_cast<uint4*>(base + cm_off(c, f0)) = make_uint4(q[0], q[1], q[2], q[3]);
}
// the same 8 values as bf16(v) at feature f of `hi` and, at the same place of
// `lo`, as bf16(v - bf16(v)); conversions in pairs (a single one runs at 16 a
// clock on the unit of sin, cos and exp, a pair at 64)
PTY_DEVI void st8_split(unsigned char* hi, int f, unsigned char* lo, int f_lo, int c, const u64 (&v)[4]) {
  uint32_t q[4], r[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float a, b;
    upk(v[j], a, b);
    q[j] = pack_bf16x2(a, b);
    upk(sub2(v[j], pk(__uint_as_float(q[j] << 16), __uint_as_float(q[j] & 0xffff0000u))), a, b);
    r[j] = pack_bf16x2(a, b);
  }
  *reinterpret_cast<uint4*>(hi + cm_off(c, f)) = make_uint4(q[0], q[1], q[2], q[3]);
  *reinterpret_cast<uint4*>(lo + cm_off(c, f_lo)) = make_uint4(r[0], r[1], r[2], r[3]);
}

// sin and cos of a pair after Cody-Waite reduction by 2 pi (two-constant split of
// 2 pi: the float nearest 2 pi plus its residual), then the SFU on [-pi, pi].
// The nearest integer comes from adding and taking off 1.5 2^23 (rintf runs at 16 a
// clock on the unit that sin, cos and exp need), with the argument's sign: the sum then
// stays where floats are whole numbers, every one below 2^22 turns and even ones beyond.
// (Against a positive constant, turns below -2^22 came out as halves, and the phase off
// by pi.)  The sign comes from a saturated product: as bit operations, whose unit the
// BF16 conversions load, forward and backward of 4,194,304 coordinates take 1836 us, this
// way 1795, without the sign 1766.
PTY_DEVI void sincos_rr(u64 a, u64* s, u64* c) {
  float a0, a1;
  upk(a, a0, a1);
  const u64 pos = pk(__saturatef(fmaf(a0, 1e30f, 0.5f)), __saturatef(fmaf(a1, 1e30f, 0.5f)));  // 1, or 0 where negative
  const u64 m = fma2(pos, pk(25165824.f), pk(-12582912.f));
  const u64 k = sub2(fma2(a, pk(0.159154943091895336f), m), m);
  u64 r = fma2(k, pk(-6.28318548202514648f), a);
  r = fma2(k, pk(1.74845553e-7f), r);
  float r0, r1, s0, s1, c0, c1;
  upk(r, r0, r1);
  __sincosf(r0, &s0, &c0);
  __sincosf(r1, &s1, &c1);
  *s = pk(s0, s1);
  *c = pk(c0, c1);
}

// exp(x) = 2^(x log2 e) of a pair, down to the smallest floats (flushing those below the
// normal range to zero would save 0.7 % of the forward and backward together)
PTY_DEVI u64 exp_fast(u64 x) {
  float a, b, ya, yb;
  upk(mul2(x, pk(1.44269504088896341f)), a, b);
  asm("ex2.approx.f32 %0, %1;" : "=f"(ya) : "f"(a));
  asm("ex2.approx.f32 %0, %1;" : "=f"(yb) : "f"(b));
  return pk(ya, yb);
}

// ---- GEMM issue helpers (single thread) --------------------------------------
// D[128 x N] (+)= A[128 x K] * B[N x K]^T, A activations (K-major), B weights (K-major)
PTY_DEVI void gemm_act_w(uint32_t d, uint32_t sa, uint32_t sb, uint32_t nout, int N, int K, bool acc) {
  const uint32_t id = tc::idesc_bf16(128, N, false, false);
  const uint32_t lbo_b = nout * 16;
  for (int s = 0; s < K / 16; ++s)
    tc::mma(d, tc::desc(sa + s * 2 * GRP, GRP, 128), tc::desc(sb + s * 2 * lbo_b, lbo_b, 128), id,
            (acc || s > 0) ? 1u : 0u);
}
// D[128 x N] = A[128 x K] * W where W[K out][N in] is stored K-major (n contiguous): MN-major B
PTY_DEVI void gemm_act_wT(uint32_t d, uint32_t sa, uint32_t sb, uint32_t nout, int N, int K) {
  const uint32_t id = tc::idesc_bf16(128, N, false, true);
  for (int s = 0; s < K / 16; ++s)
    tc::mma(d, tc::desc(sa + s * 2 * GRP, GRP, 128), tc::desc(sb + s * 2 * 128, 128, nout * 16), id,
            s > 0 ? 1u : 0u);
}
// D[128 x N] (+)= sum over the tile's 128 rows of a_c b_c^T: both operands are
// activation buffers read MN-major (feature = M or N, row = K)
PTY_DEVI void gemm_outer(uint32_t d, uint32_t sa, uint32_t sb, int N, bool acc) {
  const uint32_t id = tc::idesc_bf16(128, N, true, true);
  for (int s = 0; s < 8; ++s)
    tc::mma(d, tc::desc(sa + s * 256, 128, GRP), tc::desc(sb + s * 256, 128, GRP), id, (acc || s > 0) ? 1u : 0u);
}

struct Args {
  const unsigned char* packed;
  const float* x;    // [N][32]
  const float2* gy;  // [N]
  int N;
  float2* y;         // [N] or null
  float* gx;         // [N][32] (or [32][N] when gx_planar) or null
  float* part;       // [gridDim.x][kPartFloats]
  int32_t* status;
  int gx_planar;     // gx feature-major: feature f of row c at gx[f * N + c]
  int x_planar;      // x feature-major: feature f of row c at x[f * N + c]
};

constexpr int kTileThreads = 256;  // threads of one tile in flight

// the tile row, half of the units and TMEM lane offset of thread st (0 .. 255) of a tile
struct Place {
  int row, hh;
  uint32_t lanes;
};
PTY_DEVI Place place(int st) {
  const int w = st >> 5, quarter = w & 3;
  return {32 * quarter + (st & 31), w >> 2, uint32_t(quarter * 32) << 16};
}

// weights, parameters and the output weights as floats into shared memory
PTY_DEVI void load_packed(const Args& a, unsigned char* w, float* par, int t, int nt) {
  for (int i = t; i < kWBytes / 16; i += nt)
    reinterpret_cast<uint4*>(w)[i] = __ldg(reinterpret_cast<const uint4*>(a.packed) + i);
  for (int i = t; i < kParFloats; i += nt) par[i] = __ldg(reinterpret_cast<const float*>(a.packed + kWBytes) + i);
  for (int i = t; i < 64; i += nt) {  // Re Wo_k at (row 0, k), Im Wo_k at (row 1, k)
    const __nv_bfloat16* wo = reinterpret_cast<const __nv_bfloat16*>(a.packed + S_WO);
    par[P_WOR + i] = __bfloat162float(wo[wm_off(i >> 5, i & 31, 16) / 2]);
  }
}

// this half's 16 of row c's 32 input features
PTY_DEVI void load_x(const Args& a, int c, int hh, u64 (&lo)[4], u64 (&hi)[4]) {
  const bool ok = c < a.N;
  if (a.x_planar) {  // per feature, a warp reads 32 consecutive rows
    const float* xp = a.x + size_t(16 * hh) * a.N + c;
    float v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = ok ? __ldg(xp + size_t(i) * a.N) : 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      lo[j] = pk(v[2 * j], v[2 * j + 1]);
      hi[j] = pk(v[8 + 2 * j], v[9 + 2 * j]);
    }
  } else {
    const float4* xp = reinterpret_cast<const float4*>(a.x + size_t(ok ? c : 0) * 32 + 16 * hh);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const float4 u = ok ? __ldg(xp + q) : make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 v = ok ? __ldg(xp + 2 + q) : make_float4(0.f, 0.f, 0.f, 0.f);
      lo[2 * q] = pk(u.x, u.y);
      lo[2 * q + 1] = pk(u.z, u.w);
      hi[2 * q] = pk(v.x, v.y);
      hi[2 * q + 1] = pk(v.z, v.w);
    }
  }
}

// bring tile nt's features towards L2: a tile's loads are the first link of its chain
PTY_DEVI void prefetch_x(const Args& a, int nt, int ntiles, int st) {
  if (nt >= ntiles) return;
  if (a.x_planar) {  // 32 features x 512 bytes: one 64-byte piece per thread
    const int f = st >> 3, r0 = nt * 128 + (st & 7) * 16;
    if (r0 < a.N) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.x + size_t(f) * a.N + r0));
  } else {  // 128 rows x 128 bytes: 16 KB, one 64-byte piece per thread
    const size_t off = size_t(nt) * 128 * 32 + size_t(st) * 16;
    if (off < size_t(a.N) * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.x + off));
  }
}

// h1 = exp(i w1 zz) of eight units
PTY_DEVI void h_layer1(const u64 (&zz)[4], float w1, u64 (&hr)[4], u64 (&hi)[4]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) sincos_rr(mul2(zz[j], pk(w1)), &hi[j], &hr[j]);
}
// h = exp(i w (r + i i)) of eight units
PTY_DEVI void h_complex(const u64 (&r)[4], const u64 (&i)[4], float w, u64 (&hr)[4], u64 (&hi)[4]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const u64 amp = exp_fast(mul2(i[j], pk(-w)));
    u64 s, co;
    sincos_rr(mul2(r[j], pk(w)), &s, &co);
    hr[j] = mul2(amp, co);
    hi[j] = mul2(amp, s);
  }
}
// eight columns at taddr, plus the eight floats at b
PTY_DEVI void ld8_bias(uint32_t taddr, const float* b, u64 (&v)[4]) {
  float z[8];
  tc::ld8(taddr, z);
  const ulonglong2 p = reinterpret_cast<const ulonglong2*>(b)[0], q = reinterpret_cast<const ulonglong2*>(b)[1];
  v[0] = add2(pk(z[0], z[1]), p.x);
  v[1] = add2(pk(z[2], z[3]), p.y);
  v[2] = add2(pk(z[4], z[5]), q.x);
  v[3] = add2(pk(z[6], z[7]), q.y);
}
PTY_DEVI void ld8x2(uint32_t ta, u64 (&va)[4], uint32_t tb, u64 (&vb)[4]) {
  float x[8], y[8];
  tc::ld8x2(ta, x, tb, y);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    va[j] = pk(x[2 * j], x[2 * j + 1]);
    vb[j] = pk(y[2 * j], y[2 * j + 1]);
  }
}
PTY_DEVI void bias8(u64 (&v)[4], const float* b) {
  const ulonglong2 p = reinterpret_cast<const ulonglong2*>(b)[0], q = reinterpret_cast<const ulonglong2*>(b)[1];
  v[0] = add2(v[0], p.x);
  v[1] = add2(v[1], p.y);
  v[2] = add2(v[2], q.x);
  v[3] = add2(v[3], q.y);
}
// back through h = exp(i w z): om += Re(conj(G_h) i z h), r + i i <- conj(i w h) G_h
PTY_DEVI void grad_z(u64 (&r)[4], u64 (&i)[4], const u64 (&hr)[4], const u64 (&hi)[4], const u64 (&gr)[4],
                     const u64 (&gi)[4], float w, u64& om) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const u64 nhi = mul2(hi[j], pk(-1.f));
    const u64 p = fma2(i[j], nhi, mul2(r[j], hr[j])), q = fma2(i[j], hr[j], mul2(r[j], hi[j]));
    om = add2(om, sub2(mul2(gi[j], p), mul2(gr[j], q)));
    r[j] = mul2(fma2(hr[j], gi[j], mul2(nhi, gr[j])), pk(w));
    i[j] = mul2(fma2(hr[j], gr[j], mul2(hi[j], gi[j])), pk(-w));
  }
}

// barrier of one slot's threads that also agrees on `bad`
PTY_DEVI bool slot_barrier_or(int slot, bool bad) {
  uint32_t any;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 q, %2, 0;\n\t"
      "barrier.cta.red.or.pred p, %1, %3, q;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(any)
      : "r"(1 + slot), "r"(uint32_t(bad)), "n"(kTileThreads)
      : "memory");
  return any != 0;
}

// ---- forward ---------------------------------------------------------------------
constexpr int kFwdSlots = 4;  // tiles in flight: 4 x 256 threads, one CTA per SM
constexpr int F_HI = 0;              // bf16(h) of the running layer: 8 groups
constexpr int F_LO = F_HI + 8 * GRP;  // h - bf16(h): 8 groups
constexpr int F_X = F_LO + 8 * GRP;   // x of the next tile: 4 groups
constexpr int kFwdSlotBytes = F_X + 4 * GRP;
constexpr int F_W = kFwdSlots * kFwdSlotBytes;
constexpr int F_PAR = F_W + kWBytes;
constexpr int F_BAR = F_PAR + kParSmem * 4;  // one per slot
constexpr int F_NEXT = F_BAR + kFwdSlots * 8;  // tile counter, then each slot's next tile
constexpr int F_TMEM = F_NEXT + 4 * (kFwdSlots + 1);
constexpr int F_SMEM = int(pty_align_up_c(F_TMEM + 8, 128));
static_assert(P_B1 % 4 == 0 && P_B2R % 4 == 0 && F_PAR % 16 == 0 && F_BAR % 8 == 0, "alignment");
static_assert(F_SMEM <= 232448, "shared-memory budget");
// TMEM columns per slot: z1, z2, z3 in turn (64), the output (16)
constexpr uint32_t kColsFwd = 512, kColsFwdSlot = 128, T_OUT = 64;

__global__ void __launch_bounds__(kFwdSlots* kTileThreads, 1) k_cmlp_fwd(const Args a) {
  extern __shared__ __align__(1024) unsigned char sm[];
  const int t = threadIdx.x, slot = t / kTileThreads, st = t % kTileThreads;
  const Place pl = place(st);
  const int row = pl.row, hh = pl.hh;
  unsigned char* sl = sm + slot * kFwdSlotBytes;
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + F_BAR) + slot;
  int* counter = reinterpret_cast<int*>(sm + F_NEXT);
  volatile int* next = reinterpret_cast<int*>(sm + F_NEXT) + 1 + slot;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(sm + F_TMEM);
  float* par = reinterpret_cast<float*>(sm + F_PAR);
  const uint32_t sb = tc::smem_addr(sl), wb = tc::smem_addr(sm) + F_W;
  load_packed(a, sm + F_W, par, t, kFwdSlots * kTileThreads);
  if (t == 0) {
    for (int i = 0; i < kFwdSlots; ++i) mbar_init(reinterpret_cast<uint64_t*>(sm + F_BAR) + i, 1);
    fence_mbar_init();
    *counter = kFwdSlots;
  }
  if (t < 32) {
    tc::tmem_alloc(tslot, kColsFwd);
    tc::tmem_relinquish();
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tm = *tslot, tz = tm + slot * kColsFwdSlot, lz = tz + pl.lanes;
  const float w1 = par[P_W1], w2 = par[P_W2], w3 = par[P_W3];
  uint32_t phase = 0;
  bool bad = false, abort = false;

  // operands written -> the slot's first thread issues `issue` -> its threads wait
  // for the result; a wait that ran out is agreed on at the next step's barrier
  auto step = [&](auto issue) {
    tc::fence_smem_async();
    tc::fence_before();
    abort = slot_barrier_or(slot, bad);
    if (abort) return;
    tc::fence_after();
    if (st == 0) {
      issue();
      tc::commit(bar);
    }
    bad = bad || !mbar_wait_bounded(bar, phase);
    phase ^= 1u;
    tc::fence_after();
  };
  auto output = [&] {
    gemm_act_w(tz + T_OUT, sb + F_HI, wb + S_WO, 16, 16, 64, false);
    gemm_act_w(tz + T_OUT, sb + F_LO, wb + S_WO, 16, 16, 64, true);
  };
  auto store_y = [&](int tile) {
    if (hh == 0) {  // warp-uniform
      float d[8];
      tc::ld8(lz + T_OUT, d);
      const int c = tile * 128 + row;
      if (c < a.N) a.y[c] = make_float2(d[0] + par[P_BOR], d[1] + par[P_BOI]);
    }
  };

  // The CTA's tiles are blockIdx + i gridDim; its slots take i from a shared
  // counter (the scheduler favours some warps, and equal shares left the SM with
  // 3 tiles in flight on average)
  const int ntiles = (a.N + 127) / 128;
  auto tile_of = [&](int i) { return int(blockIdx.x) + i * int(gridDim.x); };
  int tile = tile_of(slot), last = -1;
  u64 xa[4], xb[4];
  if (tile < ntiles) {
    load_x(a, tile * 128 + row, hh, xa, xb);
    st8(sl + F_X, row, 16 * hh, xa);
    st8(sl + F_X, row, 16 * hh + 8, xb);
  }
  while (tile < ntiles) {
    if (st == 0) *next = tile_of(atomicAdd(counter, 1));  // published by the next two barriers
    step([&] {
      gemm_act_w(tz, sb + F_X, wb + S_W1, 32, 32, 32, false);
      if (last >= 0) output();  // of the tile before, whose h3 is in place
    });
    if (abort) break;
    if (last >= 0) store_y(last);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int u = 16 * hh + 8 * q;
      u64 z[4], hr[4], hi[4];
      ld8_bias(lz + u, par + P_B1 + u, z);
      h_layer1(z, w1, hr, hi);
      st8_split(sl + F_HI, u, sl + F_LO, u, row, hr);
      st8_split(sl + F_HI, 32 + u, sl + F_LO, 32 + u, row, hi);
    }
    step([&] {
      gemm_act_w(tz, sb + F_HI, wb + S_W2, 64, 64, 64, false);
      gemm_act_w(tz, sb + F_LO, wb + S_W2, 64, 64, 64, true);
    });
    if (abort) break;
    last = tile;
    tile = *next;
    prefetch_x(a, tile, ntiles, st);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int u = 16 * hh + 8 * q;
      u64 r[4], i[4], hr[4], hi[4];
      ld8x2(lz + u, r, lz + 32 + u, i);
      bias8(r, par + P_B2R + u);
      bias8(i, par + P_B2I + u);
      h_complex(r, i, w2, hr, hi);
      st8_split(sl + F_HI, u, sl + F_LO, u, row, hr);
      st8_split(sl + F_HI, 32 + u, sl + F_LO, 32 + u, row, hi);
    }
    if (tile < ntiles) load_x(a, tile * 128 + row, hh, xa, xb);  // lands while z3 is formed
    step([&] {
      gemm_act_w(tz, sb + F_HI, wb + S_W3, 64, 64, 64, false);
      gemm_act_w(tz, sb + F_LO, wb + S_W3, 64, 64, 64, true);
    });
    if (abort) break;
    if (tile < ntiles) {
      st8(sl + F_X, row, 16 * hh, xa);
      st8(sl + F_X, row, 16 * hh + 8, xb);
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int u = 16 * hh + 8 * q;
      u64 r[4], i[4], hr[4], hi[4];
      ld8x2(lz + u, r, lz + 32 + u, i);
      bias8(r, par + P_B3R + u);
      bias8(i, par + P_B3I + u);
      h_complex(r, i, w3, hr, hi);
      st8_split(sl + F_HI, u, sl + F_LO, u, row, hr);
      st8_split(sl + F_HI, 32 + u, sl + F_LO, 32 + u, row, hi);
    }
  }
  if (!abort && last >= 0) {
    step(output);
    if (!abort) store_y(last);
  }
  if (abort || bad) mbar_wait_bounded(bar, phase ^ 1u);  // let the slot's last MMAs drain
  tc::fence_before();
  if (__syncthreads_or(bad) && t == 0) pty_raise(a.status, PTYCHO_ERR_TIMEOUT);
  if (t < 32) tc::tmem_free(tm, kColsFwd);
}

// ---- backward --------------------------------------------------------------------
constexpr int kSlots = 2;                                 // tiles in flight per CTA
constexpr int kBwdThreads = kSlots * kTileThreads;
// per tile: every MMA reads 16-group A footprints (unused accumulator rows take
// whatever follows an operand), all inside the tile's own buffers
constexpr int B_GZ1 = 0;               // G_z1: 4 groups
constexpr int B_GY = B_GZ1 + 4 * GRP;  // (G_yr, G_yi, 0 ...): 2 groups, rows 32, 33 of the G_z1 accumulator
constexpr int B_GZ = B_GY + 2 * GRP;   // G_z3 (8), G_z2 (8)
constexpr int B_LO = B_GZ;             // h - bf16(h) of layers 1, 2: dead before G_z3 is written
constexpr int B_H3 = B_GZ + 8 * GRP;   // bf16(h3): its MMA completes before G_z2 is written
constexpr int B_H = B_GZ + 16 * GRP;   // bf16(h2) (8), bf16(h1) (8), ones (1)
constexpr int B_X = B_H + 17 * GRP;    // x (4), ones (1): two buffers, tiles alternate
constexpr int kXBytes = 5 * GRP;
constexpr int kSlotBytes = B_X + 2 * kXBytes + GRP;  // and a group of padding
static_assert(B_GZ1 + 16 * GRP <= kSlotBytes && B_H + 18 * GRP <= kSlotBytes, "MMA footprints");
constexpr int B_W = kSlots * kSlotBytes;
constexpr int B_PAR = B_W + kWBytes;
constexpr int B_Y = B_PAR + kParSmem * 4;            // output partials: [slot][128] float2
constexpr int B_RED = B_Y + kSlots * 128 * 8;        // 3 sums of 16 warps
constexpr int B_BAR = B_RED + 3 * 16 * 4;            // per slot: chain, both accumulations done
constexpr int B_TMEM = B_BAR + kSlots * 3 * 8;
constexpr int B_SMEM = int(pty_align_up_c(B_TMEM + 8, 128));
static_assert(B_PAR % 16 == 0 && B_Y % 8 == 0 && B_BAR % 8 == 0 && B_SMEM <= 232448, "shared-memory budget");
// TMEM columns: the accumulators, then per slot z1 / z3 / G_h2 / G_h1 (64) and z2 / G_h3 / G_x (64)
constexpr uint32_t T_ACC = 0, T_ACC1 = 144, T_ACCO = 192, T_SLOT = 256, kColsBwd = 512;

__global__ void __launch_bounds__(kBwdThreads, 1) k_cmlp_bwd(const Args a) {
  extern __shared__ __align__(1024) unsigned char sm[];
  const int t = threadIdx.x, w = t >> 5;
  const int slot = t / kTileThreads;
  const int st = t % kTileThreads;
  const Place pl = place(st);
  const int row = pl.row, hh = pl.hh;
  unsigned char* sl = sm + slot * kSlotBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + B_BAR);
  uint64_t *chain = bars, *done_o = bars + kSlots, *done_a = bars + 2 * kSlots;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(sm + B_TMEM);
  float* par = reinterpret_cast<float*>(sm + B_PAR);
  float* red = reinterpret_cast<float*>(sm + B_RED);
  const uint32_t sbase = tc::smem_addr(sm);

  load_packed(a, sm + B_W, par, t, kBwdThreads);
  if (hh == 1) {  // the second feature group of G_y stays zero
    const u64 zero[4] = {0, 0, 0, 0};
    st8(sl + B_GY, row, 8, zero);
  } else {  // ones columns; the other features of those groups are not used
    const __nv_bfloat16 one = __float2bfloat16(1.0f);
    *reinterpret_cast<__nv_bfloat16*>(sl + B_H + cm_off(row, 128)) = one;
    *reinterpret_cast<__nv_bfloat16*>(sl + B_X + cm_off(row, 32)) = one;
    *reinterpret_cast<__nv_bfloat16*>(sl + B_X + kXBytes + cm_off(row, 32)) = one;
  }
  if (t == 0) {
    for (int i = 0; i < 3 * kSlots; ++i) mbar_init(bars + i, 1);
    fence_mbar_init();
  }
  if (w == 0) {
    tc::tmem_alloc(tslot, kColsBwd);
    tc::tmem_relinquish();
  }
  tc::fence_smem_async();
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tm = *tslot;
  const int ntiles = (a.N + 127) / 128;
  // the CTA's tiles in order: q = 0 .. nq-1 is tile q gridDim + blockIdx, on slot q % kSlots
  const int nq = (ntiles - int(blockIdx.x) + int(gridDim.x) - 1) / int(gridDim.x);
  bool bad = false;
  u64 om1 = 0, om2 = 0, om3 = 0;  // pairs of partial sums

  {
    const float w1 = par[P_W1], w2 = par[P_W2], w3 = par[P_W3];
    const uint32_t ta = tm + T_SLOT + 128 * slot, tb = ta + 64;  // the slot's columns
    const uint32_t la = ta + pl.lanes, lb = tb + pl.lanes;
    const uint32_t sb = sbase + slot * kSlotBytes, wb = sbase + B_W;
    float2* ybuf = reinterpret_cast<float2*>(sm + B_Y) + slot * 128;
    uint32_t phase = 0;
    bool abort = false;
    // operands written -> the slot's first thread issues `issue` and, behind it,
    // `accumulate` -> its threads wait for the result of `issue`
    auto step = [&](auto issue, auto accumulate) {
      tc::fence_smem_async();
      tc::fence_before();
      abort = slot_barrier_or(slot, bad);
      if (abort) return;
      tc::fence_after();
      if (st == 0) {
        issue();
        tc::commit(chain + slot);
        accumulate();
      }
      bad = bad || !mbar_wait_bounded(chain + slot, phase);
      phase ^= 1u;
      tc::fence_after();
    };
    auto nothing = [] {};
    // the two slots add into the same columns: tile q after tile q - 1 has been added
    auto after_previous = [&](uint64_t* done, int q) {
      if (q > 0) bad = bad || !mbar_wait_bounded(done + (q - 1) % kSlots, ((q - 1) / kSlots) & 1);
      tc::fence_after();
    };
    u64 xa[4], xb[4];
    float2 gn = make_float2(0.f, 0.f);
    auto load_in = [&](int tile) {
      const int c = tile * 128 + row;
      load_x(a, c, hh, xa, xb);
      gn = c < a.N ? __ldg(a.gy + c) : make_float2(0.f, 0.f);
    };
    if (slot < nq) load_in(slot * gridDim.x + blockIdx.x);
    for (int q = slot; q < nq; q += kSlots) {
      const int tile = q * gridDim.x + blockIdx.x;
      const int c = tile * 128 + row;
      const bool valid = c < a.N;
      const uint32_t par_q = (q / kSlots) & 1;
      // -- inputs ------------------------------------------------------------------------
      const int bx = B_X + int(par_q) * kXBytes;
      st8(sl + bx, row, 16 * hh, xa);
      st8(sl + bx, row, 16 * hh + 8, xb);
      prefetch_x(a, tile + kSlots * gridDim.x, ntiles, st);
      step([&] { gemm_act_w(ta, sb + bx, wb + S_W1, 32, 32, 32, false); }, nothing);
      if (abort) break;
      // the tile before: its accumulation has read every buffer written from here on
      if (q >= kSlots) bad = bad || !mbar_wait_bounded(done_a + slot, par_q ^ 1u);
      if (hh == 0) {
        const u64 v[4] = {pk(gn.x, gn.y), 0, 0, 0};
        st8(sl + B_GY, row, 0, v);
      }
      // -- layer 1 (zz = z1 + b1 is kept for its gradient) -------------------------------
      u64 zz[2][4];
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const int u = 16 * hh + 8 * p;
        u64 hr[4], hi[4];
        ld8_bias(la + u, par + P_B1 + u, zz[p]);
        h_layer1(zz[p], w1, hr, hi);
        st8_split(sl + B_H, 64 + u, sl + B_LO, u, row, hr);
        st8_split(sl + B_H, 96 + u, sl + B_LO, 32 + u, row, hi);
      }
      step([&] {
        gemm_act_w(tb, sb + B_H + 8 * GRP, wb + S_W2, 64, 64, 64, false);
        gemm_act_w(tb, sb + B_LO, wb + S_W2, 64, 64, 64, true);
      }, nothing);
      if (abort) break;
      // -- layer 2 (z2 + b2 is kept for its gradient) -------------------------------------
      u64 z2r[2][4], z2i[2][4];
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const int u = 16 * hh + 8 * p;
        u64 hr[4], hi[4];
        ld8x2(lb + u, z2r[p], lb + 32 + u, z2i[p]);
        bias8(z2r[p], par + P_B2R + u);
        bias8(z2i[p], par + P_B2I + u);
        h_complex(z2r[p], z2i[p], w2, hr, hi);
        st8_split(sl + B_H, u, sl + B_LO, u, row, hr);
        st8_split(sl + B_H, 32 + u, sl + B_LO, 32 + u, row, hi);
      }
      step([&] {  // z3, and G_h3 = Wo_r^T G_y
        gemm_act_w(ta, sb + B_H, wb + S_W3, 64, 64, 64, false);
        gemm_act_w(ta, sb + B_LO, wb + S_W3, 64, 64, 64, true);
        gemm_act_wT(tb, sb + B_GY, wb + S_WO, 16, 64, 16);
      }, nothing);
      if (abort) break;
      // -- layer 3, the output, and G_z3 = conj(i w3 h3) G_h3 ------------------------------
      float2 yp = make_float2(0.f, 0.f);
#pragma unroll 1
      for (int p = 0; p < 2; ++p) {
        const int u = 16 * hh + 8 * p;
        u64 r[4], i[4], hr[4], hi[4], gr[4], gi[4];
        ld8x2(la + u, r, la + 32 + u, i);
        bias8(r, par + P_B3R + u);
        bias8(i, par + P_B3I + u);
        h_complex(r, i, w3, hr, hi);
        ld8x2(lb + u, gr, lb + 32 + u, gi);
        st8(sl + B_H3, row, u, hr);
        st8(sl + B_H3, row, 32 + u, hi);
        if (a.y) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float h0, h1, k0, k1;
            upk(hr[j], h0, h1);
            upk(hi[j], k0, k1);
            const float* wr = par + P_WOR + u + 2 * j;
            const float* wi = par + P_WOI + u + 2 * j;
            yp.x = fmaf(wr[0], h0, fmaf(-wi[0], k0, fmaf(wr[1], h1, fmaf(-wi[1], k1, yp.x))));
            yp.y = fmaf(wr[0], k0, fmaf(wi[0], h0, fmaf(wr[1], k1, fmaf(wi[1], h1, yp.y))));
          }
        }
        grad_z(r, i, hr, hi, gr, gi, w3, om3);
        st8(sl + B_GZ, row, u, r);
        st8(sl + B_GZ, row, 32 + u, i);
      }
      if (a.y && hh == 1) ybuf[row] = yp;
      step([&] { gemm_act_wT(ta, sb + B_GZ, wb + S_W3, 64, 64, 64); },
           [&] {
             after_previous(done_o, q);
             gemm_outer(tm + T_ACCO, sb + B_GY, sb + B_H3, 64, q > 0);
             tc::commit(done_o + slot);
           });
      if (abort) break;
      if (a.y && hh == 0 && valid) {
        const float2 o = ybuf[row];
        a.y[c] = make_float2(yp.x + o.x + par[P_BOR], yp.y + o.y + par[P_BOI]);
      }
      // -- G_z2 = conj(i w2 h2) G_h2 (written over h3: wait for its accumulation) ---------------
      bad = bad || !mbar_wait_bounded(done_o + slot, par_q);
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const int u = 16 * hh + 8 * p;
        u64 gr[4], gi[4], hr[4], hi[4];
        ld8x2(la + u, gr, la + 32 + u, gi);
        h_complex(z2r[p], z2i[p], w2, hr, hi);  // again: 32 registers less than keeping it
        grad_z(z2r[p], z2i[p], hr, hi, gr, gi, w2, om2);
        st8(sl + B_GZ, row, 64 + u, z2r[p]);
        st8(sl + B_GZ, row, 96 + u, z2i[p]);
      }
      step([&] { gemm_act_wT(ta, sb + B_GZ + 8 * GRP, wb + S_W2, 64, 64, 64); }, nothing);
      if (abort) break;
      // -- G_z1 = Re(conj(G_h1) i w1 h1) ----------------------------------------------------
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const int u = 16 * hh + 8 * p;
        u64 gr[4], gi[4];
        ld8x2(la + u, gr, la + 32 + u, gi);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          u64 sn, co;
          sincos_rr(mul2(zz[p][j], pk(w1)), &sn, &co);
          const u64 v = fma2(co, gi[j], mul2(mul2(sn, pk(-1.f)), gr[j]));
          om1 = fma2(zz[p][j], v, om1);
          gr[j] = mul2(v, pk(w1));
        }
        st8(sl + B_GZ1, row, u, gr);
      }
      if (q + kSlots < nq) load_in(tile + kSlots * gridDim.x);  // lands while G_x is formed
      step([&] { gemm_act_wT(tb, sb + B_GZ1, wb + S_W1, 32, 32, 32); },
           [&] {
             after_previous(done_a, q);
             gemm_outer(tm + T_ACC, sb + B_GZ, sb + B_H, 144, q > 0);
             gemm_outer(tm + T_ACC1, sb + B_GZ1, sb + bx, 48, q > 0);
             tc::commit(done_a + slot);
           });
      if (abort) break;
      if (a.gx) {
        float d[16];
        tc::ld16(lb + 16 * hh, d);
        if (valid) {
          if (a.gx_planar) {  // per feature, a warp stores 32 consecutive rows
#pragma unroll
            for (int i = 0; i < 16; ++i) a.gx[size_t(16 * hh + i) * a.N + c] = d[i];
          } else {
            float4* gp = reinterpret_cast<float4*>(a.gx + size_t(c) * 32 + 16 * hh);
#pragma unroll
            for (int i = 0; i < 4; ++i) gp[i] = make_float4(d[4 * i], d[4 * i + 1], d[4 * i + 2], d[4 * i + 3]);
          }
        }
      }
      // the last tile's accumulation is read below
      if (q + kSlots >= nq) bad = bad || !mbar_wait_bounded(done_a + slot, par_q);
    }
    if (abort || bad) mbar_wait_bounded(chain + slot, phase ^ 1u);  // let the slot's last MMAs drain
  }

  tc::fence_before();
  const bool abort = __syncthreads_or(bad);
  tc::fence_after();
  if (abort && t == 0) pty_raise(a.status, PTYCHO_ERR_TIMEOUT);
  if (!abort) {
    // -- raw accumulators -> this CTA's partial: warp w reads lane quarter w & 3,
    //    16-column chunk w >> 2 of each accumulator -------------------------------------
    float* P = a.part + size_t(blockIdx.x) * kPartFloats;
    {
      const int chunk = w >> 2;
      const uint32_t lo = tm + pl.lanes;
      float d[16];
      const bool top = row < 64;  // rows 0..63: W3 real form and b3; rows 64..127: W2 real form and b2
      tc::ld16(lo + T_ACC + (top ? 0 : 64) + 16 * chunk, d);
      float* pw = P + (top ? R_W3 + row * 64 : R_W2 + (row - 64) * 64) + 16 * chunk;
#pragma unroll
      for (int i = 0; i < 16; ++i) pw[i] = d[i];
      if (chunk == 0) {
        tc::ld16(lo + T_ACC + 128, d);
        P[top ? R_B3 + row : R_B2 + row - 64] = d[0];
      }
      if ((w & 3) == 0) {  // rows 0..31: W1, b1 ; rows 0,1: Wo real form
        if (chunk < 2) {
          tc::ld16(lo + T_ACC1 + 16 * chunk, d);
#pragma unroll
          for (int i = 0; i < 16; ++i) P[R_W1 + row * 32 + 16 * chunk + i] = d[i];
        }
        if (chunk == 2) {
          tc::ld16(lo + T_ACC1 + 32, d);
          P[R_B1 + row] = d[0];
        }
        tc::ld16(lo + T_ACCO + 16 * chunk, d);
        if (row < 2) {
#pragma unroll
          for (int i = 0; i < 16; ++i) P[R_WO + row * 64 + 16 * chunk + i] = d[i];
        }
      }
      if (w == 1) {  // rows 32, 33 of the G_z1 accumulator: G_y against the ones column
        tc::ld16(lo + T_ACC1 + 32, d);
        if (row < 34) P[R_BO + row - 32] = d[0];
      }
      // omega gradients: fixed shuffle tree, then warps in order
      const u64 om[3] = {om1, om2, om3};
#pragma unroll
      for (int l = 0; l < 3; ++l) {
        float x, y;
        upk(om[l], x, y);
        x += y;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if ((t & 31) == 0) red[16 * l + w] = x;
      }
    }
    __syncthreads();
    if (t < 3) {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < 16; ++i) s += red[16 * t + i];  // warps in order
      P[R_OM + t] = s;
    }
  }
  tc::fence_before();
  __syncthreads();
  if (w == 0) tc::tmem_free(tm, kColsBwd);
}

// sum the CTA partials in a fixed order and fold the real-form blocks
// Block b owns outputs 32 b .. 32 b + 31, one per lane, so each warp's loads of
// one partial touch neighbouring raw entries; warp k sums partials k, k + 8, ...
// in order and the eight warp sums are added in warp order.
__global__ void __launch_bounds__(256) k_cmlp_reduce(const float* __restrict__ part, int nparts,
                                                     float* __restrict__ grad) {
  __shared__ float wsum[8][32];
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const int e = blockIdx.x * 32 + lane;
  // each output is a (sign-weighted) sum of at most two raw entries
  int i0 = -1, i1 = -1;
  float s1 = 0.f;
  if (e < G_B1) {
    i0 = R_W1 + (e - G_W1);
  } else if (e < G_OM1) {
    i0 = R_B1 + (e - G_B1);
  } else if (e == G_OM1) {
    i0 = R_OM + 0;
  } else if (e == G_OM1 + 1) {
  } else if (e < G_B2 || (e >= G_W3 && e < G_B3)) {  // complex W2 / W3 [o][i][re,im]
    const bool l2 = e < G_B2;
    const int base = l2 ? R_W2 : R_W3;
    const int j = e - (l2 ? G_W2 : G_W3);
    const int o = j / 64, i = (j % 64) / 2, im = j & 1;
    if (!im) {  // P + S
      i0 = base + o * 64 + i;
      i1 = base + (32 + o) * 64 + 32 + i;
      s1 = 1.f;
    } else {  // R - Q
      i0 = base + (32 + o) * 64 + i;
      i1 = base + o * 64 + 32 + i;
      s1 = -1.f;
    }
  } else if (e < G_OM2 || (e >= G_B3 && e < G_OM3)) {  // complex b2 / b3
    const bool l2 = e < G_OM2;
    const int j = e - (l2 ? G_B2 : G_B3);
    i0 = (l2 ? R_B2 : R_B3) + (j & 1) * 32 + j / 2;
  } else if (e == G_OM2) {
    i0 = R_OM + 1;
  } else if (e == G_OM3) {
    i0 = R_OM + 2;
  } else if (e >= G_WO && e < G_BO) {
    const int j = e - G_WO;
    const int i = j / 2, im = j & 1;
    if (!im) {
      i0 = R_WO + i;
      i1 = R_WO + 64 + 32 + i;
      s1 = 1.f;
    } else {
      i0 = R_WO + 64 + i;
      i1 = R_WO + 32 + i;
      s1 = -1.f;
    }
  } else if (e >= G_BO) {
    i0 = R_BO + (e - G_BO);
  }
  float acc = 0.f;
  if (e < kGradFloats && i0 >= 0) {
    int p = wp;
    for (; p + 24 < nparts; p += 32) {  // four partials' loads in flight, added in order
      float v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float* P = part + size_t(p + 8 * k) * kPartFloats;
        v[k] = P[i0];
        if (i1 >= 0) v[k] = fmaf(s1, P[i1], v[k]);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) acc += v[k];
    }
    for (; p < nparts; p += 8) {
      const float* P = part + size_t(p) * kPartFloats;
      float v = P[i0];
      if (i1 >= 0) v = fmaf(s1, P[i1], v);
      acc += v;
    }
  }
  wsum[wp][lane] = acc;
  __syncthreads();
  if (wp == 0 && e < kGradFloats) {
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) t += wsum[k][lane];  // warps in order
    grad[e] = t;
  }
}

// pack torch-layout parameters into the kernel's bf16 operand blob + fp32 block
struct PackArgs {
  const float *W1, *b1, *w1, *W2, *b2, *w2, *W3, *b3, *w3, *Wo, *bo;
  unsigned char* out;
};

__global__ void __launch_bounds__(256) k_cmlp_pack(const PackArgs p) {
  const int e = blockIdx.x * 256 + threadIdx.x;
  __nv_bfloat16* wb = reinterpret_cast<__nv_bfloat16*>(p.out);
  float* fb = reinterpret_cast<float*>(p.out + kWBytes);
  if (e < 1024) {  // W1 [32 out][32 in]
    const int n = e / 32, k = e % 32;
    wb[(S_W1 + wm_off(n, k, 32)) / 2] = __float2bfloat16(p.W1[e]);
  } else if (e < 1024 + 2 * 4096) {  // Wr2, Wr3: [[A,-B],[B,A]]
    const int j = e - 1024;
    const int layer = j / 4096, r = (j % 4096) / 64, k = j % 64;
    const float* W = layer ? p.W3 : p.W2;  // complex [32][32] interleaved
    const int ro = r % 32, ko = k % 32;
    const float A = W[2 * (ro * 32 + ko)], B = W[2 * (ro * 32 + ko) + 1];
    const float v = (r < 32) ? (k < 32 ? A : -B) : (k < 32 ? B : A);
    wb[((layer ? S_W3 : S_W2) + wm_off(r, k, 64)) / 2] = __float2bfloat16(v);
  } else if (e < 1024 + 8192 + 1024) {  // Wor [16][64]: row 0 = [Re Wo, -Im Wo], row 1 = [Im Wo, Re Wo]
    const int j = e - 1024 - 8192;
    const int r = j / 64, k = j % 64;
    float v = 0.f;
    if (r < 2) {
      const int ko = k % 32;
      const float A = p.Wo[2 * ko], B = p.Wo[2 * ko + 1];
      v = (r == 0) ? (k < 32 ? A : -B) : (k < 32 ? B : A);
    }
    wb[(S_WO + wm_off(r, k, 16)) / 2] = __float2bfloat16(v);
  } else if (e < 1024 + 8192 + 1024 + kParFloats) {
    const int j = e - 1024 - 8192 - 1024;
    float v = 0.f;
    if (j < 32) v = p.b1[j];
    else if (j < 64) v = p.b2[2 * (j - 32)];
    else if (j < 96) v = p.b2[2 * (j - 64) + 1];
    else if (j < 128) v = p.b3[2 * (j - 96)];
    else if (j < 160) v = p.b3[2 * (j - 128) + 1];
    else if (j == P_BOR) v = p.bo[0];
    else if (j == P_BOI) v = p.bo[1];
    else if (j == P_W1) v = p.w1[0];
    else if (j == P_W2) v = p.w2[0];
    else if (j == P_W3) v = p.w3[0];
    fb[j] = v;
  }
}

template <typename K>
static int launch(K kern, int threads, int smem, const Args& a, cudaStream_t s, int* grid_out) {
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
    return PTYCHO_ERR_LAUNCH;
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const int ntiles = (a.N + 127) / 128;
  const int grid = ntiles < nsm ? ntiles : nsm;  // one CTA per SM: each allocates all of TMEM
  if (grid_out) *grid_out = grid;
  if (grid == 0) return PTYCHO_OK;
  kern<<<grid, threads, smem, s>>>(a);
  return cudaGetLastError() == cudaSuccess ? PTYCHO_OK : PTYCHO_ERR_LAUNCH;
}

}  // namespace cm
}  // namespace pty

using namespace pty;

extern "C" {

size_t ptycho_cmlp_packed_bytes(void) { return cm::kPackedBytes; }

int ptycho_cmlp_grad_floats(void) { return cm::kGradFloats; }

int ptycho_cmlp_pack(const float* W1, const float* b1, const float* omega1, const float* W2, const float* b2,
                     const float* omega2, const float* W3, const float* b3, const float* omega3, const float* Wo,
                     const float* bo, void* packed, ptycho_stream_t stream) {
  if (!W1 || !b1 || !omega1 || !W2 || !b2 || !omega2 || !W3 || !b3 || !omega3 || !Wo || !bo || !packed)
    return PTYCHO_ERR_INVALID_ARG;
  if (!pty_aligned(packed, 16)) return PTYCHO_ERR_MISALIGNED;
  cm::PackArgs p{W1, b1, omega1, W2, b2, omega2, W3, b3, omega3, Wo, bo, static_cast<unsigned char*>(packed)};
  const int total = 1024 + 8192 + 1024 + cm::kParFloats;
  cm::k_cmlp_pack<<<(total + 255) / 256, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(p);
  return cudaGetLastError() == cudaSuccess ? PTYCHO_OK : PTYCHO_ERR_LAUNCH;
}

static int cmlp_forward(int planar, const void* packed, const float* x, int N, float* y, int32_t* status_out,
                        ptycho_stream_t stream) {
  if (!packed || N < 0 || (N > 0 && (!x || !y))) return PTYCHO_ERR_INVALID_ARG;
  if (!pty_aligned(packed, 16) || !pty_aligned(x, planar ? 4 : 16) || !pty_aligned(y, 8))
    return PTYCHO_ERR_MISALIGNED;
  cm::Args a{static_cast<const unsigned char*>(packed), x, nullptr, N, reinterpret_cast<float2*>(y), nullptr,
             nullptr, status_out, 0, planar};
  return cm::launch(cm::k_cmlp_fwd, cm::kFwdSlots * cm::kTileThreads, cm::F_SMEM, a,
                    reinterpret_cast<cudaStream_t>(stream), nullptr);
}

int ptycho_cmlp_forward(const void* packed, const float* x, int N, float* y, int32_t* status_out,
                        ptycho_stream_t stream) {
  return cmlp_forward(0, packed, x, N, y, status_out, stream);
}

int ptycho_cmlp_forward_planar(const void* packed, const float* x_planar, int N, float* y, int32_t* status_out,
                               ptycho_stream_t stream) {
  return cmlp_forward(1, packed, x_planar, N, y, status_out, stream);
}

size_t ptycho_cmlp_backward_workspace_size(int N) {
  if (N < 0) return 0;
  const int ntiles = (N + 127) / 128;
  const int parts = ntiles < 1024 ? ntiles : 1024;  // at most one partial per SM is used
  return pty_align_up(size_t(parts > 0 ? parts : 1) * cm::kPartFloats * sizeof(float), 256);
}

static int cmlp_backward(int planar, const void* packed, const float* x, const float* gy, int N, float* gx, float* grad,
                         float* y, void* workspace, size_t workspace_bytes, int32_t* status_out,
                         ptycho_stream_t stream) {
  if (!packed || !grad || N < 0 || (N > 0 && (!x || !gy))) return PTYCHO_ERR_INVALID_ARG;
  const size_t ax = planar ? 4 : 16;  // feature-major values are read and written one by one
  if (!pty_aligned(packed, 16) || !pty_aligned(x, ax) || !pty_aligned(gy, 8) || !pty_aligned(gx, ax) ||
      !pty_aligned(y, 8))
    return PTYCHO_ERR_MISALIGNED;
  if (!workspace || workspace_bytes < ptycho_cmlp_backward_workspace_size(N)) return PTYCHO_ERR_WORKSPACE;
  {  // the persistent grid writes one partial per CTA: min(tiles, SMs) <= the sized count
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const int ntiles = (N + 127) / 128;
    const int grid = ntiles < nsm ? ntiles : nsm;
    if (size_t(grid) * cm::kPartFloats * sizeof(float) > workspace_bytes) return PTYCHO_ERR_WORKSPACE;
  }
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (N == 0) {
    cudaMemsetAsync(grad, 0, sizeof(float) * cm::kGradFloats, s);
    return cudaGetLastError() == cudaSuccess ? PTYCHO_OK : PTYCHO_ERR_LAUNCH;
  }
  cm::Args a{static_cast<const unsigned char*>(packed), x, reinterpret_cast<const float2*>(gy), N,
             reinterpret_cast<float2*>(y), gx, static_cast<float*>(workspace), status_out, planar, planar};
  int grid = 0;
  int st = cm::launch(cm::k_cmlp_bwd, cm::kBwdThreads, cm::B_SMEM, a, s, &grid);
  if (st) return st;
  cm::k_cmlp_reduce<<<(cm::kGradFloats + 31) / 32, 256, 0, s>>>(static_cast<const float*>(workspace), grid,
                                                                  grad);
  return cudaGetLastError() == cudaSuccess ? PTYCHO_OK : PTYCHO_ERR_LAUNCH;
}

int ptycho_cmlp_backward(const void* packed, const float* x, const float* gy, int N, float* gx, float* grad,
                         float* y, void* workspace, size_t workspace_bytes, int32_t* status_out,
                         ptycho_stream_t stream) {
  return cmlp_backward(0, packed, x, gy, N, gx, grad, y, workspace, workspace_bytes, status_out, stream);
}

int ptycho_cmlp_backward_planar(const void* packed, const float* x, const float* gy, int N, float* gx,
                                float* grad, float* y, void* workspace, size_t workspace_bytes,
                                int32_t* status_out, ptycho_stream_t stream) {
  return cmlp_backward(1, packed, x, gy, N, gx, grad, y, workspace, workspace_bytes, status_out, stream);
}

}  // extern "C"
