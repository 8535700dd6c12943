// elmm_packed.cuh -- the wall-free tendency of a velocity component
// (tendency_dev<C>) for one cell (float, double) or, on the mixed path, a pair
// of x-adjacent cells in packed FP32x2 arithmetic (sm_100 FFMA2 / FADD2 /
// FMUL2: one instruction per operation pair).
#pragma once

#include <cuda_runtime.h>

namespace elmm {

struct F2 {
  float2 v;
};

__device__ __forceinline__ F2 bc2(float a) { return F2{make_float2(a, a)}; }
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { return F2{__fadd2_rn(a.v, b.v)}; }
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { return F2{__fmul2_rn(a.v, b.v)}; }
// a - b: the product b * (-1) is exact, so this is one rounding of a - b
__device__ __forceinline__ F2 operator-(F2 a, F2 b) { return F2{__ffma2_rn(b.v, make_float2(-1.f, -1.f), a.v)}; }
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) { return F2{__ffma2_rn(a.v, b.v, c.v)}; }

// Pair accessor over the momentum plane ring: the thread's two cells sit at
// o and o + 1 of a slot (o even, so pairs at even offsets are 8-byte
// aligned); a pair at an odd x offset is assembled from its two aligned
// neighbours.
template <int WB, int SPW>
struct Ring2 {
  const float *__restrict__ p[3];  // planes k-1, k, k+1
  int o;
  __device__ __forceinline__ float2 ld(const float *q) const { return *reinterpret_cast<const float2 *>(q); }
  __device__ __forceinline__ F2 g(int f, int dx, int dy, int dz) const {
    const float *b = p[dz + 1] + f * WB + o + dy * SPW;
    if ((dx & 1) == 0) return F2{ld(b + dx)};
    const float2 lo = ld(b + dx - 1), hi = ld(b + dx + 1);
    return F2{make_float2(lo.y, hi.x)};
  }
};

// Arithmetic on one value (float, double) or on a pair (F2) in the same source.
__device__ __forceinline__ float cst(float a, float) { return a; }
__device__ __forceinline__ double cst(float a, double) { return (double)a; }
__device__ __forceinline__ F2 cst(float a, F2) { return bc2(a); }
__device__ __forceinline__ float fm(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fm(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ F2 fm(F2 a, F2 b, F2 c) { return fma2(a, b, c); }

// per-tile constants of the tendencies (broadcast to a pair)
template <typename N>
struct MomKN {
  N A[3], r[3], q[3];  // cA, rec2, rec2 / 4
};

// Stretched z (CDU/CDV/CDW_variable_z, src/advection_variable_z.f90:15-324,
// and MomentumDiffusion_variable_z_nobranch_2ord, src/momentum_diffusion.f90:
// 298-420): the divisions by dzPr(k), dzW(k) and the centred differences of
// zPr, zW become multiplications by per-level factors computed once in FP64
// (rounded to FP32 on the mixed path).
// Table rows of Dom::kz2:
enum {
  KZ_AUV = 0,   // 1 / (4 dzPr(k))                    U, V advection through z faces
  KZ_BUV = 1,   // 1 / (4 (zPr(k+1) - zPr(k-1)))       U, V advective form, W averaged over 4
  KZ_D1UV = 2,  // 1 / (dzW(k) dzPr(k))                U, V diffusion through the top face
  KZ_D2UV = 3,  // 1 / (dzW(k-1) dzPr(k))              ... the bottom face
  KZ_AW = 4,    // 1 / (4 dzW(k))                      W advection
  KZ_BW = 5,    // 1 / (zW(k+1) - zW(k-1))             W advective form
  KZ_D1W = 6,   // 1 / (dzPr(k+1) dzW(k))              W diffusion, top
  KZ_D2W = 7,   // 1 / (dzPr(k) dzW(k))                W diffusion, bottom
  KZ_RDZW = 8,  // 1 / dzW(k)                          pressure gradient of W
  kZ2 = 9
};
template <typename N>
struct KZN {
  N auv, buv, d1uv, d2uv, aw, bw, d1w, d2w;
};

// The per-level offsets of U (o) and V (p) on planes k-1, k, k+1 (the mixed
// path stores U and V as deviations from them; see Dom::voff).
template <typename N>
struct VelOffN {
  N o[3], p[3];
};

// One velocity component's tendency without wall corrections: the
// skew-symmetric CDS2 advection (advection.f90:15-327,
// advection_variable_z.f90:15-324 with VZ) and the explicit diffusion
// (momentum_diffusion.f90:169-420).  OFF: the FP32 state, whose U and V hold
// deviations from per-level offsets (O); the offsets enter only where the
// full value is needed, so that every difference of neighbouring values is a
// difference of stored ones and no rounded products of the full ~several m/s
// velocity are subtracted, whose noise the projection would turn into
// pressure.
//
// The two forms of the advection share their factors, so along each axis
// they are summed before they are evaluated.  With values f, neighbours f+,
// f- and the transporting velocity's sums B, D on the two faces (twice their
// face values):
//   along itself   A (f+ - f-) (f+ + f- + 4 f),                 A = 1 / (4 d)
//   across         A ((f+ - f-) (B + D) + (B - D) (f+ + f-) / 2 + (B - D) f)
// where (f+ + f) B - (f + f-) D = ((f+ - f-) (B + D) + (f+ + 2 f + f-) (B - D)) / 2
// and the advective form adds A / 2 (f+ - f-) (B + D).  That and fused
// multiply-adds take some 58 operations a component where the two forms term
// by term took 105; the kernel is bound by their issue and latency (with
// buoyancy, 256 x 256 x 128: FP32 152 -> 127 us, 3.96 TB/s of its 15 words a
// cell; FP64, whose form before was the reference's with its divisions, 408
// -> 234 us, 4.3 TB/s).  bt: the buoyancy of W.
template <int C, bool VZ, bool OFF, typename N, typename RT>
__device__ __forceinline__ N tendency_dev(const MomKN<N> &K, const RT &R, const VelOffN<N> &O, N bt,
                                          const KZN<N> *Z) {
  const N half = cst(0.5f, N{}), two = cst(2.f, N{}), four = cst(4.f, N{});
  N a;
  if constexpr (C < 2) {
    // the component f of axis C, the other horizontal component g; offsets
    // along the component's own axis and across it
#define F(al, cr, dz) (C == 0 ? R.g(0, al, cr, dz) : R.g(1, cr, al, dz))
#define G(al, cr, dz) (C == 0 ? R.g(1, al, cr, dz) : R.g(0, cr, al, dz))
#define H(al, dz) (C == 0 ? R.g(2, al, 0, dz) : R.g(2, 0, al, dz))
#define M(al, cr, dz) (C == 0 ? R.g(3, al, cr, dz) : R.g(3, cr, al, dz))
    const N Ka = K.A[C], Kc = K.A[1 - C], Kz = K.A[2];
    const N *o = C == 0 ? O.o : O.p, *p = C == 0 ? O.p : O.o;
    const N f = F(0, 0, 0), fe = F(1, 0, 0), fw = F(-1, 0, 0), fn = F(0, 1, 0), fs = F(0, -1, 0);
    const N ft = F(0, 0, 1), fb = F(0, 0, -1);
    N s = fm(four, f, fe + fw);
    if (OFF) s = fm(cst(6.f, N{}), o[1], s);
    N acc = (Ka * (fe - fw)) * s;
    {
      const N B = G(1, 0, 0) + G(0, 0, 0), D = G(1, -1, 0) + G(0, -1, 0), BpD = B + D, BmD = B - D, df = fn - fs;
      N t = fm(half, fn + fs, f);
      if (OFF) t = fm(two, o[1], t);
      const N y = fm(BmD, t, df * (OFF ? fm(four, p[1], BpD) : BpD));
      acc = fm(Kc, y, acc);
    }
    {
      const N P = H(1, 0) + H(0, 0), Q = H(1, -1) + H(0, -1), PpQ = P + Q, PmQ = P - Q;
      N df = ft - fb, t = fm(two, f, ft + fb);
      if (OFF) {
        df = df + (o[2] - o[0]);
        t = t + fm(two, o[1], o[2] + o[0]);
      }
      if (VZ) {
        const N c2 = half * Z->auv;
        acc = fm(df * PpQ, c2 + Z->buv, acc);
        acc = fm(t * PmQ, c2, acc);
      } else {
        acc = fm(Kz, fm(half, t * PmQ, df * PpQ), acc);
      }
    }
    a = acc * cst(-0.5f, N{});
    const N n0 = M(0, 0, 0), ne = M(1, 0, 0), s0 = ne + n0;
    a = fm(K.r[C], fm(n0, fw - f, ne * (fe - f)), a);
    const N sN = s0 + (M(1, 1, 0) + M(0, 1, 0)), sS = s0 + (M(1, -1, 0) + M(0, -1, 0));
    a = fm(K.q[1 - C], fm(sS, fs - f, sN * (fn - f)), a);
    const N sT = s0 + (M(1, 0, 1) + M(0, 0, 1)), sB = s0 + (M(1, 0, -1) + M(0, 0, -1));
    N dT = ft - f, dB = fb - f;
    if (OFF) {
      dT = dT + (o[2] - o[1]);
      dB = dB + (o[0] - o[1]);
    }
    if (VZ) {
      const N q = cst(0.25f, N{});
      a = fm(sT * dT, q * Z->d1uv, a);
      a = fm(sB * dB, q * Z->d2uv, a);
    } else {
      a = fm(K.q[2], fm(sB, dB, sT * dT), a);
    }
#undef F
#undef G
#undef H
#undef M
  } else {
#define FU(dx, dy, dz) R.g(0, dx, dy, dz)
#define FV(dx, dy, dz) R.g(1, dx, dy, dz)
#define FN(dx, dy, dz) R.g(3, dx, dy, dz)
    const N w = R.g(2, 0, 0, 0), we = R.g(2, 1, 0, 0), ww = R.g(2, -1, 0, 0), wn = R.g(2, 0, 1, 0);
    const N ws = R.g(2, 0, -1, 0), wt = R.g(2, 0, 0, 1), wb = R.g(2, 0, 0, -1);
    N acc;
    if (VZ) acc = (wt - wb) * fm(Z->aw, fm(two, w, wt + wb), Z->bw * w);
    else acc = (K.A[2] * (wt - wb)) * fm(four, w, wt + wb);
    {
      const N B = FV(0, 0, 1) + FV(0, 0, 0), D = FV(0, -1, 1) + FV(0, -1, 0), BpD = B + D;
      const N y = fm(B - D, fm(half, wn + ws, w), (wn - ws) * (OFF ? fm(two, O.p[1] + O.p[2], BpD) : BpD));
      acc = fm(K.A[1], y, acc);
    }
    {
      const N B = FU(0, 0, 1) + FU(0, 0, 0), D = FU(-1, 0, 1) + FU(-1, 0, 0), BpD = B + D;
      const N x = fm(B - D, fm(half, we + ww, w), (we - ww) * (OFF ? fm(two, O.o[1] + O.o[2], BpD) : BpD));
      acc = fm(K.A[0], x, acc);
    }
    a = fm(acc, cst(-0.5f, N{}), bt);
    const N n0 = FN(0, 0, 0), nt = FN(0, 0, 1), s0 = nt + n0;
    const N sE = s0 + (FN(1, 0, 1) + FN(1, 0, 0)), sW = s0 + (FN(-1, 0, 1) + FN(-1, 0, 0));
    a = fm(K.q[0], fm(sW, ww - w, sE * (we - w)), a);
    const N sN = s0 + (FN(0, 1, 1) + FN(0, 1, 0)), sS = s0 + (FN(0, -1, 1) + FN(0, -1, 0));
    a = fm(K.q[1], fm(sS, ws - w, sN * (wn - w)), a);
    if (VZ) {
      a = fm(nt * (wt - w), Z->d1w, a);
      a = fm(n0 * (wb - w), Z->d2w, a);
    } else {
      a = fm(K.r[2], fm(n0, wb - w, nt * (wt - w)), a);
    }
#undef FU
#undef FV
#undef FN
  }
  return a;
}

}  // namespace elmm
