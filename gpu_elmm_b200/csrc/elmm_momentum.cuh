// elmm_momentum.cuh -- Convection + OtherTerms of one RK3 stage in one pass:
// CDS2 skew-symmetric advection (advection.f90:15-327,
// advection_variable_z.f90:15-324), explicit diffusion with the wall-flux
// corrections (momentum_diffusion.f90:169-420 and the wmfluxes-*-inc.f90
// includes), the RK combine (dynamics.f90:266-354, :450-478), the
// old-pressure gradient (dynamics.f90:58-199) and U2 += U (tsteps.f90:352-354).
//
// A block owns an MX x MY column of cells and marches up a chunk of L.kc
// planes.  U, V, W, Viscosity and Pr of each plane (with a one-cell halo in
// x and y) and the old Ustar (tile only) arrive by tensor-map TMA in a ring
// of kRingSlots plane slots in shared memory, requested several planes ahead
// of their use.  Every input cell is thus read from HBM once per chunk
// instead of once per stencil use.  The SGS kernel, k_sgs, streams U, V, W
// the same way.
#pragma once

#include <type_traits>

#include "elmm_common.cuh"
#include "elmm_packed.cuh"
#include "elmm_stream.cuh"

namespace elmm {

struct StageCoef {
  double rho, beta, alpha2;  // RK_rho, RK_beta, 2*RK_alpha of the stage
  int stage;
};

// MKC: the planes of a column the marching kernels start from (the host
// halves it on small grids, the autotuner tries up to kMaxChunk)
constexpr int MX = 32, MY = 8, MKC = 16, kMaxChunk = 32;
// per-tile context in shared memory: everything the stencil code reads
// besides the fields, so that no descriptor load sits on its critical path
template <typename T>
struct MomCtx {
  T cA[3], rec2[3];
  int wallmask;  // bit s: wall-model fluxes on side s
  int vz;
  int ext[3][3];
  const double *dzPr, *dzW;
  const T *fluxp[kFaces], *fluxm[kFaces];
  const unsigned char *bskip[3];
};

// called by every thread of the block, a value or two each (one thread alone
// took longer over its chain of loads than a short column of planes)
template <typename T>
__device__ __forceinline__ void fill_ctx(MomCtx<T> &m, const Dom<T> &d) {
  const int t = threadIdx.x;
  if (t < 9) {
    m.ext[t / 3][t % 3] = d.ext[t / 3][t % 3];
  } else if (t < 12) {
    m.cA[t - 9] = (T)d.cA[t - 9];
    m.rec2[t - 9] = (T)d.rec2[t - 9];
    m.bskip[t - 9] = d.bskip[t - 9];
  } else if (t == 12) {
    int wm = 0;
#pragma unroll
    for (int f = 0; f < 6; f++) wm |= d.wall[f] ? (1 << f) : 0;
    m.wallmask = wm;
    m.vz = d.vz;
  } else if (t == 13) {
    m.dzPr = d.dzPr; m.dzW = d.dzW;
  } else if (t >= 32 && t < 32 + kFaces) {
    m.fluxp[t - 32] = d.wm_fluxp[t - 32];
    m.fluxm[t - 32] = d.wm_fluxm[t - 32];
  }
}

// one value, or the two of a pair, from a plane of values; 0 where the byte
// mask (or null) is set
__device__ __forceinline__ float wall_ld(const float *p, float) { return p[0]; }
__device__ __forceinline__ double wall_ld(const double *p, double) { return p[0]; }
__device__ __forceinline__ F2 wall_ld(const float *p, F2) { return F2{make_float2(p[0], p[1])}; }
__device__ __forceinline__ float wall_keep(float a, const unsigned char *m) { return m && m[0] ? 0.f : a; }
__device__ __forceinline__ double wall_keep(double a, const unsigned char *m) { return m && m[0] ? 0.0 : a; }
__device__ __forceinline__ F2 wall_keep(F2 a, const unsigned char *m) {
  return m ? F2{make_float2(m[0] ? 0.f : a.v.x, m[1] ? 0.f : a.v.y)} : a;
}
__device__ __forceinline__ float wall_scale(float v, float) { return v; }
__device__ __forceinline__ double wall_scale(double v, double) { return v; }
__device__ __forceinline__ F2 wall_scale(float v, F2) { return bc2(v); }

// The wall-model corrections at the bottom and top: the diffusive flux
// through the face towards the wall taken back, the wall-model flux added
// (the wmfluxes-*-inc.f90 includes); with OFF on stored deviations, where a
// difference across levels is the stored difference plus the difference of
// the offsets (O, see tendency_dev).  For one cell or a pair (F2) whose first
// cell is (i, j); x and y are periodic for every domain, so no other side has
// a wall.  In the packed form: with one cell at a time the wall planes took a
// tile two to four planes' time, which on a small grid was the kernel's.
template <int C, bool OFF, typename T, typename N, typename RT>
__device__ __forceinline__ N wall_dev(const MomCtx<T> &m, const RT &R, const VelOffN<N> &O, int i, int j, int k) {
#define FN(dx, dy, dz) R.g(3, dx, dy, dz)
  const int *e = m.ext[C];
  const long long pxy = (long long)(i - 1) + (long long)e[0] * (j - 1);
  const N one = N{}, n0 = FN(0, 0, 0);
  const T rz = m.rec2[2];
  N a = cst(0.f, one);
  const N f = R.g(C, 0, 0, 0);
  // the viscosity sum of U's or V's face dz away (four times its mean)
  auto sum = [&](int dz) {
    return C == 0 ? ((FN(1, 0, 0) + FN(1, 0, dz)) + n0) + FN(0, 0, dz) : ((FN(0, 1, 0) + FN(0, 1, dz)) + n0) + FN(0, 0, dz);
  };
  const N *o = C == 0 ? O.o : O.p;
  if ((m.wallmask & (1 << SIDE_BO)) && k == 1) {
    N df = f - R.g(C, 0, 0, -1), c;
    if (C < 2) {
      if (OFF) df = df + (o[1] - o[0]);
      const T r = m.vz ? (T)(1.0 / m.dzW[k - 1 + 2] / m.dzPr[k + 2]) : rz;
      c = sum(-1) * df * wall_scale(r * (T)0.25, one);
    } else {
      const T r = m.vz ? (T)(1.0 / m.dzPr[k + 2] / m.dzW[k + 2]) : rz;
      c = n0 * df * wall_scale(r, one);
    }
    a = a + wall_keep(c + wall_ld(m.fluxp[C * 6 + SIDE_BO] + pxy, one), m.bskip[C] ? m.bskip[C] + pxy : nullptr);
  }
  if ((m.wallmask & (1 << SIDE_TO)) && k == e[2]) {
    N df = R.g(C, 0, 0, 1) - f, c;
    if (C < 2) {
      if (OFF) df = df + (o[2] - o[1]);
      const T r = m.vz ? (T)(1.0 / m.dzW[k + 2] / m.dzPr[k + 2]) : rz;
      c = sum(1) * df * wall_scale(r * (T)0.25, one);
    } else {
      const T r = m.vz ? (T)(1.0 / m.dzPr[k + 1 + 2] / m.dzW[k + 2]) : rz;
      c = FN(0, 0, 1) * df * wall_scale(r, one);
    }
    a = a - (c + wall_ld(m.fluxm[C * 6 + SIDE_TO] + pxy, one));
  }
#undef FN
  return a;
}

// Layout of one ring slot (one plane k of the tile): NWF "wide" fields with
// the x/y halo (rows j0-1..j0+MY, columns i0-XO..i0+MX+XO-1) and NNF
// "narrow" fields of the tile's own cells (rows j0..j0+MY-1, columns
// i0..i0+MX-1).  XO = 16 bytes of halo on each side keeps every copied row
// segment 16-byte aligned in global and shared memory.
template <typename T, int NWF, int NNF>
struct SlotLayout {
  static constexpr int XO = 16 / (int)sizeof(T);
  static constexpr int SPW = MX + 2 * XO;  // wide row
  static constexpr int WROWS = MY + 2;
  static constexpr int WB = ((WROWS * SPW * (int)sizeof(T) + 127) / 128) * 128 / (int)sizeof(T);  // wide block
  static constexpr int NB = ((MY * MX * (int)sizeof(T) + 127) / 128) * 128 / (int)sizeof(T);      // narrow block
  static constexpr int WIDE = NWF * WB;
  static constexpr int SIZE = WIDE + NNF * NB;  // elements per slot (a multiple of 128 bytes)
  static constexpr int BYTES = SIZE * (int)sizeof(T);
  static constexpr uint32_t WBOX = WROWS * SPW * sizeof(T);  // bytes one wide box delivers
  static constexpr uint32_t NBOX = MY * MX * sizeof(T);
};

// ring accessor: field f (wide), offsets (dx,dy) of the thread's cell and
// plane k+dz
template <typename T, int NWF, int NNF>
struct WideRing {
  typedef SlotLayout<T, NWF, NNF> Lay;
  const T *__restrict__ p[3];
  int o;
  __device__ __forceinline__ T g(int f, int dx, int dy, int dz) const {
    return p[dz + 1][f * Lay::WB + o + dy * Lay::SPW + dx];
  }
};

// Issues the tensor-map loads of plane kk of the tile into one slot: one
// box per field (thread 0 only).
template <typename T, int NWF, int NNF>
__device__ __forceinline__ void issue_plane(T *slot, uint64_t *bar, const CUtensorMap *maps, const int *wide,
                                            const int *narrow, bool with_narrow, int aln, int i0, int j0, int kk) {
  typedef SlotLayout<T, NWF, NNF> Lay;
  const uint32_t bytes = NWF * Lay::WBOX + (with_narrow ? NNF * Lay::NBOX : 0u);
  mbar_expect_tx(bar, bytes);
  const int xw = aln - 1 + i0 - Lay::XO, xn = aln - 1 + i0;
#pragma unroll
  for (int f = 0; f < NWF; f++) tma_load_3d(slot + f * Lay::WB, maps + BOX_WIDE * F_COUNT + wide[f], xw, j0 - 1, kk, bar);
  if (with_narrow) {
#pragma unroll
    for (int f = 0; f < NNF; f++)
      tma_load_3d(slot + Lay::WIDE + f * Lay::NB, maps + BOX_NARROW * F_COUNT + narrow[f], xn, j0, kk, bar);
  }
}

// The momentum kernel's planes: U, V, W, Viscosity, P wide; the old Ustar,
// Vstar, Wstar narrow (stages 2 and 3), and on the FP32 path also the
// potential temperature of the stage as a fourth narrow field (buoyancy),
// from its own tensor maps (tmapT: one per value buffer).
template <typename T, int NNF>
__device__ __forceinline__ void issue_mom_plane(T *slot, uint64_t *bar, const CUtensorMap *maps,
                                                const CUtensorMap *tmapT, bool with_star, int aln, int i0, int j0,
                                                int kk) {
  typedef SlotLayout<T, 5, NNF> Lay;
  const uint32_t bytes = 5 * Lay::WBOX + (with_star ? 3 * Lay::NBOX : 0u) + (tmapT ? Lay::NBOX : 0u);
  mbar_expect_tx(bar, bytes);
  const int xw = aln - 1 + i0 - Lay::XO, xn = aln - 1 + i0;
  const int wide[5] = {F_U, F_V, F_W, F_NU, F_P};
#pragma unroll
  for (int f = 0; f < 5; f++) tma_load_3d(slot + f * Lay::WB, maps + BOX_WIDE * F_COUNT + wide[f], xw, j0 - 1, kk, bar);
  if (with_star) {
#pragma unroll
    for (int f = 0; f < 3; f++)
      tma_load_3d(slot + Lay::WIDE + f * Lay::NB, maps + BOX_NARROW * F_COUNT + F_US + f, xn, j0, kk, bar);
  }
  if (NNF == 4 && tmapT) tma_load_3d(slot + Lay::WIDE + 3 * Lay::NB, tmapT, xn, j0, kk, bar);
}

constexpr int kRingSlots = 5;

// Cells per thread along x and ring slots of the momentum kernel: FP32
// threads compute two x-adjacent cells with packed FP32x2 arithmetic
// (elmm_packed.cuh); a four-slot ring leaves room for four 128-thread blocks
// per SM.  FP64 keeps one cell per thread and five slots.
// nnf: narrow fields per slot (FP32 adds the temperature; the FP64 slots
// would not leave room for two blocks per SM and read it from global memory).
template <typename T>
struct MomShape {
  static constexpr int cpt = 1, slots = 5, threads = MX * MY, min_blocks = 2, nnf = 3;
};
template <>
struct MomShape<float> {
  static constexpr int cpt = 2, slots = 4, threads = MX * MY / 2, min_blocks = 4, nnf = 4;
};

// L.kc: planes of a tile's column (a tuning choice: every cell's arithmetic
// is the same for any of them)
template <typename T>
__global__ void __launch_bounds__(MomShape<T>::threads, MomShape<T>::min_blocks)
    k_momentum(const Dom<T> *__restrict__ doms, Launch L, StageCoef sc) {
  constexpr int NNF = MomShape<T>::nnf;
  typedef SlotLayout<T, 5, NNF> Lay;
  constexpr int CPT = MomShape<T>::cpt, NSL = MomShape<T>::slots, TXN = MX / CPT;
  extern __shared__ __align__(128) unsigned char dyn_smem[];
  T *ring = reinterpret_cast<T *>(dyn_smem);
  __shared__ __align__(8) uint64_t bars[NSL];
  __shared__ MomCtx<T> ctx;
  // mixed path: offsets of U and V on planes k0-1 .. k0+kc of the tile (see Dom::voff)
  __shared__ float soff[2][kMaxChunk + 2];
  __shared__ int abort_flag;
  const int tx = threadIdx.x % TXN, ty = threadIdx.x / TXN;
  // tensor copies need 128-byte aligned destinations
  if (smem_addr(ring) & 127u) {
    if (threadIdx.x == 0) doms[0].flags[1] = 1;
    return;
  }
  if (threadIdx.x == 0) {
    for (int s2 = 0; s2 < NSL; s2++) mbar_init(&bars[s2], 1);
    abort_flag = 0;
    fence_async_shared();
  }
  __syncthreads();
  uint32_t phase = 0;  // bit s: parity of the next wait on slot s
  for (int t = blockIdx.x; t < L.total; t += gridDim.x) {
    const int di = find_dom(L.starts, L.nd, t);
    const Dom<T> &d = doms[di];
    int lt = t - __ldg(L.starts + di);
    const int ntx = (d.nx + MX - 1) / MX, nty = (d.ny + MY - 1) / MY;
    const int bx = lt % ntx; lt /= ntx;
    const int by = lt % nty;
    const int bk = lt / nty;
    const int i0 = bx * MX + 1, j0 = by * MY + 1, k0 = bk * L.kc + 1;
    const int k1 = min(k0 + L.kc - 1, d.nz);
    const int i = i0 + CPT * tx, j = j0 + ty;  // the thread's first cell
    const int nx = d.nx, ny = d.ny;
    const long long plane = d.plane;
    const bool stage1 = sc.stage == 1;
    const CUtensorMap *maps = reinterpret_cast<const CUtensorMap *>(d.tmaps);
    // the temperature of the stage start through the ring (FP32 with buoyancy)
    const CUtensorMap *tmapT = (NNF == 4 && d.buoy && d.tmapT)
                                   ? reinterpret_cast<const CUtensorMap *>(d.tmapT) + (sc.stage - 1) % 3
                                   : nullptr;
    // (asm memory clobbers in the loop below reload what is not in a register)
    const int skip = d.skip_plane, wait_limit = d.wait_limit, aln = d.aln;
    __syncthreads();  // every slot and the context of the previous tile are free
    if (threadIdx.x == 0) {
      fence_async_shared();
      for (int kk = k0 - 1; kk <= min(k0 - 1 + NSL - 1, k1 + 1); kk++)
        if (kk != skip)
          issue_mom_plane<T, NNF>(ring + (kk % NSL) * Lay::SIZE, &bars[kk % NSL], maps, tmapT, !stage1, aln, i0, j0,
                                  kk);
    }
    fill_ctx(ctx, d);
    if constexpr (sizeof(T) == 4) {
      if (threadIdx.x < 2 * (kMaxChunk + 2)) {
        const int c = threadIdx.x / (kMaxChunk + 2), kk = k0 - 1 + threadIdx.x % (kMaxChunk + 2);
        soff[c][kk - k0 + 1] = kk <= d.nz + 1 ? __ldg(d.voff + c * (d.nz + 2) + kk) : 0.f;
      }
    }
    __syncthreads();  // the context is written
    const T dt = (T)d.dt;
    const double coefd = sc.alpha2 * d.dt;
    const T coef = (T)coefd;
    const T gx = (T)(-coefd / d.dx), gy = (T)(-coefd / d.dy), gz = (T)(-coefd / d.dz);
    const T rdt = stage1 ? (T)0 : (T)sc.rho * dt, bdt = (T)sc.beta * dt;  // of the old and the new tendency
    const int kU = d.ext[0][2], kV = d.ext[1][2], kW = d.ext[2][2];
    const bool vz = d.vz != 0;
    // the mean pressure gradient's increments
    const T fx = d.prgx_on ? (-coef) * (T)d.prgx : (T)0, fy = d.prgy_on ? (-coef) * (T)d.prgy : (T)0;
    T *__restrict__ U2o = d.U2;
    T *__restrict__ V2o = d.V2;
    T *__restrict__ W2o = d.W2;
    T *__restrict__ Us = d.Us;
    T *__restrict__ Vs = d.Vs;
    T *__restrict__ Ws = d.Ws;
    const int o = (ty + 1) * Lay::SPW + (CPT * tx + Lay::XO);
    const bool inside0 = i <= nx && j <= ny;
    long long c = bidx(d, inside0 ? i : 1, inside0 ? j : 1, k0);
    const int nz = d.nz, nzp = nz + 2;
    // the walls (x and y are periodic): bottom and top
    const int wmask = (d.wall[SIDE_BO] ? 1 << SIDE_BO : 0) | (d.wall[SIDE_TO] ? 1 << SIDE_TO : 0);
    // both cells of the thread's pair have all three components (the pairs of
    // a partial tile past the last cell take the per-cell path)
    const bool pair_full = i + CPT - 1 <= min(d.ext[0][0], min(d.ext[1][0], d.ext[2][0])) &&
                           j <= min(d.ext[0][1], min(d.ext[1][1], d.ext[2][1]));
    // buoyancy of W (BuoyancyForce, src/dynamics.f90:679-688): A = g / T_ref;
    // with theta stored as theta - T_ref the constant term cancels exactly
    const bool buoy = d.buoy != 0;
    const T bA2 = (T)(d.grav / d.tref / 2.0);
    const T bsub = buoy && d.toff == 0 ? (T)(d.grav / d.tref * d.tref) : (T)0;
    const T *__restrict__ Tm = buoy ? d.slot[0].buf[(sc.stage - 1) % 3] : nullptr;  // theta at the stage start
    MomKN<F2> K2;
    if constexpr (CPT == 2) {
      for (int a = 0; a < 3; a++) {
        K2.A[a] = bc2((float)ctx.cA[a]);
        K2.r[a] = bc2((float)ctx.rec2[a]);
        K2.q[a] = bc2(0.25f * (float)ctx.rec2[a]);
      }
    }
    const T *__restrict__ kz2 = d.kz2;
    // FP64: the temperature of levels k and k + 1 rides along, that of k + 2
    // is on its way while level k is computed (its slots would not leave room
    // for two blocks per SM; loaded at their use, the two values were the
    // kernel's largest stall: 0.41 -> 0.385 ms at 256 x 256 x 128)
    T th0 = (T)0, th1 = (T)0;
    if (NNF == 3 && buoy && inside0) {
      th0 = ld(Tm, c);
      th1 = ld(Tm, c + plane);
    }
    // the wait for a plane's copies; a plane whose copies were issued always
    // lands before the block moves on or gives up (so no copy into this
    // block's shared memory outlives it): a lowered limit only cuts the wait
    // on a skipped one
    auto landed = [&](int kk, int s2) {
      bool w = mbar_wait(&bars[s2], (phase >> s2) & 1u, wait_limit);
      if (!w && kk != skip) w = mbar_wait(&bars[s2], (phase >> s2) & 1u);
      phase ^= 1u << s2;
      return w;
    };
    int sm = (k0 - 1) % NSL, s0 = k0 % NSL, sp = (k0 + 1) % NSL;  // slots of planes k-1, k, k+1
    bool ok = landed(k0 - 1, sm);
    ok &= landed(k0, s0);
    for (int k = k0; k <= k1; k++) {
      T th2 = (T)0;
      if (NNF == 3 && buoy && inside0 && k < k1) th2 = ld(Tm, c + 2 * plane);
      ok &= landed(k + 1, sp);
      if (!ok) { abort_flag = 1; d.flags[1] = 1; }
      const bool wallhere = ((wmask >> SIDE_BO) & (k == 1)) | ((wmask >> SIDE_TO) & (k >= nz - 1));
      const T *p0s = ring + sm * Lay::SIZE, *p1s = ring + s0 * Lay::SIZE, *p2s = ring + sp * Lay::SIZE;
      if (CPT == 2 && ok && pair_full && k <= min(kU, kV)) {
        if constexpr (CPT == 2) {
          // two cells per thread, every operation on a pair
          Ring2<Lay::WB, Lay::SPW> R2;
          R2.p[0] = p0s; R2.p[1] = p1s; R2.p[2] = p2s;
          R2.o = o;
          // the stencils take the offsets of U and V separately
          // (tendency_dev); the RK combine below works on the stored
          // deviations (U2 is stored the same way)
          VelOffN<F2> O;
#pragma unroll
          for (int q = 0; q < 3; q++) { O.o[q] = bc2(soff[0][k - k0 + q]); O.p[q] = bc2(soff[1][k - k0 + q]); }
          const float *nar = p1s + Lay::WIDE + ty * MX + CPT * tx;
          F2 btp = bc2(0.f);
          if (buoy) {
            const int ot = Lay::WIDE + 3 * Lay::NB + ty * MX + CPT * tx;  // the temperature, narrow field 3
            btp = bc2(bA2) * (F2{*reinterpret_cast<const float2 *>(p2s + ot)} +
                              F2{*reinterpret_cast<const float2 *>(p1s + ot)});
          }
          F2 tu, tv, tw;
          F2 gz2 = bc2(gz);
          const F2 zero = bc2(0.f);
          if (!vz) {
            tu = tendency_dev<0, false, true>(K2, R2, O, zero, (const KZN<F2> *)nullptr);
            tv = tendency_dev<1, false, true>(K2, R2, O, zero, (const KZN<F2> *)nullptr);
            tw = tendency_dev<2, false, true>(K2, R2, O, btp, (const KZN<F2> *)nullptr);
          } else {
            const float *kz = kz2 + k;
            KZN<F2> Z;
            Z.auv = bc2(__ldg(kz + KZ_AUV * nzp)); Z.buv = bc2(__ldg(kz + KZ_BUV * nzp));
            Z.d1uv = bc2(__ldg(kz + KZ_D1UV * nzp)); Z.d2uv = bc2(__ldg(kz + KZ_D2UV * nzp));
            Z.aw = bc2(__ldg(kz + KZ_AW * nzp)); Z.bw = bc2(__ldg(kz + KZ_BW * nzp));
            Z.d1w = bc2(__ldg(kz + KZ_D1W * nzp)); Z.d2w = bc2(__ldg(kz + KZ_D2W * nzp));
            gz2 = bc2((-coef) * __ldg(kz + KZ_RDZW * nzp));
            tu = tendency_dev<0, true, true>(K2, R2, O, zero, &Z);
            tv = tendency_dev<1, true, true>(K2, R2, O, zero, &Z);
            tw = tendency_dev<2, true, true>(K2, R2, O, btp, &Z);
          }
          if (wallhere) {
            tu = tu + wall_dev<0, true>(ctx, R2, O, i, j, k);
            tv = tv + wall_dev<1, true>(ctx, R2, O, i, j, k);
            tw = tw + wall_dev<2, true>(ctx, R2, O, i, j, k);
          }
          // the increments of the stage summed, then added; the pressure's
          // reference offset cancels in its differences
          const F2 p0 = R2.g(4, 0, 0, 0), rd = bc2(rdt), bd = bc2(bdt);
          F2 u2 = fm(bd, tu, fm(bc2(gx), R2.g(4, 1, 0, 0) - p0, bc2(fx)));
          F2 v2 = fm(bd, tv, fm(bc2(gy), R2.g(4, 0, 1, 0) - p0, bc2(fy)));
          F2 w2 = fm(bd, tw, gz2 * (R2.g(4, 0, 0, 1) - p0));
          if (!stage1) {
            u2 = fm(rd, F2{*reinterpret_cast<const float2 *>(nar)}, u2);
            v2 = fm(rd, F2{*reinterpret_cast<const float2 *>(nar + Lay::NB)}, v2);
            w2 = fm(rd, F2{*reinterpret_cast<const float2 *>(nar + 2 * Lay::NB)}, w2);
          }
          u2 = u2 + R2.g(0, 0, 0, 0);
          v2 = v2 + R2.g(1, 0, 0, 0);
          w2 = w2 + R2.g(2, 0, 0, 0);
          *reinterpret_cast<float2 *>(Us + c) = tu.v;
          *reinterpret_cast<float2 *>(U2o + c) = u2.v;
          *reinterpret_cast<float2 *>(Vs + c) = tv.v;
          *reinterpret_cast<float2 *>(V2o + c) = v2.v;
          if (k <= kW) {
            *reinterpret_cast<float2 *>(Ws + c) = tw.v;
            *reinterpret_cast<float2 *>(W2o + c) = w2.v;
          }
        }
      } else if (ok) {
        constexpr bool OFF = sizeof(T) == 4;
#pragma unroll 1
        for (int q = 0; q < CPT; q++) {
          const int iq = i + q;
          if (!(iq <= nx && j <= ny)) continue;
          WideRing<T, 5, 3> R;
          R.p[0] = p0s; R.p[1] = p1s; R.p[2] = p2s;
          R.o = o + q;
          const T *nar = p1s + Lay::WIDE + ty * MX + CPT * tx + q;  // narrow blocks are NB apart
          const long long cq = c + q;
          // all shared-memory reads first, then the stores: a global store in
          // between would make the compiler reload every shared value it may
          // alias
          const bool doU = iq <= d.ext[0][0] && j <= d.ext[0][1] && k <= kU;
          const bool doV = iq <= d.ext[1][0] && j <= d.ext[1][1] && k <= kV;
          const bool doW = iq <= d.ext[2][0] && j <= d.ext[2][1] && k <= kW;
          T bt = (T)0;
          if (buoy) {
            if constexpr (NNF == 4) {  // the temperature of planes k+1 and k from the ring
              const int ot = Lay::WIDE + 3 * Lay::NB + ty * MX + CPT * tx + q;
              bt = bA2 * (p2s[ot] + p1s[ot]);
            } else {
              bt = bA2 * (th1 + th0) - bsub;
            }
          }
          VelOffN<T> O;
#pragma unroll
          for (int q3 = 0; q3 < 3; q3++) {
            O.o[q3] = OFF ? (T)soff[0][k - k0 + q3] : (T)0;
            O.p[q3] = OFF ? (T)soff[1][k - k0 + q3] : (T)0;
          }
          MomKN<T> K1;
#pragma unroll
          for (int a3 = 0; a3 < 3; a3++) {
            K1.A[a3] = ctx.cA[a3];
            K1.r[a3] = ctx.rec2[a3];
            K1.q[a3] = (T)0.25 * ctx.rec2[a3];
          }
          T tu, tv, tw, gzk = gz;
          if (!vz) {
            tu = tendency_dev<0, false, OFF>(K1, R, O, (T)0, (const KZN<T> *)nullptr);
            tv = tendency_dev<1, false, OFF>(K1, R, O, (T)0, (const KZN<T> *)nullptr);
            tw = tendency_dev<2, false, OFF>(K1, R, O, bt, (const KZN<T> *)nullptr);
          } else {
            const T *kz = kz2 + k;
            KZN<T> Z1;
            Z1.auv = __ldg(kz + KZ_AUV * nzp); Z1.buv = __ldg(kz + KZ_BUV * nzp);
            Z1.d1uv = __ldg(kz + KZ_D1UV * nzp); Z1.d2uv = __ldg(kz + KZ_D2UV * nzp);
            Z1.aw = __ldg(kz + KZ_AW * nzp); Z1.bw = __ldg(kz + KZ_BW * nzp);
            Z1.d1w = __ldg(kz + KZ_D1W * nzp); Z1.d2w = __ldg(kz + KZ_D2W * nzp);
            gzk = (-coef) * __ldg(kz + KZ_RDZW * nzp);
            tu = tendency_dev<0, true, OFF>(K1, R, O, (T)0, &Z1);
            tv = tendency_dev<1, true, OFF>(K1, R, O, (T)0, &Z1);
            tw = tendency_dev<2, true, OFF>(K1, R, O, bt, &Z1);
          }
          if (wallhere) {
            tu = tu + wall_dev<0, OFF>(ctx, R, O, iq, j, k);
            tv = tv + wall_dev<1, OFF>(ctx, R, O, iq, j, k);
            tw = tw + wall_dev<2, OFF>(ctx, R, O, iq, j, k);
          }
          const T p0 = R.g(4, 0, 0, 0);
          T u2 = fm(bdt, tu, fm(gx, R.g(4, 1, 0, 0) - p0, fx));
          T v2 = fm(bdt, tv, fm(gy, R.g(4, 0, 1, 0) - p0, fy));
          T w2 = fm(bdt, tw, gzk * (R.g(4, 0, 0, 1) - p0));
          if (!stage1) {
            u2 = fm(rdt, nar[0], u2);
            v2 = fm(rdt, nar[Lay::NB], v2);
            w2 = fm(rdt, nar[2 * Lay::NB], w2);
          }
          u2 = u2 + R.g(0, 0, 0, 0);
          v2 = v2 + R.g(1, 0, 0, 0);
          w2 = w2 + R.g(2, 0, 0, 0);
          if (doU) { Us[cq] = tu; U2o[cq] = u2; }
          if (doV) { Vs[cq] = tv; V2o[cq] = v2; }
          if (doW) { Ws[cq] = tw; W2o[cq] = w2; }
        }
      }
      th0 = th1;
      th1 = th2;
      __syncthreads();  // plane k-1 is no longer read
      if (abort_flag) {
        // a plane did not arrive: wait (bounded) for the copies still in
        // flight into this block's shared memory, then give up
        if (threadIdx.x == 0)
          for (int kk = k + 2; kk <= min(k - 1 + NSL - 1, k1 + 1); kk++) {
            const int s2 = kk % NSL;
            if (kk != skip) mbar_wait(&bars[s2], (phase >> s2) & 1u);  // issued copies land: the full limit
            phase ^= 1u << s2;
          }
        return;
      }
      const int kn = k - 1 + NSL;
      if (threadIdx.x == 0 && kn <= k1 + 1 && kn != skip) {
        fence_async_shared();
        issue_mom_plane<T, NNF>(ring + sm * Lay::SIZE, &bars[sm], maps, tmapT, !stage1, aln, i0, j0, kn);
      }
      c += plane;
      sm = s0;
      s0 = sp;
      sp = sp + 1 == NSL ? 0 : sp + 1;
    }
  }
}

// ---------------------------------------------------------------- k_sgs
// SubgridStresses (src/dynamics.f90:869-908): Smagorinsky viscosity
// (SGS_Smag / NuSmag / StrainIJ, src/subgrid.f90:30-67, :170-209) from a
// ring of U, V, W planes (the ghosts of BoundViscosity,
// src/scalarboundaries.f90:326-431, are filled afterwards by k_ghosts).
// Cells next to a wall-model side compute the wall fluxes of the velocity
// points there.
template <typename T>
struct SgsK {  // factors of NuSmag at one level k
  T rdx, rdy, r4dx, r4dy, rdz, r2zz, wc2;
  // mixed path: the part of the z differences of U and V (D02, D12) that
  // comes from their per-level offsets, 2 (off(k+1) - off(k-1)) r2zz, in
  // shared memory per plane of the tile (the ring holds the stored
  // deviations; every other difference is taken within one level, where the
  // offset cancels)
  const float *du, *dv;
};

// One cell (float, double) or a pair (F2).  The divisions by the (uniform)
// spacings of StrainIJ are multiplications by reciprocals computed once; the
// symmetric pairs of the strain tensor are formed once, 2 S = 2 sum D_aa^2 +
// sum (D_ab + D_ba)^2, with fused multiply-adds: 36 operations where the
// nine terms of Strainu took 68 (256 x 256 x 128, k_sgs and k_wm_points one
// after the other: FP32 93 -> 78 us, FP64 154 -> 132).  The square root is taken per cell.
__device__ __forceinline__ float root(float a) { return sqrtf(a); }
__device__ __forceinline__ double root(double a) { return sqrt(a); }
__device__ __forceinline__ F2 root(F2 a) { return F2{make_float2(sqrtf(a.v.x), sqrtf(a.v.y))}; }
template <bool OFF, typename T, typename N, typename RT>
__device__ __forceinline__ N nusmag(const SgsK<T> &q, const RT &R, N) {
#define GU(dx, dy, dz) R.g(0, dx, dy, dz)
#define GV(dx, dy, dz) R.g(1, dx, dy, dz)
#define GW(dx, dy, dz) R.g(2, dx, dy, dz)
  auto k = [](T v) { return wall_scale(v, N{}); };  // a factor, broadcast to a pair
  const N r4dx = k(q.r4dx), r4dy = k(q.r4dy), r2zz = k(q.r2zz);
  const N d0 = (GU(0, 0, 0) - GU(-1, 0, 0)) * k(q.rdx), d1 = (GV(0, 0, 0) - GV(0, -1, 0)) * k(q.rdy),
          d2 = (GW(0, 0, 0) - GW(0, 0, -1)) * k(q.rdz);
  const N S = fm(d2, d2, fm(d1, d1, d0 * d0));
  const N uy = (GU(0, 1, 0) + GU(-1, 1, 0)) - (GU(0, -1, 0) + GU(-1, -1, 0));
  const N vx = (GV(1, 0, 0) + GV(1, -1, 0)) - (GV(-1, 0, 0) + GV(-1, -1, 0));
  const N t01 = fm(uy, r4dy, vx * r4dx);
  const N uz = (GU(0, 0, 1) + GU(-1, 0, 1)) - (GU(0, 0, -1) + GU(-1, 0, -1));
  const N wx = (GW(1, 0, 0) + GW(1, 0, -1)) - (GW(-1, 0, 0) + GW(-1, 0, -1));
  const N t02 = fm(wx, r4dx, OFF ? fm(uz, r2zz, k((T)*q.du)) : uz * r2zz);
  const N vz = (GV(0, 0, 1) + GV(0, -1, 1)) - (GV(0, 0, -1) + GV(0, -1, -1));
  const N wy = (GW(0, 1, 0) + GW(0, 1, -1)) - (GW(0, -1, 0) + GW(0, -1, -1));
  const N t12 = fm(wy, r4dy, OFF ? fm(vz, r2zz, k((T)*q.dv)) : vz * r2zz);
#undef GU
#undef GV
#undef GW
  return root(fm(t12, t12, fm(t02, t02, fm(t01, t01, S + S)))) * k(q.wc2);
}

// ComputeTDiff (src/scalar_diffusion.f90:983-1009): the temperature
// diffusivity from the viscosity, constant Pr_sgs = 0.6
// (src/scalar_diffusion.f90:22)
template <typename T>
__device__ __forceinline__ T tdiff_of(T nu, T nu_mol, T kappa_mol) {
  return nu_mol > 0 ? (nu - nu_mol) / (T)0.6 + kappa_mol : nu / (T)0.6;
}

// Cells per thread of k_sgs: two for FP32 (packed arithmetic), one for FP64.
template <typename T>
struct SgsShape {
  static constexpr int cpt = 1, threads = MX * MY, min_blocks = 3;
};
template <>
struct SgsShape<float> {
  static constexpr int cpt = 2, threads = MX * MY / 2, min_blocks = 7;
};

// init: 0 a stage (viscosity and diffusivity), 1 the initial viscosity and
// diffusivity after the projection, 2 the autotuner's timing launches (a
// stage's arithmetic; its outputs the real stage overwrites).  The
// wall-model points are k_wm_points'.
template <typename T>
__global__ void __launch_bounds__(SgsShape<T>::threads, SgsShape<T>::min_blocks)
    k_sgs(const Dom<T> *__restrict__ doms, Launch L, int init) {
  // planes of U, V, W (tile plus one-cell halo) arrive by tensor-map TMA in
  // a ring of kRingSlots slots, as in k_momentum
  typedef SlotLayout<T, 3, 0> Lay;
  constexpr int CPT = SgsShape<T>::cpt, TXN = MX / CPT;
  extern __shared__ __align__(128) unsigned char dyn_smem[];
  T *ring = reinterpret_cast<T *>(dyn_smem);
  __shared__ __align__(8) uint64_t bars[kRingSlots];
  __shared__ int abort_flag;
  // the factors 1/dzPr, 1/(2 (zPr(k+1) - zPr(k-1))), (width Cs)^2 of the tile's planes
  __shared__ T sfac[3][kMaxChunk];
  // mixed path: the z-difference parts du, dv of the tile's planes (SgsK)
  __shared__ float sdz[2][kMaxChunk];
  const int tx = threadIdx.x % TXN, ty = threadIdx.x / TXN;
  if (smem_addr(ring) & 127u) {  // tensor copies need 128-byte aligned destinations
    if (threadIdx.x == 0) doms[0].flags[1] = 1;
    return;
  }
  if (threadIdx.x == 0) {
    for (int s2 = 0; s2 < kRingSlots; s2++) mbar_init(&bars[s2], 1);
    abort_flag = 0;
    fence_async_shared();
  }
  __syncthreads();
  uint32_t phase = 0;  // bit s: parity of the next wait on slot s
  for (int t = blockIdx.x; t < L.total; t += gridDim.x) {
    const int di = find_dom(L.starts, L.nd, t);
    const Dom<T> &d = doms[di];
    int lt = t - __ldg(L.starts + di);
    const int ntx = (d.nx + MX - 1) / MX, nty = (d.ny + MY - 1) / MY;
    const int bx = lt % ntx; lt /= ntx;
    const int by = lt % nty;
    const int bk = lt / nty;
    const int i0 = bx * MX + 1, j0 = by * MY + 1, k0 = bk * L.kc + 1;
    const int k1 = min(k0 + L.kc - 1, d.nz);
    const int i = i0 + CPT * tx, j = j0 + ty;  // the thread's first cell
    const int nx = d.nx, ny = d.ny, nz = d.nz;
    const int wide[3] = {F_U, F_V, F_W};
    const int none[1] = {0};
    const CUtensorMap *maps = reinterpret_cast<const CUtensorMap *>(d.tmaps);
    const int skip = d.skip_plane, wait_limit = d.wait_limit, aln = d.aln;
    __syncthreads();  // every slot and the level factors of the previous tile are free
    if (threadIdx.x == 0) {
      fence_async_shared();
      for (int kk = k0 - 1; kk <= min(k0 - 1 + kRingSlots - 1, k1 + 1); kk++)
        if (kk != skip)
          issue_plane<T, 3, 0>(ring + (kk % kRingSlots) * Lay::SIZE, &bars[kk % kRingSlots], maps, wide, none, false,
                               aln, i0, j0, kk);
    }
    if constexpr (sizeof(T) == 4) {
      if (threadIdx.x < 2 * kMaxChunk) {
        const int c = threadIdx.x / kMaxChunk, kk = k0 + threadIdx.x % kMaxChunk;
        if (kk <= k1) {
          const float *o = d.voff + c * (d.nz + 2);
          sdz[c][kk - k0] = 2.f * (__ldg(o + kk + 1) - __ldg(o + kk - 1)) * (float)d.sgs_r2zz[kk];
        }
      }
    }
    if (threadIdx.x < 3 * kMaxChunk) {
      const int c = threadIdx.x / kMaxChunk, kk = k0 + threadIdx.x % kMaxChunk;
      const double *tab = c == 0 ? d.sgs_rdz : c == 1 ? d.sgs_r2zz : d.sgs_wc2;
      if (kk <= k1) sfac[c][kk - k0] = (T)tab[kk];
    }
    __syncthreads();  // the factors are written
    const T num = (T)d.nu_mol;
    const bool sgs = d.sgs != 0, addmol = d.nu_mol > 0;
    // the scalar diffusivity too: every stage with buoyancy (ComputeTDiff,
    // src/dynamics.f90:904), and once after the initial projection whenever
    // a scalar is transported (src/initial.f90:4296-4313, which uses the
    // first formula of ComputeTDiff for any molecular viscosity)
    const bool buoy = d.tdiff_live != 0 || (init == 1 && d.nslot > 0);
    const T kap = (T)d.kappa_mol;
    SgsK<T> q;
    q.rdx = (T)(1.0 / d.dx); q.rdy = (T)(1.0 / d.dy);
    q.r4dx = (T)(1.0 / (4 * d.dx)); q.r4dy = (T)(1.0 / (4 * d.dy));
    T *__restrict__ nu = d.nu;
    T *__restrict__ td_out = d.TDiff;
    const int o = (ty + 1) * Lay::SPW + (CPT * tx + Lay::XO);
    const bool inside0 = i <= nx && j <= ny;
    const bool pair_inside = i + CPT - 1 <= nx && j <= ny;
    long long c = bidx(d, inside0 ? i : 1, inside0 ? j : 1, k0);
    const long long plane = d.plane;
    auto landed = [&](int kk, int s2) {  // as in k_momentum
      bool w = mbar_wait(&bars[s2], (phase >> s2) & 1u, wait_limit);
      if (!w && kk != skip) w = mbar_wait(&bars[s2], (phase >> s2) & 1u);
      phase ^= 1u << s2;
      return w;
    };
    int sm = (k0 - 1) % kRingSlots, s0 = k0 % kRingSlots, sp = (k0 + 1) % kRingSlots;  // slots of planes k-1, k, k+1
    bool ok = landed(k0 - 1, sm);
    ok &= landed(k0, s0);
    for (int k = k0; k <= k1; k++) {
      q.rdz = sfac[0][k - k0]; q.r2zz = sfac[1][k - k0]; q.wc2 = sfac[2][k - k0];
      q.du = &sdz[0][k - k0];
      q.dv = &sdz[1][k - k0];
      ok &= landed(k + 1, sp);
      if (!ok) { abort_flag = 1; d.flags[1] = 1; }
      const T *p0s = ring + sm * Lay::SIZE, *p1s = ring + s0 * Lay::SIZE, *p2s = ring + sp * Lay::SIZE;
      if (ok && CPT == 2 && sgs && pair_inside) {
        if constexpr (CPT == 2) {
          Ring2<Lay::WB, Lay::SPW> R2;
          R2.p[0] = p0s; R2.p[1] = p1s; R2.p[2] = p2s;
          R2.o = o;
          F2 v = nusmag<true>(q, R2, F2{});
          if (addmol) v = v + bc2(num);
          *reinterpret_cast<float2 *>(nu + c) = v.v;
          // the periodic x ghosts of the row's end cells (the ghost pass covers y and z)
          if (i == 1) nu[c + nx] = v.v.x;
          if (i + 1 == nx) nu[c + 1 - nx] = v.v.y;
          if (buoy) {
            const float2 td = init == 1 ? make_float2((v.v.x - num) / 0.6f + kap, (v.v.y - num) / 0.6f + kap)
                                   : make_float2(tdiff_of(v.v.x, num, kap), tdiff_of(v.v.y, num, kap));
            *reinterpret_cast<float2 *>(td_out + c) = td;
          }
        }
      } else if (ok) {
#pragma unroll
        for (int qc = 0; qc < CPT; qc++) {
          if (!(i + qc <= nx && j <= ny)) continue;
          WideRing<T, 3, 0> R;
          R.p[0] = p0s; R.p[1] = p1s; R.p[2] = p2s;
          R.o = o + qc;
          T v = num;
          if (sgs) {
            v = nusmag<sizeof(T) == 4>(q, R, T{});
            if (addmol) v = v + num;
          }
          nu[c + qc] = v;
          if (i + qc == 1) nu[c + qc + nx] = v;  // periodic x ghosts (the ghost pass covers y and z)
          if (i + qc == nx) nu[c + qc - nx] = v;
          if (buoy) td_out[c + qc] = init == 1 ? (v - num) / (T)0.6 + kap : tdiff_of(v, num, kap);
        }
      }
      __syncthreads();  // plane k-1 is no longer read
      if (abort_flag) {
        // a plane did not arrive: wait (bounded) for the copies still in
        // flight into this block's shared memory, then give up
        if (threadIdx.x == 0)
          for (int kk = k + 2; kk <= min(k - 1 + kRingSlots - 1, k1 + 1); kk++) {
            const int s2 = kk % kRingSlots;
            if (kk != skip) mbar_wait(&bars[s2], (phase >> s2) & 1u);  // issued copies land: the full limit
            phase ^= 1u << s2;
          }
        return;
      }
      const int kn = k - 1 + kRingSlots;
      if (threadIdx.x == 0 && kn <= k1 + 1 && kn != skip) {
        fence_async_shared();
        issue_plane<T, 3, 0>(ring + sm * Lay::SIZE, &bars[sm], maps, wide, none, false,
                             aln, i0, j0, kn);
      }
      c += plane;
      sm = s0;
      s0 = sp;
      sp = sp + 1 == kRingSlots ? 0 : sp + 1;
    }
  }
}

}  // namespace elmm
