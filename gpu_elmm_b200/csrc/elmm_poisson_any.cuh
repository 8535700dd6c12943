// elmm_poisson_any.cuh -- the x and y transforms of the Poisson problem
// (src/poisson.f90:76-210, the PoisFFT replacement) for every length that
// factors into 2, 3 and 5 and has no register FFT of its own
// (fft_reg_supported and fft_reg_y, elmm_fftreg.cuh), and for
// elmm_poisson_solve_noalloc.
//
// A length is split into few large radices (up to 16: two passes to 256,
// three to 4096), each pass one decimation-in-frequency butterfly per thread
// in registers, in place, with one barrier a pass.  Sequences lie interleaved
// in shared memory, element n of sequence s at n * pitch + s with s the
// fastest lane index: neighbouring lanes share a twiddle and read neighbouring
// words, and one division by the pass's block length serves a whole butterfly.
//
// Bound by instructions and the latency of a tile's passes, not by memory:
// 512 x 512 x 128, FP32, against radices 2 to 5 on strided sequences with two
// buffers (the form before): y 0.637 -> 0.080 ms, x forward 0.868 -> 0.228,
// x inverse 0.395 -> 0.213 (512 itself now has a register transform: 0.086,
// 0.148 and 0.077); 135 x 135 x 75: y 20 -> 16 us, x 56 -> 24 and 26 -> 19.
#pragma once

#include "elmm_poisson_reg.cuh"

namespace elmm {

// FFT factorisations and x tile of one domain
struct PoisPlan {
  FFTFactors fx, fy;
  int nsx;  // complex sequences (pairs of rows) of an x tile, a power of two
};

constexpr int kFFTThreads = 256, kFFTThreadsX = 128;
// the longest axes of the generic transforms: 8 rows (x) or TyOf columns (y)
// twice in shared memory
constexpr int kRowsX = 8;
// an x tile: two buffers of at most this many bytes together, of which six
// (FP32) or four (FP64) blocks share an SM: each pass is a chain of a
// shared-memory round trip, the butterfly and a barrier, and small blocks
// fill each other's (135 x 135 x 75, FP32: forward 28 us with tiles of 50 KB
// and 256 threads, 24 with these)
constexpr int kTileBytesX = 25 << 10, kMaxSeqX = 32;

template <typename T> struct TyOf;
template <> struct TyOf<double> { static constexpr int v = 8; };
template <> struct TyOf<float> { static constexpr int v = 16; };

__host__ __device__ constexpr int fft_any_pitch(int ns) { return ns + 1; }
template <typename T>
inline size_t fft_any_smem_x(int n, int ns) {
  return 2 * sizeof(typename Vec2<T>::type) * (size_t)n * fft_any_pitch(ns);
}
template <typename T>
inline size_t fft_any_smem_y(int n) {
  return sizeof(typename Vec2<T>::type) * (size_t)n * TyOf<T>::v;
}
// the sequences of an x tile of length n
template <typename T>
inline int fft_any_seqs(int n) {
  int ns = kMaxSeqX;
  while (ns > 1 && fft_any_smem_x<T>(n, ns) > (size_t)kTileBytesX) ns /= 2;
  return ns;
}

// calls f(std::integral_constant<int, R>) for the radix R of a pass
template <typename F>
__device__ __forceinline__ void fft_radix(int R, F &&f) {
  switch (R) {
    case 2: f(std::integral_constant<int, 2>{}); break;
    case 3: f(std::integral_constant<int, 3>{}); break;
    case 4: f(std::integral_constant<int, 4>{}); break;
    case 5: f(std::integral_constant<int, 5>{}); break;
    case 6: f(std::integral_constant<int, 6>{}); break;
    case 8: f(std::integral_constant<int, 8>{}); break;
    case 9: f(std::integral_constant<int, 9>{}); break;
    case 10: f(std::integral_constant<int, 10>{}); break;
    case 12: f(std::integral_constant<int, 12>{}); break;
    case 15: f(std::integral_constant<int, 15>{}); break;
    default: f(std::integral_constant<int, 16>{}); break;
  }
}

// where butterfly q of pass p sits: block of length len = R M, offset m in it
struct DifPos {
  int base, m;
};
__device__ __forceinline__ DifPos dif_pos(const FFTFactors &f, int p, int q) {
  const int M = f.M[p];
  const int blk = M == 1 ? q : (int)__umulhi((unsigned)q, f.magic[p]);
  const int m = q - blk * M;
  return DifPos{blk * M * f.fac[p] + m, m};
}
// the frequency of point 0 of the last pass's butterfly q (its points are
// n / R apart): the radices' digits of q in reverse
__device__ __forceinline__ int dif_freq(const FFTFactors &f, int q) {
  int k = 0;
  for (int t = f.nfac - 2; t >= 1; t--) {
    const int r = q / f.fac[t];
    k += (q - r * f.fac[t]) * f.step[t];
    q = r;
  }
  return k + q;
}

// the R-point DFT of a pass and, unless it is the last, the twiddles
// W_len^(m k) (table W_n)
template <typename T, typename T2, int R, bool INV, bool LAST>
__device__ __forceinline__ void dif_core(T2 (&v)[R], int m, int step, const T2 *__restrict__ tw) {
  dft_reg<T, T2, R, INV>(v);
  if (!LAST) {
    const int ms = m * step;
#pragma unroll
    for (int k = 1; k < R; k++) {
      T2 w = __ldg(tw + ms * k);
      if (INV) w.y = -w.y;
      v[k] = cmul(v[k], w);
    }
  }
}

// ------------------------------------------------------------- y (both)
// One pass of the C interleaved columns of a y tile: the first reads the
// columns from S, the last writes them back in natural order, the rest works
// in place in shared memory.
template <typename T, bool INV, bool FIRST, bool LAST>
__device__ __forceinline__ void ffty_pass(const FFTFactors &f, int p, typename Vec2<T>::type *buf,
                                          typename Vec2<T>::type *S, int sp, int ncol,
                                          const typename Vec2<T>::type *__restrict__ tw) {
  typedef typename Vec2<T>::type T2;
  constexpr int C = TyOf<T>::v;
  const int c = threadIdx.x % C;
  const bool ok = c < ncol;
  fft_radix(f.fac[p], [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int nb = f.n / R, M = f.M[p], step = f.step[p];
    for (int q = threadIdx.x / C; q < nb; q += kFFTThreads / C) {
      const DifPos at = dif_pos(f, p, q);
      T2 v[R];
#pragma unroll
      for (int r = 0; r < R; r++) {
        if (FIRST) {
          if (ok) v[r] = S[(long long)(at.base + r * M) * sp + c];
          else { v[r].x = 0; v[r].y = 0; }
        } else {
          v[r] = buf[(at.base + r * M) * C + c];
        }
      }
      dif_core<T, T2, R, INV, LAST>(v, at.m, step, tw);
      if (LAST) {
        const int k0 = dif_freq(f, q);
#pragma unroll
        for (int r = 0; r < R; r++)
          if (ok) S[(long long)(k0 + r * nb) * sp + c] = v[r];
      } else {
#pragma unroll
        for (int r = 0; r < R; r++) buf[(at.base + r * M) * C + c] = v[r];
      }
    }
  });
}

// Complex FFT along y of TyOf columns (kx) of one k plane of S, in place.
template <typename T, bool INV>
__global__ void __launch_bounds__(kFFTThreads, sizeof(T) == 4 ? 3 : 2)
    k_ffty_any(const Dom<T> *__restrict__ doms, Launch L, const PoisPlan *__restrict__ plans, int gate) {
  typedef typename Vec2<T>::type T2;
  constexpr int C = TyOf<T>::v;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T2 *buf = reinterpret_cast<T2 *>(smem_raw);
  for (int t = blockIdx.x; t < L.total; t += gridDim.x) {
    const int di = find_dom(L.starts, L.nd, t);
    const Dom<T> &d = doms[di];
    if (gate && !*d.refine_flag) continue;  // defect-correction sweep not needed
    const FFTFactors &f = plans[di].fy;
    const int lt = t - __ldg(L.starts + di);
    const int ncx = (d.nxh + C - 1) / C;
    const int k = lt / ncx, kx0 = (lt - k * ncx) * C;
    T2 *S = d.S + (long long)k * d.ny * d.spitch + kx0;
    const int sp = d.spitch, ncol = d.nxh - kx0, np = f.nfac;
    if (np == 1) {
      ffty_pass<T, INV, true, true>(f, 0, buf, S, sp, ncol, d.twy);
      continue;
    }
    ffty_pass<T, INV, true, false>(f, 0, buf, S, sp, ncol, d.twy);
    for (int p = 1; p < np - 1; p++) {
      __syncthreads();
      ffty_pass<T, INV, false, false>(f, p, buf, S, sp, ncol, d.twy);
    }
    __syncthreads();
    ffty_pass<T, INV, false, true>(f, np - 1, buf, S, sp, ncol, d.twy);
    __syncthreads();  // the next tile reuses buf
  }
}

// ------------------------------------------------------------ x (both)
// The passes of the ns interleaved sequences of an x tile in buf; the result
// lands in natural order in out.  Ends with a barrier.
template <typename T, bool INV>
__device__ __forceinline__ void fftx_passes(const FFTFactors &f, int ns, typename Vec2<T>::type *buf,
                                            typename Vec2<T>::type *out,
                                            const typename Vec2<T>::type *__restrict__ tw) {
  typedef typename Vec2<T>::type T2;
  const int pitch = fft_any_pitch(ns), s = threadIdx.x & (ns - 1), np = f.nfac;
  const int q0 = threadIdx.x / ns, dq = kFFTThreadsX / ns;
  for (int p = 0; p < np - 1; p++) {
    fft_radix(f.fac[p], [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      const int nb = f.n / R, Mp = f.M[p] * pitch, step = f.step[p];
      for (int q = q0; q < nb; q += dq) {
        const DifPos at = dif_pos(f, p, q);
        const int base = at.base * pitch + s;
        T2 v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = buf[base + r * Mp];
        dif_core<T, T2, R, INV, false>(v, at.m, step, tw);
#pragma unroll
        for (int r = 0; r < R; r++) buf[base + r * Mp] = v[r];
      }
    });
    __syncthreads();
  }
  fft_radix(f.fac[np - 1], [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int nb = f.n / R, nbp = nb * pitch;
    for (int q = q0; q < nb; q += dq) {
      const int base = q * R * pitch + s;
      T2 v[R];
#pragma unroll
      for (int r = 0; r < R; r++) v[r] = buf[base + r * pitch];
      dif_core<T, T2, R, INV, true>(v, 0, 0, tw);
      const int o0 = dif_freq(f, q) * pitch + s;
#pragma unroll
      for (int r = 0; r < R; r++) out[o0 + r * nbp] = v[r];
    }
  });
  __syncthreads();
}

// The rows of x tile lt: rows of them from r0 on, those before end in use.
// Across levels, or (Dom::wrows) from the start of each level.
struct XRows {
  int r0, end;
};
template <typename T>
__device__ __forceinline__ XRows x_rows(const Dom<T> &d, int lt, int rows) {
  if (!d.wrows) return XRows{lt * rows, d.ny * d.nz};
  const int np = d.wtiles(), k = lt / np;
  return XRows{k * d.ny + (lt - k * np) * rows, (k + 1) * d.ny};
}

// the right-hand sides of an x tile's rows into buf, VE cells a task: the
// divergence of PrePoisson (pressure.f90:688-717) from vectors of VE cells of
// a row; and the tile's sum of W2
template <typename T, int VE>
__device__ __forceinline__ void fftx_stage(const Dom<T> &d, typename Vec2<T>::type *buf, const RhsRow<T> *rinfo, XRows xr,
                                           int ns, double coef, int rhs_from_phi, TileSum &ls) {
  typedef typename Vec2<T>::type T2;
  const int pitch = fft_any_pitch(ns), nch = d.nx / VE, ny = d.ny, r0 = xr.r0, nrows = xr.end;
  const T rdt2 = (T)(1.0 / coef);
  const T rdx = (T)(1.0 / d.dx), rdy = (T)(1.0 / d.dy), rdz = (T)(1.0 / d.dz);
  auto row = [](const T *p, T (&v)[VE]) {
    if constexpr (VE == 1) v[0] = __ldg(p);
    else Row16<T>::ld(p, v);
  };
  for (int task = threadIdx.x; task < ns * nch; task += kFFTThreadsX) {
    const int sq = task / nch, c = task - sq * nch;
    T rhs[2][VE];
    if (rhs_from_phi) {
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int q = r0 + 2 * sq + h, k = q / ny + 1, j = q - (k - 1) * ny + 1;
        T ph[VE];
#pragma unroll
        for (int e = 0; e < VE; e++) ph[e] = (T)0;
        if (q < nrows) row(d.Phi + bidx(d, 1, j, k) + (long long)c * VE, ph);  // rows past the end are not read
#pragma unroll
        for (int e = 0; e < VE; e++) rhs[h][e] = ph[e] * rdt2;
      }
    } else {
      // the loads of both rows, then the arithmetic
      T uc[2][VE], vc[2][VE], vs[2][VE], wc[2][VE], wb[2][VE], uw0[2], rdzk[2];
#pragma unroll
      for (int h = 0; h < 2; h++) {
#pragma unroll
        for (int e = 0; e < VE; e++) uc[h][e] = vc[h][e] = vs[h][e] = wc[h][e] = wb[h][e] = (T)0;
        uw0[h] = (T)0;
        rdzk[h] = rdz;
        const int q = r0 + 2 * sq + h;
        if (q < nrows) {
          const RhsRow<T> &r = rinfo[2 * sq + h];
          const long long c0 = r.c0 + (long long)c * VE;
          row(d.U2 + c0, uc[h]);
          row(d.V2 + c0, vc[h]);
          row(d.V2 + c0 + r.o_vs, vs[h]);
          row(d.W2 + c0 + r.o_wc, wc[h]);
          row(d.W2 + c0 + r.o_wb, wb[h]);
          uw0[h] = c == 0 ? r.s_uw1 * ld((const T *)d.U2, c0 + r.o_uw1) : ld((const T *)d.U2, c0 - 1);
          rdzk[h] = r.rdz;
        }
      }
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const RhsRow<T> &r = rinfo[2 * sq + h];
#pragma unroll
        for (int e = 0; e < VE; e++) {
          const T uw = e == 0 ? uw0[h] : uc[h][e - 1];
          const T vse = r.s_vs * vs[h][e];
          const T wce = r.s_wc * wc[h][e], wbe = r.s_wb * wb[h][e];
          const T div = (uc[h][e] - uw) * rdx + (vc[h][e] - vse) * rdy + (wce - wbe) * rdzk[h];
          rhs[h][e] = div * rdt2;
        }
        if (d.wrows > 0) ls.add(wc[h], r);
      }
    }
#pragma unroll
    for (int e = 0; e < VE; e++) buf[(c * VE + e) * pitch + sq] = T2{rhs[0][e], rhs[1][e]};
  }
}

// Divergence right-hand side (or the one already stored in Phi) and the real
// FFT along x of 2 nsx rows, two real rows a complex sequence, split into
// their half spectra.
template <typename T>
__global__ void __launch_bounds__(kFFTThreadsX, sizeof(T) == 4 ? 6 : 4)
    k_fftx_fwd_any(const Dom<T> *__restrict__ doms, Launch L, const PoisPlan *__restrict__ plans, double coef_alpha2,
                   int use_dt, int rhs_from_phi, int gate) {
  typedef typename Vec2<T>::type T2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ RhsRow<T> rinfo[2 * kMaxSeqX];
  __shared__ double wred[kFFTThreadsX / 32];
  T2 *buf = reinterpret_cast<T2 *>(smem_raw);
  for (int t = blockIdx.x; t < L.total; t += gridDim.x) {
    const int di = find_dom(L.starts, L.nd, t);
    const Dom<T> &d = doms[di];
    if (gate && !*d.refine_flag) continue;
    const PoisPlan &pl = plans[di];
    const int N = d.nx, ny = d.ny, ns = pl.nsx, pitch = fft_any_pitch(ns);
    const XRows xr = x_rows(d, t - __ldg(L.starts + di), 2 * ns);
    const int r0 = xr.r0, nrows = xr.end;
    const double coef = use_dt ? coef_alpha2 * d.dt : coef_alpha2;
    T2 *out = buf + N * pitch;
    if (!rhs_from_phi && threadIdx.x < 2 * ns) {
      const int q = min(r0 + (int)threadIdx.x, nrows - 1);
      const int k = q / ny + 1;
      rinfo[threadIdx.x] = rhs_row(d, q - (k - 1) * ny + 1, k);
    }
    __syncthreads();
    const bool sums = d.wrows > 0 && !rhs_from_phi;
    TileSum ls{0};
    if (N % Row16<T>::n == 0) fftx_stage<T, Row16<T>::n>(d, buf, rinfo, xr, ns, coef, rhs_from_phi, ls);
    else fftx_stage<T, 1>(d, buf, rinfo, xr, ns, coef, rhs_from_phi, ls);
    if (sums) ls.warp_sum(wred);
    __syncthreads();
    if (sums) TileSum::put<kFFTThreadsX / 32>(wred, d.wpart + (t - __ldg(L.starts + di)));
    fftx_passes<T, false>(pl.fx, ns, buf, out, d.twx);
    // Z = FFT(a + i b): A_m = (Z_m + conj Z_{N-m}) / 2, B_m = (Z_m - conj Z_{N-m}) / 2i;
    // a warp takes 32 modes of a sequence
    const int nxh = d.nxh, lane = threadIdx.x & 31, ntask = ns * ((nxh + 31) / 32);
    for (int w = threadIdx.x / 32; w < ntask; w += kFFTThreadsX / 32) {
      const int s = w & (ns - 1), m = (w / ns) * 32 + lane, ra = r0 + 2 * s;
      if (m >= nxh || ra >= nrows) continue;
      const T2 zk = out[m * pitch + s], zc = out[(m == 0 ? 0 : N - m) * pitch + s];
      T2 A, B;
      A.x = (zk.x + zc.x) * (T)0.5;
      A.y = (zk.y - zc.y) * (T)0.5;
      B.x = (zk.y + zc.y) * (T)0.5;
      B.y = (zc.x - zk.x) * (T)0.5;
      d.S[(long long)ra * d.spitch + m] = A;
      if (ra + 1 < nrows) d.S[(long long)(ra + 1) * d.spitch + m] = B;
    }
    __syncthreads();  // the next tile reuses the buffers and rinfo
  }
}

// Inverse real FFT along x of 2 nsx rows -> interior of Phi: Z_m = A_m + i B_m
// with the Hermitian completion A_{N-m} = conj(A_m); A_0 and A_{N/2} are real
// for a real row.
template <typename T>
__global__ void __launch_bounds__(kFFTThreadsX, sizeof(T) == 4 ? 6 : 4)
    k_fftx_inv_any(const Dom<T> *__restrict__ doms, Launch L, const PoisPlan *__restrict__ plans, int gate) {
  typedef typename Vec2<T>::type T2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T2 *buf = reinterpret_cast<T2 *>(smem_raw);
  for (int t = blockIdx.x; t < L.total; t += gridDim.x) {
    const int di = find_dom(L.starts, L.nd, t);
    const Dom<T> &d = doms[di];
    if (gate && !*d.refine_flag) continue;
    const PoisPlan &pl = plans[di];
    const int N = d.nx, ny = d.ny, ns = pl.nsx, pitch = fft_any_pitch(ns);
    const XRows xr = x_rows(d, t - __ldg(L.starts + di), 2 * ns);
    const int r0 = xr.r0, nrows = xr.end, nxh = d.nxh, lane = threadIdx.x & 31;
    T2 *out = buf + N * pitch;
    // a warp takes 32 modes of a sequence, kLoads of them at a time
    constexpr int NW = kFFTThreadsX / 32, kLoads = 4;
    const int nm = ns * ((nxh + 31) / 32);
    for (int w0 = threadIdx.x / 32; w0 < nm; w0 += NW * kLoads) {
      T2 A[kLoads], B[kLoads];
#pragma unroll
      for (int u = 0; u < kLoads; u++) {
        const int w = w0 + u * NW, s = w & (ns - 1), m = (w / ns) * 32 + lane, ra = r0 + 2 * s;
        A[u].x = 0; A[u].y = 0; B[u].x = 0; B[u].y = 0;
        if (w < nm && m < nxh) {
          if (ra < nrows) A[u] = d.S[(long long)ra * d.spitch + m];
          if (ra + 1 < nrows) B[u] = d.S[(long long)(ra + 1) * d.spitch + m];
        }
      }
#pragma unroll
      for (int u = 0; u < kLoads; u++) {
        const int w = w0 + u * NW, s = w & (ns - 1), m = (w / ns) * 32 + lane;
        if (w >= nm || m >= nxh) continue;
        const bool real = m == 0 || 2 * m == N;
        if (real) { A[u].y = 0; B[u].y = 0; }
        buf[m * pitch + s] = T2{A[u].x - B[u].y, A[u].y + B[u].x};
        if (!real) buf[(N - m) * pitch + s] = T2{A[u].x + B[u].y, B[u].x - A[u].y};
      }
    }
    __syncthreads();
    fftx_passes<T, true>(pl.fx, ns, buf, out, d.twx);
    const int ni = ns * ((N + 31) / 32);
    for (int w = threadIdx.x / 32; w < ni; w += kFFTThreadsX / 32) {
      const int s = w & (ns - 1), i = (w / ns) * 32 + lane, ra = r0 + 2 * s;
      if (i >= N || ra >= nrows) continue;
      const T2 z = out[i * pitch + s];
      const int ka = ra / ny, kb = (ra + 1) / ny;
      d.Phi[bidx(d, i + 1, ra - ka * ny + 1, ka + 1)] = z.x;
      if (ra + 1 < nrows) d.Phi[bidx(d, i + 1, ra + 1 - kb * ny + 1, kb + 1)] = z.y;
    }
    __syncthreads();  // the next tile reuses the buffers
  }
}

}  // namespace elmm
