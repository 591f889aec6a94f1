// Row and column passes of a layer step, complex128 bulk, any side n = n1 n2
// with n1, n2 up to 32 (`line_shape`).
//
// A line is transformed in block fixed point (dtmm_fx.cuh) in two steps of
// register DFTs by n1 (first step) and n2 (second step) threads of a block;
// one call site serves every transform of a kernel, so the code of a launch
// is the two lengths it uses.  FP64 arithmetic remains where the voxels'
// operators act.
//
// What bounds them (256 x 256, nine windows, ten images, one layer): in FP64
// arithmetic with shared-memory radix passes the row pass took 2.68 ms and
// the column pass 0.66 ms, both at the FP64 pipe's rate; here 0.90 and 0.13
// ms.  The row pass keeps the FP64 pipe 71 % busy, with 12 warps a SM (168
// registers, 72 KB a block); applying the operators in fixed point as well
// halved its FP64 work and took the same time (1.5 x the instructions, the
// same warps), so they stay in FP64.
//
// Slots: entry (k, s) of the exchange lies at k + P s with P = n2 | 1 (an odd
// pitch, so that a column of it and a row of it are both free of bank
// conflicts), and point x = k + n2 m of the line at k + P m: every thread reads
// and writes the same slots within a step, one barrier separates the steps.
//   inverse  step 1  thread t < n1: x[t + n1 m], DFT n2, twiddle, slots k + P t
//            step 2  thread k < n2: slots k + P s, DFT n1, slots k + P m
//   forward  step 1  thread t < n2: slots t + P m, DFT n1, twiddle, slots t + P k
//            step 2  thread k < n1: slots s + P k, DFT n2, X[k + n1 m]
// A first-step thread of the forward transform holds what it wrote in the
// second step of the inverse one.
#pragma once

#include <type_traits>

#include "dtmm_fx.cuh"
#include "dtmm_layer.cuh"

namespace dtmm {

struct LineGeom {
  int n1, n2, pitch;  // pitch P = n2 | 1; a line takes n1 P slots
};

constexpr int kLineMax = 64;  // lines of a block at most

// Launch bounds: the largest block and the blocks of a SM, by the points a thread
// holds (maxl) and the side (cn1 maxl; cn1 0: run-time lengths).  The passes wait
// on shared memory and on 64-bit multiplies, so warps in flight count for more than
// spills to L1: 12 warps of 168 registers a SM as 3 x 128 threads, or 10 as 2 x 160
// where that holds eight lines of 18 or 20 points a thread.  Against one block of
// 256 threads at 255 registers (5 to 8 warps), ten layers, row pass: side 300, one
// window 2.16 -> 1.35 ms, nine windows 14.0 -> 9.5; side 125 3.64 -> 2.81 and 24.5 ->
// 17.6; side 432 4.14 -> 3.61 and 28.6 -> 23.7 (its column pass 2.22 -> 2.63).  Four
// blocks at 128 registers for up to 12 points lost up to 9 % (side 120, 144).
// Above 520 points shared memory leaves one or two such blocks, and the run-time
// kernels spill four times as much at 168 registers (1024 points: 199 -> 209 ms).
constexpr int line_threads(int maxl, int cn1) {
  return maxl <= 16 ? 128 : (cn1 == 0 || cn1 * maxl > 520 ? 256 : (maxl <= 20 ? 160 : 128));
}
constexpr int line_blocks(int maxl, int cn1) {
  return line_threads(maxl, cn1) == 128 ? 3 : (line_threads(maxl, cn1) == 160 ? 2 : 1);
}

// slot of (k, m): a compile-time power-of-two n2 swizzles (no padding, three
// 256-point blocks of eight complex128 lines a SM instead of two), others pad
template <int CN2>
__host__ __device__ __forceinline__ constexpr int line_pitch(int n2) {
  return CN2 != 0 && is_pow2(CN2) ? n2 : (n2 | 1);
}
template <int CN2>
__device__ __forceinline__ int line_slot(int k, int m, int pitch) {
  if constexpr (CN2 != 0 && is_pow2(CN2))
    return (k ^ (m & (CN2 - 1))) + CN2 * m;
  else
    return k + pitch * m;
}

// the DFT of a step: n1 x n2 known at compile time (CN1 > 0) or run-time lengths
template <int MAXL, int CN1, int CN2, typename R = fx>
__device__ __forceinline__ void step_dft(cpx<R> (&v)[MAXL], bool roleA, int len) {
  if constexpr (CN1 == 0) {
    line_dft<R, MAXL>(v, len);
  } else if constexpr (CN1 == CN2) {
    RegDFTg<R, CN1, false>::run(v);
  } else {
    if (roleA)
      RegDFTg<R, CN2, false>::run(v);
    else
      RegDFTg<R, CN1, false>::run(v);
  }
}

__device__ __forceinline__ cpx<fx> line_tw(cpx<double> w) { return mk<fx>(fx(w.re), fx(w.im)); }

// The scale of a line from its threads' words in shared memory (part), one
// barrier.  The caller's next barrier precedes the next call.
constexpr int kPartPitch = 33;
template <int MAXL>
__device__ __forceinline__ void line_scale(const cpx<double> (&d)[MAXL], int len, int nthr, int t, bool act, int line,
                                           unsigned* part, int& emax, int& g1, int& g2, int lo, int hi) {
  if (act) part[line * kPartPitch + t] = fx_part<MAXL>(d, len, lo, hi);
  __syncthreads();
  if (act) fx_scale(part + line * kPartPitch, nthr, emax, g1, g2);
}

// the entries in fixed point; entries lo <= i < hi hold zeros for every thread
template <int MAXL>
__device__ __forceinline__ void line_in(cpx<fx> (&v)[MAXL], const cpx<double> (&d)[MAXL], int len, int emax, int guard,
                                        int lo, int hi) {
#pragma unroll
  for (int i = 0; i < MAXL; ++i) {
    if (i >= len) break;
    v[i] = mk<fx>(fx(0, 0), fx(0, 0));
    if (i < lo || i >= hi) v[i] = mk<fx>(to_fx(d[i].re, emax, guard), to_fx(d[i].im, emax, guard));
  }
}

// a result beyond the exponents that from_fx scales; a line with an infinity
// or a NaN is NaN
static __device__ __noinline__ double line_out_slow(long long v, int emax, int k) {
  return emax == 0x7ff ? bitsd(0x7ff8000000000000LL) : ldexp((double)v, k);
}

__device__ __forceinline__ cpx<double> line_out(cpx<fx> a, int emax, int guard) {
  const int k = fx_kexp(emax, guard);
  if (fx_plain(emax)) return mk<double>(from_fx(a.re, k), from_fx(a.im, k));
  return mk<double>(line_out_slow(a.re.v, emax, k), line_out_slow(a.im.v, emax, k));
}

// exp(i arg k): k in turns for real FP64 arguments
__device__ __forceinline__ cpx<double> line_phase(double arg, double k, int rest) { return turn_of(arg * k, rest); }
__device__ __forceinline__ cpx<double> line_phase(cpx<double> arg, double k, int) { return phase_of<double>(arg, k); }

template <typename T>
__device__ __forceinline__ cpx<T> swapc(cpx<T> a) {
  return mk<T>(a.im, a.re);
}

// ---------------------------------------------------------------------------
// Row pass (see RowParams): one row of G wavelengths x PB polarisations of one
// ray.  Threads: lines x max(n1, n2).
// ---------------------------------------------------------------------------
template <int C, bool REAL, int MAXL, int CN1, int CN2>
__global__ void __launch_bounds__(line_threads(MAXL, CN1), line_blocks(MAXL, CN1))
    k_row_line(RowParams p, Grid g, LineGeom s, int limW, const cpx<double>* __restrict__ U,
               cpx<double>* __restrict__ X) {
  using T = typename std::conditional<REAL, double, cpx<double>>::type;
  __shared__ double s_kph[kLineMax];
  __shared__ int s_krest[kLineMax];
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_scale[kLineMax];  // emax << 8 | second-step guard bits of each line
  const int n1 = CN1 ? CN1 : s.n1, n2 = CN2 ? CN2 : s.n2;
  const int H = g.H, W = CN1 ? CN1 * CN2 : g.W, P = line_pitch<CN2>(n2), LS = n1 * P;
  const auto slot = [&](int k, int m) { return line_slot<CN2>(k, m, P); };
  const int ngrp = (g.nlam + p.G - 1) / p.G;
  const int npg = (g.npol + p.PB - 1) / p.PB;
  const int y = p.groups_inner ? blockIdx.y : blockIdx.x;
  const int gi = p.groups_inner ? blockIdx.x : blockIdx.y;
  const int pg = gi % npg, rg = gi / npg;
  const int ray = rg / ngrp, grp = rg - ray * ngrp;
  const int lam0 = grp * p.G, pol0 = pg * p.PB;
  const int G = min(p.G, g.nlam - lam0);
  const int NP = min(p.PB, g.npol - pol0);
  const int nlines = G * NP * C, lmaxn = p.G * p.PB * C;
  cpx<double>* acc = (cpx<double>*)smem_raw;                    // [lines][LS]
  cpx<double>* buf = acc + (size_t)lmaxn * LS;             // [lines][LS] exchange, then the transformed row
  cpx<fx>* tw = (cpx<fx>*)(buf + (size_t)lmaxn * LS);   // [W] W^(t k) at k n1 + t
  unsigned* s_part = (unsigned*)(tw + W);             // [lines][kPartPitch]
  const int HW = H * W, nwin = p.nx * p.ny;
  for (int e = threadIdx.x; e < W; e += blockDim.x) tw[e] = line_tw(((const cpx<double>*)p.tw)[(e % n1) * (e / n1)]);
  for (int e = threadIdx.x; e < nlines * LS; e += blockDim.x) acc[e] = mk<double>(0, 0);
  // k0 of every wavelength, in turns per unit where the phases are formed in turns
  for (int gl = threadIdx.x; gl < G; gl += blockDim.x) {
    const double k = p.ks[lam0 + gl] * p.dir;
    const TurnScale t = REAL ? turn_scale(k) : TurnScale{k, 0};
    s_kph[gl] = t.k;
    s_krest[gl] = t.rest;
  }
  grid_release();
  grid_wait();  // the column pass's rows
  __syncthreads();
  const double sc = (double)p.in_scale;
  const int lineA = threadIdx.x / n1, tA = threadIdx.x - lineA * n1;
  const int lineB = threadIdx.x / n2, tB = threadIdx.x - lineB * n2;
  const unsigned rcp2 = (65536u + n2 - 1) / n2;  // x / n2 = x rcp2 >> 16 for x < 1024
  int w = -1;
  for (;;) {
    // the next window with something in it; past the last one the forward transform
    bool fwd = false;
    for (;;) {
      if (++w >= nwin) {
        fwd = true;
        break;
      }
      // window w = i ny + j; rows j outermost, as the sums are formed
      const int j = w / p.nx, i = w - j * p.nx, ww = i * p.ny + j;
      if (p.win_only >= 0 && ww != p.win_only) continue;
      if (p.wzero != nullptr && p.wzero[ray * nwin + ww]) continue;
      break;
    }
    const int j = w / p.nx, i = w - j * p.nx, ww = i * p.ny + j;
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      const bool roleA = (half == 0) != fwd;
      const int line = roleA ? lineA : lineB, t = roleA ? tA : tB;
      const int len = CN1 != 0 && CN1 == CN2 ? CN1 : (roleA ? n2 : n1);
      const bool act = line < nlines;
      const int c = line % C, im = line / C;
      const int gl = im / NP, pol = pol0 + im - gl * NP;
      const int lam = lam0 + gl;
      const size_t img = ((size_t)ray * g.npol + pol) * g.nlam + lam;
      cpx<double>* bl = buf + (size_t)line * LS;
      cpx<fx>* fl = (cpx<fx>*)bl;
      cpx<fx> v[MAXL];
      int emax = 0, g1 = 0, guard = 0;
      if (half == 0) {
        cpx<double> d[MAXL];
        // entries m in [lo, hi) lie beyond the band for every thread
        const int lo = fwd ? len : limW / n1 + 1, hi = fwd ? len : (W - limW) / n1;
        if (act) {
          if (fwd) {
            const cpx<double>* al = acc + (size_t)line * LS;
#pragma unroll
            for (int m = 0; m < MAXL; ++m) {
              if (m >= len) break;
              d[m] = al[slot(t, m)];
            }
          } else {
            const cpx<double>* src = U + (size_t)(p.win_only >= 0 ? 0 : j) * g.NI * C * HW + ((img * C + c) * H + y) * W;
            const double* cxl = (p.cx && p.use_cx) ? (const double*)p.cx + (((size_t)ray * p.nx + i) * g.nlam + lam) * W : nullptr;
            const int lim = (int)p.blim[lam];
#pragma unroll
            for (int m = 0; m < MAXL; ++m) {
              if (m >= len) break;
              const int xk = t + n1 * m;
              const int ax = xk < (W + 1) / 2 ? xk : W - xk;
              cpx<double> a = mk<double>((double)0, (double)0);
              if ((m < lo || m >= hi) && ax <= lim) {
                a = src[xk];
                if (cxl) a = a * cxl[xk];
              }
              d[m] = swapc(a);
            }
          }
        }
        line_scale<MAXL>(d, len, roleA ? n1 : n2, t, act, line, s_part, emax, g1, guard, lo, hi);
        if (act && t == 0) s_scale[line] = emax << 8 | guard;
        if (act) line_in<MAXL>(v, d, len, emax, g1, lo, hi);
      } else if (act) {
        emax = s_scale[line] >> 8;
        guard = s_scale[line] & 0xff;
#pragma unroll
        for (int m = 0; m < MAXL; ++m) {
          if (m >= len) break;
          v[m] = fl[roleA ? slot(m, t) : slot(t, m)];
        }
      }
      if (act) {
        step_dft<MAXL, CN1, CN2>(v, roleA, len);
        if (half == 0) {
          // twiddle W^(t k), then the slots of (k, s = t)
          const int wo = fwd ? t * n1 : t, ws = fwd ? 1 : n1;
          fl[slot(fwd ? t : 0, fwd ? 0 : t)] = fx_shift(v[0], guard - g1);
#pragma unroll
          for (int k = 1; k < MAXL; ++k) {
            if (k >= len) break;
            fl[slot(fwd ? t : k, fwd ? k : t)] = fx_shift(v[k] * tw[wo + ws * k], guard - g1);
          }
        } else if (!fwd) {
#pragma unroll
          for (int m = 0; m < MAXL; ++m) {
            if (m >= len) break;
            bl[slot(t, m)] = swapc(line_out(v[m], emax, guard));
          }
        } else {
          cpx<double>* dst = X + ((img * C + c) * H + y) * W + t;
#pragma unroll
          for (int m = 0; m < MAXL; ++m) {
            if (m >= len) break;
            // band_out: the next column pass reads the columns inside the band only
            if (p.band_out && m > limW / n1 && m < (W - limW) / n1) continue;
            const cpx<double> r = line_out(v[m], emax, guard);
            dst[n1 * m] = p.accumulate ? dst[n1 * m] + r : r;
          }
        }
      }
      __syncthreads();
    }
    if (fwd) break;
    // the voxels' operators of the window
    const int rs = p.rec_stride;
    const T* opw = (const T*)p.op + (((size_t)ray * nwin + ww) * HW + (size_t)y * W) * rs;
    constexpr int NR = C == 4 ? OP_REC : REC_BLOCK;
    for (int x = threadIdx.x; x < W; x += blockDim.x) {
      T rec[NR];
      load_planes<NR, T>(opw, W, x, rec);
      const int xm = (int)((x * rcp2) >> 16), q = slot(x - xm * n2, xm);
      const T* ef = rec;
      const T* eb = rec + (C == 4 ? REC_BLOCK : 0);
      for (int gl = 0; gl < G; ++gl) {
        const double kph = s_kph[gl];
        const int kr = s_krest[gl];
        cpx<double> qf, dpf, qb, dpb;
        {
          const cpx<double> f0 = line_phase(ef[4], kph, kr), f1 = line_phase(ef[5], kph, kr);
          qf = f1 * sc;
          dpf = f0 - f1;
        }
        if (C == 4) {
          const cpx<double> b0 = line_phase(eb[4], kph, kr), b1 = line_phase(eb[5], kph, kr);
          qb = b1 * sc;
          dpb = b0 - b1;
        }
        for (int pol = 0; pol < NP; ++pol) {
          const int l0 = (gl * NP + pol) * C;
          const cpx<double>* h = buf + (size_t)l0 * LS + q;
          cpx<double>* a = acc + (size_t)l0 * LS + q;
          if (C == 4) {
            cpx<double> a0 = a[0], a1 = a[LS], a2 = a[2 * LS], a3 = a[3 * LS];
            apply_block<double, T>(ef, qf, dpf, h[0], h[2 * LS], a0, a2);
            apply_block<double, T>(eb, qb, dpb, h[LS], h[3 * LS], a1, a3);
            a[0] = a0; a[LS] = a1; a[2 * LS] = a2; a[3 * LS] = a3;
          } else {
            cpx<double> a0 = a[0], a1 = a[LS];
            apply_block<double, T>(ef, qf, dpf, h[0], h[LS], a0, a1);
            a[0] = a0; a[LS] = a1;
          }
        }
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Plain row transforms of `nlines` lines, src -> dst (the same array for in
// place: a block reads its lines before it writes them), times `scale`; lpb
// lines a block.
// ---------------------------------------------------------------------------
template <int MAXL>
__global__ void __launch_bounds__(line_threads(MAXL, 0), line_blocks(MAXL, 0))
    k_rows_line(const cpx<double>* src, cpx<double>* dst, int nlines, int W, LineGeom s, int inv,
                const cpx<double>* __restrict__ twg, double scale, int lpb) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_scale[kLineMax];  // emax << 8 | second-step guard bits of each line
  const int P = s.pitch, LS = s.n1 * P;
  cpx<fx>* buf = (cpx<fx>*)smem_raw;
  cpx<fx>* tw = buf + (size_t)lpb * LS;
  unsigned* s_part = (unsigned*)(tw + W);  // [lines][kPartPitch]
  for (int e = threadIdx.x; e < W; e += blockDim.x) tw[e] = line_tw(twg[(e % s.n1) * (e / s.n1)]);
  __syncthreads();
  const int nl = min(lpb, nlines - (int)blockIdx.x * lpb);
#pragma unroll 1
  for (int half = 0; half < 2; ++half) {
    const bool roleA = half == 0;
    const int n = roleA ? s.n1 : s.n2, len = roleA ? s.n2 : s.n1;
    const int line = threadIdx.x / n, t = threadIdx.x - line * n;
    const bool act = line < nl;
    const size_t off = ((size_t)blockIdx.x * lpb + line) * W;
    cpx<fx>* fl = buf + (size_t)line * LS;
    cpx<fx> v[MAXL];
    int emax = 0, g1 = 0, guard = 0;
    if (half == 0) {
      cpx<double> d[MAXL];
      const int lo = len, hi = len;
      if (act) {
#pragma unroll
        for (int m = 0; m < MAXL; ++m) {
          if (m >= len) break;
          const cpx<double> a = src[off + t + s.n1 * m];
          d[m] = inv ? swapc(a) : a;
        }
      }
      line_scale<MAXL>(d, len, n, t, act, line, s_part, emax, g1, guard, lo, hi);
      if (act && t == 0) s_scale[line] = emax << 8 | guard;
      if (act) line_in<MAXL>(v, d, len, emax, g1, lo, hi);
    } else if (act) {
      emax = s_scale[line] >> 8;
      guard = s_scale[line] & 0xff;
#pragma unroll
      for (int m = 0; m < MAXL; ++m) {
        if (m >= len) break;
        v[m] = fl[t + P * m];
      }
    }
    if (act) {
      line_dft<fx, MAXL>(v, len);
      if (half == 0) {
        fl[P * t] = fx_shift(v[0], guard - g1);
#pragma unroll
        for (int k = 1; k < MAXL; ++k) {
          if (k >= len) break;
          fl[P * t + k] = fx_shift(v[k] * tw[t + s.n1 * k], guard - g1);
        }
      } else {
#pragma unroll
        for (int m = 0; m < MAXL; ++m) {
          if (m >= len) break;
          const cpx<double> r = line_out(v[m], emax, guard);
          dst[off + t + s.n2 * m] = (inv ? swapc(r) : r) * scale;
        }
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Column pass (see ColParams): tc columns x max(cin, cout) components of one
// image, threads: lines x max(n1, n2), consecutive threads on consecutive
// columns.  Tile element (slot, line) at slot * lines + line.  limH: entries
// with |frequency index| along y beyond it are zero after a KOP_DIAG table.
// ---------------------------------------------------------------------------
template <int MAXL, int CN1, int CN2>
__global__ void __launch_bounds__(line_threads(MAXL, CN1), line_blocks(MAXL, CN1))
    k_col_line(ColParams p, Grid g, LineGeom s, int limH, const cpx<double>* __restrict__ X,
               cpx<double>* __restrict__ U) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_scale[kLineMax];  // emax << 8 | second-step guard bits of each line
  const int n1 = CN1 ? CN1 : s.n1, n2 = CN2 ? CN2 : s.n2;
  const int H = CN1 ? CN1 * CN2 : g.H, W = g.W, TX = p.tc;
  const int CM = max(p.cin, p.cout), NL = CM * TX;
  const int img = blockIdx.y;
  const int tile = (p.tile_lo > 0 && (int)blockIdx.x >= p.tile_lo) ? p.tile_hi0 + ((int)blockIdx.x - p.tile_lo)
                                                                    : (int)blockIdx.x;
  const int x0 = tile * TX;
  const int lam = img_lam(g, img), ray = img_ray(g, img);
  const bool diag = p.kop == KOP_DIAG;
  bool band_x = true;  // the thread's column is read
  grid_release();
  grid_wait();  // the row pass's columns, and the readers of U
  if ((p.band_skip == 2 && diag) || p.xband) {  // tiles beyond the band: nothing is read from them, or zeros
    const int lim = (int)p.blim[lam];
    bool any = false;
    for (int xc = 0; xc < TX && x0 + xc < W; ++xc) {
      const int xk = x0 + xc;
      any = any || (xk < (W + 1) / 2 ? xk : W - xk) <= lim;
    }
    const int line = threadIdx.x % NL, c = line / TX, kx = x0 + line - c * TX;
    if (!any) {
      if (!diag && c < p.cout && kx < W)
        for (int jj = 0; jj < p.ny; ++jj) {
          cpx<double>* udst = U + ((size_t)jj * g.NI * p.cout + (size_t)img * p.cout + c) * H * W + kx;
          for (int y = threadIdx.x / NL; y < H; y += blockDim.x / NL) udst[(size_t)y * W] = mk<double>(0.0, 0.0);
        }
      return;
    }
    if (p.xband) band_x = (kx < (W + 1) / 2 ? kx : W - kx) <= lim;
  }
  cpx<fx>* tile_x = (cpx<fx>*)smem_raw;                                    // [H][NL] exchange
  cpx<double>* tile_s = (cpx<double>*)(p.ny > 1 ? tile_x + (size_t)H * NL : tile_x);  // [H][NL] spectra along y
  cpx<fx>* tw = tile_x + (size_t)H * NL * (p.ny > 1 ? 2 : 1);
  unsigned* s_part = (unsigned*)(tw + H);  // [lines][kPartPitch]
  for (int e = threadIdx.x; e < H; e += blockDim.x)
    tw[e] = line_tw(((const cpx<double>*)p.tw)[(e % n1) * (e / n1)]);
  __syncthreads();
  const int line = threadIdx.x % NL, t = threadIdx.x / NL;
  const int c = line / TX, xc = line - c * TX, kx = x0 + xc;
  const bool in_x = kx < W;
  const double sc = (double)p.out_scale;
  // halves: 0, 1 the forward transform (skipped without do_fwd), then two per window row
#pragma unroll 1
  for (int q = p.do_fwd ? 0 : 1; q < 2 + 2 * p.ny; ++q) {
    const bool fwd = q < 2;
    const int half = q & 1;
    const bool roleA = (half == 0) != fwd;  // n1 threads with n2 points
    const int n = roleA ? n1 : n2, len = CN1 != 0 && CN1 == CN2 ? CN1 : (roleA ? n2 : n1);
    const int nc = fwd ? p.cin : p.cout;
    const bool act = t < n && c < nc;
    const int jj = (q - 2) >> 1, j = p.j_only >= 0 ? p.j_only : jj;
    cpx<fx> v[MAXL];
    int emax = 0, g1 = 0, guard = 0;
    const bool skip_dft = (q == 1 && !p.do_fwd) || (!fwd && !p.inverse_out);
    if (half == 0) {
      cpx<double> d[MAXL];
      // entries m in [lo, hi) lie beyond the band for every thread
      const bool cut = !fwd && diag;
      const int lo = cut ? limH / n1 + 1 : len, hi = cut ? (H - limH) / n1 : len;
      if (act) {
        if (fwd) {
          const cpx<double>* src = X + ((size_t)img * p.cin + c) * H * W + kx;
#pragma unroll
          for (int m = 0; m < MAXL; ++m) {
            if (m >= len) break;
            d[m] = in_x && band_x ? src[(size_t)(t + n2 * m) * W] : mk<double>(0.0, 0.0);
          }
        } else {
          const double* cyj = p.cy ? (const double*)p.cy + (((size_t)ray * p.cy_rows + j) * g.nlam + lam) * H : nullptr;
#pragma unroll
          for (int m = 0; m < MAXL; ++m) {
            if (m >= len) break;
            const int k = t + n1 * m;
            const int ak = k < (H + 1) / 2 ? k : H - k;
            cpx<double> a = mk<double>((double)0, (double)0);
            if (!diag || ak <= limH) {
              a = tile_s[(m + n2 * t) * NL + line];
              if (cyj) a = a * cyj[k];
            }
            d[m] = swapc(a);
          }
          if (!p.inverse_out) {  // stays along ky
            if (in_x) {
              cpx<double>* dst = U + ((size_t)jj * g.NI * p.cout + (size_t)img * p.cout + c) * H * W + kx;
#pragma unroll
              for (int m = 0; m < MAXL; ++m) {
                if (m >= len) break;
                dst[(size_t)(t + n1 * m) * W] = swapc(d[m]);
              }
            }
          }
        }
      }
      if (skip_dft) continue;
      line_scale<MAXL>(d, len, n, t, act, line, s_part, emax, g1, guard, lo, hi);
      if (act && t == 0) s_scale[line] = emax << 8 | guard;
      if (act) line_in<MAXL>(v, d, len, emax, g1, lo, hi);
    } else {
      if (!fwd && skip_dft) continue;
      if (act && !skip_dft) {
        emax = s_scale[line] >> 8;
        guard = s_scale[line] & 0xff;
        const int o = roleA ? n2 * t : t, st = roleA ? 1 : n2;
#pragma unroll
        for (int m = 0; m < MAXL; ++m) {
          if (m >= len) break;
          v[m] = tile_x[(size_t)(o + st * m) * NL + line];
        }
      }
    }
    if (act && !skip_dft) step_dft<MAXL, CN1, CN2>(v, roleA, len);
    if (half == 0) {
      if (act) {
        const int wo = fwd ? t * n1 : t, ws = fwd ? 1 : n1;
        const int o = fwd ? t : n2 * t, st = fwd ? n2 : 1;
        tile_x[(size_t)o * NL + line] = fx_shift(v[0], guard - g1);
#pragma unroll
        for (int k = 1; k < MAXL; ++k) {
          if (k >= len) break;
          tile_x[(size_t)(o + st * k) * NL + line] = fx_shift(v[k] * tw[wo + ws * k], guard - g1);
        }
      }
      __syncthreads();
    } else if (fwd) {
      // spectra k = t + n1 m through the k-space operator into the thread's own slots m + n2 t
      if (act) {
        const cpx<double>* ek = (diag && in_x) ? (const cpx<double>*)p.ktab + (((size_t)lam * W + kx) * H) * 2 +
                                                ((((c & 1) == 0) || p.cin == 2) ? 0 : 1)
                                          : nullptr;
        const cpx<double>* src = X + ((size_t)img * p.cin + c) * H * W + kx;
#pragma unroll
        for (int m = 0; m < MAXL; ++m) {
          if (m >= len) break;
          const int k = t + n1 * m;
          const int ak = k < (H + 1) / 2 ? k : H - k;
          cpx<double> a = mk<double>((double)0, (double)0);
          if (!diag || ak <= limH) {
            a = skip_dft ? (in_x && band_x ? src[(size_t)k * W] : a) : line_out(v[m], emax, guard);
            if (ek) a = a * ek[(size_t)k * 2];
            if (p.kop != KOP_MAT) a = a * sc;
          }
          tile_s[(size_t)(m + n2 * t) * NL + line] = a;
        }
      }
      if (p.kop == KOP_MAT) {
        __syncthreads();
        // one point k, column xc and every component a turn
        for (int e = threadIdx.x; e < H * TX; e += blockDim.x) {
          const int sl = e / TX, xe = e - sl * TX;
          const int kt = sl / n2, k = kt + n1 * (sl - kt * n2);  // slot m + n2 t holds k = t + n1 m
          cpx<double>* z = tile_s + (size_t)sl * NL + xe;
          cpx<double> vin[4], vout[4];
          for (int ci = 0; ci < p.cin; ++ci) vin[ci] = z[ci * TX];
          const bool out = x0 + xe < W;
          const cpx<double>* mt = (const cpx<double>*)p.ktab + ray * p.ktab_ray_stride +
                             (((size_t)lam * H + k) * W + x0 + xe) * p.cout * p.cin;
          for (int co = 0; co < p.cout; ++co) {
            cpx<double> a = mk<double>((double)0, (double)0);
            if (out)
              for (int ci = 0; ci < p.cin; ++ci) a = cfma(mt[co * p.cin + ci], vin[ci], a);
            vout[co] = a * sc;
          }
          for (int co = 0; co < p.cout; ++co) z[co * TX] = vout[co];
        }
        __syncthreads();
      }
    } else {
      if (act && in_x) {
        cpx<double>* dst = U + ((size_t)jj * g.NI * p.cout + (size_t)img * p.cout + c) * H * W + kx;
#pragma unroll
        for (int m = 0; m < MAXL; ++m) {
          if (m >= len) break;
          dst[(size_t)(t + n2 * m) * W] = swapc(line_out(v[m], emax, guard));
        }
      }
      __syncthreads();  // the exchange is read before the next window row writes it
    }
  }
}

// ---------------------------------------------------------------------------
// Launch glue.  The sides of DTMM_LINE_SIDES have row (real operator records) and
// column kernels with n1 x n2 (the most even split) known at compile time, instantiated
// in dtmm_line_<a..o>.cu: no switch and few spills, so that more blocks fit a SM.  Which
// sides these are is a choice, not a rule: multiples of 16 and of 5 and a few others from 45 to
// 1024, those of the tests, the benchmark and perf/cases.py among them, 53 of the 135 in that
// range that split, for the size of the library (2 MB a side).
// Ten layers, run-time lengths -> these (row / column pass, ms): side 48, one window
// .28 / .33 -> .21 / .24; 112, nine windows 6.9 / 1.24 -> 5.3 / .99; 200 14.4 / 3.2 ->
// 6.6 / 1.6; 320 19.0 / 4.2 -> 11.3 / 2.1; 512 38.2 / 8.5 -> 32.3 / 6.5; 1024 199 / 29.7 ->
// 170 / 24.0.  Every other side takes the run-time kernels of dtmm_line_any*.cu, or where
// those lose (Engine::line_loses) the shared-memory passes.
// ---------------------------------------------------------------------------
struct LineLaunch {
  dim3 grid;
  int threads;
  size_t smem;
  cudaStream_t st;
  LineGeom geom;
  int maxl, lim;  // lim: band limit of the transformed axis
  bool pdl = false;  // programmatic dependency on the previous kernel (row and column passes)
};

#define DTMM_LINE_SIDES(X) \
  X(5, 9) X(5, 10) X(5, 15) X(5, 25) X(6, 8) X(6, 10) X(7, 9) X(7, 25) X(8, 8) X(8, 9) X(8, 10) X(8, 12) \
  X(8, 14) X(8, 16) X(9, 10) X(9, 15) X(10, 10) X(10, 11) X(10, 12) X(10, 14) X(10, 15) X(10, 16) X(10, 20) \
  X(10, 25) X(11, 20) X(12, 12) X(12, 14) X(12, 15) X(12, 16) X(14, 14) X(14, 15) X(14, 16) X(14, 20) X(14, 25) \
  X(15, 15) X(15, 16) X(15, 18) X(15, 20) X(15, 22) X(16, 16) X(16, 18) X(16, 20) X(16, 21) X(16, 22) X(16, 24) \
  X(16, 28) X(16, 32) X(18, 20) X(18, 24) X(20, 20) X(20, 24) X(20, 32) X(32, 32)

inline bool line_side(int n1, int n2) {
#define DTMM_LINE_IS(A, B) \
  if (n1 == A && n2 == B) return true;
  DTMM_LINE_SIDES(DTMM_LINE_IS)
#undef DTMM_LINE_IS
  return false;
}
// threads a row (complex records: real = false) or column kernel's block may have
inline int line_most(const LineShape& ls, bool real) {
  return real && line_side(ls.n1, ls.n2) ? line_threads(ls.n2, ls.n1) : line_threads(ls.maxl, 0);
}
// slots of a row kernel's line per n1: what line_pitch gives there
inline int line_row_pitch(const LineShape& ls, bool real) {
  return real && line_side(ls.n1, ls.n2) && is_pow2(ls.n2) ? ls.n2 : (ls.n2 | 1);
}

template <typename K, typename... A>
cudaError_t line_launch(K kern, const LineLaunch& L, A... a) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.smem);
  if (e != cudaSuccess) return e;
  return launch_with(L.pdl, kern, L.grid, L.threads, L.smem, L.st, a...);
}

template <int C, bool REAL, int MAXL, int CN1, int CN2>
cudaError_t row_line_launch(const LineLaunch& L, const RowParams& p, const Grid& g, const void* U, void* X) {
  return line_launch(k_row_line<C, REAL, MAXL, CN1, CN2>, L, p, g, L.geom, L.lim, (const cpx<double>*)U, (cpx<double>*)X);
}
template <int MAXL, int CN1, int CN2>
cudaError_t col_line_launch(const LineLaunch& L, const ColParams& p, const Grid& g, const void* in, void* out) {
  return line_launch(k_col_line<MAXL, CN1, CN2>, L, p, g, L.geom, L.lim, (const cpx<double>*)in, (cpx<double>*)out);
}

#define DTMM_LINE_DECLARE(A, B)                                                                                     \
  cudaError_t row_line_##A##_##B(int C, const LineLaunch& L, const RowParams& p, const Grid& g, const void* U, void* X); \
  cudaError_t col_line_##A##_##B(const LineLaunch& L, const ColParams& p, const Grid& g, const void* in, void* out);
#define DTMM_LINE_DEFINE(A, B)                                                                                      \
  cudaError_t row_line_##A##_##B(int C, const LineLaunch& L, const RowParams& p, const Grid& g, const void* U, void* X) { \
    return C == 4 ? row_line_launch<4, true, B, A, B>(L, p, g, U, X) : row_line_launch<2, true, B, A, B>(L, p, g, U, X); \
  }                                                                                                                 \
  cudaError_t col_line_##A##_##B(const LineLaunch& L, const ColParams& p, const Grid& g, const void* in, void* out) { \
    return col_line_launch<B, A, B>(L, p, g, in, out);                                                              \
  }
DTMM_LINE_SIDES(DTMM_LINE_DECLARE)

// run-time lengths
cudaError_t row_line_any4(bool real, const LineLaunch& L, const RowParams& p, const Grid& g, const void* U, void* X);
cudaError_t row_line_any2(bool real, const LineLaunch& L, const RowParams& p, const Grid& g, const void* U, void* X);
cudaError_t col_line_any(const LineLaunch& L, const ColParams& p, const Grid& g, const void* in, void* out);
cudaError_t rows_line(const LineLaunch& L, const void* src, void* dst, int nlines, int W, bool inv, const void* tw,
                      double scale, int lpb);

inline cudaError_t row_line(int C, bool real, const LineLaunch& L, const RowParams& p, const Grid& g, const void* U, void* X) {
  if (real) {
#define DTMM_LINE_ROW(A, B) \
  if (L.geom.n1 == A && L.geom.n2 == B) return row_line_##A##_##B(C, L, p, g, U, X);
    DTMM_LINE_SIDES(DTMM_LINE_ROW)
#undef DTMM_LINE_ROW
  }
  return C == 4 ? row_line_any4(real, L, p, g, U, X) : row_line_any2(real, L, p, g, U, X);
}
inline cudaError_t col_line(const LineLaunch& L, const ColParams& p, const Grid& g, const void* in, void* out) {
#define DTMM_LINE_COL(A, B) \
  if (L.geom.n1 == A && L.geom.n2 == B) return col_line_##A##_##B(L, p, g, in, out);
  DTMM_LINE_SIDES(DTMM_LINE_COL)
#undef DTMM_LINE_COL
  return col_line_any(L, p, g, in, out);
}

}  // namespace dtmm
