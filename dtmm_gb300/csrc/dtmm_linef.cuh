// Row and column passes of a layer step, complex64 bulk, for the sides without
// a register transform of their own (dtmm_regkern.cuh): any n = n1 n2 with n1,
// n2 up to 32 (`line_shape`), two steps of register DFTs.  Slots, threads and
// steps are those of dtmm_linekern.cuh, in FP32 arithmetic.  The sides of
// DTMM_LINEF_SIDES have n1 and n2 at compile time: no switch over lengths, index
// arithmetic by constants and no spills at fewer registers.  They are the sides of the
// complex128 table (a choice, dtmm_linekern.cuh) up to 360 without a register transform.
//
// In shared-memory mixed-radix passes (prime by prime, every column of the
// grid, the whole band) 330-point rows of 8 images took 114 us a layer and
// 250-point columns 72 us; with run-time lengths 66 and 44 us; at compile time 33
// and 30 us (a launch is two to three waves of blocks: latency, and in the first
// step of 10 x 25 three of five threads wait).  Twenty layers, seven rays, run-time
// lengths -> compile time (row / column pass, ms): side 48 .46 / .39 -> .36 / .28; 100
// 1.60 / .79 -> .93 / .60; 200 8.6 / 4.0 -> 4.3 / 2.3; 300 6.6 / 3.4 -> 3.5 / 2.3; 350 6.5 /
// 3.0 -> 3.3 / 2.1.
#pragma once

#include <type_traits>

#include "dtmm_linekern.cuh"

namespace dtmm {

// Launch bounds.  Threads follow the length class that `line_shape` chose the side by;
// blocks a SM as many as the registers allow with few spills.  Rows of 22 and 25 points
// a thread spill at 80 registers and still gain by three blocks of 256 threads instead
// of two (side 350, seven rays 4.24 -> 3.31 ms, three window rows 3.30 -> 2.80), their
// columns lose (2.10 -> 2.43).  Eight blocks of 128 threads instead of six for up to 12
// points: 5 % faster for one window, 3 % slower for nine.
constexpr int linef_threads(int maxl, int cn1, int cn2) {
  return maxl <= 16 && (cn1 == 0 || (line_len_ok(cn1, 16) && line_len_ok(cn2, 16))) ? 128 : 256;
}
constexpr int linef_row_blocks(int maxl, int cn1, int cn2) {
  return linef_threads(maxl, cn1, cn2) == 128 ? (cn1 ? 6 : 5) : (cn1 ? 3 : 2);
}
constexpr int linef_col_blocks(int maxl, int cn1) { return maxl <= (cn1 ? 20 : 16) ? 3 : 2; }

// W^(t k) at k n1 + t
__device__ __forceinline__ void linef_tw(cpx<float>* tw, const void* twg, int n, int n1) {
  for (int e = threadIdx.x; e < n; e += blockDim.x) tw[e] = ((const cpx<float>*)twg)[(e % n1) * (e / n1)];
}

// Row pass (see RowParams): one row of G wavelengths x PB polarisations of one
// ray.  Threads: lines x max(n1, n2).  p.xr < 0: one window, in place.
template <int C, bool REAL, int MAXL, int CN1, int CN2>
__global__ void __launch_bounds__(linef_threads(MAXL, CN1, CN2), linef_row_blocks(MAXL, CN1, CN2))
    k_row_linef(RowParams p, Grid g, LineGeom s, int limW, const cpx<float>* __restrict__ U, cpx<float>* __restrict__ X) {
  using T = typename std::conditional<REAL, float, cpx<float>>::type;
  __shared__ float s_kph[kLineMax];
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n1 = CN1 ? CN1 : s.n1, n2 = CN1 ? CN2 : s.n2, H = g.H, W = CN1 ? CN1 * CN2 : g.W;
  const int P = CN1 ? (CN2 | 1) : s.pitch, LS = n1 * P;
  const int ngrp = (g.nlam + p.G - 1) / p.G, npg = (g.npol + p.PB - 1) / p.PB;
  const int y = p.groups_inner ? blockIdx.y : blockIdx.x;
  const int gi = p.groups_inner ? blockIdx.x : blockIdx.y;
  const int pg = gi % npg, rg = gi / npg;
  const int ray = rg / ngrp, grp = rg - ray * ngrp;
  const int lam0 = grp * p.G, pol0 = pg * p.PB;
  const int G = min(p.G, g.nlam - lam0), NP = min(p.PB, g.npol - pol0);
  const int nlines = G * NP * C, lmaxn = p.G * p.PB * C;
  const bool one = p.xr < 0;
  cpx<float>* acc = (cpx<float>*)smem_raw;                       // [lines][LS]
  cpx<float>* buf = acc + (one ? 0 : (size_t)lmaxn * LS);        // [lines][LS] exchange, then the transformed row
  cpx<float>* tw = buf + (size_t)lmaxn * LS;                     // [W]
  const int HW = H * W, nwin = p.nx * p.ny;
  linef_tw(tw, p.tw, W, n1);
  if (!one)
    for (int e = threadIdx.x; e < nlines * LS; e += blockDim.x) acc[e] = mk<float>(0, 0);
  for (int gl = threadIdx.x; gl < G; gl += blockDim.x) s_kph[gl] = (float)(p.ks[lam0 + gl] * p.dir);
  grid_release();
  grid_wait();  // the column pass's rows
  __syncthreads();
  const float sc = (float)p.in_scale;
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
      const int j = w / p.nx, i = w - j * p.nx, ww = i * p.ny + j;
      if (p.win_only >= 0 && ww != p.win_only) continue;
      if (p.wzero != nullptr && p.wzero[ray * nwin + ww]) continue;
      break;
    }
    const int j = w / p.nx, i = w - j * p.nx, ww = i * p.ny + j;
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      const bool roleA = (half == 0) != fwd;
      const int line = roleA ? lineA : lineB, t = roleA ? tA : tB, len = roleA ? n2 : n1;
      const bool act = line < nlines;
      if (act) {
        const int c = line % C, im = line / C;
        const int gl = im / NP, pol = pol0 + im - gl * NP, lam = lam0 + gl;
        const size_t img = ((size_t)ray * g.npol + pol) * g.nlam + lam;
        cpx<float>* bl = buf + (size_t)line * LS;
        cpx<float> v[MAXL];
        if (half == 0 && !fwd) {
          const cpx<float>* src = U + (size_t)(p.win_only >= 0 ? 0 : j) * g.NI * C * HW + ((img * C + c) * H + y) * W;
          const float* cxl = (p.cx && p.use_cx) ? (const float*)p.cx + (((size_t)ray * p.nx + i) * g.nlam + lam) * W : nullptr;
          const int lim = (int)p.blim[lam];
          const int lo = limW / n1 + 1, hi = (W - limW) / n1;  // entries m in [lo, hi) lie beyond the band
#pragma unroll
          for (int m = 0; m < MAXL; ++m) {
            if (m >= len) break;
            v[m] = mk<float>(0.0f, 0.0f);
            if (m < lo || m >= hi) {
              const int xk = t + n1 * m;
              if ((xk < (W + 1) / 2 ? xk : W - xk) <= lim) {
                cpx<float> a = src[xk];
                if (cxl) a = a * cxl[xk];
                v[m] = swapc(a);
              }
            }
          }
        } else {
          // forward, first step: the accumulated row's slots (t, m); second steps: the exchange's
          const cpx<float>* rl = half == 0 ? acc + (size_t)line * LS : bl;
          const int o = half == 1 && roleA ? P * t : t, st = half == 1 && roleA ? 1 : P;
#pragma unroll
          for (int m = 0; m < MAXL; ++m) {
            if (m >= len) break;
            v[m] = rl[o + st * m];
          }
        }
        step_dft<MAXL, CN1, CN2>(v, roleA, len);
        if (half == 0) {
          const int wo = fwd ? t * n1 : t, ws = fwd ? 1 : n1;
          const int o = fwd ? t : P * t, st = fwd ? P : 1;
          bl[o] = v[0];
#pragma unroll
          for (int k = 1; k < MAXL; ++k) {
            if (k >= len) break;
            bl[o + st * k] = v[k] * tw[wo + ws * k];
          }
        } else if (!fwd) {
#pragma unroll
          for (int m = 0; m < MAXL; ++m) {
            if (m >= len) break;
            bl[t + P * m] = swapc(v[m]);
          }
        } else {
          cpx<float>* dst = X + ((img * C + c) * H + y) * W + t;
#pragma unroll
          for (int m = 0; m < MAXL; ++m) {
            if (m >= len) break;
            // band_out: the next column pass reads the columns inside the band only
            if (!(p.band_out && m > limW / n1 && m < (W - limW) / n1)) *dst = p.accumulate ? *dst + v[m] : v[m];
            dst += n1;
          }
        }
      }
      __syncthreads();
    }
    if (fwd) break;
    // the voxels' operators of the window
    const T* opw = (const T*)p.op + (((size_t)ray * nwin + ww) * HW + (size_t)y * W) * p.rec_stride;
    constexpr int NR = C == 4 ? OP_REC : REC_BLOCK;
    for (int x = threadIdx.x; x < W; x += blockDim.x) {
      T rec[NR];
      load_planes<NR, T>(opw, W, x, rec);
      const int xm = (int)((x * rcp2) >> 16), q = x - xm * n2 + P * xm;
      const T* ef = rec;
      const T* eb = rec + (C == 4 ? REC_BLOCK : 0);
      for (int gl = 0; gl < G; ++gl) {
        const float kph = s_kph[gl];
        cpx<float> qf, dpf, qb, dpb;
        {
          const cpx<float> f0 = phase_of(ef[4], kph), f1 = phase_of(ef[5], kph);
          qf = f1 * sc;
          dpf = f0 - f1;
        }
        if (C == 4) {
          const cpx<float> b0 = phase_of(eb[4], kph), b1 = phase_of(eb[5], kph);
          qb = b1 * sc;
          dpb = b0 - b1;
        }
        for (int pol = 0; pol < NP; ++pol) {
          const int l0 = (gl * NP + pol) * C;
          const cpx<float>* h = buf + (size_t)l0 * LS + q;
          cpx<float>* a = acc + (size_t)l0 * LS + q;
          cpx<float> r[C];
#pragma unroll
          for (int c = 0; c < C; ++c) r[c] = one ? mk<float>(0.0f, 0.0f) : a[c * LS];
          if constexpr (C == 4) {
            apply_block<float, T>(ef, qf, dpf, h[0], h[2 * LS], r[0], r[2]);
            apply_block<float, T>(eb, qb, dpb, h[LS], h[3 * LS], r[1], r[3]);
          } else {
            apply_block<float, T>(ef, qf, dpf, h[0], h[LS], r[0], r[1]);
          }
#pragma unroll
          for (int c = 0; c < C; ++c) a[c * LS] = r[c];
        }
      }
    }
    __syncthreads();
  }
}

// Plain row transforms of `nlines` lines, src -> dst (in place allowed), times
// `scale`; lpb lines a block.
template <int MAXL>
__global__ void __launch_bounds__(MAXL <= 16 ? 128 : 256, MAXL <= 16 ? 5 : 2)
    k_rows_linef(const cpx<float>* src, cpx<float>* dst, int nlines, int W, LineGeom s, int inv,
                 const cpx<float>* __restrict__ twg, float scale, int lpb) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int P = s.pitch, LS = s.n1 * P;
  cpx<float>* buf = (cpx<float>*)smem_raw;
  cpx<float>* tw = buf + (size_t)lpb * LS;
  linef_tw(tw, twg, W, s.n1);
  __syncthreads();
  const int nl = min(lpb, nlines - (int)blockIdx.x * lpb);
#pragma unroll 1
  for (int half = 0; half < 2; ++half) {
    const int n = half == 0 ? s.n1 : s.n2, len = half == 0 ? s.n2 : s.n1;
    const int line = threadIdx.x / n, t = threadIdx.x - line * n;
    if (line < nl) {
      const size_t off = ((size_t)blockIdx.x * lpb + line) * W;
      cpx<float>* fl = buf + (size_t)line * LS;
      const cpx<float>* in = half == 0 ? src + off + t : fl + t;
      const int st = half == 0 ? s.n1 : P;
      cpx<float> v[MAXL];
#pragma unroll
      for (int m = 0; m < MAXL; ++m) {
        if (m >= len) break;
        const cpx<float> a = in[st * m];
        v[m] = half == 0 && inv ? swapc(a) : a;
      }
      line_dft<float, MAXL>(v, len);
      if (half == 0) {
        fl[P * t] = v[0];
#pragma unroll
        for (int k = 1; k < MAXL; ++k) {
          if (k >= len) break;
          fl[P * t + k] = v[k] * tw[t + s.n1 * k];
        }
      } else {
#pragma unroll
        for (int m = 0; m < MAXL; ++m) {
          if (m >= len) break;
          dst[off + t + s.n2 * m] = (inv ? swapc(v[m]) : v[m]) * scale;
        }
      }
    }
    __syncthreads();
  }
}

// Column pass (see ColParams): tc columns x max(cin, cout) components of one
// image; tile element (slot, line) at slot * lines + line, slot m + n2 t for
// ky = t + n1 m.  limH: entries beyond it along y are zero after a KOP_DIAG table.
template <int MAXL, int CN1, int CN2>
__global__ void __launch_bounds__(256, linef_col_blocks(MAXL, CN1))
    k_col_linef(ColParams p, Grid g, LineGeom s, int limH, const cpx<float>* __restrict__ X, cpx<float>* __restrict__ U) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n1 = CN1 ? CN1 : s.n1, n2 = CN1 ? CN2 : s.n2, H = CN1 ? CN1 * CN2 : g.H, W = g.W, TX = p.tc;
  const int CM = max(p.cin, p.cout), NL = CM * TX;
  const int img = blockIdx.y;
  const int tile = (p.tile_lo > 0 && (int)blockIdx.x >= p.tile_lo) ? p.tile_hi0 + ((int)blockIdx.x - p.tile_lo)
                                                                    : (int)blockIdx.x;
  const int x0 = tile * TX;
  const int lam = img_lam(g, img), ray = img_ray(g, img);
  const bool diag = p.kop == KOP_DIAG;
  const int line = threadIdx.x % NL, t = threadIdx.x / NL;
  const int c = line / TX, kx = x0 + line - c * TX;
  const bool in_x = kx < W;
  bool live = in_x;  // the column is read
  grid_release();
  grid_wait();  // the row pass's columns, and the readers of U
  if ((p.band_skip == 2 && diag) || p.xband) {
    const int lim = (int)p.blim[lam];
    bool any = false;
    for (int xc = 0; xc < TX && x0 + xc < W; ++xc) {
      const int xk = x0 + xc;
      any = any || (xk < (W + 1) / 2 ? xk : W - xk) <= lim;
    }
    if (!any) {
      if (!diag && c < p.cout && in_x)
        for (int jj = 0; jj < p.ny; ++jj) {
          cpx<float>* udst = U + ((size_t)jj * g.NI * p.cout + (size_t)img * p.cout + c) * H * W + kx;
          for (int y = t; y < H; y += blockDim.x / NL) udst[(size_t)y * W] = mk<float>(0.0f, 0.0f);
        }
      return;
    }
    if (p.xband) live = in_x && (kx < (W + 1) / 2 ? kx : W - kx) <= lim;
  }
  cpx<float>* tile_x = (cpx<float>*)smem_raw;                              // [H][NL] exchange
  cpx<float>* tile_s = p.ny > 1 ? tile_x + (size_t)H * NL : tile_x;        // [H][NL] spectra along y
  cpx<float>* tw = tile_x + (size_t)H * NL * (p.ny > 1 ? 2 : 1);
  linef_tw(tw, p.tw, H, n1);
  __syncthreads();
  const float sc = (float)p.out_scale;
  // halves: 0, 1 the forward transform (skipped without do_fwd), then two per window row
#pragma unroll 1
  for (int q = p.do_fwd ? 0 : 1; q < 2 + 2 * p.ny; ++q) {
    const bool fwd = q < 2;
    const int half = q & 1;
    const bool roleA = (half == 0) != fwd;  // n1 threads with n2 points
    const int n = roleA ? n1 : n2, len = roleA ? n2 : n1;
    const bool act = t < n && c < (fwd ? p.cin : p.cout);
    const int jj = (q - 2) >> 1, j = p.j_only >= 0 ? p.j_only : jj;
    const bool skip_dft = (q == 1 && !p.do_fwd) || (!fwd && !p.inverse_out);
    if (skip_dft && !fwd && half == 1) continue;
    if (act) {
      cpx<float> v[MAXL];
      if (fwd && (half == 0 || skip_dft)) {
        // rows y = t + n2 m, or without a forward transform ky = t + n1 m
        const cpx<float>* src = X + (((size_t)img * p.cin + c) * H + t) * W + kx;
        const int step = n * W;
#pragma unroll
        for (int m = 0; m < MAXL; ++m) {
          if (m >= len) break;
          v[m] = live ? *src : mk<float>(0.0f, 0.0f);
          src += step;
        }
      } else if (half == 0) {
        const float* cyj = p.cy ? (const float*)p.cy + (((size_t)ray * p.cy_rows + j) * g.nlam + lam) * H : nullptr;
        const int lo = diag ? limH / n1 + 1 : len, hi = diag ? (H - limH) / n1 : len;  // beyond the band
#pragma unroll
        for (int m = 0; m < MAXL; ++m) {
          if (m >= len) break;
          cpx<float> a = mk<float>(0.0f, 0.0f);
          if (m < lo || m >= hi) {
            a = tile_s[(size_t)(m + n2 * t) * NL + line];
            if (cyj) a = a * cyj[t + n1 * m];
          }
          v[m] = skip_dft ? a : swapc(a);
        }
      } else {
        const cpx<float>* z = tile_x + (size_t)(roleA ? n2 * t : t) * NL + line;
        const int st = (roleA ? 1 : n2) * NL;
#pragma unroll
        for (int m = 0; m < MAXL; ++m) {
          if (m >= len) break;
          v[m] = z[st * m];
        }
      }
      if (!skip_dft) step_dft<MAXL, CN1, CN2>(v, roleA, len);
      if (half == 0 && !skip_dft) {
        const int wo = fwd ? t * n1 : t, ws = fwd ? 1 : n1;
        cpx<float>* z = tile_x + (size_t)(fwd ? t : n2 * t) * NL + line;
        const int st = (fwd ? n2 : 1) * NL;
        z[0] = v[0];
#pragma unroll
        for (int k = 1; k < MAXL; ++k) {
          if (k >= len) break;
          z[st * k] = v[k] * tw[wo + ws * k];
        }
      } else if (fwd) {
        // spectra k = t + n1 m through the diagonal table into the thread's own slots
        const cpx<float>* ek = (diag && in_x) ? (const cpx<float>*)p.ktab + (((size_t)lam * W + kx) * H + t) * 2 +
                                                    ((((c & 1) == 0) || p.cin == 2) ? 0 : 1)
                                              : nullptr;
        const int lo = diag ? limH / n1 + 1 : len, hi = diag ? (H - limH) / n1 : len;
        cpx<float>* z = tile_s + (size_t)(n2 * t) * NL + line;
#pragma unroll
        for (int m = 0; m < MAXL; ++m) {
          if (m >= len) break;
          cpx<float> a = mk<float>(0.0f, 0.0f);
          if (m < lo || m >= hi) {
            a = v[m];
            if (ek) a = a * ek[(size_t)n1 * m * 2];
            if (p.kop != KOP_MAT) a = a * sc;
          }
          z[NL * m] = a;
        }
      } else if (in_x) {
        // window row j: y = t + n2 m, or without an inverse transform ky = t + n1 m
        cpx<float>* dst = U + (((size_t)jj * g.NI * p.cout + (size_t)img * p.cout + c) * H + t) * W + kx;
        const int step = n * W;
#pragma unroll
        for (int m = 0; m < MAXL; ++m) {
          if (m >= len) break;
          *dst = skip_dft ? v[m] : swapc(v[m]);
          dst += step;
        }
      }
    }
    if (fwd && half == 1 && p.kop == KOP_MAT) {
      __syncthreads();
      // one point k, column xc and every component a turn
      for (int e = threadIdx.x; e < H * TX; e += blockDim.x) {
        const int sl = e / TX, xe = e - sl * TX;
        const int kt = sl / n2, k = kt + n1 * (sl - kt * n2);
        if (x0 + xe >= W) continue;
        cpx<float>* z = tile_s + (size_t)sl * NL + xe;
        const cpx<float>* mt = (const cpx<float>*)p.ktab + ray * p.ktab_ray_stride +
                               (((size_t)lam * H + k) * W + x0 + xe) * p.cout * p.cin;
        cpx<float> in[4];
#pragma unroll
        for (int ci = 0; ci < 4; ++ci)
          if (ci < p.cin) in[ci] = z[ci * TX];
#pragma unroll
        for (int o = 0; o < 4; ++o) {
          if (o >= p.cout) break;
          cpx<float> a = mk<float>(0.0f, 0.0f);
#pragma unroll
          for (int ci = 0; ci < 4; ++ci)
            if (ci < p.cin) a = cfma(mt[o * p.cin + ci], in[ci], a);
          z[o * TX] = a * sc;
        }
      }
    }
    // (a thread reads back its own slots after the diagonal table)
    if (!(fwd && half == 1 && p.kop != KOP_MAT)) __syncthreads();
  }
}

// Sides with kernels of their own (real operator records), instantiated in dtmm_linef_<a..d>.cu
#define DTMM_LINEF_SIDES(X) \
  X(5, 9) X(5, 10) X(5, 15) X(5, 25) X(6, 8) X(6, 10) X(7, 9) X(7, 25) X(8, 9) X(9, 10) X(9, 15) X(10, 10) \
  X(10, 11) X(10, 12) X(10, 14) X(10, 15) X(10, 20) X(10, 25) X(11, 20) X(12, 14) X(12, 15) X(14, 14) X(14, 15) \
  X(14, 20) X(14, 25) X(15, 15) X(15, 18) X(15, 20) X(15, 22) X(16, 22) X(18, 20)
inline bool linef_side(int n1, int n2) {
#define DTMM_LINEF_IS(A, B) \
  if (n1 == A && n2 == B) return true;
  DTMM_LINEF_SIDES(DTMM_LINEF_IS)
#undef DTMM_LINEF_IS
  return false;
}
#define DTMM_LINEF_DECLARE(A, B)                                                                                     \
  cudaError_t row_linef_##A##_##B(int C, const LineLaunch& L, const RowParams& p, const Grid& g, const void* U, void* X); \
  cudaError_t col_linef_##A##_##B(const LineLaunch& L, const ColParams& p, const Grid& g, const void* in, void* out);
#define DTMM_LINEF_DEFINE(A, B)                                                                                      \
  cudaError_t row_linef_##A##_##B(int C, const LineLaunch& L, const RowParams& p, const Grid& g, const void* U, void* X) { \
    return line_launch(C == 4 ? k_row_linef<4, true, B, A, B> : k_row_linef<2, true, B, A, B>, L, p, g, L.geom, L.lim, \
                       (const cpx<float>*)U, (cpx<float>*)X);                                                        \
  }                                                                                                                  \
  cudaError_t col_linef_##A##_##B(const LineLaunch& L, const ColParams& p, const Grid& g, const void* in, void* out) { \
    return line_launch(k_col_linef<B, A, B>, L, p, g, L.geom, L.lim, (const cpx<float>*)in, (cpx<float>*)out);       \
  }
DTMM_LINEF_SIDES(DTMM_LINEF_DECLARE)

cudaError_t row_linef(int C, bool real, const LineLaunch& L, const RowParams& p, const Grid& g, const void* U, void* X);
cudaError_t col_linef(const LineLaunch& L, const ColParams& p, const Grid& g, const void* in, void* out);
cudaError_t rows_linef(const LineLaunch& L, const void* src, void* dst, int nlines, int W, bool inv, const void* tw,
                       double scale, int lpb);

}  // namespace dtmm
