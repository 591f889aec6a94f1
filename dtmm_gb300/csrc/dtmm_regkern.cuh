// Row and column passes of a layer step with register line transforms
// (complex64 bulk, every side N = N1 * N2 that `reg_lanes` lists).
//
// Each (image, component) line is transformed by a group of N1 lanes
// (`TwoStep`); the groups synchronise with their own lane mask, so a warp may
// hold lines of different activity.  Work per block:
//   row pass     one row y of G wavelengths x PB polarisations of one ray:
//                for each window, the weighted row is inverse-transformed into
//                the line's row buffer, the per-voxel operator accumulates into
//                the line's accumulator, and the accumulator is transformed
//                forward and stored (natural order throughout);
//   column pass  TX columns x C components of one image: forward column
//                transforms, the k-space operator, then per window row j:
//                spectra * cy_j -> inverse transform (k_layer_col_reg).
//
// The kernels are instantiated per side in separate translation units
// (dtmm_reg_*.cu) through DTMM_REG_DEFINE; the engine reaches them through the
// row_reg_<N> / col_reg_<N> functions declared at the end.
#pragma once

#include <type_traits>

#include "dtmm_layer.cuh"
#include "dtmm_regfft.cuh"

namespace dtmm {

// lanes [g * N1, g * N1 + N1) of the calling lane's group
template <int N1>
__device__ __forceinline__ unsigned group_mask() {
  if constexpr (N1 >= 32) {
    return 0xffffffffu;
  } else {
    const unsigned lane = threadIdx.x & 31u;
    return ((1u << N1) - 1u) << (lane & ~(unsigned)(N1 - 1));
  }
}

// wavelengths per row block at most (the engine caps row_group here)
constexpr int kMaxRowGroup = 64;

// row buffer stride (complex elements): with N1 = 4 or 8 several line groups
// share a half-warp, and a stride of W + 4 (W + 8) puts their exchange slots
// on disjoint banks; W is a multiple of 16 for every listed side
__host__ __device__ constexpr int reg_row_stride(int n1, int w) { return n1 == 4 ? w + 4 : (n1 == 8 ? w + 8 : w); }

// Band variants of the row pass.  The window rows arrive band-limited: every
// entry with |f_x| beyond the wavelength's band limit lim is zero.  Variant
// b > 0 loads only the entries m < KB and m >= N2 - KB of a lane (KB =
// row_band_slots) and runs the sparse step-1 DFT; it is exact when every
// wavelength of the launch has lim < KB N1 (the other entries then lie
// beyond the band: t + N1 m >= N1 KB for m >= KB on the positive side,
// W - (t + N1 m) > N1 KB for m < N2 - KB on the negative side).
__host__ __device__ constexpr int row_band_slots(int n2, int b) {
  return b == 0 ? 0 : ((b == 1 ? n2 / 8 : n2 / 4) > 1 ? (b == 1 ? n2 / 8 : n2 / 4) : 1);
}
__host__ __device__ constexpr bool row_band_ok(int n2, int b) { return b == 0 || 2 * row_band_slots(n2, b) < n2; }

// largest block of the register row pass for an n-point row (its launch bounds)
__host__ __device__ constexpr int reg_row_max_threads(int n) {
  return reg_lanes(n) > 0 && n / reg_lanes(n) >= 32 ? 512 : 256;
}

// the band variant of an n-point row for the largest band limit of a launch
__host__ __device__ constexpr int row_band_pick(int n, int lim) {
  const int n1 = reg_lanes(n), n2 = n1 > 0 ? n / n1 : 0;
  for (int b = 1; b <= 2; ++b)
    if (n1 > 0 && row_band_ok(n2, b) && lim < row_band_slots(n2, b) * n1) return b;
  return 0;
}

// Launch bounds: rows of up to 16 points per lane, and single-window rows, keep
// at most 80 registers, so that six 128-thread blocks share an SM (measured 8 %
// faster than four at 117 registers for 256-point rows); with several windows
// and more than 16 points per lane the spills of that cost more than the warps
// (320 points, nine windows: 244 us a layer, 221 with 128 registers); 32 points
// per lane need the registers of a whole 512-thread block.
// XR > 0 (several windows, 16 points a lane): the block holds kXrLines lines and
// W / XR threads, and each thread keeps the accumulators of its XR pixels in
// registers across the windows: no second set of lines and no shared-memory
// read-modify-write per window (nine windows, one layer: 128 points 40 -> 31 us,
// 256 points of the 2x2 method 66 -> 48 us).  Four 128-thread blocks a SM: five at 96
// registers spill next to nothing and are slower (256 points of the 4x4 method 95 ->
// 101 us a launch, 128 points 29 -> 34), six at 80 as well (99, 38): shared memory bounds it.
// XR = -1: one window (one window in all).  There is nothing
// to accumulate: the operators' results replace the transformed rows in place,
// without the second set of lines (half the shared memory, so twice the blocks
// a SM) and its clearing, reads and writes.  320 points, 70
// images: 166 -> 146 us a layer.
constexpr int kXrLines = 8;
// pixels a thread of that variant (0: the side has none): 16 points a lane, 128
// registers a thread with the accumulators; with 32 points a lane (168 registers)
// it took 1.35 ms a layer for 1024-point rows against 1.27 ms in shared memory
__host__ __device__ constexpr int xr_pixels(int n) {
  const int n1 = reg_lanes(n);
  return n1 > 0 && n == 16 * n1 ? n / (kXrLines * n1) : 0;
}
template <typename R, int C, bool REAL, int N1, int N2, int BAND, int XR = 0>
__global__ void __launch_bounds__(XR > 0 ? (N1 * N2) / (XR > 0 ? XR : 1) : (N2 >= 32 ? 512 : 256),
                                  XR > 0 ? 512 / (kXrLines * N1) : (N2 >= 32 ? 1 : (XR == 0 && N2 > 16 ? 2 : 3)))
    k_layer_row_reg(RowParams p, Grid g, const cpx<R>* __restrict__ U, cpx<R>* __restrict__ X) {
  constexpr bool ONE = XR < 0;
  constexpr int XL = kXrLines;
  using T = typename std::conditional<REAL, R, cpx<R>>::type;
  using TS = TwoStep<N1, N2>;
  constexpr int W = N1 * N2;
  constexpr int LS = reg_row_stride(N1, W);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int H = g.H;
  const int ngrp = (g.nlam + p.G - 1) / p.G;
  const int npg = (g.npol + p.PB - 1) / p.PB;
  // groups_inner: the groups of one row are neighbours in the launch order,
  // so that the row's operator records (shared by every wavelength and
  // polarisation) come from HBM once and from L2 for the other groups
  const int y = p.groups_inner ? blockIdx.y : blockIdx.x;
  const int gi = p.groups_inner ? blockIdx.x : blockIdx.y;
  const int pg = gi % npg, rg = gi / npg;
  const int ray = rg / ngrp, grp = rg - ray * ngrp;
  const int lam0 = grp * p.G, pol0 = pg * p.PB;
  const int G = min(p.G, g.nlam - lam0);
  const int NP = min(p.PB, g.npol - pol0);  // polarisations of this block
  const int nlines = G * NP * C;
  cpx<R>* acc = (cpx<R>*)smem_raw;                  // [lines][LS]
  cpx<R>* tmp = acc + (XR != 0 ? 0 : (size_t)p.G * p.PB * C * LS);  // [lines][LS] exchange and transformed rows
  cpx<R>* tw = tmp + (size_t)p.G * p.PB * C * LS;   // [W]  twiddles, lane-major (TwoStep::twiddle_entry)
  const int HW = H * W;
  const int nwin = p.nx * p.ny;
  for (int e = threadIdx.x; e < W; e += blockDim.x) tw[e] = TS::twiddle_entry((const cpx<R>*)p.tw, e);
  if (XR == 0)
    for (int e = threadIdx.x; e < nlines * LS; e += blockDim.x) acc[e] = mk<R>(0, 0);
  cpx<R> racc[XR > 0 ? XR : 1][XL];
  if (XR > 0) {
#pragma unroll
    for (int k = 0; k < (XR > 0 ? XR : 1); ++k)
#pragma unroll
      for (int l = 0; l < XL; ++l) racc[k][l] = mk<R>((R)0, (R)0);
  }
  // phase scale k0 * direction of each wavelength of the block (formed once, in FP64)
  __shared__ R s_kph[kMaxRowGroup];
  __shared__ int s_lim[kMaxRowGroup];  // band limit of each wavelength (columns beyond read as zero)
  for (int g2 = threadIdx.x; g2 < G; g2 += blockDim.x) {
    s_kph[g2] = (R)(p.ks[lam0 + g2] * p.dir);
    s_lim[g2] = (int)p.blim[lam0 + g2];
  }
  const R sc = (R)p.in_scale;  // det of each block's records
  grid_release();
  grid_wait();  // the column pass's rows
  __syncthreads();
  const int line = threadIdx.x / N1, t = threadIdx.x % N1;
  const bool active = line < nlines;
  const unsigned gm = group_mask<N1>();
  // the lane's twiddles W_N^(t k1) in registers when they are few
  constexpr bool TWREG = N2 <= 8;
  cpx<R> trow[TWREG ? N2 : 1];
  if (TWREG) {
#pragma unroll
    for (int k1 = 0; k1 < (TWREG ? N2 : 1); ++k1) trow[k1] = tw[k1 * N1 + t];
  }
  const int c = line % C, im = line / C;
  const int gl = im / NP, pol = pol0 + im - gl * NP;
  const int lam = lam0 + gl;
  const int img = (ray * g.npol + pol) * g.nlam + lam;
  cpx<R>* xl = tmp + (size_t)line * LS;
  for (int j = 0; j < p.ny; ++j) {
    // a single-window chain reads the one window row the column pass emitted
    const cpx<R>* Uj = U + (size_t)(p.win_only >= 0 ? 0 : j) * g.NI * C * HW;
    for (int i = 0; i < p.nx; ++i) {
      const int w = i * p.ny + j;
      if (p.win_only >= 0 && w != p.win_only) continue;
      if (p.wzero != nullptr && p.wzero[ray * nwin + w]) continue;
      if (active) {
        const cpx<R>* src = Uj + (((size_t)img * C + c) * H + y) * W;
        const R* cxl = (p.cx && p.use_cx) ? (const R*)p.cx + (((size_t)ray * p.nx + i) * g.nlam + lam) * W : nullptr;
        cpx<R> v[N2];
        const int lim = s_lim[gl];
        constexpr int KB = row_band_slots(N2, BAND);
#pragma unroll
        for (int m = 0; m < N2; ++m) {
          if (BAND == 0 || m < KB || m >= N2 - KB) {
            const int xk = t + N1 * m;
            const int fx = xk < (W + 1) / 2 ? xk : W - xk;  // |fsigned(xk)|
            cpx<R> a = fx <= lim ? src[xk] : mk<R>((R)0, (R)0);
            v[m] = cxl ? a * cxl[xk] : a;
          } else {
            v[m] = mk<R>((R)0, (R)0);
          }
        }
        TS::template step1<R, true, BAND == 0 ? full_mask(N2) : band_mask(N2, KB)>(v, xl, 1, TWREG ? trow : nullptr,
                                                                                    tw, t);
        __syncwarp(gm);
        cpx<R> u[TS::J][N1];
        TS::template step2<R, true>(u, xl, 1, t);
        __syncwarp(gm);  // every read of the exchange precedes the results that overwrite it
        TS::template store<R>(u, xl, 1, t);  // the 1/W of the inverse rides on the operator's 1/det
      }
      __syncthreads();
      const int rs = p.rec_stride;
      const T* opw = (const T*)p.op + (((size_t)ray * nwin + w) * HW + (size_t)y * W) * rs;
      // XU pixels per thread and round: their records are loaded together, so
      // that several rounds of global loads are in flight (long rows hold
      // few blocks per SM)
      constexpr int XU = (C == 2 && N2 >= 32) ? 4 : 1;
      constexpr int NR = C == 4 ? OP_REC : REC_BLOCK;  // records this pass reads per voxel
      if constexpr (XR > 0) {
        // pixels threadIdx.x + k W / XR of the block's images b (full blocks of one
        // or two polarisations, which share their wavelength's phases)
#pragma unroll
        for (int k = 0; k < (XR > 0 ? XR : 1); ++k) {
          const int x = threadIdx.x + k * (W / (XR > 0 ? XR : 1));
          T rec[NR];
          load_planes<NR, T>(opw, W, x, rec);
          const T* ef = rec;
          const T* eb = rec + (C == 4 ? REC_BLOCK : 0);
          cpx<R> qf, dpf, qb, dpb;
#pragma unroll
          for (int b = 0; b < XL / C; ++b) {
            if (b % 2 == 0 || NP == 1) {
              const R kph = s_kph[NP == 1 ? b : b / 2];
              const cpx<R> f0 = phase_of(ef[4], kph), f1 = phase_of(ef[5], kph);
              qf = f1 * sc;
              dpf = f0 - f1;
              if (C == 4) {
                const cpx<R> b0 = phase_of(eb[4], kph), b1 = phase_of(eb[5], kph);
                qb = b1 * sc;
                dpb = b0 - b1;
              }
            }
            const cpx<R>* h = tmp + (size_t)(C * b) * LS + x;
            if (C == 4) {
              apply_block<R, T>(ef, qf, dpf, h[0], h[2 * LS], racc[k][C * b], racc[k][C * b + 2 % C]);
              apply_block<R, T>(eb, qb, dpb, h[LS], h[3 * LS], racc[k][C * b + 1], racc[k][C * b + 3 % C]);
            } else {
              apply_block<R, T>(ef, qf, dpf, h[0], h[LS], racc[k][C * b], racc[k][C * b + 1]);
            }
          }
        }
        __syncthreads();
        continue;
      }
      for (int x0 = threadIdx.x; x0 < W; x0 += XU * blockDim.x) {
        T rec[XU][NR];
#pragma unroll
        for (int k = 0; k < XU; ++k) {
          const int x = x0 + k * blockDim.x;
          if (x >= W) break;
          load_planes<NR, T>(opw, W, x, rec[k]);
        }
#pragma unroll
        for (int k = 0; k < XU; ++k) {
          const int x = x0 + k * blockDim.x;
          if (x >= W) break;
          const T* ef = rec[k];
          const T* eb = rec[k] + (C == 4 ? REC_BLOCK : 0);
          for (int g2 = 0; g2 < G; ++g2) {
            const R kph = s_kph[g2];
            // projector form of each block: q = p1 scale, dp = p0 - p1
            cpx<R> qf, dpf, qb, dpb;
            {
              const cpx<R> f0 = phase_of(ef[4], kph), f1 = phase_of(ef[5], kph);
              qf = f1 * sc;
              dpf = f0 - f1;
            }
            if (C == 4) {
              const cpx<R> b0 = phase_of(eb[4], kph), b1 = phase_of(eb[5], kph);
              qb = b1 * sc;
              dpb = b0 - b1;
            }
            for (int q = 0; q < NP; ++q) {
              const int l0 = (g2 * NP + q) * C;
              const cpx<R>* h = tmp + (size_t)l0 * LS + x;
              cpx<R>* a = acc + (size_t)l0 * LS + x;
              if constexpr (ONE) {
                const cpx<R> z = mk<R>((R)0, (R)0);
                cpx<R> a0 = z, a1 = z, a2 = z, a3 = z;
                if (C == 4) {
                  apply_block<R, T>(ef, qf, dpf, h[0], h[2 * LS], a0, a2);
                  apply_block<R, T>(eb, qb, dpb, h[LS], h[3 * LS], a1, a3);
                  a[0] = a0; a[LS] = a1; a[2 * LS] = a2; a[3 * LS] = a3;
                } else {
                  apply_block<R, T>(ef, qf, dpf, h[0], h[LS], a0, a1);
                  a[0] = a0; a[LS] = a1;
                }
              } else if (C == 4) {
                cpx<R> a0 = a[0], a1 = a[LS], a2 = a[2 * LS], a3 = a[3 * LS];
                apply_block<R, T>(ef, qf, dpf, h[0], h[2 * LS], a0, a2);
                apply_block<R, T>(eb, qb, dpb, h[LS], h[3 * LS], a1, a3);
                a[0] = a0; a[LS] = a1; a[2 * LS] = a2; a[3 * LS] = a3;
              } else {
                cpx<R> a0 = a[0], a1 = a[LS];
                apply_block<R, T>(ef, qf, dpf, h[0], h[LS], a0, a1);
                a[0] = a0; a[LS] = a1;
              }
            }
          }
        }
      }
      __syncthreads();
    }
  }
  if constexpr (XR > 0) {  // the accumulators into the rows of the forward transform
#pragma unroll
    for (int k = 0; k < (XR > 0 ? XR : 1); ++k)
#pragma unroll
      for (int l = 0; l < XL; ++l) acc[(size_t)l * LS + threadIdx.x + k * (W / (XR > 0 ? XR : 1))] = racc[k][l];
    __syncthreads();
  }
  if (active) {
    cpx<R> v[N2];
    const cpx<R>* al = acc + (size_t)line * LS;
#pragma unroll
    for (int m = 0; m < N2; ++m) v[m] = al[t + N1 * m];
    if (XR != 0) __syncwarp(gm);  // the line is read before the exchange overwrites it
    TS::template step1<R, false>(v, xl, 1, TWREG ? trow : nullptr, tw, t);
    __syncwarp(gm);
    cpx<R> u[TS::J][N1];
    TS::template step2<R, false>(u, xl, 1, t);
    cpx<R>* dst = X + (((size_t)img * C + c) * H + y) * W;
    constexpr int KBO = row_band_slots(N2, BAND);
    if constexpr (TS::EVEN) {
      TS::template to_lane_order<R>(u, v);
#pragma unroll
      for (int m = 0; m < N2; ++m) {
        // band_out: the next column pass reads the columns inside the band only
        if (BAND != 0 && m >= KBO && m < N2 - KBO && p.band_out) continue;
        dst[t + N1 * m] = p.accumulate ? dst[t + N1 * m] + v[m] : v[m];
      }
    } else {
      // straight from the second step's registers: N1 (or the last round's
      // N2 % N1) consecutive points a store
#pragma unroll
      for (int j = 0; j < TS::J; ++j) {
        const int k1 = t + N1 * j;
        if (k1 < N2) {
#pragma unroll
          for (int k2 = 0; k2 < N1; ++k2) {
            const int e = k1 + N2 * k2;
            if (BAND != 0 && e >= KBO * N1 && e < W - KBO * N1 && p.band_out) continue;
            dst[e] = p.accumulate ? dst[e] + u[j][k2] : u[j][k2];
          }
        }
      }
    }
  }
}

// Plain row FFT of `nlines` lines of N = N1 * N2 points, natural order in
// and out, src -> dst (the same array for in place: a line's group reads it
// completely before it writes), times `scale`; blockDim / N1 lines per block.
template <typename R, int N1, int N2, bool INV>
__global__ void __launch_bounds__(256) k_fft_rows_reg(const cpx<R>* src, cpx<R>* dst, int nlines,
                                                     const cpx<R>* __restrict__ twg, R scale) {
  using TS = TwoStep<N1, N2>;
  constexpr int W = N1 * N2;
  constexpr int LS = reg_row_stride(N1, W);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cpx<R>* tw = (cpx<R>*)smem_raw;  // [W] twiddles, lane-major
  cpx<R>* xb = tw + W;             // [lines per block][LS] exchange
  for (int e = threadIdx.x; e < W; e += blockDim.x) tw[e] = TS::twiddle_entry(twg, e);
  __syncthreads();
  const int lpb = blockDim.x / N1;
  const int li = threadIdx.x / N1, t = threadIdx.x % N1;
  const int line = blockIdx.x * lpb + li;
  if (li >= lpb || line >= nlines) return;  // whole lane groups leave together
  const unsigned gm = group_mask<N1>();
  cpx<R>* xl = xb + (size_t)li * LS;
  const cpx<R>* in = src + (size_t)line * W;
  cpx<R>* out = dst + (size_t)line * W;
  cpx<R> v[N2];
#pragma unroll
  for (int m = 0; m < N2; ++m) v[m] = in[t + N1 * m];
  TS::template step1<R, INV>(v, xl, 1, nullptr, tw, t);
  __syncwarp(gm);
  cpx<R> u[TS::J][N1];
  TS::template step2<R, INV>(u, xl, 1, t);
  if constexpr (TS::EVEN) {
    TS::template to_lane_order<R>(u, v);
#pragma unroll
    for (int m = 0; m < N2; ++m) out[t + N1 * m] = v[m] * scale;
  } else {
    __syncwarp(gm);
    TS::template store<R>(u, xl, 1, t, scale);
    __syncwarp(gm);
#pragma unroll
    for (int m = 0; m < N2; ++m) out[t + N1 * m] = xl[t + N1 * m];
  }
}

// Split of the column pass, n = n1 n2: the most even one (up to 32 each).
__host__ __device__ constexpr int col_n1(int n) {
  int best = 0;
  for (int a = 1; a * a <= n; ++a)
    if (n % a == 0 && n / a <= 32) best = a;
  return best;
}
__host__ __device__ constexpr int col_pitch(int n) { return (n / col_n1(n)) | 1; }
__host__ __device__ constexpr int col_threads_per_line(int n) { return n / col_n1(n); }
// lines of a block at most: tiles of four columns of four components
constexpr int kColLines = 16;
__host__ __device__ constexpr size_t col_smem(int n, int lines) {
  return ((size_t)lines * col_n1(n) * col_pitch(n) + n) * 2 * sizeof(float);
}
// threads of a block at most (whole warps), and blocks a SM: 24 warps while
// that leaves 80 registers a thread
__host__ __device__ constexpr int col_max_threads(int n) { return (kColLines * col_threads_per_line(n) + 31) / 32 * 32; }
__host__ __device__ constexpr int col_min_blocks(int n) {
  return 768 / col_max_threads(n) > 1 ? 768 / col_max_threads(n) : 1;
}
// band variant of an n-point column for the largest band limit (as row_band_pick)
__host__ __device__ constexpr int col_band_pick(int n, int lim) {
  const int n1 = col_n1(n), n2 = n / n1;
  for (int b = 1; b <= 2; ++b)
    if (row_band_ok(n2, b) && lim < row_band_slots(n2, b) * n1) return b;
  return 0;
}

// Column pass, complex64 bulk, k-space operator KOP_NONE, KOP_DIAG or KOP_MAT
// (cin x cout per k).  TX columns x max(cin, cout) components of one image;
// consecutive threads on consecutive columns, n2 (the larger factor) threads a
// line.  A thread loads its points of the forward transform's first step from
// global memory straight into registers and stores the inverse transform's
// results from registers, so a line passes through shared memory once per
// transform (exchange slots (k, s) at k + P s, P = n2 | 1, lines innermost):
//   forward  t < n2: y = t + n2 m, DFT n1, twiddle  -> slots t + P k
//            t < n1: slots s + P t, DFT n2          -> ky = t + n1 m, in registers
//   inverse  t < n1: x cy_j, DFT n2, twiddle        -> slots k + P t
//            t < n2: slots t + P s, DFT n1          -> y = t + n2 m
// BAND > 0 (KOP_DIAG): the table is zero beyond betamax and the axis' band
// limit is below KB n1, so only the entries m < KB and m >= n2 - KB exist: the
// forward transform forms no others and the inverse one runs the sparse DFT.
// Latency-bound (a launch is one to four waves of blocks); staging the columns
// through shared memory on the way in and out, as before, took 27 us for 256
// points (three window rows, 18 images), 249 us for 1024 (five rows, 6 images,
// two components) and 121 us for 320 (70 images), this takes 20, 120 and 83.
template <typename R, int N, int BAND>
__global__ void __launch_bounds__(col_max_threads(N), col_min_blocks(N))
    k_layer_col_reg(ColParams p, Grid g, const cpx<R>* __restrict__ X, cpx<R>* __restrict__ U) {
  constexpr int H = N, N1 = col_n1(N), N2 = N / N1, P = N2 | 1;
  constexpr bool D = BAND != 0;  // KOP_DIAG between two transforms: nothing else is compiled in
  constexpr int KB = row_band_slots(N2, BAND);
  constexpr unsigned MASK = BAND == 0 ? full_mask(N2) : band_mask(N2, KB);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int W = g.W, TX = p.tc, CM = max(p.cin, p.cout), NL = CM * TX;
  cpx<R>* tile = (cpx<R>*)smem_raw;         // [N1 P][NL]
  cpx<R>* tw = tile + (size_t)N1 * P * NL;  // [H] W^(t k) at k N1 + t, t < N1
  const int img = blockIdx.y;
  // tile_lo > 0: the launch covers the in-band tiles only, tiles [0, tile_lo)
  // and from tile_hi0 on (the others write nothing with band_skip 2)
  const int bx = (p.tile_lo > 0 && (int)blockIdx.x >= p.tile_lo) ? p.tile_hi0 + ((int)blockIdx.x - p.tile_lo)
                                                                  : (int)blockIdx.x;
  const int x0 = bx * TX;
  const int lam = img_lam(g, img), ray = img_ray(g, img);
  const int line = threadIdx.x % NL, t = threadIdx.x / NL;
  const int c = line / TX, kx = x0 + (line - c * TX);
  const bool in_x = kx < W;
  bool live = in_x;  // the column is read
  grid_release();
  grid_wait();  // the row pass's columns, and the readers of U
  if ((p.band_skip && p.kop == KOP_DIAG) || p.xband) {
    const int lim = (int)p.blim[lam];
    bool any = false;
    for (int xc = 0; xc < TX && x0 + xc < W; ++xc) {
      const int xk = x0 + xc;
      any = any || (xk < (W + 1) / 2 ? xk : W - xk) <= lim;
    }
    if (!any) {  // the whole block leaves together
      if (p.band_skip == 1 || p.kop != KOP_DIAG) {
        if (c < p.cout && in_x)
          for (int jj = 0; jj < p.ny; ++jj) {
            cpx<R>* udst = U + ((size_t)jj * g.NI * p.cout + (size_t)img * p.cout + c) * H * W + kx;
            for (int y = t; y < H; y += blockDim.x / NL) udst[(size_t)y * W] = mk<R>((R)0, (R)0);
          }
      }
      return;
    }
    if (p.xband) live = in_x && (kx < (W + 1) / 2 ? kx : W - kx) <= lim;
  }
  cpx<R> v[N2];
  if (D || p.do_fwd) {
    // (loads first: the twiddle table fills while they are in flight)
    cpx<R> u[N1];
    const bool act = t < N2 && c < p.cin;
    if (act) {
      const cpx<R>* src = X + (((size_t)img * p.cin + c) * H + t) * W + kx;
#pragma unroll
      for (int m = 0; m < N1; ++m) {
        u[m] = live ? *src : mk<R>((R)0, (R)0);
        src += N2 * W;
      }
    }
    for (int e = threadIdx.x; e < H; e += blockDim.x) tw[e] = ((const cpx<R>*)p.tw)[(e % N1) * (e / N1)];
    __syncthreads();
    if (act) {
      RegDFTg<R, N1, false>::run(u);
      tile[(size_t)t * NL + line] = u[0];
#pragma unroll
      for (int k = 1; k < N1; ++k) tile[(size_t)(t + P * k) * NL + line] = u[k] * tw[t * N1 + k];
    }
    __syncthreads();
    if (t < N1 && c < p.cin) {
#pragma unroll
      for (int m = 0; m < N2; ++m) v[m] = tile[(size_t)(m + P * t) * NL + line];
      RegDFTg<R, N2, false>::run(v);
    }
  } else {
    for (int e = threadIdx.x; e < H; e += blockDim.x) tw[e] = ((const cpx<R>*)p.tw)[(e % N1) * (e / N1)];
    if (t < N1 && c < p.cin) {
      const cpx<R>* src = X + (((size_t)img * p.cin + c) * H + t) * W + kx;
#pragma unroll
      for (int m = 0; m < N2; ++m) {
        v[m] = live ? *src : mk<R>((R)0, (R)0);
        src += N1 * W;
      }
    }
    __syncthreads();
  }
  const R sc = (R)p.out_scale;
  if (!D && p.kop == KOP_MAT) {
    // the matrix per k across a column's components, one point a turn, through the thread's own slots
    if (t < N1 && c < p.cin) {
#pragma unroll
      for (int m = 0; m < N2; ++m) tile[(size_t)(m + P * t) * NL + line] = v[m];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < H * TX; e += blockDim.x) {
      const int k = e / TX, xe = e - k * TX, kt = k % N1, km = k / N1;
      if (x0 + xe >= W) continue;
      cpx<R>* z = tile + (size_t)(km + P * kt) * NL + xe;
      const cpx<R>* mt = (const cpx<R>*)p.ktab + ray * p.ktab_ray_stride +
                         (((size_t)lam * H + k) * W + x0 + xe) * p.cout * p.cin;
      cpx<R> in[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (i < p.cin) in[i] = z[i * TX];
#pragma unroll
      for (int o = 0; o < 4; ++o) {
        if (o >= p.cout) break;
        cpx<R> a = mk<R>((R)0, (R)0);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (i < p.cin) a = cfma(mt[o * p.cin + i], in[i], a);
        z[o * TX] = a * sc;
      }
    }
    __syncthreads();
    if (t < N1 && c < p.cout) {
#pragma unroll
      for (int m = 0; m < N2; ++m) v[m] = tile[(size_t)(m + P * t) * NL + line];
    }
  } else if (t < N1 && c < p.cin) {
    if (D || p.kop == KOP_DIAG) {
      if (in_x) {
        const cpx<R>* ek = (const cpx<R>*)p.ktab + (((size_t)lam * W + kx) * H + t) * 2 +
                           ((((c & 1) == 0) || p.cin == 2) ? 0 : 1);
#pragma unroll
        for (int m = 0; m < N2; ++m)
          if (BAND == 0 || m < KB || m >= N2 - KB) v[m] = v[m] * (ek[(size_t)m * N1 * 2] * sc);
      }
    } else {
#pragma unroll
      for (int m = 0; m < N2; ++m) v[m] = v[m] * sc;
    }
  }
  for (int jj = 0; jj < p.ny; ++jj) {
    const int j = p.j_only >= 0 ? p.j_only : jj;
    cpx<R>* udst = U + ((size_t)jj * g.NI * p.cout + (size_t)img * p.cout + c) * H * W + kx;
    if (t < N1 && c < p.cout) {
      const R* cyj = p.cy ? (const R*)p.cy + (((size_t)ray * p.cy_rows + j) * g.nlam + lam) * H + t : nullptr;
      cpx<R> w[N2];
#pragma unroll
      for (int m = 0; m < N2; ++m) {
        if (BAND == 0 || m < KB || m >= N2 - KB)
          w[m] = cyj ? v[m] * cyj[N1 * m] : v[m];
        else
          w[m] = mk<R>((R)0, (R)0);
      }
      if (D || p.inverse_out) {
        RegDFTs<R, N2, true, MASK>::run(w);
        tile[(size_t)P * t * NL + line] = w[0];
#pragma unroll
        for (int k = 1; k < N2; ++k) {
          cpx<R> f = tw[k * N1 + t];
          f.im = -f.im;
          tile[(size_t)(k + P * t) * NL + line] = w[k] * f;
        }
      } else if (in_x) {
        cpx<R>* o = udst + (size_t)t * W;
#pragma unroll
        for (int m = 0; m < N2; ++m) {
          *o = w[m];
          o += N1 * W;
        }
      }
    }
    if (!D && !p.inverse_out) continue;
    __syncthreads();
    if (t < N2 && c < p.cout) {
      cpx<R> u[N1];
#pragma unroll
      for (int m = 0; m < N1; ++m) u[m] = tile[(size_t)(t + P * m) * NL + line];
      RegDFTg<R, N1, true>::run(u);
      if (in_x) {
        cpx<R>* o = udst + (size_t)t * W;
#pragma unroll
        for (int m = 0; m < N1; ++m) {
          *o = u[m];
          o += N2 * W;
        }
      }
    }
    __syncthreads();  // the exchange is read before the next window row writes it
  }
}

// ---------------------------------------------------------------------------
// launch glue: one function per side, defined by DTMM_REG_DEFINE in the
// dtmm_reg_*.cu units.  Geometry (grid, threads, shared bytes) comes from the
// engine; a variant that is not instantiated returns cudaErrorNotSupported.
// ---------------------------------------------------------------------------
struct RegLaunch {
  dim3 grid;
  int threads;
  size_t smem;
  cudaStream_t st;
  bool pdl = false;  // programmatic dependency on the previous kernel (row and column passes)
};

// row variants: every (C, REAL) for power-of-two sides, real records for the others
__host__ __device__ constexpr bool reg_row_variant(int n, bool real) { return reg_lanes(n) > 0 && (real || is_pow2(n)); }

template <int N1, int N2, int C, bool REAL, int BAND = 0, int XR = 0>
cudaError_t row_reg_variant(const RegLaunch& L, const RowParams& p, const Grid& g, const void* U, void* X) {
  auto kern = k_layer_row_reg<float, C, REAL, N1, N2, BAND, XR>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.smem);
  if (e != cudaSuccess) return e;
  return launch_with(L.pdl, kern, L.grid, L.threads, L.smem, L.st, p, g, (const cpx<float>*)U, (cpx<float>*)X);
}

// real records with a band variant b (row_band_pick), every (C, REAL) dense
// (p.xr: the variant, RowParams)
template <int N1, int N2, int C>
cudaError_t row_reg_real(int band, const RegLaunch& L, const RowParams& p, const Grid& g, const void* U, void* X) {
  if constexpr (xr_pixels(N1 * N2) > 0) {
    constexpr int XR = xr_pixels(N1 * N2);
    if (p.xr > 0) {
      if (band == 1) return row_reg_variant<N1, N2, C, true, 1, XR>(L, p, g, U, X);
      if (band == 2) return row_reg_variant<N1, N2, C, true, 2, XR>(L, p, g, U, X);
      return row_reg_variant<N1, N2, C, true, 0, XR>(L, p, g, U, X);
    }
  }
  if (p.xr < 0) {
    if constexpr (row_band_ok(N2, 1))
      if (band == 1) return row_reg_variant<N1, N2, C, true, 1, -1>(L, p, g, U, X);
    if constexpr (row_band_ok(N2, 2))
      if (band == 2) return row_reg_variant<N1, N2, C, true, 2, -1>(L, p, g, U, X);
    return row_reg_variant<N1, N2, C, true, 0, -1>(L, p, g, U, X);
  }
  if constexpr (row_band_ok(N2, 1))
    if (band == 1) return row_reg_variant<N1, N2, C, true, 1>(L, p, g, U, X);
  if constexpr (row_band_ok(N2, 2))
    if (band == 2) return row_reg_variant<N1, N2, C, true, 2>(L, p, g, U, X);
  return row_reg_variant<N1, N2, C, true, 0>(L, p, g, U, X);
}

template <int N1, int N2>
cudaError_t row_reg_launch(int C, bool real, int band, const RegLaunch& L, const RowParams& p, const Grid& g,
                           const void* U, void* X) {
  constexpr int N = N1 * N2;
  if (C == 4 && real) return row_reg_real<N1, N2, 4>(band, L, p, g, U, X);
  if (C == 2 && real) return row_reg_real<N1, N2, 2>(band, L, p, g, U, X);
  if constexpr (is_pow2(N)) {
    if (C == 4) return row_reg_variant<N1, N2, 4, false>(L, p, g, U, X);
    if (C == 2) return row_reg_variant<N1, N2, 2, false>(L, p, g, U, X);
  }
  return cudaErrorNotSupported;
}

template <int N, int BAND>
cudaError_t col_reg_variant(const RegLaunch& L, const ColParams& p, const Grid& g, const void* in, void* out) {
  auto kern = k_layer_col_reg<float, N, BAND>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.smem);
  if (e != cudaSuccess) return e;
  return launch_with(L.pdl, kern, L.grid, L.threads, L.smem, L.st, p, g, (const cpx<float>*)in, (cpx<float>*)out);
}

// band variants (col_band_pick of the H axis) for the diagonal operator between
// a forward and an inverse transform; the caller passes band 0 otherwise
template <int N>
cudaError_t col_reg_launch(int band, const RegLaunch& L, const ColParams& p, const Grid& g, const void* in, void* out) {
  constexpr int n2 = N / col_n1(N);
  if constexpr (row_band_ok(n2, 1))
    if (band == 1) return col_reg_variant<N, 1>(L, p, g, in, out);
  if constexpr (row_band_ok(n2, 2))
    if (band == 2) return col_reg_variant<N, 2>(L, p, g, in, out);
  return col_reg_variant<N, 0>(L, p, g, in, out);
}

template <int N1, int N2>
cudaError_t fft_rows_reg_launch(bool inv, const RegLaunch& L, const void* src, void* dst, int nlines, const void* tw,
                                float scale) {
  auto kern = inv ? k_fft_rows_reg<float, N1, N2, true> : k_fft_rows_reg<float, N1, N2, false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.smem);
  if (e != cudaSuccess) return e;
  kern<<<L.grid, L.threads, L.smem, L.st>>>((const cpx<float>*)src, (cpx<float>*)dst, nlines,
                                             (const cpx<float>*)tw, scale);
  return cudaGetLastError();
}

#define DTMM_REG_SIDES(X) \
  X(64) X(80) X(96) X(112) X(128) X(144) X(160) X(192) X(224) X(240) X(256) X(288) X(320) X(336) X(384) X(400) \
  X(432) X(448) X(480) X(512) X(1024)

#define DTMM_REG_DECLARE(N)                                                                                      \
  cudaError_t row_reg_##N(int C, bool real, int band, const RegLaunch& L, const RowParams& p, const Grid& g,     \
                          const void* U, void* X);                                                             \
  cudaError_t col_reg_##N(int band, const RegLaunch& L, const ColParams& p, const Grid& g, const void* in,       \
                          void* out);                                                                          \
  cudaError_t fft_rows_reg_##N(bool inv, const RegLaunch& L, const void* src, void* dst, int nlines, const void* tw, \
                               float scale);

#define DTMM_REG_DEFINE(N)                                                                                       \
  cudaError_t row_reg_##N(int C, bool real, int band, const RegLaunch& L, const RowParams& p, const Grid& g,     \
                          const void* U, void* X) {                                                            \
    return row_reg_launch<reg_lanes(N), N / reg_lanes(N)>(C, real, band, L, p, g, U, X);                       \
  }                                                                                                            \
  cudaError_t col_reg_##N(int band, const RegLaunch& L, const ColParams& p, const Grid& g, const void* in,       \
                          void* out) {                                                                         \
    return col_reg_launch<N>(band, L, p, g, in, out);                             \
  }                                                                                                            \
  cudaError_t fft_rows_reg_##N(bool inv, const RegLaunch& L, const void* src, void* dst, int nlines, const void* tw, \
                               float scale) {                                                                  \
    return fft_rows_reg_launch<reg_lanes(N), N / reg_lanes(N)>(inv, L, src, dst, nlines, tw, scale);           \
  }

DTMM_REG_SIDES(DTMM_REG_DECLARE)

// dispatch on the side (cudaErrorNotSupported for a side without a transform)
inline cudaError_t row_reg_dispatch(int n, int C, bool real, int band, const RegLaunch& L, const RowParams& p,
                                    const Grid& g, const void* U, void* X) {
  switch (n) {
#define DTMM_REG_ROW_CASE(N) \
  case N: return row_reg_##N(C, real, band, L, p, g, U, X);
    DTMM_REG_SIDES(DTMM_REG_ROW_CASE)
#undef DTMM_REG_ROW_CASE
    default: return cudaErrorNotSupported;
  }
}

inline cudaError_t col_reg_dispatch(int n, int band, const RegLaunch& L, const ColParams& p, const Grid& g,
                                    const void* in, void* out) {
  switch (n) {
#define DTMM_REG_COL_CASE(N) \
  case N: return col_reg_##N(band, L, p, g, in, out);
    DTMM_REG_SIDES(DTMM_REG_COL_CASE)
#undef DTMM_REG_COL_CASE
    default: return cudaErrorNotSupported;
  }
}

inline cudaError_t fft_rows_reg_dispatch(int n, bool inv, const RegLaunch& L, const void* src, void* dst, int nlines,
                                         const void* tw, float scale) {
  switch (n) {
#define DTMM_REG_FFT_CASE(N) \
  case N: return fft_rows_reg_##N(inv, L, src, dst, nlines, tw, scale);
    DTMM_REG_SIDES(DTMM_REG_FFT_CASE)
#undef DTMM_REG_FFT_CASE
    default: return cudaErrorNotSupported;
  }
}

}  // namespace dtmm
