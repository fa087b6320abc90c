// Spectral kernels of the Poisson solve (potential.py:7-29 of the reference):
//
//   x_r2c    real rows -> half-spectrum rows   (R2C along x, via a length-n/2 complex FFT)
//   y_pass   complex FFT along y, forward or inverse
//   z_green  forward FFT along z, multiply by the Green function, inverse FFT along z
//   x_c2r    half-spectrum rows -> real rows   (C2R along x)
//
// Every kernel is specialised for one grid size N and is persistent over a work list
// that may span many simulations of that size: a CTA finds its simulation from the
// work prefix.  Each N is instantiated in its own translation unit (pm_spectral_n.cu
// compiled with -DPM_N=<N>), so that register allocation is per size and the build
// runs in parallel.
#pragma once
#include <cudaTypedefs.h>

#include "pm_common.cuh"
#include "pm_deposit.cuh"
#include "pm_fft.cuh"
#include "pm_tma.cuh"

namespace pm {

constexpr int SP_NT = 256;          // threads per CTA of every spectral kernel
constexpr int SP_ELEMS = 8192;      // complex elements held per CTA (64 KB)

// ---------------------------------------------------------------------------------
// Per-n configuration
// ---------------------------------------------------------------------------------
__host__ __device__ constexpr int cx_rows(int n) {
  // rows of the x passes per CTA: ~SP_ELEMS complex, a multiple of 8, at most n*n
  return (SP_ELEMS / (n / 2)) / 8 * 8 > n * n ? n * n : (SP_ELEMS / (n / 2)) / 8 * 8;
}
// Line passes: units of bundles of 16 columns (8 on 384 and above, where a bundle is 24 KB and more),
// one unit to a TMA stage of a persistent CTA.  Thin CTAs, two to four to an SM with one or two
// bundles to a unit, cover one another's barriers and copies, and give a small grid enough units
// for 152 SMs: with 64 KB stages a 64^3 grid had 24 (y 5.2 us -> 3.3, z 7.3 -> 4.2); 128: y 8.2 ->
// 5.8; 192 (512 threads on two bundles -> 256 on one, three CTAs): a Poisson solve 91 -> 82 us;
// 256 the same with two CTAs: 40 resident steps 10.74 -> 10.56 ms.  768 and 1024 keep one CTA with
// 48 / 64 KB stages.  (8-wide bundles on 256 and 192: z 20% and 4% slower.)
__host__ __device__ constexpr bool line_small(int n) { return n == 512 || n == 384; }
__host__ __device__ constexpr bool line_thin(int n) { return n >= 32 && n <= 256; }
// columns of a line-pass bundle
__host__ __device__ constexpr int cline_width(int n) { return n >= 512 || line_small(n) ? 8 : 16; }
// bundles per unit (per TMA stage)
__host__ __device__ constexpr int cline_bpc(int n) {
  if (line_thin(n)) return n >= 128 ? 1 : 2;
  return line_small(n) ? SP_ELEMS / 2 / (n * 8)
                       : (SP_ELEMS / (n * cline_width(n)) < 1 ? 1 : SP_ELEMS / (n * cline_width(n)));
}
__host__ __device__ constexpr int chalf(int n) { return n / 2 + 1; }
__host__ __device__ constexpr int cbundles_per_plane(int n) {
  return (chalf(n) + cline_width(n) - 1) / cline_width(n);
}

__host__ __device__ constexpr int cpitch(int n) { return (chalf(n) + 15) / 16 * 16; }
// Line passes that stream through a TMA ring: boxes of at most 256 rows tiling n.
__host__ __device__ constexpr int line_box_rows(int n) { return n <= 256 ? n : (n % 256 == 0 ? 256 : n / 2); }
__host__ __device__ constexpr bool tma_lines(int n) { return n >= 32 && line_box_rows(n) <= 256; }
// Threads of a line-pass CTA and CTAs per SM.  (768, transformed line by
// line, runs 1024 threads.)
__host__ __device__ constexpr int line_nt(int n) {
  return line_small(n) || n == 96 || n == 192 || n == 256 ? 256 : (line_thin(n) ? 128 : (n == 768 ? 1024 : 512));
}
__host__ __device__ constexpr int line_ctas_per_sm(int n) {
  return line_small(n) || n == 256 ? 2 : (n == 96 || n == 192 ? 3 : (line_thin(n) ? 4 : 1));
}
// The z pass with the Green function (the turn) has plans of its own (pm_fft.cuh: TurnPlan), and on
// the larger grids its own threads, CTAs per SM and ring stages, as thin as every thread still
// has a transform of the larger radix to do.  Measured in us a launch:
//   512  16 x 32, 128 threads, 3 CTAs of 2 stages 256 (8 x 8 x 8 on pairs of lines, 2 x 256 threads,
//        288; 2 CTAs of 3 stages 284; 256 threads, half idle in the radix-32 pass, 299)
//   384  24 x 16, 128 threads, 4 CTAs of 2 stages 113 (256 threads 190, 3 CTAs of 3 stages 117)
//   768  24 x 32, 256 threads, 2 CTAs of 2 stages 1.05 ms (one CTA of 3 stages 1.22, 2 of one stage
//        1.20; 3, 4, 8, 8 with 1024 threads 2.9)
//   1024 32 x 32, 256 threads 2.36 ms (16, 8, 8 with 512 threads 2.67; 2 CTAs of one stage the same)
// Bundles of 4 columns on 768 and 1024 (32-byte rows for the copies) take twice the time.
__host__ __device__ constexpr int turn_stages(int n) { return n == 512 || n == 384 || n == 768 ? 2 : 3; }
__host__ __device__ constexpr int turn_nt(int n) {
  return n == 512 || n == 384 ? 128 : (n >= 768 ? 256 : line_nt(n));
}
__host__ __device__ constexpr int turn_ctas_per_sm(int n) {
  return n == 384 ? 4 : (n == 512 ? 3 : (n == 768 ? 2 : line_ctas_per_sm(n)));
}
constexpr int TMA_STAGES = 3;
__host__ __device__ constexpr size_t tma_stage_bytes(int n) {
  return (size_t)n * cline_width(n) * cline_bpc(n) * sizeof(float2);
}
__host__ __device__ constexpr size_t tma_smem_bytes(int n, bool turn) {
  return (turn ? turn_stages(n) * tma_stage_bytes(n) : TMA_STAGES * tma_stage_bytes(n)) + 64;
}
__host__ __device__ constexpr bool line_turn(int mode) { return mode == 2 || mode == 3 || mode == 6; }

// x passes with the row transform in registers (n >= 32): a row of M = n/2 complex points is held
// by T lanes of a warp and transformed in passes of radix A, (B,) C, M = A C or A B C, through an
// exchange buffer of the row that only its warp synchronises on
// (n: radices, T) -- 32: 4x4, 4; 48: 4x6, 2; 64: 8x4, 4; 96: 4x12, 4; 128: 8x8, 8; 192: 8x12, 4;
// 256: 16x8, 8; 384: 8x24, 8; 512: 16x16, 16; 768: 8x8x6, 16; 1024: 8x8x8, 32, inverse 16x32, 16
// (the radix-3 rows with the smaller factor first: x C2R per 134M cells 96: 0.119 -> 0.115,
// 192: 0.315 -> 0.257, 384: 0.269 -> 0.256 ms.  1024 in two passes holds 32 points, 64 registers, a
// lane: the C2R pass, which is alone in its kernel, 1.90 -> 1.39 ms, but the fused deposit, left with
// two CTAs per SM, 3.35 -> 3.67; the plain R2C keeps the fused one's plan, and so its bits.  768 in
// two passes would hold 48 points.)
__host__ __device__ constexpr bool xrow_ok(int n) { return n >= 32; }
__host__ __device__ constexpr int xrow_A(int n, bool inv) {
  if (n == 1024) return inv ? 16 : 8;
  return n >= 768 ? 8 : (n % 3 == 0 ? (n <= 96 ? 4 : 8) : (n >= 256 ? 16 : (n == 32 ? 4 : 8)));
}
__host__ __device__ constexpr int xrow_B(int n, bool inv) { return n == 768 || (n == 1024 && !inv) ? 8 : 1; }
__host__ __device__ constexpr int xrow_C(int n, bool inv) { return n / 2 / (xrow_A(n, inv) * xrow_B(n, inv)); }
__host__ __device__ constexpr int xrow_T(int n, bool inv) {
  return n == 1024 && !inv ? 32 : (n >= 768 || n == 512 ? 16 : (n == 48 ? 2 : (n % 3 == 0 && n != 384 ? 4 : (n <= 64 ? 4 : 8))));
}
__host__ __device__ constexpr int xrow_rows_per_warp(int n, bool inv) { return 32 / xrow_T(n, inv); }
// rows of a work unit, which a warp takes: one unit for both directions
__host__ __device__ constexpr int xrow_unit_rows(int n) {
  return xrow_rows_per_warp(n, true) > xrow_rows_per_warp(n, false) ? xrow_rows_per_warp(n, true)
                                                                    : xrow_rows_per_warp(n, false);
}
// complex elements of a row's exchange buffer: C rows of A (padded) in two passes; in three,
// the row with one element of padding after every A
__host__ __device__ constexpr int xrow_exchange(int n, bool inv) {
  return xrow_B(n, inv) == 1 ? xrow_C(n, inv) * (xrow_A(n, inv) + 1) : n / 2 + n / 2 / xrow_A(n, inv);
}
// threads of a row-transform CTA: up to 8 warps, their exchange buffers within 40 KB of
// static shared memory
__host__ __device__ constexpr int xrow_warp_bytes(int n, bool inv) { return xrow_rows_per_warp(n, inv) * xrow_exchange(n, inv) * 8; }
__host__ __device__ constexpr int xrow_nt(int n, bool inv) {
  const int warps = 40960 / xrow_warp_bytes(n, inv);
  return 32 * (warps < 8 ? (warps < 1 ? 1 : warps) : 8);
}

__host__ __device__ constexpr size_t x_smem_bytes(int n) {
  return (size_t)(n / 2 + 1) * (cx_rows(n) + 1) * sizeof(float2);
}
__host__ __device__ constexpr size_t line_smem_bytes(int n) {
  return (size_t)n * cline_width(n) * cline_bpc(n) * sizeof(float2);
}
// ---------------------------------------------------------------------------------
// x_r2c
// ---------------------------------------------------------------------------------
template <int N>
__device__ __forceinline__ void x_r2c_body(const Sim& S, int unit, float2* s) {
  constexpr int M = N / 2, NR = cx_rows(N), LS = NR + 1;
  constexpr int NT = SP_NT;
  const long long nrows = (long long)N * N;
  const long long row0 = (long long)unit * NR;
  const float2* __restrict__ src = reinterpret_cast<const float2*>(S.rho);
  // load NR rows of M complex (pairs of reals), transposed into s[j][r]
  constexpr int NU = NR * M;
  constexpr int KU = (NU + NT - 1) / NT;
  float2 buf[KU];
#pragma unroll
  for (int k = 0; k < KU; ++k) {
    const int u = threadIdx.x + k * NT;
    const int r = u / M, j = u % M;
    buf[k] = make_float2(0.f, 0.f);
    if ((NU % NT == 0 || u < NU) && row0 + r < nrows) buf[k] = __ldg(&src[(row0 + r) * M + j]);
  }
#pragma unroll
  for (int k = 0; k < KU; ++k) {
    const int u = threadIdx.x + k * NT;
    if (NU % NT == 0 || u < NU) s[(u % M) * LS + u / M] = buf[k];
  }
  __syncthreads();
  fft_lines<M, NR, LS, NT, false>(s, S.tw, 2);
  // untangle: X[k] = E[k] + W^k O[k], k = 0..M
  float2* __restrict__ dst = S.spec;
  const int P = S.pitch;
  for (int u = threadIdx.x; u < NR * (M + 1); u += NT) {
    const int r = u / (M + 1), k = u % (M + 1);
    if (row0 + r >= nrows) continue;
    const float2 zk = s[(k == M ? 0 : k) * LS + r];
    const float2 zc = conjf2(s[(k == 0 ? 0 : M - k) * LS + r]);
    const float2 e = cscale(cadd(zk, zc), 0.5f);
    const float2 o = cscale(mul_mi<false>(csub(zk, zc)), 0.5f);
    const float2 w = __ldg(&S.tw[k]);
    dst[(row0 + r) * P + k] = cadd(e, cmul(w, o));
  }
}

template <int N>
__global__ void __launch_bounds__(SP_NT) k_x_r2c(const Sim* __restrict__ sims, Work w) {
  chain_begin();
  extern __shared__ float4 smem_f4[];
  float2* s = reinterpret_cast<float2*>(smem_f4);
  for (int unit = blockIdx.x; unit < w.total; unit += gridDim.x) {
    const int si = locate_sim(w, unit);
    x_r2c_body<N>(sims[si], unit - __ldg(&w.prefix[si]), s);
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------
// x_c2r
// ---------------------------------------------------------------------------------
template <int N>
__device__ __forceinline__ void x_c2r_body(const Sim& S, int unit, float2* s) {
  constexpr int M = N / 2, NR = cx_rows(N), LS = NR + 1;
  constexpr int NT = SP_NT;
  const long long nrows = (long long)N * N;
  const long long row0 = (long long)unit * NR;
  const float2* __restrict__ src = S.spec;
  const int P = S.pitch;
  constexpr int NU = NR * (M + 1);
  constexpr int KU = (NU + NT - 1) / NT;
  float2 buf[KU];
#pragma unroll
  for (int k = 0; k < KU; ++k) {
    const int u = threadIdx.x + k * NT;
    const int r = u / (M + 1), j = u % (M + 1);
    buf[k] = make_float2(0.f, 0.f);
    if ((NU % NT == 0 || u < NU) && row0 + r < nrows) buf[k] = __ldg(&src[(row0 + r) * P + j]);
  }
#pragma unroll
  for (int k = 0; k < KU; ++k) {
    const int u = threadIdx.x + k * NT;
    if (NU % NT == 0 || u < NU) s[(u % (M + 1)) * LS + u / (M + 1)] = buf[k];
  }
  __syncthreads();
  // tangle: Z[k] = (X[k] + X*[M-k]) + i W^-k (X[k] - X*[M-k]), handled in pairs (k, M-k)
  for (int u = threadIdx.x; u < NR * (M / 2 + 1); u += NT) {
    const int r = u / (M / 2 + 1), k = u % (M / 2 + 1);
    const float2 xk = s[k * LS + r];
    const float2 xm = s[(M - k) * LS + r];
    const float2 a = cadd(xk, conjf2(xm));
    const float2 b = csub(xk, conjf2(xm));
    const float2 w = __ldg(&S.tw[k]);
    const float2 t = cmul(conjf2(w), b);
    const float2 zk = make_float2(a.x - t.y, a.y + t.x);  // a + i t
    s[k * LS + r] = zk;
    if (k != 0 && 2 * k != M) {
      const float2 t2 = cmul(w, conjf2(b));
      s[(M - k) * LS + r] = make_float2(a.x - t2.y, -a.y + t2.x);  // conj(a) + i t2
    }
  }
  __syncthreads();
  fft_lines<M, NR, LS, NT, true>(s, S.tw, 2);
  float2* __restrict__ dst = reinterpret_cast<float2*>(S.phi);
  for (int u = threadIdx.x; u < NR * M; u += NT) {
    const int r = u / M, j = u % M;
    if (row0 + r < nrows) dst[(row0 + r) * M + j] = s[j * LS + r];
  }
}

template <int N>
__global__ void __launch_bounds__(SP_NT) k_x_c2r(const Sim* __restrict__ sims, Work w) {
  chain_begin();
  extern __shared__ float4 smem_f4[];
  float2* s = reinterpret_cast<float2*>(smem_f4);
  for (int unit = blockIdx.x; unit < w.total; unit += gridDim.x) {
    const int si = locate_sim(w, unit);
    x_c2r_body<N>(sims[si], unit - __ldg(&w.prefix[si]), s);
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------
// line passes (y, and z with the Green multiply)
// ---------------------------------------------------------------------------------
// Bundles are BW consecutive kx of one plane; plane = z for the y pass, y for the z pass.
template <int N, bool ZAXIS>
__device__ __forceinline__ void load_bundles(const Sim& S, int unit, float2* s) {
  constexpr int BW = cline_width(N), BPC = cline_bpc(N), NL = BW * BPC, LS = NL;
  constexpr int W = chalf(N), NBP = cbundles_per_plane(N);
  constexpr int U = BW / 2;              // float4 units per bundle row
  constexpr int NU = BPC * N * U;
  constexpr int NT = SP_NT;
  constexpr int KU = (NU + NT - 1) / NT;
  const long long P = S.pitch;
  const int nb = N * NBP;
  const float2* __restrict__ src = S.spec;
  float4 buf[KU];
#pragma unroll
  for (int k = 0; k < KU; ++k) {
    const int u = threadIdx.x + k * NT;
    const int i = u / (N * U), rem = u % (N * U);
    const int j = rem / U, c = (rem % U) * 2;
    const int b = unit * BPC + i;
    buf[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if ((NU % NT == 0 || u < NU) && b < nb) {
      const int plane = b / NBP, kx0 = (b % NBP) * BW;
      if (kx0 + c < W) {
        buf[k] = __ldg(reinterpret_cast<const float4*>(src + (ZAXIS ? spec_row(N, plane, j) : spec_row(N, j, plane)) * P + kx0 + c));
        if (kx0 + c + 1 >= W) { buf[k].z = 0.f; buf[k].w = 0.f; }
      }
    }
  }
#pragma unroll
  for (int k = 0; k < KU; ++k) {
    const int u = threadIdx.x + k * NT;
    if (NU % NT == 0 || u < NU) {
      const int i = u / (N * U), rem = u % (N * U);
      const int j = rem / U, c = (rem % U) * 2;
      *reinterpret_cast<float4*>(&s[j * LS + i * BW + c]) = buf[k];
    }
  }
}

template <int N, bool ZAXIS>
__device__ __forceinline__ void store_bundles(const Sim& S, int unit, const float2* s) {
  constexpr int BW = cline_width(N), BPC = cline_bpc(N), NL = BW * BPC, LS = NL;
  constexpr int W = chalf(N), NBP = cbundles_per_plane(N);
  constexpr int U = BW / 2;
  constexpr int NU = BPC * N * U;
  constexpr int NT = SP_NT;
  const long long P = S.pitch;
  const int nb = N * NBP;
  float2* __restrict__ dst = S.spec;
  for (int u = threadIdx.x; u < NU; u += NT) {
    const int i = u / (N * U), rem = u % (N * U);
    const int j = rem / U, c = (rem % U) * 2;
    const int b = unit * BPC + i;
    if (b >= nb) continue;
    const int plane = b / NBP, kx0 = (b % NBP) * BW;
    if (kx0 + c < W)
      *reinterpret_cast<float4*>(dst + (ZAXIS ? spec_row(N, plane, j) : spec_row(N, j, plane)) * P + kx0 + c) =
          *reinterpret_cast<const float4*>(&s[j * LS + i * BW + c]);
  }
}

// Plain transform of the bundles of one unit along y (ZAXIS false) or z.
template <int N, bool ZAXIS, bool INV>
__device__ __forceinline__ void line_body(const Sim& S, int unit, float2* s) {
  constexpr int NL = cline_width(N) * cline_bpc(N);
  load_bundles<N, ZAXIS>(S, unit, s);
  __syncthreads();
  fft_lines<N, NL, NL, SP_NT, INV>(s, S.tw, 1);
  store_bundles<N, ZAXIS>(S, unit, s);
}

template <int N, bool ZAXIS, bool INV>
__global__ void __launch_bounds__(SP_NT) k_line_pass(const Sim* __restrict__ sims, Work w) {
  chain_begin();
  extern __shared__ float4 smem_f4[];
  float2* s = reinterpret_cast<float2*>(smem_f4);
  for (int unit = blockIdx.x; unit < w.total; unit += gridDim.x) {
    const int si = locate_sim(w, unit);
    line_body<N, ZAXIS, INV>(sims[si], unit - __ldg(&w.prefix[si]), s);
    __syncthreads();
  }
}

// Green function of potential.py:15 / fourier_utils.py:15-16 (k = 0 -> 0), including
// the 1/n^3 of the unnormalised inverse transforms (folded into S.green).
// GRAD: the spectral gradient of axis S.grad_axis - 1 as well (times -i sin(k_d)).
template <int N, bool TABLE, bool GRAD>
__device__ __forceinline__ void z_body(const Sim& S, int unit, float2* s) {
  constexpr int BW = cline_width(N), BPC = cline_bpc(N), NL = BW * BPC;
  constexpr int NBP = cbundles_per_plane(N), W = chalf(N);
  load_bundles<N, true>(S, unit, s);
  __syncthreads();
  fft_lines<N, NL, NL, SP_NT, false>(s, S.tw, 1);
  const float g0 = S.green;
  const float* __restrict__ s2 = S.s2;
  for (int e = threadIdx.x; e < N * NL; e += SP_NT) {
    const int kz = e / NL, line = e % NL;
    const int i = line / BW, c = line % BW;
    const int b = unit * BPC + i;
    const int ky = b / NBP, kx = (b % NBP) * BW + c;
    float g = 0.f;
    if (kx < W && ky < N) {
      if (TABLE) {
        g = g0 * __ldg(&S.fgrid[((long long)kz * N + ky) * N + kx]);
      } else if ((kx | ky | kz) != 0) {
        const float den = __ldg(&s2[kx]) + __ldg(&s2[ky]) + __ldg(&s2[kz]);
        g = __fdividef(g0, den);
      }
    }
    const float2 v = s[e];
    if (GRAD) {  // times -i sin(k_d): the spectral central difference along axis d
      const float sg =
          kx < W && ky < N ? g * __ldg(&S.sn[S.grad_axis == 1 ? kx : (S.grad_axis == 2 ? ky : kz)]) : 0.f;
      s[e] = make_float2(sg * v.y, -sg * v.x);
    } else {
      s[e] = make_float2(v.x * g, v.y * g);
    }
  }
  __syncthreads();
  fft_lines<N, NL, NL, SP_NT, true>(s, S.tw, 1);
  store_bundles<N, true>(S, unit, s);
}

template <int N, bool TABLE, bool GRAD = false>
__global__ void __launch_bounds__(SP_NT) k_z_green(const Sim* __restrict__ sims, Work w) {
  chain_begin();
  extern __shared__ float4 smem_f4[];
  float2* s = reinterpret_cast<float2*>(smem_f4);
  for (int unit = blockIdx.x; unit < w.total; unit += gridDim.x) {
    const int si = locate_sim(w, unit);
    z_body<N, TABLE, GRAD>(sims[si], unit - __ldg(&w.prefix[si]), s);
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------
// TMA-streamed line pass (y forward / y inverse / z Green) over one or many simulations.
//
// Persistent CTA with a shared-memory ring of STAGES stages (3; the turn on 384, 512 and 768: 2).  A unit is BPC bundles of one
// simulation; a bundle is BW consecutive kx of one plane, loaded as N / BOX TMA boxes of
// {2 BW floats, BOX rows} with the simulation's tensor map (maps[2 s] for y, maps[2 s + 1]
// for z, in device memory).  One elected thread issues the loads of unit i+1 while all
// threads transform unit i; finished bundles leave by TMA bulk store, and a stage is
// refilled only once the store issued from it STAGES - 1 iterations earlier has finished
// reading it.  Stages hold the bundles blocked (Blocked layout of pm_fft.cuh).
// ---------------------------------------------------------------------------------
// Green function of potential.py:15 / fourier_utils.py:15-16 (k = 0 -> 0; the 1/n^3 of the
// unnormalised inverse transforms is folded into g0) for element kz of line `line` of a unit
// of the z pass whose first bundle is b0.
template <int N, bool TABLE, bool GRAD = false>
struct GreenEpi {
  float g0;
  const float* s2;
  const float* fgrid;
  int b0, cnt;
  const float* sn;  // GRAD, the spectral gradient of axis grad_axis - 1: times -i sin(k_d) as well
  int grad_axis;
  __device__ __forceinline__ float2 operator()(float2 v, int kz, int line) const {
    constexpr int BW = cline_width(N), NBP = cbundles_per_plane(N), W = chalf(N);
    const int i = line / BW, b = b0 + i;
    const int ky = b / NBP, kx = (b % NBP) * BW + line % BW;
    float g = 0.f;
    if (i < cnt && kx < W) {
      if (TABLE) g = g0 * __ldg(&fgrid[((long long)kz * N + ky) * N + kx]);
      else if ((kx | ky | kz) != 0) g = __fdividef(g0, __ldg(&s2[kx]) + __ldg(&s2[ky]) + __ldg(&s2[kz]));
    }
    if (GRAD) {
      const float sg = i < cnt && kx < W ? g * __ldg(&sn[grad_axis == 1 ? kx : (grad_axis == 2 ? ky : kz)]) : 0.f;
      return make_float2(sg * v.y, -sg * v.x);
    }
    return make_float2(v.x * g, v.y * g);
  }
};

// MODE 0: y forward, 1: y inverse, 2: z Green, 3: z Green (caller table), 4: z forward, 5: z inverse,
// 6: z Green times -i sin(k_d) (spectral gradient of axis S.grad_axis - 1)
template <int N, int MODE>
__global__ void __launch_bounds__(line_turn(MODE) ? turn_nt(N) : line_nt(N),
                                  line_turn(MODE) ? turn_ctas_per_sm(N) : line_ctas_per_sm(N))
    k_line_tma(const CUtensorMap* __restrict__ maps, const Sim* __restrict__ sims, Work w, int* err) {
  constexpr int STAGES = line_turn(MODE) ? turn_stages(N) : TMA_STAGES;
  constexpr int BW = cline_width(N), BPC = cline_bpc(N), NL = BW * BPC;
  constexpr int BOX = line_box_rows(N), NBOX = N / BOX;
  constexpr int NBP = cbundles_per_plane(N), W = chalf(N), NB = N * NBP;
  constexpr unsigned STAGE = (unsigned)tma_stage_bytes(N);
  constexpr unsigned BUNDLE = (unsigned)N * BW * sizeof(float2);
  constexpr bool ZAX = MODE >= 2;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  float2* stg0 = reinterpret_cast<float2*>(smem_raw);
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw + STAGES * STAGE);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 0; i < STAGES; ++i) mbar_init(&bar[i], 1);
    fence_mbar_init();
  }
  __syncthreads();
  chain_begin();
  auto stage_ptr = [&](int st) { return stg0 + (size_t)st * (STAGE / sizeof(float2)); };
  // unit -> (simulation, first bundle, bundles in the unit)
  auto unit_info = [&](int unit, int& si, int& b0, int& cnt) {
    si = locate_sim(w, unit);
    b0 = (unit - __ldg(&w.prefix[si])) * BPC;
    cnt = NB - b0 < BPC ? NB - b0 : BPC;
  };
  // (the map's axes: 2 kx, y in its block, z, block of y)
  auto coords = [&](int b, int box, int& c0, int& c1, int& c2, int& c3) {
    constexpr int YB = spec_block(N);
    const int plane = b / NBP, kx0 = (b % NBP) * BW, y = ZAX ? plane : box * BOX;
    c0 = 2 * kx0;
    c1 = y % YB;
    c2 = ZAX ? box * BOX : plane;
    c3 = y / YB;
  };
  auto issue_load = [&](int unit, int st) {
    int si, b0, cnt;
    unit_info(unit, si, b0, cnt);
    const CUtensorMap* tm = &maps[2 * si + (ZAX ? 1 : 0)];
    mbar_expect_tx(&bar[st], (unsigned)cnt * BUNDLE);
    for (int i = 0; i < cnt; ++i)
#pragma unroll
      for (int box = 0; box < NBOX; ++box) {
        int c0, c1, c2, c3;
        coords(b0 + i, box, c0, c1, c2, c3);
        tma_load_4d(stage_ptr(st) + (i * N + box * BOX) * BW, tm, c0, c1, c2, c3, &bar[st]);
      }
  };
  int unit = blockIdx.x;
  if (threadIdx.x == 0 && unit < w.total) issue_load(unit, 0);
  unsigned parity = 0;  // bit st: parity of the next phase of stage st
  for (int it = 0; unit < w.total; unit += gridDim.x, ++it) {
    const int st = it % STAGES;
    const int next = unit + gridDim.x;
    if (threadIdx.x == 0 && next < w.total) {
      bulk_wait_read<STAGES - 2>();  // the store that last read the stage is done
      issue_load(next, (it + 1) % STAGES);
    }
    const bool ok = mbar_wait(&bar[st], (parity >> st) & 1u);
    parity ^= 1u << st;
    if (__syncthreads_or(!ok)) {
      if (threadIdx.x == 0) set_error(err, ERR_TIMEOUT);
      break;
    }
    int si, b0, cnt;
    unit_info(unit, si, b0, cnt);
    const Sim& S = sims[si];
    float2* s = stage_ptr(st);
    if (MODE == 0 || MODE == 4) {
      fft_lines_blocked<N, NL, BW, line_nt(N), false>(s, S.tw, 1);
    } else if (MODE == 1 || MODE == 5) {
      fft_lines_blocked<N, NL, BW, line_nt(N), true>(s, S.tw, 1);
    } else {
      // forward z transform, the Green function, inverse z transform (meeting in registers)
      const GreenEpi<N, MODE == 3, MODE == 6> epi{S.green, S.s2, S.fgrid, b0, cnt, S.sn, S.grad_axis};
      fft_lines_blocked_turn<N, NL, BW, turn_nt(N)>(s, S.tw, 1, epi);
    }
    fence_proxy_async_smem();
    __syncthreads();
    if (threadIdx.x == 0) {
      const CUtensorMap* tm = &maps[2 * si + (ZAX ? 1 : 0)];
      for (int i = 0; i < cnt; ++i)
#pragma unroll
        for (int box = 0; box < NBOX; ++box) {
          int c0, c1, c2, c3;
          coords(b0 + i, box, c0, c1, c2, c3);
          tma_store_4d(tm, c0, c1, c2, c3, s + (i * N + box * BOX) * BW);
        }
      bulk_commit();
    }
  }
  if (threadIdx.x == 0) bulk_wait<0>();
}

// ---------------------------------------------------------------------------------
// x passes, row transform in registers (xrow_ok sizes).  T lanes of a warp own one row of M
// complex points.  Two passes, M = A C, j = C a + b, k = c + A d:
//   pass 1  lane t, b = t + T i: A-point DFT over a of z[C a + b], times w_M^(b c)
//   (shared-memory exchange inside the row, synchronised by the warp alone)
//   pass 2  lane t, c = t + T i: C-point DFT over b -> Z[c + A d]
// Three passes, M = A B C: Stockham passes of radix A, B, C on the row's exchange buffer, element
// e at e + e / A (pass 1 stores A e + r: without the padding all lanes would hit one bank).
// R2C: z[j] = x[2j] + i x[2j+1] read straight from the density rows, Z untangled into the
// half spectrum.  C2R: the spectrum row is tangled into pass 1, and z written as pairs of reals.
// Loads and stores of T lanes are consecutive (coalesced).  A work unit is the 32 / T rows of one
// warp (of the direction that takes more).
// ---------------------------------------------------------------------------------
// A row's passes; v holds z[(M / A) a + t + T i] on entry, o holds Z[t + T i + (M / C) d] on exit.
// rb: the row's exchange buffer.
// A-point and C-point DFTs of a lane
template <int N, bool INV> constexpr int xrow_NB1 = N / 2 / xrow_A(N, INV) / xrow_T(N, INV);
template <int N, bool INV> constexpr int xrow_NB2 = N / 2 / xrow_C(N, INV) / xrow_T(N, INV);

// The twiddles between a row's passes, in shared memory in the order in which the lanes use them.  Read
// from the table by their exponent, the lanes' words lie up to 15 apart -- 8 to 16 cache lines a
// load, a quarter to a half of the L1 wavefronts of the x passes.  From 256 cells a side (x C2R of
// 384^3 88 -> 77 us, 512^3 171 -> 167, 768^3 721 -> 643, 1024^3 1.38 -> 1.31 ms), in the fused deposit
// from 192 (256^3 59 -> 55 us, 512^3 400 -> 356, 768^3 1.60 -> 1.42 ms, 1024^3 3.33 -> 3.16; eight
// 192^3 204 -> 193 us); shorter rows have few lines to a load (192 x passes 15.4 -> 16.2).
__host__ __device__ constexpr bool xrow_table(int n, bool fused) { return n >= (fused ? 192 : 256); }
// j's of the third pass that are in the table (three CTAs of the fused deposit on 1024 leave 2.7 KB each)
__host__ __device__ constexpr int xrow_table_j(int n, bool inv) {
  return n == 1024 ? xrow_T(n, inv) : n / 2 / xrow_C(n, inv);
}
template <int N, bool INV, bool FUSED>
__host__ __device__ constexpr int xrow_table_size() {
  constexpr int M = N / 2, A = xrow_A(N, INV), B = xrow_B(N, INV), C = xrow_C(N, INV);
  return !xrow_table(N, FUSED) ? 1 : (B == 1 ? (A - 1) * (M / A) : (B - 1) * A + (C - 1) * xrow_table_j(N, INV));
}
// Filled by the CTA, which synchronises.  Two passes: w_M^(b c) at (c - 1) M / A + b; three:
// w_M^(r k M / (A B)) at (r - 1) A + k, then w_M^(r j) at (r - 1) J + j, j < J = xrow_table_j.
template <int N, bool INV, bool FUSED, int NT>
__device__ __forceinline__ void xrow_table_fill(float2* wt, const float2* __restrict__ tw) {
  constexpr int M = N / 2, A = xrow_A(N, INV), B = xrow_B(N, INV), C = xrow_C(N, INV);
  constexpr int J = xrow_table_j(N, INV);
  if (!xrow_table(N, FUSED)) return;
  for (int e = threadIdx.x; e < xrow_table_size<N, INV, FUSED>(); e += NT) {
    int m;
    if (B == 1) m = (e / (M / A) + 1) * (e % (M / A));
    else if (e < (B - 1) * A) m = (e / A + 1) * (e % A) * (M / (A * B));
    else m = ((e - (B - 1) * A) / J + 1) * ((e - (B - 1) * A) % J);
    float2 w = __ldg(&tw[m % M * 2]);
    if (INV) w.y = -w.y;
    wt[e] = w;
  }
}

template <int N, bool INV, bool FUSED>
__device__ __forceinline__ void xrow_transform(float2 (&v)[xrow_NB1<N, INV>][xrow_A(N, INV)],
                                               float2 (&o)[xrow_NB2<N, INV>][xrow_C(N, INV)], float2* rb, int t,
                                               const float2* __restrict__ tw, const float2* wt) {
  constexpr int M = N / 2, A = xrow_A(N, INV), B = xrow_B(N, INV), C = xrow_C(N, INV), T = xrow_T(N, INV);
  constexpr int NB1 = xrow_NB1<N, INV>, NB2 = xrow_NB2<N, INV>;
  // w_M^m, at place e of the table (if it is there)
  auto twiddle = [&](int m, int e, bool in = true) {
    if (xrow_table(N, FUSED) && in) return wt[e];
    float2 w = __ldg(&tw[m * 2]);
    if (INV) w.y = -w.y;
    return w;
  };
  if constexpr (B == 1) {
#pragma unroll
    for (int i = 0; i < NB1; ++i) {
      const int b = t + T * i;
      DFT<A, INV>::run(v[i]);
#pragma unroll
      for (int c = 1; c < A; ++c) v[i][c] = cmul(v[i][c], twiddle((b * c) % M, (c - 1) * (M / A) + b));
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < NB1; ++i)
#pragma unroll
      for (int c = 0; c < A; ++c) rb[(t + T * i) * (A + 1) + c] = v[i][c];
    __syncwarp();
#pragma unroll
    for (int i = 0; i < NB2; ++i) {
#pragma unroll
      for (int b = 0; b < C; ++b) o[i][b] = rb[b * (A + 1) + t + T * i];
      DFT<C, INV>::run(o[i]);
    }
  } else {
    constexpr int NB = M / B / T, J = xrow_table_j(N, INV);  // NB: B-point DFTs of a lane
    static_assert(M / B % T == 0, "row plan");
    auto at = [](int e) { return e + e / A; };
    __syncwarp();
#pragma unroll
    for (int i = 0; i < NB1; ++i) {
      DFT<A, INV>::run(v[i]);
#pragma unroll
      for (int r = 0; r < A; ++r) rb[at((t + T * i) * A + r)] = v[i][r];
    }
    __syncwarp();
    float2 u[NB][B];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      const int j = t + T * i, k = j % A;
#pragma unroll
      for (int r = 0; r < B; ++r) u[i][r] = rb[at(j + r * (M / B))];
#pragma unroll
      for (int r = 1; r < B; ++r) u[i][r] = cmul(u[i][r], twiddle(r * k * (M / (A * B)), (r - 1) * A + k));
      DFT<B, INV>::run(u[i]);
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      const int j = t + T * i, k = j % A, base = (j - k) * B + k;
#pragma unroll
      for (int r = 0; r < B; ++r) rb[at(base + r * A)] = u[i][r];
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < NB2; ++i) {
      const int j = t + T * i;
#pragma unroll
      for (int r = 0; r < C; ++r) o[i][r] = rb[at(j + r * (M / C))];
#pragma unroll
      for (int r = 1; r < C; ++r) o[i][r] = cmul(o[i][r], twiddle(r * j, (B - 1) * A + (r - 1) * J + j, T * i < J));
      DFT<C, INV>::run(o[i]);
    }
  }
}

// The ends of a row work on the pairs (k, M - k).  Lane t holds the K = M / T elements t + T m: the
// partner of element m is element K - 1 - m of lane T - t -- lane 0's is its own K - m, and k = 0
// goes with k = M -- so each lane takes the pairs of its lower half, with the partners brought by
// shuffles.  (Through the exchange buffer, every element written once and read twice, the ends
// took more of the shared-memory pipe than the transform itself: x C2R of 192^3 20.6 -> 17.7 us, 512^3
// 195 -> 174, R2C of 192^3 21.5 -> 15.7, the fused deposit of 1024^3 3.64 -> 3.35 ms.)  Lane 0 is one pair ahead in the
// upper half (its k = M / 2, alone, starts it), so that the T elements of a step are consecutive
// and aligned there too.
template <int T>
__device__ __forceinline__ float2 xrow_partner(float2 v, int t) {
  const int src = (T - t) & (T - 1);
  return make_float2(__shfl_sync(FULL, v.x, src, T), __shfl_sync(FULL, v.y, src, T));
}
__device__ __forceinline__ float2 cselect(bool c, float2 a, float2 b) { return make_float2(c ? a.x : b.x, c ? a.y : b.y); }

// R2C end of a row: Z (in o) is untangled into the half-spectrum row dst[0..M] (if `store`).
// Every lane of the warp calls it.
template <int N>
__device__ __forceinline__ void xrow_untangle_store(const float2 (&o)[xrow_NB2<N, false>][xrow_C(N, false)], int t,
                                                    const float2* __restrict__ tw, float2* __restrict__ dst, bool store) {
  constexpr int M = N / 2, T = xrow_T(N, false), NB = xrow_NB2<N, false>, K = M / T;
  static_assert(K % 2 == 0 && (T & (T - 1)) == 0, "pairs of a lane");
  // X[k] = E + W^k O, X[M - k] = conj(E - W^k O)
  float2 up = conjf2(o[K / 2 % NB][K / 2 / NB]);  // lane 0: X[M / 2]
#pragma unroll
  for (int m = K / 2 - 1; m >= 0; --m) {
    const int j = K - 1 - m, j0 = (K - m) % K, k = t + T * m;
    const float2 zk = o[m % NB][m / NB];
    const float2 zc = conjf2(xrow_partner<T>(cselect(t == 0, o[j0 % NB][j0 / NB], o[j % NB][j / NB]), t));
    const float2 e = cscale(cadd(zk, zc), 0.5f);
    const float2 od = cscale(mul_mi<false>(csub(zk, zc)), 0.5f);
    const float2 wo = cmul(__ldg(&tw[k]), od);
    const float2 xm = conjf2(csub(e, wo));
    if (store) {
      dst[k] = cadd(e, wo);
      dst[(t == 0 ? M - T : M - t) - T * m] = cselect(t == 0, up, xm);
    }
    up = xm;
  }
  if (store && t == 0) dst[M] = up;
}

// C2R start of a row: the half-spectrum row src[0..M] is loaded and tangled into pass 1's input,
// Z[k] = (X[k] + X*[M-k]) + i W^-k (X[k] - X*[M-k]).  Every lane of the warp calls it.
template <int N>
__device__ __forceinline__ void xrow_load_tangle(float2 (&v)[xrow_NB1<N, true>][xrow_A(N, true)], int t,
                                                 const float2* __restrict__ tw, const float2* __restrict__ src) {
  constexpr int M = N / 2, T = xrow_T(N, true), NB = xrow_NB1<N, true>, K = M / T;
  static_assert(K % 2 == 0 && (T & (T - 1)) == 0, "pairs of a lane");
#pragma unroll
  for (int m = 0; m < K; ++m) v[m % NB][m / NB] = __ldg(&src[t + T * m]);
  const float2 top = t == 0 ? __ldg(&src[M]) : make_float2(0.f, 0.f);
  float2 up = v[K / 2 % NB][K / 2 / NB];  // lane 0: Z[M / 2] = 2 conj(X[M / 2])
  up = make_float2(2.f * up.x, -2.f * up.y);
#pragma unroll
  for (int m = K / 2 - 1; m >= 0; --m) {
    const int j = K - 1 - m, j0 = K - m;
    const float2 xk = v[m % NB][m / NB];
    const float2 x0 = m == 0 ? top : v[j0 % K % NB][j0 % K / NB];
    const float2 xm = xrow_partner<T>(cselect(t == 0, x0, v[j % NB][j / NB]), t);
    const float2 ap = cadd(xk, conjf2(xm)), bm = csub(xk, conjf2(xm));
    const float2 tt = cmul(conjf2(__ldg(&tw[t + T * m])), bm);
    v[m % NB][m / NB] = make_float2(ap.x - tt.y, ap.y + tt.x);
    const float2 back = xrow_partner<T>(make_float2(ap.x + tt.y, tt.x - ap.y), t);
    v[j % NB][j / NB] = cselect(t == 0, up, back);
    up = back;
  }
}

template <int N, bool C2R>
__global__ void __launch_bounds__(xrow_nt(N, C2R)) k_x_row(const Sim* __restrict__ sims, Work w) {
  chain_begin();
  constexpr int XR_NT = xrow_nt(N, C2R);
  constexpr int M = N / 2, A = xrow_A(N, C2R), B = xrow_B(N, C2R), C = xrow_C(N, C2R), T = xrow_T(N, C2R), RPW = 32 / T;
  constexpr int UR = xrow_unit_rows(N), RB = xrow_exchange(N, C2R);  // exchange buffer of a row
  constexpr int NB1 = xrow_NB1<N, C2R>, NB2 = xrow_NB2<N, C2R>;
  static_assert(A * B * C == M && NB1 * A * T == M && NB2 * C * T == M, "row plan");
  __shared__ float2 sbuf[XR_NT / 32][RPW][RB];
  __shared__ float2 wt[xrow_table_size<N, C2R, false>()];
  if (xrow_table(N, false)) {
    xrow_table_fill<N, C2R, false, XR_NT>(wt, sims[locate_sim(w, 0)].tw);
    __syncthreads();
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int sub = lane / T, t = lane % T;
  float2* rb = sbuf[wid][sub];
  const long long nw = (long long)gridDim.x * (XR_NT / 32);
  for (long long unit = (long long)blockIdx.x * (XR_NT / 32) + wid; unit < w.total; unit += nw) {
    const int si = locate_sim(w, (int)unit);
    const Sim& S = sims[si];
    const float2* __restrict__ tw = S.tw;
    long long row = ((long long)unit - __ldg(&w.prefix[si])) * UR + sub;
#pragma unroll 1
    for (int r = 0; r < UR; r += RPW, row += RPW) {
      float2 v[NB1][A];
      float2 o[NB2][C];
      if constexpr (!C2R) {
        const float2* __restrict__ src = reinterpret_cast<const float2*>(S.rho) + row * M;
#pragma unroll
        for (int i = 0; i < NB1; ++i)
#pragma unroll
          for (int a = 0; a < A; ++a) v[i][a] = __ldg(&src[M / A * a + t + T * i]);
        xrow_transform<N, false, false>(v, o, rb, t, tw, wt);
        xrow_untangle_store<N>(o, t, tw, S.spec + spec_row(N, (int)(row % N), (int)(row / N)) * S.pitch, true);
      } else {
        xrow_load_tangle<N>(v, t, tw, S.spec + spec_row(N, (int)(row % N), (int)(row / N)) * S.pitch);
        xrow_transform<N, true, false>(v, o, rb, t, tw, wt);
        float2* __restrict__ dst = reinterpret_cast<float2*>(S.phi) + row * M;
#pragma unroll
        for (int i = 0; i < NB2; ++i)
#pragma unroll
          for (int d = 0; d < C; ++d) dst[t + T * i + M / C * d] = o[i][d];
      }
    }
  }
}

// Tensor map of a half spectrum seen as float32 [y / YB][z][y % YB][2*pitch] (spec_row): boxes of BOX
// rows, {2 BW, min(YB, BOX), 1, rest} for the y pass and {2 BW, 1, BOX, 1} for the z pass.
inline bool encode_spectrum_map(CUtensorMap* tm, const void* spec, int n, bool zaxis) {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !p)
      return false;
    fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  const cuuint64_t row = (cuuint64_t)2 * cpitch(n);
  const cuuint32_t box_rows = (cuuint32_t)line_box_rows(n);
  const cuuint32_t yb = (cuuint32_t)spec_block(n), yrows = yb < box_rows ? yb : box_rows;
  cuuint64_t dims[4] = {row, yb, (cuuint64_t)n, (cuuint64_t)n / yb};
  cuuint64_t strides[3] = {row * 4, row * 4 * yb, row * 4 * yb * (cuuint64_t)n};
  cuuint32_t box[4] = {(cuuint32_t)(2 * cline_width(n)), zaxis ? 1u : yrows, zaxis ? box_rows : 1u,
                       zaxis ? 1u : box_rows / yrows};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  return fn(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<void*>(spec), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// ---------------------------------------------------------------------------------
// fused deposit + x R2C (the sizes with a register row transform): a CTA deposits tiles of
// TZ x TY rows into shared memory (pm_deposit.cuh), transforms each row along x in place and
// writes the half-spectrum rows, so the density grid never goes to HBM.
// ---------------------------------------------------------------------------------
__host__ __device__ constexpr bool deposit_r2c_ok(int n) { return xrow_ok(n); }
// words of a tile row: its cells, or the exchange buffer of its transform, which overlays them
__host__ __device__ constexpr int dep_row_words(int n) {
  return 2 * xrow_exchange(n, false) > n ? 2 * xrow_exchange(n, false) : n;
}
__host__ __device__ constexpr size_t dep_tile_bytes(int n) { return (size_t)TZ * TY * dep_row_words(n) * sizeof(unsigned); }
constexpr int DEP_ROW_NT = 256;  // threads (the 16 rows of a 1024 tile take them twice: 3.95 ms, 512 threads 4.34)
// Tiles per CTA: the row transform of a tile's 16 rows keeps 16 / T warps busy (T lanes per row),
// so on the sizes with T < 16 a CTA takes several tiles at once -- its warps split into one
// group per tile for the particle loop and share all the rows in the transform.
__host__ __device__ constexpr int dep_tiles(int n) {
  return n == 1024 ? 1 : (16 / xrow_T(n, false) > 4 ? 4 : 16 / xrow_T(n, false));
}
// CTAs per SM, which bounds the registers of a thread: four (64) where the row plan leaves few
// spills (512: 423 us, three 466; 256 in an ensemble 234, three 262; 64 and 96 lose 10%), else three
// (192: 134, two 144; 768: 1589, two 1717); five spill (512: 495; all before the row ends and
// twiddles below).  The 512 grid now takes 356 us, the 1024 grid 3.16 ms (442 us and 6.12 ms with a low
// and a coarse word for every cell at three CTAs).
__host__ __device__ constexpr int dep_ctas_bound(int n) { return n == 128 || n == 256 || n == 512 ? 4 : 3; }

// The tile at place i of the order (`order`, optional, lists the tiles dense-first): its
// simulation and first row / plane (false: none).
template <int N>
__device__ __forceinline__ bool dep_tile(const Work& w, const unsigned* __restrict__ order, int i, int& si, int& y0,
                                         int& z0) {
  si = 0; y0 = z0 = 0;
  if (i >= w.total) return false;
  const int unit = order ? (int)__ldg(&order[i]) : i;
  si = locate_sim(w, unit);
  const int local = unit - __ldg(&w.prefix[si]);
  y0 = (local % (N / TY)) * TY;
  z0 = (local / (N / TY)) * TZ;
  return true;
}

// The x R2C of the NL rows of each tile (or plane of one): row r's sums at acc + r * stride (TWO: its high words dep_row_words further
// on); T lanes to a row, whose exchange buffer overlays its low words once they are read.  A
// batch is the rows that the CTA's warps hold at once.  f(tg): whether to store tile tg's rows and
// where they belong; `between` runs in warp 0 before the first transform, `after` behind the
// last; every row is left zero.  rows: all of the TPB * NL, or the first ones.
template <int N, int NT, int TPB, int NL, bool TWO, class H, class F, class G>
__device__ __forceinline__ void dep_transform(const Sim* __restrict__ sims, unsigned* acc, int stride, const TileSum* s_ts,
                                              const float2* wt, H tile, F between, G after, int rows = TPB * NL) {
  constexpr int M = N / 2, A = xrow_A(N, false), C = xrow_C(N, false), T = xrow_T(N, false), RPW = 32 / T;
  constexpr int NB1 = xrow_NB1<N, false>, NB2 = xrow_NB2<N, false>;
  constexpr int BROWS = NT / 32 * RPW, NBATCH = (TPB * NL + BROWS - 1) / BROWS;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane / T, t = lane % T;
#pragma unroll 1
  for (int batch = 0; batch < NBATCH; ++batch) {
    if (batch * BROWS + warp * RPW >= rows) break;  // warp-uniform
    // (where a warp holds more rows than there are, its other lanes repeat the last one)
    const int R0 = batch * BROWS + warp * RPW + sub, R = (!TWO && TPB * NL % RPW == 0) || R0 < rows ? R0 : rows - 1;
    const int tg = R / NL, r = R % NL;
    unsigned* row = acc + R * stride;
    float2* rb = reinterpret_cast<float2*>(row);
    int si, y0, z0;
    const bool has = tile(tg, si, y0, z0) && R == R0;
    const Sim& S = sims[si];
    const TileSum ts = s_ts[tg];
    float2 v2[NB1][A];
    float2 o2[NB2][C];
    const uint2* l2 = reinterpret_cast<const uint2*>(row);
    const uint2* h2 = reinterpret_cast<const uint2*>(row + dep_row_words(N));
#pragma unroll
    for (int i = 0; i < NB1; ++i)
#pragma unroll
      for (int a = 0; a < A; ++a) {
        const int j = M / A * a + t + T * i;  // z[j] = x[2j] + i x[2j+1]
        const uint2 l = l2[j];
        if (!TWO) {
          v2[i][a] = make_float2(word_to_float(l.x, ts.ms), word_to_float(l.y, ts.ms));
        } else {
          const uint2 h = h2[j];
          v2[i][a] = make_float2(fixed_to_float(l.x, h.x, ts.ms), fixed_to_float(l.y, h.y, ts.ms));
        }
      }
    if (warp == 0 && batch == 0) between();
    xrow_transform<N, false, true>(v2, o2, rb, t, S.tw, wt);
    xrow_untangle_store<N>(o2, t, S.tw, S.spec + spec_row(N, y0 + r % TY, z0 + r / TY) * S.pitch, has);
    __syncwarp();  // the row's lanes are done with its words
    uint4* z4 = reinterpret_cast<uint4*>(row);
    for (int i = t; i < stride / 4; i += T) z4[i] = make_uint4(0u, 0u, 0u, 0u);
    if (warp == 0 && (batch == NBATCH - 1 || (batch + 1) * BROWS >= rows)) after();
  }
}

// Source entries from which on a tile of two-word sums is taken apart by planes (k_deposit_r2c_dense).
constexpr unsigned DEP_HEAVY = 16384;

template <int N>
__global__ void __launch_bounds__(DEP_ROW_NT, dep_ctas_bound(N))
    k_deposit_r2c(const Sim* __restrict__ sims, Work w, Parts p, const unsigned* __restrict__ perm,
                  const unsigned* __restrict__ row_start, const unsigned* __restrict__ group_max, int* err,
                  unsigned* __restrict__ next_tile, const unsigned* __restrict__ order, unsigned* __restrict__ dense) {
  constexpr int NT = DEP_ROW_NT, NL = TZ * TY, TPB = dep_tiles(N);
  constexpr int RS = dep_row_words(N);  // words from a tile row to the next
  constexpr int NTT = NT / TPB;         // threads per tile group
  static_assert(TPB * 8 <= 32 && NT % (TPB * 32) == 0, "one warp loads the run tables of a CTA's tiles");
  static_assert(RS % 4 == 0, "rows zeroed 4 words at a time");
  extern __shared__ uint4 acc_raw[];
  // run tables of the CTA's tiles (7 runs each: first sorted index, and inclusive offsets)
  __shared__ unsigned s_begin[TPB][8];
  __shared__ unsigned s_off[TPB][8];
  __shared__ TileSum s_ts[2][TPB];  // of the tiles at hand and the next ones, in turn
  __shared__ int s_next;
  __shared__ float2 wt[xrow_table_size<N, false, true>()];
  unsigned* acc = reinterpret_cast<unsigned*>(acc_raw);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // warp 0: the run tables of the tiles at places idx .. idx + TPB - 1 (8 lanes per tile)
  auto load_tables = [&](int idx) -> RunLoad {
    RunLoad v;
    int si, y0, z0;
    if (dep_tile<N>(w, order, idx + (lane >> 3), si, y0, z0))
      v = run_load<BINS_MAXIMA>(sims[si], row_start, group_max, y0, z0, lane & 7);
    return v;
  };
  // warp 0: stores the tables and how the tiles' sums are held; a tile with two-word sums goes to
  // the list of k_deposit_r2c_dense (at its back if heavy) and is left out here
  auto store_tables = [&](const RunLoad& v, int idx, TileSum* ts) {
    const int tj = lane < TPB * 8 ? lane >> 3 : 0;
    unsigned total;
    const TileSum t = run_table(v, lane, s_begin[tj], s_off[tj], lane < TPB * 8, total);
    if (lane < TPB * 8 && (lane & 7) == 0) {
      ts[tj] = t;
      if (t.s == 0) {
        const bool heavy = total >= DEP_HEAVY;
        const unsigned at = atomicAdd(next_tile + (heavy ? 3 : 1), 1u);
        dense[heavy ? w.total - 1 - at : at] = (unsigned)(idx + tj);
      }
    }
  };
  // Tiles are taken from a counter (zero at launch) after the first, TPB per CTA: a tile's
  // work is its particle count, which clustering makes very uneven, so a fixed stride
  // leaves the CTAs that drew the dense tiles running alone at the end.  Warp 0 takes the next
  // tiles and loads their run tables before the transform and stores them after it, so that
  // the loads' latency hides behind it (the particle loops are over).
  int next = 0, turn = 0;
  RunLoad nl;
  auto take = [&]() {
    next = __shfl_sync(FULL, lane == 0 ? (int)gridDim.x * TPB + (int)atomicAdd(next_tile, (unsigned)TPB) : 0, 0);
    if (next < w.total) nl = load_tables(next);
  };
  auto store = [&]() {
    if (next < w.total) store_tables(nl, next, s_ts[turn ^ 1]);
    if (lane == 0) s_next = next;
  };
  // The accumulators start zero, and each row is zeroed again by its transform lanes once
  // they are done with it, so a tile needs no zeroing phase and barrier of its own
  // (0.468 -> 0.460 ms early, 0.604 -> 0.587 ms at step 980, 256^3 on 512^3).
  for (int i = threadIdx.x; i < TPB * NL * RS / 4; i += NT) acc_raw[i] = make_uint4(0u, 0u, 0u, 0u);
  chain_begin();
  xrow_table_fill<N, false, true, NT>(wt, sims[locate_sim(w, 0)].tw);
  int idx = blockIdx.x * TPB;
  if (warp == 0 && idx < w.total) store_tables(load_tables(idx), idx, s_ts[0]);
  __syncthreads();
  for (; idx < w.total; turn ^= 1) {
    {  // the particles of this group's tile (a group without a tile has an empty table)
      const int g = threadIdx.x / NTT, gtid = threadIdx.x % NTT;
      int si, y0, z0;
      dep_tile<N>(w, order, idx + g, si, y0, z0);
      const TileSum ts = s_ts[turn][g];
      if (ts.s)
        deposit_tile<POS_DISP, NTT, true, N>(sims[si], p, perm, err, y0, z0, acc + g * NL * RS, nullptr, RS, s_begin[g],
                                             s_off[g], ts, make_int2(0, TZ), gtid);
    }
    __syncthreads();
    bool any = false;  // (without a one-word tile there is nothing to transform)
#pragma unroll
    for (int j = 0; j < TPB; ++j) any = any || s_ts[turn][j].s;
    if (any) {
      dep_transform<N, NT, TPB, NL, false>(
          sims, acc, RS, s_ts[turn], wt,
          [&](int tg, int& si, int& y0, int& z0) { return dep_tile<N>(w, order, idx + tg, si, y0, z0) && s_ts[turn][tg].s; },
          take, store);
    } else if (warp == 0) {
      take();
      store();
    }
    __syncthreads();
    idx = s_next;
  }
}

// The tiles that k_deposit_r2c left: those with two-word sums.  A kernel of its own: next to the
// one-word path its registers and code cost that path 10% (442 -> 498 us on the 512 grid).  A unit of
// work, taken from a counter, is a whole tile (half of one on 1024, where four planes would leave room for one
// CTA).  Planes are units of their own, and read every particle up to twice, in two cases:
// * heavy tiles, which come first: the heart of a large halo is one tile, whose atomics on a few
//   cells alone would otherwise outlast the rest of the kernel (256^3 particles on 512^3 at step 980
//   of 1000: all tiles whole 385 us, heavy from 8192 entries on 236, from 16384 on 213 -- these with
//   256 threads; with 512 178; all by planes 254);
// * fewer tiles than CTAs (128^3 particles on 128^3 at step 20: 47 us whole, 34 by planes).
// By planes alone a state with most of its tiles dense takes twice the time (256^3 on 256^3 early 466 us
// against 242; 357^3 on 512^3 1423 against 745).  512 threads, 2 CTAs per SM, against 256
// threads and up to 4: 1024^3 late 1736 against 2104 us, 96^3 on 128^3 late 64 against 90, the dense early
// states 745 against 723 and 242 against 212; 384 threads lie between.
constexpr int DEP_DENSE_NT = 512;
__host__ __device__ constexpr int dep_dense_planes(int n) { return n == 1024 ? 2 : TZ; }  // planes of a large unit
__host__ __device__ constexpr int dep_dense_stride(int n) { return dep_row_words(n) + n; }  // low words, high words
__host__ __device__ constexpr size_t dep_dense_bytes(int n) {
  return (size_t)dep_dense_planes(n) * TY * dep_dense_stride(n) * sizeof(unsigned);
}
__host__ __device__ constexpr int dep_dense_ctas(int n) {
  const int by_smem = (int)((220 * 1024) / (dep_dense_bytes(n) + 6 * 1024));
  return by_smem > 2 ? 2 : by_smem;
}

template <int N>
__global__ void __launch_bounds__(DEP_DENSE_NT, dep_dense_ctas(N))
    k_deposit_r2c_dense(const Sim* __restrict__ sims, Work w, Parts p, const unsigned* __restrict__ perm,
                        const unsigned* __restrict__ row_start, int* err, unsigned* __restrict__ next_tile,
                        const unsigned* __restrict__ order, const unsigned* __restrict__ dense) {
  constexpr int NT = DEP_DENSE_NT, RS = dep_dense_stride(N), PU = dep_dense_planes(N);
  static_assert(RS % 4 == 0, "rows zeroed 4 words at a time");
  extern __shared__ uint4 acc_raw[];
  __shared__ unsigned s_begin[8];
  __shared__ unsigned s_off[8];
  __shared__ unsigned s_next;
  __shared__ float2 wt[xrow_table_size<N, false, true>()];
  unsigned* acc = reinterpret_cast<unsigned*>(acc_raw);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  chain_begin();
  const unsigned light = next_tile[1], heavy = next_tile[3] * TZ;
  const int pu = light < gridDim.x ? 1 : PU;  // planes of a unit of a light tile
  const unsigned count = heavy + light * (unsigned)(TZ / pu);
  if (blockIdx.x >= count) return;
  for (int i = threadIdx.x; i < PU * TY * RS / 4; i += NT) acc_raw[i] = make_uint4(0u, 0u, 0u, 0u);
  xrow_table_fill<N, false, true, NT>(wt, sims[locate_sim(w, 0)].tw);
  // unit u: planes p0 .. p1 - 1 of a tile (a heavy one from the back of the list, a light one from its front)
  auto unit = [&](unsigned u, int& si, int& y0, int& z0, int& p0, int& p1) {
    const bool hv = u < heavy;
    const unsigned v = hv ? u : u - heavy, k = hv ? 1u : (unsigned)pu, parts = TZ / k;
    p0 = (int)(v % parts * k);
    p1 = p0 + (int)k;
    dep_tile<N>(w, order, (int)dense[hv ? (unsigned)w.total - 1 - v / parts : v / parts], si, y0, z0);
  };
  // warp 0 takes the next unit and loads its run table before the transform and stores it after
  unsigned i = blockIdx.x, next = 0, total;
  RunLoad nl;
  auto load = [&](unsigned u) {
    int si, y0, z0, p0, p1;
    unit(u, si, y0, z0, p0, p1);
    nl = plane_load(sims[si], row_start, y0, z0, p0, p1, lane & 7);
  };
  auto take = [&]() {
    next = __shfl_sync(FULL, lane == 0 ? gridDim.x + atomicAdd(next_tile + 2, 1u) : 0u, 0);
    if (next < count) load(next);
  };
  auto store = [&]() {
    if (next < count) run_table(nl, lane, s_begin, s_off, lane < 8, total);
    if (lane == 0) s_next = next;
  };
  if (warp == 0) {
    load(i);
    run_table(nl, lane, s_begin, s_off, lane < 8, total);
  }
  __syncthreads();
  while (i < count) {
    int si, y0, z0, p0, p1;
    unit(i, si, y0, z0, p0, p1);
    const TileSum ts{0, sims[si].mass_scale};
    deposit_tile<POS_DISP, NT, false, N>(sims[si], p, perm, err, y0, z0, acc, acc + dep_row_words(N), RS, s_begin, s_off, ts,
                                         make_int2(p0, p1), threadIdx.x);
    __syncthreads();
    dep_transform<N, NT, 1, PU * TY, true>(
        sims, acc, RS, &ts, wt, [&](int, int& a, int& b, int& c) { a = si; b = y0; c = z0 + p0; return true; }, take,
        store, (p1 - p0) * TY);
    __syncthreads();
    i = s_next;
  }
}

template <int N>
cudaError_t deposit_r2c_launch(const Sim* sims, Work w, Parts p, const unsigned* perm, const unsigned* row_start,
                               const unsigned* group_max, int* err, unsigned* next_tile, const unsigned* order,
                               unsigned* dense, int ctas, Launch st) {
  if constexpr (!deposit_r2c_ok(N)) {
    return cudaErrorNotSupported;
  } else {
    static DeviceOnce once;
    const size_t sm = dep_tiles(N) * dep_tile_bytes(N);
    const size_t smd = dep_dense_bytes(N);
    const cudaError_t ie = once.run([&]() {
      cudaError_t e = cudaFuncSetAttribute(k_deposit_r2c<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
      if (!e) e = cudaFuncSetAttribute(k_deposit_r2c<N>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
      if (!e)
        e = cudaFuncSetAttribute(k_deposit_r2c_dense<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smd);
      if (!e) e = cudaFuncSetAttribute(k_deposit_r2c_dense<N>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
      return e;
    });
    if (ie) return ie;
    if (ctas <= 0) return cudaSuccess;  // attribute setup only
    constexpr int NT = DEP_ROW_NT, TPB = dep_tiles(N);
    if (ctas > (w.total + TPB - 1) / TPB) ctas = (w.total + TPB - 1) / TPB;  // TPB tiles per CTA
    if (ctas <= 0) return cudaSuccess;
    launch_chained(k_deposit_r2c<N>, ctas, NT, sm, st, sims, w, p, perm, row_start, group_max, err, next_tile, order,
                   dense);
    if (cudaError_t e = cudaGetLastError()) return e;
    const int cap = device_sms() * dep_dense_ctas(N), few = w.total < cap / TZ ? w.total * TZ : cap;
    launch_chained(k_deposit_r2c_dense<N>, few, DEP_DENSE_NT, smd, st, sims, w, p, perm, row_start, err, next_tile,
                   order, dense);
    return cudaGetLastError();
  }
}

template <typename K>
static cudaError_t max_shared(K kern, size_t bytes) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (!e) e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  return e;
}

template <int N>
cudaError_t spectral_launch(SpecKind kind, const Sim* sims, Work w, int ctas, Launch st,
                            const CUtensorMap* maps, int* err) {
  static DeviceOnce once;
  const size_t xs = x_smem_bytes(N), ls = line_smem_bytes(N);
  const cudaError_t ie = once.run([&]() -> cudaError_t {
    if constexpr (tma_lines(N)) {
      cudaError_t e = max_shared(k_line_tma<N, 0>, tma_smem_bytes(N, false));
      if (!e) e = max_shared(k_line_tma<N, 1>, tma_smem_bytes(N, false));
      if (!e) e = max_shared(k_line_tma<N, 2>, tma_smem_bytes(N, true));
      if (!e) e = max_shared(k_line_tma<N, 3>, tma_smem_bytes(N, true));
      if (!e) e = max_shared(k_line_tma<N, 4>, tma_smem_bytes(N, false));
      if (!e) e = max_shared(k_line_tma<N, 5>, tma_smem_bytes(N, false));
      if (!e) e = max_shared(k_line_tma<N, 6>, tma_smem_bytes(N, true));
      if (e) return e;
    }
    cudaError_t e = cudaSuccess;
    if constexpr (!xrow_ok(N)) {
      e = max_shared(k_x_r2c<N>, xs);
      if (!e) e = max_shared(k_x_c2r<N>, xs);
    }
    if (!e) e = max_shared(k_line_pass<N, false, false>, ls);
    if (!e) e = max_shared(k_line_pass<N, false, true>, ls);
    if (!e) e = max_shared(k_line_pass<N, true, false>, ls);
    if (!e) e = max_shared(k_line_pass<N, true, true>, ls);
    if (!e) e = max_shared(k_z_green<N, false>, ls);
    if (!e) e = max_shared(k_z_green<N, true>, ls);
    if (!e) e = max_shared(k_z_green<N, false, true>, ls);
    return e;
  });
  if (ie) return ie;
  if (kind == SPEC_PREPARE) return cudaSuccess;
  if constexpr (xrow_ok(N)) {
    if (kind == SPEC_X_R2C || kind == SPEC_X_C2R) {
      // ctas: the cap on the CTAs of the persistent row transform (the batch engine tunes it)
      const int nt = xrow_nt(N, kind == SPEC_X_C2R);
      const int per = nt / 32, want = (w.total + per - 1) / per, cap = ctas > 0 ? ctas : device_sms() * 8;
      const int g = want < cap ? want : cap;
      if (kind == SPEC_X_R2C) launch_chained(k_x_row<N, false>, g, nt, 0, st, sims, w);
      else launch_chained(k_x_row<N, true>, g, nt, 0, st, sims, w);
      return cudaGetLastError();
    }
  }
  if constexpr (!xrow_ok(N)) {
    if (kind == SPEC_X_R2C || kind == SPEC_X_C2R) {
      if (kind == SPEC_X_R2C) launch_chained(k_x_r2c<N>, ctas, SP_NT, xs, st, sims, w);
      else launch_chained(k_x_c2r<N>, ctas, SP_NT, xs, st, sims, w);
      return cudaGetLastError();
    }
  }
  if constexpr (tma_lines(N)) {
    if (maps) {
      const bool turn = kind == SPEC_Z_GREEN || kind == SPEC_Z_TABLE || kind == SPEC_Z_GRAD;
      const size_t sm = tma_smem_bytes(N, turn);
      const int nt = turn ? turn_nt(N) : line_nt(N);
      const int lcap = (turn ? turn_ctas_per_sm(N) : line_ctas_per_sm(N)) * device_sms();
      const int grid = w.total < lcap ? w.total : lcap;
      switch (kind) {
        case SPEC_Y_FWD: launch_chained(k_line_tma<N, 0>, grid, nt, sm, st, maps, sims, w, err); return cudaGetLastError();
        case SPEC_Y_INV: launch_chained(k_line_tma<N, 1>, grid, nt, sm, st, maps, sims, w, err); return cudaGetLastError();
        case SPEC_Z_GREEN: launch_chained(k_line_tma<N, 2>, grid, nt, sm, st, maps, sims, w, err); return cudaGetLastError();
        case SPEC_Z_TABLE: launch_chained(k_line_tma<N, 3>, grid, nt, sm, st, maps, sims, w, err); return cudaGetLastError();
        case SPEC_Z_FWD: launch_chained(k_line_tma<N, 4>, grid, nt, sm, st, maps, sims, w, err); return cudaGetLastError();
        case SPEC_Z_INV: launch_chained(k_line_tma<N, 5>, grid, nt, sm, st, maps, sims, w, err); return cudaGetLastError();
        case SPEC_Z_GRAD: launch_chained(k_line_tma<N, 6>, grid, nt, sm, st, maps, sims, w, err); return cudaGetLastError();
        default: break;
      }
    }
  }
  switch (kind) {
    case SPEC_Y_FWD: launch_chained(k_line_pass<N, false, false>, ctas, SP_NT, ls, st, sims, w); break;
    case SPEC_Y_INV: launch_chained(k_line_pass<N, false, true>, ctas, SP_NT, ls, st, sims, w); break;
    case SPEC_Z_FWD: launch_chained(k_line_pass<N, true, false>, ctas, SP_NT, ls, st, sims, w); break;
    case SPEC_Z_INV: launch_chained(k_line_pass<N, true, true>, ctas, SP_NT, ls, st, sims, w); break;
    case SPEC_Z_GREEN: launch_chained(k_z_green<N, false>, ctas, SP_NT, ls, st, sims, w); break;
    case SPEC_Z_TABLE: launch_chained(k_z_green<N, true>, ctas, SP_NT, ls, st, sims, w); break;
    case SPEC_Z_GRAD: launch_chained(k_z_green<N, false, true>, ctas, SP_NT, ls, st, sims, w); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace pm
