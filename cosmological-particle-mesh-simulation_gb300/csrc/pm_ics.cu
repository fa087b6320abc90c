// Initial conditions on the device: the Gaussian random field of
// src/gaussian_random_field.py:9-123 and the Zel'dovich positions and velocities of
// src/zeldovich.py:10-100, computed with the engine's float32 spectral passes.
//
// Input: the two float32 streams of accepted uniform numbers in (-1, 1) of the reference's
// rejection loop (gaussian_random_field.py:35-50; numpy RandomState, drawn by the caller).
// Everything else runs here:
//   * the polar Box-Muller transform (gaussian_random_field.py:53-61), float32 as in the
//     reference, with the float64 recomputation of pairs whose float32 u^2 + v^2 rounds
//     to >= 1 (the reference would produce NaN there);
//   * the power spectrum and its normalisation sum (gaussian_random_field.py:65-123) in
//     float64: the k-dependence is tabulated once per integer |m|^2 (k = 2 pi |m| / box),
//     the sum over the full grid is reduced in a fixed order (deterministic);
//   * Re(ifftn(rho_k)) (gaussian_random_field.py:24-29): the real part of the inverse
//     transform of a non-Hermitian rho_k is the inverse real transform of its Hermitian
//     part (rho_k[k] + conj(rho_k[-k])) / 2, which is built directly in the half spectrum;
//   * fftn of that field, the potential -rho_k / |l|^2 (k = 0 -> 0), -i l_d pot_k * res,
//     and Re(ifftn(.)) * force_resolution per direction (zeldovich.py:17-69), up to 256^3 the
//     three directions together; the planes where l_d sits at the Nyquist
//     frequency have no Hermitian part and are zero;
//   * lattice + Dt * disp + jitter, modulo N_CELLS, and A f H Dt * disp
//     (zeldovich.py:71-100), stored as float32.
//     The jitter is the numpy PCG64 stream of uniform(-2, 2) (x, then y, then z draws),
//     generated here by jumping the 128-bit LCG to each block's first draw.
//
// GB300 issues two float64 operations per SM and clock, against 128 in float32, so the work per
// grid point keeps out of them: the factors that depend on |m|^2 alone are tabulated in float64
// and held as float32 pairs (48 bits and more), and products and sums with them are carried as
// pairs (Dekker's and Knuth's error-free transformations), rounded to float32 once at the end.
// 128^3: spectra of the displacements 170 -> 18 us, particles 227 -> 44, field 59 -> 19; the whole
// call 772 -> 268, with 18 launches instead of 30.
#include "pm_host.cuh"
#include "pm_pair.cuh"

using namespace pm;

namespace {

constexpr int NORM_BLOCKS = 512;  // fixed grid: the reduction order is the same on every device
constexpr int NORM_NT = 256;
constexpr int IC_NT = 256;
constexpr int JIT_NT = 256;       // threads of the particle kernel
constexpr int JIT_ROUNDS = 16;    // particles per thread

// ---- the power spectrum shape (gaussian_random_field.py:65-123) -----------------------
struct Shape {
  double kscale;  // 2 pi / box: k = kscale * sqrt(m2)
  double gamma;   // OMEGA_M0 * H0 * exp(-OMEGA_B0 - OMEGA_B0 / OMEGA_M0)
  double power;
  int lcdm;
};

__device__ double lcdm_transfer(double k, double gamma) {
  const double q = k / gamma;
  const double a = 16.1 * q, b = 5.46 * q, c = 6.71 * q;
  const double f1 = sqrt(1.0 + 3.89 * q + a * a + b * b * b + (c * c) * (c * c));
  double f2 = 0.0;
  if (q != 0.0) {
    const double l = log(1.0 + 2.34 * q), d = 2.34 * q;
    f2 = (l * l) / (d * d);
  }
  return f2 / f1;
}

// Tables of a call: shape[m2] = S(m2), the summand of the normalisation, which is also P(k) / A
// for k != 0; disp[m2] = coef / (l0 m2), so that m_d disp[m2] = coef l_d / |l|^2; and the lattice
// coordinate of each index (numpy's linspace and + 0.5).
struct TableArgs {
  int m2max, n;
  double* shape;
  float2* disp;
  float2* space;
  double coef_l0;       // coef / l0
  double step, stop;    // lattice step and last point
  Shape sp;
};

__global__ void k_tables(TableArgs t) {
  chain_begin();
  const int m2 = blockIdx.x * blockDim.x + threadIdx.x;
  if (m2 < t.n)
    t.space[m2] = split(__dadd_rn(m2 == t.n - 1 && t.n > 1 ? t.stop : __dmul_rn((double)m2, t.step), 0.5));
  if (m2 > t.m2max) return;
  const Shape& sp = t.sp;
  const double k = sp.kscale * sqrt((double)m2);
  double s;
  if (sp.power >= 0.0) {
    const double kp = m2 != 0 ? pow(k, sp.power) : 0.0;
    s = sp.lcdm ? kp * lcdm_transfer(k, sp.gamma) : kp;
  } else {
    const double kinv = m2 != 0 ? pow(k, -sp.power) : 0.0;
    s = kinv != 0.0 ? 1.0 / kinv : 0.0;
  }
  t.shape[m2] = s;
  t.disp[m2] = m2 != 0 ? split(t.coef_l0 / (double)m2) : make_float2(0.f, 0.f);
}

__device__ __forceinline__ int signed_freq(int m, int n) { return m < n / 2 ? m : m - n; }
__device__ __forceinline__ int sq(int m) { return m * m; }

__device__ __forceinline__ double block_sum(double v, double* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += red[i];
  return t;
}

// Partial sums of S over the full grid, evaluated on the half spectrum (kx in [0, n/2])
// with weight 2 for the columns that stand for two full-grid columns.
__global__ void __launch_bounds__(NORM_NT) k_norm_partial(const double* __restrict__ shape, int n,
                                                           double* __restrict__ partial) {
  chain_begin();
  __shared__ double red[NORM_NT / 32];
  const int w = n / 2 + 1;
  const long long total = (long long)n * n * w;
  double acc = 0.0;
  for (long long e = (long long)blockIdx.x * NORM_NT + threadIdx.x; e < total; e += (long long)NORM_BLOCKS * NORM_NT) {
    const int kx = (int)(e % w);
    const long long r = e / w;
    const int ky = (int)(r % n), kz = (int)(r / n);
    const int m2 = sq(signed_freq(kx, n)) + sq(signed_freq(ky, n)) + sq(signed_freq(kz, n));
    const double wt = (kx == 0 || 2 * kx == n) ? 1.0 : 2.0;
    acc += wt * __ldg(&shape[m2]);
  }
  const double t = block_sum(acc, red);
  if (threadIdx.x == 0) partial[blockIdx.x] = t;
}

// A = 64 H0^2 Npix^2 / sum (gaussian_random_field.py:104-121), one block, fixed order.
__global__ void __launch_bounds__(NORM_NT) k_norm_final(const double* __restrict__ partial, double sigma_npix2,
                                                         double* __restrict__ norm) {
  chain_begin();
  __shared__ double red[NORM_NT / 32];
  double acc = 0.0;
  for (int i = threadIdx.x; i < NORM_BLOCKS; i += NORM_NT) acc += partial[i];
  const double t = block_sum(acc, red);
  if (threadIdx.x == 0) norm[0] = sigma_npix2 / t;
}

// amp[m2] = sqrt(P Dt^2) / 2 / n^3 of the field, P = A S(m2) (p0 A for k = 0)
__global__ void k_amp(const double* __restrict__ shape, const double* __restrict__ norm, int m2max, double p0, double d2,
                      double inv_n3, float2* __restrict__ amp) {
  chain_begin();
  const int m2 = blockIdx.x * blockDim.x + threadIdx.x;
  if (m2 > m2max) return;
  const double p = norm[0] * (m2 != 0 ? shape[m2] : p0);
  amp[m2] = split(sqrt(p * d2) * inv_n3 * 0.5);
}

// ---- Gaussian random numbers (gaussian_random_field.py:53-61) -------------------------
__device__ __forceinline__ float2 box_muller(float u, float v) {
  const float s = __fadd_rn(__fmul_rn(u, u), __fmul_rn(v, v));
  float t = __fdiv_rn(-2.0f * logf(s), s);
  if (!(t > 0.0f)) {  // float32 rounding took s to >= 1: float64, clamped at 0
    const double s64 = (double)u * (double)u + (double)v * (double)v;
    const double t64 = -2.0 * log(s64) / s64;
    t = (isfinite(t64) && t64 > 0.0) ? (float)t64 : 0.0f;
  }
  const float r = __fsqrt_rn(t);
  return make_float2(__fmul_rn(u, r), __fmul_rn(v, r));
}

struct GrfArgs {
  int n, pitch;
  const float* u;
  const float* v;
  const float2* amp;
  float2* spec;
};

// Hermitian part of rho_k = sqrt(P Dt^2) (f1 + i f2) over the half spectrum, scaled by 1/n^3.
__global__ void __launch_bounds__(IC_NT) k_grf_fill(GrfArgs g) {
  chain_begin();
  const int n = g.n, P = g.pitch, h = n / 2;
  const long long total = (long long)n * n * P;
  for (long long e = (long long)blockIdx.x * IC_NT + threadIdx.x; e < total; e += (long long)gridDim.x * IC_NT) {
    const int kx = (int)(e % P);
    const int r = (int)(e / P);
    const int ky = spec_row_y(n, r), kz = spec_row_z(n, r);
    float2 out = make_float2(0.f, 0.f);
    if (kx <= h) {
      const int m2 = sq(signed_freq(kx, n)) + sq(signed_freq(ky, n)) + sq(signed_freq(kz, n));
      const float2 amp = __ldg(&g.amp[m2]);
      const long long i = ((long long)kz * n + ky) * n + kx;
      const int my = ky == 0 ? 0 : n - ky, mz = kz == 0 ? 0 : n - kz, mx = kx == 0 ? 0 : n - kx;
      const long long j = ((long long)mz * n + my) * n + mx;
      const float2 a = box_muller(__ldg(&g.u[i]), __ldg(&g.v[i]));
      const float2 b = box_muller(__ldg(&g.u[j]), __ldg(&g.v[j]));
      const float2 sx = two_sum(a.x, b.x), sy = two_sum(a.y, -b.y);
      const float2 px = pair_mul(amp, sx.x), py = pair_mul(amp, sy.x);
      out = make_float2(px.x + (px.y + amp.x * sx.y), py.x + (py.y + amp.x * sy.y));
    }
    g.spec[e] = out;
  }
}

// ---- Zel'dovich displacement spectrum (zeldovich.py:17-69) ------------------------------
struct ZelArgs {
  int n, pitch;
  const float2* disp;  // coef / (l0 m2)
  const float2* in;    // fftn of the density (half spectrum)
  float2* out[3];      // i l_d coef / |l|^2 times it along axis d of the (n, n, n) array (0 = slowest,
                       // the z of [z][y][x]); null: not wanted; one of them may be `in`
};

__global__ void __launch_bounds__(IC_NT) k_zeld_spectrum(ZelArgs z) {
  chain_begin();
  const int n = z.n, P = z.pitch, h = n / 2;
  const long long total = (long long)n * n * P;
  for (long long e = (long long)blockIdx.x * IC_NT + threadIdx.x; e < total; e += (long long)gridDim.x * IC_NT) {
    const int kx = (int)(e % P);
    const int r = (int)(e / P);
    const int ky = spec_row_y(n, r), kz = spec_row_z(n, r);
    const bool mode = kx <= h && (kx | ky | kz) != 0;
    float2 re = make_float2(0.f, 0.f), im = re;  // disp[m2] * v
    if (mode) {
      const int m2 = sq(signed_freq(kx, n)) + sq(signed_freq(ky, n)) + sq(signed_freq(kz, n));
      const float2 c = __ldg(&z.disp[m2]), v = z.in[e];
      re = pair_mul(c, v.x);
      im = pair_mul(c, v.y);
    }
    #pragma unroll
    for (int d = 0; d < 3; ++d) {
      if (!z.out[d]) continue;
      const int kd = d == 0 ? kz : (d == 1 ? ky : kx);
      float2 o = make_float2(0.f, 0.f);
      if (mode && kd != h) {  // i * m_d * (disp v)
        const float m = (float)signed_freq(kd, n);
        const float2 a = pair_mul(im, m), b = pair_mul(re, m);
        o = make_float2(-(a.x + a.y), b.x + b.y);
      }
      z.out[d][e] = o;
    }
  }
}

// ---- numpy PCG64 (128-bit LCG, XSL-RR output) -------------------------------------------
typedef unsigned __int128 u128;

__host__ __device__ __forceinline__ u128 pcg_mult() {
  return ((u128)0x2360ED051FC65DA4ull << 64) | (u128)0x4385DF649FCCF645ull;
}

// State after `delta` more steps of state' = state * M + inc (Brown's jump-ahead).
__host__ __device__ inline u128 pcg_advance(u128 state, u128 inc, unsigned long long delta) {
  u128 cur_mult = pcg_mult(), cur_plus = inc, acc_mult = 1, acc_plus = 0;
  while (delta > 0) {
    if (delta & 1ull) {
      acc_mult *= cur_mult;
      acc_plus = acc_plus * cur_mult + cur_plus;
    }
    cur_plus = (cur_mult + 1) * cur_plus;
    cur_mult *= cur_mult;
    delta >>= 1;
  }
  return acc_mult * state + acc_plus;
}

__host__ __device__ __forceinline__ unsigned long long pcg_output(u128 s) {
  const unsigned long long x = (unsigned long long)(s >> 64) ^ (unsigned long long)s;
  const unsigned rot = (unsigned)(s >> 122);
  return (x >> rot) | (x << ((64u - rot) & 63u));
}

// uniform(-2, 2) of numpy's Generator, -2 + 4 ((next >> 11) 2^-53), as a pair: the 53-bit
// integer (next >> 11) - 2^52 is cut into its upper 24 bits, the next 24 and 5 dropped ones
// (2^-46 of a cell).
__device__ __forceinline__ float2 jitter_pair(unsigned long long x) {
  const long long v = (long long)(x >> 11) - (1ll << 52);
  const int hi = (int)(v >> 29), mid = (int)((v >> 5) & 0xffffffll);
  return make_float2((float)hi * (1.f / 4194304.f), (float)mid * (1.f / 70368744177664.f));
}

struct PartArgs {
  int n, first;           // particles per side, axis of blockIdx.y = 0
  long long np;           // n^3
  const float* disp[3];   // displacement field along each axis (n^3, already * force_resolution)
  const float2* space;    // lattice coordinate per axis index (zeldovich.py:79)
  float2 lin;             // Dt(A_INIT)
  float2 vcoef;           // A_INIT * f_0 * h_0 * Dt
  float ncells;
  const ulonglong2* jump; // JIT_NT entries of (M^(t+1), 1 + M + .. + M^t), low and high words
  unsigned long long st_hi, st_lo, inc_hi, inc_lo;  // PCG64 state before the first draw
  float* pos;             // (3, np)
  float* vel;
};

// A block takes JIT_NT * JIT_ROUNDS consecutive particles of axis first + blockIdx.y (coalesced); its
// first thread jumps the generator there, and thread t reaches its draws by one jump of t + 1
// steps and then jumps of JIT_NT (one 128-bit multiply-add each).
__global__ void __launch_bounds__(JIT_NT) k_zeld_particles(PartArgs a) {
  chain_begin();
  __shared__ unsigned long long s_base[2];
  const int dir = a.first + blockIdx.y;
  const long long p0 = (long long)blockIdx.x * (JIT_NT * JIT_ROUNDS);
  const u128 inc = ((u128)a.inc_hi << 64) | a.inc_lo;
  if (threadIdx.x == 0) {
    // draw number dir * np + p is the (dir * np + p + 1)-th step of the generator
    const u128 b = pcg_advance(((u128)a.st_hi << 64) | a.st_lo, inc, (unsigned long long)(dir * a.np + p0));
    s_base[0] = (unsigned long long)b;
    s_base[1] = (unsigned long long)(b >> 64);
  }
  auto word = [](ulonglong2 w) { return ((u128)w.y << 64) | w.x; };
  const u128 m = word(__ldg(&a.jump[2 * threadIdx.x])), c = word(__ldg(&a.jump[2 * threadIdx.x + 1]));
  const u128 mr = word(__ldg(&a.jump[2 * (JIT_NT - 1)])), cr = word(__ldg(&a.jump[2 * (JIT_NT - 1) + 1])) * inc;
  __syncthreads();
  u128 s = m * (((u128)s_base[1] << 64) | s_base[0]) + c * inc;
  const unsigned u = (unsigned)a.n;
  const float* __restrict__ disp = a.disp[dir];
  float* __restrict__ pos = a.pos + dir * a.np;
  float* __restrict__ vel = a.vel + dir * a.np;
  for (int k = 0; k < JIT_ROUNDS; ++k, s = mr * s + cr) {
    const long long p = p0 + k * JIT_NT + threadIdx.x;
    if (p >= a.np) break;
    const float2 jit = jitter_pair(pcg_output(s));
    const unsigned i = (unsigned)p;
    const unsigned id = dir == 0 ? i / (u * u) : (dir == 1 ? i / u % u : i % u);
    const float d = __ldg(&disp[p]);
    const float2 x0 = __ldg(&a.space[id]), ld = pair_mul(a.lin, d);
    const float2 t1 = two_sum(x0.x, ld.x), t2 = two_sum(t1.x, jit.x);
    const float lo = __fadd_rn(__fadd_rn(__fadd_rn(x0.y, ld.y), jit.y), __fadd_rn(t1.y, t2.y));
    pos[p] = pair_mod(two_sum(t2.x, lo), a.ncells);
    const float2 v = pair_mul(a.vcoef, d);
    vel[p] = __fadd_rn(v.x, v.y);
  }
}

}  // namespace

// descriptors of an object's transforms
enum IcSim : int { SIM_FIELD_INV = 0, SIM_FIELD_FWD, SIM_DISP, IC_SIMS = SIM_DISP + 3 };

// Directions of the displacement whose transforms run together.  Three keep the launches of a small
// lattice few and its passes full (128^3: 18 launches instead of 28) and make their spectra in one pass, but
// take three spectra and grids where one after another takes two and one: 3.3 GB instead of 1.7 at
// 512^3 and 26 instead of 13 at 1024^3, for 7.1 ms instead of 8.1 at 512^3.
constexpr int ic_together(int n) { return n <= 256 ? 3 : 1; }

struct pm_ics {
  int n = 0, device = 0, sms = 1, m2max = 0;
  Tables tab;
  DBuf pool;              // all of the object's memory, one after another:
  Sim* d_sim = nullptr;   // (down to d_err: written by create)
  CUtensorMap* d_maps = nullptr;  // null: no tensor maps
  int* d_prefix = nullptr;
  ulonglong2* jump = nullptr;
  int* d_err = nullptr;
  double *shape = nullptr, *partial = nullptr, *norm = nullptr;
  float2 *amp = nullptr, *disp = nullptr, *space = nullptr;
  float2* spec[3] = {};
  float* grid[3] = {};
  int h_err = 0;
  std::string err;
};

namespace {

int ic_fail(pm_ics* g, int code, const std::string& msg) {
  if (g) g->err = msg;
  return code;
}

int ic_cuda(pm_ics* g, cudaError_t e, const char* where) {
  return ic_fail(g, e == cudaErrorMemoryAllocation ? PM_ERR_OOM : PM_ERR_CUDA,
                 std::string(where) + ": " + cudaGetErrorString(e));
}

#define IC_CK(call, where)                                 \
  do {                                                     \
    cudaError_t e_ = (call);                               \
    if (e_ != cudaSuccess) return ic_cuda(g, e_, where);   \
  } while (0)

// cosmology.py:11-36 with the cosmology list [OMEGA_M0, OMEGA_LAMBDA0, OMEGA_K0]
double cosmo_H(double a, double h0, double om, double ol, double ok) {
  return std::sqrt(std::pow(h0, 2.0) * (om / std::pow(a, 3.0) + ok / std::pow(a, 2.0) + ol));
}
double cosmo_Dt(double a, double om, double ol, double ok) {
  (void)ok;
  return 5.0 / 2.0 / om / (std::pow(om, 4.0 / 7.0) - ol + (1.0 + om / 2.0) * (1.0 + ol / 70.0)) * a;
}

}  // namespace

extern "C" {

int pm_ics_create(int n_parts, int device, pm_ics** out) {
  if (!out) return PM_ERR_ARG;
  *out = nullptr;
  if (!spectral_supported(n_parts)) return PM_ERR_ARG;
  pm_ics* g = new pm_ics();
  g->n = n_parts;
  g->device = device;
  const int n = n_parts, h = n / 2;
  g->m2max = 3 * h * h;
  // (sb: a multiple of 128 bytes, which the tensor maps and the row transforms rely on)
  const size_t sb = (size_t)n * n * spec_pitch(n) * sizeof(float2), gb = (size_t)n * n * n * sizeof(float);
  cudaError_t e = cudaSetDevice(device);
  if (!e) g->sms = sm_count(device);
  if (!e) e = g->tab.build(n);
  size_t at = 0;
  auto part = [&](size_t bytes) {
    const size_t o = at;
    at += (bytes + 255) / 256 * 256;
    return o;
  };
  const size_t tables = (size_t)(g->m2max + 1);
  const int ngrids = ic_together(n), nspecs = ngrids < 2 ? 2 : ngrids;
  const size_t o_sim = part(IC_SIMS * sizeof(Sim)), o_maps = part(2 * IC_SIMS * sizeof(CUtensorMap)),
               o_pre = part(8 * sizeof(int)), o_jump = part(2 * JIT_NT * sizeof(ulonglong2)), o_err = part(sizeof(int)),
               filled = at, o_shape = part(tables * sizeof(double)), o_amp = part(tables * sizeof(float2)),
               o_disp = part(tables * sizeof(float2)), o_partial = part(NORM_BLOCKS * sizeof(double)),
               o_norm = part(sizeof(double)), o_space = part(n * sizeof(float2)), o_spec = part(nspecs * sb),
               o_grid = part(ngrids * gb);
  if (!e) e = g->pool.ensure(at);
  if (!e) {
    char* base = g->pool.as<char>();
    g->d_sim = reinterpret_cast<Sim*>(base + o_sim);
    g->d_prefix = reinterpret_cast<int*>(base + o_pre);
    g->jump = reinterpret_cast<ulonglong2*>(base + o_jump);
    g->d_err = reinterpret_cast<int*>(base + o_err);
    g->shape = reinterpret_cast<double*>(base + o_shape);
    g->amp = reinterpret_cast<float2*>(base + o_amp);
    g->disp = reinterpret_cast<float2*>(base + o_disp);
    g->partial = reinterpret_cast<double*>(base + o_partial);
    g->norm = reinterpret_cast<double*>(base + o_norm);
    g->space = reinterpret_cast<float2*>(base + o_space);
    for (int i = 0; i < nspecs; ++i) g->spec[i] = reinterpret_cast<float2*>(base + o_spec + i * sb);
    for (int i = 0; i < ngrids; ++i) g->grid[i] = reinterpret_cast<float*>(base + o_grid + i * gb);
    std::vector<char> h(filled, 0);
    // descriptors: the field's inverse and forward transforms, the displacements' inverses
    bool ok = true;
    for (int i = 0; i < IC_SIMS; ++i) {
      const int sp = i == SIM_FIELD_INV ? 1 : (i == SIM_FIELD_FWD ? 0 : (ngrids == 3 ? i - SIM_DISP : 1));
      const int gr = i < SIM_DISP || ngrids == 1 ? 0 : i - SIM_DISP;
      Sim d{};
      d.n = n;
      d.pitch = spec_pitch(n);
      d.s2 = g->tab.s2.as<float>();
      d.tw = g->tab.tw.as<float2>();
      d.spec = g->spec[sp];
      d.rho = d.phi = g->grid[gr];
      std::memcpy(h.data() + o_sim + i * sizeof(Sim), &d, sizeof(d));
      CUtensorMap m[2];
      std::memset(m, 0, sizeof(m));
      ok = ok && spectral_encode_maps(n, d.spec, m);
      std::memcpy(h.data() + o_maps + 2 * i * sizeof(CUtensorMap), m, sizeof(m));
    }
    if (ok) g->d_maps = reinterpret_cast<CUtensorMap*>(base + o_maps);
    const int ux = (int)spectral_units(SPEC_X_R2C, n), ul = (int)spectral_units(SPEC_Y_FWD, n);
    const int pre[8] = {0, ux, 2 * ux, 3 * ux, 0, ul, 2 * ul, 3 * ul};
    std::memcpy(h.data() + o_pre, pre, sizeof(pre));
    u128 m = 1, c = 0;  // the generator's jumps by 1 .. JIT_NT steps
    for (int t = 0; t < JIT_NT; ++t) {
      c = c * pcg_mult() + 1;  // 1 + M + .. + M^t
      m *= pcg_mult();
      const unsigned long long w[4] = {(unsigned long long)m, (unsigned long long)(m >> 64), (unsigned long long)c,
                                       (unsigned long long)(c >> 64)};
      std::memcpy(h.data() + o_jump + t * sizeof(w), w, sizeof(w));
    }
    e = cudaMemcpy(g->pool.p, h.data(), filled, cudaMemcpyHostToDevice);
  }
  if (!e) e = spectral_dispatch(SPEC_PREPARE, n, nullptr, Work(), 0, nullptr);
  if (!e) e = cudaDeviceSynchronize();
  if (e) {
    pm_ics_destroy(g);
    return e == cudaErrorMemoryAllocation ? PM_ERR_OOM : PM_ERR_CUDA;
  }
  *out = g;
  return PM_OK;
}

void pm_ics_destroy(pm_ics* g) {
  if (!g) return;
  cudaSetDevice(g->device);
  g->pool.release();
  g->tab.release();
  delete g;
}

const char* pm_ics_last_error(const pm_ics* g) { return g ? g->err.c_str() : "null initial-conditions object"; }

int pm_ics_generate(pm_ics* g, const pm_config* cfg, const pm_ic_params* ic, const float* u, const float* v,
                    float* positions, float* velocities, float* grf, void* stream) {
  if (!g) return PM_ERR_ARG;
  if (!cfg || !ic || !u || !v || !positions || !velocities) return ic_fail(g, PM_ERR_ARG, "null argument");
  if (cfg->n_parts != g->n) return ic_fail(g, PM_ERR_ARG, "n_parts differs from the object's size");
  if (cfg->n_cells <= 0 || !(cfg->box_size > 0.0) || !(cfg->omega_m0 != 0.0) || !(cfg->a_init > 0.0))
    return ic_fail(g, PM_ERR_ARG, "invalid configuration");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  IC_CK(cudaSetDevice(g->device), "set device");
  const int n = g->n, pitch = spec_pitch(n);
  const long long np = (long long)n * n * n;
  const double om = cfg->omega_m0, ob = cfg->omega_b0, ok = cfg->omega_k0, ol = cfg->omega_lambda0,
               h0 = cfg->h0, a0 = cfg->a_init, box = cfg->box_size, ncells = cfg->n_cells;

  const Launch lc(st, n <= 256);  // (pm_launch.cuh)
  const double npix = (double)np, res = ncells / n, fres = ncells / box;

  // power spectrum, its normalisation and the other tables
  TableArgs ta;
  ta.m2max = g->m2max;
  ta.n = n;
  ta.shape = g->shape;
  ta.disp = g->disp;
  ta.space = g->space;
  // l(m) = (2 pi n / box) fftfreq(n)[m] = l0 m; the displacement spectrum times resolution,
  // force resolution and the 1/n^3 of ifftn
  ta.coef_l0 = res * fres / npix / (2.0 * M_PI / box);
  ta.stop = ncells - res;
  ta.step = n > 1 ? ta.stop / (n - 1) : 0.0;
  ta.sp.kscale = 2.0 * M_PI / box;
  ta.sp.gamma = om * h0 * std::exp(-ob - ob / om);
  ta.sp.power = ic->power;
  ta.sp.lcdm = ic->lcdm_transfer ? 1 : 0;
  const int tb = (g->m2max + 128) / 128;
  IC_CK(launch_chained(k_tables, tb, 128, 0, lc, ta), "tables");
  IC_CK(launch_chained(k_norm_partial, NORM_BLOCKS, NORM_NT, 0, lc, g->shape, n, g->partial),
        "norm");
  IC_CK(launch_chained(k_norm_final, 1, NORM_NT, 0, lc, g->partial,
                       64.0 * std::pow(h0, 2.0) * (npix * npix), g->norm),
        "norm final");
  const double lin = cosmo_Dt(a0, om, ol, ok);
  // P(k = 0) / A: the reference's k**POWER * lcdm (or div) at k = 0
  const double p0 = (ic->power >= 0.0 && !ic->lcdm_transfer && ic->power == 0.0) ? 1.0 : 0.0;
  IC_CK(launch_chained(k_amp, tb, 128, 0, lc, g->shape, g->norm, g->m2max, p0, lin * lin,
                       1.0 / npix, g->amp),
        "amplitudes");
  GrfArgs ga;
  ga.n = n;
  ga.pitch = pitch;
  ga.u = u;
  ga.v = v;
  ga.amp = g->amp;
  ga.spec = g->spec[1];
  const int ew = grid_for(((long long)n * n * pitch + IC_NT - 1) / IC_NT, g->sms, 8);
  IC_CK(launch_chained(k_grf_fill, ew, IC_NT, 0, lc, ga), "grf fill");

  const Sim* ds = g->d_sim;
  const CUtensorMap* maps = g->d_maps;
  int* err = g->d_err;
  const int* pre = g->d_prefix;
  // one transform pass of `count` descriptors from `first` on
  auto pass = [&](SpecKind kind, int first, int count, const char* what) -> int {
    const bool xk = kind == SPEC_X_R2C || kind == SPEC_X_C2R;
    const Work w{pre + (xk ? 0 : 4), count, count * (int)spectral_units(kind, n)};
    IC_CK(spectral_dispatch(kind, n, ds + first, w, grid_for(w.total, g->sms, 8), lc, maps ? maps + 2 * first : nullptr,
                            err),
          what);
    return PM_OK;
  };
  auto inverse = [&](int first, int count, const char* what) -> int {
    if (int r = pass(SPEC_Z_INV, first, count, what)) return r;
    if (int r = pass(SPEC_Y_INV, first, count, what)) return r;
    return pass(SPEC_X_C2R, first, count, what);
  };
  if (int r = inverse(SIM_FIELD_INV, 1, "grf inverse")) return r;
  if (grf)
    IC_CK(cudaMemcpyAsync(grf, g->grid[0], (size_t)np * sizeof(float), cudaMemcpyDeviceToDevice, st), "grf out");

  // fftn of the field (zeldovich.py:17)
  if (int r = pass(SPEC_X_R2C, SIM_FIELD_FWD, 1, "r2c")) return r;
  if (int r = pass(SPEC_Y_FWD, SIM_FIELD_FWD, 1, "y fwd")) return r;
  if (int r = pass(SPEC_Z_FWD, SIM_FIELD_FWD, 1, "z fwd")) return r;

  const double f0 = 1.0 / std::sqrt((om + ok * a0 + ol * std::pow(a0, 3.0)) / a0);
  const double hh = cosmo_H(a0, h0, om, ol, ok);
  ZelArgs za;
  PartArgs pa;
  za.n = n;
  za.pitch = pitch;
  za.disp = g->disp;
  za.in = g->spec[0];
  pa.n = n;
  pa.np = np;
  pa.space = g->space;
  pa.lin = split(lin);
  pa.vcoef = split(a0 * f0 * hh * lin);
  pa.ncells = (float)ncells;
  pa.jump = g->jump;
  pa.st_hi = ic->jitter_state[0];
  pa.st_lo = ic->jitter_state[1];
  pa.inc_hi = ic->jitter_inc[0];
  pa.inc_lo = ic->jitter_inc[1];
  pa.pos = positions;
  pa.vel = velocities;
  const unsigned pb = (unsigned)((np + JIT_NT * JIT_ROUNDS - 1) / (JIT_NT * JIT_ROUNDS));
  const int together = ic_together(n);
  for (int first = 0; first < 3; first += together) {
    pa.first = first;
    for (int d = 0; d < 3; ++d) {
      const bool now = d >= first && d < first + together;
      za.out[d] = now ? g->spec[together == 3 ? d : 1] : nullptr;
      pa.disp[d] = now ? g->grid[together == 3 ? d : 0] : nullptr;
    }
    IC_CK(launch_chained(k_zeld_spectrum, ew, IC_NT, 0, lc, za), "displacement spectrum");
    if (int r = inverse(SIM_DISP + first, together, "displacement inverse")) return r;
    k_zeld_particles<<<dim3(pb, together), JIT_NT, 0, st>>>(pa);
    IC_CK(cudaGetLastError(), "particles");
  }
  // device-side checks of the TMA passes (bounded waits): read back once
  IC_CK(cudaMemcpyAsync(&g->h_err, g->d_err, sizeof(int), cudaMemcpyDeviceToHost, st), "err");
  IC_CK(cudaStreamSynchronize(st), "sync");
  const int bits = g->h_err;
  if (bits) {
    cudaMemsetAsync(g->d_err, 0, sizeof(int), st);
    return ic_fail(g, PM_ERR_DEVICE, "device check failed in the spectral passes (bits " + std::to_string(bits) + ")");
  }
  return PM_OK;
}

}  // extern "C"
