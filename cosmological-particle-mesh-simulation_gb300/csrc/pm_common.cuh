// Shared device/host declarations of the GB300 particle-mesh engine.
//
// Data layout in HBM (one simulation):
//   real grids (density, potential)  float  [z][y][x], n^3
//   half spectrum                    float2 rows of kx in [0, n/2], row pitch `pitch` (a multiple
//                                    of 16 complex = 128 B), rows in the order of spec_row
//   particles                        structure of arrays, one float per axis and
//                                    per quantity (the reference's (3, Np) layout)
// Many simulations share one launch per phase: every kernel receives the device
// array of `Sim` descriptors and a per-phase work prefix (CTA -> simulation).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "pm_launch.cuh"

#include <atomic>
#include <mutex>

#define PM_FIX_BITS 26          // CIC weights are accumulated as integers w * 2^26
#define PM_MAX_N 1024

namespace pm {

constexpr int PM_MAX_DEVICES = 64;

// Kernel attributes (dynamic shared-memory limits, carve-outs) are state of each device,
// not of the process: DeviceOnce runs a set-up function once for every device it is called
// on (the current device), under a lock, and remembers the devices whose set-up succeeded.
struct DeviceOnce {
  std::atomic<unsigned long long> done{0};
  std::mutex m;
  template <class F>
  cudaError_t run(F fn) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e) return e;
    if (dev < 0 || dev >= PM_MAX_DEVICES) return cudaErrorInvalidDevice;
    const unsigned long long bit = 1ull << dev;
    if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
    std::lock_guard<std::mutex> g(m);
    if (done.load(std::memory_order_relaxed) & bit) return cudaSuccess;
    e = fn();
    if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
    return e;
  }
};

// Streaming multiprocessors of the current device (cached per device).
inline int device_sms() {
  static std::atomic<int> cache[PM_MAX_DEVICES];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= PM_MAX_DEVICES) return 1;
  int v = cache[dev].load(std::memory_order_relaxed);
  if (v <= 0) {
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 1;
    cache[dev].store(v, std::memory_order_relaxed);
  }
  return v;
}

enum : int {
  ERR_OK = 0,
  ERR_CELL_RANGE = 1,   // a particle cell fell outside the grid (NaN/Inf position)
  ERR_SOURCE_ROW = 2,   // deposit: particle outside the tile's source rows (sort broken)
  ERR_NONFINITE = 4,    // kick/drift produced a non-finite coordinate
  ERR_TIMEOUT = 8,      // a bounded wait on an asynchronous copy gave up
};

// Row bins: the drop-in step and the resident engine group particles by x-row and, inside a row, by
// blocks of 128 cells (256 above 512 cells a side; the last block may be short).  The deposit
// needs rows only, but the lanes of the kick then read potential taps next to one another:
// resident kick 516 -> 469 us early and 489 -> 453 us clustered (256^3 on 512^3), for 6 us more in
// the sort.  Blocks of 64 cells give the kick 2-6 us more and cost the sort 6; 32 cells, 20.
__host__ __device__ constexpr int x_shift(int n) { return n <= 512 ? 7 : 8; }
__host__ __device__ constexpr int x_bins(int n) { return ((n - 1) >> x_shift(n)) + 1; }
__host__ __device__ constexpr unsigned row_bins(int n) { return (unsigned)n * (unsigned)n * (unsigned)x_bins(n); }

// Place of the row (y, z) of a half spectrum: [z][y], and from 768 cells a side on the planes of one
// block of 32 y together, [y / 32][z][y % 32].  The z pass walks a column through all planes, and
// with a plane of 2.5 or 4.3 MB between its rows every row is in a memory page of its own; in
// blocks both the y and the z pass stay within some tens of pages (z of 1024: 3.48 -> 2.67 ms, y
// the same; blocks of 8 to 64 alike).  On 512 (1.1 MB) z gains 1% and y loses 5%.
__host__ __device__ constexpr int spec_block(int n) { return n >= 768 ? 32 : n; }
__host__ __device__ constexpr long long spec_row(int n, int y, int z) {
  const int b = spec_block(n);
  return ((long long)(y / b) * n + z) * b + y % b;
}
// the y and z of row r
__host__ __device__ constexpr int spec_row_y(int n, long long r) {
  const int b = spec_block(n);
  return (int)(r / ((long long)b * n)) * b + (int)(r % b);
}
__host__ __device__ constexpr int spec_row_z(int n, long long r) { return (int)(r / spec_block(n) % n); }

enum PosMode : int { POS_ABS = 0, POS_DISP = 1 };

// Device-side description of one simulation.  All pointers are device pointers.
struct Sim {
  int n;            // grid cells per side
  int pitch;        // spectrum row pitch in complex elements
  int np1;          // particles per side of the Lagrangian lattice (0: unknown)
  int xbits;        // bits of x in the cell key
  int ty, tz;       // deposit tile: tz planes x ty rows of full x-rows
  int flags;
  int q_step;       // n / np1 when np1 divides n (lattice q = q_step i + 1/2); 0: use the tables
  long long np;        // particle count
  long long part_off;  // first position of this simulation in the sorted order (and in the
                       // state the kick writes: the batch particle arrays after a step)
  long long slot_off;  // first particle slot of this simulation in the state being read by the
                       // keys kernel (differs from part_off right after a retirement)
  unsigned row_base;   // first global row (xbits != 0) or row-bin (xbits == 0) of this simulation
  int started;         // 0 until the first step of the plan (step_coefficients)
  float* rho;          // density n^3 (output of the deposit)
  float2* spec;        // half spectrum (rows in the order of spec_row)
  float* phi;          // potential n^3
  const float* fgrid;  // optional caller Green table n^3 (nullptr: computed in-kernel)
  const float* s2;     // sin^2(pi m / n), m < n
  const float2* tw;    // exp(-2 pi i m / n), m < n
  const int* q_int;    // lattice coordinate, integer part, np1 entries
  const float* q_frac; // lattice coordinate, fractional part, np1 entries
  const float* sn;     // sin(2 pi m / n), m < n (spectral gradient)
  // spectral gradient: grad_axis = d + 1 makes the z pass multiply by -i sin(k_d) as well as
  // by the Green function, so that the inverse passes give the force grid of axis d; grad, for
  // the kick, holds the three force grids (nullptr: central differences of phi)
  int grad_axis, pad2;
  const float* grad[3];
  // per-step coefficients
  float mass_scale;    // particle mass * 2^-PM_FIX_BITS
  float green;         // -3 Om / (8 a) / n^3
  float kick;          // da * f(a + da)
  float drift;         // da * f(a + da) / (a + da)^2
  // time state (fp64, advanced on the device in resident mode)
  double a, da, om, ol, ok, h0;
  int step, nsteps, active, fix_f;
};

// The coefficients of the step at hand, in fp64 (integrate.py:11-13, potential.py:15,
// cosmology.py:20-27); every step but a plan's first moves the scale factor on.  (A resident step
// has one thread per simulation do it in the sort's scatter: a kernel of its own took 4 us.)
__device__ __forceinline__ void step_coefficients(Sim& S) {
  if (S.started) {
    S.a += S.da;
    S.step += 1;
  }
  S.started = 1;
  const double a = S.a, da = S.da, a1 = a + da;
  const double n3 = (double)S.n * S.n * S.n;
  S.green = (float)(-3.0 * S.om / 8.0 / a / n3);
  // integrate.py:12 passes [H0, OL, OK]: H0 in the Omega_m slot unless fix_f is set
  const double om_slot = S.fix_f ? S.om : S.h0;
  const double fa1 = 1.0 / sqrt((om_slot + S.ok * a1 + S.ol * a1 * a1 * a1) / a1);
  S.kick = (float)(da * fa1);
  S.drift = (float)(da / (a1 * a1) * fa1);
}

// CTA -> simulation map of one phase: prefix[s] = first work unit of simulation s.
struct Work {
  const int* prefix;  // nsims + 1 entries (device)
  int nsims;
  int total;          // prefix[nsims]
};

// Work table of a drop-in call (one simulation): (0, units) of each phase.
enum CallPhase : int { CALL_KEYS = 0, CALL_DEP, CALL_X, CALL_LINE, CALL_PHASES };
struct CallWork {
  int prefix[CALL_PHASES][2];
};

// Particle arrays of a batch (structure of arrays, indexed by slot).
struct Parts {
  float* x; float* y; float* z;       // positions (POS_ABS) or displacements (POS_DISP)
  float* vx; float* vy; float* vz;
  unsigned* id;                        // Lagrangian particle index (POS_DISP)
  // cell record (POS_DISP, optional), one 16-byte word per particle: the base cell packed
  // x | y << 10 | z << 20 (CELL_BAD if not finite) and the bits of the three in-cell offsets,
  // exactly as computed from the displacement.  The kick writes it with the state so that the
  // deposit reads the cell instead of recomputing it, with one 16-byte load (four separate
  // arrays measured 0.520 -> 0.485 ms per deposit, 256^3 on 512^3).
  uint4* rec;
};

__device__ __forceinline__ int locate_sim(const Work& w, int unit) {
  int lo = 0, hi = w.nsims - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(&w.prefix[mid]) <= unit) lo = mid; else hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ void set_error(int* err, int code) {
  if (err) atomicOr(err, code);
}

// ---------------------------------------------------------------------------------
// Launchers (defined in the .cu files, called by the engine)
// ---------------------------------------------------------------------------------
// spectral passes: one kernel per grid size n (supported n: spectral_supported)
enum SpecKind : int { SPEC_X_R2C = 0, SPEC_Y_FWD, SPEC_Z_GREEN, SPEC_Z_TABLE, SPEC_Y_INV, SPEC_X_C2R,
                      SPEC_Z_FWD, SPEC_Z_INV, /* plain z transforms (initial conditions) */
                      SPEC_Z_GRAD, /* z Green times -i sin(k_d): spectral gradient of axis grad_axis - 1 */
                      SPEC_PREPARE /* only set kernel attributes */ };
// maps: device array of tensor maps, two per simulation of `sims` (y pass, z pass; see
// spectral_encode_maps) -- enables the TMA-streamed line passes; nullptr falls back to
// plain loads.  Every kernel finds its simulation through the work prefix.
template <int N>
cudaError_t spectral_launch(SpecKind kind, const Sim* sims, Work w, int ctas, Launch st,
                            const CUtensorMap* maps, int* err);
// Encodes the y- and z-pass tensor maps of a half spectrum of size n (false if n has no
// TMA line pass).
bool spectral_encode_maps(int n, const void* spec, CUtensorMap out[2]);
bool spectral_supported(int n);
// work units (CTAs' worth of work) of one spectral pass for a grid of size n
long long spectral_units(SpecKind kind, int n);
// resident CTAs per SM of a spectral pass for size n (for persistent grid sizing)
cudaError_t spectral_dispatch(SpecKind kind, int n, const Sim* sims, Work w, int ctas, Launch st,
                              const CUtensorMap* maps = nullptr, int* err = nullptr);
cudaError_t launch_fourier_grid(const Sim* sims, int ctas, Launch st);
// fused deposit + x R2C (the density grid is not written); ctas <= 0 only prepares.
// next_tile: four device words, 0 at the start: the tile counter, and of `dense`, a list (room for
// w.total) of the tiles whose sums need two words, the count from its front, the counter of its work and
// the count from its back.  order (optional, w.total entries): the tiles in the order to
// take them (launch_tile_order).
template <int N>
cudaError_t deposit_r2c_launch(const Sim* sims, Work w, Parts p, const unsigned* perm, const unsigned* row_start,
                               const unsigned* group_max, int* err, unsigned* next_tile, const unsigned* order,
                               unsigned* dense, int ctas, Launch st);
bool deposit_r2c_supported(int n);
bool xrow_supported(int n);  // the x passes of size n transform rows in registers (their grid is tunable)
int deposit_r2c_ctas_per_sm(int n);  // resident CTAs per SM of the fused deposit
cudaError_t deposit_r2c_dispatch(int n, const Sim* sims, Work w, Parts p, const unsigned* perm,
                                 const unsigned* row_start, const unsigned* group_max, int* err, unsigned* next_tile,
                                 const unsigned* order, unsigned* dense, int ctas, Launch st);

// sum of the first n_slices planes of an n^3 grid, float64 n^2 output (pm_diagnostics.cu)
cudaError_t launch_project(const float* rho, int n, int n_slices, double* out, int ctas, cudaStream_t st);
// shell-averaged power spectrum of a half spectrum (pm_diagnostics.cu): out = (k, P, modes) for bins
// 1 .. nbins - 1; nbins <= n / 2 + 1; partial holds pk_partial_doubles(nbins) doubles
int pk_ctas();
size_t pk_partial_doubles(int nbins);
cudaError_t launch_power_spectrum(const float2* spec, int n, int pitch, int nbins, double box, double* partial,
                                  double* out, cudaStream_t st);

// particle kernels
cudaError_t launch_keys_abs(const Sim* sims, const Work& w, Parts p, unsigned* keys, unsigned* vals,
                            int* err, int ctas, Launch st);
cudaError_t launch_keys_disp(const Sim* sims, const Work& w, Parts p, unsigned* keys, unsigned* vals,
                             int* err, int ctas, Launch st);
cudaError_t launch_row_start(const unsigned* keys, long long n, int xbits, unsigned nrows,
                             unsigned* row_start, Launch st);
cudaError_t launch_deposit(const Sim* sims, const Work& w, Parts p, const unsigned* perm,
                           const unsigned* row_start, const unsigned* group_max, int mode, int* err, int ctas,
                           size_t smem, Launch st);
constexpr int KICK_UNIT = 512;  // particles per work unit of the kick
// resident kick: the state in row order (through perm), the next keys and their row histogram
cudaError_t launch_kick(const Sim* sims, const Work& w, Parts in, Parts out, const unsigned* perm,
                        unsigned* keys_next, int* err, int ctas, Launch st, unsigned* row_count);
// ---- drop-in step on (3, np) arrays in the caller's order (see pm_particles.cu) ----
// descriptor and work table of one call (from kernel arguments); zero_bytes: a multiple of 16
cudaError_t launch_call_begin(Sim* dsim, CallWork* dwork, const Sim& sim, const CallWork& work, void* zero,
                              size_t zero_bytes, Launch st);
// np1: particles per side when np = np1^3 (they may be in lattice order), else 0
// row key and rank inside its row of every particle; count (zero before) ends as the row counts;
// vote (np1; 0 before): positive if the particles are in lattice order
cudaError_t launch_row_rank(const float* pos, long long np, int np1, int n, unsigned* count, unsigned* keys,
                            unsigned* ranks, int* err, float* copy, int* vote, Launch st);
// cell records in row order, taken in boxes of the lattice if the vote is for it; place: in the keys,
// out each particle's place in row order
cudaError_t launch_row_place(const float* pos, long long np, int np1, int n, const unsigned* row_start,
                             const unsigned* ranks, unsigned* place, uint4* rec, const int* vote, Launch st);
// rec: in the cell records, out the forces (3 floats in the first words of each entry)
cudaError_t launch_force(const Sim* sims, long long np, uint4* rec, int sms, Launch st);
cudaError_t launch_advance(const Sim* sims, long long np, const uint4* force, const unsigned* place,
                           const float* pos, const float* vel, float* pos_out, float* vel_out, int* err, Launch st);
cudaError_t deposit_prepare();  // sets kernel attributes of the current device (call before graph capture)
// order of the fused deposit's tiles (dense tiles first); counts: 2 device words, 0 when the kernel starts
cudaError_t launch_tile_order(const Sim* sims, const Work& w, const unsigned* row_start, unsigned* order,
                              unsigned* counts, int sms, Launch st);
cudaError_t launch_abs_to_disp(const float* pos, const float* vel, long long np, int np1, int n,
                               const int* q_int, const float* q_frac, Parts out, long long off,
                               Launch st, const unsigned* order);
// keys[i] = row bin (rows in tile order) of the cell of absolute position i
cudaError_t launch_row_keys_abs(const float* pos, long long np, int n, unsigned* keys, Launch st);
cudaError_t launch_disp_to_abs(Parts in, long long off, long long np, int np1, int n, const int* q_int,
                               const float* q_frac, float* pos, float* vel, Launch st);
size_t deposit_smem_bytes(int n, int ty, int tz);

// radix sort of (key, value) pairs, stable, LSD, digits of up to 9 bits
struct SortScratch {
  unsigned* keys_alt; unsigned* vals_alt;
  unsigned* hist;     // 256 * max_blocks
  unsigned* digit_tot;
  long long capacity; int max_blocks;
};
constexpr int SORT_TILE = 4096;
size_t sort_scratch_hist_entries(long long n);
constexpr int SORT_DIGIT_TOTALS = 512;  // entries of SortScratch::digit_tot
int radix_sort_passes(int bits);
// sets the sort's kernel attributes on the current device (once per device; radix_sort calls it)
cudaError_t sort_prepare();
// Sorts keys[0,n) / vals[0,n) on key bits [begin_bit, begin_bit + bits).  Returns via
// *in_alt whether the result sits in the scratch (alt) buffers.  When gen_vals is set,
// vals are not read on the first pass and the identity 0..n-1 is used instead.
cudaError_t radix_sort(unsigned* keys, unsigned* vals, long long n, int begin_bit, int bits, bool gen_vals,
                       const SortScratch& s, bool* in_alt, Launch st);
// Groups n row keys (< nrows) by row: row_start[0..nrows] (exclusive prefix of the row
// counts) and perm[j] = index of the j-th key in row order (order inside a row not
// specified).  Scratch: count and cursor (nrows each), block_sums (row_sort_block_sums).
size_t row_sort_block_sums(unsigned nrows);
// counted: count already holds the row histogram of keys (else it is zeroed and computed here);
// zero: count is cleared once read; group_max: see row_scan; clear: nclear words set to 0; sims:
// nsims simulations brought to the step at hand (step_coefficients).
cudaError_t row_counting_sort(const unsigned* keys, long long n, unsigned nrows, unsigned* count,
                              unsigned* row_start, unsigned* cursor, unsigned* block_sums, unsigned* perm, int* err,
                              int sms, Launch st, bool counted = false, bool zero = false,
                              unsigned* group_max = nullptr, unsigned* clear = nullptr, int nclear = 0, Sim* sims = nullptr,
                              int nsims = 0);
// row_start[0..nrows]: exclusive prefix of count; cursor (optional): a copy of its first nrows
// entries; zero: count is cleared once read; group_max (optional): the largest count of each 16
// consecutive bins, for the deposit (pm_deposit.cuh).  All arrays 16-byte aligned.
cudaError_t row_scan(unsigned* count, unsigned nrows, unsigned* row_start, unsigned* cursor, unsigned* block_sums,
                     bool zero, Launch st, unsigned* group_max = nullptr);
int row_scan_launches(unsigned nrows);  // its kernels
// count[r] = number of keys equal to r (count zeroed first)
cudaError_t row_histogram(const unsigned* keys, long long n, unsigned nrows, unsigned* count, int* err, int sms,
                          Launch st);

}  // namespace pm
