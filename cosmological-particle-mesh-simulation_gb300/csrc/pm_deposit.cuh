// Deterministic CIC deposit of one tile (density.py:7-48 of the reference).
//
// A tile is TZ x TY full x-rows.  The particles whose base cell lies in the tile's source
// rows (the tile plus one row and one plane below, periodic: 7 runs of the row-sorted
// order) are found through the row starts; their CIC weights that land inside the tile are
// added to integer accumulators in shared memory (TileSum: one 32-bit word per cell where the
// number of its source entries allows, else a low word and a high word).  Integer sums do
// not depend on the order of the atomics, so the deposit is bit-identical run to run.
#pragma once
#include <type_traits>

#include "pm_cells.cuh"

namespace pm {

constexpr int DEP_NT = 512;

// A two-word sum: the carry out of the low word, seen from the value that was there, is added to the
// high word.  It is rare, so a corner takes one atomic, as in a one-word sum; a second one for every
// corner (a word of q >> 12, from which the carries follow) cost the halos' tiles more (256^3
// particles on 512^3 at steps 400 / 600 / 980 of 1000: 222 / 266 / 338 us -> 175 / 216 / 254).
__device__ __forceinline__ void acc_add(unsigned* lo, unsigned* hi, int i, unsigned q) {
  if (atomicAdd(&lo[i], q) > ~q) atomicAdd(&hi[i], 1u);
}

// The exact sum V of low word l and high word h, rounded to float32, times scale.  V < 2^46 (a
// million particles in a cell), so V = a 2^23 + b with a, b < 2^23; each is exact as a float
// (2^23 + a has a as its mantissa), and fmaf(a, 2^23, b) rounds once: the value of a
// round-to-nearest 64-bit conversion, computed on the FP32 pipe (GB300 issues 64-bit integer
// conversions to its narrow FP64 pipe).  __fmul_rn: a contraction of the product with the transform's first sums would
// make the fused deposit differ from the written density.
__device__ __forceinline__ float fixed_to_float(unsigned l, unsigned h, float scale) {
  const unsigned a = (h << 9) | (l >> 23), b = l & 0x7fffffu;
  const float fa = __uint_as_float(0x4B000000u | a) - 8388608.f;
  const float fb = __uint_as_float(0x4B000000u | b) - 8388608.f;
  return __fmul_rn(fmaf(fa, 8388608.f, fb), scale);
}

// How a tile's sums are held.  Every corner weight is quantised to an integer q <= 2^s and
// added with integer atomics, so a cell's sum -- and the float made from it -- does not depend
// on the order of the additions.  A tile of up to ONE_WORD_TOTAL - 1 source entries sums in one 32-bit
// word per cell (one atomic per corner), at the largest s <= 26 that cannot overflow.  A cell
// receives at most one corner from each particle in four rows (y, y - 1, z, z - 1) and two cells of
// each (x, x - 1), which lie in one row bin or two adjacent ones: at most 4 or 8 times the largest count of a
// row bin of the tile and its three lower neighbours, and at most the tile's source entries, which
// alone would allow s = 20 to 26 (256^3 on 512^3 early: 21; with the bins 23 to 24).
// Denser tiles sum at 2^-26 in a low word and a high word: bounds from the
// bins would put most of them in one word too, but at s = 20 to 22, and the quantisation would
// then be the largest error of their density -- one particle per cell of 256^3, uniform:
// 3.4e-7 in relative L2 instead of 3.2e-8.
constexpr unsigned ONE_WORD_TOTAL = 4096;

struct TileSum {
  int s;     // one-word quantisation 2^s; 0: two-word sums at 2^-26
  float ms;  // particle mass * 2^-(quantisation bits): the float of a sum times ms is its mass
};

// total: source entries of the tile; cap: a cell receives at most that many corners
__device__ __forceinline__ TileSum tile_sum(unsigned total, unsigned cap, float mass_scale) {
  const int bits = 32 - __clz(min(total, cap));  // entries of a cell < 2^bits
  TileSum t;
  t.s = total < ONE_WORD_TOTAL ? min(PM_FIX_BITS, 32 - bits) : 0;
  // mass_scale = mass * 2^-26; one-word sums at 2^-s: times 2^(26 - s), exactly
  t.ms = t.s ? mass_scale * __uint_as_float((unsigned)(127 + PM_FIX_BITS - t.s) << 23) : mass_scale;
  return t;
}

// A one-word sum as a float, times scale (exact split l = a 2^23 + b, one rounding).
__device__ __forceinline__ float word_to_float(unsigned l, float scale) {
  const float fa = __uint_as_float(0x4B000000u | (l >> 23)) - 8388608.f;
  const float fb = __uint_as_float(0x4B000000u | (l & 0x7fffffu)) - 8388608.f;
  return __fmul_rn(fmaf(fa, 8388608.f, fb), scale);
}

// The float of a cell's sum: low word l (and, for two-word tiles, high word h).
__device__ __forceinline__ float sum_to_float(const TileSum& t, unsigned l, unsigned h) {
  return t.s ? word_to_float(l, t.ms) : fixed_to_float(l, h, t.ms);
}

// Adds the 8 quantised weights q of a particle with base cell (cx, ly, lz) (ly, lz relative
// to the tile, in [-1, TY-1] x [-1, TZ-1]) to the tile accumulators; tile row r of lo / hi
// starts at word r * rs.  The corners go row by row (weights 0 1 | 2 4 | 3 5 | 6 7 of the
// order of cic_weights lie in rows (y, z), (y + 1, z), (y, z + 1), (y + 1, z + 1)); a row
// outside the tile is skipped (a neighbouring tile adds it).  Four row predicates instead of a
// test per corner measured 0.490 -> 0.468 ms per deposit (256^3 on 512^3).  ONE: one-word
// sums of the whole tile (lo only); else two-word sums of the tile's planes z.x .. z.y - 1, the
// first of which is at the start of lo and hi.
template <bool ONE>
__device__ __forceinline__ void deposit_particle(unsigned* lo, unsigned* hi, int n, int rs, int cx, int ly, int lz,
                                                 int2 z, const unsigned (&q)[8]) {
  const int x1 = cx + 1 == n ? 0 : cx + 1;
  const bool y0 = ly >= 0, y1 = ly + 1 < TY;
  const bool z0 = ONE ? lz >= 0 : (lz >= z.x && lz < z.y);
  const bool z1 = ONE ? lz + 1 < TZ : (lz + 1 >= z.x && lz + 1 < z.y);
  const int base = ((ONE ? lz : lz - z.x) * TY + ly) * rs;
  auto add = [&](int i, unsigned v) {
    if (ONE) atomicAdd(&lo[i], v);  // result unused: a non-returning shared-memory reduction
    else acc_add(lo, hi, i, v);
  };
  if (y0 && z0) { add(base + cx, q[0]); add(base + x1, q[1]); }
  if (y1 && z0) { add(base + rs + cx, q[2]); add(base + rs + x1, q[4]); }
  if (y0 && z1) { add(base + TY * rs + cx, q[3]); add(base + TY * rs + x1, q[5]); }
  if (y1 && z1) { add(base + (TY + 1) * rs + cx, q[6]); add(base + (TY + 1) * rs + x1, q[7]); }
}

// CIC weights of a particle quantised to qscale = 2^s.
// qscale is a power of two, so scaling the x factor by it is exact and each product equals
// cic_weights' weight times qscale bit for bit (same association: (a_x a_y) a_z).
__device__ __forceinline__ void quantised_weights(const Cell& c, float qscale, unsigned (&q)[8]) {
  const float tx = (1.f - c.fx) * qscale, fx = c.fx * qscale;
  const float ty = 1.f - c.fy, tz = 1.f - c.fz, fy = c.fy, fz = c.fz;
  q[0] = __float2uint_rn(tx * ty * tz);
  q[1] = __float2uint_rn(fx * ty * tz);
  q[2] = __float2uint_rn(tx * fy * tz);
  q[3] = __float2uint_rn(tx * ty * fz);
  q[4] = __float2uint_rn(fx * fy * tz);
  q[5] = __float2uint_rn(fx * ty * fz);
  q[6] = __float2uint_rn(tx * fy * fz);
  q[7] = __float2uint_rn(fx * fy * fz);
}

// (Pre-adding the weights of lanes that share a cell, with __match_any_sync and a warp
// reduction, would cut the same-address atomics of clustered tiles, but the match alone made
// the deposit 6x slower on GB300.)
template <bool ONE>
__device__ __forceinline__ void deposit_entry(unsigned* lo, unsigned* hi, int n, int rs, float qscale, bool ok,
                                              const Cell& c, int ly, int lz, int2 z) {
  if (ok) {
    unsigned q[8];
    quantised_weights(c, qscale, q);
    deposit_particle<ONE>(lo, hi, n, rs, c.x, ly, lz, z, q);
  }
}

// Source ranges of a tile: the particles whose base cell lies in the tile's rows or one row
// / plane below (periodic) are, in the row-sorted order, 7 runs of consecutive rows (rows
// are numbered tile by tile, TZ x TY inside a tile):
//   0: the tile itself (16 rows)            1: the tile below in z, its last plane (TY rows)
//   2-5: the tile below in y, its last row of each plane    6: the diagonal tile, last row
constexpr int NRUN = 7;

// The run table of a tile: source entry f belongs to the last run r with off[r] <= f, and
// sits at place f + delta[r] (= begin[r] + f - off[r]) of the row-sorted order.
//
// RunTable searches the table in shared memory (a chain of dependent loads before the
// permutation load can issue, but no registers); RunRegs holds it in 14 registers and finds
// the run with compares and selects.  The fused deposit takes RunRegs (0.535 -> 0.521 ms early,
// 0.716 -> 0.636 ms at step 980, 256^3 on 512^3); the standalone deposit, at 40 registers a
// thread, keeps RunTable.
struct RunTable {
  const unsigned *begin, *off;
  __device__ __forceinline__ RunTable(const unsigned* s_begin, const unsigned* s_off) : begin(s_begin), off(s_off) {}
  // Slot of source entry f (0xffffffff past the end): its place in the row-sorted order,
  // through the permutation when there is one (else the state is in row order).
  __device__ __forceinline__ unsigned slot(const unsigned* __restrict__ perm, unsigned f, unsigned total) const {
    if (f >= total) return 0xffffffffu;
    int r = 0;  // last run with off[r] <= f
    if (off[4] <= f) r = 4;
    if (off[r + 2] <= f) r += 2;
    if (r + 1 < NRUN && off[r + 1] <= f) r += 1;
    const unsigned pos = begin[r] + (f - off[r]);
    return perm ? __ldg(&perm[pos]) : pos;
  }
};

struct RunRegs {
  unsigned off[NRUN], delta[NRUN];
  __device__ __forceinline__ RunRegs(const unsigned* s_begin, const unsigned* s_off) {
#pragma unroll
    for (int r = 0; r < NRUN; ++r) {
      off[r] = s_off[r];
      delta[r] = s_begin[r] - s_off[r];
    }
  }
  // Slot of source entry f (0xffffffff past the end): its place in the row-sorted order,
  // through the permutation when there is one (else the state is in row order).
  __device__ __forceinline__ unsigned slot(const unsigned* __restrict__ perm, unsigned f, unsigned total) const {
    if (f >= total) return 0xffffffffu;
    unsigned d = delta[0];
#pragma unroll
    for (int r = 1; r < NRUN; ++r) d = f >= off[r] ? delta[r] : d;
    const unsigned pos = f + d;
    return perm ? __ldg(&perm[pos]) : pos;
  }
};

// Base cell of a source particle relative to the tile, from its loaded words; false if
// absent or bad.  NN: the grid size when known at compile time (0: S.n).
template <int MODE, int NN>
__device__ __forceinline__ bool source_cell(const Sim& S, const Parts& p, const RawCell& raw, int y0, int z0,
                                            int* err, Cell& c, int& ly, int& lz) {
  if (!raw.present) return false;
  c = raw_cell<MODE>(S, p, raw);
  const int n = NN ? NN : S.n;
  int dy = c.y - y0, dz = c.z - z0;
  if (dy >= n - 1) dy -= n;
  if (dz >= n - 1) dz -= n;
  const bool ok = c.ok && dy >= -1 && dy < TY && dz >= -1 && dz < TZ;
  if (!ok) set_error(err, c.ok ? ERR_SOURCE_ROW : ERR_CELL_RANGE);
  ly = dy;
  lz = dz;
  return ok;
}

// The 7 runs of the tile at (y0, z0): lane r < NRUN of a group of eight loads the first sorted
// index and the particle count of run r; and, unless MAX is BINS_NOT, the largest row bin count of the
// tile and the three below it (all lanes of the group) -- BINS_MAXIMA: group_max holds the maxima of 16
// consecutive row bins, a tile's bins being x_bins such groups; BINS_STARTS: from row_start, where a
// kernel to make the maxima would cost more (4 us of a 60 us call), all 32 lanes of a warp for one
// tile (lane32), each with the maximum of its part.
enum BinsMode : int { BINS_NOT = 0, BINS_MAXIMA, BINS_STARTS };

struct RunLoad {
  unsigned beg = 0, cnt = 0, bin_max = 0;
  int per_row = 1;         // row bins to a row
  float mass_scale = 0.f;  // of the simulation
};

template <int MAX>
__device__ __forceinline__ RunLoad run_load(const Sim& S, const unsigned* __restrict__ row_start,
                                            const unsigned* __restrict__ group_max, int y0, int z0, int lane,
                                            int lane32 = 0) {
  RunLoad v;
  const int n = S.n;
  const int ym = y0 == 0 ? n - TY : y0 - TY, zm = z0 == 0 ? n - TZ : z0 - TZ;  // tiles below
  const int ntile_y = n / TY;
  const unsigned t_own = (unsigned)(z0 / TZ) * ntile_y + y0 / TY;
  const unsigned t_zb = (unsigned)(zm / TZ) * ntile_y + y0 / TY;
  const unsigned t_yb = (unsigned)(z0 / TZ) * ntile_y + ym / TY;
  const unsigned t_c = (unsigned)(zm / TZ) * ntile_y + ym / TY;
  const unsigned per_row = S.xbits ? 1u : (unsigned)x_bins(n);  // entries of row_start per x-row
  v.per_row = (int)per_row;
  v.mass_scale = S.mass_scale;
  if (lane < NRUN) {
    unsigned r0, nr;
    if (lane == 0) { r0 = t_own * (TZ * TY); nr = TZ * TY; }
    else if (lane == 1) { r0 = t_zb * (TZ * TY) + (TZ - 1) * TY; nr = TY; }
    else if (lane < 6) { r0 = t_yb * (TZ * TY) + (lane - 2) * TY + TY - 1; nr = 1; }
    else { r0 = t_c * (TZ * TY) + (TZ - 1) * TY + TY - 1; nr = 1; }
    const unsigned* s = row_start + (S.row_base + r0 * per_row);
    v.beg = __ldg(s);
    v.cnt = __ldg(s + nr * per_row) - v.beg;
  }
  if (MAX != BINS_NOT) {
    const unsigned each = MAX == BINS_MAXIMA ? per_row : per_row * (TZ * TY);  // words of a tile
    for (unsigned i = MAX == BINS_MAXIMA ? lane : lane32; i < 4 * each; i += MAX == BINS_MAXIMA ? 8 : 32) {
      const unsigned t = i / each;
      const unsigned tile = t == 0 ? t_own : (t == 1 ? t_zb : (t == 2 ? t_yb : t_c)), at = tile * each + i % each;
      const unsigned* b = MAX == BINS_MAXIMA ? group_max + S.row_base / (TZ * TY) + at : row_start + (S.row_base + at);
      v.bin_max = max(v.bin_max, MAX == BINS_MAXIMA ? __ldg(b) : __ldg(b + 1) - __ldg(b));
    }
  }
  return v;
}

// The runs of planes z0 + p0 .. z0 + p1 - 1 of the tile alone: their rows and those of the plane below
// them, and the row before each of these planes.
__device__ __forceinline__ RunLoad plane_load(const Sim& S, const unsigned* __restrict__ row_start, int y0, int z0, int p0,
                                              int p1, int lane) {
  RunLoad v;
  const int n = S.n, ym = y0 == 0 ? n - 1 : y0 - 1, own = p0 > 0 ? p0 - 1 : 0, p = p0 - 3 + lane;
  int y = y0, z = z0 + own, rows = (p1 - own) * TY;  // lane 0: the tile's own
  if (lane == 1) { z = z0 - 1; rows = p0 == 0 ? TY : 0; }
  if (lane >= 2) { y = ym; z = z0 + p; rows = lane < NRUN && p < p1 ? 1 : 0; }
  if (rows == 0) return v;
  const unsigned per_row = S.xbits ? 1u : (unsigned)x_bins(n);
  const unsigned* s = row_start + (S.row_base + row_number(y, z < 0 ? n - 1 : z, n) * per_row);
  v.beg = __ldg(s);
  v.cnt = __ldg(s + rows * per_row) - v.beg;
  return v;
}

// Warp-wide (all 32 lanes call it): the run table (first sorted index, and the inclusive scan
// of the counts) of the tile whose runs the 8 lanes of this lane's group of eight loaded
// (lane & 7 = the run).  The lanes with `write` store their group's table at s_begin / s_off
// (NRUN and NRUN + 1 words).  total: the tile's source entries.  Returns how its sums are held.
__device__ __forceinline__ TileSum run_table(const RunLoad& v, int lane, unsigned* s_begin, unsigned* s_off,
                                             bool write, unsigned& total) {
  const int r = lane & 7;
  unsigned incl = v.cnt, m = v.bin_max;
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    const unsigned t = __shfl_up_sync(FULL, incl, o, 8);
    if (r >= o) incl += t;
    m = max(m, __shfl_xor_sync(FULL, m, o, 8));
  }
  total = __shfl_sync(FULL, incl, NRUN - 1, 8);
  if (write) {
    if (r < NRUN) {
      s_begin[r] = v.beg;
      s_off[r + 1] = incl;
    }
    if (r == 0) s_off[0] = 0;
  }
  const unsigned cap = m < (1u << 28) ? m * (v.per_row > 1 ? 8u : 4u) : 0xffffffffu;
  return tile_sum(total, cap, v.mass_scale);
}

// The particle loop of a tile: two source entries per lane and iteration, so that their
// loads overlap; the slots (the permutation entries) of the next iteration are in flight
// while this one adds its particles.
template <int MODE, int NT, bool ONE, int NN>
__device__ __forceinline__ void deposit_sources(const Sim& S, const Parts& p, const unsigned* __restrict__ perm,
                                                int* err, int y0, int z0, unsigned* lo, unsigned* hi, int rs,
                                                const unsigned* s_begin, const unsigned* s_off, unsigned total,
                                                float qscale, int tid, int2 z) {
  const int lane = tid & 31, warp = tid >> 5;
  const int n = NN ? NN : S.n;
  using Runs = typename std::conditional<NN != 0, RunRegs, RunTable>::type;
  const Runs runs(s_begin, s_off);
  unsigned base = (unsigned)warp * 32u;
  unsigned sl0 = runs.slot(perm, base + lane, total);
  unsigned sl1 = runs.slot(perm, base + NT + lane, total);
  for (; base < total; base += 2 * NT) {
    const RawCell q0 = load_raw_cell<MODE>(p, sl0), q1 = load_raw_cell<MODE>(p, sl1);
    sl0 = runs.slot(perm, base + 2 * NT + lane, total);
    sl1 = runs.slot(perm, base + 3 * NT + lane, total);
    Cell c0, c1;
    int ly0 = 0, lz0 = 0, ly1 = 0, lz1 = 0;
    const bool ok0 = source_cell<MODE, NN>(S, p, q0, y0, z0, err, c0, ly0, lz0);
    const bool ok1 = source_cell<MODE, NN>(S, p, q1, y0, z0, err, c1, ly1, lz1);
    deposit_entry<ONE>(lo, hi, n, rs, qscale, ok0, c0, ly0, lz0, z);
    deposit_entry<ONE>(lo, hi, n, rs, qscale, ok1, c1, ly1, lz1, z);
  }
}

// Adds the tile at (y0, z0) of simulation S to zeroed accumulators, row r at word r * rs: one-word sums
// (ONE, ts.s) of its TZ * TY rows of n cells in lo; two-word sums of its planes z.x .. z.y - 1 in lo
// and hi.  s_begin / s_off: the tile's run table.  Done by NT threads, tid = 0 .. NT - 1 (a whole
// CTA, or a group of its warps with one tile each); the caller synchronises.  NN: the grid size
// when known at compile time (0: S.n).
template <int MODE, int NT, bool ONE, int NN = 0>
__device__ __forceinline__ void deposit_tile(const Sim& S, const Parts& p, const unsigned* __restrict__ perm, int* err,
                                             int y0, int z0, unsigned* lo, unsigned* hi, int rs, const unsigned* s_begin,
                                             const unsigned* s_off, const TileSum& ts, int2 z, int tid) {
  const float qscale = ONE ? __uint_as_float((unsigned)(127 + ts.s) << 23) : (float)(1u << PM_FIX_BITS);
  deposit_sources<MODE, NT, ONE, NN>(S, p, perm, err, y0, z0, lo, hi, rs, s_begin, s_off, s_off[NRUN], qscale, tid, z);
}

}  // namespace pm
