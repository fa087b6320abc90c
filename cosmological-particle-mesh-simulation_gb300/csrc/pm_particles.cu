// Particle-side kernels of one PM step:
//
//   keys     cell key of every particle            (density.py:19-21 / integrate.py:20)
//   rows     start of every x-row in the sorted particle order
//   deposit  deterministic CIC deposit             (density.py:7-48)
//   kick     CIC gather of the central-difference force, kick and drift
//                                                  (integrate.py:15-97)
//
// Cells, weights and keys are defined in pm_cells.cuh, the deposit's accumulation in
// pm_deposit.cuh (shared with the fused deposit + x-transform kernel).
#include "pm_cells.cuh"
#include "pm_deposit.cuh"
#include "pm_tma.cuh"

namespace pm {

constexpr int KICK_NT = 256;
constexpr int KICK_PPT = KICK_UNIT / KICK_NT;  // particles per thread of the kick
constexpr int KEY_NT = 256;

// ---------------------------------------------------------------------------------
// keys
// ---------------------------------------------------------------------------------
template <int MODE>
__global__ void __launch_bounds__(KEY_NT) k_keys(const Sim* __restrict__ sims, Work w, Parts p,
                                                 unsigned* __restrict__ keys,
                                                 unsigned* __restrict__ vals, int* err) {
  chain_begin();
  for (int unit = blockIdx.x; unit < w.total; unit += gridDim.x) {
    const int si = locate_sim(w, unit);
    const Sim& S = sims[si];
    const long long i = (long long)(unit - __ldg(&w.prefix[si])) * KEY_NT + threadIdx.x;
    if (i >= S.np) continue;
    const long long slot = S.slot_off + i;
    // from the state itself (the cell records, if any, are written here)
    Cell c;
    if (MODE == POS_ABS) {
      c = cell_abs(p.x[slot], p.y[slot], p.z[slot], S.n);
    } else {
      c = cell_disp(S, p.id[slot], p.x[slot], p.y[slot], p.z[slot]);
      if (p.rec) store_cell_record(p, slot, c);
    }
    if (!c.ok) { set_error(err, ERR_CELL_RANGE); c.x = c.y = c.z = 0; }
    keys[slot] = cell_key(S, c);
    if (vals) vals[slot] = (unsigned)slot;
  }
}

// ---------------------------------------------------------------------------------
// rows: row_start[r] = first sorted index whose row >= r, for r in [0, nrows]
// (keys with row >= nrows, e.g. the sentinel of an empty slot, count as row nrows)
// ---------------------------------------------------------------------------------
__global__ void k_row_start(const unsigned* __restrict__ keys, long long n, int xbits, unsigned nrows,
                            unsigned* __restrict__ row_start) {
  chain_begin();
  for (long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x; s <= n;
       s += (long long)gridDim.x * blockDim.x) {
    long long rp = -1, rc = nrows;
    if (s > 0) { rp = keys[s - 1] >> xbits; if (rp > nrows) rp = nrows; }
    if (s < n) { rc = keys[s] >> xbits; if (rc > nrows) rc = nrows; }
    for (long long r = rp + 1; r <= rc; ++r) row_start[r] = (unsigned)s;
  }
}

// ---------------------------------------------------------------------------------
// deposit: one CTA per tile (pm_deposit.cuh), then the tile's rows are written once
// ---------------------------------------------------------------------------------
// Words of a cell's sum that there is room for: two up to 512 cells, at three CTAs per SM; above, tiles
// in two words are done half their planes at a time.
__host__ __device__ constexpr int deposit_words(int n) { return n <= 512 ? 2 : 1; }

template <int MODE, int BINS>
__global__ void __launch_bounds__(DEP_NT, 3) k_deposit(const Sim* __restrict__ sims, Work w, Parts p,
                                                       const unsigned* __restrict__ perm,
                                                       const unsigned* __restrict__ row_start,
                                                       const unsigned* __restrict__ group_max, int* err) {
  chain_begin();
  extern __shared__ uint4 acc_raw[];
  __shared__ unsigned s_begin[NRUN];
  __shared__ unsigned s_off[NRUN + 1];
  __shared__ TileSum s_ts;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned* acc = reinterpret_cast<unsigned*>(acc_raw);
  for (int unit = blockIdx.x; unit < w.total; unit += gridDim.x) {
    const int si = locate_sim(w, unit);
    const Sim& S = sims[si];
    const int local = unit - __ldg(&w.prefix[si]);
    const int n = S.n;
    const int ntile_y = n / TY;
    const int y0 = (local % ntile_y) * TY, z0 = (local / ntile_y) * TZ;
    if (warp == 0) {
      unsigned total;
      RunLoad v = run_load<BINS>(S, row_start, group_max, y0, z0, lane & 7, lane);
      if (BINS == BINS_STARTS) v.bin_max = __reduce_max_sync(FULL, v.bin_max);
      const TileSum t = run_table(v, lane, s_begin, s_off, lane < 8, total);
      if (lane == 0) s_ts = t;
    }
    const int words = deposit_words(n);  // of a cell
    for (int i = threadIdx.x; i < words * TZ * TY * n / 4; i += DEP_NT) acc_raw[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    const TileSum ts = s_ts;
    const int rows = ts.s || words == 2 ? TZ * TY : TZ * TY / 2;
    for (int half = 0; half < TZ * TY / rows; ++half) {
      if (ts.s)
        deposit_tile<MODE, DEP_NT, true>(S, p, perm, err, y0, z0, acc, nullptr, n, s_begin, s_off, ts, make_int2(0, TZ),
                                         threadIdx.x);
      else  // low words, then high words (of half the planes at a time)
        deposit_tile<MODE, DEP_NT, false>(S, p, perm, err, y0, z0, acc, acc + rows * n, n, s_begin, s_off, ts,
                                          make_int2(half * rows / TY, (half + 1) * rows / TY), threadIdx.x);
      __syncthreads();
      for (int r = warp; r < rows; r += DEP_NT / 32) {
        const int row = half * rows + r;
        uint4* l4 = reinterpret_cast<uint4*>(acc + r * n);
        uint4* h4 = reinterpret_cast<uint4*>(acc + (r + rows) * n);  // (two-word tiles)
        float4* dst = reinterpret_cast<float4*>(S.rho + ((long long)(z0 + row / TY) * n + (y0 + row % TY)) * n);
        for (int x4 = lane; x4 < n / 4; x4 += 32) {
          const uint4 l = l4[x4], h = ts.s ? make_uint4(0u, 0u, 0u, 0u) : h4[x4];
          dst[x4] = make_float4(sum_to_float(ts, l.x, h.x), sum_to_float(ts, l.y, h.y), sum_to_float(ts, l.z, h.z),
                                sum_to_float(ts, l.w, h.w));
          if (!ts.s) l4[x4] = h4[x4] = make_uint4(0u, 0u, 0u, 0u);  // for the other half
        }
      }
      __syncthreads();
    }
  }
}

// ---------------------------------------------------------------------------------
// kick / drift
//
// For each particle: CIC weights of its base cell, the central difference
// phi[c - e_a] - phi[c + e_a] at the 8 corners for each axis a, interpolated with the
// weights and halved (integrate.py:84-92), then v_a += kick * g_a and
// x_a += drift * v_a (integrate.py:94-95).  All three axes use the cell and weights
// of the position before the step, as the reference's three sweeps do.
//
// Resident (k_kick): displacements; the particle that is i-th in sorted order is written to
//          output slot sort_off + i, together with its cell key for the next step.
// Drop-in: k_force in row order, k_advance in the caller's order (below).
// ---------------------------------------------------------------------------------
// Potential rows around a particle, read from global memory: row(oy, oz) is the x-row at
// (y + oy, z + oz) (periodic), oy, oz in {-1, 0, 1, 2}.  The taps are scalar loads: at one
// particle per several cells each lane of a warp reads its own sector, and 16-byte chunk
// loads of the x-1 .. x+2 windows measured 1.5x slower on GB300.
struct GlobalRows {
  const float* phi;
  int n, ys[4], zs[4];  // y - 1, y, y + 1, y + 2 and the same for z, wrapped
  __device__ __forceinline__ GlobalRows(const float* p, int nn, int y, int z) : phi(p), n(nn) {
    ys[1] = y; ys[0] = y == 0 ? n - 1 : y - 1; ys[2] = y + 1 == n ? 0 : y + 1; ys[3] = ys[2] + 1 == n ? 0 : ys[2] + 1;
    zs[1] = z; zs[0] = z == 0 ? n - 1 : z - 1; zs[2] = z + 1 == n ? 0 : z + 1; zs[3] = zs[2] + 1 == n ? 0 : zs[2] + 1;
  }
  __device__ __forceinline__ const float* row(int oy, int oz) const {
    return phi + (size_t)(unsigned)(zs[oz + 1] * n + ys[oy + 1]) * (unsigned)n;
  }
  __device__ __forceinline__ float ld(const float* p) const { return __ldg(p); }
};

// integrate.py:54-97: the 32 potential taps of the three finite-difference gradients at the
// 8 CIC corners, combined with the CIC weights in the reference's order.
template <class ROWS>
__device__ __forceinline__ void gather_taps(const ROWS& R, int n, const Cell& c, float g[3]) {
  float w[8];
  cic_weights(c, w);
  const int xm = c.x == 0 ? n - 1 : c.x - 1, x1 = c.x + 1 == n ? 0 : c.x + 1, x2 = x1 + 1 == n ? 0 : x1 + 1;
  const int x0 = c.x;
  // the 12 x-rows the 32 taps lie in
  const float* r00 = R.row(0, 0); const float* r10 = R.row(1, 0);
  const float* r01 = R.row(0, 1); const float* r11 = R.row(1, 1);
  const float* rm0 = R.row(-1, 0); const float* rm1 = R.row(-1, 1);
  const float* r20 = R.row(2, 0); const float* r21 = R.row(2, 1);
  const float* r0m = R.row(0, -1); const float* r1m = R.row(1, -1);
  const float* r02 = R.row(0, 2); const float* r12 = R.row(1, 2);
  // x gradient taps: rows (y0|y1, z0|z1) at xm, x0, x1, x2   (naming a<y><z><x>)
  const float a00m = R.ld(r00 + xm), a000 = R.ld(r00 + x0), a001 = R.ld(r00 + x1), a002 = R.ld(r00 + x2);
  const float a10m = R.ld(r10 + xm), a100 = R.ld(r10 + x0), a101 = R.ld(r10 + x1), a102 = R.ld(r10 + x2);
  const float a01m = R.ld(r01 + xm), a010 = R.ld(r01 + x0), a011 = R.ld(r01 + x1), a012 = R.ld(r01 + x2);
  const float a11m = R.ld(r11 + xm), a110 = R.ld(r11 + x0), a111 = R.ld(r11 + x1), a112 = R.ld(r11 + x2);
  // y extension rows ym, y2 at x0, x1 (z0, z1)
  const float bm00 = R.ld(rm0 + x0), bm01 = R.ld(rm0 + x1), b200 = R.ld(r20 + x0), b201 = R.ld(r20 + x1);
  const float bm10 = R.ld(rm1 + x0), bm11 = R.ld(rm1 + x1), b210 = R.ld(r21 + x0), b211 = R.ld(r21 + x1);
  // z extension planes zm, z2 at (x0|x1, y0|y1)
  const float cm00 = R.ld(r0m + x0), cm01 = R.ld(r0m + x1), cm10 = R.ld(r1m + x0), cm11 = R.ld(r1m + x1);
  const float c200 = R.ld(r02 + x0), c201 = R.ld(r02 + x1), c210 = R.ld(r12 + x0), c211 = R.ld(r12 + x1);
  // x axis: g(o) = phi[x+ox-1] - phi[x+ox+1]   (corner naming g<ox><oy><oz>)
  const float gx000 = a00m - a001, gx100 = a000 - a002;
  const float gx010 = a10m - a101, gx110 = a100 - a102;
  const float gx001 = a01m - a011, gx101 = a010 - a012;
  const float gx011 = a11m - a111, gx111 = a110 - a112;
  // y axis: g(o) = phi[y+oy-1] - phi[y+oy+1]
  const float gy000 = bm00 - a100, gy100 = bm01 - a101;
  const float gy010 = a000 - b200, gy110 = a001 - b201;
  const float gy001 = bm10 - a110, gy101 = bm11 - a111;
  const float gy011 = a010 - b210, gy111 = a011 - b211;
  // z axis: g(o) = phi[z+oz-1] - phi[z+oz+1]
  const float gz000 = cm00 - a010, gz100 = cm01 - a011;
  const float gz010 = cm10 - a110, gz110 = cm11 - a111;
  const float gz001 = a000 - c200, gz101 = a001 - c201;
  const float gz011 = a100 - c210, gz111 = a101 - c211;
  // integrate.py:92 order: g*t0 + g_x*t1 + g_y*t2 + g_z*t3 + g_xy*t4 + g_xz*t5 + g_yz*t6 + g_xyz*t7
  g[0] = (gx000 * w[0] + gx100 * w[1] + gx010 * w[2] + gx001 * w[3] + gx110 * w[4] + gx101 * w[5] +
          gx011 * w[6] + gx111 * w[7]) * 0.5f;
  g[1] = (gy000 * w[0] + gy100 * w[1] + gy010 * w[2] + gy001 * w[3] + gy110 * w[4] + gy101 * w[5] +
          gy011 * w[6] + gy111 * w[7]) * 0.5f;
  g[2] = (gz000 * w[0] + gz100 * w[1] + gz010 * w[2] + gz001 * w[3] + gz110 * w[4] + gz101 * w[5] +
          gz011 * w[6] + gz111 * w[7]) * 0.5f;
}

__device__ __forceinline__ void gather_force(const float* __restrict__ phi, int n, const Cell& c, float g[3]) {
  gather_taps(GlobalRows(phi, n, c.y, c.z), n, c, g);
}

// The same force from the three force grids of the spectral gradient (each already the halved
// central difference, -i sin(k_d) phi_k transformed back): 8 taps per axis at the CIC corners,
// combined with the weights in the order of integrate.py:92.
__device__ __forceinline__ void gather_grad(const Sim& S, const Cell& c, float g[3]) {
  float w[8];
  cic_weights(c, w);
  const int n = S.n;
  const int x0 = c.x, x1 = c.x + 1 == n ? 0 : c.x + 1;
  const int y1 = c.y + 1 == n ? 0 : c.y + 1, z1 = c.z + 1 == n ? 0 : c.z + 1;
  const size_t r00 = ((size_t)c.z * n + c.y) * n, r10 = ((size_t)c.z * n + y1) * n;
  const size_t r01 = ((size_t)z1 * n + c.y) * n, r11 = ((size_t)z1 * n + y1) * n;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float* __restrict__ G = S.grad[d];
    g[d] = __ldg(&G[r00 + x0]) * w[0] + __ldg(&G[r00 + x1]) * w[1] + __ldg(&G[r10 + x0]) * w[2] +
           __ldg(&G[r01 + x0]) * w[3] + __ldg(&G[r10 + x1]) * w[4] + __ldg(&G[r01 + x1]) * w[5] +
           __ldg(&G[r11 + x0]) * w[6] + __ldg(&G[r11 + x1]) * w[7];
  }
}

// Each thread advances KICK_PPT particles, KICK_NT apart: all their loads (state, then the
// 32 potential taps each) are issued before any store, so that they overlap.
// row_count (optional, with keys_next): histogram of the next keys, for the next step's
// counting sort
__global__ void __launch_bounds__(KICK_NT, 4) k_kick(const Sim* __restrict__ sims, Work w, Parts in, Parts out,
                                                  const unsigned* __restrict__ perm,
                                                  unsigned* __restrict__ keys_next, int* err,
                                                  unsigned* __restrict__ row_count) {
  chain_begin();
  for (int unit = blockIdx.x; unit < w.total; unit += gridDim.x) {
    const int si = locate_sim(w, unit);
    const Sim& S = sims[si];
    const long long i0 = (long long)(unit - __ldg(&w.prefix[si])) * (KICK_NT * KICK_PPT) + threadIdx.x;
    long long sp[KICK_PPT], slot[KICK_PPT];
    float px[KICK_PPT], py[KICK_PPT], pz[KICK_PPT], vx[KICK_PPT], vy[KICK_PPT], vz[KICK_PPT];
    unsigned id[KICK_PPT];
    Cell c[KICK_PPT];
#pragma unroll
    for (int q = 0; q < KICK_PPT; ++q) {
      const long long i = i0 + q * KICK_NT;
      sp[q] = S.part_off + i;  // position in sorted order
      slot[q] = i < S.np ? (long long)__ldg(&perm[sp[q]]) : -1;
    }
#pragma unroll
    for (int q = 0; q < KICK_PPT; ++q) {
      const long long sl = slot[q] >= 0 ? slot[q] : 0;
      px[q] = in.x[sl]; py[q] = in.y[sl]; pz[q] = in.z[sl];
      vx[q] = in.vx[sl]; vy[q] = in.vy[sl]; vz[q] = in.vz[sl];
      id[q] = in.id[sl];
    }
#pragma unroll
    for (int q = 0; q < KICK_PPT; ++q) c[q] = cell_disp(S, id[q], px[q], py[q], pz[q]);
    float g[KICK_PPT][3];
#pragma unroll
    for (int q = 0; q < KICK_PPT; ++q) {
      g[q][0] = g[q][1] = g[q][2] = 0.f;
      if (slot[q] >= 0 && c[q].ok) gather_force(S.phi, S.n, c[q], g[q]);
    }
    unsigned key[KICK_PPT];
#pragma unroll
    for (int q = 0; q < KICK_PPT; ++q) {
      key[q] = 0xffffffffu;
      if (slot[q] < 0) continue;
      if (!c[q].ok) set_error(err, ERR_CELL_RANGE);
      const float nvx = fmaf(S.kick, g[q][0], vx[q]), nvy = fmaf(S.kick, g[q][1], vy[q]),
                  nvz = fmaf(S.kick, g[q][2], vz[q]);
      const float nx = fmaf(S.drift, nvx, px[q]), ny = fmaf(S.drift, nvy, py[q]), nz = fmaf(S.drift, nvz, pz[q]);
      if (!(isfinite(nx) && isfinite(ny) && isfinite(nz) && isfinite(nvx) && isfinite(nvy) && isfinite(nvz)))
        set_error(err, ERR_NONFINITE);
      out.x[sp[q]] = nx; out.y[sp[q]] = ny; out.z[sp[q]] = nz;
      out.vx[sp[q]] = nvx; out.vy[sp[q]] = nvy; out.vz[sp[q]] = nvz;
      out.id[sp[q]] = id[q];
      Cell cn = cell_disp(S, id[q], nx, ny, nz);
      store_cell_record(out, sp[q], cn);
      if (!cn.ok) { set_error(err, ERR_CELL_RANGE); cn.x = cn.y = cn.z = 0; }
      key[q] = cell_key(S, cn);
      keys_next[sp[q]] = key[q];
    }
    {  // the whole warp takes part: equal keys are counted once per warp
      const int lane = threadIdx.x & 31;
#pragma unroll
      for (int q = 0; q < KICK_PPT; ++q) {
        const unsigned grp = __match_any_sync(0xffffffffu, key[q]);
        if (key[q] != 0xffffffffu && lane == __ffs(grp) - 1) atomicAdd(&row_count[key[q]], (unsigned)__popc(grp));
      }
    }
  }
}

// ---------------------------------------------------------------------------------
// drop-in step on absolute positions in the caller's order
//
// The caller's arrays are in particle order (the slowest particle index is x, the fastest grid
// axis), which scatters every grid row over memory.  Each particle crosses between the two
// orders twice, as one 16-byte word each time:
//   k_row_rank  (particle order) row key, and the particle's rank in its row from the returning
//               atomic that counts the row -- no second atomic pass is needed to place it;
//   (scan of the counts: row starts)
//   k_row_place (particle order) writes the particle's cell record to its place in row order
//               and keeps the place;
//   deposit and k_force work on the records in row order (k_force leaves the force in the
//               record's own word);
//   k_advance   (particle order) reads the force back and kicks and drifts the caller's state,
//               which is read and written in its own order only.
// Both crossings are bound by the rate of 32-byte sectors in L2 (the lines being filled or
// read are the rows' current ends, a few MB).  256^3 particles, 512^3 cells, in us: rank 145, scan 7,
// place 234 (plain order 326), force 299, advance 225; with boxes rank takes 186 and advance 256,
// whose own streams are then the ones broken up.
// ---------------------------------------------------------------------------------
constexpr int ORD_NT = 256;
constexpr int ORD_PPT = 4;  // particles per thread: their loads and atomics overlap

// The particle that element q of thread t of block b handles (-1: none).  Particles in lattice
// order (np1 > 0: np = np1^3, index (ix np1 + iy) np1 + iz) are taken in boxes of 16 iz x 4 iy x
// 16 ix, boxes along ix first: a box's particles lie in a few neighbouring rows, and the boxes in
// flight fill whole rows, so the words they write stay in L2 until their lines are full.  Plain
// order sweeps all rows once per ix plane.  np1 = 0: plain order.
// np1^3 particles in another order are better off in plain order (k_row_place, 256^3 particles with
// the lattice's axes reversed 139 us, in boxes 334; shuffled 420 and 531), so the boxes are taken
// only if the positions vote for them (lattice_vote).
struct ParticleOrder {
  long long np;
  int np1, bx, by;  // boxes per axis ix, iy
  __host__ __device__ ParticleOrder(long long n, int l) : np(n), np1(l), bx((l + 15) / 16), by((l + 3) / 4) {}
  __host__ long long blocks() const {  // enough for both orders
    const long long plain = (np + ORD_NT * ORD_PPT - 1) / (ORD_NT * ORD_PPT), boxes = (long long)bx * by * bx;
    return np1 && boxes > plain ? boxes : plain;
  }
  __device__ __forceinline__ long long at(int q) const {
    if (!np1) {
      const long long i = (long long)blockIdx.x * (ORD_NT * ORD_PPT) + q * ORD_NT + threadIdx.x;
      return i < np ? i : -1;
    }
    const int b = blockIdx.x, x0 = b % bx * 16, y0 = b / bx % by * 4, z0 = b / (bx * by) * 16;
    const int e = q * ORD_NT + threadIdx.x;
    const int ix = x0 + (e >> 6), iy = y0 + ((e >> 4) & 3), iz = z0 + (e & 15);
    return ix < np1 && iy < np1 && iz < np1 ? ((long long)ix * np1 + iy) * np1 + iz : -1;
  }
};

// A warp's vote on the order of the np1^3 particles, of which its lanes hold (x, y, z) of 32
// consecutive ones from i0 on: along a lattice line (iz) the z of a particle and of one m further on
// are m n / np1 cells apart, and their x and y about the same; m n / np1 is kept to n / 4, far beyond the
// displacements of neighbours relative to one another in most of the box.  Votes are summed.
__device__ __forceinline__ void lattice_vote(int np1, int n, long long i0, float x, float y, float z, int* vote) {
  const int left = np1 - 1 - (int)(i0 % np1), m = min(min(31, np1 / 4), left);  // (warp-uniform)
  if (m < 1) return;
  const float fn = (float)n;
  auto apart = [&](float v) {  // to the nearest image
    const float d = __shfl_sync(FULL, v, m) - __shfl_sync(FULL, v, 0);
    return fabsf(d - fn * rintf(d / fn));
  };
  const float dx = apart(x), dy = apart(y), dz = apart(z);
  if ((threadIdx.x & 31) == 0) atomicAdd(vote, dz > 2.f * fmaxf(dx, dy) ? 1 : -1);
}

// np1 (optional): whether np = np1^3 particles are in lattice order is voted on by every 16th block
// (vote: 0 before; positive: yes).
// copy (optional): the positions are also written there (they are read once, e.g. from host
// memory, and leave a device copy)
__global__ void __launch_bounds__(ORD_NT) k_row_rank(const float* __restrict__ pos, ParticleOrder ord, int n,
                                                     unsigned* __restrict__ count, unsigned* __restrict__ keys,
                                                     unsigned* __restrict__ ranks, int* err,
                                                     float* __restrict__ copy, int np1, int* __restrict__ vote) {
  chain_begin();
  const int lane = threadIdx.x & 31;
  const long long np = ord.np;
  float x[ORD_PPT], y[ORD_PPT], z[ORD_PPT];
#pragma unroll
  for (int q = 0; q < ORD_PPT; ++q) {
    const long long i = ord.at(q);
    x[q] = y[q] = z[q] = 0.f;
    if (i >= 0) { x[q] = pos[i]; y[q] = pos[np + i]; z[q] = pos[2 * np + i]; }
  }
  if (np1 && blockIdx.x % 16 == 0) {
    const long long i0 = (long long)blockIdx.x * (ORD_NT * ORD_PPT) + threadIdx.x - lane;
    if (i0 + 31 < np) lattice_vote(np1, n, i0, x[0], y[0], z[0], vote);
  }
  unsigned key[ORD_PPT], grp[ORD_PPT], base[ORD_PPT];
#pragma unroll
  for (int q = 0; q < ORD_PPT; ++q) {
    const long long i = ord.at(q);
    key[q] = 0xffffffffu;
    if (i >= 0) {
      if (copy) { copy[i] = x[q]; copy[np + i] = y[q]; copy[2 * np + i] = z[q]; }
      const Cell c = cell_abs(x[q], y[q], z[q], n);
      if (!c.ok) set_error(err, ERR_CELL_RANGE);
      key[q] = c.ok ? row_bin(c, n) : 0u;
    }
    // equal keys of a warp share one atomic
    grp[q] = __match_any_sync(FULL, key[q]);
    base[q] = 0;
    if (key[q] != 0xffffffffu && lane == __ffs(grp[q]) - 1) base[q] = atomicAdd(&count[key[q]], (unsigned)__popc(grp[q]));
  }
#pragma unroll
  for (int q = 0; q < ORD_PPT; ++q) {
    const long long i = ord.at(q);
    const unsigned b = __shfl_sync(FULL, base[q], __ffs(grp[q]) - 1);
    if (i >= 0) {
      keys[i] = key[q];
      ranks[i] = b + __popc(grp[q] & ((1u << lane) - 1u));
    }
  }
}

// place: in the row key of each particle, out its place in row order; vote: k_row_rank's
__global__ void __launch_bounds__(ORD_NT) k_row_place(const float* __restrict__ pos, ParticleOrder ord, int n,
                                                      const unsigned* __restrict__ row_start,
                                                      const unsigned* __restrict__ ranks, unsigned* __restrict__ place,
                                                      uint4* __restrict__ rec, const int* __restrict__ vote) {
  chain_begin();
  const long long np = ord.np;
  if (ord.np1 && *vote <= 0) ord.np1 = 0;
  Parts out{};
  out.rec = rec;
#pragma unroll
  for (int q = 0; q < ORD_PPT; ++q) {
    const long long i = ord.at(q);
    if (i < 0) continue;
    const Cell c = cell_abs(pos[i], pos[np + i], pos[2 * np + i], n);
    const unsigned slot = __ldg(&row_start[place[i]]) + ranks[i];
    store_cell_record(out, slot, c);
    place[i] = slot;
  }
}

// The force (gx, gy, gz) at every record, in row order, over the record's own word.  Two
// particles per thread, as k_kick.
__global__ void __launch_bounds__(KICK_NT, 4) k_force(const Sim* __restrict__ sims, uint4* __restrict__ rec) {
  chain_begin();
  const Sim& S = sims[0];
  const long long units = (S.np + KICK_UNIT - 1) / KICK_UNIT;
  for (long long unit = blockIdx.x; unit < units; unit += gridDim.x) {
    const long long i0 = unit * KICK_UNIT + threadIdx.x;
    Cell c[KICK_PPT];
    float g[KICK_PPT][3];
#pragma unroll
    for (int q = 0; q < KICK_PPT; ++q) {
      const long long i = i0 + q * KICK_NT;
      c[q] = record_cell(i < S.np ? rec[i] : make_uint4(CELL_BAD, 0u, 0u, 0u));
    }
#pragma unroll
    for (int q = 0; q < KICK_PPT; ++q) {
      g[q][0] = g[q][1] = g[q][2] = 0.f;
      if (c[q].ok) {
        if (S.grad[0]) gather_grad(S, c[q], g[q]);  // spectral gradient: three force grids
        else gather_force(S.phi, S.n, c[q], g[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < KICK_PPT; ++q) {
      const long long i = i0 + q * KICK_NT;
      if (i < S.np)
        rec[i] = make_uint4(__float_as_uint(g[q][0]), __float_as_uint(g[q][1]), __float_as_uint(g[q][2]), 0u);
    }
  }
}

// Kick and drift (integrate.py:94-95) of the caller's state with the forces in row order;
// positions may arrive as exactly n: the canonical value drifts and is wrapped into [0, n).
// pos_out / vel_out may be pos / vel, or host memory.
__global__ void __launch_bounds__(ORD_NT) k_advance(const Sim* __restrict__ sims, ParticleOrder ord,
                                                    const uint4* __restrict__ force,
                                                    const unsigned* __restrict__ place, const float* pos,
                                                    const float* vel, float* pos_out, float* vel_out, int* err) {
  chain_begin();
  const Sim& S = sims[0];
  const long long np = ord.np;
  const float kk = S.kick, dr = S.drift, fn = (float)S.n;
  uint4 g[ORD_PPT];
  float p[ORD_PPT][3], v[ORD_PPT][3];
#pragma unroll
  for (int q = 0; q < ORD_PPT; ++q) {
    const long long i = ord.at(q);
    if (i >= 0) g[q] = __ldg(&force[__ldg(&place[i])]);
  }
#pragma unroll
  for (int q = 0; q < ORD_PPT; ++q) {
    const long long i = ord.at(q);
#pragma unroll
    for (int d = 0; d < 3; ++d)
      if (i >= 0) { p[q][d] = pos[d * np + i]; v[q][d] = vel[d * np + i]; }
  }
#pragma unroll
  for (int q = 0; q < ORD_PPT; ++q) {
    const long long i = ord.at(q);
    if (i < 0) continue;
    const float f[3] = {__uint_as_float(g[q].x), __uint_as_float(g[q].y), __uint_as_float(g[q].z)};
    bool ok = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const float nv = fmaf(kk, f[d], v[q][d]);
      const float nx = canon(fmaf(dr, nv, canon(p[q][d], fn)), fn);
      ok = ok && isfinite(nv) && isfinite(nx);
      pos_out[d * np + i] = nx;
      vel_out[d * np + i] = nv;
    }
    if (!ok) set_error(err, ERR_NONFINITE);
  }
}

// Writes a call's descriptor and work table to device memory (they arrive as kernel arguments:
// no staging of host memory, and the call can be captured) and zeroes `nzero` 16-byte words.
__global__ void k_call_begin(Sim* __restrict__ dsim, CallWork* __restrict__ dwork, Sim sim, CallWork work,
                             uint4* __restrict__ zero, long long nzero) {
  chain_begin();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t == 0) {
    *dsim = sim;
    *dwork = work;
  }
  for (long long i = t; i < nzero; i += (long long)gridDim.x * blockDim.x) zero[i] = make_uint4(0u, 0u, 0u, 0u);
}

// ---------------------------------------------------------------------------------
// resident-state conversion: absolute (3, np) arrays in particle order <-> displacement
// state at slots [off, off + np)
// ---------------------------------------------------------------------------------
// row bin of the cell of every absolute position
__global__ void k_row_keys_abs(const float* __restrict__ pos, long long np, int n, unsigned* __restrict__ keys) {
  chain_begin();
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < np;
       i += (long long)gridDim.x * blockDim.x) {
    const Cell c = cell_abs(pos[i], pos[np + i], pos[2 * np + i], n);
    keys[i] = c.ok ? row_bin(c, n) : 0u;
  }
}

// Both conversions cross between particle order and row order, one float at a time and one array
// after another (blockIdx.y: x y z vx vy vz, so that the blocks of one array run together): the
// lines of one array that are being filled or read then stay in L2, where those of six at once do
// not.  The slots are taken in chunks of one deposit tile's mean particle count, all z of one y
// before the next y (row order has y before z): the particles in flight then cover whole lines
// of the lattice (z is the fastest particle index).  For a clustered state the chunks only
// roughly follow the tiles; every order gives the same result.  256^3 / 512^3 particles: to
// displacements 1.12 / 14.1 ms (all arrays at once, slot order) -> 0.44 / 9.0, back 2.79 / 28.8 ->
// 0.82 / 16.1; without the chunks 0.52 / 11.1 and 0.81 / 19.5.  The way back reads its slots
// evict-first, which leaves L2 to the lines being filled: 0.78 / 14.3 (its stores evict-first as well 24;
// several slots' loads issued together 0.79 / 17; a quarter of the CTAs 0.95 / 20).  Bound by
// the rate of 32-byte sectors in L2, one per float (123 G/s at 256^3).
struct ChunkOrder {
  long long np;
  int side;  // tiles per axis
  unsigned size;
  __host__ ChunkOrder(long long p, int n) : np(p), side(n / TY) {
    size = (unsigned)((p + (long long)side * side - 1) / ((long long)side * side));
  }
  // f(s) for every slot s < np of this block's chunks
  template <class F>
  __device__ __forceinline__ void each(F f) const {
    for (int c = blockIdx.x; c < side * side; c += gridDim.x) {
      const long long s0 = (long long)(c % side * side + c / side) * size;
      for (unsigned j = threadIdx.x; j < size && s0 + j < np; j += blockDim.x) f(s0 + j);
    }
  }
};

// slot off + s takes particle order[s]
__global__ void k_abs_to_disp(const float* __restrict__ pos, const float* __restrict__ vel, ChunkOrder chunks,
                              int np1, int n, const int* __restrict__ q_int, const float* __restrict__ q_frac,
                              Parts out, long long off, const unsigned* __restrict__ order) {
  chain_begin();
  const long long np = chunks.np;
  const float fn = (float)n, half = 0.5f * fn;
  const unsigned u1 = (unsigned)np1;
  const int k = blockIdx.y % 3;
  const bool is_vel = blockIdx.y >= 3;
  const float* __restrict__ src = (is_vel ? vel : pos) + k * np;
  float* __restrict__ dst = (is_vel ? (k == 0 ? out.vx : (k == 1 ? out.vy : out.vz))
                                    : (k == 0 ? out.x : (k == 1 ? out.y : out.z))) + off;
  chunks.each([&](long long s) {
    const unsigned i = __ldg(&order[s]);  // the particle
    const float v = src[i];
    if (is_vel) {
      dst[s] = v;
      return;
    }
    const unsigned iz = i % u1, t = i / u1, iy = t % u1, ix = t / u1;
    const unsigned l = k == 0 ? ix : (k == 1 ? iy : iz);
    const float q = (float)__ldg(&q_int[l]) + __ldg(&q_frac[l]);
    float d = v - q;
    if (d >= half) d -= fn;
    if (d < -half) d += fn;
    dst[s] = d;
    if (k == 0) out.id[off + s] = pack_lattice(ix, iy, iz);
  });
}

__global__ void k_disp_to_abs(Parts in, long long off, ChunkOrder chunks, int np1, int n,
                              const int* __restrict__ q_int, const float* __restrict__ q_frac,
                              float* __restrict__ pos, float* __restrict__ vel) {
  chain_begin();
  const long long np = chunks.np;
  const float fn = (float)n;
  const int k = blockIdx.y % 3;
  const bool is_vel = blockIdx.y >= 3;
  const float* __restrict__ src = (is_vel ? (k == 0 ? in.vx : (k == 1 ? in.vy : in.vz))
                                          : (k == 0 ? in.x : (k == 1 ? in.y : in.z))) + off;
  const unsigned* __restrict__ ids = in.id + off;
  float* __restrict__ dst = (is_vel ? vel : pos) + k * np;
  chunks.each([&](long long j) {
    const unsigned pid = __ldcs(&ids[j]);
    const unsigned ax[3] = {pid >> 20, (pid >> 10) & 1023u, pid & 1023u};
    const long long id = ((long long)ax[0] * np1 + ax[1]) * np1 + ax[2];
    float v = __ldcs(&src[j]);
    if (!is_vel) {
      const unsigned l = k == 0 ? ax[0] : (k == 1 ? ax[1] : ax[2]);
      const float s = __ldg(&q_frac[l]) + v;
      const float fl = floorf(s);
      float x = (float)wrap_int(__ldg(&q_int[l]) + (int)fl, n) + (s - fl);
      if (x >= fn) x -= fn;
      v = x;
    }
    dst[id] = v;
  });
}

// ---------------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------------
cudaError_t launch_abs_to_disp(const float* pos, const float* vel, long long np, int np1, int n,
                               const int* q_int, const float* q_frac, Parts out, long long off,
                               Launch st, const unsigned* order) {
  const ChunkOrder c(np, n);
  const int b = c.side * c.side < 152 * 16 ? c.side * c.side : 152 * 16;
  k_abs_to_disp<<<dim3((unsigned)b, 6), 256, 0, st>>>(pos, vel, c, np1, n, q_int, q_frac, out, off, order);
  return cudaGetLastError();
}

cudaError_t launch_row_keys_abs(const float* pos, long long np, int n, unsigned* keys, Launch st) {
  long long b = (np + 255) / 256;
  if (b > 152 * 32) b = 152 * 32;
  launch_chained(k_row_keys_abs, (int)(b > 0 ? b : 1), 256, 0, st, pos, np, n, keys);
  return cudaGetLastError();
}

cudaError_t launch_disp_to_abs(Parts in, long long off, long long np, int np1, int n, const int* q_int,
                               const float* q_frac, float* pos, float* vel, Launch st) {
  const ChunkOrder c(np, n);
  const int b = c.side * c.side < 152 * 16 ? c.side * c.side : 152 * 16;
  k_disp_to_abs<<<dim3((unsigned)b, 6), 256, 0, st>>>(in, off, c, np1, n, q_int, q_frac, pos, vel);
  return cudaGetLastError();
}

cudaError_t deposit_prepare() {
  static DeviceOnce once;
  return once.run([]() {
    int sm = 0;
    for (int n = 16; n <= PM_MAX_N; n *= 2) sm = std::max(sm, (int)deposit_smem_bytes(n, TY, TZ));
    cudaError_t e = cudaSuccess;
    for (auto k : {k_deposit<POS_ABS, BINS_STARTS>, k_deposit<POS_DISP, BINS_MAXIMA>}) {
      if (!e) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
      if (!e) e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    }
    return e;
  });
}

size_t deposit_smem_bytes(int n, int ty, int tz) { return (size_t)n * ty * tz * deposit_words(n) * sizeof(unsigned); }

cudaError_t launch_keys_abs(const Sim* sims, const Work& w, Parts p, unsigned* keys, unsigned* vals,
                            int* err, int ctas, Launch st) {
  launch_chained(k_keys<POS_ABS>, ctas, KEY_NT, 0, st, sims, w, p, keys, vals, err);
  return cudaGetLastError();
}
cudaError_t launch_keys_disp(const Sim* sims, const Work& w, Parts p, unsigned* keys, unsigned* vals,
                             int* err, int ctas, Launch st) {
  launch_chained(k_keys<POS_DISP>, ctas, KEY_NT, 0, st, sims, w, p, keys, vals, err);
  return cudaGetLastError();
}

cudaError_t launch_row_start(const unsigned* keys, long long n, int xbits, unsigned nrows,
                             unsigned* row_start, Launch st) {
  long long work = n + 1;
  int ctas = (int)((work + 255) / 256);
  if (ctas > 152 * 16) ctas = 152 * 16;
  launch_chained(k_row_start, ctas, 256, 0, st, keys, n, xbits, nrows, row_start);
  return cudaGetLastError();
}

// Order in which the fused deposit takes its tiles: the dense tiles first.  A tile's work is
// its source-entry count, which clustering makes very uneven; a dense tile taken late runs on
// alone after the others have finished.  Tiles with more than twice the mean count go to the
// front of `order`, the others to the back (their order within each part is immaterial: a
// tile's sums do not depend on when it runs).  counts[0], counts[1]: zero at launch.
__global__ void k_tile_order(const Sim* __restrict__ sims, Work w, const unsigned* __restrict__ row_start,
                             unsigned* __restrict__ order, unsigned* __restrict__ counts) {
  chain_begin();
  for (int unit = blockIdx.x * blockDim.x + threadIdx.x; unit < w.total; unit += gridDim.x * blockDim.x) {
    const int si = locate_sim(w, unit);
    const Sim& S = sims[si];
    const int n = S.n, local = unit - __ldg(&w.prefix[si]);
    const int y0 = (local % (n / TY)) * TY, z0 = (local / (n / TY)) * TZ;
    unsigned cnt = 0;
#pragma unroll
    for (int r = 0; r < NRUN; ++r) cnt += run_load<BINS_NOT>(S, row_start, nullptr, y0, z0, r).cnt;
    // mean source entries per tile: each particle once, plus its tile's last plane / row / corner
    const double ntiles = (double)(n / TY) * (n / TZ);
    const double mean = (double)S.np * (1.0 + 1.0 / TZ + 1.0 / TY + 1.0 / (TY * TZ)) / ntiles;
    if (cnt > 2.0 * mean) order[atomicAdd(&counts[0], 1u)] = (unsigned)unit;
    else order[w.total - 1 - (int)atomicAdd(&counts[1], 1u)] = (unsigned)unit;
  }
}

cudaError_t launch_tile_order(const Sim* sims, const Work& w, const unsigned* row_start, unsigned* order,
                              unsigned* counts, int sms, Launch st) {
  if (w.total <= 0) return cudaSuccess;
  const int ctas = std::min((w.total + 255) / 256, 4 * sms);
  launch_chained(k_tile_order, ctas, 256, 0, st, sims, w, row_start, order, counts);
  return cudaGetLastError();
}

cudaError_t launch_deposit(const Sim* sims, const Work& w, Parts p, const unsigned* perm,
                           const unsigned* row_start, const unsigned* group_max, int mode, int* err, int ctas,
                           size_t smem, Launch st) {
  if (cudaError_t e = deposit_prepare()) return e;
  // (absolute positions come without bin maxima)
  auto kernel = mode == POS_ABS ? k_deposit<POS_ABS, BINS_STARTS> : k_deposit<POS_DISP, BINS_MAXIMA>;
  launch_chained(kernel, ctas, DEP_NT, smem, st, sims, w, p, perm, row_start, group_max, err);
  return cudaGetLastError();
}

cudaError_t launch_kick(const Sim* sims, const Work& w, Parts in, Parts out, const unsigned* perm,
                        unsigned* keys_next, int* err, int ctas, Launch st, unsigned* row_count) {
  k_kick<<<ctas, KICK_NT, 0, st>>>(sims, w, in, out, perm, keys_next, err, row_count);
  return cudaGetLastError();
}

cudaError_t launch_call_begin(Sim* dsim, CallWork* dwork, const Sim& sim, const CallWork& work, void* zero,
                              size_t zero_bytes, Launch st) {
  const long long nz = (long long)(zero_bytes / sizeof(uint4));
  const long long want = (nz + 1023) / 1024;  // four words per thread
  launch_chained(k_call_begin, (int)(want < 1 ? 1 : (want > 1024 ? 1024 : want)), 256, 0, st, dsim, dwork, sim, work, static_cast<uint4*>(zero), nz);
  return cudaGetLastError();
}

cudaError_t launch_row_rank(const float* pos, long long np, int np1, int n, unsigned* count, unsigned* keys,
                            unsigned* ranks, int* err, float* copy, int* vote, Launch st) {
  const ParticleOrder o(np, 0);
  launch_chained(k_row_rank, (int)o.blocks(), ORD_NT, 0, st, pos, o, n, count, keys, ranks, err, copy, np1, vote);
  return cudaGetLastError();
}

cudaError_t launch_row_place(const float* pos, long long np, int np1, int n, const unsigned* row_start,
                             const unsigned* ranks, unsigned* place, uint4* rec, const int* vote, Launch st) {
  const ParticleOrder o(np, np1);
  launch_chained(k_row_place, (int)o.blocks(), ORD_NT, 0, st, pos, o, n, row_start, ranks, place, rec, vote);
  return cudaGetLastError();
}

cudaError_t launch_force(const Sim* sims, long long np, uint4* rec, int sms, Launch st) {
  const long long units = (np + KICK_UNIT - 1) / KICK_UNIT, cap = (long long)sms * 16;
  launch_chained(k_force, (int)(units < cap ? units : cap), KICK_NT, 0, st, sims, rec);
  return cudaGetLastError();
}

cudaError_t launch_advance(const Sim* sims, long long np, const uint4* force, const unsigned* place,
                           const float* pos, const float* vel, float* pos_out, float* vel_out, int* err,
                           Launch st) {
  const ParticleOrder o(np, 0);
  launch_chained(k_advance, (int)o.blocks(), ORD_NT, 0, st, sims, o, force, place, pos, vel, pos_out, vel_out, err);
  return cudaGetLastError();
}

}  // namespace pm
