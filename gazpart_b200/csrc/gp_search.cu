// gp_search.cu -- binning, neighbour search, greedy matching and the data-movement
// kernels of the collision step.
#include <cooperative_groups.h>

#include "gp_types.h"
#include "gp_launch.h"

namespace cg = cooperative_groups;

namespace gp {

// COLLISION on the device (collision.f90:7-200 with NPROC=1).
//
// The reference lists candidate pairs box by box (collision_detection_connectivity.f90:
// 145-207): for each box IJK, for each particle NP1 of the box in ascending index,
// first the later particles of the same box, then every particle of the 13 forward
// neighbour boxes COLBOX(IJK)%CON(1..NCON) in order.  It then walks that list and lets
// a pair collide only if neither particle has collided yet this step
// (collision_interaction.f90:190-419).
//
// Device formulation (same result):
//  1. particles are binned into a search grid whose cell edge is at least twice the
//     largest bounding radius max(EMAJ, EMAJ/APR); a pair can only be in contact if
//     its bounding spheres overlap (each contact point must lie inside the other body,
//     ellipsoid_contact_detection.f90:125), so a half-stencil sweep over that grid
//     finds every pair that could collide;
//  2. for each such pair the reference's box ids decide whether the reference lists it
//     at all and in which orientation, and give its position in the reference list as
//     the key (IJK of HOME, index of HOME, stencil slot, index of NEAR);
//  3. contacts and NVREL are evaluated for all of them on the pre-collision state (a
//     pair is only ever evaluated while both its particles are unmodified);
//  4. the lexicographically-first maximal matching of the colliding pairs under that key
//     -- which is what the sequential COLOR walk produces -- is computed in parallel
//     rounds (a pair is accepted when it holds the smallest key at both endpoints);
//  5. COLLISION_RESPONSE is applied to the accepted pairs (disjoint, so race free).

// Canonical slot of the 13 forward neighbour offsets in COLBOX order
// (collision_box_connectivity.f90:127-312: boxes 9,12,15,17,18,20,21,22,23,24,25,26,27),
// indexed by (dI+1)*9 + (dJ+1)*3 + (dK+1); 0 = not a forward offset.
__constant__ int8_t c_fwd_slot[27] = {
    // dI = -1: (dJ,dK) = (-1,-1) (-1,0) (-1,1) (0,-1) (0,0) (0,1) (1,-1) (1,0) (1,1)
    0, 0, 0, 0, 0, 8, 0, 0, 11,
    // dI = 0
    0, 0, 6, 0, 0, 9, 0, 4, 12,
    // dI = +1
    0, 2, 7, 0, 3, 10, 1, 5, 13};

__device__ __forceinline__ int wrap_delta(int d, int n, bool periodic) {
  if (periodic) {
    if (d == n - 1) return -1;
    if (d == -(n - 1)) return 1;
  }
  return d;
}


// 1. search-grid cell of every particle (counting pass)
// ---------------------------------------------------------------------------
__device__ __forceinline__ int cell_coord(double v, double ih, int n) {
  const double f = v * ih;
  int c = (f >= 0.0) ? (f < (double)n ? (int)f : n - 1) : 0;
  return c;
}

// First cell of the row (cy, cz); cells are numbered x-fastest.
__device__ __forceinline__ int32_t cell_row(const InstDev &I, int cy, int cz) {
  return (int32_t)I.cell_begin + (cz * I.nfy + cy) * I.nfx;
}
__device__ __forceinline__ void cell_coords(const InstDev &I, int32_t cell, int &cx, int &cy, int &cz) {
  const int l = cell - (int32_t)I.cell_begin, t = l / I.nfx;
  cx = l - t * I.nfx;
  cz = t / I.nfy;
  cy = t - cz * I.nfy;
}

// Of the `grid` blocks that fill the chip (eight per SM: the binning waits for its scattered
// accesses, 16.8 M particles 0.65 ms with four; 0.58 with eight, half of the scatter's then
// waiting for the others' registers, 0.52 with all of them resident) only those that get a
// particle: 10,000 particles 19 us with eight per SM, 17 so.
constexpr int kBinThreads = 256;
static int bin_blocks(int64_t n, int grid) {
  return (int)std::max<int64_t>(1, std::min<int64_t>(grid, (n + kBinThreads - 1) / kBinThreads));
}

// Also clears what the rest of the collision phase counts in (also in a step after a halted
// one, whose scan and search still run): a clearing pass of its own costs a launch each.
__global__ void k_bin_count(const InstDev *__restrict__ insts, const PoolView *__restrict__ pv, int64_t n,
                            SearchArrays sa, PhaseClear clear, const Status *st) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x, gid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  for (int64_t k = gid; k < clear.tiles; k += stride) clear.tile_state[k] = 0ull;
  if (blockIdx.x == 0) {
    if (threadIdx.x < clear.ncounters && (clear.counter_mask >> threadIdx.x) & 1u) clear.counters[threadIdx.x] = 0ull;
    if (clear.bins != nullptr)
      for (int k = threadIdx.x; k < clear.nbins; k += blockDim.x) clear.bins[k] = 0u;
  }
  if (step_halted(st)) return;
  const PoolView P = *pv;
  const int64_t nround = (n + stride - 1) / stride * stride;   // whole warps stay in the loop
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nround; i += stride) {
    int32_t c = -1;
    if (i < n) {
      const int inst = P.inst[i];
      if (inst >= 0) {
        const InstDev &I = insts[inst];
        const int cx = cell_coord(P.st[0][i], I.ihfx, I.nfx);
        const int cy = cell_coord(P.st[1][i], I.ihfy, I.nfy);
        const int cz = cell_coord(P.st[2][i], I.ihfz, I.nfz);
        c = cell_row(I, cy, cz) + cx;
      }
      sa.cell_of[i] = c;
    }
    // particles are kept in cell order, so neighbouring lanes usually share a cell:
    // one atomic per cell per warp
    const unsigned peers = __match_any_sync(0xffffffffu, c);
    const int leader = __ffs(peers) - 1;
    if (c >= 0 && (int)(threadIdx.x & 31) == leader) atomicAdd(&sa.cell_count[c], __popc(peers));
  }
}

void launch_bin_count(const InstDev *insts, const PoolView *pv, int64_t n, SearchArrays sa, Status *st, int grid,
                      const PhaseClear &clear, cudaStream_t s) {
  k_bin_count<<<bin_blocks(n, grid), kBinThreads, 0, s>>>(insts, pv, n, sa, clear, st);
}

// ---------------------------------------------------------------------------
// 2. exclusive scan, one pass
// ---------------------------------------------------------------------------
// Blocks take tiles of 2048 counts in order from a counter. A tile publishes its sum at once
// and its inclusive prefix as soon as it has it; a block adds up the sums before its tile
// back to the nearest prefix (the decoupled look-back of D. Merrill and M. Garland, NVIDIA
// NVR-2016-002).  The tiles before a block's were taken by blocks that are running, so the
// wait ends; it is bounded all the same.  One launch instead of three to five.
// state[0] is the counter, state[1 + t] tile t: status (1 sum, 2 prefix) << 32 | value; all
// zero at the launch.
constexpr int kScanThreads = 512, kScanPer = 4, kScanBlock = kScanThreads * kScanPer;

__global__ void __launch_bounds__(kScanThreads) k_scan(const int32_t *__restrict__ in, int32_t *__restrict__ out,
                                                       int64_t n, unsigned long long *state,
                                                       float *__restrict__ clear, Status *st) {
  __shared__ int32_t warp_tot[kScanThreads / 32];
  __shared__ int64_t tile_s;
  __shared__ int32_t before_s;
  if (threadIdx.x == 0) tile_s = (int64_t)atomicAdd(&state[0], 1ull);
  __syncthreads();
  const int64_t tile = tile_s, base = tile * kScanBlock + (int64_t)threadIdx.x * kScanPer;
  int32_t v[kScanPer];
  int32_t run = 0;
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) {
    const int64_t idx = base + k;
    v[k] = (idx < n) ? in[idx] : 0;
    const int32_t t = v[k];
    v[k] = run;
    run += t;
  }
  // inclusive warp scan of per-thread totals
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int32_t x = run;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_tot[wid] = x;
  __syncthreads();
  if (wid == 0) {
    int32_t w = (lane < kScanThreads / 32) ? warp_tot[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < kScanThreads / 32) warp_tot[lane] = w;
    const int32_t total = __shfl_sync(0xffffffffu, w, kScanThreads / 32 - 1);
    volatile unsigned long long *tiles = state + 1;
    if (lane == 0) tiles[tile] = ((tile == 0 ? 2ull : 1ull) << 32) | (unsigned)total;
    int32_t before = 0;
    if (tile > 0) {
      // look back 32 tiles at a time, lane 0 at the nearest
      int64_t at = tile - 1;
      for (int spin = 0;;) {
        const int64_t k = at - lane;
        const unsigned long long e = k >= 0 ? tiles[k] : (2ull << 32);
        const int status = (int)(e >> 32);
        if (__any_sync(0xffffffffu, status == 0)) {
          if (++spin > (1 << 24)) {   // cannot happen
            if (lane == 0) set_error(st, GP_ETIMEOUT, tile);
            break;
          }
          continue;
        }
        const unsigned whole = __ballot_sync(0xffffffffu, status == 2);
        const int last = whole ? __ffs(whole) - 1 : 31;   // the nearest prefix ends the sum
        before += __reduce_add_sync(0xffffffffu, lane <= last ? (int32_t)(unsigned)e : 0);
        if (whole) break;
        at -= 32;
      }
      if (lane == 0) tiles[tile] = (2ull << 32) | (unsigned)(before + total);
    }
    if (lane == 0) before_s = before;
  }
  __syncthreads();
  const int32_t excl = before_s + x - run + (wid > 0 ? warp_tot[wid - 1] : 0);
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) {
    const int64_t idx = base + k;
    if (idx < n) {
      out[idx] = v[k] + excl;
      if (clear != nullptr) clear[idx] = 0.f;
    }
  }
}

int64_t scan_tiles(int64_t n) { return (n + 1 + kScanBlock - 1) / kScanBlock + 1; }

// out[0..n] = exclusive scan of in[0..n-1], out[n] = total.  in[n] must be readable
// as zero (the caller allocates n+1 counters, and n+1 values of clear).
void launch_scan(const int32_t *in, int32_t *out, int64_t n, unsigned long long *state, float *clear, Status *st,
                 cudaStream_t s) {
  k_scan<<<(unsigned)(scan_tiles(n) - 1), kScanThreads, 0, s>>>(in, out, n + 1, state, clear, st);
}

// ---------------------------------------------------------------------------
// 3. scatter into cell order, out-of-grid check (collision_detection_connectivity.f90:74-89)
// ---------------------------------------------------------------------------
// 0-based coordinate of v in the reference's box grid, or -1 outside it.
__device__ __forceinline__ int box_coord(double v, double vmin, double edge, int nbox) {
  const double f = (v - vmin) / edge;
  if (!(f > -1.0 && f < 2.0e9)) return -1;
  const int k = (int)f + 1;
  return (k >= 1 && k <= nbox) ? k - 1 : -1;
}
// Whether box_coord has a box for v, without its division well inside the grid.
__device__ __forceinline__ bool in_boxes(double v, double vmin, double edge, int nbox) {
  const double d = v - vmin;
  return (d >= 0.0 && d <= (double)nbox * edge * (1.0 - 1e-9)) || box_coord(v, vmin, edge, nbox) >= 0;
}

// The counting pass's counts are taken back to zero here, one place after the other, so
// that the next binning finds them clear.  Only what nearly every candidate of the search
// is judged by goes into sorted order (20 bytes a particle); the few candidates that pass
// read the pool.  What bounds it is the scattered traffic: with sixteen sorted columns
// (112 bytes written, 100 read) and three arrays of cells cleared by themselves the whole
// binning took 1.07 ms at 16.8 M particles, with these two 0.52 (B200).  Numbering the
// cells in bricks of 4 x 4 x 8, 4 x 4 x 4 or 2 x 2 x 8 for the gather's sake left the
// gather as it was (3.22 ms each) and took 0.04 more in the search.
__global__ void __launch_bounds__(kBinThreads, 8) k_bin_scatter(const InstDev *__restrict__ insts, const PoolView *__restrict__ pv, int64_t n,
                              SearchArrays sa, Status *st) {
  if (step_halted(st)) return;
  const PoolView P = *pv;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t nround = (n + stride - 1) / stride * stride;
  const int lane = threadIdx.x & 31;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nround; i += stride) {
    const int32_t c = (i < n) ? sa.cell_of[i] : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, c);
    const int leader = __ffs(peers) - 1;
    double x = 0.0, y = 0.0, z = 0.0;
    float small = 0.f, w = 0.f;
    if (c >= 0) {
      const int inst = P.inst[i];
      const InstDev &I = insts[inst];
      x = P.st[0][i]; y = P.st[1][i]; z = P.st[2][i];
      const double rb = fmax(P.pc[0][i], P.pc[1][i]);
      // w carries the bounding radius, negated for particles above the small-particle cut
      w = rb > I.rcut ? -(float)rb : (float)rb;
      if (rb <= I.rcut) small = __double2float_ru(rb);   // a float rounded up bounds the radius
      if (!(in_boxes(x, I.xminbox, I.dxbox, I.nxbox) && in_boxes(y, I.yminbox, I.dybox, I.nybox) &&
            in_boxes(z, I.zminbox, I.dzbox, I.nzbox)))
        set_error(st, GP_EOUT_OF_GRID, (long long)P.id[i], inst);
    }
    // non-negative floats order like their bits
    const unsigned most = __reduce_max_sync(peers, (unsigned)__float_as_int(small));
    int base = 0;
    if (c >= 0 && lane == leader) {
      base = atomicSub(&sa.cell_count[c], __popc(peers)) - __popc(peers);
      if (most != 0u) atomicMax(reinterpret_cast<int *>(sa.cell_rmax) + c, (int)most);
    }
    base = __shfl_sync(0xffffffffu, base, leader);
    if (c < 0) continue;
    const int pos = sa.cell_start[c] + base + __popc(peers & ((1u << lane) - 1u));
    sa.sorted[pos] = (int32_t)i;
    sa.spk[pos] = make_float4((float)x, (float)y, (float)z, w);
  }
}

void launch_bin_scatter(const InstDev *insts, const PoolView *pv, int64_t n, SearchArrays sa, Status *st, int grid,
                        cudaStream_t s) {
  k_bin_scatter<<<bin_blocks(n, grid), kBinThreads, 0, s>>>(insts, pv, n, sa, st);
}

// ---------------------------------------------------------------------------
// 4. half-stencil sweep of the search grid, reference adjacency and order key
// ---------------------------------------------------------------------------
// mark (non-null when the next step's integrate runs speculatively): both particles of
// a stored pair are flagged, since the response may change their velocities.
__device__ __forceinline__ void emit_pair(PairRec *pairs, unsigned long long *npairs, int64_t cap, const PairRec &r,
                                          uint32_t *mark, Status *st) {
  cg::coalesced_group g = cg::coalesced_threads();
  unsigned long long base = 0;
  if (g.thread_rank() == 0) base = atomicAdd(npairs, (unsigned long long)g.size());
  base = g.shfl(base, 0);
  const unsigned long long slot = base + g.thread_rank();
  if ((int64_t)slot < cap) {
    pairs[slot] = r;
    if (mark != nullptr) {
      mark[r.home] = 1u;
      mark[r.near] = 1u;
    }
  } else {
    atomicAdd(&st->overflow, 1ull);
    atomicMax(&st->pairs_needed, slot + 1ull);
    set_error(st, GP_EPAIR_OVERFLOW, (long long)r.home);
  }
}

// A home particle as the conservative float test of its candidates reads it: position,
// bounding radius, its instance's box lengths, the slack with the sign of x periodicity
// (32 bytes).
struct HomeF {
  float x, y, z, r, lx, ly, lz, slack;
};

__device__ __forceinline__ HomeF home_f(const InstDev &I, const float4 p) {
  return {p.x, p.y, p.z, fabsf(p.w), (float)I.lx, (float)I.ly, (float)I.lz,
          I.periodicity != 0 ? I.slack : -I.slack};
}

// The conservative float test of candidate qs (sorted position) against a home at sorted
// position s: rounding moves the float distance by less than 7e-7 of the largest box
// length, the slack is 2e-6 of it.  Nearly every candidate of the sweep fails it, so it
// reads only the candidate's float record.
// kLarge: the home particle is above the cut and sweeps a full stencil; it takes every
// small candidate and the large ones that follow it in sorted order.  Otherwise the home
// particle is small, sweeps the half stencil and leaves large candidates to them.
template <bool kLarge>
__device__ __forceinline__ bool near_float(const float4 c, int32_t qs, int32_t s, const HomeF &h) {
  if (c.w < 0.f && (!kLarge || qs <= s)) return false;
  float fx = c.x - h.x, fy = c.y - h.y, fz = c.z - h.z;
  if (h.slack > 0.f && fabsf(fx) > 0.5f * h.lx) fx = fx - copysignf(h.lx, fx);
  if (fabsf(fy) > 0.5f * h.ly) fy = fy - copysignf(h.ly, fy);
  if (fabsf(fz) > 0.5f * h.lz) fz = fz - copysignf(h.lz, fz);
  const float rf = h.r + fabsf(c.w) + fabsf(h.slack);
  return fx * fx + fy * fy + fz * fz <= rf * rf;
}

// What the exact tests of a pair take of one particle, from the pool: position, squared
// semi-axes and bounding radius, symmetry axis in the lab frame (first column of R(q)).
struct PairEnd {
  double x, y, z, r, a2, b2, ex, ey, ez;
};
__device__ __forceinline__ PairEnd pair_end(const PoolView &P, int32_t i) {
  PairEnd e;
  e.x = P.st[0][i]; e.y = P.st[1][i]; e.z = P.st[2][i];
  const double ea = P.pc[0][i], eb = P.pc[1][i];
  const double q0 = P.st[6][i], q1 = P.st[7][i], q2 = P.st[8][i], q3 = P.st[9][i];
  e.r = fmax(ea, eb);
  e.a2 = ea * ea;
  e.b2 = eb * eb;
  e.ex = 1.0 - 2.0 * (q2 * q2 + q3 * q3);
  e.ey = 2.0 * (q1 * q2 + q0 * q3);
  e.ez = 2.0 * (q1 * q3 - q0 * q2);
  return e;
}

// One candidate (sorted positions s, qs) of the sweep that passed near_float: FP64
// bounding-sphere test, centre-line separation test, reference box adjacency, then emission
// with the reference's ordering keys.
// Out of line, so that its FP64 state takes no registers from the sweep.
static __device__ __noinline__ void search_candidate(const InstDev *__restrict__ insts, const PoolView *pv,
                                                     const int32_t *sorted, uint32_t *mark, int32_t s, int32_t qs,
                                                     PairRec *pairs, unsigned long long *npairs, int64_t cap,
                                                     Status *st) {
  const PoolView &P = *pv;
  const int32_t pslot = sorted[s], qslot = sorted[qs];
  const InstDev &I = insts[P.inst[pslot]];
  const bool perx = I.periodicity != 0;
  const PairEnd p = pair_end(P, pslot), q = pair_end(P, qslot);
  double dx = q.x - p.x, dy = q.y - p.y, dz = q.z - p.z;
  if (perx && fabs(dx) > I.lx / 2) dx = dx - copysign(I.lx, dx);
  if (fabs(dy) > I.ly / 2.) dy = dy - copysign(I.ly, dy);
  if (fabs(dz) > I.lz / 2.) dz = dz - copysign(I.lz, dz);
  const double rr = (p.r + q.r) * (1.0 + 1e-9);
  const double d2 = dx * dx + dy * dy + dz * dz;
  if (d2 > rr * rr) return;
  // Support-function test along the centre line: for unit d, the extent of a
  // spheroid is h(d) = sqrt(b^2 + (a^2-b^2)(e.d)^2).  If h_p + h_q < |d| the two
  // bodies are disjoint, so no contact point can lie inside the other body
  // (ellipsoid_contact_detection.f90:125) and the reference cannot flag the pair.
  if (d2 > 0.0) {
    const double dist = sqrt(d2), inv = 1.0 / dist;
    const double ux = dx * inv, uy = dy * inv, uz = dz * inv;
    const double cp = p.ex * ux + p.ey * uy + p.ez * uz;
    const double cq = q.ex * ux + q.ey * uy + q.ez * uz;
    const double hp = sqrt(fmax(p.b2 + (p.a2 - p.b2) * cp * cp, 0.0));
    const double hq = sqrt(fmax(q.b2 + (q.a2 - q.b2) * cq * cq, 0.0));
    if (hp + hq < dist * (1.0 - 1e-9)) return;
  }
  atomicAdd(&st->n_near, 1ull);
  // reference adjacency of the two boxes (collision_box_connectivity.f90)
  const int pi = box_coord(p.x, I.xminbox, I.dxbox, I.nxbox), pj = box_coord(p.y, I.yminbox, I.dybox, I.nybox);
  const int pk = box_coord(p.z, I.zminbox, I.dzbox, I.nzbox);
  const int qi = box_coord(q.x, I.xminbox, I.dxbox, I.nxbox), qj = box_coord(q.y, I.yminbox, I.dybox, I.nybox);
  const int qk = box_coord(q.z, I.zminbox, I.dzbox, I.nzbox);
  if ((pi | pj | pk | qi | qj | qk) < 0) return;   // already reported as out of grid
  const int di = wrap_delta(qi - pi, I.nxbox, perx);
  const int dj = wrap_delta(qj - pj, I.nybox, true);
  const int dk = wrap_delta(qk - pk, I.nzbox, true);
  if (di < -1 || di > 1 || dj < -1 || dj > 1 || dk < -1 || dk > 1) return;
  const int32_t idp = P.id[pslot], idq = P.id[qslot];
  PairRec r;
  int slot;
  bool home_is_p;
  if (di == 0 && dj == 0 && dk == 0) {
    slot = 0;
    home_is_p = idp < idq;
  } else {
    const int idx = (di + 1) * 9 + (dj + 1) * 3 + (dk + 1);
    slot = c_fwd_slot[idx];
    home_is_p = slot > 0;
    if (!home_is_p) slot = c_fwd_slot[26 - idx];
  }
  // the home's box (both particles' box where slot = 0)
  const int hi = home_is_p ? pi : qi, hj = home_is_p ? pj : qj, hk = home_is_p ? pk : qk;
  const unsigned long long ijk =
      (unsigned long long)(hi + 1) + (unsigned long long)hj * I.nxbox + (unsigned long long)hk * I.nxbox * I.nybox;
  const int32_t idh = home_is_p ? idp : idq, idn = home_is_p ? idq : idp;
  r.home = home_is_p ? pslot : qslot;
  r.near = home_is_p ? qslot : pslot;
  r.k1 = ijk;
  r.k2 = ((unsigned long long)idh << 34) | ((unsigned long long)slot << 30) | (unsigned long long)idn;
  emit_pair(pairs, npairs, cap, r, mark, st);
}

__device__ __forceinline__ int wrap_cell(int c, int n) { return c < 0 ? c + n : (c >= n ? c - n : c); }

// Pair search over the search grid.  The cell edge is at least twice the cut radius,
// so two small particles (bounding radius <= cut) can only meet in the same or an
// adjacent cell; a small particle sweeps the half stencil of its cell: the 13 forward
// neighbours that follow it in (z, y, x) order, (cx+1, cy, cz), the three cells
// cx-1..cx+1 of row (cy+1, cz) and the nine of layer cz+1.  Cells are numbered
// x-fastest, so these are five x-rows, each one or two contiguous ranges of sorted
// particles; the home cell is swept from the next sorted particle on.  A large particle (radius above the
// cut, rare) sweeps every cell within its radius plus the largest radius.  Every pair is
// visited exactly once.
#ifndef GP_SEARCH_MIN_BLOCKS
#define GP_SEARCH_MIN_BLOCKS 4
#endif

constexpr int kSearchThreads = 288;
constexpr int kMaxRanges = 10;   // 5 rows, each at most two contiguous ranges

// Each lane takes one home particle (32 consecutive sorted particles per warp) and works
// out the ranges of sorted particles its half stencil must test: the five forward rows
// of cells, trimmed to the cells within reach; the rows' cell records are requested in two
// batches, each before the first of them is looked at.  The warp then tests all its homes'
// candidates together, 32 at a time: candidate idx of the warp's concatenated lists goes
// to lane idx mod 32, which looks up the owning home and range in shared memory.  Lanes
// stay busy however unevenly the candidates fall among the homes.  The candidates that pass
// wait in the warp's queue until there are 32 for the exact tests, or the warp has no more
// homes: one at a time in their lanes they held up the whole warp, once for 32 homes at
// 16.8 M particles and seven times in a packed ensemble.  Homes above the cut
// radius sweep their wide stencil afterwards, each on its own lane.  Everything up to the
// candidates that pass is FP32, widened by the slack that covers its rounding; about one
// candidate in 100 passes and reads its two particles from the pool.  What bounds it is the
// latency of the lookups, half of it in forming the ranges, with 36 warps an SM (1.28 ms at
// 16.8 M particles with 32, 1.24 with 40: what then spills goes through an L1 that the lookups
// fill; 1.23 with one batch).
// Measured (B200): 16.8 M particles 1.55 ms -> 1.20, 1 M 0.080 -> 0.069, 20,000 packed 0.041
// -> 0.031.
__global__ void __launch_bounds__(kSearchThreads, GP_SEARCH_MIN_BLOCKS) k_search(
    const InstDev *__restrict__ insts, const PoolView *__restrict__ pv, int64_t n, SearchArrays sa,
    PairRec *__restrict__ pairs, unsigned long long *npairs, int64_t cap, Status *st) {
  // no halt test here: this kernel is what raises the flag, and a later block must not
  // skip its pairs because an earlier one overflowed (the count it leaves in
  // pairs_needed sizes the buffers).  In a step after a halted one the binning did not
  // run and every cell is empty (its counts are zero between binnings), so the sweep finds
  // nothing.
  __shared__ HomeF homesf[kSearchThreads];
  __shared__ int32_t rstart[kSearchThreads][kMaxRanges];   // first sorted particle of a range
  __shared__ int32_t rcum[kSearchThreads][kMaxRanges];     // candidates of the home before it
  __shared__ int8_t rnum[kSearchThreads];
  __shared__ int2 passed[kSearchThreads / 32][64];  // candidates for the exact tests
  constexpr unsigned kFull = 0xffffffffu;
  const PoolView &P = *pv;
  const int t = threadIdx.x, lane = t & 31, wbase = t & ~31;
  const unsigned before = (1u << lane) - 1u;
  int2 *queue = passed[t >> 5];
  int nq = 0;
  const int64_t nact = sa.cell_start[sa.ncells];
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t s0 = (int64_t)blockIdx.x * blockDim.x + wbase; s0 < nact; s0 += stride) {
    const int64_t s = s0 + lane;
    int nr = 0;
    int32_t c = 0;
    bool large = false;
    if (s < nact) {
      const float4 p = sa.spk[s];
      const int32_t pslot = sa.sorted[s], cell = sa.cell_of[pslot];
      const InstDev &I = insts[P.inst[pslot]];
      homesf[t] = home_f(I, p);
      large = p.w < 0.f;
      if (!large) {
        int cx, cy, cz;
        cell_coords(I, cell, cx, cy, cz);
        const int nfx = I.nfx, nfy = I.nfy, nfz = I.nfz;
        const bool perx = I.periodicity != 0;
        const int xl = cx > 0 ? cx - 1 : nfx - 1, xr = cx + 1 < nfx ? cx + 1 : 0;
        const int yu = wrap_cell(cy + 1, nfy), zu = wrap_cell(cz + 1, nfz);
        const int32_t rows[5] = {cell_row(I, cy, cz), cell_row(I, yu, cz), cell_row(I, wrap_cell(cy - 1, nfy), zu),
                                 cell_row(I, cy, zu), cell_row(I, yu, zu)};
        // the row's three cells: where the left begins, the middle begins and ends, the right
        // ends, and the largest radius in each
        int32_t sl[5], sm[5], se[5], sr[5];
        float ml[5], mm[5], mr[5];
        // Small candidates have radius <= rcut, so only cells whose box comes within
        // R = rp + rcut of this particle can hold a partner: rows and end cells farther
        // away are skipped (distances to the neighbour boxes from the offsets inside the
        // home cell, shortened by the slack).
        const float e = I.slack, rp = p.w * (1.0f + 1e-6f);
        const float hx = (float)I.hfx, hy = (float)I.hfy, hz = (float)I.hfz;
        const float R = rp + (float)I.rcut * (1.0f + 1e-6f), R2 = R * R;
        const float fx = p.x - cx * hx, fy = p.y - cy * hy, fz = p.z - cz * hz;
        const float dxl = fmaxf(fx - e, 0.f), dxh = fmaxf(hx - fx - e, 0.f);
        const float dyl = fmaxf(fy - e, 0.f), dyh = fmaxf(hy - fy - e, 0.f);
        const float dzh = fmaxf(hz - fz - e, 0.f);
        const bool left_ok = (cx - 1 >= 0 || perx), right_ok = (cx + 1 < nfx || perx);
        auto add = [&](int32_t a0, int32_t a1) {
          if (a1 > a0) {
            rstart[t][nr] = a0;
            rcum[t][nr] = c;
            c += a1 - a0;
            ++nr;
          }
        };
        auto request = [&](int r) {
          const int32_t row = rows[r];
          sl[r] = sm[r] = 0;
          ml[r] = mm[r] = 0.f;
          if (r > 0) {   // the home's own row begins at the home
            sl[r] = __ldg(sa.cell_start + row + xl);
            sm[r] = __ldg(sa.cell_start + row + cx);
            ml[r] = __ldg(sa.cell_rmax + row + xl);
            mm[r] = __ldg(sa.cell_rmax + row + cx);
          }
          se[r] = __ldg(sa.cell_start + row + cx + 1);
          sr[r] = __ldg(sa.cell_start + row + xr + 1);
          mr[r] = __ldg(sa.cell_rmax + row + xr);
        };
        request(0); request(1);
#pragma unroll
        for (int r = 0; r < 5; ++r) {
          if (r == 2) { request(2); request(3); request(4); }
          const float dyb = r == 2 ? dyl : (r == 3 ? 0.f : dyh);
          const float dyz2 = r == 0 ? 0.f : (r == 1 ? dyh * dyh : dyb * dyb + dzh * dzh);
          // each cell within reach of its own largest radius
          auto reaches = [&](float most, float d2) {
            const float m = rp + most;
            return d2 <= R2 && d2 <= m * m;
          };
          const bool row_ok = dyz2 <= R2;
          const bool use_l = r > 0 && row_ok && left_ok && reaches(ml[r], dxl * dxl + dyz2);
          const bool use_r = row_ok && right_ok && reaches(mr[r], dxh * dxh + dyz2);
          // the home cell from s+1 on; its neighbours' middle cell whenever an end is used
          const bool use_m = r == 0 || use_l || use_r || (row_ok && reaches(mm[r], dyz2));
          int32_t a0 = r == 0 ? (int32_t)s + 1 : sm[r], a1 = use_m ? se[r] : a0;
          if (use_l && cx > 0) a0 = sl[r];
          if (use_r && cx + 1 < nfx) a1 = sr[r];
          if ((use_l && cx == 0) || (use_r && cx + 1 == nfx)) {   // nfx >= 3: one of the two
            const int32_t row = rows[r];
            const int32_t b0 = use_l && cx == 0 ? sl[r] : __ldg(sa.cell_start + row);
            const int32_t b1 = use_l && cx == 0 ? __ldg(sa.cell_start + row + nfx) : sr[r];
            add(b0, b1);
          }
          add(a0, a1);
        }
      }
    }
    rnum[t] = (int8_t)nr;
    __syncwarp();
    // the warp's candidate lists, concatenated in lane order
    int32_t incl = c;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int32_t v = __shfl_up_sync(kFull, incl, d);
      if (lane >= d) incl += v;
    }
    const int32_t total = __shfl_sync(kFull, incl, 31);
    const int32_t excl = incl - c;
    for (int32_t base = 0; base < total; base += 32) {
      const int32_t idx = base + lane;
      // the last lane o whose list starts at or before idx owns it
      int o = 0;
#pragma unroll
      for (int step = 16; step > 0; step >>= 1) {
        const int32_t e = __shfl_sync(kFull, excl, (o + step) & 31);
        if (o + step < 32 && e <= idx) o += step;
      }
      const int32_t eo = __shfl_sync(kFull, excl, o);
      bool pass = false;
      int32_t q = 0;
      if (idx < total) {
        const int to = wbase + o;
        const int32_t k = idx - eo;
        int j = 0;
        const int no = rnum[to];
        while (j + 1 < no && rcum[to][j + 1] <= k) ++j;
        q = rstart[to][j] + (k - rcum[to][j]);
        pass = near_float<false>(sa.spk[q], q, 0, homesf[to]);
      }
      const unsigned m = __ballot_sync(kFull, pass);
      if (m != 0u) {
        if (pass) queue[nq + __popc(m & before)] = make_int2((int32_t)(s0 + o), q);
        nq += __popc(m);
        __syncwarp();
        if (nq >= 32) {
          nq -= 32;
          const int2 e = queue[nq + lane];
          search_candidate(insts, &P, sa.sorted, sa.mark, e.x, e.y, pairs, npairs, cap, st);
          __syncwarp();
        }
      }
    }
    if (large) {
      // a particle above the cut: every cell within its radius plus the largest radius
      const int32_t pslot = sa.sorted[s];
      const InstDev &I = insts[P.inst[pslot]];
      const int nfx = I.nfx, nfy = I.nfy, nfz = I.nfz;
      int cx, cy, cz;
      cell_coords(I, sa.cell_of[pslot], cx, cy, cz);
      const HomeF hf = homesf[t];
      const bool perx = I.periodicity != 0;
      const double reach = (fmax(P.pc[0][pslot], P.pc[1][pslot]) + I.rmax) * (1.0 + 1.0e-6);
      const int rx = (int)ceil(reach / I.hfx), ry = (int)ceil(reach / I.hfy), rz = (int)ceil(reach / I.hfz);
      const bool ally = 2 * ry + 1 >= nfy, allz = 2 * rz + 1 >= nfz, allx = 2 * rx + 1 >= nfx;
      const int y0 = ally ? 0 : cy - ry, y1 = ally ? nfy - 1 : cy + ry;
      const int z0 = allz ? 0 : cz - rz, z1 = allz ? nfz - 1 : cz + rz;
      int lo = allx ? 0 : cx - rx, hi = allx ? nfx - 1 : cx + rx;
      if (!perx) { lo = max(lo, 0); hi = min(hi, nfx - 1); }
      for (int zz = z0; zz <= z1; ++zz) {
        const int wz = wrap_cell(zz, nfz);
        for (int yy = y0; yy <= y1; ++yy) {
          const int32_t row = cell_row(I, wrap_cell(yy, nfy), wz);
          for (int x = lo; x <= hi;) {
            const int w = wrap_cell(x, nfx), len = min(nfx - w, hi - x + 1);   // up to the row's end
            const int32_t q1 = sa.cell_start[row + w + len];
            for (int32_t qs = sa.cell_start[row + w]; qs < q1; ++qs)
              if (qs != s && near_float<true>(sa.spk[qs], qs, (int32_t)s, hf))
                search_candidate(insts, &P, sa.sorted, sa.mark, (int32_t)s, qs, pairs, npairs, cap, st);
            x += len;
          }
        }
      }
    }
    __syncwarp();   // the records are rewritten by the warp's next 32 homes
  }
  if (lane < nq) search_candidate(insts, &P, sa.sorted, sa.mark, queue[lane].x, queue[lane].y, pairs, npairs, cap, st);
}

void launch_search(const InstDev *insts, const PoolView *pv, int64_t n, SearchArrays sa, PairRec *pairs, unsigned long long *npairs,
                   int64_t cap_pairs, Status *st, int grid, cudaStream_t s) {
  k_search<<<grid, kSearchThreads, 0, s>>>(insts, pv, n, sa, pairs, npairs, cap_pairs, st);
}

// ---------------------------------------------------------------------------
// 5. lexicographically-first maximal matching of the colliding pairs
//    (the outcome of the COLOR walk, collision_interaction.f90:190-207,397-398)
// ---------------------------------------------------------------------------
// Rounds over the live pairs: each particle's smallest live key (A), the pairs that hold it
// at both ends are accepted and colour their particles (B), pairs with a coloured particle
// die and the others give their particles back (C).  A particle's smallest key is kept as
// the index of the pair that has it, so a round takes three barriers (five with the two key
// words kept apart).  What bounds it is the latency of the scattered accesses between two
// barriers, so from kMatchAlone pairs on eight blocks of a cluster share the pairs, and its
// barrier takes the place of the block's.  Measured (B200, with the response): 50,900 pairs
// 0.88 ms in one block with five barriers -> 0.16; 3,260 pairs 0.068 alone, 0.041 shared;
// 861 pairs 0.031 alone, 0.037 shared.
constexpr int kMatchThreads = 1024, kMatchBlocks = 8;
constexpr int64_t kMatchAlone = 2048;

__device__ __forceinline__ bool key_less(const CollRec &a, const CollRec &b) {
  return a.k1 < b.k1 || (a.k1 == b.k1 && a.k2 < b.k2);
}

// best[p] <- e if pair e's key is below that of the pair held there (~0: none)
__device__ __forceinline__ void hold_smallest(uint32_t *best, const CollRec *coll, uint32_t e, const CollRec &r) {
  uint32_t cur = atomicCAS(best, ~0u, e);
  while (cur != ~0u && key_less(r, coll[cur])) {   // keys only fall, so this ends
    const uint32_t was = atomicCAS(best, cur, e);
    if (was == cur) break;
    cur = was;
  }
}

__global__ void __cluster_dims__(kMatchBlocks, 1, 1) __launch_bounds__(kMatchThreads)
    k_match(const CollRec *__restrict__ coll, const unsigned long long *__restrict__ ncoll, int64_t cap,
            unsigned long long *best64, int8_t *matched, int8_t *state, Status *st) {
  if (step_halted(st)) return;
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ unsigned left[2];   // live pairs after an even and an odd round (block 0's are used)
  const int64_t nc = (int64_t)min(*ncoll, (unsigned long long)cap);
  const bool alone = nc <= kMatchAlone;
  if (alone && blockIdx.x != 0) return;
  // one 32-bit index a particle, at the particle's own 64-bit word (all ones at rest)
  uint32_t *best = reinterpret_cast<uint32_t *>(best64);
  const int64_t first = (alone ? 0 : (int64_t)blockIdx.x * kMatchThreads) + threadIdx.x;
  const int64_t stride = alone ? kMatchThreads : kMatchThreads * kMatchBlocks;
  auto sync = [&]() {
    if (alone) __syncthreads(); else cluster.sync();
  };
  unsigned *const left0 = cluster.map_shared_rank(left, 0);
  if (threadIdx.x < 2) left[threadIdx.x] = 0u;
  for (int64_t e = first; e < nc; e += stride) state[e] = 0;
  sync();
  bool live = nc > 0;
  for (int64_t round = 0; live; ++round) {
    for (int64_t e = first; e < nc; e += stride) {
      if (state[e] != 0) continue;
      const CollRec &r = coll[e];
      hold_smallest(best + 2 * (int64_t)r.home, coll, (uint32_t)e, r);
      hold_smallest(best + 2 * (int64_t)r.near, coll, (uint32_t)e, r);
    }
    sync();
    if (blockIdx.x == 0 && threadIdx.x == 0) left[(round + 1) & 1] = 0u;
    for (int64_t e = first; e < nc; e += stride) {
      if (state[e] != 0) continue;
      const CollRec &r = coll[e];
      if (__ldcg(best + 2 * (int64_t)r.home) == (uint32_t)e && __ldcg(best + 2 * (int64_t)r.near) == (uint32_t)e) {
        state[e] = 1;
        __stcg(matched + r.home, (int8_t)1);
        __stcg(matched + r.near, (int8_t)1);
      }
    }
    sync();
    unsigned cnt = 0;
    for (int64_t e = first; e < nc; e += stride) {
      if (state[e] != 0) continue;
      const CollRec &r = coll[e];
      if (__ldcg(matched + r.home) || __ldcg(matched + r.near)) {
        state[e] = 2;
      } else {
        __stcg(best + 2 * (int64_t)r.home, ~0u);
        __stcg(best + 2 * (int64_t)r.near, ~0u);
        ++cnt;
      }
    }
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if ((threadIdx.x & 31) == 0 && cnt) atomicAdd(left0 + (round & 1), cnt);
    sync();
    live = *(volatile unsigned *)(left0 + (round & 1)) != 0u;
    if (live && round > nc) {   // every round accepts at least one pair; cannot happen
      if (first == 0) set_error(st, GP_ETIMEOUT, round);
      live = false;
    }
  }
  for (int64_t e = first; e < nc; e += stride) {
    const CollRec &r = coll[e];
    __stcg(best + 2 * (int64_t)r.home, ~0u);
    __stcg(best + 2 * (int64_t)r.near, ~0u);
    __stcg(matched + r.home, (int8_t)0);
    __stcg(matched + r.near, (int8_t)0);
  }
  if (!alone) cluster.sync();   // block 0's counters stay until every block has read them
}

void launch_match(const CollRec *coll, const unsigned long long *ncoll, int64_t cap_coll, unsigned long long *best1,
                  int8_t *matched, int8_t *state, Status *st, cudaStream_t s) {
  k_match<<<kMatchBlocks, kMatchThreads, 0, s>>>(coll, ncoll, cap_coll, best1, matched, state, st);
}

// ---------------------------------------------------------------------------
// Data movement
// ---------------------------------------------------------------------------
// Internal field layout from a reference-layout or interior source (one component).
template <typename T>
__global__ void k_field_layout(T *__restrict__ dst, int nx, int ny, int nz, int ncomp, int comp,
                               const double *__restrict__ src, int src_layout, int ghost_mode) {
  const int64_t sx = nx + 3, sy = ny + 4, sz = nz + 4;
  const int64_t total = sx * sy * sz;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int ix = (int)(t % sx), jy = (int)((t / sx) % sy), kz = (int)(t / (sx * sy));
    int i = ix;
    if (ix == 0) i = nx;
    else if (ix == nx + 1) i = 1;
    else if (ix == nx + 2) i = 2;
    const int j = jy - 1, k = kz - 1;   // reference indices, -1..N+2
    double v;
    if (src_layout == GP_LAYOUT_REFERENCE) {
      v = src[(int64_t)(i - 1) + (int64_t)nx * ((int64_t)(j + 1) + (int64_t)(ny + 4) * (int64_t)(k + 1))];
    } else {
      const bool inside = (j >= 1 && j <= ny && k >= 1 && k <= nz);
      if (!inside && ghost_mode == GP_GHOST_ZERO) {
        v = 0.0;
      } else {
        const int jj = (j < 1) ? j + ny : (j > ny ? j - ny : j);
        const int kk = (k < 1) ? k + nz : (k > nz ? k - nz : k);
        v = src[(int64_t)(i - 1) + (int64_t)nx * ((int64_t)(jj - 1) + (int64_t)ny * (int64_t)(kk - 1))];
      }
    }
    dst[t * ncomp + comp] = (T)v;
  }
}

void launch_field_layout(void *dst, int prec, int nx, int ny, int nz, int ncomp, int comp, const double *src,
                         int src_layout, int ghost_mode, cudaStream_t s) {
  const int grid = 148 * 8;
  if (prec == GP_PREC_MIXED)
    k_field_layout<float><<<grid, 256, 0, s>>>(static_cast<float *>(dst), nx, ny, nz, ncomp, comp, src, src_layout,
                                                ghost_mode);
  else
    k_field_layout<double><<<grid, 256, 0, s>>>(static_cast<double *>(dst), nx, ny, nz, ncomp, comp, src,
                                                 src_layout, ghost_mode);
}

// A node's components in one go, a warp to a row of nodes: six coalesced reads and whole
// sectors written by one instruction each, where k_field_layout, one component a launch,
// writes 8 bytes of each 64-byte node.  Bound by memory.  Measured (B200, 128^3, FP64
// field): six launches 174 us -> 44 (89 with 16-byte stores, two to a sector).
template <typename T, bool kVorticity>
__global__ void __launch_bounds__(256) k_field_nodes(T *__restrict__ dst, int nx, int ny, int nz,
                                                     const double *__restrict__ vel,
                                                     const double *__restrict__ vort) {
  static_assert(kFieldStride == 8, "a node is eight values");
  const int sx = nx + 3, sy = ny + 4, sz = nz + 4, lane = threadIdx.x & 31;
  const int64_t np = (int64_t)nx * ny * nz;
  const unsigned rows = (unsigned)sy * (unsigned)sz, warps = gridDim.x * (blockDim.x >> 5);
  for (unsigned row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); row < rows; row += warps) {
    const int kz = (int)(row / (unsigned)sy), jy = (int)(row - (unsigned)kz * (unsigned)sy);
    const int j = jy - 1, k = kz - 1;   // reference indices, -1..N+2
    const bool inside = j >= 1 && j <= ny && k >= 1 && k <= nz;
    const int jj = (j < 1) ? j + ny : (j > ny ? j - ny : j), kk = (k < 1) ? k + nz : (k > nz ? k - nz : k);
    const int64_t from = (int64_t)nx * ((int64_t)(jj - 1) + (int64_t)ny * (int64_t)(kk - 1));
    T *out = dst + (int64_t)row * sx * kFieldStride;
    for (int ix = lane; ix < sx; ix += 32) {
      const int64_t e = from + (ix == 0 ? nx - 1 : (ix > nx ? ix - nx - 1 : ix - 1));
      alignas(16) T v[kFieldStride] = {};
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        v[c] = (T)vel[c * np + e];
        if (kVorticity) v[3 + c] = inside ? (T)vort[c * np + e] : (T)0;
      }
      T *o = out + (int64_t)ix * kFieldStride;
      if (kVorticity) {
        if constexpr (sizeof(T) == 8) {
          asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(o), "d"(v[0]), "d"(v[1]), "d"(v[2]), "d"(v[3])
                       : "memory");
          asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(o + 4), "d"(v[4]), "d"(v[5]), "d"(v[6]), "d"(v[7])
                       : "memory");
        } else {
          asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(o), "f"(v[0]), "f"(v[1]),
                       "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                       : "memory");
        }
      } else {
#pragma unroll
        for (int c = 0; c < 3; ++c) o[c] = v[c];
      }
    }
  }
}

void launch_field_nodes(void *dst, int prec, int nx, int ny, int nz, const double *vel, const double *vort,
                        cudaStream_t s) {
  const int grid = 148 * 8;
  auto run = [&](auto *d) {
    using T = std::remove_pointer_t<decltype(d)>;
    if (vort) k_field_nodes<T, true><<<grid, 256, 0, s>>>(d, nx, ny, nz, vel, vort);
    else k_field_nodes<T, false><<<grid, 256, 0, s>>>(d, nx, ny, nz, vel, vort);
  };
  if (prec == GP_PREC_MIXED) run(static_cast<float *>(dst));
  else run(static_cast<double *>(dst));
}

// Retires class `inst`: its particles leave the binning, and the next advance drops them.
__global__ void k_retire(const PoolView *__restrict__ pv, int64_t n, int inst) {
  const PoolView P = *pv;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    if (P.inst[i] == inst) P.inst[i] = -1;
}

void launch_retire(const PoolView *pv, int64_t n, int inst, cudaStream_t s) {
  if (n > 0) k_retire<<<148 * 8, 256, 0, s>>>(pv, n, inst);
}

// One class into pool slots [begin, begin+n): particle k of the class is column entry
// src + k of the staged arrays (leading dimension ld); ids are 0-based within the class.
__global__ void k_init_pool(const PoolView *__restrict__ pv, int64_t begin, int64_t n, int inst,
                            const double *__restrict__ cols, const double *__restrict__ pcs, ConstRow row,
                            int64_t ld, int64_t src) {
  const PoolView P = *pv;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = begin + k, e = src + k;
#pragma unroll
    for (int c = 0; c < kNState; ++c) P.st[c][i] = cols[c * ld + e];
#pragma unroll
    for (int c = 0; c < kNConst; ++c) P.pc[c][i] = pcs ? pcs[c * ld + e] : row.v[c];
    P.id[i] = (int32_t)k;
    P.inst[i] = inst;
  }
}

void launch_init_pool(const PoolView *pv, int64_t begin, int64_t n, int inst, const double *cols, const double *pcs,
                      const ConstRow &row, int64_t ld, int64_t src, cudaStream_t s) {
  if (n <= 0) return;
  k_init_pool<<<148 * 8, 256, 0, s>>>(pv, begin, n, inst, cols, pcs, row, ld, src);
}

__global__ void k_iota(int32_t *a, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    a[i] = (int32_t)i;
}

void launch_iota(int32_t *a, int64_t n, cudaStream_t s) {
  if (n > 0) k_iota<<<148 * 8, 256, 0, s>>>(a, n);
}

// The slots are in class order and, within a class, in cell order, so classes on one field
// each sweep the whole of it, one after the other, and read it from HBM again.  Taken by the
// fraction of its class that lies before it, a run's neighbours in time are the other
// classes' runs at the same height, and the field passes through the L2 once.
// Run t belongs to the class of its middle slot m (or, the last one, of the last slot); runs
// are ordered by ((m - begin) / count, class), and a run's place is the number of runs of
// each class before it.
__global__ void k_run_order(const InstDev *__restrict__ insts, int ninst, int64_t n, int32_t *__restrict__ order) {
  const int64_t nruns = (n + kOrderedRun - 1) / kOrderedRun;
  constexpr int64_t kMid = kOrderedRun / 2;
  // first run whose middle is at slot x or later
  auto run_from = [&](int64_t x) { return min((x + kOrderedRun - 1 - kMid) / kOrderedRun, nruns); };
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nruns; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t m = t * kOrderedRun + kMid, slot = min(m, n - 1);
    int own = 0;
    while (own < ninst - 1 && !(slot < insts[own].begin + insts[own].count)) ++own;
    const int64_t mine = insts[own].count, f = m - insts[own].begin;
    int64_t place = 0;
    for (int k = 0; k < ninst; ++k) {
      const int64_t b = insts[k].begin, cnt = insts[k].count;
      if (cnt == 0) continue;
      // the last run's middle may lie past the last class
      const int64_t first = run_from(b), end = b + cnt == n ? nruns : run_from(b + cnt);
      // middles m' of class k with (m' - b) / cnt before f / mine: m' - b < x
      const int64_t v = f * cnt, q = v / mine;
      const int64_t x = (k < own || v % mine != 0) ? q + 1 : q;
      place += k == own ? t - first : min(max(run_from(b + x), first), end) - first;
    }
    order[place] = (int32_t)t;
  }
}

void launch_run_order(const InstDev *insts, int ninst, int64_t n, int32_t *order, cudaStream_t s) {
  if (n > 0) k_run_order<<<148 * 4, 128, 0, s>>>(insts, ninst, n, order);
}

// COLLISION_BOX_CONNECTIVITY (collision_box_connectivity.f90:42-322), NPROC=1.
__global__ void k_connectivity(int NXB, int NYB, int NZB, int periodicity, int32_t *ncon, int32_t *con) {
  const int64_t nbox = (int64_t)NXB * NYB * NZB;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nbox; t += (int64_t)gridDim.x * blockDim.x) {
    const int i0 = (int)(t % NXB) + 1, j0 = (int)((t / NXB) % NYB) + 1, k0 = (int)(t / ((int64_t)NXB * NYB)) + 1;
    auto BOX = [&](int i, int j, int k) { return (int32_t)(i + (j - 1) * NXB + (k - 1) * NXB * NYB); };
    int im1 = i0 - 1, ip1 = i0 + 1, jm1 = j0 - 1, jp1 = j0 + 1, km1 = k0 - 1, kp1 = k0 + 1;
    if (im1 < 1 && periodicity) im1 = NXB;
    if (ip1 > NXB && periodicity) ip1 = 1;
    if (jm1 < 1) jm1 = NYB;
    if (jp1 > NYB) jp1 = 1;
    if (km1 < 1) km1 = NZB;
    if (kp1 > NZB) kp1 = 1;
    int32_t c[27];
    int nn = 0;
    if (km1 >= 1 && jp1 <= NYB && ip1 <= NXB) c[nn++] = BOX(ip1, jp1, km1);   // box 9
    if (jm1 >= 1 && ip1 <= NXB) c[nn++] = BOX(ip1, jm1, k0);                  // box 12
    if (ip1 <= NXB) c[nn++] = BOX(ip1, j0, k0);                                // box 15
    if (jp1 <= NYB) {
      c[nn++] = BOX(i0, jp1, k0);                                               // box 17
      if (ip1 <= NXB) c[nn++] = BOX(ip1, jp1, k0);                             // box 18
    }
    if (kp1 <= NZB) {
      if (jm1 >= 1) {
        c[nn++] = BOX(i0, jm1, kp1);                                            // box 20
        if (ip1 <= NXB) c[nn++] = BOX(ip1, jm1, kp1);                          // box 21
      }
      if (im1 >= 1) c[nn++] = BOX(im1, j0, kp1);                               // box 22
      c[nn++] = BOX(i0, j0, kp1);                                               // box 23
      if (ip1 <= NXB) c[nn++] = BOX(ip1, j0, kp1);                             // box 24
      if (jp1 <= NYB) {
        if (im1 >= 1) c[nn++] = BOX(im1, jp1, kp1);                            // box 25
        c[nn++] = BOX(i0, jp1, kp1);                                            // box 26
        if (ip1 <= NXB) c[nn++] = BOX(ip1, jp1, kp1);                          // box 27
      }
    }
    const int64_t ijk = (i0 - 1) + (int64_t)(j0 - 1) * NXB + (int64_t)(k0 - 1) * NXB * NYB;
    ncon[ijk] = nn;
    for (int q = 0; q < 27; ++q) con[ijk * 27 + q] = (q < nn) ? c[q] : 0;
  }
}

void launch_connectivity(int nxb, int nyb, int nzb, int periodicity, int32_t *ncon, int32_t *con, cudaStream_t s) {
  k_connectivity<<<148 * 8, 128, 0, s>>>(nxb, nyb, nzb, periodicity, ncon, con);
}

}  // namespace gp
