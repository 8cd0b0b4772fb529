// gp_launch.h -- host-side launchers of the device kernels (one per translation unit
// so that the FP64 path can be compiled without FMA contraction).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include "gp_types.h"

namespace gp {

struct TailRec;   // gp_contact.cuh

// --- gp_kernels_fp64.cu (FP64 path, -fmad=false) ---
// ADV_PARTICLE_ELLP: advances particle perm[j] of *pv into slot j of *pv_alt, then swaps
// the two views (so *pv is current afterwards) and takes the gather's ticket back to zero.
// With mark non-null, the speculative pass: marked particles are left to
// launch_integrate_fix_*, which does both.  done: a counter, zero between launches.
// order (may be null): the order in which the gather takes runs of kOrderedRun slots
// (launch_run_order).
void launch_gather_fp64(const InstDev *insts, const PoolView *pv, const int32_t *perm, int64_t n,
                      const int32_t *order, double *const *fluid, unsigned long long *ticket, Status *st, int grid, cudaStream_t s);
void launch_integrate_fp64(const InstDev *insts, PoolView *pv, PoolView *pv_alt, const int32_t *perm, int64_t n,
                         double *const *fluid, Status *st, int grid, unsigned long long *done,
                         unsigned long long *ticket, cudaStream_t s, uint32_t *mark = nullptr);
void launch_integrate_fix_fp64(const InstDev *insts, PoolView *pv, PoolView *pv_alt, const PairRec *pairs,
                             const unsigned long long *npairs, int64_t cap_pairs, double *const *fluid,
                             uint32_t *mark, Status *st, int grid, unsigned long long *done,
                             unsigned long long *ticket, cudaStream_t s);
// order (or null): the indices of the points in the order to take them, as
// launch_point_order leaves them (bins: rows of mesh cells cut into runs of 2^shift cells,
// ny * nz * ((nx >> shift) + 1) of them; count: bins + 1 zeros; start: bins + 1; state:
// scan_tiles(bins) zeros; key, order: n).
void launch_interp(const InstDev *inst, bool mixed, int comp, int64_t n, const int32_t *order, const double *x,
                   const double *y, const double *z, double *out, Status *st, cudaStream_t s);
void launch_point_order(const InstDev *inst, int64_t n, int shift, int64_t bins, const double *x, const double *y,
                        const double *z, uint32_t *key, int32_t *count, int32_t *start,
                        unsigned long long *state, int32_t *order, Status *st, cudaStream_t s);
void launch_frozen_interp(const double *xain, const double *yain, const double *zain, int nx, int ny, int nz,
                          const double *uain, int64_t n, const double *x, const double *y, const double *z,
                          double *out, Status *st, cudaStream_t s);
int contact_grid_blocks();
void launch_contact(const InstDev *insts, const PoolView *pv, const PairRec *pairs, const unsigned long long *npairs,
                    int64_t cap_pairs, const TailRec *in, const unsigned long long *nin, int64_t cap_in,
                    CollRec *coll, unsigned long long *ncoll, int64_t cap_coll, unsigned long long *queue,
                    ContactStatRec *cst, unsigned long long *ncst, int64_t cap_cst, TailRec *out,
                    unsigned long long *nout, int64_t cap_out, int budget, const uint32_t *order,
                    uint32_t *hist, int64_t nhist, Status *st, int grid, cudaStream_t s);
size_t tail_record_bytes();
// The contact queue's order (gp_contact.cu): order[0, *nsolve) are the candidate pairs that
// are not proven apart, longest predicted solve first; the record hist[0, nhist) is cleared
// for this phase's solves.  bins holds 2 * kQueueBins counters, zero at the launch; key one
// byte per pair slot.
constexpr int kQueueBins = 256;
void launch_queue_order(const InstDev *insts, const PoolView *pv, const PairRec *pairs,
                        const unsigned long long *npairs, int64_t cap_pairs, uint32_t *hist, int64_t nhist,
                        uint8_t *key, uint32_t *bins, uint32_t *order, unsigned long long *nsolve, const Status *st,
                        int grid, cudaStream_t s);
void launch_response(const InstDev *insts, const PoolView *pv, const CollRec *coll, const unsigned long long *ncoll,
                     int64_t cap_coll, const int8_t *state, int32_t *acc_list, unsigned long long *nacc, Status *st,
                     int grid, cudaStream_t s);
// per-routine drop-ins (n items; all pointers device)
void launch_force_batch(int64_t n, const double *pcs /*n*10*/, double visc, const double *up,
                        const double *uf, const double *quat, double *fdrag, double *flift, Status *st,
                        cudaStream_t s);
void launch_torque_batch(int64_t n, const double *pcs, double visc, const double *omega, const double *quat,
                         const double *pup, const double *pufap, const double *pvort, double *tp, double *tr,
                         Status *st, cudaStream_t s);
void launch_quat_batch(int64_t n, double *quat, const double *omega, double dt, cudaStream_t s);
void launch_euler_batch(int64_t n, const double *ip /*n*3*/, double dt, double *omega, cudaStream_t s);
void launch_contact_batch(int64_t n, const double *shapes /*n*4: a1 b1 a2 b2*/, const double *centres,
                          const double *quats, int32_t *flag, double *e1, double *e2, double *cn, cudaStream_t s);
void launch_response_batch(int64_t n, double ecp, double mup, const double *ip /*n*3*/, double *p1 /*n*10*/,
                           double *p2, const double *r1, const double *r2, const double *nrm, Status *st,
                           cudaStream_t s);

// --- gp_gather_tma.cu: the FP32 gather with each stencil box staged by the TMA ---
// make_field_map: tensor map over one FP32 field slot ([z][y][x][8], the interior sizes
// given); gather_tma_prepare: the kernel's shared-memory limit, once, outside any stream
// capture; launch_gather_tma: as launch_gather_mixed, for instances that all read the
// mapped field.
int make_field_map(const void *field, int nx, int ny, int nz, CUtensorMap *out);
int gather_tma_prepare();
size_t gather_tma_smem_bytes();
void launch_gather_tma(const CUtensorMap &map, const InstDev *insts, const PoolView *pv, const int32_t *perm,
                       int64_t n, double *const *fluid, unsigned long long *ticket, Status *st, int grid,
                       cudaStream_t s);

// --- gp_stats.cu (-fmad=false) ---
void launch_stat_partfluid(const InstDev *insts, const PoolView *pv, int64_t n, int inst, double *const *fluid,
                           const int32_t *groups, int ngroups, double rhof, double ppi, double *partial,
                           int nblocks, double *out, Status *st, cudaStream_t s);
void launch_collision_stats(const CollRec *coll, const unsigned long long *ncoll, int64_t cap_coll,
                            const int8_t *state, unsigned long long *best1, unsigned long long *best2,
                            const ContactStatRec *rec, const unsigned long long *nrec, int64_t cap_rec,
                            const PoolView *pv, const int32_t *const *group_tab, const int32_t *ngroups, double *acc,
                            unsigned long long *steps, Status *st, cudaStream_t s);

// --- gp_kernels_mixed.cu ---
void launch_gather_mixed(const InstDev *insts, const PoolView *pv, const int32_t *perm, int64_t n,
                      const int32_t *order, double *const *fluid, unsigned long long *ticket, Status *st, int grid, cudaStream_t s);
void launch_integrate_mixed(const InstDev *insts, PoolView *pv, PoolView *pv_alt, const int32_t *perm, int64_t n,
                         double *const *fluid, Status *st, int grid, unsigned long long *done,
                         unsigned long long *ticket, cudaStream_t s, uint32_t *mark = nullptr);
void launch_integrate_fix_mixed(const InstDev *insts, PoolView *pv, PoolView *pv_alt, const PairRec *pairs,
                             const unsigned long long *npairs, int64_t cap_pairs, double *const *fluid,
                             uint32_t *mark, Status *st, int grid, unsigned long long *done,
                             unsigned long long *ticket, cudaStream_t s);
void launch_iota(int32_t *a, int64_t n, cudaStream_t s);

// --- gp_search.cu ---
// What k_bin_count clears for the phases after it.
struct PhaseClear {
  unsigned long long *counters;     // those of the first ncounters (at most 32) in counter_mask
  unsigned counter_mask;
  int ncounters;
  uint32_t *bins;                   // or null
  int nbins;
  unsigned long long *tile_state;   // the scan's
  int64_t tiles;
};
void launch_bin_count(const InstDev *insts, const PoolView *pv, int64_t n, SearchArrays sa, Status *st, int grid,
                      const PhaseClear &clear, cudaStream_t s);
// Exclusive scan of n counts; state: scan_tiles(n) words, zero at the launch; clears
// clear[0..n] on the way where it is not null.
int64_t scan_tiles(int64_t n);
void launch_scan(const int32_t *in, int32_t *out, int64_t n, unsigned long long *state, float *clear, Status *st,
                 cudaStream_t s);
void launch_bin_scatter(const InstDev *insts, const PoolView *pv, int64_t n, SearchArrays sa, Status *st, int grid,
                        cudaStream_t s);
void launch_search(const InstDev *insts, const PoolView *pv, int64_t n, SearchArrays sa, PairRec *pairs, unsigned long long *npairs,
                   int64_t cap_pairs, Status *st, int grid, cudaStream_t s);
void launch_match(const CollRec *coll, const unsigned long long *ncoll, int64_t cap_coll, unsigned long long *best1,
                  int8_t *matched, int8_t *state, Status *st, cudaStream_t s);
// All nodes of an internal field from interior arrays, three components back to back each:
// the velocity with periodic ghosts and, unless null, the vorticity with zero ghosts.
void launch_field_nodes(void *dst, int prec, int nx, int ny, int nz, const double *vel, const double *vort,
                        cudaStream_t s);
// The same into a context's field slot (of the same mesh); returns when it is done.
int couple_field(gp_ctx *c, int32_t field, const double *vel, const double *vort);
void launch_field_layout(void *dst, int prec, int nx, int ny, int nz, int ncomp, int comp, const double *src,
                         int src_layout, int ghost_mode, cudaStream_t s);
void launch_retire(const PoolView *pv, int64_t n, int inst, cudaStream_t s);
// One particle's constants, as an argument.
struct ConstRow {
  double v[kNConst];
};
// Particles of one class into pool slots [begin, begin + n) from columns of leading dimension
// ld, from row src on; pcs null: all have the constants `row`.
void launch_init_pool(const PoolView *pv, int64_t begin, int64_t n, int inst, const double *cols, const double *pcs,
                      const ConstRow &row, int64_t ld, int64_t src, cudaStream_t s);
// A permutation of the runs of kOrderedRun slots in [0, n), the classes' (instances with
// begin and count set) interleaved by the fraction of the class that lies before them.
void launch_run_order(const InstDev *insts, int ninst, int64_t n, int32_t *order, cudaStream_t s);
void launch_connectivity(int nxb, int nyb, int nzb, int periodicity, int32_t *ncon, int32_t *con, cudaStream_t s);

// --- gp_state.cu: the state columns between the caller's order and the pool's ---
// state columns as bits (x y z u v w qa qb qc qd ox oy oz = bits 0..12); the copies take
// these five sets
constexpr unsigned kAllStateCols = (1u << kNState) - 1u;
constexpr unsigned kColsPosQuat = 0x3C7u;    // x y z qa qb qc qd: final once the integrate is done
constexpr unsigned kColsVelSpin = 0x1C38u;   // u v w ox oy oz: the response may still change them
constexpr unsigned kColsPos = 0x7u;          // x y z: all the gather reads
// (kAllStateCols & ~kColsPos is the fifth)
struct StateCols {
  double *p[kNState];   // device pointers; the entries outside the copy's set are not used
};
// alt: the pool's other buffer, of capacity cap, used as workspace (its contents are dead
// between two advances); count: the caller's entries per column; only >= 0: that class
// alone, at offset 0.
void launch_read_state(const InstDev *insts, const PoolView *pv, const PoolView *alt, int64_t cap, int64_t n,
                       int only, const StateCols &out, int64_t count, cudaStream_t s,
                       unsigned mask = kAllStateCols);
void launch_write_state(const InstDev *insts, const PoolView *pv, const PoolView *alt, int64_t cap, int64_t n,
                        const StateCols &in, int64_t count, cudaStream_t s, unsigned mask = kAllStateCols);
void launch_fluid_out(const InstDev *insts, const PoolView *pv, int64_t n, double *const *fluid, double *fout,
                      int64_t count, cudaStream_t s);

}  // namespace gp
