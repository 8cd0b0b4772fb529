// gp_state.cu -- the state columns between the caller's order and the pool's.
//
// The pool holds the particles in cell order, the caller holds them by class and index,
// and the two orders have nothing to do with each other, so one side of every copy is a
// random access.  Taken column by column (13 scattered 8-byte words a particle) each word
// costs a 32-byte sector of L2 or a burst of DRAM; that is the shortest way while the
// columns fit the L2.  Beyond it the copy goes through rows: a particle's columns side by
// side in one aligned row of up to 128 bytes, so that the random access moves whole lines,
// and the conversion between rows and columns on the other side is a streamed transpose in
// shared memory.  The rows live in the pool's other buffer, whose contents are dead
// between two advances, so they cost no memory.
#include "gp_launch.h"
#include "gp_types.h"

namespace gp {
namespace {

constexpr int kTile = 256;   // particles (and threads) a block

__host__ __device__ constexpr int bits(unsigned m) { return m ? (int)(m & 1u) + bits(m >> 1) : 0; }
__host__ __device__ constexpr int nth_bit(unsigned m, int k) {
  int b = 0;
  for (;; ++b) {
    if ((m >> b) & 1u) {
      if (k == 0) return b;
      --k;
    }
  }
}

template <unsigned kMask>
struct Rows {
  static constexpr int kCols = bits(kMask);
  static constexpr int kPitch = kCols <= 4 ? 4 : (kCols <= 8 ? 8 : 16);   // doubles a row
  static constexpr int kPad = kCols | 1;   // doubles a particle in shared memory: odd, so
                                           // that a column is read without bank conflicts
  static constexpr int kParts = kPitch / 2;                               // 16-byte parts a row
};

// Row g of the rows kept in the 23 columns of buffer `alt`, `per` rows to a column.
template <int kPitch>
__device__ __forceinline__ double *row_ptr(double *const *cols, uint32_t per, int64_t g) {
  const uint32_t c = (uint32_t)g / per;
  return cols[c] + (size_t)((uint32_t)g - c * per) * kPitch;
}

// The pool buffer's columns, state first, as the rows' storage.
__device__ __forceinline__ void row_columns(const PoolView *alt, double **cols) {
  if (threadIdx.x < kNState) cols[threadIdx.x] = alt->st[threadIdx.x];
  else if (threadIdx.x < kNState + kNConst) cols[threadIdx.x] = alt->pc[threadIdx.x - kNState];
  __syncthreads();
}

__device__ __forceinline__ int64_t caller_index(const InstDev *__restrict__ insts, const PoolView &P, int64_t i,
                                                int only, int64_t count) {
  const int inst = P.inst[i];
  if (inst < 0 || (only >= 0 && inst != only)) return -1;
  const int64_t g = (only >= 0 ? 0 : insts[inst].begin) + P.id[i];
  return (g < 0 || g >= count) ? -1 : g;
}

// rows <- the tile's columns in s, or s <- rows; row of particle t is rows index at(t) (< 0:
// none).  kParts neighbouring lanes move one row.
template <unsigned kMask, bool kStore, class At>
__device__ __forceinline__ void move_rows(double *s, double *const *cols, uint32_t per, int here, At at) {
  using R = Rows<kMask>;
  for (int e = threadIdx.x; e < here * R::kParts; e += kTile) {
    const int t = e / R::kParts, p = e % R::kParts;
    const int64_t g = at(t);
    if (g < 0) continue;
    double2 *row = reinterpret_cast<double2 *>(row_ptr<R::kPitch>(cols, per, g)) + p;
    double *v = s + t * R::kPad + 2 * p;
    if (kStore) {
      *row = make_double2(2 * p < R::kCols ? v[0] : 0.0, 2 * p + 1 < R::kCols ? v[1] : 0.0);
    } else if (2 * p < R::kCols) {
      const double2 d = *row;
      v[0] = d.x;
      if (2 * p + 1 < R::kCols) v[1] = d.y;
    }
  }
}

// caller's columns -> rows (kIn), rows -> caller's columns
template <unsigned kMask, bool kIn>
__global__ void __launch_bounds__(kTile) k_rows_caller(StateCols io, const PoolView *__restrict__ alt, uint32_t per,
                                                       int64_t count) {
  using R = Rows<kMask>;
  __shared__ double s[kTile * R::kPad];
  __shared__ double *cols[kNState + kNConst];
  row_columns(alt, cols);
  for (int64_t g0 = (int64_t)blockIdx.x * kTile; g0 < count; g0 += (int64_t)gridDim.x * kTile) {
    const int here = (int)min((int64_t)kTile, count - g0), t = threadIdx.x;
    auto at = [&](int k) { return g0 + k; };
    if (kIn) {
      if (t < here) {
#pragma unroll
        for (int k = 0; k < R::kCols; ++k) s[t * R::kPad + k] = io.p[nth_bit(kMask, k)][g0 + t];
      }
      __syncthreads();
      move_rows<kMask, true>(s, cols, per, here, at);
    } else {
      move_rows<kMask, false>(s, cols, per, here, at);
      __syncthreads();
      if (t < here) {
#pragma unroll
        for (int k = 0; k < R::kCols; ++k) io.p[nth_bit(kMask, k)][g0 + t] = s[t * R::kPad + k];
      }
    }
    __syncthreads();
  }
}

// rows -> pool (kIn), pool -> rows
template <unsigned kMask, bool kIn>
__global__ void __launch_bounds__(kTile) k_rows_pool(const InstDev *__restrict__ insts,
                                                     const PoolView *__restrict__ pv,
                                                     const PoolView *__restrict__ alt, uint32_t per, int64_t n,
                                                     int only, int64_t count) {
  using R = Rows<kMask>;
  __shared__ double s[kTile * R::kPad];
  __shared__ int32_t row_of[kTile];
  __shared__ double *cols[kNState + kNConst];
  row_columns(alt, cols);
  for (int64_t i0 = (int64_t)blockIdx.x * kTile; i0 < n; i0 += (int64_t)gridDim.x * kTile) {
    const int here = (int)min((int64_t)kTile, n - i0), t = threadIdx.x;
    const int64_t g = t < here ? caller_index(insts, *pv, i0 + t, only, count) : -1;
    row_of[t] = (int32_t)g;
    auto at = [&](int k) { return (int64_t)row_of[k]; };
    if (!kIn && g >= 0) {
#pragma unroll
      for (int k = 0; k < R::kCols; ++k) s[t * R::kPad + k] = pv->st[nth_bit(kMask, k)][i0 + t];
    }
    __syncthreads();
    move_rows<kMask, !kIn>(s, cols, per, here, at);
    __syncthreads();
    if (kIn && g >= 0) {
#pragma unroll
      for (int k = 0; k < R::kCols; ++k) pv->st[nth_bit(kMask, k)][i0 + t] = s[t * R::kPad + k];
    }
    __syncthreads();
  }
}

// Column by column, without rows.
template <unsigned kMask, bool kIn>
__global__ void __launch_bounds__(kTile) k_direct(const InstDev *__restrict__ insts, const PoolView *__restrict__ pv,
                                                  int64_t n, int only, StateCols io, int64_t count) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t g = caller_index(insts, *pv, i, only, count);
    if (g < 0) continue;
#pragma unroll
    for (int k = 0; k < kNState; ++k) {
      if (!((kMask >> k) & 1u)) continue;
      if (kIn) pv->st[k][i] = io.p[k][g];
      else io.p[k][g] = pv->st[k][i];
    }
  }
}

// The interpolated field at the particles into the caller's order (fout: 6 columns of count).
__global__ void k_fluid_out(const InstDev *__restrict__ insts, const PoolView *__restrict__ pv, int64_t n,
                            double *const *__restrict__ fluid, double *__restrict__ fout, int64_t count) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t g = caller_index(insts, *pv, i, -1, count);
    if (g < 0) continue;
#pragma unroll
    for (int c = 0; c < kNFluid; ++c) fout[c * count + g] = fluid[c][i];
  }
}

int grid_of(int64_t n) { return (int)min((n + kTile - 1) / kTile, (int64_t)148 * 8); }

// From this many particles on the copy goes through rows.  All 13 columns, us a call with
// its launch and wait (B200), column by column / through rows:
//                   600,000    800,000      1 M       1.6 M      1.8 M       2 M       16.8 M
//   into the pool    59 / 98    81 / 130  108 / 157  216 / 232  261 / 254  327 / 279  5183 / 2128
//   out of it        84 / 100  155 / 131  258 / 159  633 / 234  752 / 252  863 / 277  9828 / 2060
// (13 staging copies and a column-by-column kernel before: 5780 and 10419 at 16.8 M, 82
// and 74 at 10,000 where it now takes 28 and 23.)  Scattered writes leave the L2's reach
// first.
constexpr int64_t kRowsFromIn = 1600000, kRowsFromOut = 800000;

template <unsigned kMask, bool kIn>
void move_state(const InstDev *insts, const PoolView *pv, const PoolView *alt, int64_t cap, int64_t n, int only,
                StateCols io, int64_t count, cudaStream_t s) {
  const int64_t per = cap / Rows<kMask>::kPitch;   // rows a column of the other buffer holds
  if (count < (kIn ? kRowsFromIn : kRowsFromOut) || per * (kNState + kNConst) < count) {
    k_direct<kMask, kIn><<<grid_of(n), kTile, 0, s>>>(insts, pv, n, only, io, count);
  } else if (kIn) {
    k_rows_caller<kMask, true><<<grid_of(count), kTile, 0, s>>>(io, alt, (uint32_t)per, count);
    k_rows_pool<kMask, true><<<grid_of(n), kTile, 0, s>>>(insts, pv, alt, (uint32_t)per, n, only, count);
  } else {
    k_rows_pool<kMask, false><<<grid_of(n), kTile, 0, s>>>(insts, pv, alt, (uint32_t)per, n, only, count);
    k_rows_caller<kMask, false><<<grid_of(count), kTile, 0, s>>>(io, alt, (uint32_t)per, count);
  }
}

template <bool kIn>
void move_masked(const InstDev *insts, const PoolView *pv, const PoolView *alt, int64_t cap, int64_t n, int only,
                 StateCols io, int64_t count, unsigned mask, cudaStream_t s) {
  if (n <= 0) return;
  switch (mask) {
    case kColsPos: return move_state<kColsPos, kIn>(insts, pv, alt, cap, n, only, io, count, s);
    case kAllStateCols & ~kColsPos:
      return move_state<kAllStateCols & ~kColsPos, kIn>(insts, pv, alt, cap, n, only, io, count, s);
    case kColsPosQuat: return move_state<kColsPosQuat, kIn>(insts, pv, alt, cap, n, only, io, count, s);
    case kColsVelSpin: return move_state<kColsVelSpin, kIn>(insts, pv, alt, cap, n, only, io, count, s);
    default: return move_state<kAllStateCols, kIn>(insts, pv, alt, cap, n, only, io, count, s);
  }
}

}  // namespace

void launch_read_state(const InstDev *insts, const PoolView *pv, const PoolView *alt, int64_t cap, int64_t n,
                       int only, const StateCols &out, int64_t count, cudaStream_t s, unsigned mask) {
  move_masked<false>(insts, pv, alt, cap, n, only, out, count, mask, s);
}

void launch_write_state(const InstDev *insts, const PoolView *pv, const PoolView *alt, int64_t cap, int64_t n,
                        const StateCols &in, int64_t count, cudaStream_t s, unsigned mask) {
  move_masked<true>(insts, pv, alt, cap, n, -1, in, count, mask, s);
}

void launch_fluid_out(const InstDev *insts, const PoolView *pv, int64_t n, double *const *fluid, double *fout,
                      int64_t count, cudaStream_t s) {
  if (n > 0) k_fluid_out<<<grid_of(n), kTile, 0, s>>>(insts, pv, n, fluid, fout, count);
}

}  // namespace gp
