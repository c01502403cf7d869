// The wall-normal tridiagonal solve with each column split over the threads
// of a block (ssolve_trid, mod_poisson_solver.cc:317-357).
//
// The serial sweep is a chain of 2 nz dependent operations per system, and its
// forward values make a round trip through memory.  Here a block owns 16 lanes
// of systems and cuts their columns into 16 segments of ceil(nz / 16) planes,
// a half warp each, held in registers:
//   1. forward elimination of the segment from a zero incoming value, and the
//      product of its multipliers: (E, M), to shared memory;
//   2. the segment's true incoming value from the (E, M) of the segments
//      below it, and the elimination again from there, in place;
//   3. and 4. the same downwards for the back substitution.
// The elimination is a first-order linear recurrence with known multipliers,
// so step 2 continues exactly where the segment below ends, up to the
// rounding of the combined incoming value; the multipliers of the diagonally
// dominant systems are at most 1 in magnitude, so that rounding is not
// amplified.  The reciprocal of a zero last pivot is 0 in the table, which
// keeps the rule of the singular mode (last unknown = 0).
//
// A lane holds the two systems 2m, 2m+1 of a packed x pair (on large FP32
// grids also those of the packed y pair): they share the wavenumber, hence
// the pivots and every multiplier, which is what keeps the instruction count
// below the memory time.
//
// What bounds it: memory, where the segments are whole.  Every value is read once
// and written once, all loads of a thread are in flight at once, and several
// blocks per SM overlap their loads, sweeps and stores.  Segments that are not
// whole leave threads idle and pay the guarded code, so large planes of other
// columns stay with the serial sweeps (trid_split_pays).  Measured against the serial streaming sweep, per
// solve: FP64 768 x 384 x 256 0.42 -> 0.31 ms (a copy in the same access pattern
// takes 0.20), 256 x 192 x 128 28 -> 22 us, 128 x 64 x 64 10 -> 3 us; mixed 0.23 ->
// 0.17 ms, 52 -> 16 us, 22 -> 3 us.  Tried and slower at the large size: one
// system per lane (0.96 and 0.60 ms: instructions and spills), segments over
// the CTAs of a cluster with the (E, M) read through distributed shared memory
// (0.83 and 0.33 ms, 10 us at any size), one block of 512 threads per SM
// (0.34 and 0.17 ms: nothing overlaps its sweeps).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <type_traits>

#include "plc_device.cuh"
#include "plc_internal.h"

namespace plc {

namespace {

constexpr int kSeg = 16;    // segments of a column
constexpr int kLanes = 16;  // lanes of a block: 128- or 256-byte rows of a plane
constexpr int kThreads = kSeg * kLanes;

__device__ __forceinline__ double fma_a(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float fma_a(float a, float b, float c) { return fmaf(a, b, c); }

template <class T>
struct Pair;
template <>
struct Pair<double> {
  using V = double2;
};
template <>
struct Pair<float> {
  using V = float2;
};

// A lane's systems: `NS` rows of a packed x pair, first element at q, rows
// `row` elements apart; the pivot column rp; which of the pair's components
// and rows are the lane's own to store (the pairs (0, 1) of either direction
// hold two wavenumbers, each with a lane of its own).
template <class T, class A>
struct Lane {
  T *q;
  const A *rp;
  bool st_x[2], st_y[2];
};

// (E, M) of the segments, for both sweeps
template <class A, int NS>
struct Share {
  A v[2][kSeg][2 * NS + 1][kLanes];
};

// Barrier of the block, reached by each warp at one of two places of the program
// (solve_columns).  __syncthreads is defined where the whole block takes the
// same path; the barrier by its number counts warps wherever they arrive.
__device__ __forceinline__ void segment_barrier() {
  __syncwarp();
  asm volatile("barrier.cta.sync.aligned 0;" ::: "memory");
}

// The solve of one segment: n planes from k0 (FULL: n == CH; n <= 0: an
// empty segment, E = 0 and M = 1).
template <class T, class A, int NS, int CH, bool FULL>
__device__ __forceinline__ void solve_segment(const Lane<T, A> &L, long long plane, long long row,
                                              long long PS, const A *__restrict__ ca,
                                              const A *__restrict__ cc, int k0, int n,
                                              Share<A, NS> &sh) {
  using V = typename Pair<T>::V;
  constexpr int C = 2 * NS;
  const int lane = threadIdx.x % kLanes, seg = threadIdx.x / kLanes;
  A x[CH][C], r[CH], r_below = A(0);
  {
    const T *qs = L.q + k0 * plane;
    const A *rs = L.rp + k0 * PS;
#pragma unroll
    for (int s = 0; s < CH; ++s)
      if (FULL || s < n) {
#pragma unroll
        for (int y = 0; y < NS; ++y) {
          const V v = __ldcs(reinterpret_cast<const V *>(qs + y * row));
          x[s][2 * y] = A(v.x);
          x[s][2 * y + 1] = A(v.y);
        }
        r[s] = __ldg(rs);
        qs += plane;
        rs += PS;
      }
    if (k0 > 0 && (FULL || n > 0)) r_below = __ldg(L.rp + (k0 - 1) * PS);
  }
  // the negative multiplier of plane k0 + s (zero for the first: a[0] = 0)
  auto mul = [&](int s) -> A { return -(__ldg(ca + k0 + s) * (s ? r[s ? s - 1 : 0] : r_below)); };
  {
    A e[C], m = A(1);
#pragma unroll
    for (int c = 0; c < C; ++c) e[c] = A(0);
#pragma unroll
    for (int s = 0; s < CH; ++s)
      if (FULL || s < n) {
        const A t = mul(s);
#pragma unroll
        for (int c = 0; c < C; ++c) e[c] = fma_a(t, e[c], x[s][c]);
        m *= t;
      }
#pragma unroll
    for (int c = 0; c < C; ++c) sh.v[0][seg][c][lane] = e[c];
    sh.v[0][seg][C][lane] = m;
  }
  segment_barrier();
  {
    A e[C];
#pragma unroll
    for (int c = 0; c < C; ++c) e[c] = A(0);
    for (int s = 0; s < seg; ++s) {
      const A m = sh.v[0][s][C][lane];
#pragma unroll
      for (int c = 0; c < C; ++c) e[c] = fma_a(m, e[c], sh.v[0][s][c][lane]);
    }
#pragma unroll
    for (int s = 0; s < CH; ++s)
      if (FULL || s < n) {
        const A t = mul(s);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          e[c] = fma_a(t, e[c], x[s][c]);
          x[s][c] = e[c] * r[s];
        }
      }
  }
  // from here on x[s] holds the forward value times the pivot, r[s] the
  // negative multiplier of the back substitution, x(k) - (c(k) r(k)) x(k+1)
  {
    A e[C], m = A(1);
#pragma unroll
    for (int c = 0; c < C; ++c) e[c] = A(0);
#pragma unroll
    for (int s = CH - 1; s >= 0; --s)
      if (FULL || s < n) {
        r[s] *= -__ldg(cc + k0 + s);
#pragma unroll
        for (int c = 0; c < C; ++c) e[c] = fma_a(r[s], e[c], x[s][c]);
        m *= r[s];
      }
#pragma unroll
    for (int c = 0; c < C; ++c) sh.v[1][seg][c][lane] = e[c];
    sh.v[1][seg][C][lane] = m;
  }
  segment_barrier();
  {
    A e[C];
#pragma unroll
    for (int c = 0; c < C; ++c) e[c] = A(0);
    for (int s = kSeg - 1; s > seg; --s) {
      const A m = sh.v[1][s][C][lane];
#pragma unroll
      for (int c = 0; c < C; ++c) e[c] = fma_a(m, e[c], sh.v[1][s][c][lane]);
    }
    T *qs = L.q + (k0 + (FULL ? CH : n) - 1) * plane;
    const bool whole = L.st_x[0] && L.st_x[1];
#pragma unroll
    for (int s = CH - 1; s >= 0; --s)
      if (FULL || s < n) {
#pragma unroll
        for (int c = 0; c < C; ++c) e[c] = fma_a(r[s], e[c], x[s][c]);
#pragma unroll
        for (int y = 0; y < NS; ++y) {
          T *p = qs + y * row;
          if (L.st_y[y]) {
            if (whole) {
              V v;
              v.x = T(e[2 * y]);
              v.y = T(e[2 * y + 1]);
              *reinterpret_cast<V *>(p) = v;
            } else if (L.st_x[0]) {
              p[0] = T(e[2 * y]);
            } else {
              p[1] = T(e[2 * y + 1]);
            }
          }
        }
        qs -= plane;
      }
  }
}

// planes of a segment
__host__ __device__ __forceinline__ int split_planes(int nz) { return (nz + kSeg - 1) / kSeg; }

template <class T, class A, int NS, int CH>
__device__ __forceinline__ void solve_columns(const Lane<T, A> &L, int nz, long long plane,
                                              long long row, long long PS, const A *ca,
                                              const A *cc, void *smem) {
  const int np = split_planes(nz);
  const int k0 = (int)threadIdx.x / kLanes * np, n = min(np, nz - k0);
  Share<A, NS> &sh = *static_cast<Share<A, NS> *>(smem);
  // (the two segments of a warp take the same side: both hold the block's barriers)
  if (__all_sync(0xffffffffu, n == CH))
    solve_segment<T, A, NS, CH, true>(L, plane, row, PS, ca, cc, k0, n, sh);
  else
    solve_segment<T, A, NS, CH, false>(L, plane, row, PS, ca, cc, n > 0 ? k0 : 0, n, sh);
}

// packed index -> wavenumber
__device__ __forceinline__ int wave_of(int i, int n) {
  return i == 0 ? 0 : (i == 1 ? n >> 1 : i >> 1);
}
// wavenumber m of n: the first packed index of its pair, which components are its own
__device__ __forceinline__ int pair_of(int m, int n, bool (&own)[2]) {
  own[0] = m != n >> 1;
  own[1] = m != 0;
  return (m == 0 || m == n >> 1) ? 0 : 2 * m;
}

// resident blocks per SM that the registers of a segment length leave room for
constexpr int split_resident(int ch) { return ch <= 4 ? 4 : (ch <= 8 ? 3 : 2); }

// FP64: a lane per packed x pair and row
template <int CH>
__global__ void __launch_bounds__(kThreads, split_resident(CH))
    k_trid_split(int nx, int ny, int nz, const double *__restrict__ rpiv,
                 const double *__restrict__ a, const double *__restrict__ c,
                 double *__restrict__ var) {
  __shared__ Share<double, 1> sh;
  const int MX = (nx >> 1) + 1, lanes = MX * ny;
  const long long plane = (long long)nx * ny, PS = (long long)MX * ((ny >> 1) + 1);
  const int t0 = (int)(blockIdx.x * kLanes + threadIdx.x % kLanes), t = min(t0, lanes - 1);
  const int j = t / MX, mx = t - j * MX;
  Lane<double, double> L;
  L.q = var + (long long)j * nx + pair_of(mx, nx, L.st_x);
  L.rp = rpiv + (long long)wave_of(j, ny) * MX + mx;
  L.st_y[0] = t0 < lanes;
  solve_columns<double, double, 1, CH>(L, nz, plane, nx, PS, a, c, &sh);
}

// A mixed-form channel: the systems whose packed x and y indices are both
// below kLowModes (the lowest wavenumbers, with the largest amplification,
// and the pinned singular mode) are solved by blocks of their own in FP64
// with the FP64 pivots; all others in FP32, a lane per packed x pair and row
// or, NS = 2, per packed pair of both directions.
struct SplitMember {
  int nx, ny, nz, low_blocks, blocks;
  const float *rpiv32, *a32, *c32;
  const double *rpiv, *a, *c;
  float *var;
};

__host__ __device__ __forceinline__ int low_waves(int nx) {
  const int MX = (nx >> 1) + 1;
  return MX < kLowModes / 2 + 1 ? MX : kLowModes / 2 + 1;
}
__host__ __device__ __forceinline__ int low_rows(int ny) { return ny < kLowModes ? ny : kLowModes; }

// the solve of block b of a channel (its low-mode blocks come first)
template <int CH, int NS>
__device__ __forceinline__ void split_mixed(const SplitMember &M, int b, void *smem) {
  const int nx = M.nx, ny = M.ny, lane = (int)threadIdx.x % kLanes;
  const int MX = (nx >> 1) + 1, MY = (ny >> 1) + 1;
  const long long plane = (long long)nx * ny, PS = (long long)MX * MY;
  if (b < M.low_blocks) {
    const int W = low_waves(nx), lanes = W * low_rows(ny);
    const int t0 = b * kLanes + lane, t = min(t0, lanes - 1), j = t / W, q = t - j * W;
    const int mx = q < kLowModes / 2 ? q : nx >> 1;
    Lane<float, double> L;
    L.q = M.var + (long long)j * nx + pair_of(mx, nx, L.st_x);
    L.rp = M.rpiv + (long long)wave_of(j, ny) * MX + mx;
    L.st_y[0] = t0 < lanes;
    solve_columns<float, double, 1, CH>(L, M.nz, plane, nx, PS, M.a, M.c, smem);
  } else {
    const int lanes = MX * (NS == 2 ? MY : ny);
    const int t0 = (b - M.low_blocks) * kLanes + lane, t = min(t0, lanes - 1);
    const int row = t / MX, mx = t - row * MX;  // NS = 2: of wavenumber row; else of packed row
    const int my = NS == 2 ? row : wave_of(row, ny);
    Lane<float, float> L;
    const int i0 = pair_of(mx, nx, L.st_x);
    int j0 = row;
    if (NS == 2)
      j0 = pair_of(my, ny, L.st_y);
    else
      L.st_y[0] = true;
    const bool low = (mx < kLowModes / 2 || mx == nx >> 1) && (my < kLowModes / 2 || my == ny >> 1);
    if (low || t0 >= lanes) L.st_y[0] = L.st_y[1] = false;
    L.q = M.var + (long long)j0 * nx + i0;
    L.rp = M.rpiv32 + (long long)my * MX + mx;
    solve_columns<float, float, NS, CH>(L, M.nz, plane, nx, PS, M.a32, M.c32, smem);
  }
}

// (both kinds of block share the memory)
constexpr size_t kSplitShare =
    std::max(sizeof(Share<double, 1>), sizeof(Share<float, 2>));

template <int CH, int NS>
__global__ void __launch_bounds__(kThreads, split_resident(CH))
    k_trid_split_mixed(const __grid_constant__ SplitMember M) {
  __shared__ __align__(16) unsigned char sh[kSplitShare];
  split_mixed<CH, NS>(M, (int)blockIdx.x, sh);
}

// the mixed-form channels of an ensemble: block b works for channel m,
// start[m] <= b < start[m + 1], with that channel's own segments, so each
// channel's result is that of its own launch
struct SplitBatch {
  int n;
  int start[kBatchMax + 1];
  SplitMember m[kBatchMax];
};
static_assert(sizeof(SplitBatch) <= 32000, "kernel parameters are limited to 32764 bytes");

// compiled segment lengths
__host__ __device__ __forceinline__ int split_ch(int np) { return np <= 4 ? 4 : (np <= 8 ? 8 : 16); }
static_assert(kTridSplitMax == 16 * kSeg, "the longest compiled segment is 16 planes");

template <int CHMAX>
__global__ void __launch_bounds__(kThreads, split_resident(CHMAX))
    k_trid_split_mixed_batch(const __grid_constant__ SplitBatch b) {
  __shared__ __align__(16) unsigned char sh[kSplitShare];
  batch_grid_sync();
  const int q = batch_member(b.start, b.n, (int)blockIdx.x), lb = (int)blockIdx.x - b.start[q];
  const SplitMember &M = b.m[q];
  switch (split_ch(split_planes(M.nz))) {
    case 4: split_mixed<4, 1>(M, lb, sh); break;
    case 8: split_mixed<8, 1>(M, lb, sh); break;
    default:
      if constexpr (CHMAX > 8) split_mixed<16, 1>(M, lb, sh);
      break;
  }
}

// A lane per packed pair of both directions halves the instructions, but also
// the blocks: worth it once they still fill the device several times.
bool split_quads(const plc_ctx *c) {
  return (long long)(c->nx / 2 + 1) * (c->ny / 2 + 1) >= (long long)kLanes * 8 * c->device_sms;
}

SplitMember split_member(const plc_ctx *c, bool quads) {
  const int low = low_waves(c->nx) * low_rows(c->ny);
  const int main = (c->nx / 2 + 1) * (quads ? c->ny / 2 + 1 : c->ny);
  const int lb = (low + kLanes - 1) / kLanes;
  return SplitMember{c->nx,       c->ny,     c->nz,
                     lb,          lb + (main + kLanes - 1) / kLanes,
                     c->d_rpiv32, c->d_ac32, c->d_ac32 + c->nz, c->d_rpiv, c->d_ac,
                     c->d_ac + c->nz, c->f_field[PLC_SPEC]};
}

// f(CH) with the segment length as a compile-time constant
template <class F>
void split_dispatch(int nz, F &&f) {
  switch (split_ch(split_planes(nz))) {
    case 4: f(std::integral_constant<int, 4>{}); break;
    case 8: f(std::integral_constant<int, 8>{}); break;
    default: f(std::integral_constant<int, 16>{}); break;
  }
}

}  // namespace

cudaError_t launch_trid_split(const plc_ctx *c, double *var, cudaStream_t s) {
  split_dispatch(c->nz, [&](auto CH) {
    const int lanes = (c->nx / 2 + 1) * c->ny;
    k_trid_split<decltype(CH)::value><<<(lanes + kLanes - 1) / kLanes, kThreads, 0, s>>>(
        c->nx, c->ny, c->nz, c->d_rpiv, c->d_ac, c->d_ac + c->nz, var);
  });
  return cudaGetLastError();
}

cudaError_t launch_trid_split(const plc_ctx *c, float *var, cudaStream_t s) {
  const bool quads = split_quads(c);
  SplitMember M = split_member(c, quads);
  M.var = var;
  split_dispatch(c->nz, [&](auto CH) {
    constexpr int ch = decltype(CH)::value;
    if (quads)
      k_trid_split_mixed<ch, 2><<<M.blocks, kThreads, 0, s>>>(M);
    else
      k_trid_split_mixed<ch, 1><<<M.blocks, kThreads, 0, s>>>(M);
  });
  return cudaGetLastError();
}

cudaError_t launch_trid_split_batch(plc_ctx *const *cs, int n, cudaStream_t s, bool pdl) {
  for (int q0 = 0; q0 < n; q0 += kBatchMax) {
    SplitBatch b;
    std::memset(&b, 0, sizeof b);
    b.n = std::min(kBatchMax, n - q0);
    int tot = 0, nzmax = 0;
    for (int q = 0; q < b.n; ++q) {
      b.m[q] = split_member(cs[q0 + q], false);
      b.start[q] = tot;
      tot += b.m[q].blocks;
      nzmax = std::max(nzmax, cs[q0 + q]->nz);
    }
    b.start[b.n] = tot;
    // segments of at most 8 planes need half the registers
    const dim3 block(kThreads);
    const cudaError_t e =
        split_planes(nzmax) <= 8
            ? launch_batched(k_trid_split_mixed_batch<8>, (unsigned)tot, block, 0, s, b, pdl)
            : launch_batched(k_trid_split_mixed_batch<16>, (unsigned)tot, block, 0, s, b, pdl);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace plc
