// Tensor-core kernels of the learned initialiser's generator (plc_gen.cu):
// BF16 channels-last 3-D convolutions as implicit GEMMs on tcgen05 with FP32
// accumulators in tensor memory, periodic in x and y and zero-padded in z
// (the walls) -- the forward pass, the input gradient (the same kernel) and
// the weight gradient.
//
// Tensors are [b][z][y][x][c] with c fastest.  A 3x3x3 convolution is
//   Y[m][co] = sum_{tap, ci} W[tap][co][ci] * X[m + off(tap)][ci],
// tap = (dz+1)*9 + (dy+1)*3 + (dx+1), off(tap) = (dz, dy, dx); the adjoint
// (gradient with respect to X) is the same convolution of dY with the
// weights W'[tap][ci][co] = W[26 - tap][co][ci].
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "plc_device.cuh"

namespace plc {
namespace gen {

using bf16 = __nv_bfloat16;

__device__ __forceinline__ float lrelu(float h) { return h > 0.f ? h : 0.2f * h; }

struct Shape {
  int B, Z, Y, X;  // batch and spatial extents
  __host__ __device__ long long voxels() const { return (long long)B * Z * Y * X; }
};

// voxel m -> (b, z, y, x); 32-bit arithmetic (plc_gen_create keeps every
// tensor below 2^31 voxels), a 64-bit division being a long software routine
__device__ __forceinline__ void unflatten(const Shape &s, long long m, int &b, int &z, int &y,
                                          int &x) {
  const unsigned um = (unsigned)m, X = (unsigned)s.X, Y = (unsigned)s.Y, Z = (unsigned)s.Z;
  unsigned r = um / X;
  x = (int)(um - r * X);
  const unsigned r2 = r / Y;
  y = (int)(r - r2 * Y);
  const unsigned r3 = r2 / Z;
  z = (int)(r2 - r3 * Z);
  b = (int)r3;
}
// the voxel at offset (dz, dy, dx) from (b, z, y, x): periodic in x, y; -1
// outside the walls in z
__device__ __forceinline__ long long shifted(const Shape &s, int b, int z, int y, int x, int dz,
                                             int dy, int dx) {
  const int zz = z + dz;
  if (zz < 0 || zz >= s.Z) return -1;
  int yy = y + dy, xx = x + dx;
  yy = yy < 0 ? yy + s.Y : (yy >= s.Y ? yy - s.Y : yy);
  xx = xx < 0 ? xx + s.X : (xx >= s.X ? xx - s.X : xx);
  return (((long long)b * s.Z + zz) * s.Y + yy) * s.X + xx;
}

// ===========================================================================
// The convolution on the 5th-generation tensor cores (tcgen05): a
// block of 128 threads owns 128 voxels x N output channels (N = Co <= 128),
// with the FP32 accumulator tile in tensor memory (TMEM).  K = 27 taps x Ci
// in steps of 16 channels; kTcG steps form a stage: the im2col rows of A and
// the weight rows of B in the K-major core-matrix layout of the UMMA
// descriptors without swizzle (8 rows x 16 bytes per core matrix, the two
// 8-channel halves of a step 128 bytes apart, 8-row groups 256 bytes apart).
// Stages rotate through kTcNB buffers filled by cp.async (zero fill for the
// walls) two stages ahead: thread 0 issues a stage's tcgen05.mma and commits
// them to that buffer's mbarrier, which the threads wait on before refilling
// the buffer.  The epilogue reads the accumulators with tcgen05.ld (warp w
// owns TMEM lanes 32w..32w+31, i.e. voxels) and stores FP32 rows.  Every wait
// is bounded; on a timeout the block flags *err, skips its stores and still
// releases its TMEM.
// ===========================================================================
constexpr int kTcM = 128;
constexpr int kTcG = 2;                        // 16-channel K steps per buffer
constexpr int kTcNB = 3;                       // buffers: copies run two stages ahead of the MMAs
constexpr int kTcABytes = kTcM * 16 * 2;       // 4 KB per step
constexpr long long kTcWaitLimit = 1ll << 24;  // mbarrier polls before giving up

__device__ __forceinline__ unsigned tc_smem_u32(const void *p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
// UMMA shared-memory descriptor, K-major, no swizzle: start address, leading
// byte offset (between the two K halves), stride byte offset (between 8-row
// groups), version 1
__device__ __forceinline__ unsigned long long tc_desc(unsigned saddr) {
  return (unsigned long long)((saddr >> 4) & 0x3FFF) | ((unsigned long long)(128 >> 4) << 16) |
         ((unsigned long long)(256 >> 4) << 32) | (1ull << 46);
}
// instruction descriptor: F32 accumulator, BF16 A and B, both K-major, M = 128
__host__ __device__ constexpr unsigned tc_idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(n >> 3) << 17) | ((unsigned)(kTcM >> 4) << 24);
}
__device__ __forceinline__ bool tc_wait(unsigned long long *bar, unsigned parity) {
  const unsigned a = tc_smem_u32(bar);
  for (long long it = 0; it < kTcWaitLimit; ++it) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// Tensor memory: the instructions are .sync.aligned, so that the lanes of a warp,
// which may have parted at a predicate before, meet first.
// cols columns, their address to *base (by one warp, which also gives them back)
__device__ __forceinline__ void tc_alloc(unsigned *base, unsigned cols) {
  __syncwarp();
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   tc_smem_u32(base)),
               "r"(cols));
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
}
__device__ __forceinline__ void tc_dealloc(unsigned base, unsigned cols) {
  __syncwarp();
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols));
}
// 16 columns from addr of the warp's 32 lanes (with the wait in one statement: no use
// of the registers can be moved between the two)
__device__ __forceinline__ void tc_ld16(unsigned addr, unsigned (&r)[16]) {
  __syncwarp();
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
      "%14,%15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(addr)
      : "memory");
}

// 16-byte asynchronous copy global -> shared; src_bytes 0 fills zeros
__device__ __forceinline__ void tc_cp16(void *dst, const void *src, unsigned src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(tc_smem_u32(dst)), "l"(src),
               "r"(src_bytes)
               : "memory");
}

__device__ __forceinline__ void tc_cp16s(unsigned dst, const void *src, unsigned src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes)
               : "memory");
}

// A/B core-matrix layout offset (bytes) of row r, channel half h of one step
__device__ __forceinline__ int tc_off(int r, int h) { return (r >> 3) * 256 + h * 128 + (r & 7) * 16; }

template <int N>
__global__ void __launch_bounds__(128) k_conv3d_tc(Shape s, const bf16 *__restrict__ X,
                                                   const bf16 *__restrict__ W, float *__restrict__ Y,
                                                   int Ci, int *err) {
  constexpr int kNCols = N <= 32 ? 32 : (N <= 64 ? 64 : 128);  // TMEM columns (power of 2)
  constexpr int kBBytes = N * 16 * 2;
  constexpr int kBuf = kTcG * (kTcABytes + kBBytes);
  extern __shared__ __align__(1024) unsigned char tc_smem[];
  __shared__ __align__(8) unsigned long long bar[kTcNB];
  __shared__ unsigned tmem_base_s;
  __shared__ int fail_s;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const long long M = s.voxels();
  const long long m0 = (long long)blockIdx.x * kTcM;
  unsigned char *buf0 = reinterpret_cast<unsigned char *>(
      (reinterpret_cast<unsigned long long>(tc_smem) + 1023ull) & ~1023ull);

  if (warp == 0) {
    tc_alloc(&tmem_base_s, kNCols);
  }
  if (t == 0) {
    for (int q = 0; q < kTcNB; ++q)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem_u32(&bar[q])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fail_s = 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = tmem_base_s;

  // this thread's A row: voxel m0 + t
  const long long am = m0 + t;
  int ab = 0, az = 0, ay = 0, ax = 0;
  if (am < M) unflatten(s, am, ab, az, ay, ax);
  const int CC = Ci / 16;  // K steps per tap
  const int KT = 27 * CC;
  const int nstage = (KT + kTcG - 1) / kTcG;
  // copies of stage st into buffer st % kTcNB (one commit group per stage)
  auto load_stage = [&](int st) {
    unsigned char *A = buf0 + (st % kTcNB) * kBuf;
    unsigned char *Bm = A + kTcG * kTcABytes;
#pragma unroll
    for (int g = 0; g < kTcG; ++g) {
      const int kk = st * kTcG + g;
      if (kk >= KT) break;
      unsigned char *Ag = A + g * kTcABytes;
      unsigned char *Bg = Bm + g * kBBytes;
      const int tap = kk / CC, c0 = (kk - tap * CC) * 16;
      const int dz = tap / 9 - 1, dy = (tap / 3) % 3 - 1, dx = tap % 3 - 1;
      const long long src = am < M ? shifted(s, ab, az, ay, ax, dz, dy, dx) : -1;
      const bf16 *xs = src >= 0 ? X + src * Ci + c0 : X;
      tc_cp16(Ag + tc_off(t, 0), xs, src >= 0 ? 16u : 0u);
      tc_cp16(Ag + tc_off(t, 1), src >= 0 ? xs + 8 : X, src >= 0 ? 16u : 0u);
      for (int e = t; e < 2 * N; e += 128) {
        const int n = e >> 1, h = e & 1;
        tc_cp16(Bg + tc_off(n, h), W + ((long long)tap * N + n) * Ci + c0 + h * 8, 16u);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  load_stage(0);
  if (nstage > 1) load_stage(1);
  bool ok = true;
  for (int st = 0; st < nstage; ++st) {
    const int b = st % kTcNB;
    unsigned char *A = buf0 + b * kBuf;
    unsigned char *Bm = A + kTcG * kTcABytes;
    if (st + 1 < nstage)
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    else
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    // the copies become visible to the tensor core's async proxy
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (t == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int g = 0; g < kTcG; ++g) {
        const int kk = st * kTcG + g;
        if (kk >= KT) break;
        const unsigned long long da = tc_desc(tc_smem_u32(A + g * kTcABytes));
        const unsigned long long db = tc_desc(tc_smem_u32(Bm + g * kBBytes));
        const unsigned acc = kk > 0 ? 1u : 0u;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
            :
            : "r"(tmem), "l"(da), "l"(db), "r"(tc_idesc(N)), "r"(acc), "r"(0u), "r"(0u), "r"(0u),
              "r"(0u));
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       tc_smem_u32(&bar[b]))
                   : "memory");
    }
    if (st + 2 < nstage) {
      // buffer (st + 2) % kTcNB was read by the MMAs of stage st - 1
      if (st >= 1) {
        if (t == 0 && !tc_wait(&bar[(st - 1) % kTcNB], (unsigned)(((st - 1) / kTcNB) & 1)))
          fail_s = 1;
        __syncthreads();
        if (fail_s) {
          ok = false;
          break;
        }
      }
      load_stage(st + 2);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  // all MMAs complete: the last commit covers every earlier tcgen05 operation
  if (ok) {
    const int last = nstage - 1;
    if (t == 0 && !tc_wait(&bar[last % kTcNB], (unsigned)((last / kTcNB) & 1))) fail_s = 1;
    __syncthreads();
    ok = !fail_s;
  }
  if (ok) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const long long row = m0 + warp * 32 + lane;
#pragma unroll
    for (int c0 = 0; c0 < N; c0 += 16) {
      unsigned r[16];
      const unsigned addr = tmem + ((unsigned)(warp * 32) << 16) + (unsigned)c0;
      tc_ld16(addr, r);
      if (row < M) {
        float4 *dst = reinterpret_cast<float4 *>(Y + row * N + c0);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          dst[q] = make_float4(__uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]),
                               __uint_as_float(r[4 * q + 2]), __uint_as_float(r[4 * q + 3]));
      }
    }
  } else if (t == 0) {
    atomicExch(err, 1);
    // let the MMAs still in flight finish (bounded) before the TMEM goes back
    for (int q = 0; q < kTcNB; ++q) tc_wait(&bar[q], 0);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    tc_dealloc(tmem, kNCols);
  }
}

template <int N, int G = kTcG, int NB = kTcNB>
constexpr size_t tc_smem_bytes() {
  return NB * (size_t)G * (kTcABytes + N * 16 * 2) + 1024;
}


// ---------------------------------------------------------------------------
// Weight gradient on tcgen05: D[co][ci] (+)= sum_m dY[m][co] X[m + off(tap)][ci]
// for one tap over a range of voxels (split K), M = 128 (co, zero-padded
// above Co), N = Ci <= 128, K = 16 voxels per MMA.  Both operands are staged
// MN-major (channels contiguous, as they lie in memory): element (mn, k) of
// a step at (mn/8)*256 + (k/8)*128 + (k%8)*16 + (mn%8)*2 bytes, i.e. stride
// byte offset 256 between 8-channel groups and leading byte offset 128
// between the two 8-voxel halves.  The block's tile is added to dW with
// FP32 atomics.
// ---------------------------------------------------------------------------
__host__ __device__ constexpr unsigned tc_idesc_mn(int n) {
  return tc_idesc(n) | (1u << 15) | (1u << 16);  // A and B MN-major
}
// byte offset of channel mn, voxel k of one MN-major step
__device__ __forceinline__ int tc_off_mn(int mn, int k) {
  return (mn >> 3) * 256 + (k >> 3) * 128 + (k & 7) * 16;
}

constexpr int kWgG = 2;   // K steps (16 voxels each) per buffer of the weight gradient
constexpr int kWgNB = 3;  // buffers: the copies run two stages ahead of the MMAs

template <int N>
__global__ void __launch_bounds__(128) k_conv3d_wgrad_tc(Shape s, const bf16 *__restrict__ dY,
                                                         const bf16 *__restrict__ X,
                                                         float *__restrict__ dW, int Co,
                                                         long long chunk, int *err) {
  constexpr int kNCols = N <= 32 ? 32 : (N <= 64 ? 64 : 128);
  constexpr int kBBytes = N * 16 * 2;
  constexpr int kBuf = kWgG * (kTcABytes + kBBytes);
  extern __shared__ __align__(1024) unsigned char tc_smem[];
  __shared__ __align__(8) unsigned long long bar[kWgNB];
  __shared__ unsigned tmem_base_s;
  __shared__ int fail_s;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int tap = blockIdx.z;
  const int dz = tap / 9 - 1, dy = (tap / 3) % 3 - 1, dx = tap % 3 - 1;
  const long long M = s.voxels();
  const long long k0 = (long long)blockIdx.x * chunk;
  const long long k1 = k0 + chunk < M ? k0 + chunk : M;
  unsigned char *buf0 = reinterpret_cast<unsigned char *>(
      (reinterpret_cast<unsigned long long>(tc_smem) + 1023ull) & ~1023ull);

  if (warp == 0) {
    tc_alloc(&tmem_base_s, kNCols);
  }
  if (t == 0) {
    for (int q = 0; q < kWgNB; ++q)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem_u32(&bar[q])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fail_s = 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = tmem_base_s;

  const long long nsteps = (k1 - k0 + 15) / 16;
  const int nstage = (int)((nsteps + kWgG - 1) / kWgG);
  const int ca = Co / 8, cb = N / 8;  // 16-byte channel chunks of a voxel row
  // the copies of stage st into buffer st % kWgNB (one commit group per stage)
  auto load_stage = [&](int st) {
    unsigned char *A = buf0 + (st % kWgNB) * kBuf;
    unsigned char *Bm = A + kWgG * kTcABytes;
#pragma unroll
    for (int g = 0; g < kWgG; ++g) {
      const long long step = (long long)st * kWgG + g;
      unsigned char *Ag = A + g * kTcABytes;
      unsigned char *Bg = Bm + g * kBBytes;
      const long long mb = k0 + step * 16;
      for (int e = t; e < 16 * 16; e += 128) {  // A: 16 voxels x 128 co
        const int k = e >> 4, q = e & 15;
        const long long m = mb + k;
        const bool v = step < nsteps && q < ca && m < k1;
        tc_cp16(Ag + tc_off_mn(q * 8, k), v ? (const void *)(dY + m * Co + q * 8) : (const void *)dY,
                v ? 16u : 0u);
      }
      for (int e = t; e < 16 * cb; e += 128) {  // B: 16 voxels x N ci of the shifted input
        const int k = e / cb, q = e - k * cb;
        const long long m = mb + k;
        long long src = -1;
        if (step < nsteps && m < k1) {
          int bb, z, y, x;
          unflatten(s, m, bb, z, y, x);
          src = shifted(s, bb, z, y, x, dz, dy, dx);
        }
        tc_cp16(Bg + tc_off_mn(q * 8, k), src >= 0 ? (const void *)(X + src * N + q * 8) : (const void *)X,
                src >= 0 ? 16u : 0u);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  load_stage(0);
  if (nstage > 1) load_stage(1);
  bool ok = true;
  for (int st = 0; st < nstage; ++st) {
    const int b = st % kWgNB;
    unsigned char *A = buf0 + b * kBuf;
    unsigned char *Bm = A + kWgG * kTcABytes;
    // stage st's copies landed (stage st + 1 may still be in flight)
    if (st + 1 < nstage)
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    else
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (t == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int g = 0; g < kWgG; ++g) {
        const long long step = (long long)st * kWgG + g;
        if (step >= nsteps) break;
        const unsigned long long da = tc_desc(tc_smem_u32(A + g * kTcABytes));
        const unsigned long long db = tc_desc(tc_smem_u32(Bm + g * kBBytes));
        const unsigned acc = step > 0 ? 1u : 0u;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
            :
            : "r"(tmem), "l"(da), "l"(db), "r"(tc_idesc_mn(N)), "r"(acc), "r"(0u), "r"(0u),
              "r"(0u), "r"(0u));
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       tc_smem_u32(&bar[b]))
                   : "memory");
    }
    if (st + 2 < nstage) {
      // buffer (st + 2) % kWgNB was read by the MMAs of stage st - 1
      if (st >= 1) {
        if (t == 0 && !tc_wait(&bar[(st - 1) % kWgNB], (unsigned)(((st - 1) / kWgNB) & 1)))
          fail_s = 1;
        __syncthreads();
        if (fail_s) {
          ok = false;
          break;
        }
      }
      load_stage(st + 2);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (ok && nstage > 0) {
    const int last = nstage - 1;
    if (t == 0 && !tc_wait(&bar[last % kWgNB], (unsigned)((last / kWgNB) & 1))) fail_s = 1;
    __syncthreads();
    ok = !fail_s;
  }
  if (ok && nstage > 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int co = warp * 32 + lane;
#pragma unroll
    for (int c0 = 0; c0 < N; c0 += 16) {
      unsigned r[16];
      const unsigned addr = tmem + ((unsigned)(warp * 32) << 16) + (unsigned)c0;
      tc_ld16(addr, r);
      if (co < Co) {
        float *dst = dW + ((long long)tap * Co + co) * N + c0;
#pragma unroll
        for (int q = 0; q < 16; ++q) atomicAdd(dst + q, __uint_as_float(r[q]));
      }
    }
  } else if (!ok && t == 0) {
    atomicExch(err, 1);
    for (int q = 0; q < kWgNB; ++q) tc_wait(&bar[q], 0);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    tc_dealloc(tmem, kNCols);
  }
}

// ===========================================================================
// Convolution and weight gradient over halo tiles.
//
// The kernels above copy the im2col rows of every tap, 27 reads of each input
// value from L2, which is what bounded them (64 -> 32 channels on 4 x 64 x 48 x 64
// voxels: 0.91 ms forward, 2.07 ms weight gradient; here 0.34 and 0.49).  Here a plane (b, z) is
// numbered by padded positions p = y * (X + 2) + x + 1: the neighbour at (dz,
// dy, dx) of the output at p is the input at p + dy * (X + 2) + dx of plane
// z + dz, for every p whose x is not one of the two padding columns.  A tile of
// consecutive positions therefore needs one run of consecutive rows of three
// planes, and with the rows of a group of 8 channels 16 bytes apart in shared
// memory a tap is only another start address of the UMMA operand.  Outputs at
// padding positions are computed and dropped (2 of X + 2).
// ===========================================================================

// divisions by the extents that the copies' index arithmetic needs
struct HaloDiv {
  FastDiv XP, X, YX;
  explicit HaloDiv(const Shape &s) : XP(s.X + 2), X(s.X), YX(s.Y * s.X) {}
};

// Row q of a halo tile whose first output position is p0: its voxel within the
// plane, periodic in y and x (rows that only padding outputs read map to some
// voxel of the plane).
__device__ __forceinline__ int halo_voxel(const Shape &s, const HaloDiv &d, int p0, int q) {
  const int XP = s.X + 2;
  const int pos = p0 - (XP + 1) + q + 2 * XP;  // not negative; two rows up
  const int row = d.XP.div(pos);
  int x = pos - row * XP - 1, y = row - 2;
  while (y < 0) y += s.Y;
  while (y >= s.Y) y -= s.Y;
  x = x < 0 ? s.X - 1 : (x >= s.X ? 0 : x);
  return y * s.X + x;
}

// Low word of a UMMA shared-memory descriptor without swizzle: start address and
// leading byte offset (K-major: between the K halves; MN-major: between the
// 8-voxel groups of K), both in units of 16 bytes; the start address of
// shared memory never carries out of its 14 bits, so that a neighbouring operand
// is one 32-bit addition away.  High word: stride byte offset (K-major: between
// 8-row groups; MN-major: between 8-channel groups) in the same units.
__device__ __forceinline__ unsigned tc_desc_lo(unsigned saddr, unsigned lbo16) {
  return (saddr >> 4) | (lbo16 << 16);
}
__device__ __forceinline__ unsigned tc_desc_hi(unsigned sbo16) { return sbo16 | (1u << 14); }
// (one thread issues every MMA of a block one after another: the descriptors
// cost it a few instructions each, not the twenty of assembling them anew)
__device__ __forceinline__ void tc_mma(unsigned d, unsigned a_lo, unsigned a_hi, unsigned b_lo,
                                       unsigned b_hi, unsigned idesc, unsigned acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %2};\n\tmov.b64 db, {%3, %4};\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, {%7, %7, %7, %7}, p;\n\t}"
      :
      : "r"(d), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(acc), "r"(0u));
}
__device__ __forceinline__ void tc_commit(unsigned long long *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   tc_smem_u32(bar))
               : "memory");
}
constexpr int tc_cols(int n) { return n <= 32 ? 32 : (n <= 64 ? 64 : (n <= 128 ? 128 : (n <= 256 ? 256 : 512))); }

constexpr int kHaloThreads = 256;
constexpr int kHaloM = 256;  // positions of a convolution tile: two MMA tiles of 128

// rows of a convolution's halo tile, = 2 (mod 4): the two rows and four channel
// groups that 8 lanes copy together fall on different banks
__host__ __device__ inline int halo_rows(int X) {
  const int r = kHaloM + 2 * (X + 3);
  return r + ((2 - r) & 3);
}
// one plane of the tile and the weights of its nine taps
__host__ __device__ inline size_t halo_smem(int X, int ci, int nb) {
  return (size_t)(ci * 2 + 4) * halo_rows(X) + (size_t)9 * ci * nb * 2 + 128;
}

// What the epilogue of a convolution does with its FP32 sums: stores them (pre,
// if not null) and, with film, h = gamma * sum + beta, gamma = 1 + A0 + A1 r and
// beta = B0 + B1 r per sample, plane and channel, as BF16 lrelu(h) (act) or FP32 h
// (out).
struct ConvOut {
  float *pre = nullptr;
  const float *film = nullptr;  // A0, A1, B0, B1 [z][c]
  const float *r = nullptr;     // [b]
  bf16 *act = nullptr;
  float *out = nullptr;
};

// Forward convolution and input gradient: a block owns 256 positions of a plane
// x NB of the N output channels and takes the three input planes one after
// another, each with its nine taps' weights in one buffer; the resident blocks
// overlap their copies and MMAs.  The MMAs of an accumulator run over the taps
// and, within a tap, over the 16-channel steps, the order of k_conv3d_tc: the
// same sums bit for bit, so that no BF16 rounding downstream moves.  Waits and
// errors as there.
template <int NB>
__global__ void __launch_bounds__(kHaloThreads) k_conv3d_halo(Shape s, const bf16 *__restrict__ X,
                                                              const bf16 *__restrict__ W,
                                                              ConvOut o, int Ci, int N, int tiles,
                                                              HaloDiv d, int *err) {
  constexpr int kCols = tc_cols(2 * NB);
  __shared__ float gam[NB], bet[NB];
  extern __shared__ __align__(128) unsigned char halo_sm[];
  __shared__ __align__(8) unsigned long long bar;
  __shared__ unsigned tmem_base_s;
  __shared__ int fail_s;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int XP = s.X + 2, PP = s.Y * XP, R = halo_rows(s.X);
  const int pl = (int)blockIdx.x / tiles, p0 = ((int)blockIdx.x - pl * tiles) * kHaloM;
  const int nmt = PP - p0 > 128 ? 2 : 1;  // MMA tiles with positions of the plane
  const int used = nmt * 128 + 2 * (XP + 1);
  const int z = pl % s.Z, n0 = (int)blockIdx.y * NB, groups = Ci / 8;
  // [8-channel group][row], [tap][8-channel group][n], the rows' elements in a plane
  unsigned char *A = halo_sm, *Bm = halo_sm + (size_t)16 * groups * R;
  int *src_row = reinterpret_cast<int *>(Bm + (size_t)9 * groups * NB * 16);
  for (int r = t; r < used; r += kHaloThreads) src_row[r] = halo_voxel(s, d, p0, r) * Ci;
  if (o.film && t < NB) {
    const long long zc = (long long)s.Z * N, q = (long long)z * N + n0 + t;
    const float rb = o.r[pl / s.Z];
    gam[t] = 1.f + o.film[q] + o.film[zc + q] * rb;
    bet[t] = o.film[2 * zc + q] + o.film[3 * zc + q] * rb;
  }

  if (warp == 0) {
    tc_alloc(&tmem_base_s, kCols);
  }
  if (t == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem_u32(&bar)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fail_s = 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = tmem_base_s;

  const long long plane = (long long)s.Y * s.X;
  bool ok = true;
  for (int dz = 0; dz < 3; ++dz) {
    if (dz) {  // the MMAs of the plane before have read the buffer
      if (t == 0 && !tc_wait(&bar, (unsigned)((dz - 1) & 1))) fail_s = 1;
      __syncthreads();
      if (fail_s) {
        ok = false;
        break;
      }
    }
    const bool in = z + dz - 1 >= 0 && z + dz - 1 < s.Z;
    const bf16 *Xp = X + ((long long)pl + dz - 1) * plane * Ci;
    const int g0 = t & 3;
    for (int r = t >> 2; r < used; r += kHaloThreads / 4) {
      const bf16 *src = in ? Xp + src_row[r] + g0 * 8 : X;
      unsigned dst = tc_smem_u32(A) + (unsigned)(g0 * R + r) * 16u;
      for (int g = g0; g < groups; g += 4) {
        tc_cp16s(dst, src, in ? 16u : 0u);
        src += in ? 32 : 0;
        dst += 64u * (unsigned)R;
      }
    }
    // rows tap * NB + n of the weights
    const bf16 *Wp = W + ((long long)dz * 9 * N + n0) * Ci + g0 * 8;
    for (int rr = t >> 2; rr < 9 * NB; rr += kHaloThreads / 4) {
      const int tap = rr / NB, n = rr - tap * NB;
      const bf16 *src = Wp + (tap * N + n) * Ci;
      unsigned dst = tc_smem_u32(Bm) + (unsigned)((tap * groups + g0) * NB + n) * 16u;
      for (int g = g0; g < groups; g += 4) {
        tc_cp16s(dst, src, 16u);
        src += 32;
        dst += 64u * NB;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (t == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const unsigned a0 = tc_desc_lo(tc_smem_u32(A), (unsigned)R);
      unsigned b_lo = tc_desc_lo(tc_smem_u32(Bm), NB);
      const unsigned hi = tc_desc_hi(8);
#pragma unroll
      for (int tap = 0; tap < 9; ++tap) {
        unsigned a_lo = a0 + (unsigned)((XP + 1) + (tap / 3 - 1) * XP + (tap % 3 - 1));
        for (int c = 0; c < groups; c += 2) {
          tc_mma(tmem, a_lo, hi, b_lo, hi, tc_idesc(NB), (unsigned)(dz | tap | c));
          if (nmt == 2)
            tc_mma(tmem + NB, a_lo + 128, hi, b_lo, hi, tc_idesc(NB), (unsigned)(dz | tap | c));
          a_lo += 2 * (unsigned)R;
          b_lo += 2 * NB;
        }
      }
      tc_commit(&bar);
    }
  }
  if (ok) {
    if (t == 0 && !tc_wait(&bar, 0)) fail_s = 1;  // the third phase
    __syncthreads();
    ok = !fail_s;
  }
  if (ok) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int mt = warp >> 2, p = p0 + mt * 128 + (warp & 3) * 32 + lane;
    const int y = p / XP, x = p - y * XP - 1;
    const bool valid = p < PP && x >= 0 && x < s.X;
    const long long at = ((long long)pl * plane + (long long)y * s.X + x) * N + n0;
    if (mt < nmt) {
#pragma unroll
      for (int c0 = 0; c0 < NB; c0 += 16) {
        unsigned r[16];
        tc_ld16(tmem + ((unsigned)((warp & 3) * 32) << 16) + (unsigned)(mt * NB + c0), r);
        if (valid) {
          if (o.pre) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
              reinterpret_cast<float4 *>(o.pre + at + c0)[q] =
                  make_float4(__uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]),
                              __uint_as_float(r[4 * q + 2]), __uint_as_float(r[4 * q + 3]));
          }
          if (o.film) {
            float h[16];
#pragma unroll
            for (int q = 0; q < 16; ++q) h[q] = gam[c0 + q] * __uint_as_float(r[q]) + bet[c0 + q];
            if (o.act) {
              __align__(16) __nv_bfloat162 a[8];
#pragma unroll
              for (int q = 0; q < 8; ++q)
                a[q] = __floats2bfloat162_rn(lrelu(h[2 * q]), lrelu(h[2 * q + 1]));
              uint4 *dst = reinterpret_cast<uint4 *>(o.act + at + c0);
              dst[0] = reinterpret_cast<const uint4 *>(a)[0];
              dst[1] = reinterpret_cast<const uint4 *>(a)[1];
            } else {
#pragma unroll
              for (int q = 0; q < 4; ++q)
                reinterpret_cast<float4 *>(o.out + at + c0)[q] =
                    make_float4(h[4 * q], h[4 * q + 1], h[4 * q + 2], h[4 * q + 3]);
            }
          }
        }
      }
    }
  } else if (t == 0) {
    atomicExch(err, 1);
    // (MMAs still in flight end within a bounded wait before the TMEM goes back)
    tc_wait(&bar, 0);
    tc_wait(&bar, 1);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    tc_dealloc(tmem, kCols);
  }
}

// Weight gradient: D[(dz, ci)][co] of the taps (dy, dx = -1, 0, 1) of one dy
// accumulate in tensor memory over a range of voxels.  The three planes' groups
// of 8 input channels are the rows of A, 128 at a time (grid.y: row block and
// dy); K = 16 voxels per MMA, in two groups of 8 that lie in one row of the
// plane each, so X must be a multiple of 8 and a plane of 16; both operands
// MN-major.  A block walks the tiles of up to 128 voxels of its range, the
// copies of the next tile running under the MMAs of this one, and adds its
// sums to dW at the end.  Ranges, K groups and their order are those of
// k_conv3d_wgrad_tc: the same partial sums bit for bit.
constexpr int kWgM = 128;  // voxels of a tile

// rows of its halo tile, = 2 (mod 4): the two rows and four channel groups that
// 8 lanes copy together fall on different banks
__host__ __device__ inline int wg_rows(int X) {
  const int r = kWgM + 2 * (kWgM / X + 1) + 2;
  return r + ((2 - r) & 3);
}
// buffers
constexpr int wg_bufs(int co) { return co <= 48 ? 4 : 3; }
template <int CO>
size_t wg_smem(int X) {
  return wg_bufs(CO) * ((size_t)16 * 16 * wg_rows(X) + (size_t)kWgM * CO * 2) + 128;
}

template <int CO>
__global__ void __launch_bounds__(kHaloThreads + 32)
    k_conv3d_wgrad_halo(Shape s, const bf16 *__restrict__ dY, const bf16 *__restrict__ X,
                        float *__restrict__ dW, int Ci, long long chunk, HaloDiv d, int *err) {
  constexpr int kCols = tc_cols(3 * CO), G = CO / 8, NB = wg_bufs(CO);
  extern __shared__ __align__(128) unsigned char halo_sm[];
  __shared__ __align__(8) unsigned long long full[NB], empty[NB];
  __shared__ unsigned kdesc[NB][kWgM / 16];  // per K step: row of its first voxel, offset to the 8 others
  __shared__ unsigned tmem_base_s;
  __shared__ int fail_s;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int XP = s.X + 2, R = wg_rows(s.X), YX = s.Y * s.X;
  const int mb = (int)blockIdx.y / 3, dy = (int)blockIdx.y % 3 - 1;
  const long long M = s.voxels();
  const int k0 = (int)(blockIdx.x * chunk), k1 = (int)(k0 + chunk < M ? k0 + chunk : M);
  const int buf_bytes = 256 * R + kWgM * CO * 2;

  if (warp == 0) {
    tc_alloc(&tmem_base_s, kCols);
  }
  if (t == 0) {
    for (int q = 0; q < NB; ++q) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(tc_smem_u32(&full[q])),
                   "r"(kHaloThreads));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem_u32(&empty[q])));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fail_s = 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = tmem_base_s;

  const int cg = Ci / 8;
  // this thread copies the row groups 4 q + (t & 3) of the row block: their plane
  // offset and channels (a group beyond the three planes stays zero)
  int gz[4], gc[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int g = mb * 16 + 4 * q + (t & 3);
    gz[q] = g / cg - 1;
    gc[q] = (g - g / cg * cg) * 8;
  }
  // padded position of the voxel at offset v of a plane, less one: the row of the
  // tile that its dx = -1 neighbour has
  auto pos = [&](int v) { return v + 2 * d.X.div(v); };
  // voxels of the tile that starts at v: within a plane and the range
  auto tile_len = [&](int v) { return min(min(kWgM, k1 - v), YX - (v - d.YX.div(v) * YX)); };
  auto load = [&](int v, int len, int b) {
    unsigned char *A = halo_sm + b * buf_bytes, *Bm = A + 256 * R;
    const int pl = d.YX.div(v), off = v - pl * YX, z = pl % s.Z;
    const int P0 = pos(off), used = pos(off + len - 1) + 3 - P0;
    for (int r = t >> 2; r < used; r += kHaloThreads / 4) {
      const int row = d.XP.div(P0 + r), px = P0 + r - row * XP - 1;
      int y = row + dy, x = px < 0 ? s.X - 1 : (px >= s.X ? 0 : px);
      y = y < 0 ? y + s.Y : (y >= s.Y ? y - s.Y : y);
      const long long vox = (long long)pl * YX + y * s.X + x;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const bool in = gz[q] < 2 && z + gz[q] >= 0 && z + gz[q] < s.Z;
        tc_cp16(A + ((4 * q + (t & 3)) * R + r) * 16,
                in ? X + (vox + (long long)gz[q] * YX) * Ci + gc[q] : X, in ? 16u : 0u);
      }
    }
    if (t < len / 16) {
      const int p = pos(off + 16 * t);
      kdesc[b][t] = (unsigned)(p - P0) | ((unsigned)(pos(off + 16 * t + 8) - p) << 16);
    }
    for (int e = t; e < len * G; e += kHaloThreads) {
      const int r = e / G, g = e - r * G;
      tc_cp16(Bm + (g * kWgM + r) * 16, dY + ((long long)v * CO + e * 8), 16u);
    }
  };
  // The copying warps run ahead of the MMA warp by up to NB tiles: full[b] is
  // reached when every copying thread's part of the tile in buffer b has
  // landed, empty[b] when the MMAs have read it.  (One set of threads copying
  // and issuing in turn took 2.6 us a tile of 32 x 32 channels against 1.75.)
  bool ok = true;
  int tiles = 0;
  if (warp < kHaloThreads / 32) {
    constexpr int D = NB - 2;  // tiles in flight behind the newest
    auto landed = [&](int i) {  // tile i is this thread's oldest in flight
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc_smem_u32(&full[i % NB]))
                   : "memory");
    };
    for (int v = k0; v < k1 && ok; ++tiles) {
      const int len = tile_len(v), b = tiles % NB;
      if (tiles >= NB) ok = tc_wait(&empty[b], (unsigned)((tiles / NB - 1) & 1));
      if (ok) {
        load(v, len, b);
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (tiles >= D) {
          asm volatile("cp.async.wait_group %0;" ::"n"(D) : "memory");
          landed(tiles - D);
        }
      }
      v += len;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (ok) {
      for (int i = max(0, tiles - D); i < tiles; ++i) landed(i);
      // the last commit covers every earlier tcgen05 operation
      ok = tc_wait(&empty[(tiles - 1) % NB], (unsigned)(((tiles - 1) / NB) & 1));
    }
  } else if (lane == 0) {
    const unsigned a_hi = tc_desc_hi((unsigned)R);
    for (int v = k0; v < k1; ++tiles) {
      const int len = tile_len(v), b = tiles % NB;
      ok = tc_wait(&full[b], (unsigned)((tiles / NB) & 1));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const unsigned a0 = tc_smem_u32(halo_sm + b * buf_bytes);
      const unsigned a_base = tc_desc_lo(a0, 0);
      unsigned b_lo = tc_desc_lo(a0 + 256 * R, 8);
      for (int k = 0; k < len / 16; ++k) {
        const unsigned a_lo = a_base + kdesc[b][k];
#pragma unroll
        for (int dx = 0; dx < 3; ++dx)
          tc_mma(tmem + dx * CO, a_lo + dx, a_hi, b_lo, tc_desc_hi(kWgM), tc_idesc_mn(CO),
                 (unsigned)(tiles | k));
        b_lo += 16;
      }
      tc_commit(&empty[b]);
      v += len;
    }
  }
  if (!ok) fail_s = 1;
  __syncthreads();
  ok = !fail_s;
  if (ok) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // row of D: channel ci of plane dz; the warps 0-3 and 4-7 take alternate columns
    const int row = mb * 128 + (warp & 3) * 32 + lane, dz = row / Ci, ci = row - dz * Ci;
    for (int c = warp < 8 ? (warp >> 2) * 16 : 3 * CO; c < 3 * CO; c += 32) {
      unsigned r[16];
      tc_ld16(tmem + ((unsigned)((warp & 3) * 32) << 16) + (unsigned)c, r);
      const int q = c / CO, co = c - q * CO, tap = dz * 9 + (dy + 1) * 3 + q;
      if (dz < 3) {
        float *dst = dW + ((long long)tap * CO + co) * Ci + ci;
#pragma unroll
        for (int e = 0; e < 16; ++e) atomicAdd(dst + (long long)e * Ci, __uint_as_float(r[e]));
      }
    }
  } else if (t == 0) {
    atomicExch(err, 1);
    for (int q = 0; q < 2 * NB; ++q) tc_wait(&empty[q % NB], q / NB);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    tc_dealloc(tmem, kCols);
  }
}

}  // namespace gen
}  // namespace plc
