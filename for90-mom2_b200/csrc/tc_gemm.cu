// Trailing-update GEMM of the mixed-precision LU on the sm_100a tensor cores.
//
//   C  -=  L21 * U12      (complex FP32, C = A22 of the LU, in place)
//
// Complex products are built from real ones: with C viewed as a real matrix
// (re/im interleaved rows, 2m x nc), L21 expanded to the real 2m x 2k matrix
//   Ahat[2i][2l] = Re L, Ahat[2i][2l+1] = -Im L, Ahat[2i+1][2l] = Im L,
//   Ahat[2i+1][2l+1] = Re L
// and U12 viewed as real 2k x nc (its own interleaved storage), C -= Ahat B.
// Accuracy: each operand is split into two FP16 numbers, high part and
// remainder, after scalings by powers of two: per column of L21 (and inversely
// per row of U12) one that brings the columns' largest entries level, then per
// row of L21 and per column of U12 one that puts its largest entry just below
// 2^15; the MMA accumulates hi*hi + hi*lo + lo*hi (three kind::f16 passes into
// one FP32 TMEM accumulator) and the epilogue undoes the scaling.  An entry
// keeps 22 bits, or 2^-40 of its row's (column's) largest scaled entry: rows of
// A of any sizes, which grade L by column against U by row, cost nothing, and
// what smaller entries lose beyond the 22 bits stays, in column j of the update,
// below k 2^-39 of the largest entry of column j of |L| |U|, as every column of L
// has an entry at its level.
// Three passes on TF32 parts keep no more (the tensor core cuts the remainder
// to TF32) at half the rate and twice the operand bytes.  Measured, relative
// Frobenius error of C - L U against FP64, Gaussian operands (rows and columns
// scaled by any powers of two alike), k = 16 / 48 / 64 / 128 / 256: 2.0e-7 /
// 4.3e-7 / 5.3e-7 / 9.8e-7 / 1.9e-6, with TF32 parts 3.0e-7 / 7.5e-7 / 9.6e-7 /
// 1.9e-6 / 3.7e-6.
//
// Kernel: persistent, one CTA per SM, 128 x 256 output tiles, K blocks of
// 32 halves (one 64-byte swizzle row) staged by TMA in a 4-deep ring (three
// stages can be under way while one is consumed).
//   warp 0    TMA producer (one elected lane)
//   warp 1    MMA issuer (one elected lane; tcgen05.mma cta_group::1)
//   warp 2    TMEM allocator (512 columns = two 128 x 256 accumulators)
//   warps 4-11 epilogue: tcgen05.ld the accumulator, C -= acc (coalesced);
//             two warps per 32 rows, so that enough of C is in flight to keep
//             up with the MMAs of a K = 512 tile
// Bound: with n = 15,360 and blocks of 192 columns (real K = 384) a tile's MMAs
// take 5 us, its operands 590 KB through L2 and its part of C 262 KB of HBM
// traffic; the trailing updates of the factorisation take 34 ms (with 256 columns
// 27.7, for dearer narrow updates between them; with TF32 parts, two stages and
// four epilogue warps 43.3; 18.3 at the bf16 rate).
// Every mbarrier wait is bounded; on timeout the kernel records the error,
// stops issuing work, waits (bounded) for its own copies and for the MMAs
// already issued, frees TMEM and exits.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>
#include <cstring>

#include "mom_internal.h"

namespace mom {
namespace {

constexpr int kBM = 128, kBN = 256, kBK = 32, kStages = 4;
constexpr int kTileA = kBM * kBK * 2;  // bytes of one A tile (hi or lo)
constexpr int kTileB = kBN * kBK * 2;  // bytes of one B tile
constexpr int kStageBytes = 2 * kTileA + 2 * kTileB;
constexpr int kEpiWarps = 8, kTcThreads = 128 + 32 * kEpiWarps;
constexpr int kEpiCols = 32;  // columns of C an epilogue warp has in flight
constexpr long long kDrainPolls = 1LL << 22;  // bound of the waits for work already issued

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Bounded parity wait; returns false (and raises *abort) after `limit` polls,
// or when another warp of the CTA has raised *abort.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, unsigned parity, volatile int *abort, long long limit) {
  const uint32_t a = smem_u32(bar);
  for (long long it = 0;; it++) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
    if ((it & 1023) == 1023 || it >= limit) {
      if (*abort) return false;
      if (it >= limit) {
        *abort = 1;
        return false;
      }
    }
  }
}

__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, uint64_t *bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}

// K-major, 64-byte swizzled operand tile: rows of 64 bytes, 8-row atoms of
// 512 bytes (SBO), LBO unused (1), descriptor version 1, layout SWIZZLE_64B.
__device__ __forceinline__ uint64_t sw64_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)1 << 16;           // LBO (16-byte units)
  d |= (uint64_t)(512 >> 4) << 32;  // SBO
  d |= (uint64_t)1 << 46;           // version
  d |= (uint64_t)4 << 61;           // SWIZZLE_64B
  return d;
}

// kind::f16 instruction descriptor: D f32, A/B f16, both K-major, M=128, N=256.
constexpr uint32_t kIdesc = (1u << 4) | ((uint32_t)(kBN >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);

__device__ __forceinline__ void mma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(kIdesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// K blocks up to which the epilogue brings the C that it needs next to L2: with
// few of them its read of C bounds the tile (K = 64, 7,260 unknowns: 220 to 175 us
// per update, whole calls 24.1 to 22.5 ms; 4,860 12.45 to 12.14), with more the
// prefetches only get in the operands' way (K = 192: 42.04 to 42.24 ms at 10,140).
constexpr int kAheadBlocks = 4;

struct TcArgs {
  float *C;        // real view of the complex FP32 C block
  int64_t ldc;     // in floats
  int Mr, Nc, Kp;  // real rows of C, columns, real K padded to kBK
  const float *rinv, *cinv;  // undo the scaling: per complex row, per column
  int *err;        // device error word (timeout)
  long long spin;  // polls before an mbarrier wait is declared timed out
};

__global__ void __launch_bounds__(kTcThreads, 1)
    tc_gemm_kernel(const __grid_constant__ CUtensorMap mAhi, const __grid_constant__ CUtensorMap mAlo,
                   const __grid_constant__ CUtensorMap mBhi, const __grid_constant__ CUtensorMap mBlo, TcArgs a) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // 1024-byte aligned stage buffers (swizzle atoms need 512)
  unsigned char *smem = reinterpret_cast<unsigned char *>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ uint64_t full[kStages], empty[kStages], acc_full[2], acc_empty[2], drain;
  __shared__ uint32_t tmem_base;
  __shared__ int abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int numM = a.Mr / kBM, numN = (a.Nc + kBN - 1) / kBN, ntiles = numM * numN, nk = a.Kp / kBK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], kEpiWarps);  // one arrival per epilogue warp
    }
    mbar_init(&drain, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base;
  volatile int *abort = &abort_flag;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      int s = 0;
      unsigned ph = 0;
      unsigned last_ph[kStages];
      bool pending[kStages];
      for (int i = 0; i < kStages; i++) pending[i] = false;
      for (int t = blockIdx.x; t < ntiles && !*abort; t += gridDim.x) {
        const int tm = t % numM, tn = t / numM;
        for (int kb = 0; kb < nk; kb++) {
          if (!mbar_wait(&empty[s], ph ^ 1, abort, a.spin)) break;
          unsigned char *st = smem + (size_t)s * kStageBytes;
          mbar_expect_tx(&full[s], kStageBytes);
          tma_load_2d(st, &mAhi, &full[s], kb * kBK, tm * kBM);
          tma_load_2d(st + kTileA, &mAlo, &full[s], kb * kBK, tm * kBM);
          tma_load_2d(st + 2 * kTileA, &mBhi, &full[s], kb * kBK, tn * kBN);
          tma_load_2d(st + 2 * kTileA + kTileB, &mBlo, &full[s], kb * kBK, tn * kBN);
          pending[s] = true;
          last_ph[s] = ph;
          if (++s == kStages) {
            s = 0;
            ph ^= 1;
          }
        }
      }
      // wait (bounded) until the last copy into every stage has landed: the
      // MMA warp may give up on a stage whose copy is still in flight, and
      // the CTA must not exit before its shared memory is written
      volatile int dummy = 0;
      for (int i = 0; i < kStages; i++)
        if (pending[i]) mbar_wait(&full[i], last_ph[i], &dummy, kDrainPolls);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      int s = 0;
      unsigned ph = 0;
      int it = 0;
      for (int t = blockIdx.x; t < ntiles && !*abort; t += gridDim.x, it++) {
        const int acc = it & 1;
        const unsigned acc_ph = (it >> 1) & 1;
        if (!mbar_wait(&acc_empty[acc], acc_ph ^ 1, abort, a.spin)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t d = tmem + (uint32_t)(acc * kBN);
        bool ok = true;
        for (int kb = 0; kb < nk; kb++) {
          if (!mbar_wait(&full[s], ph, abort, a.spin)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t base = smem_u32(smem + (size_t)s * kStageBytes);
          const uint32_t ahi = base, alo = base + kTileA, bhi = base + 2 * kTileA, blo = base + 2 * kTileA + kTileB;
#pragma unroll
          for (int k = 0; k < kBK / 16; k++) {
            const uint32_t off = (uint32_t)k * 32;  // 16 halves = 32 bytes along K inside the swizzle atom
            mma_f16(d, sw64_desc(ahi + off), sw64_desc(bhi + off), (kb | k) != 0);
            mma_f16(d, sw64_desc(ahi + off), sw64_desc(blo + off), 1);
            mma_f16(d, sw64_desc(alo + off), sw64_desc(bhi + off), 1);
          }
          mma_commit(&empty[s]);  // frees the stage when these MMAs complete
          if (++s == kStages) {
            s = 0;
            ph ^= 1;
          }
        }
        if (!ok) break;
        mma_commit(&acc_full[acc]);
      }
      // on abort, wait (bounded) until every MMA issued so far has completed
      // (they read the stage buffers and write TMEM, both released below)
      if (*abort) {
        volatile int dummy = 0;
        mma_commit(&drain);
        mbar_wait(&drain, 0, &dummy, kDrainPolls);
      }
    }
  } else if (warp >= 4) {
    // ---------------- epilogue ----------------
    const int ew = warp % 4;            // TMEM lanes 32*ew .. 32*ew+31
    const int half = (warp - 4) / 4;    // columns half * 128 .. of the tile
    int it = 0;
    const bool ahead = nk <= kAheadBlocks;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x, it++) {
      const int acc = it & 1;
      const unsigned acc_ph = (it >> 1) & 1;
      const int tm = t % numM, tn = t / numM;
      const int64_t row = (int64_t)tm * kBM + ew * 32 + lane;
      float *crow = a.C + row;
      const float rs = a.rinv[row >> 1];
      int ok = 1;
#pragma unroll 1
      for (int c0 = half * (kBN / 2); c0 < (half + 1) * (kBN / 2); c0 += kEpiCols) {
        const int col0 = tn * kBN + c0;
        // the loads of C in flight before the accumulator is waited for and
        // before the stores (which the compiler must assume to alias them)
        float cv[kEpiCols];
#pragma unroll
        for (int j = 0; j < kEpiCols; j++)
          cv[j] = (col0 + j < a.Nc) ? __ldcs(crow + (int64_t)(col0 + j) * a.ldc) : 0.0f;
        if (ahead) {  // the next columns' lines (or the next tile's first) on their way to L2, one per lane
          const bool last = c0 + kEpiCols == (half + 1) * (kBN / 2);
          const int tp = last ? t + (int)gridDim.x : t;
          const int cp = tp / numM * kBN + (last ? half * (kBN / 2) : c0 + kEpiCols) + lane;
          const float *line = a.C + (int64_t)(tp % numM) * kBM + ew * 32 + (int64_t)cp * a.ldc;
          if (tp < ntiles && cp < a.Nc) asm volatile("prefetch.global.L2 [%0];" ::"l"(line) : "memory");
        }
        if (c0 == half * (kBN / 2)) {
          if (lane == 0) ok = mbar_wait(&acc_full[acc], acc_ph, abort, a.spin) ? 1 : 0;
          ok = __shfl_sync(0xffffffffu, ok, 0);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        const float sc = col0 + lane < a.Nc ? a.cinv[col0 + lane] : 0.0f;
        uint32_t v[kEpiCols];
        const uint32_t taddr = tmem + ((uint32_t)(ew * 32) << 16) + (uint32_t)(acc * kBN + c0);
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
            "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
              "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
              "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
              "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
            : "r"(taddr));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < kEpiCols; j++) {
          const float cs = __shfl_sync(0xffffffffu, sc, j);
          if (col0 + j < a.Nc)
            __stcs(crow + (int64_t)(col0 + j) * a.ldc, fmaf(-(__uint_as_float(v[j]) * rs), cs, cv[j]));
        }
      }
      if (!ok) break;
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[acc]);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && abort_flag) atomicExch(a.err, 1);
  if (warp == 2) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

// Power of two that puts a magnitude with these float bits into [2^14, 2^15),
// and its reciprocal.
__device__ __forceinline__ float scale_of(unsigned bits, float *inv) {
  const int e = (int)(bits >> 23);                  // biased exponent, 0 for zero
  const int s = bits == 0u ? 0 : min(126, max(-126, 141 - e));
  *inv = __uint_as_float((unsigned)(127 - s) << 23);
  return __uint_as_float((unsigned)(127 + s) << 23);
}
__device__ __forceinline__ unsigned mag_bits(float2 z) {
  return max(__float_as_uint(fabsf(z.x)), __float_as_uint(fabsf(z.y)));
}
__device__ __forceinline__ float pow2(int e) { return __uint_as_float((unsigned)(127 + e) << 23); }

// The larger of m and the magnitude of z, if that is finite.
__device__ __forceinline__ void take_mag(unsigned &m, float2 z) {
  const unsigned v = mag_bits(z);
  if (v < 0x7f800000u) m = max(m, v);
}
__device__ __forceinline__ int level_of(unsigned bits) { return bits == 0u ? -1 : (int)(bits >> 23); }

// level[l]: biased exponent of the largest finite entry of column l of the
// complex block L (m x k, ld; tr: of the transpose of a k x m block), -1 if there
// is none.  One CTA per column (tr: per four, whose entries lie side by side).
__global__ void __launch_bounds__(256) col_level_kernel(const float2 *L, int64_t ld, int m, int k, int *level, bool tr) {
  __shared__ unsigned s_max[8][4];
  const int per = tr ? 4 : 1, l0 = blockIdx.x * per;
  unsigned b[4] = {0u, 0u, 0u, 0u};
  if (!tr) {
#pragma unroll 8
    for (int i = threadIdx.x; i < m; i += 256) take_mag(b[0], L[i + (int64_t)l0 * ld]);
  } else {
#pragma unroll 2
    for (int i = threadIdx.x; i < m; i += 256)
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (l0 + q < k) take_mag(b[q], L[l0 + q + (int64_t)i * ld]);
  }
#pragma unroll
  for (int q = 0; q < 4; q++) {
    b[q] = __reduce_max_sync(0xffffffffu, b[q]);
    if (threadIdx.x % 32 == 0) s_max[threadIdx.x / 32][q] = b[q];
  }
  __syncthreads();
  if ((int)threadIdx.x < per && l0 + (int)threadIdx.x < k) {
    unsigned v = 0u;
    for (int w = 0; w < 8; w++) v = max(v, s_max[w][threadIdx.x]);
    level[l0 + threadIdx.x] = level_of(v);
  }
}

// The levels of every operand of a blocked substitution at once: column l (TR:
// row l) of the n x n factors over the rows (columns) after its block of `rows`
// into after[l] and over those before it into before[l].  Reads the factors
// once (HBM bound, 75 us at 7,680 unknowns), where a launch per operand added 9
// us to each of the 60 updates of a solve.
template <bool TR>
__global__ void __launch_bounds__(1024) block_levels_kernel(const float2 *F, int64_t lda, int n, int rows, int *after,
                                                            int *before) {
  __shared__ unsigned s_max[2][32][33];
  const int lane = threadIdx.x % 32, wid = threadIdx.x / 32;
  // TR: a warp reads 32 rows of a column, else 32 rows of one of its column's
  const int l = TR ? blockIdx.x * 32 + lane : blockIdx.x * 4 + wid / 8;
  unsigned b[2] = {0u, 0u};
  if (l < n) {
    const int k0 = l / rows * rows, k1 = min(n, k0 + rows);
    const int first = TR ? wid : (wid % 8) * 32 + lane, step = TR ? 32 : 256;
#pragma unroll 8
    for (int i = first; i < n; i += step)
      if (i < k0 || i >= k1) take_mag(b[i < k0], TR ? F[l + (int64_t)i * lda] : F[i + (int64_t)l * lda]);
  }
#pragma unroll
  for (int q = 0; q < 2; q++) s_max[q][wid][lane] = TR ? b[q] : __reduce_max_sync(0xffffffffu, b[q]);
  __syncthreads();
  if (threadIdx.x < (TR ? 32 : 4)) {
    const int at = TR ? blockIdx.x * 32 + threadIdx.x : blockIdx.x * 4 + threadIdx.x;
    for (int q = 0; q < 2 && at < n; q++) {
      unsigned v = 0u;
      for (int w = 0; w < (TR ? 32 : 8); w++) v = max(v, TR ? s_max[q][w][threadIdx.x] : s_max[q][threadIdx.x * 8 + w][0]);
      (q ? before : after)[at] = level_of(v);
    }
  }
}
// By how many powers of two each of the k columns is raised to the highest
// level, staged by a CTA of 256 threads (every warp finds the top).
constexpr int kMaxK = 1024;
__device__ __forceinline__ void stage_raise(const int *level, int k, int *up) {
  const int tid = threadIdx.x + threadIdx.y * blockDim.x;
  int top = -1;
#pragma unroll 8
  for (int l = tid % 32; l < k; l += 32) top = max(top, level[l]);
  top = __reduce_max_sync(0xffffffffu, top);
  for (int l = tid; l < k; l += 256) up[l] = level[l] < 0 ? 0 : min(126, top - level[l]);
  __syncthreads();
}
// v = hi + lo up to FP16 rounding of the remainder
__device__ __forceinline__ void split_half(float v, __half *hi, __half *lo) {
  *hi = __float2half_rn(v);
  *lo = __float2half_rn(v - __half2float(*hi));
}

// Ahat_hi / Ahat_lo (2m x Kp halves, row-major) from the complex block L
// (m x k, ld), or (tr) from the transpose of a k x m block: L(i, l) = P[l + i
// ld], its columns raised to one level, and the rows' inverse scales.  One CTA
// (32 x 8 threads) per 32 rows and gridDim.y-th of the columns: the rows' largest
// entries first, then 32 x 32 tiles through shared memory, the
// complex block read along its contiguous direction both times (the second
// time from L2) and the expanded rows written as pairs of halves.
__global__ void __launch_bounds__(256) expand_a_kernel(const float2 *L, int64_t ld, int m, int k, int Kp, __half *hi,
                                                       __half *lo, float *rinv, const int *level, bool tr) {
  __shared__ float2 t[32][33];  // [l][i] of the tile
  __shared__ unsigned s_max[32];
  const int i0 = blockIdx.x * 32, tx = threadIdx.x, ty = threadIdx.y;
  __shared__ int s_up[kMaxK];
  if (ty == 0) s_max[tx] = 0u;
  stage_raise(level, k, s_up);
  auto at = [&](float2 z, int l) {
    const float up = pow2(s_up[l]);
    return make_float2(z.x * up, z.y * up);
  };
  if (!tr) {
    unsigned b = 0u;
    if (i0 + tx < m) {
#pragma unroll 8
      for (int l = ty; l < k; l += 8) b = max(b, mag_bits(at(L[i0 + tx + (int64_t)l * ld], l)));
    }
    atomicMax(&s_max[tx], b);
  } else {
    for (int r = ty; r < 32; r += 8) {
      unsigned b = 0u;
      if (i0 + r < m) {
#pragma unroll 8
        for (int l = tx; l < k; l += 32) b = max(b, mag_bits(at(L[l + (int64_t)(i0 + r) * ld], l)));
      }
      b = __reduce_max_sync(0xffffffffu, b);
      if (tx == 0) s_max[r] = b;
    }
  }
  for (int l0 = 32 * blockIdx.y; l0 < Kp / 2; l0 += 32 * gridDim.y) {
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
      if (!tr) {
        const int i = i0 + tx, l = l0 + r;
        t[r][tx] = (i < m && l < k) ? at(L[i + (int64_t)l * ld], l) : make_float2(0.f, 0.f);
      } else {
        const int l = l0 + tx, i = i0 + r;
        t[tx][r] = (i < m && l < k) ? at(L[l + (int64_t)i * ld], l) : make_float2(0.f, 0.f);
      }
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
      const int i = i0 + r, l = l0 + tx;
      if (i >= m || 2 * l >= Kp) continue;
      float inv;
      const float sc = scale_of(s_max[r], &inv);
      const float2 z = t[tx][r];
      if (l == 0) rinv[i] = inv;
      __half2 h, g;  // (re, im): rows 2i and 2i + 1 hold (re, -im) and (im, re)
      split_half(z.x * sc, &h.x, &g.x);
      split_half(z.y * sc, &h.y, &g.y);
      const int64_t p0 = (2 * (int64_t)i) * Kp + 2 * l, p1 = p0 + Kp;
      *reinterpret_cast<__half2 *>(hi + p0) = __halves2half2(h.x, __hneg(h.y));
      *reinterpret_cast<__half2 *>(hi + p1) = __halves2half2(h.y, h.x);
      *reinterpret_cast<__half2 *>(lo + p0) = __halves2half2(g.x, __hneg(g.y));
      *reinterpret_cast<__half2 *>(lo + p1) = __halves2half2(g.y, g.x);
    }
  }
}

// B_hi / B_lo (nc x Kp halves, K contiguous) from the complex block U (k x nc,
// ld), its rows lowered by what L's columns were raised, and the columns'
// inverse scales: one warp per column.  An entry's two scalings are one power of
// two (applied in halves, since it may leave FP32's range).
__global__ void __launch_bounds__(256) split_b_kernel(const float2 *U, int64_t ld, int k, int nc, int Kp, __half *hi,
                                                      __half *lo, float *cinv, const int *level) {
  const int lane = threadIdx.x & 31, j = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  __shared__ int s_up[kMaxK];
  const float2 *u = U + (int64_t)min(j, nc - 1) * ld;
  stage_raise(level, k, s_up);
  if (j >= nc) return;
  int b = INT_MIN;  // bits of the largest magnitude, less the powers of two
#pragma unroll 8
  for (int l = lane; l < k; l += 32) {
    const unsigned v = mag_bits(u[l]);
    if (v != 0u) b = max(b, (int)v - (s_up[l] << 23));
  }
  b = __reduce_max_sync(0xffffffffu, b);
  const int s = b == INT_MIN ? 0 : min(126, max(-126, 141 - (b >> 23)));
  if (lane == 0) cinv[j] = pow2(-s);
#pragma unroll 8
  for (int l = lane; l < Kp / 2; l += 32) {
    const float2 z = l < k ? u[l] : make_float2(0.f, 0.f);
    const int f = s - (l < k ? s_up[l] : 0);
    const float f1 = pow2(f >> 1), f2 = pow2(f - (f >> 1));
    __half2 h, g;
    split_half(z.x * f1 * f2, &h.x, &g.x);
    split_half(z.y * f1 * f2, &h.y, &g.y);
    reinterpret_cast<__half2 *>(hi + (int64_t)j * Kp)[l] = h;
    reinterpret_cast<__half2 *>(lo + (int64_t)j * Kp)[l] = g;
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// 2-D FP16 tensor map over a row-major rows x cols matrix (cols contiguous),
// box = 32 columns (64 bytes) x box_rows rows, 64-byte swizzle.
int make_map(Ctx *c, CUtensorMap *m, const __half *base, int64_t rows, int64_t cols, int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(c, MOM_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)(cols * sizeof(__half))};
  cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half *>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(c, MOM_ERR_CUDA, "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
  return MOM_OK;
}

// Real K of the expanded operands: 2 k padded with zeros to whole K blocks.
int padded_k(int k) { return (2 * k + kBK - 1) / kBK * kBK; }
size_t up256(size_t b) { return (b + 255) / 256 * 256; }

}  // namespace

// The expansion of L into the operands of tc_cgemm_update (own: room for its
// columns' levels unless they are known).
static void expand_a(Ctx *c, cudaStream_t st, const float2 *L, int64_t ldl, int m, int k, __half *ahi, __half *alo,
                     float *rinv, int *own, const int *levels, bool trans_l) {
  if (!levels) {
    col_level_kernel<<<(unsigned)(trans_l ? (k + 3) / 4 : k), 256, 0, st>>>(L, ldl, m, k, own, trans_l);
    c->launches++;
  }
  // few rows: their columns over several CTAs, each of which looks for the
  // largest entries itself (20 us for 1,664 x 256, 10 with eight)
  const int rb = (m + 31) / 32, cb = std::max(1, std::min((k + 31) / 32, 2 * c->nsm / rb));
  expand_a_kernel<<<dim3(rb, cb), dim3(32, 8), 0, st>>>(L, ldl, m, k, padded_k(k), ahi, alo, rinv, levels ? levels : own,
                                                        trans_l);
  c->launches++;
}

// The expansion of L (m x k) alone, on stream st, for calls of tc_cgemm_update
// with the same m, k and work and reuse_a.
int tc_cgemm_expand(Ctx *c, cudaStream_t st, const float2 *L, int64_t ldl, int m, int k, float *work) {
  const size_t half = up256(sizeof(__half) * 2 * (size_t)m * padded_k(k));
  char *w = reinterpret_cast<char *>(work);
  expand_a(c, st, L, ldl, m, k, (__half *)w, (__half *)(w + half), (float *)(w + 2 * half),
           (int *)(w + 2 * half + up256(sizeof(float) * m)), nullptr, false);
  MOM_CUDA(c, cudaGetLastError());
  return MOM_OK;
}

// C (m x nc complex FP32, ldc) -= L (m x k, ldl) * U (k x nc, ldu) on the
// tensor cores (two FP16 parts per operand, FP32-accurate).  m must be a
// multiple of 64, k of 16.  work: tc_cgemm_work_bytes(m, nc, k) of device
// scratch.  max_ctas > 0 caps the persistent grid.  reuse_a: work already holds
// the expansion of this L (of the previous call, or of tc_cgemm_expand, with the
// same L, m and k).  trans_l: L is given as its k x m transpose at L (ld ldl).  levels:
// those of L's columns if they are known (tc_block_levels).
int tc_cgemm_update(Ctx *c, float2 *C, int64_t ldc, const float2 *L, int64_t ldl, const float2 *U, int64_t ldu, int m,
                    int nc, int k, float *work, int *err, int max_ctas, bool reuse_a, bool trans_l, const int *levels) {
  if (m <= 0 || nc <= 0 || k <= 0) return MOM_OK;
  if ((2 * m) % kBM != 0 || (2 * k) % 32 != 0) return fail(c, MOM_ERR_ARG, "tc_cgemm_update: unsupported shape");
  for (int k0 = 0; k > kMaxK && k0 < k; k0 += kMaxK)  // (no LU or solve has that many)
    MOM_TRY(tc_cgemm_update(c, C, ldc, L + k0 * (trans_l ? 1 : ldl), ldl, U + k0, ldu, m, nc, std::min(kMaxK, k - k0), work,
                            err, max_ctas, false, trans_l));
  if (k > kMaxK) return MOM_OK;
  const int Mr = 2 * m, Kp = padded_k(k);
  char *w = reinterpret_cast<char *>(work);
  auto take = [&](size_t bytes) {
    char *p = w;
    w += up256(bytes);
    return p;
  };
  // the expansion of L first: its place must not depend on nc (tc_cgemm_expand)
  __half *ahi = (__half *)take(sizeof(__half) * (size_t)Mr * Kp), *alo = (__half *)take(sizeof(__half) * (size_t)Mr * Kp);
  float *rinv = (float *)take(sizeof(float) * m);
  int *own = (int *)take(sizeof(int) * k);
  const int *level = levels ? levels : own;
  __half *bhi = (__half *)take(sizeof(__half) * (size_t)nc * Kp), *blo = (__half *)take(sizeof(__half) * (size_t)nc * Kp);
  float *cinv = (float *)take(sizeof(float) * nc);
  if (!reuse_a) expand_a(c, c->stream, L, ldl, m, k, ahi, alo, rinv, own, levels, trans_l);
  split_b_kernel<<<(unsigned)((nc + 7) / 8), 256, 0, c->stream>>>(U, ldu, k, nc, Kp, bhi, blo, cinv, level);
  c->launches++;
  CUtensorMap mAhi, mAlo, mBhi, mBlo;
  MOM_TRY(make_map(c, &mAhi, ahi, Mr, Kp, kBM));
  MOM_TRY(make_map(c, &mAlo, alo, Mr, Kp, kBM));
  MOM_TRY(make_map(c, &mBhi, bhi, nc, Kp, kBN));
  MOM_TRY(make_map(c, &mBlo, blo, nc, Kp, kBN));
  TcArgs ta;
  ta.C = reinterpret_cast<float *>(C);
  ta.ldc = 2 * ldc;
  ta.Mr = Mr;
  ta.Nc = nc;
  ta.Kp = Kp;
  ta.rinv = rinv;
  ta.cinv = cinv;
  ta.err = err;
  ta.spin = wait_polls(c, 1);
  const int ntiles = (Mr / kBM) * ((nc + kBN - 1) / kBN);
  // persistent: one CTA per SM, or fewer when another kernel (the look-ahead
  // panel) is to run beside it
  const int cap = (max_ctas > 0 && max_ctas < c->nsm) ? max_ctas : c->nsm;
  const int grid = ntiles < cap ? ntiles : cap;
  const size_t smem = (size_t)kStages * kStageBytes + 1024;
  {
    ProfScope ps(c, kProfTc);
    tc_gemm_kernel<<<grid, kTcThreads, smem, c->stream>>>(mAhi, mAlo, mBhi, mBlo, ta);
  }
  c->launches++;
  c->tc_flops += 6.0 * Mr * (double)nc * 2 * k;  // three passes, 2 FLOP per real MAC
  MOM_CUDA(c, cudaGetLastError());
  return MOM_OK;
}

// Levels for the updates of a substitution by blocks of `rows` rows with the n x n
// factors F (trans: their transpose): after[l] for the updates of the rows after
// l's block, before[l] for those before it.
int tc_block_levels(Ctx *c, const float2 *F, int64_t lda, int n, int rows, bool trans, int *after, int *before) {
  if (trans) block_levels_kernel<true><<<(n + 31) / 32, 1024, 0, c->stream>>>(F, lda, n, rows, after, before);
  else block_levels_kernel<false><<<(n + 3) / 4, 1024, 0, c->stream>>>(F, lda, n, rows, after, before);
  c->launches++;
  MOM_CUDA(c, cudaGetLastError());
  return MOM_OK;
}

int tc_init_kernels(Ctx *c) {
  MOM_CUDA(c, cudaFuncSetAttribute(tc_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   kStages * kStageBytes + 1024));
  return MOM_OK;
}

size_t tc_cgemm_work_bytes(int m, int nc, int k) {
  const size_t Kp = padded_k(k);
  return 2 * up256(sizeof(__half) * 2 * (size_t)m * Kp) + up256(sizeof(float) * m) + up256(sizeof(int) * k) +
         2 * up256(sizeof(__half) * (size_t)nc * Kp) + up256(sizeof(float) * nc);
}

}  // namespace mom

using namespace mom;
struct mom_ctx : public Ctx {};

// Diagnostics: C -= L U (host arrays, complex FP32 interleaved, column-major,
// leading dimensions m, k, m) through the tensor-core kernel above.
extern "C" int mom_gpu_selftest_cgemm(mom_ctx *c, int32_t m, int32_t nc, int32_t k, const float *L, const float *U,
                                      float *C) {
  if (!c || !L || !U || !C || m <= 0 || nc <= 0 || k <= 0) return MOM_ERR_ARG;
  std::lock_guard<std::mutex> g(c->mu);
  MOM_CUDA(c, cudaSetDevice(c->device));
  const size_t bl = sizeof(float2) * (size_t)m * k, bu = sizeof(float2) * (size_t)k * nc,
               bc = sizeof(float2) * (size_t)m * nc, bw = tc_cgemm_work_bytes(m, nc, k);
  char *buf = nullptr;
  if (cudaMalloc(&buf, bl + bu + bc + bw + 4096) != cudaSuccess) {
    cudaGetLastError();
    return fail(c, MOM_ERR_ALLOC, "selftest allocation failed");
  }
  float2 *dL = (float2 *)buf, *dU = (float2 *)(buf + bl), *dC = (float2 *)(buf + bl + bu);
  float *dw = (float *)(buf + ((bl + bu + bc + 255) / 256) * 256);
  int rc = MOM_OK;
  cudaMemcpyAsync(dL, L, bl, cudaMemcpyHostToDevice, c->stream);
  cudaMemcpyAsync(dU, U, bu, cudaMemcpyHostToDevice, c->stream);
  cudaMemcpyAsync(dC, C, bc, cudaMemcpyHostToDevice, c->stream);
  cudaMemsetAsync(c->dinfo + 2, 0, sizeof(int), c->stream);
  rc = tc_cgemm_update(c, dC, m, dL, m, dU, k, m, nc, k, dw, c->dinfo + 2);
  int err = 0;
  if (rc == MOM_OK) {
    cudaMemcpyAsync(C, dC, bc, cudaMemcpyDeviceToHost, c->stream);
    cudaMemcpyAsync(&err, c->dinfo + 2, sizeof(int), cudaMemcpyDeviceToHost, c->stream);
    if (cudaStreamSynchronize(c->stream) != cudaSuccess) rc = fail(c, MOM_ERR_CUDA, "selftest failed");
    else if (err) rc = fail(c, MOM_ERR_TIMEOUT, "tensor-core GEMM wait timed out");
  }
  cudaStreamSynchronize(c->stream);
  cudaFree(buf);
  return rc;
}
