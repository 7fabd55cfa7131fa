// Register-resident panel factorisation of the LU on one thread-block cluster.
//
// A 64-column panel of the factorisation (partial pivoting, ZGETRF of
// linalg.f90:159-180) as four subpanels of W = 16 columns (eight of W = 8 for
// the tallest), each by
//   panel_reg_kernel  the W columns with pivoting, then the interchanges and
//                     the triangular solve on the panel's other columns;
//   rank_w_kernel     C -= L21 U12 on the panel's columns right of it.
//
// What bounds it.  The panel is a serial chain, one pivot decision per
// column; the arithmetic is small.  A column cost 2.5-3.3 us with the panel in
// a cluster's shared memory (slab swept between two exchanges, a cluster
// barrier per column) and 4.4-5.2 us with the exchange through global memory
// (above 2,816 rows in FP64, 5,632 in FP32).  Here a panel row lives in the
// registers of one thread (R rows of W columns per thread, at most 128
// registers), so the update touches no memory but the broadcast pivot row; W
// is small enough that 16,384 rows (32,768 in FP32) fit one cluster; and the
// exchange is one message per CTA and column sent straight into every CTA's
// shared memory with its arrival counted on an mbarrier (st.async): no cluster
// barrier, fence or global memory in the chain.  One 64-column panel on a B200,
// launches included: FP32 66 / 74 / 86 / 109 us at 2,048 / 4,096 / 8,192 /
// 16,384 rows (1.0 to 1.7 us per column), FP64 86 / 102 / 126 us at 2,048 /
// 4,096 / 8,192.  Of a subpanel's 15 us at 2,048 rows, 12 are its 16 columns
// (per column, in cycles: message latency and wait 300, choice of the pivot
// 170, multipliers and next column 60, candidate 100, rest of the update 300,
// row to shared memory 150, barrier and send 350) and 3 its loads, stores and
// the other columns.
//
// Rows never move during a subpanel: each thread tracks the position its rows
// have after the interchanges and stores them there at the end.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "mom_internal.h"

namespace mom {
namespace {

constexpr int kRegMaxCluster = 16;
constexpr int kPanelNb = 64;
// Polls that a wait goes on for after it ran out: the messages under way, of
// which there is one from every CTA, land in that time.
constexpr long long kPanelDrainPolls = 1LL << 22;

struct RegPanelArgs {
  void *A;
  int64_t lda;
  int64_t j0;        // first column (and row) of the 64-column panel
  int m;             // rows n - j0
  int s0, s1;        // subpanels [s0, s1) of W columns
  int *ipiv;         // ipiv[j0 ..]: pivot rows (global, 0-based)
  int *info;         // first zero pivot (1-based), 0 if none
  int *timeout;      // set when a wait ran out
  long long spin;    // polls before a wait is declared timed out
  int *map;          // [2][128] or null: the subpanels' row moves (from, to), rows from j0, 2 W per subpanel
  // blockIdx.y selects one of several matrices of the same shape
  int64_t batch_A, batch_piv, batch_map;
};

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned mapa_u32(unsigned a, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
// 16 bytes into another CTA's shared memory, counted on its mbarrier.
__device__ __forceinline__ void st_async16(unsigned addr, uint4 v, unsigned mbar) {
  asm volatile(
      "st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr),
      "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(mbar)
      : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The same in two parts, with work between them.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ bool mbar_test(unsigned bar, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}
// The same, suspended for a while.
__device__ __forceinline__ bool mbar_poll(unsigned bar, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}

__device__ __forceinline__ float mag1(float2 a) { return fabsf(a.x) + fabsf(a.y); }
__device__ __forceinline__ float mag1(double2 a) { return (float)(fabs(a.x) + fabs(a.y)); }
// a - l u and a b in the element's precision
__device__ __forceinline__ float2 nmac(float2 a, float2 l, float2 u) {
  a.x = fmaf(l.y, u.y, fmaf(-l.x, u.x, a.x));
  a.y = fmaf(-l.y, u.x, fmaf(-l.x, u.y, a.y));
  return a;
}
__device__ __forceinline__ double2 nmac(double2 a, double2 l, double2 u) {
  a.x = fma(l.y, u.y, fma(-l.x, u.x, a.x));
  a.y = fma(-l.y, u.x, fma(-l.x, u.y, a.y));
  return a;
}
__device__ __forceinline__ float2 mul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 mul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// 1 / z, zero for a zero z, with |z|^2 near one after a scaling by a power of
// two, its reciprocal by Newton-Raphson from the hardware estimate, and no
// branch, so that the chain overlaps the update.  FP32: |z|^2 and the
// reciprocal as sums of two FP32 numbers (Dekker's double-length arithmetic),
// so the quotients round once (the same in FP64 arithmetic measured 150 cycles
// more per column).
__device__ __forceinline__ float2 recip_of(float2 z) {
  const unsigned e = max(__float_as_uint(z.x) & 0x7f800000u, __float_as_uint(z.y) & 0x7f800000u);
  const float s = __uint_as_float(0x7f000000u - min(e, 0x7e800000u));
  const float x = z.x * s, y = z.y * s;
  const float p = x * x, q = y * y, d = p + q, b = d - p;
  const float lo = (p - (d - b)) + (q - b) + fmaf(x, x, -p) + fmaf(y, y, -q);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  const float rl = r * fmaf(-lo, r, fmaf(-d, r, 1.0f));
  const float xh = x * r, yh = y * r;
  const float qx = xh + (fmaf(x, r, -xh) + x * rl), qy = yh + (fmaf(y, r, -yh) + y * rl);
  return d != 0.0f ? make_float2(qx * s, -qy * s) : make_float2(0.f, 0.f);
}
// FP64: one Newton-Raphson step for the reciprocal from the FP32 estimate of
// |z|^2 (2^-104 at least after the scaling, so in FP32's range), to 2^-45, and
// one step of iterative refinement of the quotients, x / d + (x - q d) / d.
__device__ __forceinline__ double2 recip_of(double2 z) {
  const unsigned e = max((unsigned)__double2hiint(z.x) & 0x7ff00000u, (unsigned)__double2hiint(z.y) & 0x7ff00000u);
  const double s = __hiloint2double((int)(0x7fd00000u - min(e, 0x7fc00000u)), 0);
  const double x = z.x * s, y = z.y * s, d = fma(x, x, y * y);
  float r0;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"((float)d));
  const double r = fma((double)r0, fma(-d, (double)r0, 1.0), (double)r0);
  double qx = x * r, qy = y * r;
  qx = fma(fma(-qx, d, x), r, qx);
  qy = fma(fma(-qy, d, y), r, qy);
  return d != 0.0 ? make_double2(qx * s, -qy * s) : make_double2(0.0, 0.0);
}

// x[r][j] by selects (an indexed access would put the rows in local memory)
template <typename E, int W, int R>
__device__ __forceinline__ E pick_row(const E (&x)[R][W], int r, int j) {
  E v[R];
#pragma unroll
  for (int i = 0; i < R; i++) v[i] = x[i][j];
#pragma unroll
  for (int s = 1; s < R; s *= 2)
#pragma unroll
    for (int i = 0; i + s < R; i += 2 * s)
      if (r & s) v[i] = v[i + s];
  return v[0];
}

// A candidate for one column, the message of a CTA: |re| + |im| of its value
// as float bits plus one (0: no candidate), its row's present position and its
// index before the interchanges, 1 / value and the row.  Candidates compare
// by the FP32 rounding of the magnitude; ties go to the lower CTA, warp, lane
// and row.
template <typename E, int W>
struct __align__(16) PanelMsg {
  unsigned mag;
  unsigned short pos, row;
  E rp;
  alignas(16) E v[W];
};

// One cluster of gridDim.x CTAs of T threads per matrix.  Per subpanel thread t
// of CTA b holds the rows b T R + T r + t, r < R, counted from the subpanel's
// first row (W columns each).  With several subpanels in one launch the rows
// of the next one, and the columns right of it, take the rank-W update of the
// last one as they are loaded, so the cluster keeps its SMs for the whole panel
// (beside a GEMM that would take them between launches).  What other CTAs of
// the cluster wrote is read through L2 after a cluster barrier: that at a
// subpanel's end, and for the columns updated in place one whose two halves
// stand on either side of the subpanel's pivot chain.
template <typename E, int W, int R, int T>
__global__ void __launch_bounds__(T, 1) panel_reg_kernel(RegPanelArgs a) {
  using Msg = PanelMsg<E, W>;
  constexpr int kRegWarps = T / 32;
  constexpr int kMsgChunks = (int)(sizeof(Msg) / 16);
  __shared__ Msg s_in[2][kRegMaxCluster];
  __shared__ Msg s_out[2][kRegWarps];
  __shared__ unsigned s_wmag[2][kRegWarps];
  __shared__ __align__(8) unsigned long long s_bar[2];
  __shared__ E s_l11[W][W + 1];
  __shared__ __align__(16) E s_u[kPanelNb - W][W];
  __shared__ int s_src[W], s_top[W];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, cta = blockIdx.x, CL = gridDim.x;
  const unsigned bar0 = smem_u32(&s_bar[0]), bar1 = smem_u32(&s_bar[1]);
  const unsigned tx = (unsigned)(CL * sizeof(Msg));
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar1) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar0), "r"(tx) : "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar1), "r"(tx) : "memory");
  }
  E *P = reinterpret_cast<E *>(a.A) + blockIdx.y * a.batch_A + a.j0 + a.j0 * a.lda;  // the panel's first entry
  int *ipiv = a.ipiv + blockIdx.y * a.batch_piv + a.j0;
  E x[R][W];
  int pos[R];
  bool act[R];
  int m = 0, top = 0, ph = 0;  // rows of the subpanel; ph: columns exchanged before it
  bool dead = false;
  // every CTA's mbarriers are initialised before any message is sent
  cluster_barrier();
  // where this thread's pieces of a message go (16 bytes each)
  constexpr int kSend = (kRegMaxCluster * kMsgChunks + T - 1) / T;
  unsigned to_msg[kSend], to_bar[kSend];
#pragma unroll
  for (int i = 0; i < kSend; i++) {
    const int q = tid + i * T, t = q / kMsgChunks;
    to_msg[i] = mapa_u32(smem_u32(&s_in[0][cta]) + 16u * (unsigned)(q % kMsgChunks), (unsigned)(t < CL ? t : 0));
    to_bar[i] = mapa_u32(bar0, (unsigned)(t < CL ? t : 0));
  }
  // The candidate of this CTA for column c, whose values are x[.][0]: each
  // warp's best lane leaves its row in shared memory once it is up to date
  // (after `rest`), and after the barrier every thread sends its pieces of the
  // best warp's to the CTAs (one warp writing and sending its row after the
  // barrier measured 3-10% slower).  The rows alternate by column: a warp that
  // has every CTA's message may write the next one while another warp of its
  // CTA still sends its pieces of this one (to other CTAs: nothing here waits
  // for those), and is past the next barrier before it writes the one after.
  auto propose = [&](int c, auto rest) {
    unsigned bm = 0u;
    int bp = pos[0], br = 0;
    E bv = x[0][0];
#pragma unroll
    for (int r = 0; r < R; r++) {
      const unsigned g = __float_as_uint(mag1(x[r][0]));
      const unsigned gm = act[r] && g <= 0x7f800000u ? g + 1u : 0u;  // no NaN
      if (gm > bm) {
        bm = gm;
        bp = pos[r];
        br = r;
        bv = x[r][0];
      }
    }
    const unsigned wm = __reduce_max_sync(0xffffffffu, bm);
    const int best = __ffs(__ballot_sync(0xffffffffu, bm == wm)) - 1;
    const int par = (ph + c) & 1;
    const E brp = recip_of(bv);
    rest();
    if (lane == best) {
      Msg &o = s_out[par][wid];
      s_wmag[par][wid] = wm;
      o.mag = wm;
      o.pos = (unsigned short)bp;
      o.row = (unsigned short)(cta * (T * R) + br * T + tid);
      o.rp = brp;
#pragma unroll
      for (int j = 0; j < W; j++) o.v[j] = pick_row<E, W, R>(x, br, j);
    }
    __syncthreads();
    const unsigned k = s_wmag[par][lane % kRegWarps];
    const unsigned cm = __reduce_max_sync(0xffffffffu, k);
    const uint4 *src = reinterpret_cast<const uint4 *>(&s_out[par][__ffs(__ballot_sync(0xffffffffu, k == cm)) - 1]);
#pragma unroll
    for (int i = 0; i < kSend; i++) {
      const int q = tid + i * T;
      if (q < CL * kMsgChunks && !dead)
        st_async16(to_msg[i] + par * (unsigned)sizeof(s_in[0]), src[q % kMsgChunks], to_bar[i] + 8u * par);
    }
  };
  // Columns c0 .. c1: interchange, update, next candidate.  The first WIN
  // registers of a row rotate: x[.][0] is the current column, the later
  // columns follow, and the multipliers of the columns done since the window
  // began come last; so every column runs the same instructions (a fully
  // unrolled loop of 16 columns spent 40% of its time on instruction fetch).
  auto columns = [&](auto win, int first, int c0, int c1) {
    constexpr int WIN = decltype(win)::value;
#pragma unroll 1
    for (int c = c0; c < c1; c++) {
      // 1. the CTAs' messages of column c: the largest key wins
      const int par = (ph + c) & 1;
      const unsigned bar = par ? bar1 : bar0, phase = (unsigned)((ph + c) >> 1) & 1u;
      //    A wait of more than a.spin polls fails the factorisation, whichever
      //    thread it is, and goes on: every CTA sends its message, so the
      //    exchange stays in step and no phase is armed twice or left behind.
      //    Past the second limit (a message is lost) the thread is dead: it
      //    sends nothing more, which ends the other CTAs' waits in the same
      //    way, and the phase, still armed, is not armed again.
      if (!dead && !mbar_test(bar, phase)) {
        long long it = 0;
        do {
          if (++it == a.spin) atomicExch(a.timeout, 1);
          dead = it - a.spin >= kPanelDrainPolls;
        } while (!dead && !mbar_poll(bar, phase));
      }
      if (tid == 0 && !dead)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(tx) : "memory");
      const unsigned k = lane < CL ? s_in[par][lane].mag : 0u;
      const unsigned g = __reduce_max_sync(0xffffffffu, k);
      const Msg *in = &s_in[par][__ffs(__ballot_sync(0xffffffffu, k == g)) - 1];
      // no candidate at all (every entry NaN): no interchange, a failed pivot
      const bool none = g == 0u;
      int p = none ? c : (int)in->pos;
      if (p < c || p >= m) p = c;  // only in a dead thread
      E rp = {0, 0};
      if (!none) rp = in->rp;
      const bool live = rp.x != 0 || rp.y != 0;
      const int left = W - c;  // columns that are not done, this one included
      // 2. multipliers, and the next column's update
      E l[R], keep[R];
#pragma unroll
      for (int r = 0; r < R; r++) {
        if (pos[r] == p) {
          pos[r] = c;
          act[r] = false;
        } else if (pos[r] == c) {
          pos[r] = p;
        }
        l[r] = mul(x[r][0], rp);
        const bool on = act[r] && live;
        keep[r] = on ? l[r] : x[r][0];
        if (!on) l[r] = E{0, 0};
      }
      // the pivot row by 16-byte broadcasts, zero where a column is done
      constexpr int kPer = 16 / (int)sizeof(E);
      struct alignas(16) Chunk {
        E e[kPer];
      };
      const Chunk *row = reinterpret_cast<const Chunk *>(in->v);
      auto update = [&](int j, E u) {
        if (j >= left) u = E{0, 0};
#pragma unroll
        for (int r = 0; r < R; r++) x[r][j - 1] = nmac(x[r][j], l[r], u);
      };
      update(1, row[1 / kPer].e[1 % kPer]);
      // 3. off the chain: the rest of column c's update, and the records
      auto rest = [&]() {
        if (wid == 0) {
          // the pivot row's own multipliers (row c of L11), by column
          const int q = WIN < W && lane < W - WIN ? WIN + lane : left + lane - c0;
          if (lane < c) s_l11[c][lane] = in->v[q];
          top = top == p ? c : (top == c ? p : top);
          if (lane == 0) {
            s_src[c] = none ? -1 : in->row;
            if (cta == 0) {
              ipiv[first + c] = (int)a.j0 + first + p;
              if (!live) atomicCAS(a.info, 0, (int)a.j0 + first + c + 1);
            }
          }
        }
#pragma unroll
        for (int q = 2 / kPer; q < WIN / kPer; q++) {
          const Chunk u = row[q];
#pragma unroll
          for (int i = 0; i < kPer; i++) update(q * kPer + i, u.e[i]);
        }
#pragma unroll
        for (int r = 0; r < R; r++) x[r][WIN - 1] = keep[r];
      };
      if (c + 1 < W) propose(c + 1, rest);
      else rest();
    }
  };
#pragma unroll 1
  for (int s = a.s0; s < a.s1; s++) {
    const int first = s * W;        // the subpanel's first column and row
    const bool carry = s > a.s0;    // the last subpanel's update is still to do
    E *A = P + first + first * a.lda;
    m = a.m - first;
    top = lane;  // warp 0: the position of the row that began at position `lane`
    if (carry) {
      // U12 of the last subpanel on the columns from here on
      constexpr int kPer = ((kPanelNb - W) * W + T - 1) / T;
      E v[kPer];  // every load in flight before the shared stores
#pragma unroll
      for (int u = 0; u < kPer; u++) {
        const int i = tid + u * T;
        v[u] = E{0, 0};
        if (i < (kPanelNb - first) * W) v[u] = __ldcg(A - W + i % W + (i / W) * a.lda);
      }
#pragma unroll
      for (int u = 0; u < kPer; u++) {
        const int i = tid + u * T;
        if (i < (kPanelNb - first) * W) s_u[i / W][i % W] = v[u];
      }
      __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < R; r++) {
      pos[r] = cta * (T * R) + r * T + tid;
      act[r] = pos[r] < m;
#pragma unroll
      for (int j = 0; j < W; j++) {
        x[r][j] = E{0, 0};
        if (act[r]) x[r][j] = __ldcg(A + pos[r] + j * a.lda);
      }
    }
    if (carry) {
#pragma unroll 1
      for (int r0 = 0; r0 < R; r0++) {
        // one row at a time (its multipliers take W registers); the rows
        // rotate so that every access to x has a fixed index
        const int row = cta * (T * R) + r0 * T + tid;
        const bool on = row < m;
        E l[W];
#pragma unroll
        for (int k = 0; k < W; k++) {
          l[k] = E{0, 0};
          if (on) l[k] = __ldcg(A + row + (k - W) * a.lda);
        }
        E y[W];
#pragma unroll
        for (int j = 0; j < W; j++) y[j] = x[0][j];
#pragma unroll
        for (int j = 0; j < W; j++)
#pragma unroll
          for (int k = 0; k < W; k++) y[j] = nmac(y[j], l[k], s_u[j][k]);
#pragma unroll
        for (int r = 0; r + 1 < R; r++)
#pragma unroll
          for (int j = 0; j < W; j++) x[r][j] = x[r + 1][j];
#pragma unroll
        for (int j = 0; j < W; j++) x[R - 1][j] = y[j];
        // the columns right of this subpanel, in place
#pragma unroll 1
        for (int j0 = W; j0 < kPanelNb - first; j0 += 8) {
#pragma unroll
          for (int j = 0; j < 8; j++) {
            y[j] = E{0, 0};
            if (on) y[j] = __ldcg(A + row + (j0 + j) * a.lda);
          }
#pragma unroll
          for (int j = 0; j < 8; j++)
#pragma unroll
            for (int k = 0; k < W; k++) y[j] = nmac(y[j], l[k], s_u[j0 + j][k]);
#pragma unroll
          for (int j = 0; j < 8; j++)
            if (on) A[row + (j0 + j) * a.lda] = y[j];
        }
      }
      // released here, acquired before step 4, which reads these columns' rows
      // whichever CTA owns them (the messages order nothing but themselves)
      cluster_arrive();
    }
    propose(0, []() {});
    columns(std::integral_constant<int, W>{}, first, 0, W / 2);
    columns(std::integral_constant<int, W / 2>{}, first, W / 2, W);
    ph += W;
    if (wid == 0 && lane < W) s_top[lane] = top;
    // (a CTA with a dead thread stores nothing more, and its row moves are none)
    dead = __syncthreads_or(dead ? 1 : 0) != 0;
    if (s > a.s0) cluster_wait();
    if (dead && a.map && cta == 0 && tid < 2 * W) {
      int *map = a.map + blockIdx.y * a.batch_map + 2 * W * s + tid;
      map[0] = -1;
      map[128] = first;
    }
    if (!dead) {
#pragma unroll
      for (int r = 0; r < R; r++)
#pragma unroll
        for (int j = 0; j < W; j++)
          if (cta * (T * R) + r * T + tid < m) A[pos[r] + ((j + W / 2) % W) * a.lda] = x[r][j];
      // 4. the panel's other columns: the rows the interchanges move (lane i <
      //    W: row i takes the i-th pivot row; lane W + i: the place that the
      //    old row i ended at), and U12 = inv(L11) A12 on the columns to the
      //    right.  One warp per column.
      int from = -1, to = -1;
      if (lane < W) {
        from = s_src[lane];
        to = lane;
        if (from < 0) from = lane;  // failed pivot: no interchange
      } else if (lane < 2 * W && s_top[lane - W] >= W) {
        from = lane - W;
        to = s_top[lane - W];
      }
      if (a.map && cta == 0 && wid == 0 && lane < 2 * W) {
        int *map = a.map + blockIdx.y * a.batch_map + 2 * W * s + lane;
        map[0] = from < 0 ? -1 : first + from;
        map[128] = first + to;
      }
      for (int col = cta * kRegWarps + wid; col < kPanelNb - W; col += CL * kRegWarps) {
        const int cc = col < first ? col : col + W;
        E *q = P + first + (int64_t)cc * a.lda;
        E v = {0, 0};
        if (from >= 0) v = __ldcg(q + from);
        __syncwarp();
        if (cc >= first + W) {
#pragma unroll
          for (int k = 0; k < W - 1; k++) {
            E u;
            u.x = __shfl_sync(0xffffffffu, v.x, k);
            u.y = __shfl_sync(0xffffffffu, v.y, k);
            if (lane > k && lane < W) v = nmac(v, s_l11[lane][k], u);
          }
        }
        if (to >= 0) q[to] = v;
      }
    }
    // every column of the cluster is in place; and no CTA leaves while messages
    // to it can be under way: all have been waited for, or, where a thread is
    // dead, every CTA has spent kPanelDrainPolls since the last was sent
    cluster_barrier();
  }
}

// C (m x nc) -= L (m x W) U (W x nc): the rows below a subpanel on the
// panel's columns to its right (nc <= 64 - W).  Thread per two rows and kRwCols
// columns: the row's W multipliers in registers, U broadcast from shared
// memory.  Bound by the panel's traffic through L2 and the launch.
constexpr int kRwThreads = 128;
constexpr int kRwCols = 8;
template <typename E, int W>
__global__ void __launch_bounds__(kRwThreads) rank_w_kernel(const E *L, const E *U, E *C, int64_t lda, int m,
                                                            int64_t batch) {
  L += blockIdx.z * batch;
  U += blockIdx.z * batch;
  C += blockIdx.z * batch;
  __shared__ __align__(16) E su[kRwCols][W];
  const int j0 = blockIdx.y * kRwCols;
  for (int i = threadIdx.x; i < kRwCols * W; i += kRwThreads) su[i / W][i % W] = U[i % W + (j0 + i / W) * lda];
  const int i0 = blockIdx.x * (2 * kRwThreads) + threadIdx.x, i1 = i0 + kRwThreads;
  const bool v0 = i0 < m, v1 = i1 < m;
  E l0[W], l1[W];
#pragma unroll
  for (int k = 0; k < W; k++) {
    l0[k] = v0 ? L[i0 + k * lda] : E{0, 0};
    l1[k] = v1 ? L[i1 + k * lda] : E{0, 0};
  }
  E c0[kRwCols], c1[kRwCols];
#pragma unroll
  for (int j = 0; j < kRwCols; j++) {
    c0[j] = v0 ? C[i0 + (j0 + j) * lda] : E{0, 0};
    c1[j] = v1 ? C[i1 + (j0 + j) * lda] : E{0, 0};
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kRwCols; j++) {
#pragma unroll
    for (int k = 0; k < W; k++) {
      const E u = su[j][k];
      c0[j] = nmac(c0[j], l0[k], u);
      c1[j] = nmac(c1[j], l1[k], u);
    }
    if (v0) C[i0 + (j0 + j) * lda] = c0[j];
    if (v1) C[i1 + (j0 + j) * lda] = c1[j];
  }
}

// The interchanges of a panel, and U12 = inv(L11) A12, on columns outside it.
// Four lanes share a column, eight columns per warp: lane g holds the rows 4 i +
// g of the column's top 64.  The interchanges are gathers (each top row loads
// its source; the old top rows that leave are stored where they end).  The
// substitution with the unit lower L11 (staged in shared memory) goes four rows
// at a time: the four rows among the four lanes by shuffles, then every row
// below takes their four products.  The registers rotate by one row per step, so
// the loop body is the same 15 guarded row updates.  Columns left of the panel
// are only interchanged, and with them the vector that records the row order.
// Bound by the latency of its chain (loads, map, sixteen steps): 17 us in FP64,
// 13 us in FP32 under ncu, whatever the number of columns up to 3,840.  Before, a map kernel, an interchange
// kernel, the inverse of L11, a GEMM with it and a copy took about 45 us.
constexpr int kStThreads = 128, kStTile = kStThreads / 4;  // columns per CTA

template <typename E>
struct SwapTrsmArgs {
  E *A;
  int64_t lda, j0;
  int entries;              // map entries per subpanel: 2 W
  const int *map;           // [2][128], or null: no interchanges
  int *moves;               // or null: the composed moves, dst[128], src[128], count
  int64_t r0, r1;           // columns right of the panel: interchange and solve
  int64_t l0, l1;           // columns left of it: interchange
  int *perm;                // or null
  int64_t batch_A, batch_piv, batch_map;
};
constexpr int kStLd = kPanelNb + 1;  // row stride of the staged L11
template <typename E>
constexpr size_t swap_trsm_smem() {
  return sizeof(E) * kPanelNb * kStLd;
}

template <typename E>
__global__ void __launch_bounds__(kStThreads) swap_trsm_kernel(SwapTrsmArgs<E> a) {
  extern __shared__ __align__(16) unsigned char st_smem[];
  E *s_l = reinterpret_cast<E *>(st_smem);  // [row][k]
  __shared__ int2 s_map[128];               // (from, to) of the subpanels' moves
  __shared__ int s_src[kPanelNb];           // source of each top row
  __shared__ int2 s_out[128];               // old top rows that leave: (from, to)
  __shared__ int s_nout;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  E *A = a.A + blockIdx.y * a.batch_A + a.j0;
  const int64_t tr = (a.r1 - a.r0 + kStTile - 1) / kStTile;  // tiles of the right side come first
  const bool right = (int64_t)blockIdx.x < tr;
  if (right) {
    // sixteen loads in flight per thread before the shared stores
    for (int i0 = tid; i0 < kPanelNb * kPanelNb; i0 += 16 * kStThreads) {
      E v[16];
#pragma unroll
      for (int u = 0; u < 16; u++) {
        const int i = i0 + u * kStThreads;
        v[u] = A[i % kPanelNb + (a.j0 + i / kPanelNb) * a.lda];
      }
#pragma unroll
      for (int u = 0; u < 16; u++) {
        const int i = i0 + u * kStThreads;
        s_l[(i % kPanelNb) * kStLd + i / kPanelNb] = v[u];
      }
    }
  }
  if (tid < kPanelNb) s_src[tid] = tid;
  if (tid == 0) s_nout = 0;
  if (a.map) {
    const int *map = a.map + blockIdx.y * a.batch_map;
    s_map[tid] = make_int2(map[tid], map[128 + tid]);
    __syncthreads();
    // entry -> the row that its destination holds after every subpanel's
    // moves: follow the moves backwards; the last subpanel that moves a row to
    // a destination speaks for it
    const int sub = tid / a.entries, to = s_map[tid].y;
    int from = -1;
    if (s_map[tid].x >= 0) {
      from = to;
      for (int s = 128 / a.entries - 1; s >= 0; s--) {
        int hit = -1;
#pragma unroll 8
        for (int e = 0; e < a.entries; e++) {
          const int2 v = s_map[s * a.entries + e];
          if (v.x >= 0 && v.y == from) hit = v.x;
        }
        if (hit >= 0) {
          if (s > sub && from == to) {
            from = -1;
            break;
          }
          from = hit;
        }
      }
    }
    if (from >= 0 && from != to) {
      if (to < kPanelNb) s_src[to] = from;
      else s_out[atomicAdd(&s_nout, 1)] = make_int2(from, to);
    }
  }
  __syncthreads();
  const int nout = s_nout;
  if (blockIdx.x == gridDim.x - 1) {
    // by the last CTA: the row order, and the composed moves
    if (a.perm) {
      int *perm = a.perm + blockIdx.y * a.batch_piv + a.j0;
      int v = 0, o = 0;
      if (tid < kPanelNb) v = perm[s_src[tid]];
      if (tid < nout) o = perm[s_out[tid].x];
      __syncthreads();
      if (tid < kPanelNb) perm[tid] = v;
      if (tid < nout) perm[s_out[tid].y] = o;
    }
    if (a.moves) {
      const bool moved = tid < kPanelNb && s_src[tid] != tid;
      if (tid < nout) {
        a.moves[tid] = (int)a.j0 + s_out[tid].y;
        a.moves[128 + tid] = (int)a.j0 + s_out[tid].x;
      }
      __shared__ int s_cnt;
      if (tid == 0) s_cnt = nout;
      __syncthreads();
      if (moved) {
        const int at = atomicAdd(&s_cnt, 1);
        a.moves[at] = (int)a.j0 + tid;
        a.moves[128 + at] = (int)a.j0 + s_src[tid];
      }
      __syncthreads();
      if (tid == 0) a.moves[256] = s_cnt;
    }
  }
  const int64_t tile = right ? blockIdx.x : (int64_t)blockIdx.x - tr;
  const int64_t col = (right ? a.r0 : a.l0) + tile * kStTile + wid * 8 + lane / 4, end = right ? a.r1 : a.l1;
  const int g = lane & 3;
  const bool on = col < end;
  E *q = A + (on ? col : 0) * a.lda;
  E x[16];
#pragma unroll
  for (int i = 0; i < 16; i++) {
    x[i] = E{0, 0};
    const int src = s_src[4 * i + g];
    if (on && (right || src != 4 * i + g)) x[i] = q[src];
  }
  // The column's four lanes read rows that another of them stores below; the
  // loop's own barrier is not reached when no row leaves (the last panel).
  __syncwarp();
  // the rows that leave: all loads of a column before its stores
  for (int o0 = 0; o0 < nout; o0 += 64) {
    E v[16];
#pragma unroll
    for (int i = 0; i < 16; i++) {
      const int e = o0 + 4 * i + g;
      v[i] = E{0, 0};
      if (on && e < nout) v[i] = q[s_out[e].x];
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 16; i++) {
      const int e = o0 + 4 * i + g;
      if (on && e < nout) q[s_out[e].y] = v[i];
    }
  }
  if (!right) {
#pragma unroll
    for (int i = 0; i < 16; i++)
      if (on && s_src[4 * i + g] != 4 * i + g) q[4 * i + g] = x[i];
    return;
  }
#pragma unroll 1
  for (int b = 0; b < 16; b++) {
    // rows 4 b .. 4 b + 3, x[0] of the four lanes
    const E *l = s_l + (4 * b + g) * kStLd + 4 * b;
    E u[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      u[k].x = __shfl_sync(0xffffffffu, x[0].x, (lane & ~3) + k);
      u[k].y = __shfl_sync(0xffffffffu, x[0].y, (lane & ~3) + k);
      if (k < 3 && g > k) x[0] = nmac(x[0], l[k], u[k]);
    }
    if (on) q[4 * b + g] = x[0];
    // the rows below, five at a time (one by one under their own guards they
    // would wait for each other); past the end a row reads the
    // last row of L11 and is not used
#pragma unroll
    for (int h = 1; h < 16; h += 5)
      if (h < 16 - b) {
#pragma unroll
        for (int i = h; i < h + 5; i++) {
          const E *li = s_l + min(4 * (b + i) + g, kPanelNb - 1) * kStLd + 4 * b;
          E y = x[i];
#pragma unroll
          for (int k = 0; k < 4; k++) y = nmac(y, li[k], u[k]);
          x[i - 1] = y;
        }
      }
  }
}

template <typename E, int W, int R, int T>
int launch_reg(Ctx *c, const RegPanelArgs &a, int batch, cudaStream_t st) {
  // (CTAs without rows still share the work on the other columns: 64 rows on
  // one CTA take 78 us per panel, on eight 64 us)
  int CL = std::min(8, c->panel_cluster);
  while ((int64_t)T * R * CL < a.m - a.s0 * W) CL *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(CL, batch);
  cfg.blockDim = dim3(T);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CL;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  MOM_CUDA(c, cudaLaunchKernelEx(&cfg, panel_reg_kernel<E, W, R, T>, a));
  c->launches++;
  return MOM_OK;
}

// Rows a subpanel can have on one CTA, W = 16 and W = 8: what 256 threads hold
// in 128 registers each.
template <typename E> constexpr int kRows16 = sizeof(E) == 8 ? 1024 : 512;
template <typename E> constexpr int kRows8 = 2 * kRows16<E>;

// The kernel for a subpanel of a.m rows, on the largest cluster (measured, one
// 64-column panel at 4,096 rows: 8 CTAs 83 us, 16 CTAs 74 us in FP32; 117 and
// 102 us in FP64).  Few rows per thread while the cluster has room: one row on
// 128 threads (FP32 at 2,048 rows 66 us against 72 us on 256 threads, FP64 86
// against 94).  At two rows per 128 threads the broadcasts of the pivot row
// serve two rows each, which wins in FP32 (4,096 rows: 74 against 76 us), and
// in FP64, bound by its arithmetic, 256 threads win (102 against 105 us).
template <typename E>
int launch_sub(Ctx *c, int W, const RegPanelArgs &a, int batch, cudaStream_t st) {
  const int64_t rows = (a.m - a.s0 * W + c->panel_cluster - 1) / c->panel_cluster;  // per CTA of the largest cluster
  if constexpr (sizeof(E) == 8) {
    if (W == 8) return launch_reg<E, 8, 8, 256>(c, a, batch, st);
    if (rows <= 128) return launch_reg<E, 16, 1, 128>(c, a, batch, st);
    if (rows <= 256) return launch_reg<E, 16, 2, 128>(c, a, batch, st);
    if (rows <= 512) return launch_reg<E, 16, 2, 256>(c, a, batch, st);
    return launch_reg<E, 16, 4, 256>(c, a, batch, st);
  } else {
    if (W == 8) return launch_reg<E, 8, 4, 256>(c, a, batch, st);
    if (rows <= 128) return launch_reg<E, 16, 1, 128>(c, a, batch, st);
    if (rows <= 256) return launch_reg<E, 16, 1, 256>(c, a, batch, st);
    return launch_reg<E, 16, 2, 256>(c, a, batch, st);
  }
}

template <typename E, int W>
int factor_panel(Ctx *c, const PanelCall<E> &p, bool one_launch) {
  RegPanelArgs a;
  a.A = p.A;
  a.lda = p.lda;
  a.j0 = p.j0;
  a.m = (int)(p.n - p.j0);
  a.ipiv = p.ipiv;
  a.info = p.info;
  a.timeout = p.timeout;
  a.spin = wait_polls(c, 0);
  a.map = p.map;
  a.batch_A = p.batch_A;
  a.batch_piv = p.batch_piv;
  a.batch_map = p.batch_map;
  constexpr int kSub = kPanelNb / W;
  if (one_launch) {
    a.s0 = 0;
    a.s1 = kSub;
    return launch_sub<E>(c, W, a, p.batch, p.st);
  }
  for (int s = 0; s < kSub; s++) {
    a.s0 = s;
    a.s1 = s + 1;
    MOM_TRY(launch_sub<E>(c, W, a, p.batch, p.st));
    const int64_t c0 = p.j0 + s * W;
    const int nc = kPanelNb - (s + 1) * W, below = (int)(p.n - c0) - W;
    if (nc > 0 && below > 0) {
      const dim3 grid((below + 2 * kRwThreads - 1) / (2 * kRwThreads), nc / kRwCols, p.batch);
      E *L = p.A + (c0 + W) + c0 * p.lda, *U = p.A + c0 + (c0 + W) * p.lda, *C = U + W;
      rank_w_kernel<E, W><<<grid, kRwThreads, 0, p.st>>>(L, U, C, p.lda, below, p.batch_A);
      c->launches++;
      MOM_CUDA(c, cudaGetLastError());
    }
  }
  return MOM_OK;
}

template <typename E, int W, int R, int T>
bool allow_large_cluster() {
  return cudaFuncSetAttribute(panel_reg_kernel<E, W, R, T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
         cudaSuccess;
}

}  // namespace

// Largest cluster (a power of two) that the device schedules; 0 when it has
// none.  Asked once per context for the kernel that needs most of an SM.
int panel_reg_max_cluster() {
  int most = kRegMaxCluster;
  if (!(allow_large_cluster<float2, 16, 1, 128>() && allow_large_cluster<float2, 16, 2, 128>() &&
        allow_large_cluster<float2, 16, 2, 256>() && allow_large_cluster<float2, 16, 4, 256>() &&
        allow_large_cluster<float2, 8, 8, 256>() && allow_large_cluster<double2, 16, 1, 128>() &&
        allow_large_cluster<double2, 16, 1, 256>() && allow_large_cluster<double2, 16, 2, 256>() &&
        allow_large_cluster<double2, 8, 4, 256>())) {
    cudaGetLastError();
    most = 8;
  }
  for (int cl = most; cl >= 2; cl /= 2) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cl);
    cfg.blockDim = dim3(256);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cl;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int got = 0;
    if (cudaOccupancyMaxActiveClusters(&got, panel_reg_kernel<float2, 16, 4, 256>, &cfg) == cudaSuccess && got >= 1)
      return cl;
    cudaGetLastError();
  }
  return 0;
}

int64_t panel_reg_rows(const Ctx *c, bool f32) {
  return (int64_t)(f32 ? kRows8<float2> : kRows8<double2>) * c->panel_cluster;
}

// 16 columns at a time while the rows fit.  One launch for the panel if
// one_launch says so (the caller runs something else beside it).  Alone, four
// launches with the rank-16 updates on every SM between them are faster on tall
// panels (16,384 rows FP32: 110 against 147 us, 4,096 rows 73 against 93 us, FP64
// 104 against 112 us; no difference up to 1,024 rows).
template <typename E>
int panel_reg(Ctx *c, const PanelCall<E> &p, bool one_launch) {
  if (p.n - p.j0 <= (int64_t)kRows16<E> * c->panel_cluster) return factor_panel<E, 16>(c, p, one_launch);
  return factor_panel<E, 8>(c, p, one_launch);
}
template int panel_reg<float2>(Ctx *, const PanelCall<float2> &, bool);
template int panel_reg<double2>(Ctx *, const PanelCall<double2> &, bool);

template <typename E>
int swap_trsm(Ctx *c, const PanelCall<E> &p, int64_t r0, int64_t r1, int64_t l0, int64_t l1, int *perm, int *moves) {
  SwapTrsmArgs<E> a;
  a.A = p.A;
  a.lda = p.lda;
  a.j0 = p.j0;
  a.entries = p.n - p.j0 <= (int64_t)kRows16<E> * c->panel_cluster ? 32 : 16;
  a.map = p.map;
  a.r0 = r0;
  a.r1 = std::max(r0, r1);
  a.l0 = l0;
  a.l1 = std::max(l0, l1);
  a.perm = perm;
  a.moves = moves;
  a.batch_A = p.batch_A;
  a.batch_piv = p.batch_piv;
  a.batch_map = p.batch_map;
  const int64_t tiles = (a.r1 - a.r0 + kStTile - 1) / kStTile + (a.l1 - a.l0 + kStTile - 1) / kStTile;
  if (tiles == 0 && !perm && !moves) return MOM_OK;
  swap_trsm_kernel<E><<<dim3((unsigned)std::max<int64_t>(1, tiles), p.batch), kStThreads, swap_trsm_smem<E>(), p.st>>>(a);
  c->launches++;
  MOM_CUDA(c, cudaGetLastError());
  return MOM_OK;
}
template int swap_trsm<float2>(Ctx *, const PanelCall<float2> &, int64_t, int64_t, int64_t, int64_t, int *, int *);
template int swap_trsm<double2>(Ctx *, const PanelCall<double2> &, int64_t, int64_t, int64_t, int64_t, int *, int *);

int panel_init_kernels(Ctx *c) {
  MOM_CUDA(c, cudaFuncSetAttribute(swap_trsm_kernel<float2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)swap_trsm_smem<float2>()));
  MOM_CUDA(c, cudaFuncSetAttribute(swap_trsm_kernel<double2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)swap_trsm_smem<double2>()));
  return MOM_OK;
}

}  // namespace mom
