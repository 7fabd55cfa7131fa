// d(lambda^T A x) / d(permittivity) of one domain (no counterpart in the
// reference).  Included by assemble.cu after adjoint_impl.cuh and
// nfields_impl.cuh (complex helpers).
//
// The permittivity moves only k, c2 and Zsi, and d/dk of the kernels is simple:
// dG/dk = i e^{ikR} / (4 pi), dphi/dk = k e^{ikR} / (4 pi R).  So the derivative
// of a face pair's nine entries is linear in the sums of two kernels,
//   B: e^{ikR},  A: e^{ikR} / R,
// over the point pairs, times 1, rho, rho', rho . rho' and (A) rho x rho', rho
// and rho' being the points from their faces' centroids: 19 complex sums,
// which serve every objective, contracted with its weights lambda_r x_c (or the
// dense W) edge pair by edge pair.  A far pair is evaluated once for both its
// blocks: the derivatives are the same, so their weights add.  Near pairs, one
// order at a time, use the smoothed kernels (K's on its own) and the assembly's
// closed-form terms (near_static).

namespace {

struct AdjEpsArgs {
  int F, no;              // faces, objectives (1 with W)
  int tests;              // test faces per far CTA
  int64_t n, N;
  const double *qrel, *cp, *mu, *sl;  // assembly geometry
  const int *hpar;
  const unsigned *near_bits;
  int64_t nnear;
  const int *near_m, *near_n;
  const double *near_static;
  Cd k, c1, c2, Z;        // and their derivatives along eps (c1 has none)
  Cd dk, dc2, dZ;
  const double2 *lam, *xv;  // [no][n], or W
  const double2 *W;         // [n][n] column-major
  double2 *part;            // [CTA][no], the near CTAs after the far ones
};

constexpr int kEpsThreads = 128;
constexpr int kEpsTests = 8;  // most test faces per CTA
constexpr int kEpsWaves = 2;

// Sums of a kernel over a face pair's points, times 1, rho, rho', rho . rho'.
struct EpsSums {
  Cd one, r[3], s[3], rs;
};
__device__ __forceinline__ void eps_zero(EpsSums &o) {
  o.one = o.rs = Cd{0, 0};
#pragma unroll
  for (int i = 0; i < 3; i++) o.r[i] = o.s[i] = Cd{0, 0};
}
// real vector dot complex vector
__device__ __forceinline__ Cd rdot(const double *a, const Cd *b) {
  return {a[0] * b[0].re + a[1] * b[1].re + a[2] * b[2].re, a[0] * b[0].im + a[1] * b[1].im + a[2] * b[2].im};
}
// sum of a w into o, w into the point's weight times 1, rho, rho'
__device__ __forceinline__ void eps_point(EpsSums &o, double w, const double *rho, Cd one, const Cd *s) {
  const Cd t = rdot(rho, s);
  o.one = {fma(w, one.re, o.one.re), fma(w, one.im, o.one.im)};
  o.rs = {fma(w, t.re, o.rs.re), fma(w, t.im, o.rs.im)};
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const double wr = w * rho[i];
    o.r[i] = {fma(wr, one.re, o.r[i].re), fma(wr, one.im, o.r[i].im)};
    o.s[i] = {fma(w, s[i].re, o.s[i].re), fma(w, s[i].im, o.s[i].im)};
  }
}
__device__ __forceinline__ void eps_add(double w, Cd v, double x, double y, double z, Cd &one, Cd *s) {
  v = csc(v, w);
  one = cadd(one, v);
  s[0] = {fma(v.re, x, s[0].re), fma(v.im, x, s[0].im)};
  s[1] = {fma(v.re, y, s[1].re), fma(v.im, y, s[1].im)};
  s[2] = {fma(v.re, z, s[2].re), fma(v.im, z, s[2].im)};
}

// The sums over the point pairs of faces m (points qm: those of the lane) and n
// (points qn, sn apart per coordinate), d apart; X: of rho x rho' times K's
// kernel, which is A's unless NEAR.
template <int NQ, bool NEAR, int LANES>
__device__ __forceinline__ void eps_points(const AdjEpsArgs &a, const double *d, const double *qm, const double *qn,
                                           int sn, int lane, EpsSums &B, EpsSums &A, EpsSums &K, Cd *X) {
  eps_zero(B);
  eps_zero(A);
  eps_zero(K);
#pragma unroll
  for (int i = 0; i < 3; i++) X[i] = Cd{0, 0};
  const Cd k2 = cmul(a.k, a.k), z0 = {0, 0};
#pragma unroll 1
  for (int t = lane; t < NQ; t += LANES) {
    const double rho[3] = {qm[3 * t], qm[3 * t + 1], qm[3 * t + 2]};
    const double r[3] = {d[0] + rho[0], d[1] + rho[1], d[2] + rho[2]};
    Cd b0 = z0, a0 = z0, k0 = z0, b1[3] = {z0, z0, z0}, a1[3] = {z0, z0, z0}, k1[3] = {z0, z0, z0};
#pragma unroll 1
    for (int s = 0; s < NQ; s++) {
      const double x = qn[3 * s * sn], y = qn[(3 * s + 1) * sn], z = qn[(3 * s + 2) * sn];
      const double D[3] = {r[0] - x, r[1] - y, r[2] - z};
      const double R2 = D[0] * D[0] + D[1] * D[1] + D[2] * D[2];
      double iR = 0, R = 0;
      Cd e = {1.0, 0.0};
      if (R2 > 0) {
        iR = ::rsqrt(R2);
        R = R2 * iR;
        double si, cs;
        ::sincos(a.k.re * R, &si, &cs);
        const double ea = ::exp(-a.k.im * R);
        e = {ea * cs, ea * si};
      }
      const double ws = c_qw[s];
      if (NEAR) {
        // Gs = (e - 1)/R + k^2 R / 2 (ik at R = 0), dGs/dk = i (e - i k R), dphis/dk = k (e - 1)/R
        const Cd e1 = {(e.re - 1.0) * iR, e.im * iR};
        const Cd gs = R2 > 0 ? Cd{e1.re + 0.5 * k2.re * R, e1.im + 0.5 * k2.im * R} : Cd{-a.k.im, a.k.re};
        eps_add(ws, Cd{e.re + a.k.im * R, e.im - a.k.re * R}, x, y, z, b0, b1);
        eps_add(ws, gs, x, y, z, a0, a1);
        eps_add(ws, e1, x, y, z, k0, k1);
      } else {
        eps_add(ws, e, x, y, z, b0, b1);
        eps_add(ws, csc(e, iR), x, y, z, a0, a1);
      }
    }
    const double wt = c_qw[t];
    eps_point(B, wt, rho, b0, b1);
    eps_point(A, wt, rho, a0, a1);
    if (NEAR) eps_point(K, wt, rho, k0, k1);
    const Cd *x1 = NEAR ? k1 : a1;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const int j = (i + 1) % 3, l = (i + 2) % 3;
      X[i] = {fma(wt, rho[j] * x1[l].re - rho[l] * x1[j].re, X[i].re),
              fma(wt, rho[j] * x1[l].im - rho[l] * x1[j].im, X[i].im)};
    }
  }
}

// Adds the pair's derivatives, contracted with each objective's weights, to
// acc: the block (test m, source n), without NEAR also (test n, source m).
// Edge pairs i of the nine with i % LANES == lane.
template <bool NEAR, int LANES>
__device__ __forceinline__ void eps_contract(const AdjEpsArgs &a, int m, int n, const double *d, int64_t j, int lane,
                                             const EpsSums &B, const EpsSums &A, const EpsSums &K, const Cd *X,
                                             Cd *acc) {
  const int64_t N = a.N, ld = a.n;
  const Cd i1 = {0.0, 1.0};
  const Cd fB = cmul(cmul(i1, a.dk), csc(a.c1, 0.25)), fA = cmul(a.dZ, csc(a.c1, 0.25)),
           fK = csc(cmul(a.k, a.dk), 0.25);
  const Cd hB = cmul(cmul(i1, a.dk), a.c2), hA = cmul(a.dZ, a.c2);
  const Cd hd = cfma(hB, B.one, cmul(a.dc2, A.one));
  const double f4 = 1.0 / (4.0 * kPi);
  const Cd f8 = csc(cmul(a.k, a.k), 1.0 / (8.0 * kPi)), df8 = csc(cmul(a.k, a.dk), 2.0 / (8.0 * kPi));
#pragma unroll 1
  for (int i = lane; i < 9; i += LANES) {
    const int p = i / 3, q = i % 3;
    const int64_t r = a.hpar[3 * m + p], c = a.hpar[3 * n + q];
    const double s = a.sl[3 * m + p] * a.sl[3 * n + q] * kOofpi;
    const double *u = a.mu + 9 * (size_t)m + 3 * p, *v = a.mu + 9 * (size_t)n + 3 * q;
    const double uv = u[0] * v[0] + u[1] * v[1] + u[2] * v[2];
    // (rho - u) . (rho' - v)
    auto dots = [&](const EpsSums &o) {
      const Cd t = csub(csub(o.rs, rdot(u, o.s)), rdot(v, o.r));
      return Cd{fma(uv, o.one.re, t.re), fma(uv, o.one.im, t.im)};
    };
    const Cd cb = cfma(fB, dots(B), hd);
    Cd cjj = csc(cb, s), cmm = csc(cfma(a.Z, cb, cfma(fA, dots(A), cmul(hA, A.one))), s), ck = {0, 0};
    if (!NEAR || m != n) {
      // D . ((rho' - v) x (rho - u)) by the sums: rho x rho' . (v - u - d),
      // rho . (v x u - d x v), -rho' . (v x u + u x d), d . (v x u)
      const EpsSums &o = NEAR ? K : A;
      double vu[3], gx[3], gr[3], gs[3];
#pragma unroll
      for (int e = 0; e < 3; e++) {
        const int f = (e + 1) % 3, g = (e + 2) % 3;
        vu[e] = v[f] * u[g] - v[g] * u[f];
        gx[e] = v[e] - u[e] - d[e];
        gr[e] = vu[e] - (d[f] * v[g] - d[g] * v[f]);
        gs[e] = -(vu[e] + (u[f] * d[g] - u[g] * d[f]));
      }
      const double go = d[0] * vu[0] + d[1] * vu[1] + d[2] * vu[2];
      const Cd t = cadd(cadd(rdot(gx, X), rdot(gr, o.r)), rdot(gs, o.s));
      ck = csc(cmul(fK, Cd{fma(go, o.one.re, t.re), fma(go, o.one.im, t.im)}), s);
    }
    if (NEAR) {
      const double *st = a.near_static + j * 54;
      const Cd Dt = {f4 * st[i] - f8.re * st[9 + i], -f8.im * st[9 + i]};
      const Cd Ht = {f4 * st[18 + i] - f8.re * st[27 + i], -f8.im * st[27 + i]};
      const Cd S = cfma(a.c1, Dt, cmul(a.c2, Ht));
      // dS = -c1 f8' D1 + c2' H - c2 f8' H1
      const Cd dS = csub(cmul(a.dc2, Ht), cmul(df8, cadd(csc(a.c1, st[9 + i]), csc(a.c2, st[27 + i]))));
      cjj = cadd(cjj, dS);
      cmm = cadd(cmm, cfma(a.dZ, S, cmul(a.Z, dS)));
      ck = csub(ck, csc(df8, st[45 + i]));
    }
    if (a.W) {
      Cd wjj = ld_c(a.W + r + c * ld), wmm = ld_c(a.W + (r + N) + (c + N) * ld);
      Cd wk = csub(ld_c(a.W + (r + N) + c * ld), ld_c(a.W + r + (c + N) * ld));
      if (!NEAR) {
        wjj = cadd(wjj, ld_c(a.W + c + r * ld));
        wmm = cadd(wmm, ld_c(a.W + (c + N) + (r + N) * ld));
        wk = cadd(wk, csub(ld_c(a.W + (c + N) + r * ld), ld_c(a.W + c + (r + N) * ld)));
      }
      acc[0] = cfma(ck, wk, cfma(cmm, wmm, cfma(cjj, wjj, acc[0])));
      continue;
    }
#pragma unroll 1
    for (int o = 0; o < a.no; o++) {
      const double2 *l = a.lam + o * ld, *x = a.xv + o * ld;
      const Cd lj = ld_c(l + r), lm = ld_c(l + r + N), xj = ld_c(x + c), xm = ld_c(x + c + N);
      Cd wjj = cmul(lj, xj), wmm = cmul(lm, xm), wk = csub(cmul(lm, xj), cmul(lj, xm));
      if (!NEAR) {
        const Cd kj = ld_c(l + c), km = ld_c(l + c + N), yj = ld_c(x + r), ym = ld_c(x + r + N);
        wjj = cfma(kj, yj, wjj);
        wmm = cfma(km, ym, wmm);
        wk = cfms(kj, ym, cfma(km, yj, wk));
      }
      acc[o] = cfma(ck, wk, cfma(cmm, wmm, cfma(cjj, wjj, acc[o])));
    }
  }
}

__device__ __forceinline__ void eps_block_sum(int no, const Cd *acc, double2 *out) {
  __shared__ double2 red[kEpsThreads];
  for (int o = 0; o < no; o++) {
    __syncthreads();
    red[threadIdx.x] = make_double2(acc[o].re, acc[o].im);
    __syncthreads();
    for (int w = kEpsThreads / 2; w > 0; w >>= 1) {
      if (threadIdx.x < w) {
        red[threadIdx.x].x += red[threadIdx.x + w].x;
        red[threadIdx.x].y += red[threadIdx.x + w].y;
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) out[o] = red[0];
  }
}

// Far pairs m < n: thread per n, a.tests test faces per CTA.  Bound by FP64
// latency, most of it in the kernels of the 169 point pairs, so they are taken
// once for all objectives: the whole call with four sources (eight objectives)
// over 1,280 faces takes 4.75 ms, with forms per objective and a pass for each
// 18.7, with dual numbers in the moments 17.6.  The points of the CTA's faces n
// wait in shared memory, since lanes would read them 39 doubles apart otherwise.
template <int NQ>
__global__ void __launch_bounds__(kEpsThreads) adj_eps_far_kernel(AdjEpsArgs a) {
  __shared__ double s_q[3 * NQ][kEpsThreads];
  const int n0 = blockIdx.x * kEpsThreads, n = n0 + threadIdx.x, m0 = blockIdx.y * a.tests;
  Cd acc[kAdjMaxObj];
  for (int o = 0; o < a.no; o++) acc[o] = Cd{0, 0};
  if (m0 < n0 + kEpsThreads) {  // some pair has m < n
    for (int i = threadIdx.x; i < 3 * NQ * kEpsThreads; i += kEpsThreads) {
      const int f = i / (3 * NQ);
      if (n0 + f < a.F) s_q[i % (3 * NQ)][f] = a.qrel[(size_t)n0 * 3 * NQ + i];
    }
    __syncthreads();
#pragma unroll 1
    for (int m = m0; m < min(a.F, m0 + a.tests); m++) {
      if (n >= a.F || m >= n) continue;
      const int64_t bit = (int64_t)m * a.F + n;
      if ((a.near_bits[bit >> 5] >> (bit & 31)) & 1u) continue;
      const double d[3] = {a.cp[3 * m] - a.cp[3 * n], a.cp[3 * m + 1] - a.cp[3 * n + 1], a.cp[3 * m + 2] - a.cp[3 * n + 2]};
      EpsSums B, A, K;
      Cd X[3];
      eps_points<NQ, false, 1>(a, d, a.qrel + (size_t)m * 3 * NQ, &s_q[0][threadIdx.x], kEpsThreads, 0, B, A, K, X);
      eps_contract<false, 1>(a, m, n, d, 0, 0, B, A, K, X, acc);
    }
  }
  eps_block_sum(a.no, acc, a.part + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * a.no);
}

// Near pairs in each order: smoothed quadrature and closed-form terms, LANES
// threads per pair with every LANES-th test point and edge pair each.
template <int NQ, int LANES>
__global__ void __launch_bounds__(kEpsThreads) adj_eps_near_kernel(AdjEpsArgs a) {
  const int64_t idx = (int64_t)blockIdx.x * kEpsThreads + threadIdx.x;
  const int lane = (int)(idx % LANES);
  const bool live = idx / LANES < a.nnear;
  const int64_t j = live ? idx / LANES : 0;
  Cd acc[kAdjMaxObj];
  for (int o = 0; o < a.no; o++) acc[o] = Cd{0, 0};
  const int m = a.near_m[j], n = a.near_n[j];
  const double d[3] = {a.cp[3 * m] - a.cp[3 * n], a.cp[3 * m + 1] - a.cp[3 * n + 1], a.cp[3 * m + 2] - a.cp[3 * n + 2]};
  struct {
    EpsSums B, A, K;
    Cd X[3];
  } s;
  eps_points<NQ, true, LANES>(a, d, a.qrel + (size_t)m * 3 * NQ, a.qrel + (size_t)n * 3 * NQ, 1, lane, s.B, s.A, s.K, s.X);
  if (LANES > 1) {
    double *v = reinterpret_cast<double *>(&s);
#pragma unroll
    for (int i = 0; i < (int)(sizeof(s) / sizeof(double)); i++)
#pragma unroll
      for (int w = 1; w < LANES; w *= 2) v[i] += __shfl_xor_sync(0xffffffffu, v[i], w);
  }
  if (live) eps_contract<true, LANES>(a, m, n, d, j, lane, s.B, s.A, s.K, s.X, acc);
  eps_block_sum(a.no, acc, a.part + (size_t)blockIdx.x * a.no);
}

template <int NQ>
void launch_adj_eps(const dim3 &far, unsigned near, int lanes, cudaStream_t s, AdjEpsArgs a) {
  adj_eps_far_kernel<NQ><<<far, kEpsThreads, 0, s>>>(a);
  a.part += (size_t)far.x * far.y * a.no;
  if (!near) return;
  if (lanes > 1) adj_eps_near_kernel<NQ, 4><<<near, kEpsThreads, 0, s>>>(a);
  else adj_eps_near_kernel<NQ, 1><<<near, kEpsThreads, 0, s>>>(a);
}

}  // namespace
