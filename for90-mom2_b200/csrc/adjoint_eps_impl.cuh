// d(lambda^T A x) / d(permittivity) of one domain (no counterpart in the
// reference).  Included by assemble.cu after adjoint_impl.cuh and
// nfields_impl.cuh (complex helpers).
//
// The permittivity moves only k, c2 and Zsi, and d/dk of the kernels is simple:
// dG/dk = i e^{ikR} / (4 pi), dphi/dk = k e^{ikR} / (4 pi R).  So with the pair's
// weights w_JJ.. (lambda_r x_c, or the dense W) folded into bilinear forms of
// the two points first, a point pair contributes
//   B(rho, rho') e^{ikR} + A(rho, rho') e^{ikR} / R,
// B and A affine in rho' for each test point: two complex numbers and two
// forms instead of 18 dual moments and their contraction.  A far pair is
// evaluated once for both its blocks: their forms in (rho, rho') are the same,
// so their weights add.  Near pairs, one order at a time, use the smoothed
// kernels and the assembly's closed-form terms (near_static).

namespace {

struct AdjEpsArgs {
  int F;
  int64_t n, N;
  const double *qrel, *cp, *mu, *sl;  // assembly geometry
  const int *hpar;
  const unsigned *near_bits;
  int64_t nnear;
  const int *near_m, *near_n;
  const double *near_static;
  Cd k, c1, c2, Z;        // and their derivatives along eps (c1 has none)
  Cd dk, dc2, dZ;
  const double2 *lam, *xv;  // one objective, or W
  const double2 *W;         // [n][n] column-major
  double2 *part;            // far: [gridDim.y][gridDim.x]; near: the blocks after them
};

constexpr int kEpsThreads = 128;
constexpr int kEpsTests = 8;  // test faces per CTA

// The forms of one face pair: sum_pq of the weights times (rho - u_p).(rho' -
// v_q) (c0, u, v, uv), and for K times D.((rho' - v_q) x (rho - u_p)) (x: the sum
// of v x u); hB, hA: the divergence terms.
struct EpsForms {
  Cd B0, Bu[3], Bv[3], Buv, A0, Au[3], Av[3], Auv, K0, Ku[3], Kv[3], Kx[3];
};

// Adds block (test m, source n): weights w(r, c) on its 3 x 3 edge pairs, p on
// face f1 (forms' first face), q on face f2; flip: the block's test face is f2.
__device__ __forceinline__ void eps_forms(const AdjEpsArgs &a, int f1, int f2, bool flip, bool self, EpsForms &o) {
  const int64_t N = a.N, ld = a.n;
  const Cd i1 = {0.0, 1.0};
  const Cd fB = cmul(cmul(i1, a.dk), csc(a.c1, 0.25)), fA = cmul(a.dZ, csc(a.c1, 0.25)),
           fK = csc(cmul(a.k, a.dk), 0.25);
  const Cd hB = cmul(cmul(i1, a.dk), a.c2), hA2 = cmul(a.dZ, a.c2);
  const Cd z0 = {0, 0};
#pragma unroll 1
  for (int p = 0; p < 3; p++) {
    const int64_t r = a.hpar[3 * f1 + p];
    const double s1 = a.sl[3 * f1 + p];
    const double *u = a.mu + 9 * (size_t)f1 + 3 * p;
#pragma unroll 1
    for (int q = 0; q < 3; q++) {
      const int64_t c = a.hpar[3 * f2 + q];
      const double s = s1 * a.sl[3 * f2 + q];
      const double *v = a.mu + 9 * (size_t)f2 + 3 * q;
      const int64_t tr = flip ? c : r, tc = flip ? r : c;
      Cd wjj, wmm, wk;
      if (a.W) {
        wjj = ld_c(a.W + tr + tc * ld);
        wmm = ld_c(a.W + (tr + N) + (tc + N) * ld);
        wk = csub(ld_c(a.W + (tr + N) + tc * ld), ld_c(a.W + tr + (tc + N) * ld));
      } else {
        const Cd lj = ld_c(a.lam + tr), lm = ld_c(a.lam + tr + N), xj = ld_c(a.xv + tc), xm = ld_c(a.xv + tc + N);
        wjj = cmul(lj, xj);
        wmm = cmul(lm, xm);
        wk = csub(cmul(lm, xj), cmul(lj, xm));
      }
      const Cd w1 = csc(cfma(a.Z, wmm, wjj), s), w2 = csc(wmm, s);
      const Cd oB = cmul(fB, w1), oA = cmul(fA, w2), oK = self ? z0 : cmul(fK, csc(wk, s));
      const double uv = u[0] * v[0] + u[1] * v[1] + u[2] * v[2];
      o.B0 = cadd(o.B0, oB);
      o.A0 = cadd(o.A0, oA);
      o.K0 = cadd(o.K0, oK);
      // the divergence terms join the constants
      o.Buv = cadd(o.Buv, cfma(hB, w1, csc(oB, uv)));
      o.Auv = cadd(o.Auv, cfma(hA2, w2, cfma(a.dc2, w1, csc(oA, uv))));
      const double x[3] = {v[1] * u[2] - v[2] * u[1], v[2] * u[0] - v[0] * u[2], v[0] * u[1] - v[1] * u[0]};
#pragma unroll
      for (int i = 0; i < 3; i++) {
        o.Bu[i] = cadd(o.Bu[i], csc(oB, u[i]));
        o.Bv[i] = cadd(o.Bv[i], csc(oB, v[i]));
        o.Au[i] = cadd(o.Au[i], csc(oA, u[i]));
        o.Av[i] = cadd(o.Av[i], csc(oA, v[i]));
        o.Ku[i] = cadd(o.Ku[i], csc(oK, u[i]));
        o.Kv[i] = cadd(o.Kv[i], csc(oK, v[i]));
        o.Kx[i] = cadd(o.Kx[i], csc(oK, x[i]));
      }
    }
  }
}
__device__ __forceinline__ void eps_zero(EpsForms &o) {
  Cd *p = &o.B0;
#pragma unroll
  for (int i = 0; i < (int)(sizeof(EpsForms) / sizeof(Cd)); i++) p[i] = Cd{0, 0};
}
// real vector cross complex vector, and dot products
__device__ __forceinline__ Cd rdot(const double *a, const Cd *b) {
  return {a[0] * b[0].re + a[1] * b[1].re + a[2] * b[2].re, a[0] * b[0].im + a[1] * b[1].im + a[2] * b[2].im};
}
__device__ __forceinline__ void rcross(const double *a, const Cd *b, Cd *o) {
  o[0] = {a[1] * b[2].re - a[2] * b[1].re, a[1] * b[2].im - a[2] * b[1].im};
  o[1] = {a[2] * b[0].re - a[0] * b[2].re, a[2] * b[0].im - a[0] * b[2].im};
  o[2] = {a[0] * b[1].re - a[1] * b[0].re, a[0] * b[1].im - a[1] * b[0].im};
}

// Sum over the point pairs of faces m (points qm) and n (points qn, sn apart
// per coordinate); NEAR: smoothed kernels, with the K form on its own.
template <int NQ, bool NEAR>
__device__ __forceinline__ Cd eps_points(const AdjEpsArgs &a, int m, int n, const double *qm, const double *qn, int sn,
                                         const EpsForms &o) {
  double d[3];
#pragma unroll
  for (int i = 0; i < 3; i++) d[i] = a.cp[3 * m + i] - a.cp[3 * n + i];
  Cd sum = {0, 0};
  const Cd k2 = cmul(a.k, a.k);
#pragma unroll 1
  for (int t = 0; t < NQ; t++) {
    const double *rt = qm + 3 * t;
    const double rho[3] = {rt[0], rt[1], rt[2]}, r[3] = {d[0] + rho[0], d[1] + rho[1], d[2] + rho[2]};
    // the forms at this test point: constant and coefficient of rho'
    const Cd bc = csub(o.Buv, rdot(rho, o.Bv));
    Cd ac = csub(o.Auv, rdot(rho, o.Av)), bl[3], al[3], kl[3], c1[3], c2[3];
    rcross(r, o.Ku, c1);     // -(Ku x r)
    rcross(rho, o.Kv, c2);   // -(Kv x rho)
    const double rd[3] = {rho[1] * d[2] - rho[2] * d[1], rho[2] * d[0] - rho[0] * d[2], rho[0] * d[1] - rho[1] * d[0]};
    const Cd kc = cadd(rdot(d, c2), rdot(r, o.Kx));
#pragma unroll
    for (int i = 0; i < 3; i++) {
      bl[i] = csub(csc(o.B0, rho[i]), o.Bu[i]);
      al[i] = csub(csc(o.A0, rho[i]), o.Au[i]);
      kl[i] = csub(cadd(csc(o.K0, rd[i]), c1[i]), cadd(c2[i], o.Kx[i]));
    }
    if (!NEAR) {
      ac = cadd(ac, kc);
#pragma unroll
      for (int i = 0; i < 3; i++) al[i] = cadd(al[i], kl[i]);
    }
    Cd st = {0, 0};
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
        double sn, cs;
        ::sincos(a.k.re * R, &sn, &cs);
        const double ea = ::exp(-a.k.im * R);
        e = {ea * cs, ea * sn};
      }
      const Cd fB = {fma(z, bl[2].re, fma(y, bl[1].re, fma(x, bl[0].re, bc.re))),
                     fma(z, bl[2].im, fma(y, bl[1].im, fma(x, bl[0].im, bc.im)))};
      const Cd fA = {fma(z, al[2].re, fma(y, al[1].re, fma(x, al[0].re, ac.re))),
                     fma(z, al[2].im, fma(y, al[1].im, fma(x, al[0].im, ac.im)))};
      Cd v;
      if (NEAR) {
        const Cd fK = {fma(z, kl[2].re, fma(y, kl[1].re, fma(x, kl[0].re, kc.re))),
                       fma(z, kl[2].im, fma(y, kl[1].im, fma(x, kl[0].im, kc.im)))};
        // Gs = (e - 1)/R + k^2 R / 2 (ik at R = 0), dGs/dk = i (e - i k R), dphis/dk = k (e - 1)/R
        const Cd e1 = {(e.re - 1.0) * iR, e.im * iR};
        const Cd gs = R2 > 0 ? Cd{e1.re + 0.5 * k2.re * R, e1.im + 0.5 * k2.im * R} : Cd{-a.k.im, a.k.re};
        v = cfma(fK, e1, cfma(fA, gs, cmul(fB, Cd{e.re + a.k.im * R, e.im - a.k.re * R})));
      } else {
        v = cfma(fA, csc(e, iR), cmul(fB, e));
      }
      const double ws = c_qw[s];
      st = {fma(ws, v.re, st.re), fma(ws, v.im, st.im)};
    }
    const double wt = c_qw[t];
    sum = {fma(wt, st.re, sum.re), fma(wt, st.im, sum.im)};
  }
  return csc(sum, kOofpi);
}

__device__ __forceinline__ void eps_block_sum(Cd acc, double2 *out) {
  __shared__ double2 red[kEpsThreads];
  red[threadIdx.x] = make_double2(acc.re, acc.im);
  __syncthreads();
  for (int w = kEpsThreads / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
      red[threadIdx.x].x += red[threadIdx.x + w].x;
      red[threadIdx.x].y += red[threadIdx.x + w].y;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = red[0];
}

// Far pairs m < n: thread per n, kEpsTests test faces per CTA (8 fill the chip
// from about 700 faces on).  FP64 bound in latency: 43% of the pipe with two
// CTAs of 228 registers per SM; 1.78 ms per objective and domain over 1,280
// faces.  The points of the CTA's faces n wait in shared memory, since lanes
// would read them 39 doubles apart otherwise (2% slower).
template <int NQ>
__global__ void __launch_bounds__(kEpsThreads) adj_eps_far_kernel(AdjEpsArgs a) {
  __shared__ double s_q[3 * NQ][kEpsThreads];
  const int n0 = blockIdx.x * kEpsThreads, n = n0 + threadIdx.x, m0 = blockIdx.y * kEpsTests;
  Cd acc = {0, 0};
  if (m0 < n0 + kEpsThreads) {  // some pair has m < n
    for (int i = threadIdx.x; i < 3 * NQ * kEpsThreads; i += kEpsThreads) {
      const int f = i / (3 * NQ);
      if (n0 + f < a.F) s_q[i % (3 * NQ)][f] = a.qrel[(size_t)n0 * 3 * NQ + i];
    }
    __syncthreads();
#pragma unroll 1
    for (int m = m0; m < min(a.F, m0 + kEpsTests); m++) {
      if (n >= a.F || m >= n) continue;
      const int64_t bit = (int64_t)m * a.F + n;
      if ((a.near_bits[bit >> 5] >> (bit & 31)) & 1u) continue;
      EpsForms o;
      eps_zero(o);
      eps_forms(a, m, n, false, false, o);
      eps_forms(a, m, n, true, false, o);
      acc = cadd(acc, eps_points<NQ, false>(a, m, n, a.qrel + (size_t)m * 3 * NQ, &s_q[0][threadIdx.x], kEpsThreads, o));
    }
  }
  eps_block_sum(acc, a.part + (size_t)blockIdx.y * gridDim.x + blockIdx.x);
}

// Near pairs in each order: smoothed quadrature and closed-form terms.
template <int NQ>
__global__ void __launch_bounds__(kEpsThreads) adj_eps_near_kernel(AdjEpsArgs a) {
  const int64_t j = (int64_t)blockIdx.x * kEpsThreads + threadIdx.x;
  Cd acc = {0, 0};
  if (j < a.nnear) {
    const int m = a.near_m[j], n = a.near_n[j];
    EpsForms o;
    eps_zero(o);
    eps_forms(a, m, n, false, m == n, o);
    acc = eps_points<NQ, true>(a, m, n, a.qrel + (size_t)m * 3 * NQ, a.qrel + (size_t)n * 3 * NQ, 1, o);
    const double *st = a.near_static + j * 54;
    const double f4 = 1.0 / (4.0 * kPi);
    const Cd f8 = csc(cmul(a.k, a.k), 1.0 / (8.0 * kPi)), df8 = csc(cmul(a.k, a.dk), 2.0 / (8.0 * kPi));
#pragma unroll 1
    for (int p = 0; p < 3; p++)
#pragma unroll 1
      for (int q = 0; q < 3; q++) {
        const int64_t r = a.hpar[3 * m + p], c = a.hpar[3 * n + q], N = a.N, ld = a.n;
        Cd wjj, wmm, wk;
        if (a.W) {
          wjj = ld_c(a.W + r + c * ld);
          wmm = ld_c(a.W + (r + N) + (c + N) * ld);
          wk = csub(ld_c(a.W + (r + N) + c * ld), ld_c(a.W + r + (c + N) * ld));
        } else {
          const Cd lj = ld_c(a.lam + r), lm = ld_c(a.lam + r + N), xj = ld_c(a.xv + c), xm = ld_c(a.xv + c + N);
          wjj = cmul(lj, xj);
          wmm = cmul(lm, xm);
          wk = csub(cmul(lm, xj), cmul(lj, xm));
        }
        const int i = 3 * p + q;
        const Cd Dt = {f4 * st[i] - f8.re * st[9 + i], -f8.im * st[9 + i]};
        const Cd Ht = {f4 * st[18 + i] - f8.re * st[27 + i], -f8.im * st[27 + i]};
        const Cd S = cfma(a.c1, Dt, cmul(a.c2, Ht));
        // dS = -c1 f8' D1 + c2' H - c2 f8' H1
        const Cd dS = csub(cmul(a.dc2, Ht), cmul(df8, cadd(csc(a.c1, st[9 + i]), csc(a.c2, st[27 + i]))));
        acc = cfma(wjj, dS, acc);
        acc = cfma(wmm, cfma(a.dZ, S, cmul(a.Z, dS)), acc);
        acc = cfms(wk, csc(df8, st[45 + i]), acc);
      }
  }
  eps_block_sum(acc, a.part + blockIdx.x);
}

template <int NQ>
void launch_adj_eps(const dim3 &far, unsigned near, cudaStream_t s, AdjEpsArgs a) {
  adj_eps_far_kernel<NQ><<<far, kEpsThreads, 0, s>>>(a);
  a.part += (size_t)far.x * far.y;
  if (near) adj_eps_near_kernel<NQ><<<near, kEpsThreads, 0, s>>>(a);
}

}  // namespace
