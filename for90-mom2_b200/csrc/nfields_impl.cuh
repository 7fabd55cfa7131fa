// Scattered near fields of a domain's surface currents at arbitrary points
// (scat_fields, nfields.f90:29-49, with scat_fields_frags 109-197, identity
// group).  Included once, at the end of assemble.cu, so that the field
// kernel shares the closed-form static integrals (point_static) and the
// quadrature weights (c_qw) of the assembly (inside namespace mom).
//
// For point r and source face f with the RWG functions f_q = c_q (r' - p_q)
// (c_q = s_q l_q / (2 A_f), div f_q = s_q l_q / A_f) the fields need
//   K2_q = int G f_q,  K3_q = int grad'G div'f_q,  K4_q = int grad'G x f_q
// (intK2, intK3, intK4 of srcint.f90 with no test face), and with
// c1 = i w mu0, c2 = 1/(i w eps0 n^2)
//   E += x_J (c1 K2 + c2 K3) + x_M K4,   H += x_M (K2/c2 + K3/c1) - x_J K4.
// The coefficients x go in first: the face's current is the affine field
// (a rho' + b) / A of the point rho' from the centroid, so with D0 from the
// centroid to r, D = D0 - rho', grad'G = D phi / (4 pi),
// phi = e^{ikR} (1/R^3 - ik/R^2), the sums
//   g0 = sum w g,  s1 = sum w g rho',  p0 = sum w phi,  t1 = sum w phi rho'
// and p1 = sum w phi D = p0 D0 - t1 give every source's (A-free, times 1/(4 pi))
//   K2 = b g0 + a s1,  K3 = 2 a p1,  K4 = p1 x b + a D0 x t1.
// No term grows with the distance.  (In the current extended to r,
// X^ = a D0 + b, K2 = X^ g0 - a sum w g D and K4 = p1 x X^: terms of the
// distance over the face's size cancel, five digits at 1 cm from faces of 15 nm.)
// Within three average edge lengths of the face centroid the smoothed kernels
// are used and the closed-form parts (1/(4 pi)) X_m1 - (k^2/(8 pi)) X_1 are
// added, as in the reference.

namespace {

__device__ __forceinline__ Cd cadd(Cd a, Cd b) { return {a.re + b.re, a.im + b.im}; }
__device__ __forceinline__ Cd csub(Cd a, Cd b) { return {a.re - b.re, a.im - b.im}; }
__device__ __forceinline__ Cd csc(Cd a, double s) { return {a.re * s, a.im * s}; }
__host__ __device__ __forceinline__ Cd cdivd(Cd a, Cd b) {
  const double d = b.re * b.re + b.im * b.im;
  return {(a.re * b.re + a.im * b.im) / d, (a.im * b.re - a.re * b.im) / d};
}
// acc + a b, acc - a b
__device__ __forceinline__ Cd cfma(Cd a, Cd b, Cd acc) {
  return {fma(a.re, b.re, fma(-a.im, b.im, acc.re)), fma(a.re, b.im, fma(a.im, b.re, acc.im))};
}
__device__ __forceinline__ Cd cfms(Cd a, Cd b, Cd acc) {
  return {fma(-a.re, b.re, fma(a.im, b.im, acc.re)), fma(-a.re, b.im, fma(-a.im, b.re, acc.im))};
}
struct Cv {
  Cd x, y, z;
};
__device__ __forceinline__ Cv cvcross(const Cv &a, const Cv &b) {
  const Cd o = {0, 0};
  return {cfms(a.z, b.y, cfma(a.y, b.z, o)), cfms(a.x, b.z, cfma(a.z, b.x, o)), cfms(a.y, b.x, cfma(a.x, b.y, o))};
}
// real vector times complex vector
__device__ __forceinline__ Cv rvcross(const double *a, const Cv &b) {
  return {{fma(a[1], b.z.re, -a[2] * b.y.re), fma(a[1], b.z.im, -a[2] * b.y.im)},
          {fma(a[2], b.x.re, -a[0] * b.z.re), fma(a[2], b.x.im, -a[0] * b.z.im)},
          {fma(a[0], b.y.re, -a[1] * b.x.re), fma(a[0], b.y.im, -a[1] * b.x.im)}};
}
__device__ __forceinline__ Cv cvadd(const Cv &a, const Cv &b) { return {cadd(a.x, b.x), cadd(a.y, b.y), cadd(a.z, b.z)}; }
__device__ __forceinline__ Cv cvsub(const Cv &a, const Cv &b) { return {csub(a.x, b.x), csub(a.y, b.y), csub(a.z, b.z)}; }
__device__ __forceinline__ Cv cvscale(Cd s, const Cv &a) { return {cmul(s, a.x), cmul(s, a.y), cmul(s, a.z)}; }
// a D + b
__device__ __forceinline__ Cv affine(Cd a, const double *D, const Cv &b) {
  return {{fma(a.re, D[0], b.x.re), fma(a.im, D[0], b.x.im)},
          {fma(a.re, D[1], b.y.re), fma(a.im, D[1], b.y.im)},
          {fma(a.re, D[2], b.z.re), fma(a.im, D[2], b.z.im)}};
}
__device__ __forceinline__ Cd ld_c(const double2 *p) {
  const double2 v = *p;
  return {v.x, v.y};
}
__device__ __forceinline__ Cv ld_v(const double2 *p) { return {ld_c(p), ld_c(p + 1), ld_c(p + 2)}; }

// The affine current of face f about its centroid, of the J (h = 0) or M half of
// vector v: a = sum_p v_p sl_p / 2, b = -sum_p v_p sl_p mu_p / 2 into o[4] = a, b.
__device__ __forceinline__ void face_current(int f, int h, int N, const int *hpar, const double *sl, const double *mu,
                                             const double2 *v, double2 *o) {
  Cd a = {0, 0}, b[3] = {{0, 0}, {0, 0}, {0, 0}};
#pragma unroll
  for (int p = 0; p < 3; p++) {
    const double2 c = v[hpar[3 * f + p] + (h ? N : 0)];
    const double s = 0.5 * sl[3 * f + p];
    a.re += s * c.x;
    a.im += s * c.y;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const double t = s * mu[9 * (size_t)f + 3 * p + i];
      b[i].re -= t * c.x;
      b[i].im -= t * c.y;
    }
  }
  o[0] = make_double2(a.re, a.im);
#pragma unroll
  for (int i = 0; i < 3; i++) o[1 + i] = make_double2(b[i].re, b[i].im);
}

// Those of every face and of the vectors v + s ldv, s = blockIdx.y:
// coef[s][F][8] = aJ, bJ[3], aM, bM[3].
__global__ void face_current_kernel(int F, int N, const int *hpar, const double *sl, const double *mu,
                                    const double2 *v, int64_t ldv, double2 *coef) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= F) return;
  v += (size_t)blockIdx.y * ldv;
  for (int h = 0; h < 2; h++)
    face_current(f, h, N, hpar, sl, mu, v, coef + 8 * ((size_t)blockIdx.y * F + f) + 4 * h);
}

constexpr int kNfThreads = 128;
constexpr int kNfTile = 8;  // faces staged at a time

struct NfArgs {
  int F;
  const double *qrel;    // [F][NQ][3] minus the centroid
  const double *cp;      // [F][3]
  const double *area;    // [F]
  const FaceGeo *geo;    // [F]
  int N;
  const int *hpar;
  const double *sl, *mu;
  const double2 *x;      // the launch's solutions, ldx apart
  int64_t ldx;
  double thr2;           // (3 avelen)^2
  double kr, ki;         // k = ri w / c0
  Cd k2;                 // k^2
  Cd c1, c2, ic1, ic2;   // i w mu0, 1 / (i w eps0 n^2), and their reciprocals
  int nsrc;              // sources in this launch (<= NS)
  const double *pts;     // [npts][3]
  int npts, per_split;   // faces per split (blockIdx.y)
  double2 *part;         // [split][nsrc][npts][6]: E, H
};

// The closed-form parts of face n at r for the currents cur of ns sources,
// added to E, H (times 4 pi: the caller scales the sums).
__device__ __noinline__ void nfield_static(const NfArgs &a, const double *r, const double *D0, int n,
                                           const double2 *cur, int ns, Cv *E, Cv *H) {
  PointStatic<double> ps;
  point_static(r, a.geo[n], ps);
  const double iA = 1.0 / a.area[n];
  const double f4 = 1.0 / (4.0 * kPi) / kOofpi;
  const Cd f8 = {a.k2.re / (8.0 * kPi) / kOofpi, a.k2.im / (8.0 * kPi) / kOofpi};
  const Cd y0 = {f4 * ps.Sm1 - f8.re * ps.S1, -f8.im * ps.S1};
  Cd gr[3], l[3];
  double rc[3];
#pragma unroll
  for (int i = 0; i < 3; i++) {
    gr[i] = {iA * (f4 * ps.K3m1[i] - f8.re * ps.K31[i]), -iA * f8.im * ps.K31[i]};
    l[i] = {f4 * ps.mL1[i] - f8.re * ps.mL3[i] / 3.0, -f8.im * ps.mL3[i] / 3.0};
    rc[i] = ps.rho[i] - a.cp[3 * n + i];
  }
  const Cv P = {gr[0], gr[1], gr[2]}, Lv = {l[0], l[1], l[2]};
#pragma unroll 1
  for (int s = 0; s < ns; s++) {
    const double2 *c = cur + 8 * s;
    const Cd aJ = ld_c(c), aM = ld_c(c + 4), z = {iA, 0};
    const Cv bJ = ld_v(c + 1), bM = ld_v(c + 5);
    // int (a r' + b) / A over R and R: a (mL + rho S) + b S
    const Cv yJ = cvscale(z, cvadd(cvscale(aJ, Lv), cvscale(y0, affine(aJ, rc, bJ))));
    const Cv yM = cvscale(z, cvadd(cvscale(aM, Lv), cvscale(y0, affine(aM, rc, bM))));
    E[s] = cvadd(E[s], cvsub(cvadd(cvscale(a.c1, yJ), cvscale(csc(cmul(a.c2, aJ), 2.0), P)),
                             cvcross(affine(aM, D0, bM), P)));
    H[s] = cvadd(H[s], cvadd(cvadd(cvscale(a.ic2, yM), cvscale(csc(cmul(a.ic1, aM), 2.0), P)),
                             cvcross(affine(aJ, D0, bJ), P)));
  }
}

// One thread per point over the faces of its split, staged in shared memory
// in tiles (broadcast reads; neighbouring points share their near faces, so
// warps seldom diverge).  FP64-pipe bound, about 90 instructions per point and
// quadrature point; a 101 x 101 plane over 1,280 faces with one CTA per point
// and the three RWG functions of a face apart took 3.7 ms.
template <int NQ, int NS, bool LOSSLESS>
__global__ void __launch_bounds__(kNfThreads) nfield_kernel(NfArgs a) {
  constexpr int kCoef = 16 * NS, kFace = (kCoef + 3 + 3 * NQ + 1) / 2 * 2;
  __shared__ __align__(16) double s_face[kNfTile][kFace];
  const int ip = blockIdx.x * kNfThreads + threadIdx.x;
  const bool valid = ip < a.npts;
  double r[3];
#pragma unroll
  for (int i = 0; i < 3; i++) r[i] = valid ? a.pts[3 * (size_t)ip + i] : 0.0;
  Cv E[NS], H[NS];
  const Cd z0 = {0, 0};
#pragma unroll
  for (int s = 0; s < NS; s++) E[s] = H[s] = Cv{z0, z0, z0};
  const int n0 = blockIdx.y * a.per_split, n1 = min(a.F, n0 + a.per_split);
  for (int base = n0; base < n1; base += kNfTile) {
    const int cnt = min(kNfTile, n1 - base);
    __syncthreads();
    for (int e = threadIdx.x; e < cnt * 2 * NS; e += kNfThreads) {
      const int f = e / (2 * NS), s = e / 2 % NS, h = e % 2;
      double2 *o = reinterpret_cast<double2 *>(s_face[f]) + 8 * s + 4 * h;
      if (s < a.nsrc) face_current(base + f, h, a.N, a.hpar, a.sl, a.mu, a.x + s * a.ldx, o);
      else
        for (int i = 0; i < 4; i++) o[i] = make_double2(0, 0);
    }
    for (int e = threadIdx.x; e < cnt * (3 + 3 * NQ); e += kNfThreads) {
      const int f = e / (3 + 3 * NQ), k = e % (3 + 3 * NQ), n = base + f;
      s_face[f][kCoef + k] = k < 3 ? a.cp[3 * n + k] : a.qrel[(size_t)n * NQ * 3 + k - 3];
    }
    __syncthreads();
    if (!valid) continue;
#pragma unroll 1
    for (int f = 0; f < cnt; f++) {
      const double *fc = s_face[f], *fcp = fc + kCoef, *fq = fcp + 3;
      const double D0[3] = {r[0] - fcp[0], r[1] - fcp[1], r[2] - fcp[2]};
      const bool near = D0[0] * D0[0] + D0[1] * D0[1] + D0[2] * D0[2] < a.thr2;
      Cd g0 = z0, p0 = z0, s1[3] = {z0, z0, z0}, t1[3] = {z0, z0, z0};
#pragma unroll 1
      for (int j = 0; j < NQ; j++) {
        const double *q = fq + 3 * j;
        const double D[3] = {D0[0] - q[0], D0[1] - q[1], D0[2] - q[2]};
        const double R2 = D[0] * D[0] + D[1] * D[1] + D[2] * D[2], w = c_qw[j];
        Cd g, p;
        if (R2 > 0) {
          const double iR = ::rsqrt(R2), R = R2 * iR;
          double sn, cs;
          ::sincos(a.kr * R, &sn, &cs);
          const double ea = LOSSLESS ? 1.0 : ::exp(-a.ki * R);
          const double er = ea * cs, ei = ea * sn, iR2 = iR * iR, iR3 = iR2 * iR;
          const double qr = iR3 + a.ki * iR2, qi = -a.kr * iR2;  // 1/R^3 - i k / R^2
          g = {er * iR, ei * iR};
          p = {er * qr - ei * qi, er * qi + ei * qr};
          if (near) {  // green.f90 vGs / vgradGs: (e - 1)/R + k^2 R / 2, e q - 1/R^3 - k^2/(2R)
            g = {(er - 1.0) * iR + 0.5 * a.k2.re * R, ei * iR + 0.5 * a.k2.im * R};
            p = {p.re - iR3 - 0.5 * a.k2.re * iR, p.im - 0.5 * a.k2.im * iR};
          }
        } else {  // R = 0: Gs = i k / (4 pi), grad Gs = 0
          g = near ? Cd{-a.ki, a.kr} : z0;
          p = z0;
        }
        g = csc(g, w);
        p = csc(p, w);
        g0 = cadd(g0, g);
        p0 = cadd(p0, p);
#pragma unroll
        for (int i = 0; i < 3; i++) {
          s1[i] = {fma(g.re, q[i], s1[i].re), fma(g.im, q[i], s1[i].im)};
          t1[i] = {fma(p.re, q[i], t1[i].re), fma(p.im, q[i], t1[i].im)};
        }
      }
      const Cv S1 = {s1[0], s1[1], s1[2]}, T1 = {t1[0], t1[1], t1[2]}, P1 = cvsub(affine(p0, D0, Cv{z0, z0, z0}), T1);
      const Cv DT = rvcross(D0, T1);
#pragma unroll
      for (int s = 0; s < NS; s++) {
        const double2 *c = reinterpret_cast<const double2 *>(fc + 16 * s);
        const Cd aJ = ld_c(c), aM = ld_c(c + 4);
        const Cv bJ = ld_v(c + 1), bM = ld_v(c + 5);
        const Cv uj = cvadd(cvscale(g0, bJ), cvscale(aJ, S1)), um = cvadd(cvscale(g0, bM), cvscale(aM, S1));
        const Cv kj = cvadd(cvcross(P1, bJ), cvscale(aJ, DT)), km = cvadd(cvcross(P1, bM), cvscale(aM, DT));
        E[s] = cvadd(E[s], cvadd(cvadd(cvscale(a.c1, uj), cvscale(csc(cmul(a.c2, aJ), 2.0), P1)), km));
        H[s] = cvadd(H[s], cvsub(cvadd(cvscale(a.ic2, um), cvscale(csc(cmul(a.ic1, aM), 2.0), P1)), kj));
      }
      if (near) nfield_static(a, r, D0, base + f, reinterpret_cast<const double2 *>(fc), min(NS, a.nsrc), E, H);
    }
  }
  if (!valid) return;
#pragma unroll
  for (int s = 0; s < NS; s++) {
    if (s >= a.nsrc) break;
    double2 *o = a.part + (((size_t)blockIdx.y * a.nsrc + s) * a.npts + ip) * 6;
    const Cd v[6] = {E[s].x, E[s].y, E[s].z, H[s].x, H[s].y, H[s].z};
#pragma unroll
    for (int i = 0; i < 6; i++) o[i] = make_double2(kOofpi * v[i].re, kOofpi * v[i].im);
  }
}

// E, H [nsrc][npts][3]: the splits' parts, LANES threads per value with every
// LANES-th split each, added up in a fixed order.
template <int LANES>
__global__ void nfield_sum_kernel(int npts, int nsrc, int splits, const double2 *part, double2 *E, double2 *H) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, e = idx / LANES;
  const int lane = (int)(idx % LANES);
  const int64_t per = (int64_t)nsrc * npts * 6;
  double2 v = make_double2(0, 0);
  for (int s = lane; s < splits && e < per; s += LANES) {
    const double2 p = part[s * per + e];
    v.x += p.x;
    v.y += p.y;
  }
#pragma unroll
  for (int w = 1; w < LANES; w *= 2) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, w);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, w);
  }
  if (e >= per || lane != 0) return;
  const int64_t at = e / 6;
  const int i = (int)(e % 6);
  (i < 3 ? E : H)[at * 3 + i % 3] = v;
}

template <int NQ, bool LOSSLESS>
void launch_nfield_k(int ns, const dim3 &grid, cudaStream_t st, const NfArgs &a) {
  if (ns == 1) nfield_kernel<NQ, 1, LOSSLESS><<<grid, kNfThreads, 0, st>>>(a);
  else if (ns == 2) nfield_kernel<NQ, 2, LOSSLESS><<<grid, kNfThreads, 0, st>>>(a);
  else nfield_kernel<NQ, 4, LOSSLESS><<<grid, kNfThreads, 0, st>>>(a);
}
template <int NQ>
void launch_nfield(int ns, const dim3 &grid, cudaStream_t st, const NfArgs &a) {
  if (a.ki == 0.0) launch_nfield_k<NQ, true>(ns, grid, st, a);
  else launch_nfield_k<NQ, false>(ns, grid, st, a);
}

}  // namespace

// Face geometry of domain d for the field kernel (uploaded once per geometry).
static int nfield_geometry(Ctx *c, DomDev &D) {
  if (D.nf_geo) return MOM_OK;
  const int F = D.F;
  std::vector<FaceGeo> geo(F);
  for (int f = 0; f < F; f++) {
    FaceGeo &g = geo[f];
    for (int k = 0; k < 3; k++)
      for (int i = 0; i < 3; i++) {
        g.v[k][i] = D.h_fv[9 * (size_t)f + 3 * k + i];
        g.s[k][i] = D.h_fs[9 * (size_t)f + 3 * k + i];
        g.mm[k][i] = D.h_fm[9 * (size_t)f + 3 * k + i];
      }
    for (int i = 0; i < 3; i++) g.n[i] = D.h_nrm[3 * (size_t)f + i];
  }
  void *pg = nullptr;
  if (cudaMalloc(&pg, sizeof(FaceGeo) * F) != cudaSuccess) {
    cudaGetLastError();
    return fail(c, MOM_ERR_ALLOC, "near-field geometry allocation failed");
  }
  D.nf_geo = pg;
  MOM_CUDA(c, cudaMemcpyAsync(pg, geo.data(), sizeof(FaceGeo) * F, cudaMemcpyHostToDevice, c->stream));
  return MOM_OK;
}

int scat_fields(Ctx *c, int d, double omega, const double *ri, int nsrc, const double2 *X, int64_t ldx, int npts,
                const double *pts, double2 *E, double2 *H) {
  if (d < 0 || d >= c->ndom) return fail(c, MOM_ERR_ARG, "domain index out of range");
  DomDev &D = c->dom[d];
  MOM_TRY(nfield_geometry(c, D));
  const int F = D.F;
  // Faces per split: eight CTAs per SM in all, down to one face each, since a
  // split's faces are a serial chain (8 us per near face with 13 points).
  const int blocks = (npts + kNfThreads - 1) / kNfThreads;
  const int want = std::max(1, std::min(F, 8 * c->nsm / blocks));
  const int per = (F + want - 1) / want, splits = (F + per - 1) / per;
  MOM_TRY(ensure_buffer(c, &c->adj_part, &c->adj_part_bytes,
                        sizeof(double2) * 6 * (size_t)npts * std::min(nsrc, 4) * splits));
  const double k0 = omega / kC0;
  NfArgs a;
  a.F = F;
  a.qrel = D.qrel;
  a.cp = D.cp;
  a.area = D.area;
  a.geo = reinterpret_cast<const FaceGeo *>(D.nf_geo);
  a.thr2 = (D.avelen * 3) * (D.avelen * 3);
  a.kr = ri[0] * k0;
  a.ki = ri[1] * k0;
  a.k2 = {a.kr * a.kr - a.ki * a.ki, 2 * a.kr * a.ki};
  a.c1 = {0.0, omega * kMu0};
  const Cd n2 = {ri[0] * ri[0] - ri[1] * ri[1], 2 * ri[0] * ri[1]};
  const Cd den = {-omega * kEps0 * n2.im, omega * kEps0 * n2.re};  // i w eps0 n^2
  a.c2 = cdivd({1.0, 0.0}, den);
  a.ic1 = cdivd({1.0, 0.0}, a.c1);
  a.ic2 = den;
  a.pts = pts;
  a.npts = npts;
  a.per_split = per;
  a.part = (double2 *)c->adj_part;
  a.N = c->N;
  a.hpar = D.hpar;
  a.sl = D.sl;
  a.mu = D.mu;
  a.ldx = ldx;
  for (int s0 = 0; s0 < nsrc; s0 += 4) {
    const int ns = std::min(4, nsrc - s0);
    a.nsrc = ns;
    a.x = X + (size_t)s0 * ldx;
    const int nl = ns == 1 ? 1 : (ns == 2 ? 2 : 4);
    const dim3 grid(blocks, splits);
    switch (c->nq) {
      case 1: launch_nfield<1>(nl, grid, c->stream, a); break;
      case 3: launch_nfield<3>(nl, grid, c->stream, a); break;
      case 4: launch_nfield<4>(nl, grid, c->stream, a); break;
      case 7: launch_nfield<7>(nl, grid, c->stream, a); break;
      case 13: launch_nfield<13>(nl, grid, c->stream, a); break;
      default: return fail(c, MOM_ERR_ARG, "unsupported number of quadrature points");
    }
    const int64_t vals = (int64_t)ns * npts * 6;
    double2 *Eo = E + (size_t)s0 * npts * 3, *Ho = H + (size_t)s0 * npts * 3;
    if (splits > 16)  // few points (eight CTAs per SM at most: under 10,000)
      nfield_sum_kernel<32><<<(unsigned)((vals * 32 + 255) / 256), 256, 0, c->stream>>>(npts, ns, splits, a.part, Eo, Ho);
    else
      nfield_sum_kernel<1><<<(unsigned)((vals + 255) / 256), 256, 0, c->stream>>>(npts, ns, splits, a.part, Eo, Ho);
    c->launches += 2;
    MOM_CUDA(c, cudaGetLastError());
  }
  return MOM_OK;
}
