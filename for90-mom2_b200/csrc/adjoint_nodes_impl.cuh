// d(lambda^T A x) / d(vertex coordinates) in reverse mode (no counterpart in
// the reference).  Included by assemble.cu after adjoint_impl.cuh and
// nfields_impl.cuh (complex vectors, the faces' affine currents).
//
// With the currents of a face written as affine fields, t(r) = a r + b times
// 1 / area for lambda and for x (J and M), the quadrature of every face pair is
// a sum over point pairs (i on the test face, j on the source face)
//   F = sum_ij g [c1 (TJi.XJj + Z TMi.XMj) + c2 (dTJi dXJj + Z dTMi dXMj)]
//             + phi [TMi.(D x XJj) - TJi.(D x XMj)],     D = r_i - r_j,
// with T_i = w_i t(r_i), dT_i = 2 w_i a, likewise X, and g, phi the (smoothed,
// for near pairs) kernels over 4 pi.  F depends on the geometry through the
// points r_i (g, phi, D and T, X themselves), the free vertices and edge
// lengths in a, b.  So one pass over the points and faces gives every
// derivative: for each point i the fields dF/dT_i, dF/dX_i and the force
// dF/dr_i at fixed T, X; then the chain rule per face.  This costs about twice
// an FP64 assembly instead of 18 forward-mode evaluations per face pair.
//
// A source face acts through moments only.  With D0 = r_i - c_n, the field of
// face n extended to r_i is X^ = a D0 + b, X_j = w_j (X^ - a D), and D x D = 0:
//   sum g X_j = g0 X^ - a g1,  sum phi D x X_j = p1 x X^,
//   force = -p1 alpha + p2 gamma + (q2 + p0) B - p1 x eta
// with g0, g1 = sum w g {1, D}; p0, p1, p2 = sum w phi {1, D, D D};
// q2 = sum w psi D D, psi = phi'(R) / R, and alpha, gamma, B, eta bilinear in the
// point's and the face's fields.  20 complex sums per (point, face) serve all
// objectives.
//
// The closed-form integrals of near pairs add (a) their fields to dF/dT_i and
// (b) the derivative in the source face's coordinates, in forward-mode duals
// (nine per near pair and point); the derivative in r_i at fixed T is minus the
// sum over the three vertices, since the integrals move with the face.

namespace {

constexpr int kRevThreads = 128;
constexpr int kRevTile = 8;     // faces staged at a time
constexpr int kRevVals = 43;    // per point and objective: R_i (3), then 20 complex sums

struct RevArgs {
  int F, no;               // faces, objectives of a set (1 or 2, the same x); sets: blockIdx.z
  const double *qrel, *cp;
  const double2 *coef;     // [set][no + 1][F][8]: lambda of each objective, then x: aJ, bJ[3], aM, bM[3]
  const unsigned *near_bits;
  double kr, ki;
  Cd c1, c2, Z;
  int per_split;           // faces per split (blockIdx.y)
  double *part;            // [set][split][no][F NQ][kRevVals], the sets set_part doubles apart
  size_t set_part;
};

__device__ __forceinline__ Cd cvdot(const Cv &a, const Cv &b, Cd acc) {
  return cfma(a.z, b.z, cfma(a.y, b.y, cfma(a.x, b.x, acc)));
}
// symmetric matrix (xx, yy, zz, xy, xz, yz) times a vector
__device__ __forceinline__ Cv symv(const Cd *s, const Cv &v) {
  const Cd o = {0, 0};
  return {cfma(s[4], v.z, cfma(s[3], v.y, cfma(s[0], v.x, o))), cfma(s[5], v.z, cfma(s[1], v.y, cfma(s[3], v.x, o))),
          cfma(s[2], v.z, cfma(s[5], v.y, cfma(s[4], v.x, o)))};
}

// Doubles of shared memory per thread: the point's fields (T of each
// objective, X: J, M vectors and the two divergences) and the sums (dF/dT, dF/dX
// of each objective, forces).
constexpr int rev_slots(int no) { return 16 * (no + 1) + 16 * (no + 1) + 3 * no; }
template <int NQ> constexpr int rev_face_doubles(int no) { return 3 * NQ + 3 + 16 * (no + 1); }
template <int NQ> constexpr size_t rev_smem(int no) {
  return sizeof(double) * ((size_t)rev_slots(no) * kRevThreads + (size_t)kRevTile * (rev_face_doubles<NQ>(no) + 1));
}

// One thread per quadrature point; the faces of the split are staged in
// shared memory in tiles.  FP64-pipe bound: about 170 FP64 instructions per
// point pair for the kernels and sums, a thirteenth of 700 per (point, face).
template <int NQ, int NO>
__global__ void __launch_bounds__(kRevThreads) rev_field_kernel(RevArgs a) {
  extern __shared__ __align__(16) double rev_sm[];
  constexpr int kT = kRevThreads, kFace = (rev_face_doubles<NQ>(NO) + 1) / 2 * 2;
  double *s_own = rev_sm;                                   // [16 (NO + 1)][kT]
  double *s_acc = s_own + 16 * (NO + 1) * kT;               // [16 (NO + 1) + 3 NO][kT]
  double *s_face = s_acc + (16 * (NO + 1) + 3 * NO) * kT;   // [kRevTile][kFace]: coefs, cp, qrel
  const int tid = threadIdx.x;
  const int P = a.F * NQ, i = blockIdx.x * kT + tid;
  a.coef += (size_t)blockIdx.z * (NO + 1) * a.F * 8;
  a.part += blockIdx.z * a.set_part;
  const bool valid = i < P;
  const int m = valid ? i / NQ : 0, t = valid ? i % NQ : 0;
  const double w = c_qw[t];
  const double k2r = a.kr * a.kr - a.ki * a.ki, k2i = 2 * a.kr * a.ki;
  auto own_c = [&](int s, int c) -> Cd {
    return {s_own[(16 * s + 2 * c) * kT + tid], s_own[(16 * s + 2 * c + 1) * kT + tid]};
  };
  auto own_v = [&](int s, int c) -> Cv { return {own_c(s, c), own_c(s, c + 1), own_c(s, c + 2)}; };
  auto add_c = [&](int s, int c, Cd v) {
    s_acc[(16 * s + 2 * c) * kT + tid] += v.re;
    s_acc[(16 * s + 2 * c + 1) * kT + tid] += v.im;
  };
  auto add_v = [&](int s, int c, const Cv &v) {
    add_c(s, c, v.x);
    add_c(s, c + 1, v.y);
    add_c(s, c + 2, v.z);
  };
  // the point's own fields: set s < NO lambda of objective s, s = NO x; per set
  // J (0-2), M (3-5), dJ (6), dM (7)
  double r[3];
#pragma unroll
  for (int k = 0; k < 3; k++) r[k] = a.cp[3 * m + k] + a.qrel[((size_t)m * NQ + t) * 3 + k];
#pragma unroll 1
  for (int s = 0; s <= NO; s++) {
    const double2 *c = a.coef + ((size_t)s * a.F + m) * 8;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const Cd al = ld_c(c + 4 * h);
      const Cv v = affine(al, a.qrel + ((size_t)m * NQ + t) * 3, ld_v(c + 4 * h + 1));
      const Cd o[4] = {v.x, v.y, v.z, {2 * al.re, 2 * al.im}};
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int at = k < 3 ? 3 * h + k : 6 + h;
        s_own[(16 * s + 2 * at) * kT + tid] = w * o[k].re;
        s_own[(16 * s + 2 * at + 1) * kT + tid] = w * o[k].im;
      }
    }
  }
  for (int k = 0; k < 16 * (NO + 1) + 3 * NO; k++) s_acc[k * kT + tid] = 0.0;
  const int n0 = blockIdx.y * a.per_split, n1 = min(a.F, n0 + a.per_split);
  for (int base = n0; base < n1; base += kRevTile) {
    const int cnt = min(kRevTile, n1 - base);
    __syncthreads();
    for (int e = tid; e < cnt * rev_face_doubles<NQ>(NO); e += kT) {
      const int f = e / rev_face_doubles<NQ>(NO), k = e % rev_face_doubles<NQ>(NO);
      const int n = base + f;
      double v;
      if (k < 16 * (NO + 1))
        v = reinterpret_cast<const double *>(a.coef + ((size_t)(k / 16) * a.F + n) * 8)[k % 16];
      else if (k < 16 * (NO + 1) + 3) v = a.cp[3 * n + k - 16 * (NO + 1)];
      else v = a.qrel[(size_t)n * NQ * 3 + k - 16 * (NO + 1) - 3];
      s_face[f * kFace + k] = v;
    }
    __syncthreads();
    if (!valid) continue;
#pragma unroll 1
    for (int f = 0; f < cnt; f++) {
      const int n = base + f;
      const double *fc = s_face + f * kFace, *fcp = fc + 16 * (NO + 1), *fq = fcp + 3;
      const double D0[3] = {r[0] - fcp[0], r[1] - fcp[1], r[2] - fcp[2]};
      const int64_t bit = (int64_t)m * a.F + n;
      const bool near = (a.near_bits[bit >> 5] >> (bit & 31)) & 1u;
      Cd g0 = {0, 0}, g1[3] = {{0, 0}, {0, 0}, {0, 0}}, p0 = {0, 0}, p1[3] = {{0, 0}, {0, 0}, {0, 0}};
      Cd p2[6], q2[6];
#pragma unroll
      for (int k = 0; k < 6; k++) p2[k] = q2[k] = Cd{0, 0};
#pragma unroll 1
      for (int j = 0; j < NQ; j++) {
        const double D[3] = {D0[0] - fq[3 * j], D0[1] - fq[3 * j + 1], D0[2] - fq[3 * j + 2]};
        const double R2 = D[0] * D[0] + D[1] * D[1] + D[2] * D[2];
        const double wj = c_qw[j];
        Cd g, p, q;
        if (R2 > 0) {
          const double iR = ::rsqrt(R2), R = R2 * iR;
          double sn, cs;
          ::sincos(a.kr * R, &sn, &cs);
          const double ea = a.ki == 0.0 ? 1.0 : ::exp(-a.ki * R);
          const Cd e = {ea * cs, ea * sn};
          const double iR2 = iR * iR, iR3 = iR2 * iR, iR4 = iR2 * iR2, iR5 = iR4 * iR;
          g = {e.re * iR, e.im * iR};
          p = cmul(e, Cd{iR3 + a.ki * iR2, -a.kr * iR2});
          // psi = e (-3 / R^5 + 3 i k / R^4 + k^2 / R^3)
          q = cmul(e, Cd{-3 * iR5 - 3 * a.ki * iR4 + k2r * iR3, 3 * a.kr * iR4 + k2i * iR3});
          if (near) {  // the smoothed kernels (green.f90:40-97)
            g = {(e.re - 1.0) * iR + 0.5 * k2r * R, e.im * iR + 0.5 * k2i * R};
            p = {p.re - iR3 - 0.5 * k2r * iR, p.im - 0.5 * k2i * iR};
            q = {q.re + 3 * iR5 + 0.5 * k2r * iR3, q.im + 0.5 * k2i * iR3};
          }
        } else {
          g = near ? Cd{-a.ki, a.kr} : Cd{0, 0};
          p = q = Cd{0, 0};
        }
        g = csc(g, wj);
        p = csc(p, wj);
        q = csc(q, wj);
        const double DD[6] = {D[0] * D[0], D[1] * D[1], D[2] * D[2], D[0] * D[1], D[0] * D[2], D[1] * D[2]};
        g0 = cadd(g0, g);
        p0 = cadd(p0, p);
#pragma unroll
        for (int k = 0; k < 3; k++) {
          g1[k] = {fma(g.re, D[k], g1[k].re), fma(g.im, D[k], g1[k].im)};
          p1[k] = {fma(p.re, D[k], p1[k].re), fma(p.im, D[k], p1[k].im)};
        }
#pragma unroll
        for (int k = 0; k < 6; k++) {
          p2[k] = {fma(p.re, DD[k], p2[k].re), fma(p.im, DD[k], p2[k].im)};
          q2[k] = {fma(q.re, DD[k], q2[k].re), fma(q.im, DD[k], q2[k].im)};
        }
      }
      const bool self = n == m;  // no K term: phi enters through grad g only
      const Cv P1 = {p1[0], p1[1], p1[2]};
      const Cv G1 = {g1[0], g1[1], g1[2]};
      const double2 *cx = reinterpret_cast<const double2 *>(fc + 16 * NO);
      const Cd aXJ = ld_c(cx), aXM = ld_c(cx + 4);
      const Cv XJ = affine(aXJ, D0, ld_v(cx + 1)), XM = affine(aXM, D0, ld_v(cx + 5));
      // sums of g and of phi over the fields of one set (a, field^): J and M
      // into accumulator set s; sg: sign of the cross terms (T: J -, M +)
      auto fields = [&](int s, Cd aJ, Cd aM, const Cv &FJ, const Cv &FM, double sg) {
        const Cv uj = cvsub(cvscale(g0, FJ), cvscale(aJ, G1)), um = cvsub(cvscale(g0, FM), cvscale(aM, G1));
        Cv rj = cvscale(a.c1, uj), rm = cvscale(cmul(a.c1, a.Z), um);
        if (!self) {
          const Cv vj = cvcross(P1, FJ), vm = cvcross(P1, FM);
          const Cd sp = {sg, 0}, sn = {-sg, 0};
          rj = cvadd(rj, cvscale(sn, vm));
          rm = cvadd(rm, cvscale(sp, vj));
        }
        add_v(s, 0, rj);
        add_v(s, 3, rm);
        const Cd c2g = cmul(a.c2, g0);
        add_c(s, 6, csc(cmul(c2g, aJ), 2.0));
        add_c(s, 7, csc(cmul(cmul(c2g, a.Z), aM), 2.0));
      };
      fields(NO, aXJ, aXM, XJ, XM, 1.0);  // dF / dT
      const Cv OXJ = own_v(NO, 0), OXM = own_v(NO, 3);
      const Cd odXJ = own_c(NO, 6), odXM = own_c(NO, 7);
#pragma unroll 1
      for (int o = 0; o < NO; o++) {
        const double2 *ct = reinterpret_cast<const double2 *>(fc + 16 * o);
        const Cd aTJ = ld_c(ct), aTM = ld_c(ct + 4);
        const Cv TJ = affine(aTJ, D0, ld_v(ct + 1)), TM = affine(aTM, D0, ld_v(ct + 5));
        fields(o, aTJ, aTM, TJ, TM, -1.0);  // dF / dX
        const Cv OTJ = own_v(o, 0), OTM = own_v(o, 3);
        const Cd z0 = {0, 0};
        const Cd aj = cvdot(OXJ, TJ, cvdot(OTJ, XJ, z0)), am = cvdot(OXM, TM, cvdot(OTM, XM, z0));
        const Cd dj = cfma(odXJ, aTJ, cmul(own_c(o, 6), aXJ)), dm = cfma(odXM, aTM, cmul(own_c(o, 7), aXM));
        const Cd alpha = cfma(a.c1, cfma(a.Z, am, aj), csc(cmul(a.c2, cfma(a.Z, dm, dj)), 2.0));
        const Cv gj = cvadd(cvscale(aXJ, OTJ), cvscale(aTJ, OXJ)), gm = cvadd(cvscale(aXM, OTM), cvscale(aTM, OXM));
        const Cv gamma = cvscale(a.c1, cvadd(gj, cvscale(a.Z, gm)));
        Cv fo = cvsub(symv(p2, gamma), cvscale(alpha, P1));
        if (!self) {
          const Cv B = cvadd(cvsub(cvcross(XJ, OTM), cvcross(XM, OTJ)), cvsub(cvcross(TM, OXJ), cvcross(TJ, OXM)));
          const Cv eta = cvadd(cvsub(cvscale(aXJ, OTM), cvscale(aXM, OTJ)),
                               cvsub(cvscale(aTM, OXJ), cvscale(aTJ, OXM)));
          fo = cvadd(fo, cvadd(symv(q2, B), cvsub(cvscale(p0, B), cvcross(P1, eta))));
        }
        double *af = s_acc + (16 * (NO + 1) + 3 * o) * kT + tid;
        af[0] += fo.x.re;
        af[kT] += fo.y.re;
        af[2 * kT] += fo.z.re;
      }
    }
  }
  if (!valid) return;
  // per objective: R_i = Re(force + w (a . fields)), and the weighted sums that
  // the free vertices and edge lengths need: w F (12 complex: TJ, TM, XJ, XM),
  // w qrel.F (4), w Fd (4)
  const double *qr = a.qrel + ((size_t)m * NQ + t) * 3;
#pragma unroll 1
  for (int o = 0; o < NO; o++) {
    double *out = a.part + (((size_t)blockIdx.y * NO + o) * P + i) * kRevVals;
    const double *af = s_acc + (16 * (NO + 1) + 3 * o) * kT + tid;
    double R[3] = {af[0], af[kT], af[2 * kT]};
#pragma unroll 1
    for (int h = 0; h < 4; h++) {
      const int s = h < 2 ? NO : o, at = 3 * (h & 1);        // accumulator: dF/dT in set NO, dF/dX in set o
      const Cd al = ld_c(a.coef + ((size_t)(h < 2 ? o : NO) * a.F + m) * 8 + 4 * (h & 1));
      Cd S1 = {0, 0};
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const Cd F = {s_acc[(16 * s + 2 * (at + k)) * kT + tid], s_acc[(16 * s + 2 * (at + k) + 1) * kT + tid]};
        R[k] += w * (al.re * F.re - al.im * F.im);
        out[3 + 2 * (3 * h + k)] = kOofpi * w * F.re;
        out[3 + 2 * (3 * h + k) + 1] = kOofpi * w * F.im;
        S1.re += w * qr[k] * F.re;
        S1.im += w * qr[k] * F.im;
      }
      const int ad = 6 + (h & 1);
      out[27 + 2 * h] = kOofpi * S1.re;
      out[27 + 2 * h + 1] = kOofpi * S1.im;
      out[35 + 2 * h] = kOofpi * w * s_acc[(16 * s + 2 * ad) * kT + tid];
      out[35 + 2 * h + 1] = kOofpi * w * s_acc[(16 * s + 2 * ad + 1) * kT + tid];
    }
#pragma unroll
    for (int k = 0; k < 3; k++) out[k] = kOofpi * R[k];
  }
}

struct RevStaticArgs {
  AdjTopo t;
  int F, no;
  int64_t nnear;
  const int *near_m, *near_n;
  const double *qrel, *qabs, *cp, *area;
  const FaceGeo *geo;
  const double2 *coef;  // as RevArgs
  const double2 *xv;    // x on the unknowns, the sets set_x apart
  size_t set_x;
  Cd k2, c1, c2, Z;
  double *part;         // the fields' slot: [no][F NQ][kRevVals], the sets set_part apart
  size_t set_part;
  double *pair;         // [set][nnear][9][no][4]: d/d(source coordinate); minus its share of the test vertices
};

// First entry of row m of the near list (sorted by test face).
__device__ __forceinline__ int64_t near_row(const int *near_m, int64_t nnear, int m) {
  int64_t lo = 0, hi = nnear;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (near_m[mid] < m) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// Fields of the near faces' closed-form terms at every point, written as one
// more split of rev_field_kernel's output (no dF/dX and no force: those are
// rev_static_kernel's).  kStaticLanes threads per point with every
// kStaticLanes-th near face each, added up in a fixed order.  Bound by the
// latency of point_static: one thread per point took 388 us over 80 faces.
constexpr int kStaticLanes = 8;
template <int NQ>
__global__ void __launch_bounds__(64) rev_static_field_kernel(RevStaticArgs a) {
  const int P = a.F * NQ, at = blockIdx.x * blockDim.x + threadIdx.x, lane = at % kStaticLanes;
  const bool live = at / kStaticLanes < P;
  const int i = live ? at / kStaticLanes : 0;
  a.coef += (size_t)blockIdx.y * (a.no + 1) * a.F * 8;
  a.part += blockIdx.y * a.set_part;
  const int m = i / NQ, t = i % NQ;
  const double w = c_qw[t];
  const double *r = a.qabs + (size_t)i * 3;
  const double f4 = 1.0 / (4.0 * kPi);
  const Cd f8 = {a.k2.re / (8.0 * kPi), a.k2.im / (8.0 * kPi)};
  Cd F[2][4];  // J, M: field (3), divergence
  for (int h = 0; h < 2; h++)
    for (int k = 0; k < 4; k++) F[h][k] = {0, 0};
  for (int64_t j = near_row(a.near_m, a.nnear, m) + lane; j < a.nnear && a.near_m[j] == m; j += kStaticLanes) {
    const int n = a.near_n[j];
    PointStatic<double> ps;
    point_static(r, a.geo[n], ps);
    const double iA = 1.0 / a.area[n];
    const Cd y0 = {f4 * ps.Sm1 - f8.re * ps.S1, -f8.im * ps.S1};
    Cv Hn;
    Cd *hv = &Hn.x;
#pragma unroll
    for (int k = 0; k < 3; k++) hv[k] = {f4 * ps.K3m1[k] - f8.re * ps.K31[k], -f8.im * ps.K31[k]};
    const double D0[3] = {r[0] - a.cp[3 * n], r[1] - a.cp[3 * n + 1], r[2] - a.cp[3 * n + 2]};
    const double rc[3] = {ps.rho[0] - a.cp[3 * n], ps.rho[1] - a.cp[3 * n + 1], ps.rho[2] - a.cp[3 * n + 2]};
    Cv K[2];
    for (int h = 0; h < 2; h++) {
      const double2 *c = a.coef + ((size_t)a.no * a.F + n) * 8 + 4 * h;
      const Cd al = ld_c(c);
      const Cv b = ld_v(c + 1), vr = affine(al, rc, b);
      const Cd *vv = &vr.x;
      const Cd z = h ? a.Z : Cd{1.0, 0.0}, c1 = cmul(a.c1, z), c2 = cmul(a.c2, z);
      for (int k = 0; k < 3; k++) {
        const Cd l = {f4 * ps.mL1[k] - f8.re * ps.mL3[k] / 3.0, -f8.im * ps.mL3[k] / 3.0};
        const Cd Y = csc(cfma(al, l, cmul(y0, vv[k])), iA);
        F[h][k] = cfma(c1, Y, F[h][k]);
      }
      F[h][3] = cfma(c2, csc(cmul(al, y0), 2.0 * iA), F[h][3]);
      K[h] = cvcross(Hn, affine(al, D0, b));
    }
    if (n != m)
      for (int k = 0; k < 3; k++) {
        F[0][k] = csub(F[0][k], csc((&K[1].x)[k], iA));
        F[1][k] = cadd(F[1][k], csc((&K[0].x)[k], iA));
      }
  }
#pragma unroll
  for (int h = 0; h < 2; h++)
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
      for (int s = 1; s < kStaticLanes; s *= 2) {
        F[h][k].re += __shfl_xor_sync(0xffffffffu, F[h][k].re, s);
        F[h][k].im += __shfl_xor_sync(0xffffffffu, F[h][k].im, s);
      }
  if (!live || lane != 0) return;
  const double *qr = a.qrel + (size_t)i * 3;
  for (int o = 0; o < a.no; o++) {
    double *out = a.part + ((size_t)o * P + i) * kRevVals;
    for (int k = 0; k < kRevVals; k++) out[k] = 0.0;
    for (int h = 0; h < 2; h++) {
      const Cd al = ld_c(a.coef + ((size_t)o * a.F + m) * 8 + 4 * h);
      for (int k = 0; k < 3; k++) {
        const Cd f = F[h][k];
        out[k] += w * (al.re * f.re - al.im * f.im);
        out[3 + 2 * (3 * h + k)] = w * f.re;
        out[3 + 2 * (3 * h + k) + 1] = w * f.im;
        out[27 + 2 * h] += w * qr[k] * f.re;
        out[27 + 2 * h + 1] += w * qr[k] * f.im;
      }
      out[35 + 2 * h] = w * F[h][3].re;
      out[35 + 2 * h + 1] = w * F[h][3].im;
    }
  }
}

// Thread per (near pair, coordinate of its source face): the derivative of
// the closed-form terms at fixed T_i.
template <int NQ>
__global__ void __launch_bounds__(64) rev_static_kernel(RevStaticArgs a) {
  const int64_t item = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (item >= a.nnear * 9) return;
  a.coef += (size_t)blockIdx.y * (a.no + 1) * a.F * 8;
  a.xv += blockIdx.y * a.set_x;
  a.pair += (size_t)blockIdx.y * a.nnear * 36 * a.no;
  const int64_t j = item / 9;
  const int seed = (int)(item % 9);
  const int m = a.near_m[j], n = a.near_n[j];
  FaceGeoT<Dual> g;
  Dual area, cp[3], sl[3], bn[3][3];
  face_geo(a.t, n, a.t.fnode[3 * n + seed / 3], seed % 3, g, area, cp, sl, bn);
  // a and b of x about the face's first vertex
  Cx<Dual> ax[2], bx[2][3];
  for (int h = 0; h < 2; h++) {
    ax[h] = {Dual(0.0), Dual(0.0)};
    for (int k = 0; k < 3; k++) bx[h][k] = {Dual(0.0), Dual(0.0)};
    for (int p = 0; p < 3; p++) {
      const double2 v = a.xv[a.t.hpar[3 * n + p] + (h ? a.t.N : 0)];
      const Dual s = 0.5 * sl[p];
      ax[h] = cxa(ax[h], Cx<Dual>{s * v.x, s * v.y});
      for (int k = 0; k < 3; k++) {
        const Dual q = s * (bn[p][k] - g.v[0][k]);
        bx[h][k] = cxs(bx[h][k], Cx<Dual>{q * v.x, q * v.y});
      }
    }
  }
  const Dual iA = 1.0 / area;
  const double f4 = 1.0 / (4.0 * kPi);
  const double f8r = a.k2.re / (8.0 * kPi), f8i = a.k2.im / (8.0 * kPi);
  double val[2] = {0, 0}, tv[2][3] = {{0, 0, 0}, {0, 0, 0}};
#pragma unroll 1
  for (int t = 0; t < NQ; t++) {
    const double *rp = a.qabs + ((size_t)m * NQ + t) * 3;
    const Dual r[3] = {Dual(rp[0]), Dual(rp[1]), Dual(rp[2])};
    PointStatic<Dual> ps;
    point_static(r, g, ps);
    // derivative parts of Y, y, K of the J and M currents
    Cd dY[2][3], dy[2], dK[2][3];
    const Cx<Dual> y0 = {f4 * ps.Sm1 - f8r * ps.S1, -f8i * ps.S1};
    Cx<Dual> H[3];
#pragma unroll
    for (int k = 0; k < 3; k++) H[k] = {f4 * ps.K3m1[k] - f8r * ps.K31[k], -f8i * ps.K31[k]};
#pragma unroll 1
    for (int h = 0; h < 2; h++) {
      Cx<Dual> sr[3];
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const Dual dr = ps.rho[k] - g.v[0][k], dx = r[k] - g.v[0][k];
        const Cx<Dual> vr = cxa(Cx<Dual>{ax[h].re * dr, ax[h].im * dr}, bx[h][k]);
        const Cx<Dual> l = {f4 * ps.mL1[k] - f8r * ps.mL3[k] / 3.0, -f8i * ps.mL3[k] / 3.0};
        dY[h][k] = dpart(cxr(cxa(cxm(ax[h], l), cxm(y0, vr)), iA));
        sr[k] = cxr(cxa(Cx<Dual>{ax[h].re * dx, ax[h].im * dx}, bx[h][k]), iA);
      }
      dy[h] = dpart(cxr(cxm(ax[h], y0), 2.0 * iA));
      dK[h][0] = dpart(cxs(cxm(H[1], sr[2]), cxm(H[2], sr[1])));
      dK[h][1] = dpart(cxs(cxm(H[2], sr[0]), cxm(H[0], sr[2])));
      dK[h][2] = dpart(cxs(cxm(H[0], sr[1]), cxm(H[1], sr[0])));
    }
    const double w = c_qw[t];
    const double *qr = a.qrel + ((size_t)m * NQ + t) * 3;
    for (int o = 0; o < a.no; o++) {
      const double2 *c = a.coef + ((size_t)o * a.F + m) * 8;
      double e = 0;
      Cd T[2][3], dT[2];
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const Cd al = ld_c(c + 4 * h);
        const Cv v = affine(al, qr, ld_v(c + 4 * h + 1));
        T[h][0] = v.x;
        T[h][1] = v.y;
        T[h][2] = v.z;
        dT[h] = {2 * al.re, 2 * al.im};
      }
#pragma unroll
      for (int h = 0; h < 2; h++) {
        Cd s = {0, 0};
#pragma unroll
        for (int k = 0; k < 3; k++) s = cfma(T[h][k], dY[h][k], s);
        s = cfma(a.c1, s, cmul(a.c2, cmul(dT[h], dy[h])));
        if (h) s = cmul(a.Z, s);
        e += s.re;
      }
      if (m != n) {
        Cd s = {0, 0};
#pragma unroll
        for (int k = 0; k < 3; k++) s = cfms(T[0][k], dK[1][k], cfma(T[1][k], dK[0][k], s));
        e += s.re;
      }
      e *= w;
      val[o] += e;
#pragma unroll
      for (int k = 0; k < 3; k++) tv[o][k] -= e * c_qn[t][k == 0 ? 2 : k - 1];
    }
  }
  for (int o = 0; o < a.no; o++) {
    double *out = a.pair + ((size_t)item * a.no + o) * 4;
    out[0] = val[o];
    for (int k = 0; k < 3; k++) out[1 + k] = tv[o][k];
  }
}

struct RevChainArgs {
  AdjTopo t;
  int F, no, splits;
  int64_t nnear;
  const int *near_m, *near_n;
  const double *mu, *sl;
  const double2 *lam, *xv;  // the launch's objectives: [set][no][n], x (set_x apart)
  int64_t n;
  size_t set_x, set_part;
  const double *part, *pair;
  double *out;              // [set][no][F][9]
};

// One CTA per (face, objective of a set, set): the chain rule to the face's nine
// coordinates, every sum in a fixed order.  Bound by latency: the sums over
// splits and points and those over near faces are spread over the threads (one
// warp, and nine of its lanes for the near faces, took 280 us over 80 faces).
constexpr int kChainThreads = 128;
template <int NQ>
__global__ void __launch_bounds__(kChainThreads) rev_chain_kernel(RevChainArgs a) {
  constexpr int kWarps = kChainThreads / 32;
  const int f = blockIdx.x, o = blockIdx.y, lane = threadIdx.x % 32, wid = threadIdx.x / 32;
  const int P = a.F * NQ;
  a.lam += (size_t)blockIdx.z * a.no * a.n;
  a.xv += blockIdx.z * a.set_x;
  a.part += blockIdx.z * a.set_part;
  a.pair += (size_t)blockIdx.z * a.nnear * 36 * a.no;
  a.out += (size_t)blockIdx.z * a.no * a.F * 9;
  __shared__ double s_sum[9 + 40], s_w[kWarps][9 + 40], s_n[kWarps][9], s_v[9], s_u[3][3], s_l[3];
  for (int e = lane; e < 49; e += 32) {
    double acc = 0;
#pragma unroll 4
    for (int b = wid; b < a.splits * NQ; b += kWarps) {
      const int s = b / NQ, t = b % NQ;
      const double *p = a.part + (((size_t)s * a.no + o) * P + (size_t)f * NQ + t) * kRevVals;
      acc += e < 9 ? c_qn[t][e / 3 == 0 ? 2 : e / 3 - 1] * p[e % 3] : p[3 + e - 9];
    }
    s_w[wid][e] = acc;
  }
  // closed-form terms: as the source face, and as the test face
  {
    double v[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    const int64_t r0 = near_row(a.near_m, a.nnear, f);
    for (int64_t j = r0 + threadIdx.x; j < a.nnear && a.near_m[j] == f; j += kChainThreads) {
      const int mp = a.near_n[j];  // the pair (mp, f): the near relation is symmetric
      int64_t lo = near_row(a.near_m, a.nnear, mp), hi = near_row(a.near_m, a.nnear, mp + 1);
      while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (a.near_n[mid] < f) lo = mid + 1;
        else hi = mid;
      }
#pragma unroll
      for (int c = 0; c < 9; c++) {
        for (int u = 0; u < 3; u++) v[c] += a.pair[((size_t)(j * 9 + 3 * u + c % 3) * a.no + o) * 4 + 1 + c / 3];
        v[c] += a.pair[((size_t)(lo * 9 + c) * a.no + o) * 4];
      }
    }
#pragma unroll
    for (int c = 0; c < 9; c++)
#pragma unroll
      for (int s = 1; s < 32; s *= 2) v[c] += __shfl_xor_sync(0xffffffffu, v[c], s);
    if (lane == 0)
#pragma unroll
      for (int c = 0; c < 9; c++) s_n[wid][c] = v[c];
  }
  __syncthreads();
  if (wid > 0) return;
  for (int e = lane; e < 49; e += 32) {
    double acc = 0;
    for (int k = 0; k < kWarps; k++) acc += s_w[k][e];
    s_sum[e] = acc;
  }
  __syncwarp();
  const double *S = s_sum + 9;  // TJ, TM, XJ, XM: w F (3 complex each), then w qrel.F, then w Fd
  if (lane < 3) {
    const int p = lane;
    const double s = a.sl[3 * f + p];
    const double *mu = a.mu + 9 * (size_t)f + 3 * p;
    double gu[3] = {0, 0, 0}, gl = 0;
    for (int h = 0; h < 4; h++) {
      const double2 c = (h < 2 ? a.lam + (size_t)o * a.n : a.xv)[a.t.hpar[3 * f + p] + (h & 1 ? a.t.N : 0)];
      double mr = 0, mi = 0;
      for (int k = 0; k < 3; k++) {
        const double fr = S[2 * (3 * h + k)], fi = S[2 * (3 * h + k) + 1];
        gu[k] -= 0.5 * s * (c.x * fr - c.y * fi);
        mr += mu[k] * fr;
        mi += mu[k] * fi;
      }
      const double lr = 0.5 * (S[24 + 2 * h] - mr) + S[32 + 2 * h];
      const double li = 0.5 * (S[24 + 2 * h + 1] - mi) + S[32 + 2 * h + 1];
      gl += c.x * lr - c.y * li;
    }
    for (int k = 0; k < 3; k++) s_u[p][k] = gu[k];
    s_l[p] = gl;
  }
  if (lane < 9) {
    double acc = s_sum[lane];
    for (int k = 0; k < kWarps; k++) acc += s_n[k][lane];
    s_v[lane] = acc;
  }
  __syncwarp();
  if (lane < 3) {  // axis
    const int k = lane;
    auto slot = [&](int node) { return node == a.t.fnode[3 * f] ? 0 : (node == a.t.fnode[3 * f + 1] ? 1 : 2); };
    for (int p = 0; p < 3; p++) {
      s_v[3 * slot(a.t.fbn[3 * f + p]) + k] += s_u[p][k];
      const int ea = a.t.fea[3 * f + p], eb = a.t.feb[3 * f + p];
      const double s = a.sl[3 * f + p];  // sign times length
      const double d = s_l[p] * (a.t.nodes[3 * ea + k] - a.t.nodes[3 * eb + k]) / s;
      s_v[3 * slot(ea) + k] += d;
      s_v[3 * slot(eb) + k] -= d;
    }
  }
  __syncwarp();
  if (lane < 9) a.out[((size_t)o * a.F + f) * 9 + lane] = s_v[lane];
}

template <int NQ>
int rev_launch(Ctx *c, const RevArgs &ra, const RevStaticArgs &sa, const RevChainArgs &ca, int splits, int sets) {
  const int P = ra.F * NQ;
  const dim3 grid((P + kRevThreads - 1) / kRevThreads, splits, sets);
  const size_t smem = rev_smem<NQ>(ra.no);
  if (ra.no == 2) {
    MOM_CUDA(c, cudaFuncSetAttribute(rev_field_kernel<NQ, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    rev_field_kernel<NQ, 2><<<grid, kRevThreads, smem, c->stream>>>(ra);
  } else {
    MOM_CUDA(c, cudaFuncSetAttribute(rev_field_kernel<NQ, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    rev_field_kernel<NQ, 1><<<grid, kRevThreads, smem, c->stream>>>(ra);
  }
  rev_static_field_kernel<NQ><<<dim3((P * kStaticLanes + 63) / 64, sets), 64, 0, c->stream>>>(sa);
  if (sa.nnear > 0) rev_static_kernel<NQ><<<dim3((unsigned)((sa.nnear * 9 + 63) / 64), sets), 64, 0, c->stream>>>(sa);
  rev_chain_kernel<NQ><<<dim3(ca.F, ca.no, sets), kChainThreads, 0, c->stream>>>(ca);
  c->launches += sa.nnear > 0 ? 4 : 3;
  MOM_CUDA(c, cudaGetLastError());
  return MOM_OK;
}

// Sets of objectives that rev_nodes takes at once: as many as leave one split
// of the faces each in a few waves of CTAs.
int rev_sets(const Ctx *c, const DomDev &D) {
  return std::max(1, 8 * c->nsm / ((D.F * c->nq + kRevThreads - 1) / kRevThreads));
}

// d Re(lambda_o^T A_d x_o) / d(coordinates of domain d's face vertices) for
// objectives o0 .. o0 + sets no - 1, no of the same x after another:
// out[sets][no][F][9].
int rev_nodes(Ctx *c, int d, const AdjPairArgs &m, int o0, int no, int sets, std::vector<double> &out) {
  DomDev &D = c->dom[d];
  MOM_TRY(nfield_geometry(c, D));
  const int F = D.F, P = F * c->nq;
  // a few waves of two CTAs per SM, two faces at least per CTA (the sums over a
  // split's faces are a serial chain, 9 us per face with 13 points)
  const int blocks = (P + kRevThreads - 1) / kRevThreads;
  const int want = std::max(1, std::min(F / 2, 8 * c->nsm / (blocks * sets)));
  const int per = (F + want - 1) / want, splits = (F + per - 1) / per;
  const size_t b_coef = sizeof(double2) * 8 * (size_t)F * (no + 1) * sets;
  const size_t slot = sizeof(double) * kRevVals * (size_t)P * no, set_part = slot / sizeof(double) * (splits + 1);
  const size_t b_part = sizeof(double) * set_part * sets;
  const size_t b_pair = sizeof(double) * 36 * (size_t)no * std::max<int64_t>(1, D.nnear) * sets;
  const size_t b_out = sizeof(double) * 9 * (size_t)F * no * sets;
  MOM_TRY(ensure_buffer(c, &c->adj_part, &c->adj_part_bytes, b_coef + b_part + b_pair + b_out));
  char *b = (char *)c->adj_part;
  double2 *coef = (double2 *)b;
  const double2 *lam = m.lam + (size_t)o0 * m.n, *xv = m.xv + (size_t)o0 * m.n;
  const size_t set_x = (size_t)no * m.n;
  const dim3 cg((F + 127) / 128, no);
  for (int s = 0; s < sets; s++) {
    double2 *cs = coef + 8 * (size_t)F * (no + 1) * s;
    face_current_kernel<<<cg, 128, 0, c->stream>>>(F, c->N, D.hpar, D.sl, D.mu, lam + s * set_x, m.n, cs);
    face_current_kernel<<<cg.x, 128, 0, c->stream>>>(F, c->N, D.hpar, D.sl, D.mu, xv + s * set_x, m.n,
                                                     cs + 8 * (size_t)F * no);
    c->launches += 2;
  }
  RevArgs ra;
  ra.F = F;
  ra.no = no;
  ra.qrel = D.qrel;
  ra.cp = D.cp;
  ra.coef = coef;
  ra.near_bits = D.near_bits;
  ra.kr = m.kr.v;
  ra.ki = m.ki.v;
  ra.c1 = {m.c1.re.v, m.c1.im.v};
  ra.c2 = {m.c2.re.v, m.c2.im.v};
  ra.Z = {m.Zsi.re.v, m.Zsi.im.v};
  ra.per_split = per;
  ra.part = (double *)(b + b_coef);
  ra.set_part = set_part;
  RevStaticArgs sa;
  sa.t = m.t;
  sa.F = F;
  sa.no = no;
  sa.nnear = D.nnear;
  sa.near_m = D.near_m;
  sa.near_n = D.near_n;
  sa.qrel = D.qrel;
  sa.qabs = D.qabs;
  sa.cp = D.cp;
  sa.area = D.area;
  sa.geo = reinterpret_cast<const FaceGeo *>(D.nf_geo);
  sa.coef = coef;
  sa.xv = xv;
  sa.set_x = set_x;
  sa.k2 = {ra.kr * ra.kr - ra.ki * ra.ki, 2 * ra.kr * ra.ki};
  sa.c1 = ra.c1;
  sa.c2 = ra.c2;
  sa.Z = ra.Z;
  sa.part = (double *)(b + b_coef + slot * splits);
  sa.set_part = set_part;
  sa.pair = (double *)(b + b_coef + b_part);
  RevChainArgs ca;
  ca.t = m.t;
  ca.F = F;
  ca.no = no;
  ca.splits = splits + 1;
  ca.nnear = D.nnear;
  ca.near_m = D.near_m;
  ca.near_n = D.near_n;
  ca.mu = D.mu;
  ca.sl = D.sl;
  ca.lam = lam;
  ca.xv = xv;
  ca.n = m.n;
  ca.set_x = set_x;
  ca.set_part = set_part;
  ca.part = ra.part;
  ca.pair = sa.pair;
  ca.out = (double *)(b + b_coef + b_part + b_pair);
  switch (c->nq) {
    case 1: MOM_TRY(rev_launch<1>(c, ra, sa, ca, splits, sets)); break;
    case 3: MOM_TRY(rev_launch<3>(c, ra, sa, ca, splits, sets)); break;
    case 4: MOM_TRY(rev_launch<4>(c, ra, sa, ca, splits, sets)); break;
    case 7: MOM_TRY(rev_launch<7>(c, ra, sa, ca, splits, sets)); break;
    case 13: MOM_TRY(rev_launch<13>(c, ra, sa, ca, splits, sets)); break;
    default: return fail(c, MOM_ERR_ARG, "unsupported number of quadrature points");
  }
  out.resize(9 * (size_t)F * no * sets);
  MOM_CUDA(c, cudaMemcpyAsync(out.data(), ca.out, b_out, cudaMemcpyDeviceToHost, c->stream));
  MOM_CUDA(c, cudaStreamSynchronize(c->stream));
  return MOM_OK;
}

}  // namespace
