// Helper physics of the miniAero face flux: primitive variables, Roe upwind
// inviscid flux with the eigenvalue fix, and the viscous flux.  The
// arithmetic follows the reference's kernels/mini_aero_utils.hpp:6-373
// operation for operation so that results are bit-identical to its serial
// loop when neither side fuses multiply-adds; a form with fewer operations
// for the units that do fuse them follows.
#ifndef FOT_MINI_AERO_UTILS_HPP
#define FOT_MINI_AERO_UTILS_HPP

#ifndef FOT_HD
#define FOT_HD __host__ __device__ __forceinline__
#endif

// conserved (rho, rho u, rho v, rho w, E) -> primitive (rho, u, v, w, T)
FOT_HD void ma_primitives(const double *U, double *V) {
  const double gamma = 1.4, Rgas = 287.05;
  const double r = U[0];
  const double ri = 1.0 / r;
  const double u = U[1] * ri, v = U[2] * ri, w = U[3] * ri;
  const double k = 0.5 * (u * u + v * v + w * w);
  const double e = U[4] * ri - k;
  V[0] = r;
  V[1] = u;
  V[2] = v;
  V[3] = w;
  V[4] = e * (gamma - 1.0) / Rgas;
}

// y = A x for a 5x5 row-major A; y starts at y*0 and sums in column order
FOT_HD void ma_matvec5(const double *A, const double *x, double *y) {
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    double acc = y[i] * 0.0;
#pragma unroll
    for (int j = 0; j < 5; ++j) acc += 1.0 * A[5 * i + j] * x[j];
    y[i] = acc;
  }
}

FOT_HD void ma_inviscid_flux(const double *pl, const double *pr, double *flux,
                             const double *n, const double *t, const double *b,
                             unsigned fs) {
  const double efix_u = 0.1, efix_c = 0.1, gm1 = 0.4;
  const double n0 = n[0], n1 = n[fs], n2 = n[2 * fs];
  const double t0 = t[0], t1 = t[fs], t2 = t[2 * fs];
  const double b0 = b[0], b1 = b[fs], b2 = b[2 * fs];
  const double rho_l = pl[0], u_l = pl[1], v_l = pl[2], w_l = pl[3];
  const double p_l = rho_l * 287.05 * pl[4], h_l = 1004.0 * pl[4];
  const double H_l = h_l + 0.5 * (u_l * u_l + v_l * v_l + w_l * w_l);
  const double mf_l = rho_l * (n0 * u_l + n1 * v_l + n2 * w_l);
  const double rho_r = pr[0], u_r = pr[1], v_r = pr[2], w_r = pr[3];
  const double p_r = rho_r * 287.05 * pr[4], h_r = 1004.0 * pr[4];
  const double H_r = h_r + 0.5 * (u_r * u_r + v_r * v_r + w_r * w_r);
  const double mf_r = rho_r * (n0 * u_r + n1 * v_r + n2 * w_r);
  const double psum = p_l + p_r;
  flux[0] = 0.5 * (mf_l + mf_r);
  flux[1] = 0.5 * (mf_l * u_l + mf_r * u_r + n0 * psum);
  flux[2] = 0.5 * (mf_l * v_l + mf_r * v_r + n1 * psum);
  flux[3] = 0.5 * (mf_l * w_l + mf_r * w_r + n2 * psum);
  flux[4] = 0.5 * (mf_l * H_l + mf_r * H_r);

  const double nn = sqrt(n0 * n0 + n1 * n1 + n2 * n2);
  const double tn = sqrt(t0 * t0 + t1 * t1 + t2 * t2);
  const double bn = sqrt(b0 * b0 + b1 * b1 + b2 * b2);
  const double nu0 = n0 / nn, nu1 = n1 / nn, nu2 = n2 / nn;
  const double tu0 = t0 / tn, tu1 = t1 / tn, tu2 = t2 / tn;
  const double bu0 = b0 / bn, bu1 = b1 / bn, bu2 = b2 / bn;

  const double sl = sqrt(rho_l);
  const double denom = 1.0 / (sl + sqrt(rho_r));
  const double alpha = sl * denom;
  const double beta = 1.0 - alpha;
  const double ur = alpha * u_l + beta * u_r;
  const double vr = alpha * v_l + beta * v_r;
  const double wr = alpha * w_l + beta * w_r;
  const double hr = alpha * h_l + beta * h_r +
                    0.5 * alpha * beta *
                        ((u_r - u_l) * (u_r - u_l) + (v_r - v_l) * (v_r - v_l) +
                         (w_r - w_l) * (w_r - w_l));
  const double c = sqrt(gm1 * hr);
  const double nv = ur * nu0 + vr * nu1 + wr * nu2;
  const double tv = ur * tu0 + vr * tu1 + wr * tu2;
  const double bv = ur * bu0 + vr * bu1 + wr * bu2;
  const double ke = 0.5 * (ur * ur + vr * vr + wr * wr);
  const double c2i = 1.0 / (c * c);
  const double hc2i = 0.5 * c2i;
  double dq[5];
  dq[0] = rho_r - rho_l;
  dq[1] = rho_r * u_r - rho_l * u_l;
  dq[2] = rho_r * v_r - rho_l * v_l;
  dq[3] = rho_r * w_r - rho_l * w_l;
  dq[4] = (rho_r * H_r - p_r) - (rho_l * H_l - p_l);
  const double cbar = c * nn;
  const double ubar = ur * n0 + vr * n1 + wr * n2;
  const double cfl = fabs(ubar) + cbar;
  const double e1 = ubar + cbar, e2 = ubar - cbar, e3 = ubar;
  double a1 = fabs(e1), a2 = fabs(e2), a3 = fabs(e3);
  const double epuc = efix_u * cfl, epcc = efix_c * cfl;
  if (a1 < epcc) a1 = 0.5 * (e1 * e1 + epcc * epcc) / epcc;
  if (a2 < epcc) a2 = 0.5 * (e2 * e2 + epcc * epcc) / epcc;
  if (a3 < epuc) a3 = 0.5 * (e3 * e3 + epuc * epuc) / epuc;
  const double ep0 = 0.5 * (e1 + a1), ep1 = 0.5 * (e2 + a2), ep2 = 0.5 * (e3 + a3);
  const double em0 = 0.5 * (e1 - a1), em1 = 0.5 * (e2 - a2), em2 = 0.5 * (e3 - a3);
  const double gk = gm1 * (ke - hr);
  // left eigenvectors, one row per wave
  const double L[25] = {gk + c * (c - nv), c * nu0 - gm1 * ur, c * nu1 - gm1 * vr,
                        c * nu2 - gm1 * wr, gm1,
                        gk + c * (c + nv), -c * nu0 - gm1 * ur, -c * nu1 - gm1 * vr,
                        -c * nu2 - gm1 * wr, gm1,
                        ke - hr, -ur, -vr, -wr, 1.0,
                        -tv, tu0, tu1, tu2, 0.0,
                        -bv, bu0, bu1, bu2, 0.0};
  double ldq[5] = {0, 0, 0, 0, 0};
  ma_matvec5(L, dq, ldq);
  ldq[0] = (ep0 - em0) * ldq[0];
  ldq[1] = (ep1 - em1) * ldq[1];
  ldq[2] = (ep2 - em2) * ldq[2];
  ldq[3] = (ep2 - em2) * ldq[3];
  ldq[4] = (ep2 - em2) * ldq[4];
  // right eigenvectors
  const double hk = hr + ke;
  const double R[25] = {hc2i, hc2i, -gm1 * c2i, 0.0, 0.0,
                        (ur + nu0 * c) * hc2i, (ur - nu0 * c) * hc2i, -gm1 * ur * c2i, tu0, bu0,
                        (vr + nu1 * c) * hc2i, (vr - nu1 * c) * hc2i, -gm1 * vr * c2i, tu1, bu1,
                        (wr + nu2 * c) * hc2i, (wr - nu2 * c) * hc2i, -gm1 * wr * c2i, tu2, bu2,
                        (hk + c * nv) * hc2i, (hk - c * nv) * hc2i, (c * c - gm1 * hk) * c2i,
                        tv, bv};
  double rl[5] = {0, 0, 0, 0, 0};
  ma_matvec5(R, ldq, rl);
#pragma unroll
  for (int i = 0; i < 5; ++i) flux[i] -= 0.5 * rl[i];
}

FOT_HD void ma_viscous_flux(const double g[5][3], const double *prim,
                            const double *a, double *vflux, unsigned as) {
  const double T = prim[4];
  const double visc = 1.458e-6 * T * sqrt(T) / (T + 110.4);
  const double tc = visc * 1006.0 / 0.71;
  const double a0 = a[0], a1 = a[as], a2 = a[2 * as];
  const double av[3] = {a0, a1, a2};
  double div = 0;
#pragma unroll
  for (int i = 0; i < 5; ++i) vflux[i] = 0.0;
#pragma unroll
  for (int i = 0; i < 3; i++) div += g[i + 1][i];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const double delta = (i == j) ? 1 : 0;
      const double S = 0.5 * (g[i + 1][j] + g[j + 1][i]);
      const double tij = S - div * delta / 3.;
      vflux[1 + i] += (2 * visc * tij) * av[j];
      vflux[4] += (2 * visc * tij) * prim[i + 1] * av[j];
    }
    vflux[4] += tc * g[4][i] * av[i];
  }
}

// ---- the form of the contracted units -------------------------------------
// FOT_CONTRACTED is defined where multiply-adds are fused and results are
// summed in any order (the atomic executor): the same flux with fewer
// operations.  The reference's order of operations costs 22 divisions and 7
// roots a face (each a dozen FP64 instructions) and two dense 5x5 products;
// the FP64 chain behind the gathers bounded the loop.  Here the unit vectors
// come from reciprocal roots, divisions by constants are products, the
// eigenvector products are written out without their zeros and with their
// common factors taken out, and of the gradients only what the viscous flux
// needs is kept, so that their 30 values die as they are loaded: 3 divisions
// (one more where an eigenvalue is fixed) and 7 roots.
#ifdef FOT_CONTRACTED

// Sums over both sides of what the viscous flux needs of the gradients g of
// (u, v, w) and T: s[i] = (row i + column i of g) . n, the trace, grad T . n.
struct ma_gradient_sums {
  double s[3], trace, heat;
};

// One side's primitive variables extrapolated to the face.
FOT_HD void ma_side(const double *values, const double *centre, const double *grad,
                    const double *limiter, const double *face, const double *n,
                    unsigned cs, unsigned fs, double *P, ma_gradient_sums &sums) {
  const double n0 = n[0], n1 = n[fs], n2 = n[2 * fs];
  const double d0 = face[0] - centre[0];
  const double d1 = face[fs] - centre[cs];
  const double d2 = face[2 * fs] - centre[2 * cs];
  double step[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const double g0 = grad[(3 * k) * cs], g1 = grad[(3 * k + 1) * cs], g2 = grad[(3 * k + 2) * cs];
    step[k] = (d0 * g0 + d1 * g1 + d2 * g2) * limiter[k * cs];
    if (k == 0) continue;
    const double gn = g0 * n0 + g1 * n1 + g2 * n2;
    if (k == 4) {
      sums.heat += gn;
    } else {
      const double nk = k == 1 ? n0 : k == 2 ? n1 : n2;
      sums.s[k - 1] += gn;
      sums.s[0] += g0 * nk;
      sums.s[1] += g1 * nk;
      sums.s[2] += g2 * nk;
      sums.trace += k == 1 ? g0 : k == 2 ? g1 : g2;
    }
  }
  const double r = values[0];
  const double ri = 1.0 / r;
  const double u = values[cs] * ri, v = values[2 * cs] * ri, w = values[3 * cs] * ri;
  const double e = values[4 * cs] * ri - 0.5 * (u * u + v * v + w * w);
  P[0] = r + step[0];
  P[1] = u + step[1];
  P[2] = v + step[2];
  P[3] = w + step[3];
  P[4] = e * ((1.4 - 1.0) / 287.05) + step[4];
}

// The inviscid flux (Roe, with the eigenvalue fix) minus the viscous one.
FOT_HD void ma_face_flux(const double *pl, const double *pr, const ma_gradient_sums &sums,
                         double *flux, const double *n, const double *t, const double *b,
                         unsigned fs) {
  const double efix = 0.1, gm1 = 0.4;
  const double n0 = n[0], n1 = n[fs], n2 = n[2 * fs];
  const double rho_l = pl[0], u_l = pl[1], v_l = pl[2], w_l = pl[3];
  const double p_l = rho_l * (287.05 * pl[4]), h_l = 1004.0 * pl[4];
  const double H_l = h_l + 0.5 * (u_l * u_l + v_l * v_l + w_l * w_l);
  const double mf_l = rho_l * (n0 * u_l + n1 * v_l + n2 * w_l);
  const double rho_r = pr[0], u_r = pr[1], v_r = pr[2], w_r = pr[3];
  const double p_r = rho_r * (287.05 * pr[4]), h_r = 1004.0 * pr[4];
  const double H_r = h_r + 0.5 * (u_r * u_r + v_r * v_r + w_r * w_r);
  const double mf_r = rho_r * (n0 * u_r + n1 * v_r + n2 * w_r);
  const double psum = p_l + p_r;
  // viscous: tau . n and the heat flux, at the mean state
  const double T = 0.5 * (pl[4] + pr[4]);
  const double visc = 1.458e-6 * T * sqrt(T) / (T + 110.4);
  const double third = sums.trace * (1.0 / 3.0);
  const double f1 = visc * (0.5 * sums.s[0] - third * n0);
  const double f2 = visc * (0.5 * sums.s[1] - third * n1);
  const double f3 = visc * (0.5 * sums.s[2] - third * n2);
  const double f4 = 0.5 * (f1 * (u_l + u_r) + f2 * (v_l + v_r) + f3 * (w_l + w_r)) +
                    visc * (0.5 * 1006.0 / 0.71) * sums.heat;
  flux[0] = 0.5 * (mf_l + mf_r);
  flux[1] = 0.5 * (mf_l * u_l + mf_r * u_r + n0 * psum) - f1;
  flux[2] = 0.5 * (mf_l * v_l + mf_r * v_r + n1 * psum) - f2;
  flux[3] = 0.5 * (mf_l * w_l + mf_r * w_r + n2 * psum) - f3;
  flux[4] = 0.5 * (mf_l * H_l + mf_r * H_r) - f4;

  // Roe averages
  const double sl = sqrt(rho_l);
  const double alpha = sl / (sl + sqrt(rho_r));
  const double beta = 1.0 - alpha;
  const double ur = alpha * u_l + beta * u_r;
  const double vr = alpha * v_l + beta * v_r;
  const double wr = alpha * w_l + beta * w_r;
  const double hr = alpha * h_l + beta * h_r +
                    0.5 * alpha * beta *
                        ((u_r - u_l) * (u_r - u_l) + (v_r - v_l) * (v_r - v_l) +
                         (w_r - w_l) * (w_r - w_l));
  const double d0 = rho_r - rho_l;
  const double d1 = rho_r * u_r - rho_l * u_l;
  const double d2 = rho_r * v_r - rho_l * v_l;
  const double d3 = rho_r * w_r - rho_l * w_l;
  const double d4 = (rho_r * H_r - p_r) - (rho_l * H_l - p_l);
  const double ke = 0.5 * (ur * ur + vr * vr + wr * wr);
  const double cc = gm1 * hr;
  const double c = sqrt(cc);
  const double c2i = 1.0 / cc;
  // eigenvalues
  const double nsq = n0 * n0 + n1 * n1 + n2 * n2;
  const double ni = rsqrt(nsq);
  const double cbar = c * (nsq * ni);
  const double e3 = ur * n0 + vr * n1 + wr * n2;
  const double e1 = e3 + cbar, e2 = e3 - cbar;
  const double ep = efix * (fabs(e3) + cbar);
  double a1 = fabs(e1), a2 = fabs(e2), a3 = fabs(e3);
  if (a1 < ep || a2 < ep || a3 < ep) {
    const double h = 0.5 / ep;
    if (a1 < ep) a1 = (e1 * e1 + ep * ep) * h;
    if (a2 < ep) a2 = (e2 * e2 + ep * ep) * h;
    if (a3 < ep) a3 = (e3 * e3 + ep * ep) * h;
  }
  // the acoustic and entropy waves: left eigenvectors applied to d, scaled
  const double nv = e3 * ni;
  const double nm = ni * (n0 * d1 + n1 * d2 + n2 * d3);
  const double s = (ke - hr) * d0 - (ur * d1 + vr * d2 + wr * d3) + d4;
  const double w0 = a1 * (gm1 * s + c * ((c - nv) * d0 + nm));
  const double w1 = a2 * (gm1 * s + c * ((c + nv) * d0 - nm));
  const double w2 = a3 * s;
  // right eigenvectors applied to them
  const double hc2i = 0.5 * c2i;
  const double r0 = hc2i * (w0 + w1) - gm1 * c2i * w2;
  const double rn = c * hc2i * (w0 - w1);
  double r1 = ur * r0 + (rn * ni) * n0;
  double r2 = vr * r0 + (rn * ni) * n1;
  double r3 = wr * r0 + (rn * ni) * n2;
  double r4 = (hr + ke) * r0 + nv * rn + w2;
  // the two shear waves
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const double *a = k == 0 ? t : b;
    const double x = a[0], y = a[fs], z = a[2 * fs];
    const double i = rsqrt(x * x + y * y + z * z);
    const double av = i * (ur * x + vr * y + wr * z);
    const double w = a3 * (i * (x * d1 + y * d2 + z * d3) - av * d0);
    r1 += (i * w) * x;
    r2 += (i * w) * y;
    r3 += (i * w) * z;
    r4 += av * w;
  }
  flux[0] -= 0.5 * r0;
  flux[1] -= 0.5 * r1;
  flux[2] -= 0.5 * r2;
  flux[3] -= 0.5 * r3;
  flux[4] -= 0.5 * r4;
}

#endif // FOT_CONTRACTED

#endif
