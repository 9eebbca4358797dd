// mb_face_fast.cuh -- the interior face flux of the simplified flux path (the mixed form and the FP64 production form)
// for the solvers with their own sweep unit: HLLC (1), AUSM+ (4), LMRoe (12). The same scheme as face_flux of
// mb_engine.cuh (conv_physics.inc, diff_cuf_kernels.inc, diff_physics.inc) with the single-species identities, written
// for few instructions, which bounded the sweep before it (60 % of the issue slots in use, DRAM under a fifth of its peak;
// with it half of the slots are, and exposed latency bounds it):
//  - values travel in pairs, (u, v), (w, T), (rho, p): one 8-byte shared load brings two, and in FP32 one instruction
//    (add / mul / fma .f32x2, each half rounded as the scalar instruction rounds) computes on both;
//  - a divide is a multiplication by a reciprocal; in FP32 the reciprocal is one instruction (rcp.approx.ftz), where
//    the full-range divide takes about ten issue slots (measured: 12.8 divides per clock and SM against 15.8 of the
//    approximate one, which is bound by its unit and not by issue);
//  - the viscous flux contracts the gradients with the face normal instead of building the nine gradient components:
//    with the metric rows M_a (a = the three computational directions) and the differences g_a of a variable along
//    them, grad(q) . n = sum_a g_a (M_a . n), (grad u)^T n = sum_a M_a (g_a . n), div u = sum_a g_a . M_a.
// One B200, a step before and with it (the chunk rule in both): 192^3 mixed 4.01 and 3.20 ms, 64 blocks of 32^3 mixed (HLLC)
// 1.65 and 1.51 ms, 96^3 FP64 production 2.25 and 1.74 ms, the 2-D batch of 12 blocks (AUSM+, van Leer) mixed 0.82 and
// 0.69 ms, of 4 blocks FP64 production 0.565 and 0.419 ms.
#pragma once

namespace mb {

// ---- the table row of T and the interpolated values (the rows of tidx)
template <typename R>
__device__ __forceinline__ int trow(const Params& p, R T, R& td) {
  const R c = fmin(fmax(T, Cst<R>::of(p).t0), Cst<R>::of(p).t1);  // NaN -> tmin
  const int ti = (int)c;
  td = T - (R)ti;
  return ti;
}
__device__ __forceinline__ void cp_h(const Params& p, int ti, double td, double& cp, double& h) {
  const double2 a = __ldg(reinterpret_cast<const double2*>(p.tab4) + 2 * ti);
  const double2 b = __ldg(reinterpret_cast<const double2*>(p.tab4) + 2 * ti + 1);
  cp = a.x + a.y * td;
  h = b.x + b.y * td;
}
__device__ __forceinline__ void cp_h(const Params& p, int ti, float td, float& cp, float& h) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(p.tab4f) + ti);
  cp = a.x + a.y * td;
  h = a.z + a.w * td;
}
// viscosity, and the conductivity (mu cp / Pr with a Prandtl number)
__device__ __forceinline__ void mu_k(const Params& p, double T, double& mu, double& k) {
  double td;
  const int ti = trow<double>(p, T, td);
  mu = tabT(p.mu, ti, td);
  k = p.has_pr ? mu * tabT(p.cp, ti, td) * p.cd.ipr : tabT(p.k, ti, td);
}
__device__ __forceinline__ void mu_k(const Params& p, float T, float& mu, float& k) {
  float td;
  const int ti = trow<float>(p, T, td);
  const float4 a = __ldg(reinterpret_cast<const float4*>(p.tabm4f) + ti);
  mu = a.x + a.y * td;
  if (p.has_pr) {
    const float2 c = __ldg(reinterpret_cast<const float2*>(p.tab4f) + 2 * ti);
    k = mu * (c.x + c.y * td) * p.cf.ipr;
  } else {
    k = a.z + a.w * td;
  }
}

// ---- geometry: the metric row a of padded cell l and its dl component; the face record
__device__ __forceinline__ void metric(const DBlk& b, int a, int l, V2<double>& mxy, double& mz, double& dl) {
  const double* m = b.m + 9 * l + a;
  mxy = V2<double>{ld(m), ld(m + 3)};
  mz = ld(m + 6);
  dl = ld(b.dl + 3 * l + a);
}
__device__ __forceinline__ void metric(const DBlk& b, int a, int l, V2<float>& mxy, float& mz, float& dl) {
  const float4 v = __ldg(b.mdf + (a * b.npad + l));
  mxy = mk2<float>(v.x, v.y);
  mz = v.z;
  dl = v.w;
}
template <typename R> __device__ __forceinline__ R cell_dl(const DBlk& b, int a, int l);
template <> __device__ __forceinline__ double cell_dl(const DBlk& b, int a, int l) { return ld(b.dl + 3 * l + a); }
template <> __device__ __forceinline__ float cell_dl(const DBlk& b, int a, int l) {
  return ld(&b.mdf[a * b.npad + l].w);
}
__device__ __forceinline__ void face_rec(const DBlk& b, int d, int f, double& nx, double& ny, double& nz, double& area) {
  const double* q = Geo<double>::fm(b, d) + f;
  nx = ld(q); ny = ld(q + 1); nz = ld(q + 2); area = ld(q + 3);
}
__device__ __forceinline__ void face_rec(const DBlk& b, int d, int f, float& nx, float& ny, float& nz, float& area) {
  const float4 v = __ldg(reinterpret_cast<const float4*>(Geo<float>::fm(b, d) + f));  // the engine's own copy: aligned
  nx = v.x; ny = v.y; nz = v.z; area = v.w;
}

// ---- limited face states of a pair of variables: q0 = qc + s(L) lm, q1 = qd - s(R) lp, from the slopes a, b, c of the
// three cell-to-cell differences of the stencil
__device__ __forceinline__ V2<double> albada(V2<double> a, V2<double> b, V2<double> c, V2<double>& right) {
  // x y (x + y) / (x^2 + y^2) of (b, a) and of (c, b); one division for the four quotients
  const double eps = 1e-30;
  const double bx = b.x * b.x, by = b.y * b.y;
  const double d0 = fma(a.x, a.x, bx) + eps, d1 = fma(c.x, c.x, bx) + eps, d2 = fma(a.y, a.y, by) + eps,
               d3 = fma(c.y, c.y, by) + eps;
  const double p01 = d0 * d1, p23 = d2 * d3;
  const double r = 1.0 / (p01 * p23);
  const double r01 = r * p23, r23 = r * p01;
  right = V2<double>{b.x * c.x * (b.x + c.x) * (r01 * d0), b.y * c.y * (b.y + c.y) * (r23 * d2)};
  return V2<double>{b.x * a.x * (b.x + a.x) * (r01 * d1), b.y * a.y * (b.y + a.y) * (r23 * d3)};
}
// the same of one variable
__device__ __forceinline__ double albada(double a, double b, double c, double& right) {
  const double bb = b * b, d0 = fma(a, a, bb) + 1e-30, d1 = fma(c, c, bb) + 1e-30;
  const double r = 1.0 / (d0 * d1);
  right = b * c * (b + c) * (r * d0);
  return b * a * (b + a) * (r * d1);
}
__device__ __forceinline__ V2<float> albada(V2<float> a, V2<float> b, V2<float> c, V2<float>& right) {
  const V2<float> bb = fma2(b, b, dup2<float>(1e-30f));
  const V2<float> dl = fma2(a, a, bb), dr = fma2(c, c, bb);
  const V2<float> nl = (a * b) * (a + b), nr = (b * c) * (b + c);
  right = nr * mk2<float>(rcp_(lo2(dr)), rcp_(hi2(dr)));
  return nl * mk2<float>(rcp_(lo2(dl)), rcp_(hi2(dl)));
}
// one limited slope of a run-time limiter, x = forward, y = backward difference (rlimiter of mb_physics.cuh)
template <typename R>
__device__ __forceinline__ R slope_rt(int lim, R x, R y) {
  if (lim == 1) {
    R r = x;
    if (fabs(x) > fabs(y)) r = y;
    return (x * y < (R)0) ? (R)0 : r;
  }
  if (lim == 2) {  // (r + |r|) / (1 + |r|) x with r = y / x, written as 2 x |y| / (|x| + |y|) where the signs agree
    const R q = (R)2 * x * (fabs(y) * rcp_(fabs(x) + fabs(y) + (R)1e-30));
    return (x < (R)0) != (y < (R)0) ? (R)0 * q : q;
  }
  return rlimiter<R>(lim, x, y);
}

// ---- Riemann solvers on the pair states L, R: A = (u, v), w, C = (rho, p). Flux per unit area: fr, (fu, fv), (fw, fe)
template <typename R>
struct Side {
  V2<R> A;
  R w, rho, p;
  R T, cp, h;
};

template <typename R>
__device__ __forceinline__ void side_thermo(const Params& p, Side<R>& s) {
  s.T = s.p * Cst<R>::of(p).iri * rcp_(s.rho);
  R td;
  const int ti = trow<R>(p, s.T, td);
  cp_h(p, ti, td, s.cp, s.h);
}

// LMRoe (Mco floor) of lmroe_fast: the Roe averages as L + w (R - L), the dissipation of the three velocity components
// as ks U + kt dU + c n
template <typename R>
__device__ __forceinline__ void roe_pair(const Params& p, const Side<R>& L, const Side<R>& Q, R nx, R ny, R nz, R& fr,
                                         V2<R>& fuv, R& fw, R& fe) {
  const R Rg = Cst<R>::of(p).ri;
  const R sL = rsqrt_(L.rho), sR = rsqrt_(Q.rho);
  const R wr = sR * rcp_(sL + sR);
  const R rho_roe = sL * sR;
  const V2<R> dA = Q.A - L.A;
  const R dw = Q.w - L.w;
  const R kL = (R)0.5 * (lo2(L.A) * lo2(L.A) + hi2(L.A) * hi2(L.A) + L.w * L.w);
  const R kR = (R)0.5 * (lo2(Q.A) * lo2(Q.A) + hi2(Q.A) * hi2(Q.A) + Q.w * Q.w);
  const R h0L = L.h + kL, h0R = Q.h + kR;
  const R eL = L.h - Rg * L.T, eR = Q.h - Rg * Q.T;
  const V2<R> U = fma2(dup2<R>(wr), dA, L.A);
  const R W = L.w + wr * dw;
  const R T = L.T + wr * (Q.T - L.T), H = h0L + wr * (h0R - h0L), E = eL + wr * (eR - eL);
  const R cv = (R)0.5 * (L.cp + Q.cp) - Rg;
  const R u2 = lo2(U) * lo2(U) + hi2(U) * hi2(U) + W * W;
  const R a = rsqrt_(Rg * rcp_(cv) * (H - (R)0.5 * u2 + cv * T - E));
  const R ia = rcp_(a);
  const R unL = lo2(L.A) * nx + hi2(L.A) * ny + L.w * nz, unR = lo2(Q.A) * nx + hi2(Q.A) * ny + Q.w * nz;
  const R un = lo2(U) * nx + hi2(U) * ny + W * nz;
  const R dun = unR - unL;
  R phi = Cst<R>::of(p).mco;
  if (p.mach_floor) {  // Mco < 1 (from 1 on the floor is above min(1, Ma))
    const R Ma = (a > (R)0) ? (fabs(un) + rsqrt_(mx((R)0, u2 - un * un))) * ia : (R)1;
    phi = mx(phi, mn((R)1, Ma));
  }
  const R dp = (Q.p - L.p) * ia * ia;
  const R t = rho_roe * phi * dun * ia;
  const R k1 = fabs(un - a) * ((R)0.5 * (dp - t)), k5 = fabs(un + a) * ((R)0.5 * (dp + t));
  const R k4 = fabs(un) * ((Q.rho - L.rho) - dp), kt = fabs(un) * rho_roe;
  const R ks = k1 + k4 + k5;
  const R c = a * (k5 - k1) - kt * dun;
  const R fL = L.rho * unL, fR = Q.rho * unR;
  const R pn = L.p + Q.p - c;
  fr = (R)0.5 * (fL + fR - ks);
  V2<R> m = fma2(dup2<R>(fL), L.A, dup2<R>(fR) * Q.A);
  m = fma2(dup2<R>(-ks), U, m);
  m = fma2(dup2<R>(-kt), dA, m);
  m = fma2(dup2<R>(pn), mk2<R>(nx, ny), m);
  fuv = dup2<R>((R)0.5) * m;
  fw = (R)0.5 * (fL * L.w + fR * Q.w - ks * W - kt * dw + pn * nz);
  const R udu = lo2(U) * lo2(dA) + hi2(U) * hi2(dA) + W * dw;
  fe = (R)0.5 * (fL * h0L + fR * h0R - ((k1 + k5) * H + k4 * ((R)0.5 * u2) + kt * udu + c * un));
}

// HLLC with the Batten signal speeds (hllc of mb_physics.cuh): the star state of the one side the contact selects. Its
// flux F + S (U* - U) is written out: with du = S* - un, m = rho (S - un) and the mass flux fr = m S* / (S - S*), the
// pressure is p + g and the energy flux fr h0 + S* g, g = du (fr + m), so no large terms cancel. du = S* = 0 gives F, which
// takes nothing from the other side: a supersonic face stays finite beside a state that is not. The rms error of the FP32
// mass, momentum and energy fluxes over random subsonic states, against FP64: 7.4e-8, 3.7e-8 and 9.3e-8; summed as
// F + S (U* - U) 2.6e-7, 4.5e-8 and 3.3e-7.
template <typename R>
__device__ __forceinline__ void hllc_pair(const Params& p, const Side<R>& L, const Side<R>& Q, R nx, R ny, R nz, R& fr,
                                          V2<R>& fuv, R& fw, R& fe) {
  const R Rg = Cst<R>::of(p).ri;
  const R aL = rsqrt_(L.cp * Rg * L.T * rcp_(L.cp - Rg)), aR = rsqrt_(Q.cp * Rg * Q.T * rcp_(Q.cp - Rg));
  const R sL = rsqrt_(L.rho), sR = rsqrt_(Q.rho);
  const R wr = sR * rcp_(sL + sR);
  const R kL = (R)0.5 * (lo2(L.A) * lo2(L.A) + hi2(L.A) * hi2(L.A) + L.w * L.w);
  const R kR = (R)0.5 * (lo2(Q.A) * lo2(Q.A) + hi2(Q.A) * hi2(Q.A) + Q.w * Q.w);
  const R h0L = L.h + kL, h0R = Q.h + kR;
  const R eL = L.h - Rg * L.T, eR = Q.h - Rg * Q.T;
  const V2<R> U = fma2(dup2<R>(wr), Q.A - L.A, L.A);
  const R W = L.w + wr * (Q.w - L.w);
  const R T = L.T + wr * (Q.T - L.T), H = h0L + wr * (h0R - h0L), E = eL + wr * (eR - eL);
  const R cv = (R)0.5 * (L.cp + Q.cp) - Rg;
  const R u2 = lo2(U) * lo2(U) + hi2(U) * hi2(U) + W * W;
  const R a = rsqrt_(Rg * rcp_(cv) * (H - (R)0.5 * u2 + cv * T - E));
  const R unL = lo2(L.A) * nx + hi2(L.A) * ny + L.w * nz, unR = lo2(Q.A) * nx + hi2(Q.A) * ny + Q.w * nz;
  const R un = lo2(U) * nx + hi2(U) * ny + W * nz;
  const R S1 = mn(mn((R)0, unL - aL), un - a);
  const R S4 = mx(mx((R)0, unR + aR), un + a);
  const R mL = L.rho * (S1 - unL), mR = Q.rho * (S4 - unR);
  const R Ss = (Q.p - L.p + mL * unL - mR * unR) * rcp_(mL - mR);
  // (S1 >= 0: the left flux; otherwise the side of the contact, with its physical flux alone where S4 <= 0)
  const bool left = S1 >= (R)0 || Ss >= (R)0;
  const R S = left ? S1 : S4;
  const R un_ = left ? unL : unR, w = left ? L.w : Q.w, h0 = left ? h0L : h0R;
  const R mk = left ? mL : mR;  // rho (S - un)
  const V2<R> A = left ? L.A : Q.A;
  const bool star = left ? S1 < (R)0 : S4 > (R)0;
  const R du = star ? Ss - un_ : (R)0, Sx = star ? Ss : (R)0;
  fr = star ? mk * Ss * rcp_(S - Ss) : (left ? L.rho : Q.rho) * un_;
  const R g = du * (fr + mk);
  const R cn = (left ? L.p : Q.p) + g;
  fuv = fma2(dup2<R>(fr), A, dup2<R>(cn) * mk2<R>(nx, ny));
  fw = fr * w + cn * nz;
  fe = fr * h0 + Sx * g;
}

// AUSM+ (riemann_open of mb_physics.cuh, id 4)
template <typename R>
__device__ __forceinline__ void ausm_pair(const Params& p, const Side<R>& L, const Side<R>& Q, R nx, R ny, R nz, R& fr,
                                          V2<R>& fuv, R& fw, R& fe) {
  const R Rg = Cst<R>::of(p).ri;
  const R aL = rsqrt_(L.cp * Rg * L.T * rcp_(L.cp - Rg)), aR = rsqrt_(Q.cp * Rg * Q.T * rcp_(Q.cp - Rg));
  const R h0L = L.h + (R)0.5 * (lo2(L.A) * lo2(L.A) + hi2(L.A) * hi2(L.A) + L.w * L.w);
  const R h0R = Q.h + (R)0.5 * (lo2(Q.A) * lo2(Q.A) + hi2(Q.A) * hi2(Q.A) + Q.w * Q.w);
  const R ah = rsqrt_(aL * aR), ih = rcp_(ah);
  const R ML = (lo2(L.A) * nx + hi2(L.A) * ny + L.w * nz) * ih, MR = (lo2(Q.A) * nx + hi2(Q.A) * ny + Q.w * nz) * ih;
  const R qL = ML * ML - (R)1, qR = MR * MR - (R)1;
  const R pL1 = (R)0.25 * ((ML + (R)1) * (ML + (R)1)), pR1 = (R)0.25 * ((MR - (R)1) * (MR - (R)1));
  const bool iL = fabs(ML) < (R)1, iR = fabs(MR) < (R)1;
  const R Mp = iL ? pL1 + (R)0.125 * (qL * qL) : (R)0.5 * (ML + fabs(ML));
  const R pp = iL ? pL1 * ((R)2 - ML) + (R)0.1875 * ML * (qL * qL) : (R)0.5 * ((R)1 + copysign((R)1, ML));
  const R Mm = iR ? -pR1 - (R)0.125 * (qR * qR) : (R)0.5 * (MR - fabs(MR));
  const R pm = iR ? pR1 * ((R)2 + MR) - (R)0.1875 * MR * (qR * qR) : (R)0.5 * ((R)1 - copysign((R)1, MR));
  const R M = Mp + Mm, ph = pp * L.p + pm * Q.p;
  const R fp = L.rho * ah * (R)0.5 * (M + fabs(M)), fm = Q.rho * ah * (R)0.5 * (M - fabs(M));
  fr = fp + fm;
  V2<R> m = fma2(dup2<R>(fp), L.A, dup2<R>(fm) * Q.A);
  fuv = fma2(dup2<R>(ph), mk2<R>(nx, ny), m);
  fw = fp * L.w + fm * Q.w + ph * nz;
  fe = fp * h0L + fm * h0R;
}

// The net flux (convective - viscous) along +d of the face between padded cell l0 of block b and its +d neighbour (gst
// further on), into out[0..4]; where vout is given (the records), the convective one into out and the viscous one into
// vout. c gives the states: c.stencil(q, A, B, C), q = 0..3, the four cells along d (1 and 2 the face's own);
// c.transverse(e, w, A, B) the neighbours along the two other axes e in increasing order (w = 0, 1: below / above cell 1;
// 2, 3: below / above cell 2).
template <typename R, bool VISC, int RS, int LIM, typename Cells>
__device__ __forceinline__ void face_core(const Params& p, const DBlk& b, int d, int l0, int gst, int face,
                                          const Cells& c, R* out, R* vout = nullptr) {
  R nx, ny, nz, area;
  face_rec(b, d, face, nx, ny, nz, area);
  if (nx == (R)0 && ny == (R)0 && nz == (R)0) area = (R)0;  // a degenerate face carries no flux
  // ---- the viscous flux first (its four values are fewer to keep than the face's two cells)
  V2<R> vuv;
  R vw, ve;
  R dl1, dl2;
  if (VISC) {
    V2<R> GnA, GnB, Gt;  // grad(.) . n of (u, v), (w, T); (grad u)^T n, x and y
    R Gtz, div;
    auto add_axis = [&](const V2<R>& gA, const V2<R>& gB, const V2<R>& m, R z, bool first) {
      const R mn_ = lo2(m) * nx + hi2(m) * ny + z * nz;
      const R gn = lo2(gA) * nx + hi2(gA) * ny + lo2(gB) * nz;
      const R dv = lo2(gA) * lo2(m) + hi2(gA) * hi2(m) + lo2(gB) * z;
      if (first) {
        GnA = dup2<R>(mn_) * gA; GnB = dup2<R>(mn_) * gB; Gt = dup2<R>(gn) * m; Gtz = gn * z; div = dv;
      } else {
        GnA = fma2(dup2<R>(mn_), gA, GnA); GnB = fma2(dup2<R>(mn_), gB, GnB); Gt = fma2(dup2<R>(gn), m, Gt);
        Gtz = gn * z + Gtz; div = div + dv;
      }
    };
    // differences along the axes, in quarters (the normal one times 4), and metric rows in halves: the factor 1/8 goes
    // into the viscosity
    const int ab = (d == 0) ? 1 : 0, ac = (d == 2) ? 1 : 2;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int ax = e ? ac : ab;
      V2<R> a0, b0, a1, b1, a2, b2, a3, b3;
      c.transverse(e, 0, a0, b0);
      c.transverse(e, 1, a1, b1);
      c.transverse(e, 2, a2, b2);
      c.transverse(e, 3, a3, b3);
      V2<R> m, m2;
      R z, z2, dd;
      metric(b, ax, l0, m, z, dd);
      metric(b, ax, l0 + gst, m2, z2, dd);
      add_axis((a1 - a0) + (a3 - a2), (b1 - b0) + (b3 - b2), m + m2, z + z2, e == 0);
    }
    V2<R> A1, B1, C1, A2, B2, C2, m, m2;
    R z, z2;
    c.stencil(1, A1, B1, C1);
    c.stencil(2, A2, B2, C2);
    metric(b, d, l0, m, z, dl1);
    metric(b, d, l0 + gst, m2, z2, dl2);
    const V2<R> four = dup2<R>((R)4);
    add_axis(four * (A2 - A1), four * (B2 - B1), m + m2, z + z2, false);
    R mu, kap;
    mu_k(p, (hi2(C1) + hi2(C2)) * Cst<R>::of(p).iri * rcp_(lo2(C1) + lo2(C2)), mu, kap);
    const R m8 = (R)0.125 * mu;
    const R td = (R)(-2.0 / 3.0) * div;
    const V2<R> S = fma2(dup2<R>(td), mk2<R>(nx, ny), GnA + Gt);  // stress . n / (mu / 8), x and y
    const R Sz = lo2(GnB) + Gtz + td * nz;
    const V2<R> Uf = A1 + A2;
    const R wk = (lo2(S) * lo2(Uf) + hi2(S) * hi2(Uf) + Sz * (lo2(B1) + lo2(B2))) * (R)0.5;
    vuv = dup2<R>(m8) * S;
    vw = m8 * Sz;
    ve = m8 * wk + (R)0.125 * kap * hi2(GnB);
  } else {
    dl1 = cell_dl<R>(b, d, l0);
    dl2 = cell_dl<R>(b, d, l0 + gst);
  }
  // ---- the limited face states from the four cells of the stencil
  Side<R> L, Q;
  {
    const R dl0 = cell_dl<R>(b, d, l0 - gst), dl3 = cell_dl<R>(b, d, l0 + 2 * gst);
    const R i0 = (R)2 * rcp_(dl0 + dl1), i1 = (R)2 * rcp_(dl1 + dl2), i2 = (R)2 * rcp_(dl2 + dl3);
    const V2<R> I0 = dup2<R>(i0), I1 = dup2<R>(i1), I2 = dup2<R>(i2), LM = dup2<R>((R)0.5 * dl1),
                LP = dup2<R>((R)-0.5 * dl2);
    auto face_states = [&](const V2<R>& q0, const V2<R>& q1, const V2<R>& q2, const V2<R>& q3, V2<R>& l, V2<R>& r) {
      const V2<R> a = (q1 - q0) * I0, e = (q2 - q1) * I1, f = (q3 - q2) * I2;
      V2<R> sl, sr;
      if (LIM == 3) {
        sl = albada(a, e, f, sr);
      } else {
        const int lim = LIM ? LIM : p.lim;
        sl = mk2<R>(slope_rt<R>(lim, lo2(e), lo2(a)), slope_rt<R>(lim, hi2(e), hi2(a)));
        sr = mk2<R>(slope_rt<R>(lim, lo2(f), lo2(e)), slope_rt<R>(lim, hi2(f), hi2(e)));
      }
      l = fma2(sl, LM, q1);
      r = fma2(sr, LP, q2);
    };
    V2<R> A[4], B[4], C[4], l, r;
#pragma unroll
    for (int q = 0; q < 4; ++q) c.stencil(q, A[q], B[q], C[q]);
    face_states(A[0], A[1], A[2], A[3], L.A, Q.A);
    if constexpr (sizeof(R) == 4) {  // w beside a T that nobody reads: the halves are independent
      face_states(B[0], B[1], B[2], B[3], l, r);
      L.w = lo2(l); Q.w = lo2(r);
    } else {
      // w alone: the pair's one division would mix in T, which has no value where a ghost that nothing fills is read (the
      // second layer of a periodic axis one cell deep, a face without records: zero density), and w would have none either
      const R a = (lo2(B[1]) - lo2(B[0])) * i0, e = (lo2(B[2]) - lo2(B[1])) * i1, f = (lo2(B[3]) - lo2(B[2])) * i2;
      R sl, sr;
      if (LIM == 3) {
        sl = albada(a, e, f, sr);
      } else {
        const int lim = LIM ? LIM : p.lim;
        sl = slope_rt<R>(lim, e, a);
        sr = slope_rt<R>(lim, f, e);
      }
      L.w = fma(sl, (R)0.5 * dl1, lo2(B[1]));
      Q.w = fma(sr, (R)-0.5 * dl2, lo2(B[2]));
    }
    face_states(C[0], C[1], C[2], C[3], l, r);
    L.rho = mx(lo2(l), (R)1e-20); Q.rho = mx(lo2(r), (R)1e-20);
    L.p = hi2(l); Q.p = hi2(r);
  }
  side_thermo<R>(p, L);
  side_thermo<R>(p, Q);
  R fr, fw, fe;
  V2<R> fuv;
  if (RS == 12) roe_pair<R>(p, L, Q, nx, ny, nz, fr, fuv, fw, fe);
  else if (RS == 1) hllc_pair<R>(p, L, Q, nx, ny, nz, fr, fuv, fw, fe);
  else ausm_pair<R>(p, L, Q, nx, ny, nz, fr, fuv, fw, fe);
  if (VISC && vout) {
    const V2<R> G = vuv * dup2<R>(area);
    vout[0] = (R)0;
    vout[MB_IU] = lo2(G);
    vout[MB_IV] = hi2(G);
    vout[MB_IW] = vw * area;
    vout[MB_IPR] = ve * area;
  } else if (VISC) {
    fuv = fuv - vuv;
    fw = fw - vw;
    fe = fe - ve;
  }
  const V2<R> F = fuv * dup2<R>(area);
  out[0] = fr * area;
  out[MB_IU] = lo2(F);
  out[MB_IV] = hi2(F);
  out[MB_IW] = fw * area;
  out[MB_IPR] = fe * area;
}

// the cells of an interior face in the state tile
template <typename R, int TY, bool KM, int NVT>
struct TileCells {
  const Tile<R, TY, NVT, KM>& T;
  int o0, o1, o2, o3;  // the stencil
  int bm, cm, cp;      // offsets below / above along the two transverse axes: -bm, bm; cm, cp
  __device__ __forceinline__ void stencil(int q, V2<R>& A, V2<R>& B, V2<R>& C) const {
    T.load(q == 0 ? o0 : q == 1 ? o1 : q == 2 ? o2 : o3, A, B, C);
  }
  __device__ __forceinline__ void transverse(int e, int w, V2<R>& A, V2<R>& B) const {
    T.load_uvwT((w < 2 ? o1 : o2) + (e == 0 ? ((w & 1) ? bm : -bm) : ((w & 1) ? cp : cm)), A, B);
  }
};

// One interior face of direction d between cell (i,j,k) and its +d neighbour from the state tile; (ii, jj): the tile
// coordinates of the cell
template <typename R, int TY, bool VISC, int RS, int LIM, bool KM, int NVT>
__device__ __forceinline__ void face_fast(const Params& p, const DBlk& b, const Tile<R, TY, NVT, KM>& T, int d, int i,
                                          int j, int k, int ii, int jj, R* out) {
  constexpr int VS = Tile<R, TY, NVT, KM>::VS;
  // the planes k-1 .. k+2 (a mirrored block's are its one plane)
  const int S0 = slot_of<KM>(k - 1) * VS, S1 = slot_of<KM>(k) * VS, S2 = slot_of<KM>(k + 1) * VS,
            S3 = slot_of<KM>(k + 2) * VS;
  const int st = (d == 0) ? 1 : TXH;
  const int o1 = jj * TXH + ii + S1;
  const TileCells<R, TY, KM, NVT> c{T, o1 + ((d == 2) ? S0 - S1 : -st), o1, o1 + ((d == 2) ? S2 - S1 : st),
                                    o1 + ((d == 2) ? S3 - S1 : 2 * st), (d == 0) ? TXH : 1,
                                    (d == 2) ? -TXH : S0 - S1, (d == 2) ? TXH : S2 - S1};
  face_core<R, VISC, RS, LIM>(p, b, d, lin32(b, i, j, k), (d == 0) ? 1 : (d == 1 ? b.pi : b.pi * b.pj),
                              fmi32(b, d, i, j, k), c, out);
}

// the cells of a connection record's face in the state arena: the boundary cell and the ghosts of its face, filled; the
// ghost's transverse neighbours are the donor's (the rows pg[2..5] of the record's table: -b, +b, -c, +c)
template <typename R>
struct ArenaCells {
  const double* P;
  long long nc, row1, st;  // row1: the lower cell of the face
  long long own, sb, sc;   // the boundary cell's row and its transverse strides
  const long long* pg;
  R iri;
  bool low;                // the boundary cell is the upper one (a low face)
  __device__ __forceinline__ void uvwT(long long r, V2<R>& A, V2<R>& B, V2<R>& C) const {
    const R rho = (R)P[r], u = (R)P[r + nc], v = (R)P[r + 2 * nc], w = (R)P[r + 3 * nc], pr = (R)P[r + 4 * nc];
    A = mk2<R>(u, v);
    B = mk2<R>(w, pr * iri * rcp_(rho));
    C = mk2<R>(rho, pr);
  }
  __device__ __forceinline__ void stencil(int q, V2<R>& A, V2<R>& B, V2<R>& C) const { uvwT(row1 + (q - 1) * st, A, B, C); }
  __device__ __forceinline__ void transverse(int e, int w, V2<R>& A, V2<R>& B) const {
    const bool mine = (w >= 2) == low;
    const long long s = e == 0 ? sb : sc;
    const long long r = mine ? own + ((w & 1) ? s : -s) : ld_row(pg + 2 + 2 * e + (w & 1));
    V2<R> C;
    uvwT(r, A, B, C);
  }
  __device__ __forceinline__ static long long ld_row(const long long* q) { return __ldg(q); }
};

// a connection record (bc_conn_eul and bc_conn_visc of mb_engine.cuh): its contributions A and S to the row of its cell.
// The two viscous fluxes the reference averages, with the gradients of the cell and of its ghost, are one flux with the
// mean gradient (the flux is linear in it): the interior face's.
template <typename R, bool VISC, int RS, int LIM>
__device__ __forceinline__ void conn_fast(const Params& p, const DBlk& b, const double* P, int i, int j,
                                          int k, int F, const long long* __restrict__ pg, R* A, R* S) {
  const int d = (F - 1) >> 1, low = F & 1;
  const int gst = (d == 0) ? 1 : (d == 1 ? b.pi : b.pi * b.pj);
  const int l = lin32(b, i, j, k);
  const int il = (d == 0) ? i - low : i, jl = (d == 1) ? j - low : j, kl = (d == 2) ? k - low : k;
  const int sk = b.kmirror ? 0 : b.pi * b.pj;  // a mirrored block's k ghosts are its k = 1 cells
  const ArenaCells<R> c{P, p.nc, b.boff + l - low * gst, gst, b.boff + l, (d == 0) ? b.pi : 1, (d == 2) ? b.pi : sk, pg,
                        Cst<R>::of(p).iri, low != 0};
  face_core<R, VISC, RS, LIM>(p, b, d, l - low * gst, gst, fmi32(b, d, il, jl, kl), c, A, S);
  if (low) {
#pragma unroll
    for (int s = 0; s < MB_NP; ++s) {
      A[s] = -A[s];
      if (VISC) S[s] = -S[s];
    }
  }
}

}  // namespace mb
