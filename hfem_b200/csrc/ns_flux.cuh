// Compressible Navier-Stokes flux F(u, q) and its Jacobian dF/d(u, q) at one
// point, for the HDG element kernels (sm_100a).
//
// Restates application/FM/nsNew/flux_ns2dNEW.c:22-74 / flux_ns3dNEW.c (the
// reference's symbolically generated flux, viscosity mu(u) from
// FM/getViscosity.c):
//   f_rho^d = m_d
//   f_mi^d  = m_i v_d + p delta_id + tau_id
//   f_E^d   = (E + p) v_d + sum_i tau_id v_i
//             + mu gamma/(Re Pr) (q_E^d/rho - E q_rho^d/rho^2 - sum_i v_i dv_i/dx_d)
// with dv_i/dx_d = (q_mi^d - v_i q_rho^d)/rho and
// tau_ij = (mu/Re)(dv_i/dx_j + dv_j/dx_i - 2/3 delta_ij div v).
// The trace flux's stabilization tensor (ns_stab_apply) and the boundary
// fluxes (ns_fbou_dual) follow.
// Variables: w = [rho, m_1..m_nd, E, q_1 (ncu comps), .., q_nd].
//
// The Jacobian is exact forward-mode differentiation (dual numbers).
#pragma once

namespace hfem {

template <int N>
struct Dual {
    double v;
    double d[N];
};

template <int N>
__device__ __forceinline__ Dual<N> dc(double v) {
    Dual<N> r;
    r.v = v;
#pragma unroll
    for (int i = 0; i < N; i++) r.d[i] = 0.0;
    return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator+(const Dual<N>& a, const Dual<N>& b) {
    Dual<N> r;
    r.v = a.v + b.v;
#pragma unroll
    for (int i = 0; i < N; i++) r.d[i] = a.d[i] + b.d[i];
    return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator-(const Dual<N>& a, const Dual<N>& b) {
    Dual<N> r;
    r.v = a.v - b.v;
#pragma unroll
    for (int i = 0; i < N; i++) r.d[i] = a.d[i] - b.d[i];
    return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator*(const Dual<N>& a, const Dual<N>& b) {
    Dual<N> r;
    r.v = a.v * b.v;
#pragma unroll
    for (int i = 0; i < N; i++) r.d[i] = a.d[i] * b.v + a.v * b.d[i];
    return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator*(double s, const Dual<N>& a) {
    Dual<N> r;
    r.v = s * a.v;
#pragma unroll
    for (int i = 0; i < N; i++) r.d[i] = s * a.d[i];
    return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator/(const Dual<N>& a, const Dual<N>& b) {
    Dual<N> r;
    const double ib = 1.0 / b.v;
    r.v = a.v * ib;
#pragma unroll
    for (int i = 0; i < N; i++) r.d[i] = (a.d[i] - r.v * b.d[i]) * ib;
    return r;
}

template <int N>
__device__ __forceinline__ Dual<N> datan(const Dual<N>& a) {
    Dual<N> r;
    r.v = atan(a.v);
    const double h = 1.0 / (1.0 + a.v * a.v);
#pragma unroll
    for (int i = 0; i < N; i++) r.d[i] = a.d[i] * h;
    return r;
}
template <int N>
__device__ __forceinline__ Dual<N> dpow15(const Dual<N>& a) {       // a^(3/2)
    Dual<N> r;
    r.v = pow(a.v, 1.5);
    const double h = 1.5 * sqrt(a.v);
#pragma unroll
    for (int i = 0; i < N; i++) r.d[i] = a.d[i] * h;
    return r;
}

// Sutherland's law (application/FM/getViscosity.c, sutherlandLaw2d 25-146 and
// sutherlandLaw3d 275-...; app.viscosityModel 1), regularised at zero: with the
// temperature T = (rE - |m|^2/(2 rho)) / (rho gamma (gamma - 1) Mach^2) and
// a = (S + T0) T^(3/2) / (S + T0 T), S = 111, T0 = 300,
//   mu = c + a (atan(b a)/pi + 1/2),  b = 100, c = 1/2 - atan(b)/pi.
template <int ND, int M>
__device__ __forceinline__ Dual<M> ns_sutherland(const double* __restrict__ param, const Dual<M>* w) {
    using D = Dual<M>;
    const double gam = param[0], mach = param[4], S = 111.0, T0 = 300.0, b = 100.0, pi = 3.141592653589793;
    D ke = dc<M>(0.0);
#pragma unroll
    for (int i = 0; i < ND; i++) ke = ke + w[1 + i] * w[1 + i];
    const D T = (w[ND + 1] - 0.5 * (ke / w[0])) / ((gam * (gam - 1.0) * mach * mach) * w[0]);
    const D a = (S + T0) * (dpow15(T) / (dc<M>(S) + T0 * T));
    return dc<M>(0.5 - atan(b) / pi) + a * ((1.0 / pi) * datan(b * a) + dc<M>(0.5));
}

// f[d*ncu + c] for one point; w has ND+2 + (ND+2)*ND entries, each carrying M
// partial derivatives (M = nc for the full Jacobian, 1 for one column of it).
// viscous == false: the Euler flux (flux_euler2dNEW.c / flux_euler3dNEW.c), the
// same expression without the stress and heat terms.  visc_model: 0 mu = 1,
// 1 Sutherland's law (ns_sutherland); GEN false compiles the constant-viscosity
// flux alone.
template <int ND, int M, bool GEN = false>
__device__ __forceinline__ void ns_flux_dual(const double* __restrict__ param, const Dual<M>* w, Dual<M>* f,
                                             bool viscous = true, int visc_model = 0) {
    constexpr int NCU = ND + 2;
    constexpr int NC = M;
    using D = Dual<M>;
    const double gam = param[0], Re = param[2], Pr = param[3];
    const double iRe = 1.0 / Re;
    const D& rho = w[0];
    const D& E = w[ND + 1];
    D v[ND];
    D ke = dc<NC>(0.0);
#pragma unroll
    for (int i = 0; i < ND; i++) {
        v[i] = w[1 + i] / rho;
        ke = ke + v[i] * w[1 + i];
    }
    const D p = (gam - 1.0) * (E - 0.5 * ke);
    D dv[ND][ND];
#pragma unroll
    for (int d = 0; d < ND; d++)
#pragma unroll
        for (int i = 0; i < ND; i++) dv[i][d] = (w[NCU * (1 + d) + 1 + i] - v[i] * w[NCU * (1 + d)]) / rho;
    D div = dv[0][0];
#pragma unroll
    for (int i = 1; i < ND; i++) div = div + dv[i][i];
    const double kappa = gam / (Re * Pr);
    const bool vm = GEN && viscous && visc_model != 0;
    D mu = dc<NC>(1.0);
    if constexpr (GEN) {
        if (vm) mu = ns_sutherland<ND, M>(param, w);
    }
#pragma unroll
    for (int d = 0; d < ND; d++) {
        f[d * NCU + 0] = w[1 + d];
        D fe = (E + p) * v[d];
        D vdv = dc<NC>(0.0);
#pragma unroll
        for (int i = 0; i < ND; i++) {
            D t = dv[i][d] + dv[d][i];
            if (i == d) t = t - (2.0 / 3.0) * div;
            t = viscous ? iRe * (vm ? mu * t : t) : dc<NC>(0.0);   // tau_id
            D fm = w[1 + i] * v[d] + t;
            if (i == d) fm = fm + p;
            f[d * NCU + 1 + i] = fm;
            fe = fe + t * v[i];
            vdv = vdv + v[i] * dv[i][d];
        }
        const D heat = w[NCU * (1 + d) + ND + 1] / rho - E * w[NCU * (1 + d)] / (rho * rho) - vdv;
        f[d * NCU + ND + 1] = viscous ? fe + kappa * (vm ? mu * heat : heat) : fe;
    }
}

// The flux through one direction X, F(w).X = sum_d f_d X_d, and its Jacobian
// columns without dual numbers, for the element kernel's FP64 form: X is a row of
// the volume point's metric or the face point's scaled normal, so what is formed
// is what the element integrals need, and no product with a zero derivative.
// NsDir holds the terms that the columns share.
template <int ND>
struct NsDir {
    double ir, rho, E, p, v[ND], v2;
    double X[ND], q0[ND];
    double Vn, Q0n, qEn, div;   // v.X, grad(rho).X, grad(rho E).X, div v
    double Gn[ND], Hn[ND];      // sum_d dv_i/dx_d X_d,  sum_d dv_d/dx_i X_d
    double a, kap;              // mu / Re, mu gamma / (Re Pr); 0 for the Euler flux
};

// iRe = 1/Re and kappa = gamma/(Re Pr), both 0 for the Euler flux
template <int ND>
__device__ __forceinline__ void ns_dir(double gam, double iRe, double kappa, double mu, const double* w,
                                       const double* X, NsDir<ND>& s) {
    constexpr int NCU = ND + 2;
    s.rho = w[0];
    s.E = w[ND + 1];
    s.ir = 1.0 / w[0];
    s.v2 = s.Vn = s.Q0n = s.qEn = s.div = 0.0;
#pragma unroll
    for (int i = 0; i < ND; i++) {
        s.X[i] = X[i];
        s.v[i] = w[1 + i] * s.ir;
        s.v2 = fma(s.v[i], s.v[i], s.v2);
        s.Vn = fma(s.v[i], X[i], s.Vn);
        s.q0[i] = w[NCU * (1 + i)];
        s.Q0n = fma(s.q0[i], X[i], s.Q0n);
        s.qEn = fma(w[NCU * (1 + i) + ND + 1], X[i], s.qEn);
        s.Gn[i] = s.Hn[i] = 0.0;
    }
    s.p = (gam - 1.0) * fma(-0.5 * s.rho, s.v2, s.E);
#pragma unroll
    for (int d = 0; d < ND; d++)
#pragma unroll
        for (int i = 0; i < ND; i++) {
            const double g = fma(-s.v[i], s.q0[d], w[NCU * (1 + d) + 1 + i]) * s.ir;   // dv_i/dx_d
            s.Gn[i] = fma(g, X[d], s.Gn[i]);
            s.Hn[d] = fma(g, X[i], s.Hn[d]);
            if (i == d) s.div += g;
        }
    s.a = iRe * mu;
    s.kap = kappa * mu;
}

// The flux F.X alone: val(j, F_j).
template <int ND, class Val>
__device__ __forceinline__ void ns_dir_value(const NsDir<ND>& s, Val val) {
    double vt = 0.0, vG = 0.0;
    val(0, s.rho * s.Vn);
#pragma unroll
    for (int i = 0; i < ND; i++) {
        const double tn = s.a * (s.Gn[i] + s.Hn[i] - (2.0 / 3.0) * s.div * s.X[i]);
        vt = fma(s.v[i], tn, vt);
        vG = fma(s.v[i], s.Gn[i], vG);
        val(1 + i, fma(s.rho * s.v[i], s.Vn, fma(s.p, s.X[i], tn)));
    }
    const double heat = s.qEn * s.ir - s.E * s.Q0n * (s.ir * s.ir) - vG;
    val(ND + 1, fma(s.E + s.p, s.Vn, fma(s.kap, heat, vt)));
}

// The flux F.X and its columns along the conserved variables: val(j, F_j) and
// col(k, j, dF_j/du_k).  dmu[k] = dmu/du_k (GEN; NULL: constant viscosity).
template <int ND, class Val, class Col>
__device__ __forceinline__ void ns_dir_u(double gam, double iRe, double kappa, const double* dmu, const NsDir<ND>& s,
                                         Val val, Col col) {
    const double g1 = gam - 1.0, ir2 = s.ir * s.ir, c23 = 2.0 / 3.0;
    double sh[ND], tn[ND], vG = 0.0;                 // stress without mu/Re, stress, v.Gn
#pragma unroll
    for (int i = 0; i < ND; i++) {
        sh[i] = s.Gn[i] + s.Hn[i] - c23 * s.div * s.X[i];
        tn[i] = s.a * sh[i];
        vG = fma(s.v[i], s.Gn[i], vG);
    }
    const double heat = s.qEn * s.ir - s.E * s.Q0n * ir2 - vG, EP = s.E + s.p;
    ns_dir_value<ND>(s, val);
    // what a viscosity derivative adds to column k
    auto visc = [&](int k, int i) { return dmu ? iRe * dmu[k] * sh[i] : 0.0; };
    auto visc_e = [&](int k) {
        if (!dmu) return 0.0;
        double t = kappa * dmu[k] * heat;
#pragma unroll
        for (int i = 0; i < ND; i++) t = fma(iRe * dmu[k] * s.v[i], sh[i], t);
        return t;
    };
    // along rho: dv = -v/rho
    {
        double vq = 0.0;
#pragma unroll
        for (int i = 0; i < ND; i++) vq = fma(s.v[i], s.q0[i], vq);
        const double dVn = -s.Vn * s.ir, dp = 0.5 * g1 * s.v2, ddiv = fma(vq, s.ir, -s.div) * s.ir;
        double et = 0.0, vdG = 0.0;
        col(0, 0, 0.0);
#pragma unroll
        for (int i = 0; i < ND; i++) {
            const double dG = fma(s.v[i] * s.ir, s.Q0n, -s.Gn[i]) * s.ir;
            const double dH = fma(s.q0[i], s.Vn * s.ir, -s.Hn[i]) * s.ir;
            const double dt = fma(s.a, dG + dH - c23 * ddiv * s.X[i], visc(0, i));
            // stress: v.dt + dv.t; heat: -(dv.Gn + v.dGn)
            et = fma(s.v[i], fma(-tn[i], s.ir, dt), et);
            vdG = fma(s.v[i], fma(-s.Gn[i], s.ir, dG), vdG);
            col(0, 1 + i, fma(s.rho * s.v[i], dVn, fma(dp, s.X[i], dt)));
        }
        const double dheat = fma(-s.qEn, ir2, 2.0 * s.E * s.Q0n * ir2 * s.ir) - vdG;
        double mu_e = dmu ? kappa * dmu[0] * heat : 0.0;
        col(0, ND + 1, fma(dp, s.Vn, fma(EP, dVn, fma(s.kap, dheat, et + mu_e))));
    }
    // along the momentum: dv_l = 1/rho
#pragma unroll
    for (int l = 0; l < ND; l++) {
        const double dVn = s.X[l] * s.ir, dp = -g1 * s.v[l], ddiv = -s.q0[l] * ir2, dGl = -s.Q0n * ir2;
        double et = tn[l] * s.ir;
        col(1 + l, 0, s.X[l]);
#pragma unroll
        for (int i = 0; i < ND; i++) {
            const double dt = fma(s.a, (i == l ? dGl : 0.0) - s.q0[i] * dVn * s.ir - c23 * ddiv * s.X[i], visc(1 + l, i));
            et = fma(s.v[i], dt, et);
            col(1 + l, 1 + i, fma(s.rho * s.v[i], dVn, fma(dp, s.X[i], dt)) + (i == l ? s.Vn : 0.0));
        }
        const double dheat = -fma(s.Gn[l], s.ir, s.v[l] * dGl);
        double mu_e = dmu ? kappa * dmu[1 + l] * heat : 0.0;
        col(1 + l, ND + 1, fma(dp, s.Vn, fma(EP, dVn, fma(s.kap, dheat, et + mu_e))));
    }
    // along the energy
    col(ND + 1, 0, 0.0);
#pragma unroll
    for (int i = 0; i < ND; i++) col(ND + 1, 1 + i, fma(g1, s.X[i], visc(ND + 1, i)));
    col(ND + 1, ND + 1, fma(gam, s.Vn, fma(-s.kap, s.Q0n * ir2, visc_e(ND + 1))));
}

// The columns along the gradients: col(dq, m, j, dF_j/dq_{dq,m}) for the pairs
// (j, m) that depend on them (NsPairs); the flux is linear in q, so a column is
// the flux of the unit gradient.
template <int ND, class Col>
__device__ __forceinline__ void ns_dir_q(const NsDir<ND>& s, Col col) {
    const double ai = s.a * s.ir, ki = s.kap * s.ir, c23 = 2.0 / 3.0;
#pragma unroll
    for (int dq = 0; dq < ND; dq++) {
        const double X = s.X[dq];
        // m = 0: g_i = -v_i/rho
#pragma unroll
        for (int i = 0; i < ND; i++)
            col(dq, 0, 1 + i, -ai * (fma(s.v[i], X, -c23 * s.v[dq] * s.X[i]) + (i == dq ? s.Vn : 0.0)));
        col(dq, 0, ND + 1, fma(-ai, fma(s.v2, X, (1.0 - c23) * s.v[dq] * s.Vn), ki * fma(-s.E, s.ir, s.v2) * X));
        // m = 1 + l: g_l = 1/rho
#pragma unroll
        for (int l = 0; l < ND; l++) {
#pragma unroll
            for (int i = 0; i < ND; i++) {
                double t = 0.0;
                if (i == l) t = X;
                if (i == dq) t += s.X[l];
                if (l == dq) t -= c23 * s.X[i];
                col(dq, 1 + l, 1 + i, ai * t);
            }
            double e = fma(s.v[l], X, s.v[dq] * s.X[l]);
            if (l == dq) e = fma(-c23, s.Vn, e);
            col(dq, 1 + l, ND + 1, fma(ai, e, -ki * s.v[l] * X));
        }
        col(dq, ND + 1, ND + 1, ki * X);
    }
}

// The (equation j, variable m) pairs in two groups, those whose flux depends on
// the gradient of m first: j = 1..nd+1 with m = 0..nd, and (nd+1, nd+1).  The
// rest, mass with any variable and momentum with the energy, have zero d' > 0
// columns in every volume, trace and boundary flux of this file (17 of 25 pairs
// in 3D and 10 of 16 in 2D depend on gradients).
template <int ND>
struct NsPairs {
    static constexpr int NCU = ND + 2, ALL = NCU * NCU, DEP = (ND + 1) * (ND + 1) + 1;
    static __device__ __forceinline__ void at(int p, int& j, int& m) {
        if (p < DEP - 1) {
            j = 1 + p % (ND + 1);
            m = p / (ND + 1);
        } else if (p == DEP - 1) {
            j = m = ND + 1;
        } else if (p < DEP + NCU) {
            j = 0;
            m = p - DEP;
        } else {
            j = 1 + p - DEP - NCU;
            m = ND + 1;
        }
    }
};

template <int N>
__device__ __forceinline__ Dual<N> dsqrt(const Dual<N>& a) {
    Dual<N> r;
    r.v = sqrt(a.v);
    const double h = 0.5 / r.v;
#pragma unroll
    for (int i = 0; i < N; i++) r.d[i] = a.d[i] * h;
    return r;
}
template <int N>
__device__ __forceinline__ Dual<N> dabs(const Dual<N>& a) {
    return a.v < 0.0 ? (-1.0) * a : a;
}

// Free-stream far field (application/FM/fbou.cpp:126-218):
//   fb = (A_n + |A_n|)(u - uh) - (A_n - |A_n|)(ui - uh)
// with the Euler normal-flux Jacobian A_n at uh and |A_n| = R |Lambda| R^-1 in the
// closed form of application/FM/getan.c (eigenvalues un + c, un - c, un; with
// eps > 0 the eigenvalues below eps c are smoothed as there).  Column k of
// either matrix is lam3 e_k + cc1_k [1, v, h] + cc2_k [0, n, un]; the matrices
// are applied column by column without being stored.
template <int ND, int M>
__device__ __forceinline__ void ns_farfield_dual(const double* __restrict__ param, const double* ui, const double* nl,
                                                 const Dual<M>* w, const Dual<M>* uh, Dual<M>* fb) {
    constexpr int NCU = ND + 2;
    using D = Dual<M>;
    const double gam = param[0], eps = param[1], g1 = gam - 1.0;
    const D r = uh[0];
    D uv[ND], af = dc<M>(0.0), un = dc<M>(0.0);
#pragma unroll
    for (int i = 0; i < ND; i++) {
        uv[i] = uh[1 + i] / r;
        af = af + 0.5 * (uv[i] * uv[i]);
        un = un + nl[i] * uv[i];
    }
    const D E = uh[ND + 1] / r;
    const D p = g1 * (uh[ND + 1] - r * af);
    const D h = E + p / r;
    const D c2 = gam * (p / r);
    const D c = dsqrt(c2);
    D la[3] = {un + c, un - c, un}, lb[3];
#pragma unroll
    for (int m = 0; m < 3; m++) {
        lb[m] = dabs(la[m]);
        if (eps > 0.0 && lb[m].v < eps * c.v) lb[m] = 0.5 * (lb[m] * lb[m] / (eps * c) + eps * c);
    }
    const D s1a = 0.5 * (la[0] + la[1]), s2a = 0.5 * (la[0] - la[1]);
    const D s1b = 0.5 * (lb[0] + lb[1]), s2b = 0.5 * (lb[0] - lb[1]);
#pragma unroll
    for (int j = 0; j < NCU; j++) fb[j] = dc<M>(0.0);
#pragma unroll
    for (int k = 0; k < NCU; k++) {
        const D a = (k == 0) ? af : (k == ND + 1 ? dc<M>(1.0) : dc<M>(0.0) - uv[k > 0 ? k - 1 : 0]);
        const D b = (k == 0) ? dc<M>(0.0) - un : (k == ND + 1 ? dc<M>(0.0) : dc<M>(nl[k > 0 ? k - 1 : 0]));
        const D c1a = g1 * ((s1a - la[2]) * a / c2) + s2a * b / c, c2a = g1 * (s2a * a / c) + (s1a - la[2]) * b;
        const D c1b = g1 * ((s1b - lb[2]) * a / c2) + s2b * b / c, c2b = g1 * (s2b * a / c) + (s1b - lb[2]) * b;
        const D du = w[k] - uh[k], di = dc<M>(ui[k]) - uh[k];
#pragma unroll
        for (int j = 0; j < NCU; j++) {
            const D v1 = (j == 0) ? dc<M>(1.0) : (j == ND + 1 ? h : uv[j > 0 ? j - 1 : 0]);
            const D v2 = (j == 0) ? dc<M>(0.0) : (j == ND + 1 ? un : dc<M>(nl[j > 0 ? j - 1 : 0]));
            D Aa = c1a * v1 + c2a * v2, Ab = c1b * v1 + c2b * v2;
            if (j == k) {
                Aa = Aa + la[2];
                Ab = Ab + lb[2];
            }
            fb[j] = fb[j] + (Aa + Ab) * du - (Aa - Ab) * di;
        }
    }
}

// out = tau(uh) v, the convective stabilization tensor of the trace flux
// (application/FM/stabilizationTensor.cpp, getConvectiveStabilizationTensor
// 3439-3456; app.convStabMethod):
//   0 constant: param[5] v (getConstantStabilizationTensor, 9-29);
//   1 Lax-Friedrichs: lam v, lam = |un| + c at uh (3D, 221-425); the 2D routine
//     (31-218) evaluates lam at the fixed state (rho, rho u, rho v, rho E) =
//     (1, 0.9994, 0.0349, 1.7858e4) and has a zero Jacobian: restated as it is;
//   2 Roe (440-1716): |A_n(uh)| v, eigenvalues un + c, un - c, un through the
//     smooth absolute value r(x) = 2 (x (atan(b x)/pi + 1/2) - atan(b)/pi +
//     1/2) - x, b = 10, and, with eps = param[1] > 0, r < eps c replaced by
//     (r^2/(eps c) + eps c)/2; columns lam3 e_k + cc1_k [1, v, h] + cc2_k [0, n, un].
template <int ND, int M>
__device__ __forceinline__ void ns_stab_apply(int method, const double* __restrict__ param, const double* nl,
                                              const Dual<M>* uh, const Dual<M>* v, Dual<M>* out) {
    constexpr int NCU = ND + 2;
    using D = Dual<M>;
    if (method == 0) {
#pragma unroll
        for (int j = 0; j < NCU; j++) out[j] = param[5] * v[j];
        return;
    }
    const double gam = param[0], g1 = gam - 1.0, eps = param[1];
    if (method == 1) {
        D lam;
        if constexpr (ND == 2) {
            const double r = 1.0, ru = 0.9994, rv = 0.0349, rE = 1.7858e+04;
            const double uv = ru / r, vv = rv / r, af = 0.5 * (uv * uv + vv * vv), p = g1 * (rE - r * af);
            const double c = sqrt(gam * p / r), un = uv * nl[0] + vv * nl[1];
            lam = dc<M>(un >= 0 ? un + c : -un + c);
        } else {
            const D r = uh[0];
            D af = dc<M>(0.0), un = dc<M>(0.0);
#pragma unroll
            for (int i = 0; i < ND; i++) {
                const D vi = uh[1 + i] / r;
                af = af + 0.5 * (vi * vi);
                un = un + nl[i] * vi;
            }
            const D p = g1 * (uh[ND + 1] - r * af);
            const D c = dsqrt(gam * (p / r));
            lam = un.v >= 0 ? un + c : c - un;
        }
#pragma unroll
        for (int j = 0; j < NCU; j++) out[j] = lam * v[j];
        return;
    }
    const double b = 10.0, pi = 3.141592653589793;
    const D r = uh[0];
    D uv[ND], af = dc<M>(0.0), un = dc<M>(0.0);
#pragma unroll
    for (int i = 0; i < ND; i++) {
        uv[i] = uh[1 + i] / r;
        af = af + 0.5 * (uv[i] * uv[i]);
        un = un + nl[i] * uv[i];
    }
    const D E = uh[ND + 1] / r;
    const D p = g1 * (uh[ND + 1] - r * af);
    const D h = E + p / r;
    const D c2 = gam * (p / r);
    const D c = dsqrt(c2);
    D rl[3] = {un + c, un - c, un};
#pragma unroll
    for (int m = 0; m < 3; m++) {
        const D x = rl[m];
        rl[m] = 2.0 * (x * ((1.0 / pi) * datan(b * x) + dc<M>(0.5)) + dc<M>(0.5 - atan(b) / pi)) - x;
        if (eps > 0.0 && rl[m].v < eps * c.v) rl[m] = 0.5 * (rl[m] * rl[m] / (eps * c) + eps * c);
    }
    const D s1 = 0.5 * (rl[0] + rl[1]), s2 = 0.5 * (rl[0] - rl[1]), l3 = rl[2];
#pragma unroll
    for (int j = 0; j < NCU; j++) out[j] = dc<M>(0.0);
#pragma unroll
    for (int k = 0; k < NCU; k++) {
        const D a = (k == 0) ? af : (k == ND + 1 ? dc<M>(1.0) : dc<M>(0.0) - uv[k > 0 ? k - 1 : 0]);
        const D bb = (k == 0) ? dc<M>(0.0) - un : (k == ND + 1 ? dc<M>(0.0) : dc<M>(nl[k > 0 ? k - 1 : 0]));
        const D cc1 = g1 * ((s1 - l3) * a / c2) + s2 * bb / c;
        const D cc2 = g1 * (s2 * a / c) + (s1 - l3) * bb;
#pragma unroll
        for (int j = 0; j < NCU; j++) {
            const D v1 = (j == 0) ? dc<M>(1.0) : (j == ND + 1 ? h : uv[j > 0 ? j - 1 : 0]);
            const D v2 = (j == 0) ? dc<M>(0.0) : (j == ND + 1 ? un : dc<M>(nl[j > 0 ? j - 1 : 0]));
            D m = cc1 * v1 + cc2 * v2;
            if (j == k) m = m + l3;
            out[j] = out[j] + m * v[k];
        }
    }
}

// The stabilization term of fhat at one face point for the element kernel's
// flux pass: sv = tau(uh)(u - uh), sd = its derivative along uh_k (k < ncu;
// 0 otherwise), tcol = column k of tau (k < ncu).
template <int ND>
__device__ __forceinline__ void ns_stab_point(int method, const double* __restrict__ param, const double* nl,
                                           const double* uh, const double* u, int k, double* sv, double* sd,
                                           double* tcol) {
    constexpr int NCU = ND + 2;
    using DD = Dual<1>;
    DD uhd[NCU], dv[NCU], st[NCU];
#pragma unroll
    for (int m = 0; m < NCU; m++) {
        uhd[m].v = uh[m];
        uhd[m].d[0] = (m == k) ? 1.0 : 0.0;
        dv[m] = dc<1>(u[m]) - uhd[m];
    }
    ns_stab_apply<ND, 1>(method, param, nl, uhd, dv, st);
#pragma unroll
    for (int j = 0; j < NCU; j++) {
        sv[j] = st[j].v;
        sd[j] = st[j].d[0];
    }
    if (k < NCU) {
#pragma unroll
        for (int m = 0; m < NCU; m++) {
            uhd[m] = dc<1>(uh[m]);
            dv[m] = dc<1>(m == k ? 1.0 : 0.0);
        }
        ns_stab_apply<ND, 1>(method, param, nl, uhd, dv, st);
#pragma unroll
        for (int j = 0; j < NCU; j++) tcol[j] = st[j].v;
    }
}

// Boundary flux fb(u, q, uh) of the NS boundary conditions at one point
// (application/FM/fbou.cpp on a fixed mesh), in dual numbers so that one pass
// per differentiated variable gives fb and its derivative:
//   1 free-stream far field (ns_farfield_dual);
//   2 no-slip adiabatic wall: rho - rho_hat, -m_hat, and for energy the
//     interior trace flux F(uh, q).n + [tau(uh) (u - uh)]_E (ns_stab_apply);
//   5 Dirichlet: tau (ui - uh);   6 extrapolation: u - uh;
//   7 slip wall: rho - rho_hat, m - (m.n) n - m_hat, E - E_hat.
// w holds (u, q) (NC entries), uh the trace state (NCH); returns false for a
// type without a restatement.
template <int ND, int M, bool GEN = false>
__device__ __forceinline__ bool ns_fbou_dual(int bn, const double* __restrict__ param, const double* ui,
                                             const double* nl, const Dual<M>* w, const Dual<M>* uh, Dual<M>* fb,
                                             bool viscous = true, int conv_stab = 0, int visc_model = 0) {
    constexpr int NCU = ND + 2, NC = NCU * (ND + 1);
    const double tau = param[5];
    if (bn == 1) {
        ns_farfield_dual<ND, M>(param, ui, nl, w, uh, fb);
        return true;
    }
    if (bn == 2) {
        fb[0] = w[0] - uh[0];
#pragma unroll
        for (int j = 0; j < ND; j++) fb[1 + j] = dc<M>(0.0) - uh[1 + j];
        Dual<M> wf[NC], f[ND * NCU];
#pragma unroll
        for (int k = 0; k < NCU; k++) wf[k] = uh[k];
#pragma unroll
        for (int k = NCU; k < NC; k++) wf[k] = w[k];
        ns_flux_dual<ND, M, GEN>(param, wf, f, viscous, visc_model);
        Dual<M> t;
        if (!GEN || conv_stab == 0) {
            t = tau * (w[ND + 1] - uh[ND + 1]);
        } else {
            Dual<M> du[NCU], st[NCU];
#pragma unroll
            for (int k = 0; k < NCU; k++) du[k] = w[k] - uh[k];
            ns_stab_apply<ND, M>(conv_stab, param, nl, uh, du, st);
            t = st[ND + 1];
        }
#pragma unroll
        for (int d = 0; d < ND; d++) t = t + nl[d] * f[d * NCU + ND + 1];
        fb[ND + 1] = t;
        return true;
    }
    if (bn == 5) {
#pragma unroll
        for (int j = 0; j < NCU; j++) fb[j] = tau * (dc<M>(ui[j]) - uh[j]);
        return true;
    }
    if (bn == 6) {
#pragma unroll
        for (int j = 0; j < NCU; j++) fb[j] = w[j] - uh[j];
        return true;
    }
    if (bn == 7) {
        fb[0] = w[0] - uh[0];
        Dual<M> un = dc<M>(0.0);
#pragma unroll
        for (int i = 0; i < ND; i++) un = un + nl[i] * w[1 + i];
#pragma unroll
        for (int j = 0; j < ND; j++) fb[1 + j] = w[1 + j] - nl[j] * un - uh[1 + j];
        fb[ND + 1] = w[ND + 1] - uh[ND + 1];
        return true;
    }
    return false;
}

}  // namespace hfem
