// Physical-space stage on (theta, pi - theta) row pairs:
//   Phi_Derivatives           (Sphere_Physical_Space.F90:745-759) in the spectrum load,
//   fft_to_physical  (c2r)    (Fourier_Transform.F90:142-183), 14 or 20 fields,
//   sintheta_div + NL terms   (Sphere_Physical_Space.F90:98-224, 303-700),
//   Find_MyMinDT (CFL max)    (:784-813),
//   fft_to_spectral (r2c)     (Fourier_Transform.F90:100-140), 4 or 7 fields,
//   equatorial fold of PtS    (Legendre_Transforms.F90:1109-1122),
// reading the inverse Legendre output p2a[theta_h][m][par][r][f][re/im] (E, O) and
// writing the folded p2b[m][par][theta_h][r][f][re/im] for m <= l_max.  The
// reference materialises the packed (n_phi+2, r, theta, f) buffers p3a/p3b
// between these steps; here the rows of one (r, theta pair) never leave the SM.
// The transform and its layout: phi_pair.cuh.
//
// What bounds it: at most twelve warps an SM (168 registers hold the velocity or B and a batch's
// points, 8 M slots of shared memory a batch and the four outputs; at M = 1024 eight, the shared memory of
// one CTA of 256 threads, which take 238 to 255 registers), which wait in turn on loads, barriers and shared
// memory; the data pipe is 68 % busy at M = 1536.  Against one CTA of 384 threads per row with
// half-length transforms, per step: n_theta 64, N_r 48 127.6 -> 31 us; 192 polytrope, N_r 128 1331 -> 588;
// 384 anelastic MHD, N_r 128 6751 -> 3811; 512, N_r 64 hydrodynamic 4.73 -> 2.51 ms, dynamo 7.31 -> 3.82,
// anelastic MHD 7.53 -> 3.99; 768 dynamo, N_r 96 16.56 -> 12.4.  At M = 1536 the heating terms spill (384 bytes
// without B, 228 with): 768, N_r 64 polytrope 7.45 -> 6.03 ms, anelastic MHD 11.60 -> 9.31, against
// 5.62 and 8.30 without heating.
#include <cmath>
#include <vector>

#include "phi_pair.cuh"
#include "ra_internal.h"

namespace ra {

// r2c and equatorial fold of NB fields whose radix-4 pass is done (this thread's points written to
// buf): the mid passes, then per item the values Z_m, Z_{-m}, S_m and N_m times hsf(b), and
// f_even = S + N, f_odd = S - N into p2b at obase + m mstride (+ par pstride) + 2 b.
template <int M, int NB, class HS>
__device__ __forceinline__ void pair_r2c(const PhysParams& P, double* __restrict__ obase, int L, long mstride,
                                         long pstride, double2* buf, int tt, const HS& hsf) {
    using S = Pair<M>;
    constexpr int F = S::F, Q = S::Q, T = S::T, NITEM = NB * (Q / 2);
    __syncthreads();
    pair_mid_pass<M, NB, S::R2, 4 * S::R2, true>(buf, P.twq + S::TW2, tt);
    if constexpr (S::R1 > 1) {
        mid_barrier<M>(tt);
        pair_mid_pass<M, NB, S::R1, Q, true>(buf, P.twq, tt);
    }
    __syncthreads();
#pragma unroll 1
    for (int q = tt; q < NITEM; q += T) {
        int k, b;
        pair_item<M, NB>(q, k, b);
        const bool self = k == 0;
        const int kp = self ? Q / 2 : Q - k;
        const double2* fb = buf + b * M;
        const double2 w = __ldg(P.wr + (self ? kp : k));
        double2 ua[F], ub[F];
        ua[0] = fb[swz<M>(k)];
        ub[0] = fb[swz<M>(kp)];
        double2 wj = w;
#pragma unroll
        for (int j = 1; j < F; ++j) {
            const double2 a = fb[swz<M>(j * Q + k)];
            ua[j] = self ? a : cmul(a, cconj(wj));
            ub[j] = cmul(fb[swz<M>(j * Q + kp)], wj);
            if (j + 1 < F) wj = cmul(wj, w);
        }
        // a: Z at k, k + Q, -(Q - k + Q), -(Q - k); b: Z at -k, -(k + Q), kp + Q, kp
        double2 a0, a1, a2, a3, b0, b1, b2, b3, ax;
        dft_to4<F, -1>(ua, a0, a1, a2, a3, &ax);
        dft_to4<F, 1>(ub, b0, b1, b2, b3);
        const double hs = hsf(b);
        double* out = obase + 2 * b;
        auto put = [&](int m, double2 zp, double2 zm) {
            if (m < L) {
                const double2 s = make_double2(hs * (zp.x + zm.x), hs * (zp.y - zm.y));
                const double2 n = make_double2(hs * (zp.y + zm.y), hs * (zm.x - zp.x));
                *reinterpret_cast<double2*>(out + m * mstride) = cadd(s, n);
                *reinterpret_cast<double2*>(out + m * mstride + pstride) = csub(s, n);
            }
        };
        put(k, a0, self ? a0 : b0);
        put(k + Q, a1, self ? a3 : b1);
        put(kp, b3, self ? b0 : a3);
        put(kp + Q, b2, self ? b1 : a2);
        if (F == 6 && self) put(2 * Q, ax, a2);   // m = M/3 = l_max
    }
}

// One CTA = G radii of one theta pair, M/4 threads each.
template <int M, int G, int MINB, bool MAG, bool HEAT>
__global__ void __launch_bounds__(G* M / 4, MINB) physics_pair_kernel(PhysParams P) {
    constexpr int T = Pair<M>::T, NT = G * T, NTH = M / 2;
    // The next batch's spectra come in under this one's terms, except in the largest plans (two radix-8
    // mid passes): with both the staging and up to six transforms inlined their code outgrows the
    // instruction cache (M = 1536 with B, N_r = 96: 16.2 ms staged, 12.4 direct; M = 768 with B and
    // heating, N_r = 128: 3.81 / 3.83 ms, M = 384 with heating 588 / 667 us, with B, N_r = 64,
    // 451 / 515, M = 256 195 / 218).
    constexpr bool STAGED = Pair<M>::R1 < 8;
    static_assert(NT % 32 == 0, "whole warps");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double red[NT / 32];
    __shared__ double rowc_all[G][RC_COUNT];
    const int t = threadIdx.x;
    const int g = G == 1 ? 0 : t / T, tt = t - g * T;
    const int nr = P.nr;
    const int nrb = (nr + G - 1) / G;
    const int thh = blockIdx.x / nrb;
    const int r = (blockIdx.x - thh * nrb) * G + g;
    const int L = r < nr ? P.L : 0;
    double2* buf = reinterpret_cast<double2*>(smem_raw) + g * (8 * M);   // 4 fields
    double2* acc = buf + 4 * M;                                           // W, P, T, Z
    double* rowc = rowc_all[g];
    const double* rowbase = P.p2a + (long)thh * (2L * P.L * P.ncola) + (long)r * (2 * P.nfa);
    const long mstride = 2L * (P.nth / 2) * P.ncolb, pstride = (long)(P.nth / 2) * P.ncolb;
    double* obase = P.p2b + (long)thh * P.ncolb + (long)r * (2 * P.nfb);
    if (tt == 0) {   // cos and cot change sign on the north row
        const int rr = r < nr ? r : nr - 1;
        const double csc = P.trig[2 * NTH + thh], orad = P.radial[R_OVER_R * nr + rr];
        rowc[RC_RAD] = P.radial[R_RADIUS * nr + rr];
        rowc[RC_ORAD] = orad;
        rowc[RC_RHO] = P.radial[R_DENSITY * nr + rr];
        rowc[RC_DLNRHO] = P.radial[R_DLNRHO * nr + rr];
        rowc[RC_DR] = P.radial[R_DELTA_R * nr + rr];
        rowc[RC_CS] = P.trig[thh];
        rowc[RC_SN] = P.trig[NTH + thh];
        rowc[RC_CSC] = csc;
        rowc[RC_COT] = P.trig[3 * NTH + thh];
        rowc[RC_COR] = P.rotation ? P.coriolis : 0.0;
        rowc[RC_C2R] = csc * csc * orad;
        rowc[RC_HSF] = 0.5 * (P.radial[R_DENSITY * nr + rr] * P.radial[R_RADIUS * nr + rr] * csc);
        rowc[RC_VH] = P.radial[R_VISC_HEAT * nr + rr];
        rowc[RC_OH] = P.radial[R_OHM_HEAT * nr + rr];
    }   // read after pair_c2r's first barrier

    double2 vr[4], vt[4], vp[4];   // (south, north)
    double2 y[4][4];
    auto acc_at = [&](int f, int i) -> double2& { return acc[f * M + swz<M>(4 * tt + i)]; };
    if constexpr (HEAT) {
        // The anelastic form: the same terms, with the viscous heating
        // (Compute_Viscous_Heating, Sphere_Physical_Space.F90:337-443) in T's accumulator.
        // Its strain-rate components are products across fields, so the batches are
        // grouped for each component to complete inside one batch:
        //   H1: v_r, v_theta, v_phi
        //   H2: dv_r/dtheta, dv_r/dphi, dv_theta/dr, dv_phi/dr  -> 2 e_r_theta, 2 e_r_phi
        //   H3: dv_phi/dphi, omega_r, dv_theta/dphi, dv_r/dr    -> e_rr, e_theta_theta,
        //       e_phi_phi, 2 e_phi_theta (dv_theta/dtheta, dv_phi/dtheta as :226-248 form them)
        //   H4: dT/dr, dT/dtheta, dT/dphi
        {
            const int fo[3] = {A_VR, A_VT, A_VP};
            const bool dp[3] = {false, false, false};
            if constexpr (STAGED) pair_stage<M, 3>(P, rowbase, L, fo, buf, tt);
            pair_c2r<M, 3, STAGED>(P, rowbase, L, fo, dp, buf, tt, y);
            if constexpr (STAGED) {
                const int next[4] = {A_DVRDT, A_VR, A_DVTDR, A_DVPDR};
                pair_stage<M, 4>(P, rowbase, L, next, buf, tt);
            }
            const double rad = rowc[RC_RAD], orad = rowc[RC_ORAD], rho = rowc[RC_RHO], dlnrho = rowc[RC_DLNRHO];
            const double cs = rowc[RC_CS], sn = rowc[RC_SN], csc = rowc[RC_CSC], cot = rowc[RC_COT], cor = rowc[RC_COR];
            auto w0 = [&](double b, double c) { return rho * (rad * b * b + rad * c * c + cor * sn * rad * rad * c); };
            auto p0 = [&](double a, double b, double c, double ct, double co) {
                return -b * b * ct * orad - b * a * orad - b * a * dlnrho - c * c * ct * orad - cor * co * c;
            };
            auto z0 = [&](double a, double b, double c, double co) { return c * a * orad + cor * (co * b + sn * a); };
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                vr[i] = y[0][i];
                vt[i] = make_double2(y[1][i].x * csc, y[1][i].y * csc);
                vp[i] = make_double2(y[2][i].x * csc, y[2][i].y * csc);
                acc_at(0, i) = make_double2(w0(vt[i].x, vp[i].x), w0(vt[i].y, vp[i].y));
                acc_at(1, i) = make_double2(p0(vr[i].x, vt[i].x, vp[i].x, cot, cs), p0(vr[i].y, vt[i].y, vp[i].y, -cot, -cs));
                acc_at(3, i) = make_double2(z0(vr[i].x, vt[i].x, vp[i].x, cs), z0(vr[i].y, vt[i].y, vp[i].y, -cs));
            }
        }
        {
            const int fo[4] = {A_DVRDT, A_VR, A_DVTDR, A_DVPDR};
            const bool dp[4] = {false, true, false, false};
            pair_c2r<M, 4, STAGED>(P, rowbase, L, fo, dp, buf, tt, y);
            if constexpr (STAGED) {
                const int next[4] = {A_VP, A_OMR, A_VT, A_DVRDR};
                pair_stage<M, 4>(P, rowbase, L, next, buf, tt);
            }
            const double rad = rowc[RC_RAD], orad = rowc[RC_ORAD], rho = rowc[RC_RHO], csc = rowc[RC_CSC];
            const double dlnrho = rowc[RC_DLNRHO], vh = rowc[RC_VH];
            // a = sin(theta) dv_r/dtheta, b = dv_r/dphi, c = sin(theta) dv_theta/dr, d = sin(theta) dv_phi/dr
            auto terms = [&](double a, double b, double c, double d, double vrr, double vtt, double vpp, double& wv,
                             double& pv, double& zv) {
                wv += -rho * rad * vtt * a * csc - rho * rad * csc * vpp * b;
                pv += vrr * c * csc;
                zv += vrr * d * csc;
                const double erth = (a * csc - vtt) * orad + c * csc;   // 2 e_r_theta
                const double erph = (b * csc - vpp) * orad + d * csc;   // 2 e_r_phi
                const double dv = -vrr * dlnrho;                        // div u
                return vh * (erth * erth * 0.5 + erph * erph * 0.5 - dv * dv * (1.0 / 3.0));
            };
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                double2 w = acc_at(0, i), pp = acc_at(1, i), z = acc_at(3, i);
                const double hx = terms(y[0][i].x, y[1][i].x, y[2][i].x, y[3][i].x, vr[i].x, vt[i].x, vp[i].x, w.x,
                                        pp.x, z.x);
                const double hy = terms(y[0][i].y, y[1][i].y, y[2][i].y, y[3][i].y, vr[i].y, vt[i].y, vp[i].y, w.y,
                                        pp.y, z.y);
                acc_at(0, i) = w;
                acc_at(1, i) = pp;
                acc_at(2, i) = make_double2(hx, hy);
                acc_at(3, i) = z;
            }
        }
        {
            const int fo[4] = {A_VP, A_OMR, A_VT, A_DVRDR};
            const bool dp[4] = {true, false, true, false};
            pair_c2r<M, 4, STAGED>(P, rowbase, L, fo, dp, buf, tt, y);
            if constexpr (STAGED) {
                const int next[3] = {A_DTDR, A_DTDT, A_T};
                pair_stage<M, 3>(P, rowbase, L, next, buf, tt);
            }
            const double rad = rowc[RC_RAD], orad = rowc[RC_ORAD], rho = rowc[RC_RHO], csc = rowc[RC_CSC];
            const double cot = rowc[RC_COT], c2r = rowc[RC_C2R], dlnrho = rowc[RC_DLNRHO], vh = rowc[RC_VH];
            const double csc2 = csc * csc;
            // a = sin(theta) dv_phi/dphi, b = omega_r, c = sin(theta) dv_theta/dphi, x = dv_r/dr
            auto terms = [&](double a, double b, double c, double x, double vrr, double vtt, double vpp, double ct,
                             double& wv, double& pv, double& zv) {
                wv += -rho * rad * rad * vrr * x;
                pv += -vtt * x + vpp * c * c2r - vtt * a * c2r;
                zv += vtt * c * c2r + vpp * a * c2r + vtt * b;
                const double dvtdt = -vrr * (rad * dlnrho + 2.0) - rad * x - vtt * ct - a * csc2;
                const double dvpdt = rad * b + c * csc2 - vpp * ct;
                const double eff = (a * csc2 + vrr + vtt * ct) * orad;     // e_phi_phi
                const double ett = (dvtdt + vrr) * orad;                   // e_theta_theta
                const double eph = (dvpdt + c * csc2 - vpp * ct) * orad;   // 2 e_phi_theta
                return vh * (x * x + eff * eff + ett * ett + eph * eph * 0.5);
            };
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                double2 w = acc_at(0, i), pp = acc_at(1, i), tv = acc_at(2, i), z = acc_at(3, i);
                tv.x += terms(y[0][i].x, y[1][i].x, y[2][i].x, y[3][i].x, vr[i].x, vt[i].x, vp[i].x, cot, w.x, pp.x, z.x);
                tv.y += terms(y[0][i].y, y[1][i].y, y[2][i].y, y[3][i].y, vr[i].y, vt[i].y, vp[i].y, -cot, w.y, pp.y, z.y);
                acc_at(0, i) = w;
                acc_at(1, i) = pp;
                acc_at(2, i) = tv;
                acc_at(3, i) = z;
            }
        }
        {
            const int fo[3] = {A_DTDR, A_DTDT, A_T};
            const bool dp[3] = {false, false, true};
            pair_c2r<M, 3, STAGED>(P, rowbase, L, fo, dp, buf, tt, y);
            if constexpr (STAGED && MAG) {
                const int next[4] = {A_BR, A_BT, A_BP, A_CBR};
                pair_stage<M, 4>(P, rowbase, L, next, buf, tt);
            }
            const double csc = rowc[RC_CSC], orad = rowc[RC_ORAD];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const double2 d = y[0][i], a = y[1][i], b = y[2][i];
                double2& tv = acc_at(2, i);
                tv.x += -vr[i].x * d.x - a.x * csc * vt[i].x * orad - vp[i].x * b.x * csc * orad;
                tv.y += -vr[i].y * d.y - a.y * csc * vt[i].y * orad - vp[i].y * b.y * csc * orad;
            }
        }
    } else {
        // B1: v_r, v_theta, v_phi, dv_r/dr: the quadratic, Coriolis and radial-advection terms
        {
            const int fo[4] = {A_VR, A_VT, A_VP, A_DVRDR};
            const bool dp[4] = {false, false, false, false};
            if constexpr (STAGED) pair_stage<M, 4>(P, rowbase, L, fo, buf, tt);
            pair_c2r<M, 4, STAGED>(P, rowbase, L, fo, dp, buf, tt, y);
            if constexpr (STAGED) {
                const int next[4] = {A_DVRDT, A_VR, A_DVTDR, A_VT};
                pair_stage<M, 4>(P, rowbase, L, next, buf, tt);
            }
            const double rad = rowc[RC_RAD], orad = rowc[RC_ORAD], rho = rowc[RC_RHO], dlnrho = rowc[RC_DLNRHO];
            const double cs = rowc[RC_CS], sn = rowc[RC_SN], csc = rowc[RC_CSC], cot = rowc[RC_COT], cor = rowc[RC_COR];
            auto w0 = [&](double a, double b, double c, double xx) {
                return rho * (rad * b * b + rad * c * c + cor * sn * rad * rad * c) - rho * rad * rad * a * xx;
            };
            auto p0 = [&](double a, double b, double c, double xx, double ct, double co) {
                return -b * b * ct * orad - b * a * orad - b * a * dlnrho - c * c * ct * orad - cor * co * c - b * xx;
            };
            auto z0 = [&](double a, double b, double c, double co) { return c * a * orad + cor * (co * b + sn * a); };
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                vr[i] = y[0][i];
                vt[i] = make_double2(y[1][i].x * csc, y[1][i].y * csc);
                vp[i] = make_double2(y[2][i].x * csc, y[2][i].y * csc);
                const double2 x = y[3][i];
                acc_at(0, i) = make_double2(w0(vr[i].x, vt[i].x, vp[i].x, x.x), w0(vr[i].y, vt[i].y, vp[i].y, x.y));
                acc_at(1, i) = make_double2(p0(vr[i].x, vt[i].x, vp[i].x, x.x, cot, cs),
                                            p0(vr[i].y, vt[i].y, vp[i].y, x.y, -cot, -cs));
                acc_at(3, i) = make_double2(z0(vr[i].x, vt[i].x, vp[i].x, cs), z0(vr[i].y, vt[i].y, vp[i].y, -cs));
            }
        }
        // B2: dv_r/dtheta, dv_r/dphi, dv_theta/dr, dv_theta/dphi
        {
            const int fo[4] = {A_DVRDT, A_VR, A_DVTDR, A_VT};
            const bool dp[4] = {false, true, false, true};
            pair_c2r<M, 4, STAGED>(P, rowbase, L, fo, dp, buf, tt, y);
            if constexpr (STAGED) {
                const int next[4] = {A_DVPDR, A_VP, A_OMR, A_DTDR};
                pair_stage<M, 4>(P, rowbase, L, next, buf, tt);
            }
            const double rad = rowc[RC_RAD], rho = rowc[RC_RHO], csc = rowc[RC_CSC], c2r = rowc[RC_C2R];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const double2 a = y[0][i], b = y[1][i], c = y[2][i], d = y[3][i];
                double2& w = acc_at(0, i);
                double2& pp = acc_at(1, i);
                double2& z = acc_at(3, i);
                w.x += -rho * rad * vt[i].x * a.x * csc - rho * rad * csc * vp[i].x * b.x;
                w.y += -rho * rad * vt[i].y * a.y * csc - rho * rad * csc * vp[i].y * b.y;
                pp.x += vr[i].x * c.x * csc + vp[i].x * d.x * c2r;
                pp.y += vr[i].y * c.y * csc + vp[i].y * d.y * c2r;
                z.x += vt[i].x * d.x * c2r;
                z.y += vt[i].y * d.y * c2r;
            }
        }
        // B3: dv_phi/dr, dv_phi/dphi, omega_r, dT/dr (the T term's first part, written)
        {
            const int fo[4] = {A_DVPDR, A_VP, A_OMR, A_DTDR};
            const bool dp[4] = {false, true, false, false};
            pair_c2r<M, 4, STAGED>(P, rowbase, L, fo, dp, buf, tt, y);
            if constexpr (STAGED) {
                const int next[2] = {A_DTDT, A_T};
                pair_stage<M, 2>(P, rowbase, L, next, buf, tt);
            }
            const double csc = rowc[RC_CSC], c2r = rowc[RC_C2R];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const double2 a = y[0][i], b = y[1][i], c = y[2][i], d = y[3][i];
                double2& pp = acc_at(1, i);
                double2& z = acc_at(3, i);
                z.x += vr[i].x * a.x * csc + vp[i].x * b.x * c2r + vt[i].x * c.x;
                z.y += vr[i].y * a.y * csc + vp[i].y * b.y * c2r + vt[i].y * c.y;
                pp.x += -vt[i].x * b.x * c2r;
                pp.y += -vt[i].y * b.y * c2r;
                acc_at(2, i) = make_double2(-vr[i].x * d.x, -vr[i].y * d.y);
            }
        }
        // B4: dT/dtheta, dT/dphi
        {
            const int fo[2] = {A_DTDT, A_T};
            const bool dp[2] = {false, true};
            pair_c2r<M, 2, STAGED>(P, rowbase, L, fo, dp, buf, tt, y);
            if constexpr (STAGED && MAG) {
                const int next[4] = {A_BR, A_BT, A_BP, A_CBR};
                pair_stage<M, 4>(P, rowbase, L, next, buf, tt);
            }
            const double csc = rowc[RC_CSC], orad = rowc[RC_ORAD];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const double2 a = y[0][i], b = y[1][i];
                double2& tv = acc_at(2, i);
                tv.x += -a.x * csc * vt[i].x * orad - vp[i].x * b.x * csc * orad;
                tv.y += -a.y * csc * vt[i].y * orad - vp[i].y * b.y * csc * orad;
            }
        }
    }
    // CFL (Find_MyMinDT); the rho r / sin(theta) factor of the P and Z terms is a
    // row constant, applied to their spectra after the r2c (RC_HSF)
    double cmax = 0.0;
    const double orad = rowc[RC_ORAD], dr = rowc[RC_DR];
    {
        const double hfac = P.llmax * orad * orad, rfac = 1.0 / (dr * dr);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            cmax = fmax(cmax, (vt[i].x * vt[i].x + vp[i].x * vp[i].x) * hfac);
            cmax = fmax(cmax, (vt[i].y * vt[i].y + vp[i].y * vp[i].y) * hfac);
            cmax = fmax(cmax, vr[i].x * vr[i].x * rfac);
            cmax = fmax(cmax, vr[i].y * vr[i].y * rfac);
        }
    }
    if constexpr (MAG) {
        // M1: B_r, B_theta, B_phi, (curl B)_r.  The EMF u x B (Compute_EMF,
        // Sphere_Physical_Space.F90:534-581) takes their place in the FFT buffer and goes through
        // its own r2c and fold into p2b fields B_EMFT, B_EMFR, B_EMFP; B stays in registers
        // for the Lorentz force, which M2 ((curl B)_theta, (curl B)_phi) completes.
        double2 br[4], bt[4], bp[4], cbr[4];
        {
            const int fo[4] = {A_BR, A_BT, A_BP, A_CBR};
            const bool dp[4] = {false, false, false, false};
            pair_c2r<M, 4, STAGED>(P, rowbase, L, fo, dp, buf, tt, y);
            const double csc = rowc[RC_CSC], rad = rowc[RC_RAD], rho = rowc[RC_RHO];
            // the Alfven speed (:798-806)
            const double hfb = P.llmax * orad * orad / rho * P.lorentz, rfb = P.lorentz / (dr * dr * rho);
            const double cr = csc * rad;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                br[i] = y[0][i];
                bt[i] = make_double2(y[1][i].x * csc * orad, y[1][i].y * csc * orad);   // rsintheta_div
                bp[i] = make_double2(y[2][i].x * csc * orad, y[2][i].y * csc * orad);
                cbr[i] = y[3][i];
                if constexpr (HEAT) {   // Compute_Ohmic_Heating (:446-466), the (curl B)_r part
                    const double oh = rowc[RC_OH];
                    acc_at(2, i).x += cbr[i].x * cbr[i].x * oh;
                    acc_at(2, i).y += cbr[i].y * cbr[i].y * oh;
                }
                cmax = fmax(cmax, (bt[i].x * bt[i].x + bp[i].x * bp[i].x) * hfb);
                cmax = fmax(cmax, (bt[i].y * bt[i].y + bp[i].y * bp[i].y) * hfb);
                cmax = fmax(cmax, br[i].x * br[i].x * rfb);
                cmax = fmax(cmax, br[i].y * br[i].y * rfb);
            }
            auto emit = [&](int f, const double2 (&a)[4], const double2 (&b)[4], const double2 (&c)[4],
                            const double2 (&d)[4], double scale) {   // scale (a b - c d), then the radix-4 pass
                double2 u[4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    u[i] = make_double2((a[i].x * b[i].x - c[i].x * d[i].x) * scale,
                                        (a[i].y * b[i].y - c[i].y * d[i].y) * scale);
                dft4(u[0], u[1], u[2], u[3], -1);
#pragma unroll
                for (int i = 0; i < 4; ++i) buf[f * M + swz<M>(4 * tt + i)] = u[i];
            };
            emit(0, vp, br, vr, bp, cr);
            emit(1, vt, bp, vp, bt, 1.0);
            emit(2, vr, bt, vt, br, cr);
        }
        pair_r2c<M, 3>(P, obase + 2 * B_EMFT, L, mstride, pstride, buf, tt, [](int) { return 0.5; });
        // M2: (curl B)_theta, (curl B)_phi -> the Lorentz force (:512-519, 635-641, 712-718)
        {
            const int fo[2] = {A_CBT, A_CBP};
            const bool dp[2] = {false, false};
            if constexpr (STAGED) pair_stage<M, 2>(P, rowbase, L, fo, buf, tt);
            pair_c2r<M, 2, STAGED>(P, rowbase, L, fo, dp, buf, tt, y);
            const double csc = rowc[RC_CSC], rad = rowc[RC_RAD], rho = rowc[RC_RHO];
            const double lc = P.lorentz, r2lc = rad * rad * lc, lcr = lc / rho;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const double2 cbt = make_double2(y[0][i].x * csc * orad, y[0][i].y * csc * orad);
                const double2 cbp = make_double2(y[1][i].x * csc * orad, y[1][i].y * csc * orad);
                double2& w = acc_at(0, i);
                double2& pp = acc_at(1, i);
                double2& z = acc_at(3, i);
                w.x += r2lc * (cbt.x * bp[i].x - cbp.x * bt[i].x);
                w.y += r2lc * (cbt.y * bp[i].y - cbp.y * bt[i].y);
                pp.x -= lcr * (cbp.x * br[i].x - cbr[i].x * bp[i].x);
                pp.y -= lcr * (cbp.y * br[i].y - cbr[i].y * bp[i].y);
                z.x -= lcr * (cbr[i].x * bt[i].x - cbt.x * br[i].x);
                z.y -= lcr * (cbr[i].y * bt[i].y - cbt.y * br[i].y);
                if constexpr (HEAT) {   // the (curl B)_theta and (curl B)_phi parts
                    const double oh = rowc[RC_OH];
                    acc_at(2, i).x += (cbt.x * cbt.x + cbp.x * cbp.x) * oh;
                    acc_at(2, i).y += (cbt.y * cbt.y + cbp.y * cbp.y) * oh;
                }
            }
        }
    }
    // the r2c's radix-4 pass on this thread's own points of W, P, T, Z, then the rest
#pragma unroll
    for (int f = 0; f < 4; ++f) {
        double2 u[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) u[i] = acc_at(f, i);
        dft4(u[0], u[1], u[2], u[3], -1);
#pragma unroll
        for (int i = 0; i < 4; ++i) acc_at(f, i) = u[i];
    }
    const double hsf_pz = rowc[RC_HSF];   // P and Z (f = 1, 3) take the row factor
    pair_r2c<M, 4>(P, obase, L, mstride, pstride, acc, tt, [&](int f) { return (f & 1) ? hsf_pz : 0.5; });
    // CFL max over the rows
    for (int o = 16; o > 0; o >>= 1) cmax = fmax(cmax, __shfl_down_sync(0xffffffffu, cmax, o));
    if ((t & 31) == 0) red[t >> 5] = cmax;
    __syncthreads();
    if (t == 0) {
        double v = red[0];
        for (int i = 1; i < NT / 32; ++i) v = fmax(v, red[i]);
        atomicMax(P.cfl, (unsigned long long)__double_as_longlong(v));
    }
}

// n_theta, radii a CTA (whole warps; small grids want many CTAs), CTAs an SM (shared memory)
#define RA_PAIR_CASES(X) \
    X(24, 8, 4)          \
    X(32, 4, 6)          \
    X(48, 4, 4)          \
    X(64, 2, 6)          \
    X(96, 2, 4)          \
    X(128, 1, 6)         \
    X(192, 1, 4)         \
    X(256, 1, 3)         \
    X(384, 1, 2)         \
    X(512, 1, 1)         \
    X(768, 1, 1)

bool physics_pair_supported(int n_theta) {
    switch (n_theta) {
#define RA_X(NN, GG, BB) case NN:
        RA_PAIR_CASES(RA_X)
#undef RA_X
        return true;
        default: return false;
    }
}

template <int M>
static void pair_twiddles(std::vector<double>& tw) {
    using S = Pair<M>;
    const long double PI = 3.141592653589793238462643383279502884L;
    auto add = [&](int count, int ls) {
        for (int j = 0; j < count; ++j) {
            const long double a = 2.0L * PI * j / ls;
            tw.push_back((double)cosl(a));
            tw.push_back((double)sinl(a));
        }
    };
    if (S::R1 > 1) add(S::SS1, S::Q);
    add(4, 4 * S::R2);
}

// The mid passes' twiddles, built once at set-up (the step may be captured into a graph).
void physics_pair_prepare(Ctx& c) {
    if (c.d_twq) return;
    std::vector<double> tw;
    switch (c.d.nth) {
#define RA_X(NN, GG, BB) \
    case NN: pair_twiddles<2 * NN>(tw); break;
        RA_PAIR_CASES(RA_X)
#undef RA_X
        default: return;
    }
    RA_CUDA(cudaMalloc(&c.d_twq, tw.size() * sizeof(double)));
    RA_CUDA(cudaMemcpy(c.d_twq, tw.data(), tw.size() * sizeof(double), cudaMemcpyHostToDevice));
}

template <int M, int G, int MINB>
static void pair_launch(Ctx& c, const PhysParams& P) {
    const unsigned grid = (unsigned)(c.d.nth2 * ((c.d.nr + G - 1) / G));
    const size_t smem = (size_t)G * 8 * M * sizeof(double2);
    auto go = [&](auto kern) {
        RA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kern<<<grid, G * (M / 4), smem, c.stream>>>(P);
    };
    const bool heat = c.rad.heating;
    if (c.mag && heat)
        go(physics_pair_kernel<M, G, MINB, true, true>);
    else if (c.mag)
        go(physics_pair_kernel<M, G, MINB, true, false>);
    else if (heat)
        go(physics_pair_kernel<M, G, MINB, false, true>);
    else
        go(physics_pair_kernel<M, G, MINB, false, false>);
    RA_CUDA(cudaGetLastError());
    ++c.launches;
}

void launch_physics_pair(Ctx& c, PhysParams P) {
    if (!c.d_twq) throw ArgError("physics tables not prepared (physics_prepare runs at set-up)");
    P.twq = reinterpret_cast<const double2*>(c.d_twq);
    switch (c.d.nth) {
#define RA_X(NN, GG, BB) \
    case NN: pair_launch<2 * NN, GG, BB>(c, P); break;
        RA_PAIR_CASES(RA_X)
#undef RA_X
        default: throw ArgError("n_theta " + std::to_string(c.d.nth) +
                                " has no physical-space kernel instance (24..768 of the form 2^a or 3*2^a)");
    }
}

}  // namespace ra
