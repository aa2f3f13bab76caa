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
//
// Both hemispheres in one complex transform.  The south row of a field has the
// spectrum S_m = E_m + O_m, the north row N_m = E_m - O_m; the complex transform of
// length M = n_phi of Z_m = S_m + i N_m, Z_{-m} = conj(S_m) + i conj(N_m) leaves the
// south row in its real part and the north row in its imaginary part.  So every E and O
// is read once, no half-length pre- and post-processing of a real transform is
// needed, a thread holds both hemispheres of its phi points, and on the way back
// the spectra Z_m, Z_{-m} of (south term) + i (north term) give S_m and N_m, hence
// the folded f_even = S + N and f_odd = S - N, where they are.
//
// The transform, in place in shared memory, decimation in frequency for the c2r
// (digit-reversed points; the nonlinear terms are pointwise in phi) and in time for
// the r2c:  M = F x (mid radices) x 4, F = 6 where 3 divides M, else 4.
//   first pass   radix F straight from the spectrum loads.  With |m| <= l_max < M/3
//                two of the six inputs are zero (F = 6); the residues k and -k
//                use the same four X_m, so that a work item forms both
//   mid passes   radix 8 (4, 2) in shared memory
//   last pass    radix 4 in registers: thread t of a row holds the points 4t .. 4t+3 of
//                every field
// and the r2c the same backwards, its last (radix-F) pass writing to global memory.
// At M = 1536 a field point makes six 16-byte shared accesses per transform (the
// form with one complex transform of length M/2 per row and field made ten).
//
// Shared layout: position p of a field at swz(p), a permutation of the low three
// bits under which every access of the mid and last passes is conflict-free (a
// 16-byte access is served in phases of 8 lanes, one wavefront where the 8 slots
// differ modulo 8), and the first pass's writes up to one extra wavefront.
#include <cmath>
#include <vector>

#include "phi_fft.cuh"
#include "ra_internal.h"

namespace ra {

template <int M>
struct Pair {
    static constexpr int F = (M % 3 == 0) ? 6 : 4;
    static constexpr int T = M / 4;          // threads of a row pair
    static constexpr int Q = M / F;          // stride of the first pass
    static constexpr int INNER = Q / 4;      // product of the mid radices
    static constexpr int R1 = INNER == 64 ? 8 : (INNER >= 16 ? 4 : 1);   // 1: one mid pass only
    static constexpr int R2 = INNER / R1;    // the mid pass of stride 4
    static constexpr int SS1 = Q / R1;       // stride of the first mid pass
    static constexpr int TW2 = R1 > 1 ? SS1 : 0;   // offset of the second mid pass's twiddles
    static constexpr int NTW = TW2 + 4;
    static constexpr int TB = 4 * R2;        // the position bit that toggles bit 2 of the slot
    static_assert(F * R1 * R2 * 4 == M && R2 <= 8 && R2 >= 2 && (R2 & (R2 - 1)) == 0, "plan");
};

// Slot of position p.  Last pass: 8 lanes take p = 4t + i, t = 8 consecutive: bits 3-4
// vary over four pairs of lanes and permute the low two bits.  The stride-4 mid pass
// (p = TB b + j + 4i, j < 4): the two blocks b of a phase differ in bit 2.  Larger
// strides and the first pass: 8 consecutive p, permuted among themselves.
template <int M>
__device__ __forceinline__ int swz(int p) {
    return p ^ ((p >> 3) & 3) ^ ((p & Pair<M>::TB) ? 4 : 0);
}

// E and O of one (m, field): Z_m and Z_{-m} of S = E + O, N = E - O; times i m for d/dphi;
// Im X_0 = 0 as FFTW's c2r ignores it.
__device__ __forceinline__ void hemispheres(double2 e, double2 o, int m, bool dp, double2& zp, double2& zm) {
    double2 s = cadd(e, o), n = csub(e, o);
    if (dp) {
        s = make_double2(-m * s.y, m * s.x);
        n = make_double2(-m * n.y, m * n.x);
    }
    if (m == 0) s.y = n.y = 0.0;
    zp = make_double2(s.x - n.y, s.y + n.x);
    zm = make_double2(s.x + n.y, n.x - s.y);
}

// y_j = sum_i x_i exp(SGN 2 pi i i j / F) over the nonzero inputs x_0, x_1, x_{F-2}, x_{F-1}.
template <int F, int SGN>
__device__ __forceinline__ void dft_from4(double2 x0, double2 x1, double2 x2, double2 x3, double2 (&y)[F]) {
    if constexpr (F == 4) {
        dft4(x0, x1, x2, x3, SGN);
        y[0] = x0;
        y[1] = x1;
        y[2] = x2;
        y[3] = x3;
    } else {
        // j = (j mod 2, j mod 3): even inputs {0, 4} and odd inputs {1, 5}, each a 3-point sum
        const double S3 = SGN * 0.86602540378443864676;
        const double2 t = cadd(x1, x3), d = csub(x1, x3);
        const double2 p0 = cadd(x0, x2);
        const double2 a = make_double2(x0.x - 0.5 * x2.x, x0.y - 0.5 * x2.y);
        const double2 p1 = make_double2(a.x + S3 * x2.y, a.y - S3 * x2.x);
        const double2 p2 = make_double2(a.x - S3 * x2.y, a.y + S3 * x2.x);
        const double2 q1 = make_double2(S3 * d.y - 0.5 * t.x, -S3 * d.x - 0.5 * t.y);
        const double2 q2 = make_double2(-S3 * d.y - 0.5 * t.x, S3 * d.x - 0.5 * t.y);
        y[0] = cadd(p0, t);
        y[3] = csub(p0, t);
        y[4] = cadd(p1, q1);
        y[1] = csub(p1, q1);
        y[2] = cadd(p2, q2);
        y[5] = csub(p2, q2);
    }
}

// z_i = sum_j u_j exp(SGN 2 pi i i j / F) for i = 0, 1, F-2, F-1 (and i = 2 of F = 6 in z2).
template <int F, int SGN>
__device__ __forceinline__ void dft_to4(const double2 (&u)[F], double2& z0, double2& z1, double2& z3, double2& z4,
                                        double2* z2 = nullptr) {
    if constexpr (F == 4) {
        double2 a = u[0], b = u[1], c = u[2], d = u[3];
        dft4(a, b, c, d, SGN);
        z0 = a;
        z1 = b;
        z3 = c;
        z4 = d;
    } else {
        const double S3 = SGN * 0.86602540378443864676;
        auto three = [&](double2 a, double2 b, double2 c, double2* s, double2& cw, double2& wc) {
            // s = a + b + c, cw = a + b conj(w) + c w, wc = a + b w + c conj(w), w = exp(SGN 2 pi i / 3)
            const double2 t = cadd(b, c), d = csub(b, c);
            const double2 h = make_double2(a.x - 0.5 * t.x, a.y - 0.5 * t.y);
            if (s) *s = cadd(a, t);
            cw = make_double2(h.x + S3 * d.y, h.y - S3 * d.x);
            wc = make_double2(h.x - S3 * d.y, h.y + S3 * d.x);
        };
        double2 e2;
        three(cadd(u[0], u[3]), cadd(u[4], u[1]), cadd(u[2], u[5]), &z0, z3, e2);
        if (z2) *z2 = e2;
        three(csub(u[0], u[3]), csub(u[4], u[1]), csub(u[2], u[5]), nullptr, z1, z4);
    }
}

// A work item of the first (c2r) and last (r2c) pass: the residues k and Q - k of one field
// (k = 0 with Q/2, which are their own mirrors).  Items run over 8 consecutive k of one field,
// then the batch's other fields, so that the lanes of a load share the cache lines of
// neighbouring fields and a store phase covers 8 consecutive slots.
template <int M, int NB>
__device__ __forceinline__ void pair_item(int q, int& k, int& b) {
    constexpr int H = Pair<M>::Q / 2, KL = H < 8 ? H : 8;
    static_assert(H % KL == 0, "items per field");
    const int hi = q / (KL * NB);
    b = (q / KL) % NB;
    k = hi * KL + q % KL;
}

// One mid pass over NB fields of this row pair: butterfly (block, j) takes the positions
// block LS + j + m SS.  tw holds exp(2 pi i j / LS), j < SS.
template <int M, int NB, int R, int LS, bool DIT>
__device__ __forceinline__ void pair_mid_pass(double2* __restrict__ buf, const double2* __restrict__ tw, int tt) {
    constexpr int SS = LS / R, T = Pair<M>::T, PER = M / R;
#pragma unroll 1
    for (int q = tt; q < NB * PER; q += T) {
        const int f = q / PER, bi = q - f * PER, blk = bi / SS, j = bi - blk * SS;
        double2* fb = buf + f * M;
        const int base = blk * LS + j;
        double2 w1 = __ldg(tw + j);
        double2 u[R];
#pragma unroll
        for (int m = 0; m < R; ++m) u[m] = fb[swz<M>(base + m * SS)];
        if (DIT) {
            w1.y = -w1.y;
            twiddle_apply<R>(u, w1);
            dft_small(R, u, -1);
        } else {
            dft_small(R, u, +1);
            twiddle_apply<R>(u, w1);
        }
#pragma unroll
        for (int m = 0; m < R; ++m) fb[swz<M>(base + m * SS)] = u[m];
    }
}

// c2r of NB fields of this row pair (fields fo[b], d/dphi where dp[b]); on return y[b][i] holds the
// (south, north) values of field b at the row's point 4 tt + i (digit-reversed order).  L is 0 for
// a row past the last radius.
template <int M, int NB>
__device__ __forceinline__ void pair_c2r(const PhysParams& P, const double* __restrict__ rowbase, int L,
                                         const int (&fo)[NB], const bool (&dp)[NB], double2* buf, int tt,
                                         double2 (&y)[4][4]) {
    using S = Pair<M>;
    constexpr int F = S::F, Q = S::Q, T = S::T, NITEM = NB * (Q / 2);
    const long ostride = (long)P.ncola, mstride = 2L * P.ncola;
    __syncthreads();   // the buffer is free
#pragma unroll 1
    for (int q = tt; q < NITEM; q += T) {
        int k, b;
        pair_item<M, NB>(q, k, b);
        const bool self = k == 0;
        const int kp = self ? Q / 2 : Q - k;
        int f = fo[0];
        bool d = dp[0];
#pragma unroll
        for (int i = 1; i < NB; ++i)
            if (b == i) {
                f = fo[i];
                d = dp[i];
            }
        const double* base = rowbase + (long)f * 2;
        const int idx[4] = {k, k + Q, kp, kp + Q};
        double2 e[4], o[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            e[i] = o[i] = make_double2(0.0, 0.0);
            if (idx[i] < L) {
                e[i] = __ldg(reinterpret_cast<const double2*>(base + idx[i] * mstride));
                o[i] = __ldg(reinterpret_cast<const double2*>(base + idx[i] * mstride + ostride));
            }
        }
        double2 w = __ldg(P.wr + (self ? kp : k));   // exp(2 pi i k / M)
        double2 zp[4], zm[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) hemispheres(e[i], o[i], idx[i], d, zp[i], zm[i]);
        double2 ya[F], yb[F];
        const double2 zero = make_double2(0.0, 0.0);
        double2 a2 = self ? zero : zm[3];
        if (F == 6 && self && 2 * Q < L) {   // m = M/3 = l_max: inputs 2 and 4 of residue 0
            const double2 ex = __ldg(reinterpret_cast<const double2*>(base + 2 * Q * mstride));
            const double2 ox = __ldg(reinterpret_cast<const double2*>(base + 2 * Q * mstride + ostride));
            double2 xp, xm;
            hemispheres(ex, ox, 2 * Q, d, xp, xm);
            dft_from4<F, 1>(zp[0], zp[1], xm, zm[1], ya);
            const double S3 = 0.86602540378443864676;
            const double2 x1 = make_double2(-0.5 * xp.x - S3 * xp.y, -0.5 * xp.y + S3 * xp.x);
            const double2 x2 = make_double2(-0.5 * xp.x + S3 * xp.y, -0.5 * xp.y - S3 * xp.x);
#pragma unroll
            for (int j = 0; j < F; ++j) ya[j] = cadd(ya[j], j % 3 == 0 ? xp : (j % 3 == 1 ? x1 : x2));
        } else {
            dft_from4<F, 1>(zp[0], zp[1], a2, self ? zm[1] : zm[2], ya);
        }
        dft_from4<F, -1>(self ? zm[2] : zm[0], self ? zm[3] : zm[1], zp[3], zp[2], yb);
        double2* fb = buf + b * M;
        fb[swz<M>(k)] = ya[0];
        fb[swz<M>(kp)] = yb[0];
        double2 wj = w;
#pragma unroll
        for (int j = 1; j < F; ++j) {
            fb[swz<M>(j * Q + k)] = self ? ya[j] : cmul(ya[j], wj);
            fb[swz<M>(j * Q + kp)] = cmul(yb[j], cconj(wj));
            if (j + 1 < F) wj = cmul(wj, w);
        }
    }
    __syncthreads();
    if constexpr (S::R1 > 1) {
        pair_mid_pass<M, NB, S::R1, Q, false>(buf, P.twq, tt);
        __syncthreads();
    }
    pair_mid_pass<M, NB, S::R2, 4 * S::R2, false>(buf, P.twq + S::TW2, tt);
    __syncthreads();
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        double2 u[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) u[i] = buf[b * M + swz<M>(4 * tt + i)];
        dft4(u[0], u[1], u[2], u[3], 1);
#pragma unroll
        for (int i = 0; i < 4; ++i) y[b][i] = u[i];
    }
}

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
    __syncthreads();
    if constexpr (S::R1 > 1) {
        pair_mid_pass<M, NB, S::R1, Q, true>(buf, P.twq, tt);
        __syncthreads();
    }
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
            pair_c2r<M, 3>(P, rowbase, L, fo, dp, buf, tt, y);
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
            pair_c2r<M, 4>(P, rowbase, L, fo, dp, buf, tt, y);
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
            pair_c2r<M, 4>(P, rowbase, L, fo, dp, buf, tt, y);
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
            pair_c2r<M, 3>(P, rowbase, L, fo, dp, buf, tt, y);
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
            pair_c2r<M, 4>(P, rowbase, L, fo, dp, buf, tt, y);
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
            pair_c2r<M, 4>(P, rowbase, L, fo, dp, buf, tt, y);
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
            pair_c2r<M, 4>(P, rowbase, L, fo, dp, buf, tt, y);
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
            pair_c2r<M, 2>(P, rowbase, L, fo, dp, buf, tt, y);
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
            pair_c2r<M, 4>(P, rowbase, L, fo, dp, buf, tt, y);
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
            pair_c2r<M, 2>(P, rowbase, L, fo, dp, buf, tt, y);
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

// f(Pair<M> tag, G) for the n_theta with an instance; false for the others
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
