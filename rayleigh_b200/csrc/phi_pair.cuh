// The phi transform of a (theta, pi - theta) row pair, both rows in one complex FFT, in the shared
// memory of a CTA: the engine of the physical-space stage and of the device-resident transforms.
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
#pragma once

#include "phi_fft.cuh"

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

// Barrier between the two mid passes.  Where each half of the row's threads works on its own fields in
// both of them (two radix-8 passes: a field has T/2 butterflies) a half waits for itself only.
template <int M>
__device__ __forceinline__ void mid_barrier(int tt) {
    constexpr int T = Pair<M>::T;
    if constexpr (Pair<M>::R1 == 8 && Pair<M>::R2 == 8 && T % 64 == 0) {
        asm volatile("bar.sync %0, %1;" ::"r"(tt < T / 2 ? 1 : 2), "r"(T / 2) : "memory");
    } else {
        __syncthreads();
    }
}

// The first pass of NB fields (fo[b], d/dphi where dp[b]) straight from global memory.
template <int M, int NB>
__device__ __forceinline__ void pair_first(const PhysParams& P, const double* __restrict__ rowbase, int L,
                                           const int (&fo)[NB], const bool (&dp)[NB], double2* buf, int tt) {
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
}

// The spectra of NB fields (fo[b]) on their way into the FFT buffer by cp.async: E_m of field b in slot
// b M + m, O_m in slot b M + M/2 + m, m < L (0 for a row past the last radius).  The caller's use of
// the buffer ends with the barrier in here.  Called as soon as the previous batch has left the buffer,
// it brings the next one in under the nonlinear terms; loads into registers were held up by the small
// L1 that 197 KB of shared memory leave (their sectors in flight have to fit it).
template <int M, int NB>
__device__ __forceinline__ void pair_stage(const PhysParams& P, const double* __restrict__ rowbase, int L,
                                           const int (&fo)[NB], double2* buf, int tt) {
    const long ostride = (long)P.ncola, mstride = 2L * P.ncola;
    const unsigned s0 = (unsigned)__cvta_generic_to_shared(buf);
    __syncthreads();
    // eight consecutive m of one field, then the batch's other fields (their records share cache lines),
    // then the other parity
    const int n = 2 * NB * ((L + 7) & ~7);
    for (int e = tt; e < n; e += Pair<M>::T) {
        const int b = (e >> 3) % NB, hi = e / (8 * NB), par = hi & 1, m = (hi >> 1) * 8 + (e & 7);
        int f = fo[0];
#pragma unroll
        for (int i = 1; i < NB; ++i)
            if (b == i) f = fo[i];
        if (m < L)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s0 + 16 * (b * M + par * (M / 2) + m)),
                         "l"(rowbase + m * mstride + par * ostride + 2 * f)
                         : "memory");
    }
}

// The first pass of NB fields whose spectra pair_stage brought (d/dphi where dp[b]).
template <int M, int NB>
__device__ __forceinline__ void pair_first_staged(const PhysParams& P, int L, const bool (&dp)[NB], double2* buf,
                                                  int tt) {
    using S = Pair<M>;
    constexpr int F = S::F, Q = S::Q, T = S::T, H = Q / 2;
    static_assert(2 * H <= T, "one item of a field pair per thread");
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    unsigned dphi = 0;
#pragma unroll
    for (int b = 0; b < NB; ++b) dphi |= dp[b] ? 1u << b : 0u;
    // two fields at a time: every thread takes its item's values, and after the barrier the fields'
    // transforms replace them (one copy of the code for both pairs: the kernel, with up to six
    // transforms inlined, has to stay inside the instruction cache)
#pragma unroll 1
    for (int b0 = 0; b0 < NB; b0 += 2) {
        const int nf = NB - b0 < 2 ? 1 : 2;
        const bool active = tt < nf * H;
        const int b = b0 + (tt >= H ? 1 : 0), k = tt - (tt >= H ? H : 0);
        const bool self = k == 0;
        const int kp = self ? Q / 2 : Q - k;
        double2* fb = buf + b * M;
        const int idx[4] = {k, k + Q, kp, kp + Q};
        const double2 zero = make_double2(0.0, 0.0);
        double2 zp[4], zm[4], xp = zero, xm = zero, w = zero;
        if (active) {
            const bool d = (dphi >> b) & 1;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                double2 e = zero, o = zero;
                if (idx[i] < L) {
                    e = fb[idx[i]];
                    o = fb[M / 2 + idx[i]];
                }
                hemispheres(e, o, idx[i], d, zp[i], zm[i]);
            }
            if (F == 6 && self && 2 * Q < L) hemispheres(fb[2 * Q], fb[M / 2 + 2 * Q], 2 * Q, d, xp, xm);
            w = __ldg(P.wr + (self ? kp : k));   // exp(2 pi i k / M)
        }
        __syncthreads();
        if (active) {
            double2 ya[F], yb[F];
            dft_from4<F, 1>(zp[0], zp[1], self ? xm : zm[3], self ? zm[1] : zm[2], ya);
            if (F == 6 && self) {   // m = M/3 = l_max: inputs 2 (here) and 4 (above) of residue 0
                const double S3 = 0.86602540378443864676;
                const double2 x1 = make_double2(-0.5 * xp.x - S3 * xp.y, -0.5 * xp.y + S3 * xp.x);
                const double2 x2 = make_double2(-0.5 * xp.x + S3 * xp.y, -0.5 * xp.y - S3 * xp.x);
#pragma unroll
                for (int j = 0; j < F; ++j) ya[j] = cadd(ya[j], j % 3 == 0 ? xp : (j % 3 == 1 ? x1 : x2));
            }
            dft_from4<F, -1>(self ? zm[2] : zm[0], self ? zm[3] : zm[1], zp[3], zp[2], yb);
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
    }
}

// c2r of NB fields of this row pair (fields fo[b], d/dphi where dp[b]; STAGED: the spectra are on their
// way by pair_stage); on return y[b][i] holds the (south, north) values of field b at the row's point
// 4 tt + i (digit-reversed order).  L is 0 for a row past the last radius.
template <int M, int NB, bool STAGED>
__device__ __forceinline__ void pair_c2r(const PhysParams& P, const double* __restrict__ rowbase, int L,
                                         const int (&fo)[NB], const bool (&dp)[NB], double2* buf, int tt,
                                         double2 (&y)[4][4]) {
    using S = Pair<M>;
    constexpr int Q = S::Q;
    if constexpr (STAGED)
        pair_first_staged<M, NB>(P, L, dp, buf, tt);
    else
        pair_first<M, NB>(P, rowbase, L, fo, dp, buf, tt);
    __syncthreads();
    if constexpr (S::R1 > 1) {
        pair_mid_pass<M, NB, S::R1, Q, false>(buf, P.twq, tt);
        mid_barrier<M>(tt);
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

}  // namespace ra
