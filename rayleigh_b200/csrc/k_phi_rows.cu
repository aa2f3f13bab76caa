// The device-resident transforms between the Legendre products' E/O blocks and phi rows
// (ra_transform_dev; the unfold or fold of Legendre_Transforms.F90:1030-1064, 1109-1122 and
// FFT_To_Physical / FFT_To_Spectral, Fourier_Transform.F90:100-183, in one kernel each way):
//   rows_c2r  p2[theta_h][m][par][fr] (E, O) -> rows[theta][fr][n_phi + 2], the padding zero
//   rows_r2c  rows -> their packed spectra in place, and the folded p2[m][par][theta_h][fr]
// on row pairs (phi_pair.cuh), four neighbouring columns fr per T = n_phi / 4 threads.
//
// What bounds them: latency.  At n_phi = 1536 registers let one CTA of twelve warps on an SM, which waits
// on its loads (long scoreboard a third of the cycles of an instruction) and barriers; the L1 data pipe is
// 59 % busy, HBM 0.37 (c2r) and 0.56 (r2c, whose rows' spectra are 37 % of its bytes) of the copy rate.  Each
// direction reads its input once and writes its output once, where the separate relayout and in-place FFT moved
// the rows three times and the FFT, one row per CTA with a twiddle table copied to shared memory for each, ran
// at a fifth of the HBM rate (l_max 255, 512 columns, FP64 inverse call: 3303 -> 1130 us).
// The rows enter and leave in natural phi order: the points of the last pass, digit-reversed, go
// through shared memory once more, at natural index n plus one slot per F R1 points, which
// spreads the 8 lanes of a phase (their n differ by F R1) over the 8 banks.
#include "phi_pair.cuh"
#include "ra_internal.h"

namespace ra {

template <int M>
struct Rows {
    using S = Pair<M>;
    static constexpr int STEP = S::F * S::R1;
    static constexpr int LEN = M + M / STEP;      // a field's slots in natural order
    static __device__ __forceinline__ int slot(int n) { return n + n / STEP; }
    // natural index of position 4 t (the point 4 t + i is M/4 i further on)
    static __device__ __forceinline__ int natural(int t) {
        const int p = 4 * t, d0 = p / S::Q, r0 = p - d0 * S::Q;
        if constexpr (S::R1 > 1) {
            const int d1 = r0 / S::SS1, d2 = (r0 - d1 * S::SS1) / 4;
            return d0 + S::F * (d1 + S::R1 * d2);
        } else {
            return d0 + S::F * (r0 / 4);
        }
    }
};

constexpr int ROW_NB = 4;   // columns of a thread group

template <int M, int G>
__global__ void __launch_bounds__(G* M / 4) rows_c2r_kernel(PhysParams P, double* __restrict__ rows, int nfr) {
    using R = Rows<M>;
    constexpr int T = Pair<M>::T, NTH = M / 2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int t = threadIdx.x, g = G == 1 ? 0 : t / T, tt = t - g * T;
    const int thh = blockIdx.y, fr0 = (blockIdx.x * G + g) * ROW_NB;
    double2* buf = reinterpret_cast<double2*>(smem_raw) + g * (ROW_NB * R::LEN);
    const double* base = P.p2a + ((size_t)thh * P.L * 2 * nfr + fr0) * 2;
    int fo[ROW_NB];
    const bool dp[ROW_NB] = {false, false, false, false};
#pragma unroll
    for (int b = 0; b < ROW_NB; ++b) fo[b] = min(b, max(nfr - 1 - fr0, 0));   // past the last column: any, not stored
    double2 y[4][4];
    pair_c2r<M, ROW_NB, false>(P, base, fr0 < nfr ? P.L : 0, fo, dp, buf, tt, y);
    __syncthreads();   // every point is in registers
    const int n0 = R::natural(tt);
#pragma unroll
    for (int b = 0; b < ROW_NB; ++b)
#pragma unroll
        for (int i = 0; i < 4; ++i) buf[b * R::LEN + R::slot(n0 + i * T)] = y[b][i];
    __syncthreads();
#pragma unroll
    for (int b = 0; b < ROW_NB; ++b) {
        if (fr0 + b >= nfr) break;
        double* south = rows + ((size_t)thh * nfr + fr0 + b) * (M + 2);
        double* north = rows + ((size_t)(NTH - 1 - thh) * nfr + fr0 + b) * (M + 2);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int n = tt + i * T;
            const double2 v = buf[b * R::LEN + R::slot(n)];
            south[n] = v.x;
            north[n] = v.y;
        }
        if (tt < 2) south[M + tt] = north[M + tt] = 0.0;
    }
}

// z_i = sum_j u_j exp(SGN 2 pi i i j / F), every i
template <int F, int SGN>
__device__ __forceinline__ void dft_all(double2 (&u)[F]) {
    if constexpr (F == 4) {
        dft4(u[0], u[1], u[2], u[3], SGN);
    } else {
        double2 e[3] = {cadd(u[0], u[3]), cadd(u[4], u[1]), cadd(u[2], u[5])};
        double2 o[3] = {csub(u[0], u[3]), csub(u[4], u[1]), csub(u[2], u[5])};
        dft_small(3, e, SGN);   // e_k = sum_b U_b w^(kb): z_i = e_{-i mod 3} for even i
        dft_small(3, o, SGN);
        u[0] = e[0];
        u[2] = e[1];
        u[4] = e[2];
        u[3] = o[0];
        u[5] = o[1];
        u[1] = o[2];
    }
}

template <int M, int G>
__global__ void __launch_bounds__(G* M / 4) rows_r2c_kernel(PhysParams P, double* __restrict__ rows, int nfr) {
    using S = Pair<M>;
    using R = Rows<M>;
    constexpr int F = S::F, Q = S::Q, T = S::T, NTH = M / 2, NITEM = ROW_NB * (Q / 2);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int t = threadIdx.x, g = G == 1 ? 0 : t / T, tt = t - g * T;
    const int thh = blockIdx.y, fr0 = (blockIdx.x * G + g) * ROW_NB;
    double2* buf = reinterpret_cast<double2*>(smem_raw) + g * (ROW_NB * R::LEN);
    double* south = rows + ((size_t)thh * nfr + fr0) * (M + 2);
    double* north = rows + ((size_t)(NTH - 1 - thh) * nfr + fr0) * (M + 2);
#pragma unroll
    for (int b = 0; b < ROW_NB; ++b)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int n = tt + i * T;
            double2 v = make_double2(0.0, 0.0);
            if (fr0 + b < nfr) v = make_double2(south[(size_t)b * (M + 2) + n], north[(size_t)b * (M + 2) + n]);
            buf[b * R::LEN + R::slot(n)] = v;
        }
    __syncthreads();
    const int n0 = R::natural(tt);
    double2 y[ROW_NB][4];
#pragma unroll
    for (int b = 0; b < ROW_NB; ++b)
#pragma unroll
        for (int i = 0; i < 4; ++i) y[b][i] = buf[b * R::LEN + R::slot(n0 + i * T)];
    __syncthreads();
#pragma unroll
    for (int b = 0; b < ROW_NB; ++b) {
        dft4(y[b][0], y[b][1], y[b][2], y[b][3], -1);
#pragma unroll
        for (int i = 0; i < 4; ++i) buf[b * M + swz<M>(4 * tt + i)] = y[b][i];
    }
    __syncthreads();
    pair_mid_pass<M, ROW_NB, S::R2, 4 * S::R2, true>(buf, P.twq + S::TW2, tt);
    if constexpr (S::R1 > 1) {
        mid_barrier<M>(tt);
        pair_mid_pass<M, ROW_NB, S::R1, Q, true>(buf, P.twq, tt);
    }
    __syncthreads();
    const size_t mstride = (size_t)NTH * nfr * 2, pstride = mstride / 2;   // p2[m][par][theta_h][fr]
#pragma unroll 1
    for (int q = tt; q < NITEM; q += T) {
        int k, b;
        pair_item<M, ROW_NB>(q, k, b);
        if (fr0 + b >= nfr) continue;
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
        dft_all<F, -1>(ua);   // Z at k + i Q
        dft_all<F, 1>(ub);    // Z at -(k + i Q), that is at kp + (F - 1 - i) Q
        double2* srow = reinterpret_cast<double2*>(south + (size_t)b * (M + 2));
        double2* nrow = reinterpret_cast<double2*>(north + (size_t)b * (M + 2));
        double* out = P.p2b + ((size_t)thh * nfr + fr0 + b) * 2;
        auto put = [&](int m, double2 zp, double2 zm) {
            const double2 s = make_double2(0.5 * (zp.x + zm.x), 0.5 * (zp.y - zm.y));
            const double2 n = make_double2(0.5 * (zp.y + zm.y), 0.5 * (zm.x - zp.x));
            srow[m] = s;
            nrow[m] = n;
            if (m < P.L) {
                *reinterpret_cast<double2*>(out + m * mstride) = cadd(s, n);
                *reinterpret_cast<double2*>(out + m * mstride + pstride) = csub(s, n);
            }
        };
#pragma unroll
        for (int i = 0; i < F / 2; ++i) {
            put(k + i * Q, ua[i], self ? ua[(F - i) % F] : ub[i]);
            put(kp + i * Q, ub[F - 1 - i], self ? ub[i] : ua[F - 1 - i]);
        }
        if (self) put(M / 2, ua[F / 2], ua[F / 2]);
    }
}

#define RA_ROW_CASES(X) \
    X(24, 16)           \
    X(32, 8)            \
    X(48, 8)            \
    X(64, 4)            \
    X(96, 4)            \
    X(128, 2)           \
    X(192, 2)           \
    X(256, 1)           \
    X(384, 1)           \
    X(512, 1)           \
    X(768, 1)

// The pruned first pass needs l_max <= n_phi / 3 where n_phi = 3 2^a (any accepted l_max else); the
// other contexts keep the relayout and the in-place row FFT.
bool rows_pair_supported(const Ctx& c) {
    if (!c.d_twq) return false;
    return c.d.nth % 3 != 0 || c.d.L <= (2 * c.d.nth) / 3 + 1;
}

// to_rows: p2 -> rows; else rows -> rows (spectra) and p2
void launch_rows_pair(Ctx& c, bool to_rows, double* p2, double* rows, int nfr) {
    PhysParams P{};
    P.p2a = p2;
    P.p2b = p2;
    P.wr = reinterpret_cast<const double2*>(c.d_twid);
    P.twq = reinterpret_cast<const double2*>(c.d_twq);
    P.L = c.d.L;
    P.ncola = 2 * nfr;
    auto go = [&](auto kern, int len, int G) {
        const dim3 grid((unsigned)((nfr + ROW_NB * G - 1) / (ROW_NB * G)), (unsigned)c.d.nth2);
        const size_t smem = (size_t)G * ROW_NB * len * sizeof(double2);
        RA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kern<<<grid, (unsigned)(G * c.d.nphi / 4), smem, c.stream>>>(P, rows, nfr);
    };
    switch (c.d.nth) {
#define RA_X(NN, GG)                                             \
    case NN:                                                     \
        if (to_rows)                                             \
            go(rows_c2r_kernel<2 * NN, GG>, Rows<2 * NN>::LEN, GG); \
        else                                                     \
            go(rows_r2c_kernel<2 * NN, GG>, Rows<2 * NN>::LEN, GG); \
        break;
        RA_ROW_CASES(RA_X)
#undef RA_X
        default: throw ArgError("n_theta " + std::to_string(c.d.nth) + " has no row-pair transform");
    }
    RA_CUDA(cudaGetLastError());
    ++c.launches;
}

}  // namespace ra
