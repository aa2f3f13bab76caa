// The per-l implicit matrices on the device (Load_Linear_Coefficients, Set_Boundary_Conditions;
// Sphere_Linear_Terms.F90:196-1100): every row is either a sum of radius profiles times rows of the
// derivative matrices D_d, or a boundary row.  The profiles of each l (a few dozen vectors of n_r)
// come from the host, which forms them for ra_build_matrices too; the matrices, 9 n_r^2 doubles an l
// and more, are formed where the factorisation reads them.
//
// What bounds it: the writes (one 8-byte store per element; D and the profiles come from L1 / L2).
// The host formed them element by element and copied them over: 8 ms of the 9 ms of a dt change at
// l_max = 85, N_r = 64.  Products and sums are rounded one by one, in the host form's order, so that
// the two agree bit for bit.
#include "ra_internal.h"

namespace ra {

constexpr int AS_THREADS = 128;

// element (row, col) of system sys of one l
__device__ __forceinline__ double assembled(const AsmShape& S, const double* __restrict__ amp,
                                            const double* __restrict__ bamp, const double* __restrict__ D, int sys,
                                            int row, int col, int nr, int rda) {
    const int eq = row / nr, i = row - eq * nr;
    double v = 0.0;
    bool boundary = false;
    for (int q = 0; q < S.nclear; ++q) boundary = boundary || (S.clear_sys[q] == sys && S.clear_row[q] == row);
    if (boundary) {
        for (int q = 0; q < S.nbc; ++q) {
            if (S.bc_sys[q] != sys || S.bc_row[q] != row) continue;
            const int j = col - S.bc_col[q];
            if (j >= 0 && j < rda - 1)
                v = __dadd_rn(v, __dmul_rn(__ldg(bamp + q), __ldg(D + ((size_t)S.bc_d[q] * nr + i) * nr + j)));
        }
        return v;
    }
    const int var = col / nr, j = col - var * nr;
    for (int q = 0; q < S.nterm; ++q) {
        if (S.sys[q] != sys || S.eq[q] != eq || S.var[q] != var) continue;
        v = __dadd_rn(v, __dmul_rn(__ldg(amp + (size_t)q * nr + i), __ldg(D + ((size_t)S.d[q] * nr + i) * nr + j)));
    }
    return v;
}

// grid: (rows of the l's systems, l); l = 0 has its own terms
__global__ void __launch_bounds__(AS_THREADS) assemble_kernel(AsmShape S0, AsmShape S1, const double* __restrict__ amp,
                                                              const double* __restrict__ bamp,
                                                              const double* __restrict__ D, int nr, int rda,
                                                              double* __restrict__ wpt, double* __restrict__ z,
                                                              double* __restrict__ cm, double* __restrict__ am) {
    const int l = blockIdx.y;
    const AsmShape& S = l == 0 ? S0 : S1;
    int row = blockIdx.x, sys = 0, n = 3 * nr;
    double* out = wpt;
    if (row >= 3 * nr) {
        sys = 1 + (row - 3 * nr) / nr;
        row = (row - 3 * nr) % nr;
        n = nr;
        out = sys == 1 ? z : (sys == 2 ? cm : am);
    }
    out += ((size_t)l * n + row) * n;
    const double* a = amp + (size_t)l * AsmShape::MAXT * nr;
    const double* b = bamp + (size_t)l * AsmShape::MAXB;
    for (int col = threadIdx.x; col < n; col += AS_THREADS) out[col] = assembled(S, a, b, D, sys, row, col, nr, rda);
}

void launch_assemble(Ctx& c, const AsmShape& s0, const AsmShape& s1, const double* d_amp, const double* d_bamp) {
    const dim3 grid((unsigned)((c.mag ? 6 : 4) * c.d.nr), (unsigned)c.d.L);
    assemble_kernel<<<grid, AS_THREADS, 0, c.stream>>>(s0, s1, d_amp, d_bamp, c.d_D, c.d.nr, c.d.rda, c.d_Awpt, c.d_Az,
                                                       c.d_Ac, c.d_Aa);
    RA_CUDA(cudaGetLastError());
    ++c.launches;
}

}  // namespace ra
