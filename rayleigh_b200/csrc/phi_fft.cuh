// What the phi FFT kernels share: complex arithmetic, the small DFTs, the twiddle powers, and the
// operands of the physical-space stage.
#pragma once

#include <cuda_runtime.h>

namespace ra {

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }

__device__ __forceinline__ void dft4(double2& u0, double2& u1, double2& u2, double2& u3, int sign) {
    const double2 t0 = cadd(u0, u2), t1 = csub(u0, u2);
    const double2 t2 = cadd(u1, u3), d = csub(u1, u3);
    // w = sign * i : w * (x + i y) = sign * (-y + i x)
    const double2 wd = make_double2(-sign * d.y, sign * d.x);
    u0 = cadd(t0, t2);
    u2 = csub(t0, t2);
    u1 = cadd(t1, wd);
    u3 = csub(t1, wd);
}

__device__ __forceinline__ void dft_small(int R, double2* u, int sign) {
    if (R == 2) {
        const double2 a = u[0], b = u[1];
        u[0] = cadd(a, b);
        u[1] = csub(a, b);
    } else if (R == 4) {
        dft4(u[0], u[1], u[2], u[3], sign);
    } else if (R == 8) {
        const double H = 0.70710678118654752440;   // sqrt(2)/2
        double2 a0 = cadd(u[0], u[4]), a1 = cadd(u[1], u[5]), a2 = cadd(u[2], u[6]), a3 = cadd(u[3], u[7]);
        double2 b0 = csub(u[0], u[4]), b1 = csub(u[1], u[5]), b2 = csub(u[2], u[6]), b3 = csub(u[3], u[7]);
        // b_j *= exp(sign i pi j / 4)
        b1 = make_double2(H * (b1.x - sign * b1.y), H * (b1.y + sign * b1.x));
        b2 = make_double2(-sign * b2.y, sign * b2.x);
        b3 = make_double2(H * (-b3.x - sign * b3.y), H * (-b3.y + sign * b3.x));
        dft4(a0, a1, a2, a3, sign);
        dft4(b0, b1, b2, b3, sign);
        u[0] = a0; u[2] = a1; u[4] = a2; u[6] = a3;
        u[1] = b0; u[3] = b1; u[5] = b2; u[7] = b3;
    } else {  // R == 3
        const double S3 = 0.86602540378443864676;
        const double2 t = cadd(u[1], u[2]), d = csub(u[1], u[2]);
        const double2 a = make_double2(u[0].x - 0.5 * t.x, u[0].y - 0.5 * t.y);
        const double2 sd = make_double2(-sign * S3 * d.y, sign * S3 * d.x);
        u[0] = cadd(u[0], t);
        u[1] = cadd(a, sd);
        u[2] = csub(a, sd);
    }
}

// u[k] *= w^k, k = 1 .. R-1, for the butterfly's one table twiddle w: the
// powers are complex products (at most three deep, a few units in the last
// place) formed in the order they are used, w^2 = w w, w^3 = w^2 w,
// w^4 = w^2 w^2, w^5 = w^4 w, w^6 = w^4 w^2, w^7 = w^4 w^3, so that no more
// than four of them are live next to the butterfly's R values.
template <int R>
__device__ __forceinline__ void twiddle_apply(double2 (&u)[R], double2 w1) {
    static_assert(R == 2 || R == 3 || R == 4 || R == 8, "radix");
    u[1] = cmul(u[1], w1);
    if constexpr (R >= 3) {
        const double2 w2 = cmul(w1, w1);
        u[2] = cmul(u[2], w2);
        if constexpr (R >= 4) {
            const double2 w3 = cmul(w2, w1);
            u[3] = cmul(u[3], w3);
            if constexpr (R == 8) {
                const double2 w4 = cmul(w2, w2);
                u[4] = cmul(u[4], w4);
                u[5] = cmul(u[5], cmul(w4, w1));
                u[6] = cmul(u[6], cmul(w4, w2));
                u[7] = cmul(u[7], cmul(w4, w3));
            }
        }
    }
}

struct PhysParams {
    const double* p2a;
    double* p2b;
    const double* radial;   // packed radial profiles
    const double* trig;     // [4][nth]: cos, sin, csc, cot
    const double2* wr;      // [nth] exp(2 pi i k / n_phi)
    const double2* twp;     // per-pass FFT twiddles (ip_tw_off; one load per butterfly, twiddle_apply)
    const double2* twq;     // the mid passes' twiddles of the row-pair FFT
    unsigned long long* cfl;
    int L, nth, nr, ncola, ncolb;
    double coriolis;
    int rotation;
    double llmax;
    int nfa, nfb;           // fields per radius of p2a / p2b
    double lorentz;         // Lorentz_Coeff (magnetism)
};

// The row's radial and colatitude factors, kept in shared memory.
enum { RC_RAD, RC_ORAD, RC_RHO, RC_DLNRHO, RC_DR, RC_CS, RC_SN, RC_CSC, RC_COT, RC_COR, RC_C2R, RC_HSF, RC_VH, RC_OH,
       RC_COUNT };

}  // namespace ra
