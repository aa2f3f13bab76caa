// FP64 tile engine of the Legendre products: a 64 x 64 CTA tile of C += A B with the FP64
// tensor-core instruction mma.sync.m8n8k4.f64 (4 warps, 32 x 32 per warp), operands staged by
// cp.async in a ring of three k-tiles of 16.
//
// What bounds it: the FP64 tensor pipe (one mma per 16 cycles and SM quarter).  K is the number of
// l of one parity, 128 on average at l_max = 511, so that a tile is only eight k-tiles long: the
// copies of the next two k-tiles are in flight without holding registers, one barrier serves a
// k-tile, and fragments are read in 16-byte pieces, half the shared-memory instructions of
// element-wise ones (l_max 511, N_r 96 with B: inverse 12.63 -> 10.73 ms, 0.86 of DGEMM, forward 5.67 ->
// 5.12): a lane's two neighbouring rows (or columns) belong to two mma tiles, so that the
// tile's rows and columns come out permuted (acc_each knows the order), four neighbouring columns a lane.
#pragma once

#include <cuda_runtime.h>

namespace ra {

constexpr int GEMM_THREADS = 128, GA_STAGES = 3, GA_BK = 16, GA_BM = 64, GA_BN = 64;

// 32 x 32 per warp: mma tile (i, j), two columns a lane
struct Acc {
    double v[4][4][2];
    __device__ void zero() {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) v[i][j][0] = v[i][j][1] = 0.0;
    }
};

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// Copies of 16 bytes, or two of 8 where the operand is only 8-byte aligned; bytes = 0 writes zeros.
template <bool VEC>
__device__ __forceinline__ void ga_copy(double* dst, const double* src, bool ok) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
    if constexpr (VEC) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(src), "r"(ok ? 16 : 0) : "memory");
    } else {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(src), "r"(ok ? 8 : 0) : "memory");
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s + 8), "l"(src + (ok ? 1 : 0)), "r"(ok ? 8 : 0) : "memory");
    }
}

// Operand with x contiguous: element (k, x) at p[k ld + x], zero past K or X (X and ld even).
// Tile [k][x]; PAD doubles a row.
template <bool VEC, int PAD>
struct OperandX {
    static constexpr int LD = 64 + PAD, SIZE = GA_BK * LD;
    const double* p;
    long ld;
    int K, X;
    __device__ __forceinline__ void stage(double* tile, int k0) const {
#pragma unroll
        for (int i = 0; i < GA_BK * 32 / GEMM_THREADS; ++i) {
            const int e = threadIdx.x + i * GEMM_THREADS, k = e >> 5, x = (e & 31) * 2;
            const bool ok = k0 + k < K && x < X;
            ga_copy<VEC>(tile + k * LD + x, ok ? p + (long)(k0 + k) * ld + x : p, ok);
        }
    }
};

// Operand with k contiguous: element (k, x) at p[x ld + k] (K and ld even).  Tile [x][k]; rows of 24
// doubles put the two rows of a fragment phase in different halves of the banks.
struct OperandK {
    static constexpr int LD = GA_BK + 8, SIZE = 64 * LD;
    const double* p;
    long ld;
    int K, X;
    __device__ __forceinline__ void stage(double* tile, int k0) const {
#pragma unroll
        for (int i = 0; i < 64 * 8 / GEMM_THREADS; ++i) {
            const int e = threadIdx.x + i * GEMM_THREADS, x = e >> 3, k = (e & 7) * 2;
            const bool ok = k0 + k < K && x < X;
            ga_copy<true>(tile + x * LD + k, ok ? p + (long)x * ld + k0 + k : p, ok);
        }
    }
};

template <class OA, class OB>
constexpr size_t ga_smem() { return (size_t)GA_STAGES * (OA::SIZE + OB::SIZE) * sizeof(double); }

// acc += A B over K.  An operand with x contiguous: the row (column) of acc index i, lane row g is
// 16 (i / 2) + 2 g + i % 2; with k contiguous: 8 i + g.  AK, BK: which of them have k contiguous (B
// only together with A).
template <bool AK, bool BK, class OA, class OB>
__device__ __forceinline__ void gemm_async(Acc& acc, const OA& oa, const OB& ob, int K, double* sm) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, tig = lane & 3;
    const int wm = warp & 1, wn = warp >> 1;
    double* As = sm;
    double* Bs = sm + GA_STAGES * OA::SIZE;
    const int nk = (K + GA_BK - 1) / GA_BK;
    auto issue = [&](int kt) {
        if (kt < nk) {
            oa.stage(As + (kt % GA_STAGES) * OA::SIZE, kt * GA_BK);
            ob.stage(Bs + (kt % GA_STAGES) * OB::SIZE, kt * GA_BK);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
#pragma unroll
    for (int s = 0; s < GA_STAGES - 1; ++s) issue(s);
    for (int kt = 0; kt < nk; ++kt) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(GA_STAGES - 2) : "memory");
        __syncthreads();   // k-tile kt is there; every warp is done with the one whose place the next copy takes
        issue(kt + GA_STAGES - 1);
        const double* a_t = As + (kt % GA_STAGES) * OA::SIZE;
        const double* b_t = Bs + (kt % GA_STAGES) * OB::SIZE;
        if constexpr (AK) {
            // the k of a group of 8 go to two mma steps: lane tig takes k = 2 tig and 2 tig + 1
#pragma unroll
            for (int h = 0; h < GA_BK; h += 8) {
                double2 a[4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    a[i] = *reinterpret_cast<const double2*>(a_t + (wm * 32 + i * 8 + g) * OA::LD + h + 2 * tig);
                if constexpr (BK) {
                    double2 b[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        b[j] = *reinterpret_cast<const double2*>(b_t + (wn * 32 + j * 8 + g) * OB::LD + h + 2 * tig);
#pragma unroll
                    for (int s = 0; s < 2; ++s)
#pragma unroll
                        for (int i = 0; i < 4; ++i)
#pragma unroll
                            for (int j = 0; j < 4; ++j) dmma(acc.v[i][j], s ? a[i].y : a[i].x, s ? b[j].y : b[j].x);
                }
#pragma unroll
                for (int s = 0; !BK && s < 2; ++s) {
                    double2 b[2];
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        b[j] = *reinterpret_cast<const double2*>(b_t + (h + 2 * tig + s) * OB::LD + wn * 32 + j * 16 + 2 * g);
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            dmma(acc.v[i][j], s ? a[i].y : a[i].x, (j & 1) ? b[j >> 1].y : b[j >> 1].x);
                }
            }
        } else {
#pragma unroll
            for (int kk = 0; kk < GA_BK; kk += 4) {
                double2 a[2], b[2];
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    a[i] = *reinterpret_cast<const double2*>(a_t + (kk + tig) * OA::LD + wm * 32 + i * 16 + 2 * g);
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    b[j] = *reinterpret_cast<const double2*>(b_t + (kk + tig) * OB::LD + wn * 32 + j * 16 + 2 * g);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        dmma(acc.v[i][j], (i & 1) ? a[i >> 1].y : a[i >> 1].x, (j & 1) ? b[j >> 1].y : b[j >> 1].x);
            }
        }
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// Visits the accumulator two neighbouring columns at a time: f(m, n, value at n, value at n + 1), n even.
template <bool AK, class F>
__device__ __forceinline__ void acc_each(const Acc& acc, const F& f) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, tig = lane & 3;
    const int wm = warp & 1, wn = warp >> 1;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = wm * 32 + (AK ? i * 8 + g : (i >> 1) * 16 + 2 * g + (i & 1));
#pragma unroll
        for (int jp = 0; jp < 2; ++jp)
#pragma unroll
            for (int q = 0; q < 2; ++q)
                f(m, wn * 32 + jp * 16 + 4 * tig + 2 * q, acc.v[i][2 * jp][q], acc.v[i][2 * jp + 1][q]);
    }
}

}  // namespace ra
