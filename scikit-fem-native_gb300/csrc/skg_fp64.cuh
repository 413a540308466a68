// FP64 additions and products as fused multiply-adds.
//
// On GB300 a DFMA with three register operands takes 8.15 ns per warp and SM, a
// DADD or DMUL (and a DFMA with an operand from the constant bank) 9.67 ns
// (measured with eight independent chains per thread and 64 warps per SM).  The
// kernels that are bound by the FP64 pipe therefore add as a * 1 + b and
// multiply as a * b + (-0): the same results bit for bit, signs of zero
// included.  The constants are loaded through an opaque instruction, so that
// they stay in registers and the compiler does not fold them back.
#pragma once

namespace skg {

static __device__ double g_fp64_units[3] = {1.0, -0.0, 3.0};

struct Fp64 {
    double one, none, three_;

    static __device__ __forceinline__ Fp64 load() {
        Fp64 f;
        asm volatile("ld.global.f64 %0, [%1];" : "=d"(f.one) : "l"(g_fp64_units));
        asm volatile("ld.global.f64 %0, [%1];" : "=d"(f.none) : "l"(g_fp64_units + 1));
        asm volatile("ld.global.f64 %0, [%1];" : "=d"(f.three_) : "l"(g_fp64_units + 2));
        return f;
    }
    static __device__ __forceinline__ double unit() {
        double one;
        asm volatile("ld.global.f64 %0, [%1];" : "=d"(one) : "l"(g_fp64_units));
        return one;
    }
    __device__ __forceinline__ double add(double a, double b) const { return fma(a, one, b); }
    __device__ __forceinline__ double sub(double a, double b) const { return fma(a, one, -b); }
    __device__ __forceinline__ double mul(double a, double b) const { return fma(a, b, none); }
    __device__ __forceinline__ double add3(double a, double b, double c) const { return add(add(a, b), c); }
    // a0 b0 + a1 b1 + a2 b2
    __device__ __forceinline__ double dot(const double a[3], const double b[3]) const {
        return fma(a[2], b[2], fma(a[1], b[1], mul(a[0], b[0])));
    }
    // a b - c d
    __device__ __forceinline__ double cross(double a, double b, double c, double d) const {
        return fma(a, b, -mul(c, d));
    }
    // Rows 1..3 of the adjugate of M (column r = edge r, row i = coordinate i at
    // M[3 i + r]): det M times the rows of its inverse.  Returns det M.
    __device__ __forceinline__ double adjugate(const double M[9], double b[4][3]) const {
        b[1][0] = cross(M[4], M[8], M[5], M[7]);
        b[1][1] = cross(M[2], M[7], M[1], M[8]);
        b[1][2] = cross(M[1], M[5], M[2], M[4]);
        b[2][0] = cross(M[5], M[6], M[3], M[8]);
        b[2][1] = cross(M[0], M[8], M[2], M[6]);
        b[2][2] = cross(M[2], M[3], M[0], M[5]);
        b[3][0] = cross(M[3], M[7], M[4], M[6]);
        b[3][1] = cross(M[1], M[6], M[0], M[7]);
        b[3][2] = cross(M[0], M[4], M[1], M[3]);
        return fma(M[2], b[3][0], fma(M[1], b[2][0], mul(M[0], b[1][0])));
    }
};

}  // namespace skg
