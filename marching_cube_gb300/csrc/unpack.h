// Exact tsdf unpacking without a division.
//
// The reference unpacks a stored tsdf as (float)tsdf / 32766
// (cu_kinect_fusion_v1.h:253-256), an IEEE-rounded division.  Division by
// this one constant is replaced by q = RN(a * r) with r = RN(1/32766),
// followed by one correction step e = a - q*32766 (exact with an FMA) and
// q' = RN(q + e*r) -- Markstein's correction ("Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. R&D 34(1), 1990).
// tests/test_unpack_exact.py checks that q' equals the IEEE quotient for all
// 65536 int16 inputs, so kernels using it stay bit-exact with the division.
#pragma once

#include <math.h>

#if defined(__CUDACC__)
#define MCG_HD __host__ __device__ __forceinline__
#else
#define MCG_HD inline
#endif

MCG_HD float mcg_unpack_tsdf(int t) {
    const float c = 32766.0f;
    const float r = 1.0f / 32766.0f;  // correctly rounded at compile time
    const float a = (float)t;
    const float q = a * r;
    const float e = fmaf(-q, c, a);
    return fmaf(e, r, q);
}

// RN(a / b) from y = RN(1 / b): two corrections of RN(a * y) by the exact
// remainder.  With |y b - 1| <= 2^-24 b / 2 (b scaled to [1, 2)) the first
// leaves an error of half an ulp and a 2^-23 of one; the second one's is then
// below 2^-48 b / 2 (1 + 2^-22), and no quotient of 24-bit numbers lies nearer
// than 2^-48 (2 / b) to a rounding boundary, unless b's significand is all
// ones, for which mcg_div_reciprocal gives 0.  It gives 0 too where the
// remainders could underflow; with y = 0 the caller divides.  The quotient must not overflow.
MCG_HD float mcg_div_reciprocal(float b) {
    const bool plain = b > 1e-25f && b < 1e25f;
#if defined(__CUDA_ARCH__)
    const unsigned int u = __float_as_uint(b);
#else
    unsigned int u;
    __builtin_memcpy(&u, &b, 4);
#endif
    return plain && (u & 0x7fffffu) != 0x7fffffu ? 1.0f / b : 0.0f;
}

MCG_HD float mcg_div_exact(float a, float b, float y) {
    const float q = a * y;
    const float q1 = fmaf(fmaf(-q, b, a), y, q);
    return fmaf(fmaf(-q1, b, a), y, q1);
}

// Whether a position interpolated between the nodes (i + 0.5) cell and
// (i + 1.5) cell of a volume whose longest side is `side`, divided by cell,
// lies between i + 0.25 and i + 1.75: the voxel of a vertex (rounded down, less
// a half) is then i - 1, i or i + 1 and the first sample of its normal i or
// i + 1.  Every step of the interpolation is monotonic, so the position stays
// between the two nodes as rounded, and node and quotient are each off by at
// most 2^-24 of a coordinate below 2^21, an eighth.  At 2^22 that reaches the
// next voxel, with a subnormal cell anything, and where (side + 1) cell
// overflows positions are infinite or NaN (tests/test_between_nodes.py).
MCG_HD bool mcg_between_nodes(float cell, int side) {
    return cell > 1e-25f && cell < 1e25f && side <= (1 << 21);
}

// org <= i < org + n, for any i
MCG_HD bool mcg_in_tile(int i, int org, int n) {
    return (unsigned int)i - (unsigned int)org < (unsigned int)n;
}
