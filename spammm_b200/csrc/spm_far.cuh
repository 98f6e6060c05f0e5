// spm_far.cuh -- blocks of grid nodes with a far field: the Chebyshev points and interpolation weights of a
// block, and the test that an atom is far from it (the reasons for the constants stand in grid_build.cu).
#pragma once
#include <cuda_runtime.h>
#include <cmath>
#include "spm_batch.cuh"

namespace spm {

constexpr int FB = SPM_FAR_BLOCK;
constexpr int FP = 8;
constexpr int FN = FP * FP * FP;
constexpr float FAR_RATIO = 9.f;
constexpr int FAR_FEWEST = 8;        // far atoms that pay for an interpolation (it costs about 4 atoms at the nodes)

// Lagrange weights of the Chebyshev points c at the nodes of a block (L), and of a
// group's points at the points of its lower and upper blocks (T).
struct FarTab {
    float L[FB][FP];
    float T[2][FP][FP];
    float c[FP];
};

inline FarTab make_far_tab() {
    FarTab t;
    double c[FP];
    for (int k = 0; k < FP; k++) c[k] = cos((2 * k + 1) * 3.14159265358979323846 / (2 * FP));
    auto weight = [&](double x, int k) {
        double w = 1.0;
        for (int j = 0; j < FP; j++)
            if (j != k) w *= (x - c[j]) / (c[k] - c[j]);
        return w;
    };
    for (int i = 0; i < FB; i++)
        for (int k = 0; k < FP; k++) t.L[i][k] = (float)weight((2.0 * i - (FB - 1)) / (FB - 1), k);
    for (int s = 0; s < 2; s++)
        for (int i = 0; i < FP; i++)
            for (int k = 0; k < FP; k++)
                t.T[s][i][k] = (float)weight(((s ? 0.5 : -0.5) * FB + 0.5 * (FB - 1) * c[i]) / (0.5 * (2 * FB - 1)), k);
    for (int k = 0; k < FP; k++) t.c[k] = (float)c[k];
    return t;
}

// Centre and squared far distance of a cube of nodes with corner (x, y, z) and edge n.  h: half-edge,
// the largest of the three axes' and of the corner distance over sqrt(3) (skew cells).  Fixed operation
// order: batch and single builds classify alike.
struct FarCube {
    float x, y, z, lim2, h, half;
};

__device__ __forceinline__ float len3(float x, float y, float z) {
    return __fsqrt_rn(__fmaf_rn(z, z, __fmaf_rn(y, y, __fmul_rn(x, x))));
}

// Geom: p0, dA, dB, dC of the grid.
template <class Geom>
__device__ __forceinline__ FarCube far_cube(const Geom& G, int x, int y, int z, int n) {
    FarCube C;
    C.half = 0.5f * (float)(n - 1);
    const float cx = (float)x + C.half, cy = (float)y + C.half, cz = (float)z + C.half;
    C.x = __fmaf_rn(G.dB.x, cy, __fmaf_rn(G.dA.x, cx, G.p0.x));
    C.y = __fmaf_rn(G.dB.y, cy, __fmaf_rn(G.dA.y, cx, G.p0.y));
    C.z = __fmaf_rn(G.dC.z, cz, __fmaf_rn(G.dB.z, cy, __fmaf_rn(G.dA.z, cx, G.p0.z)));
    float e = fmaxf(fmaxf(len3(G.dA.x, G.dA.y, G.dA.z), len3(G.dB.x, G.dB.y, G.dB.z)), fabsf(G.dC.z));
#pragma unroll
    for (int s = 0; s < 4; s++) {
        const float sb = s & 1 ? -1.f : 1.f, sc = s & 2 ? -1.f : 1.f;
        e = fmaxf(e, __fmul_rn(0.57735027f, len3(__fmaf_rn(sb, G.dB.x, G.dA.x), __fmaf_rn(sb, G.dB.y, G.dA.y),
                                                 __fmaf_rn(sc, G.dC.z, __fmaf_rn(sb, G.dB.z, G.dA.z)))));
    }
    C.h = __fmul_rn(e, C.half);
    C.lim2 = __fmul_rn(__fmul_rn(FAR_RATIO, C.h), __fmul_rn(FAR_RATIO, C.h));
    return C;
}

}  // namespace spm
