// FP32 contours (3xTF32), one launch per phase: contour_alt_kernel_f32's schedule and tile
// operations, so its results bit for bit, without its release flags,
//   plane phase:  [A_z A_y]  D  store q  D  [A_z A_y]  -> exchange XP
//   slab phase:       [A_x]  D  store q  D  [A_x]      -> exchange XS
// The launches order the exchange (programmatic launches, as contour_any_kernel in
// contour_step.cuh): the operators of the layout and the Boltzmann tiles of a phase are copied
// while the launch before it runs, two CTAs an SM.  The persistent kernel spends half of a step
// waiting: 1.35 ms an iteration at 64^3 (Ns = 200) against 1.16 ms
// here, 0.33 against 0.22 ms at 16^3 (Ns = 100).
#pragma once
#include <cuda_runtime.h>

#include "contour_kernel_f32.cuh"
#include "contour_step.cuh"

namespace crysscft {

struct ContourStepArgsF {
    const float* in[2];   // k = 0: the initial slice; else the exchange buffer of the other layout
    float* q[2];          // k >= 1: the finished slice
    float* xout[2];       // k < U: this layout's exchange buffer
    const float* w0[2];   // k >= 1: Boltzmann factor of the finished step
    const float* w1[2];   // k < U: of the started step
    const float* ops;     // packed FP32 operators (hi/lo), x then y then z
    int plane, finish, start;
    PhiStep<float> phi;
};

template <int N, bool EO>
struct StepShapeF {
    static constexpr int LF = N + 4;
    static constexpr int AX = AxisShapeF<N, EO>::SIZE;
    static constexpr int TILE = (N * LF + 3) & ~3;
    // two work tiles, the two Boltzmann tiles, the operators of the layout (z and y, or x)
    static constexpr size_t SMEM = (size_t)(4 * TILE + 2 * AX) * sizeof(float);
};

template <int N, bool EO>
__global__ void __launch_bounds__(kContourThreads, 2) contour_step_kernel_f32(const ContourStepArgsF a) {
    using S = StepShapeF<N, EO>;
    constexpr int LF = S::LF;
    constexpr long long PLANE = (long long)N * N;
    extern __shared__ __align__(16) float stf[];
    float* T0 = stf;
    float* T1 = T0 + S::TILE;
    float* W0 = T1 + S::TILE;
    float* W1 = W0 + S::TILE;
    float* opc = W1 + S::TILE;      // A_y on planes, A_x on slabs
    float* opz = opc + S::AX;
    const bool plane = a.plane != 0;
    const int c = (int)blockIdx.x >= N ? 1 : 0, p = (int)blockIdx.x - c * N;
    const long long off = plane ? p * PLANE : (long long)p * N, gs = plane ? N : PLANE;
    const float* w0 = a.finish ? (c ? a.w0[1] : a.w0[0]) + off : nullptr;
    const float* w1 = a.start ? (c ? a.w1[1] : a.w1[0]) + off : w0;
    op_copy_async(opc, a.ops + (plane ? S::AX : 0), S::AX);
    if (plane) op_copy_async(opz, a.ops + 2 * S::AX, S::AX);
    if (a.finish) {  // the factors are older than the launch before this one
        tile_fetch_f32<N, LF>(W0, w0, gs);
        if (w1 != w0) tile_fetch_f32<N, LF>(W1, w1, gs);
    }
    cp_async_commit();
    phi_step(a.phi, PLANE * N);
    pdl_wait();
    pdl_launch_dependents();

    const float* in = (c ? a.in[1] : a.in[0]) + off;
    tile_fetch_f32<N, LF>(T0, in, gs);
    if (!a.finish) tile_fetch_f32<N, LF>(W0, w1, gs);
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
    float* cur = T0;
    float* oth = T1;
    if (a.finish) {
        ColOutF fo{plane ? T0 : T1, gs};
        fo.w0 = W0;
        fo.w1 = w1 != w0 ? W1 : W0;
        fo.qs = (c ? a.q[1] : a.q[0]) + off;
        fo.start = a.start;
        if (plane) {
            row_op_f32<N, N, LF, EO>(T0, T1, opz);
            __syncthreads();
            col_op_f32<N, N, LF, EO, kFinishDirect>(T1, fo, opc);
        } else {
            col_op_f32<N, N, LF, EO, kFinishDirect>(T0, fo, opc);
            cur = T1;
            oth = T0;
        }
        __syncthreads();
    } else {
        for (int e = threadIdx.x; e < N * N; e += kContourThreads) {
            const int r = e / N, z = e - (e / N) * N;
            T0[r * LF + z] *= W0[r * LF + z];
        }
        __syncthreads();
    }
    if (!a.start) return;
    const ColOutF xo{(c ? a.xout[1] : a.xout[0]) + off, gs};
    if (plane) {
        row_op_f32<N, N, LF, EO>(cur, oth, opz);
        __syncthreads();
        col_op_f32<N, N, LF, EO, kToGlobal>(oth, xo, opc);
    } else {
        col_op_f32<N, N, LF, EO, kToGlobal>(cur, xo, opc);
    }
}

}  // namespace crysscft
