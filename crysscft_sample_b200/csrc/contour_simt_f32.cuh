// FP32 contour steps for grids off the tensor-core kernels' sizes (odd, unequal sides, up to 64):
// two launches a step in place of three SIMT GEMM passes,
//   plane launch, unit (chain, x): D q(s), A_z, A_y -> exchange buffer
//   slab launch,  unit (chain, y): A_x, D, store q(s+1)
// A tile is in shared memory once per launch, beside the operators it needs; a thread computes
// 4 x 4 results.  Every result is the sum over j = 0 .. n-1 in that order by FMA, with D applied
// to the input of A_z and to the result of A_x: the arithmetic of the passes (axis_kernels.cuh),
// bit for bit.  The launches are programmatic, as in contour_step.cuh.
// Both chains, a step (one B200): 45^3 P1 10.6 us against 32.4 in three passes, 17 x 25 x 23 PMMM 6.2
// against 24.3, 20 x 64 x 33 P1 12.2 against 31.6.  The FMAs of a 45^3 unit take 1.7 us, the two
// waits for the launch before about 3; the rest is shared-memory latency in the K loops.
#pragma once
#include <cuda_runtime.h>

#include "contour_step.cuh"

namespace crysscft {

constexpr int kSimtMaxN = 64;
constexpr int kSimtThreads = 256;

struct ContourSimtArgsF {
    const float* in[2];   // plane: q(s); slab: the exchange buffer
    float* out[2];        // plane: the exchange buffer; slab: q(s+1)
    const float* w[2];    // Boltzmann factor of the step
    const float* opT[2];  // transposed operators (n x n): plane A_z, A_y; slab A_x
    int n[3];
    int plane;
    PhiStep<float> phi;
};

__host__ __device__ inline int simt_ld(int n) { return ((n + 3) & ~3) + 4; }
inline size_t simt_smem(int nx, int ny, int nz) {
    const size_t plane = (size_t)nz * simt_ld(ny) + (size_t)ny * simt_ld(nz) + (size_t)nz * simt_ld(nz) + (size_t)ny * simt_ld(ny);
    const size_t slab = (size_t)nx * simt_ld(nz) + (size_t)nx * simt_ld(nx);
    return (plane > slab ? plane : slab) * sizeof(float);
}

// acc[a][b] = sum_k A[k lda + 4 ty + a] B[k ldb + 4 tx + b], k ascending
__device__ __forceinline__ void simt_tile(const float* A, int lda, const float* B, int ldb, int K, float (&acc)[4][4]) {
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = 0.0f;
#pragma unroll 4
    for (int k = 0; k < K; ++k) {
        const float4 x = *reinterpret_cast<const float4*>(A + k * lda);
        const float4 y = *reinterpret_cast<const float4*>(B + k * ldb);
        const float xa[4] = {x.x, x.y, x.z, x.w}, yb[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) acc[a][b] = fmaf(xa[a], yb[b], acc[a][b]);
    }
}

__global__ void __launch_bounds__(kSimtThreads, 2) contour_simt_kernel_f32(const ContourSimtArgsF a) {
    const int nx = a.n[0], ny = a.n[1], nz = a.n[2];
    const bool plane = a.plane != 0;
    const int lx = simt_ld(nx), ly = simt_ld(ny), lz = simt_ld(nz);
    const long long psz = (long long)ny * nz;
    extern __shared__ __align__(16) float sim[];
    const int tid = threadIdx.x;
    // operators, padded rows zero-filled (their sums are not stored)
    auto put_op = [&](float* dst, const float* opT, int n, int ld) {
        for (int e = tid; e < n * ld; e += kSimtThreads) {
            const int j = e / ld, i = e - j * ld;
            dst[e] = i < n ? __ldcg(opT + j * n + i) : 0.0f;
        }
    };
    float* T = sim;  // plane: [z][y] (D q transposed); slab: [x][z]
    float* op0 = plane ? T + nz * ly + ny * lz : T + nx * lz;
    put_op(op0, a.opT[0], plane ? nz : nx, plane ? lz : lx);
    float* T2 = T + nz * ly;  // plane: [y][z] after A_z
    float* op1 = op0 + nz * lz;
    if (plane) put_op(op1, a.opT[1], ny, ly);
    phi_step(a.phi, (long long)nx * psz);
    pdl_wait();
    pdl_launch_dependents();

    const int units = nx > ny ? nx : ny;
    const int c = (int)blockIdx.x >= units ? 1 : 0, p = (int)blockIdx.x - c * units;
    if (p >= (plane ? nx : ny)) return;
    const float* in = c ? a.in[1] : a.in[0];
    float* out = c ? a.out[1] : a.out[0];
    const float* w = c ? a.w[1] : a.w[0];
    const int tx = tid & 15, ty = tid >> 4;
    float acc[4][4];
    if (plane) {
        const float* src = in + p * psz;
        const float* ws = w + p * psz;
#pragma unroll 4
        for (int e = tid; e < ny * nz; e += kSimtThreads) {
            const int y = e / nz, z = e - y * nz;
            T[z * ly + y] = __ldcg(src + e) * __ldcg(ws + e);
        }
        __syncthreads();
        if (4 * ty < ny && 4 * tx < nz) {
            simt_tile(T + 4 * ty, ly, op0 + 4 * tx, lz, nz, acc);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (4 * ty + i < ny)
                    *reinterpret_cast<float4*>(T2 + (4 * ty + i) * lz + 4 * tx) =
                        make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        }
        __syncthreads();
        if (4 * ty < ny && 4 * tx < nz) {
            simt_tile(op1 + 4 * ty, ly, T2 + 4 * tx, lz, ny, acc);
            float* dst = out + p * psz;
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (4 * ty + i < ny && 4 * tx + j < nz) __stcg(dst + (4 * ty + i) * nz + 4 * tx + j, acc[i][j]);
        }
        return;
    }
    const float* src = in + (long long)p * nz;
#pragma unroll 4
    for (int e = tid; e < nx * nz; e += kSimtThreads) {
        const int x = e / nz, z = e - x * nz;
        T[x * lz + z] = __ldcg(src + x * psz + z);
    }
    __syncthreads();
    if (4 * ty < nx && 4 * tx < nz) {
        float f[4][4];
        const float* ws = w + (long long)p * nz;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                f[i][j] = 4 * ty + i < nx && 4 * tx + j < nz ? __ldcg(ws + (4 * ty + i) * psz + 4 * tx + j) : 0.0f;
        simt_tile(op0 + 4 * ty, lx, T + 4 * tx, lz, nx, acc);
        float* dst = out + (long long)p * nz;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (4 * ty + i < nx && 4 * tx + j < nz)
                    __stcg(dst + (4 * ty + i) * psz + 4 * tx + j, acc[i][j] * f[i][j]);
    }
}

}  // namespace crysscft
