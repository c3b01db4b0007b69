// One contour step per launch for cubic grids of side 96 and 128, whose planes fit in shared
// memory once but whose whole-contour kernel (several tiles per CTA) does not.
//
// The alternating schedule of contour_alt_kernel, one phase per launch: a phase holds an n x n
// tile (x-plane in even phases, y-slab in odd ones) of each chain in shared memory, finishes
// step k-1 and starts step k on it,
//   plane phase:  [A_z A_y]  D  store q  D  [A_y]  -> exchange buffer XP
//   slab phase:   [A_z A_x]  D  store q  D  [A_x]  -> exchange buffer XS
// so a step moves the field four times (exchange in and out, q, D) where the three axis passes
// move it seven times, and takes one launch instead of three.
//
// Every axis operation works in place on one tile: a warp owns 8 ML whole lines (rows for A_z,
// columns for A_y and A_x), reads each value of them once, forms the mirrored sums and
// differences in registers, keeps all their results in its accumulators and writes them back.
// So A_z starts on a warp's rows as soon as its own copies have landed, the finishing and the
// starting column operation of a phase need no barrier between them, and one barrier (A_z to
// columns) is left per tile.  The operator blocks are those of axis_mma.cuh (kEo2, kCirc4).
#pragma once
#include <cuda_runtime.h>

#include "axis_mma.cuh"

namespace crysscft {

struct ContourStepArgs {
    const double* in[2];   // k = 0: the initial slice; else the exchange buffer of the other layout
    double* q[2];          // k >= 1: the finished slice
    double* xout[2];       // k < U: this layout's exchange buffer
    const double* w0[2];   // k >= 1: Boltzmann factor of the finished step
    const double* w1[2];   // k < U: of the started step
    const double* opz;     // packed blocks of A_z
    const double* opc;     // ... of the layout's column axis (A_y on planes, A_x on slabs)
    int nchain;
    int plane;             // 1: x-planes, 0: y-slabs
    int finish, start;     // k >= 1, k < U
};

template <int MODE, int N, int ML>
struct StepShape {
    static_assert(MODE == kEo2 || MODE == kCirc4, "block forms of 96- and 128-point axes");
    static constexpr int LF = N + 4;
    static constexpr int THREADS = N / (8 * ML) * 32;
    static constexpr int H = N / 4, G = H / 8, HALF = N / 2;
    static constexpr int LD = H + 4, LDO = HALF + 4, BLK = H * LD;
    static constexpr int OP = MODE == kEo2 ? 2 * BLK + HALF * LDO : 4 * BLK;
    static constexpr int TILE = N * LF;
    static constexpr size_t smem(bool one_op) { return (size_t)(TILE + (one_op ? 1 : 2) * OP) * sizeof(double); }
};

// acc[block][group][m] += the blocks of one axis operation on the warp's lines line0..
// ROW: lines are rows of T (values at T[line][j]), else columns (T[j][line]).
template <int MODE, int N, int ML, bool ROW>
__device__ __forceinline__ void warp_axis_mma(const double* T, const double* op, int line0,
                                              double (&acc)[4][StepShape<MODE, N, ML>::G][ML][2]) {
    using S = StepShape<MODE, N, ML>;
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int r = 0; r < S::G; ++r)
#pragma unroll
            for (int m = 0; m < ML; ++m) acc[a][r][m][0] = acc[a][r][m][1] = 0.0;
    constexpr int KS = ROW ? 1 : S::LF;               // stride of the position along the line
    const double* f = ROW ? T + (line0 + g) * S::LF : T + line0 + g;
    const double* B = op + g * S::LD + t;
    const double* OA = op + 2 * S::BLK + g * S::LDO;                   // row 8 r + g of O
    const double* OB = op + 2 * S::BLK + (S::HALF - 1 - g) * S::LDO;   // row half - 1 - (8 r + g)
    auto mma = [&](double (&d)[2], double x, double o) {
        if (ROW) dmma884(d, x, o);
        else dmma884(d, o, x);
    };
#pragma unroll
    for (int k0 = 0; k0 < S::H; k0 += 4) {
        const int j = k0 + t;
        double a0[ML], a1[ML], a2[ML], a3[ML];
#pragma unroll
        for (int m = 0; m < ML; ++m) {
            const double* fm = f + m * 8 * (ROW ? S::LF : 1);
            const double x0 = fm[j * KS], x1 = fm[(N - 1 - j) * KS];
            const double x2 = fm[(S::HALF - 1 - j) * KS], x3 = fm[(S::HALF + j) * KS];
            if constexpr (MODE == kEo2) {
                const double s = x0 + x1, d = x2 + x3;
                a0[m] = s + d;
                a1[m] = s - d;
                a2[m] = x0 - x1;  // v_j
                a3[m] = x2 - x3;  // v_{half-1-j}
            } else {
                const double u0 = x0 + x3, v0 = x0 - x3, u1 = x2 + x1, v1 = x2 - x1;
                a0[m] = u0 + u1;
                a1[m] = u0 - u1;
                a2[m] = v0 + v1;
                a3[m] = v0 - v1;
            }
        }
#pragma unroll
        for (int r = 0; r < S::G; ++r) {
            const double o0 = B[8 * r * S::LD + k0], o1 = B[S::BLK + 8 * r * S::LD + k0];
#pragma unroll
            for (int m = 0; m < ML; ++m) {
                mma(acc[0][r][m], a0[m], o0);
                mma(acc[1][r][m], a1[m], o1);
            }
            if constexpr (MODE == kEo2) {
                const double oa0 = OA[8 * r * S::LDO + j], oa1 = OA[8 * r * S::LDO + S::HALF - 1 - j];
                const double ob0 = OB[-8 * r * S::LDO + j], ob1 = OB[-8 * r * S::LDO + S::HALF - 1 - j];
#pragma unroll
                for (int m = 0; m < ML; ++m) {
                    mma(acc[2][r][m], a2[m], oa0);
                    mma(acc[3][r][m], a2[m], ob0);
                    mma(acc[2][r][m], a3[m], oa1);
                    mma(acc[3][r][m], a3[m], ob1);
                }
            } else {
                const double o2 = B[2 * S::BLK + 8 * r * S::LD + k0], o3 = B[3 * S::BLK + 8 * r * S::LD + k0];
#pragma unroll
                for (int m = 0; m < ML; ++m) {
                    mma(acc[2][r][m], a2[m], o2);
                    mma(acc[3][r][m], a3[m], o3);
                }
            }
        }
    }
}

// The four results of a pair index i from its block sums: at positions i, n-1-i, half-1-i, half+i.
template <int MODE>
__device__ __forceinline__ void pair_results(double b0, double b1, double b2, double b3, double (&y)[4]) {
    const double p1 = b0 + b1, p2 = b0 - b1;
    if constexpr (MODE == kEo2) {
        y[0] = p1 + b2;
        y[1] = p1 - b2;
        y[2] = p2 + b3;
        y[3] = p2 - b3;
    } else {
        const double v0 = b2 + b3, v1 = b2 - b3;
        y[0] = p1 + v0;
        y[3] = p1 - v0;
        y[2] = p2 + v1;
        y[1] = p2 - v1;
    }
}

template <int MODE, int N, int ML>
__global__ void __launch_bounds__(StepShape<MODE, N, ML>::THREADS, 1) contour_step_kernel(const ContourStepArgs p) {
    using S = StepShape<MODE, N, ML>;
    constexpr int LF = S::LF, G = S::G, HALF = S::HALF;
    extern __shared__ __align__(16) double stp[];
    double* T = stp;
    double* opz = stp + S::TILE;
    double* opc = p.opc == p.opz ? opz : opz + S::OP;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int line0 = warp * 8 * ML;  // this warp's rows and columns

    for (int i = threadIdx.x; i < S::OP / 2; i += S::THREADS) cp_async16(opz + 2 * i, p.opz + 2 * i);
    if (opc != opz)
        for (int i = threadIdx.x; i < S::OP / 2; i += S::THREADS) cp_async16(opc + 2 * i, p.opc + 2 * i);
    cp_async_commit();
    cp_async_wait_all();
    pdl_wait();  // everything above reads only the operators
    pdl_launch_dependents();
    __syncthreads();

    const long long gs = p.plane ? N : (long long)N * N;  // global row stride of a tile
    for (int u = blockIdx.x; u < p.nchain * N; u += gridDim.x) {
        const int c = u >= N ? 1 : 0, idx = u - c * N;
        const long long off = p.plane ? (long long)idx * N * N : (long long)idx * N;
        const double* in = (c ? p.in[1] : p.in[0]) + off;
        // this warp's rows (16-byte chunks)
#pragma unroll 8
        for (int e = lane; e < 8 * ML * (N / 2); e += 32) {
            const int r = line0 + e / (N / 2), ch = e % (N / 2);
            cp_async16(T + r * LF + 2 * ch, in + r * gs + 2 * ch);
        }
        cp_async_commit();
        cp_async_wait_all();
        __syncwarp();
        double acc[4][G][ML][2];
        // Boltzmann factors of this lane's results in (group, m) order, loaded one (group, m) ahead:
        // loaded where they are used, each of the G ML loads put its latency into the epilogue
        const int rowpos[4] = {g, N - 1 - g, HALF - 1 - g, HALF + g};  // + 8 r, - 8 r, - 8 r, + 8 r
        auto factors = [&](const double* w, int it, double2 (&f)[4]) {
            const int r = it / ML, col = line0 + 8 * (it % ML) + 2 * t;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int at = rowpos[k] + (k == 0 || k == 3 ? 8 * r : -8 * r);
                f[k] = __ldg(reinterpret_cast<const double2*>(w + at * gs + col));
            }
        };
        const double* w0 = p.finish ? (c ? p.w0[1] : p.w0[0]) + off : nullptr;
        const double* w1 = p.start ? (c ? p.w1[1] : p.w1[0]) + off : nullptr;
        if (p.finish) {
            warp_axis_mma<MODE, N, ML, true>(T, opz, line0, acc);
            __syncwarp();
#pragma unroll
            for (int r = 0; r < G; ++r)
#pragma unroll
                for (int m = 0; m < ML; ++m) {
                    double y0[4], y1[4];
                    pair_results<MODE>(acc[0][r][m][0], acc[1][r][m][0], acc[2][r][m][0], acc[3][r][m][0], y0);
                    pair_results<MODE>(acc[0][r][m][1], acc[1][r][m][1], acc[2][r][m][1], acc[3][r][m][1], y1);
                    double* row = T + (line0 + 8 * m + g) * LF;
                    const int i = 8 * r + 2 * t;
                    *reinterpret_cast<double2*>(row + i) = make_double2(y0[0], y1[0]);
                    *reinterpret_cast<double2*>(row + N - 2 - i) = make_double2(y1[1], y0[1]);
                    *reinterpret_cast<double2*>(row + HALF - 2 - i) = make_double2(y1[2], y0[2]);
                    *reinterpret_cast<double2*>(row + HALF + i) = make_double2(y0[3], y1[3]);
                }
            __syncthreads();  // every row is through A_z
            double2 fnext[4];
            factors(w0, 0, fnext);
            warp_axis_mma<MODE, N, ML, false>(T, opc, line0, acc);
            __syncwarp();
            double* q = (c ? p.q[1] : p.q[0]) + off;
            const bool other_w = w1 && w1 != w0;
#pragma unroll
            for (int it = 0; it < G * ML; ++it) {
                const int r = it / ML, m = it % ML;
                double2 f[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) f[k] = fnext[k];
                if (it + 1 < G * ML) factors(w0, it + 1, fnext);
                double y0[4], y1[4];
                pair_results<MODE>(acc[0][r][m][0], acc[1][r][m][0], acc[2][r][m][0], acc[3][r][m][0], y0);
                pair_results<MODE>(acc[0][r][m][1], acc[1][r][m][1], acc[2][r][m][1], acc[3][r][m][1], y1);
                const int col = line0 + 8 * m + 2 * t;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int at = rowpos[k] + (k == 0 || k == 3 ? 8 * r : -8 * r);
                    const double2 v = make_double2(y0[k] * f[k].x, y1[k] * f[k].y);
                    __stcs(reinterpret_cast<double2*>(q + at * gs + col), v);
                    double2 f1 = f[k];
                    if (other_w) f1 = __ldg(reinterpret_cast<const double2*>(w1 + at * gs + col));
                    *reinterpret_cast<double2*>(T + at * LF + col) = make_double2(v.x * f1.x, v.y * f1.y);
                }
            }
            __syncwarp();
        } else {
            // the first phase: D q(0) on this warp's rows
#pragma unroll 8
            for (int e = lane; e < 8 * ML * (N / 2); e += 32) {
                const int r = line0 + e / (N / 2), ch = 2 * (e % (N / 2));
                double2 v = *reinterpret_cast<double2*>(T + r * LF + ch);
                const double2 f = __ldg(reinterpret_cast<const double2*>(w1 + r * gs + ch));
                v.x *= f.x;
                v.y *= f.y;
                *reinterpret_cast<double2*>(T + r * LF + ch) = v;
            }
            __syncthreads();
        }
        if (p.start) {
            warp_axis_mma<MODE, N, ML, false>(T, opc, line0, acc);
            double* x = (c ? p.xout[1] : p.xout[0]) + off;
#pragma unroll
            for (int r = 0; r < G; ++r)
#pragma unroll
                for (int m = 0; m < ML; ++m) {
                    double y0[4], y1[4];
                    pair_results<MODE>(acc[0][r][m][0], acc[1][r][m][0], acc[2][r][m][0], acc[3][r][m][0], y0);
                    pair_results<MODE>(acc[0][r][m][1], acc[1][r][m][1], acc[2][r][m][1], acc[3][r][m][1], y1);
                    const int i = 8 * r + g, col = line0 + 8 * m + 2 * t;
                    const int at[4] = {i, N - 1 - i, HALF - 1 - i, HALF + i};
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        __stcg(reinterpret_cast<double2*>(x + at[k] * gs + col), make_double2(y0[k], y1[k]));
                }
        }
        __syncthreads();  // the columns of T are read: its rows may be fetched again
    }
}

}  // namespace crysscft
