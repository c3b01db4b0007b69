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
//
// 128^3 PMMM, both chains: 53 us a step against 87 us in three passes (256^3 iteration 17.9 -> 11.5
// ms), P1 43 against 93 us.  DMMA floor 33 us (P1 22); the rest is the 131 KB that a tile moves in
// and out four times while its SM computes nothing.  16 warps of 8 lines instead of 8 of 16 at 128
// points: the same time; at 96 points 12 warps.  Turns on the tensor pipe (the two warps of a
// scheduler one after the other, so that one stores while the other multiplies) gave P1 1.3 % and
// took 1.8 % from PMMM.  The rows are on their way before the operators have landed: the CTAs of
// the second wave find no launch to wait for, and had one latency after the other (0.3 to 0.5 %).
#pragma once
#include <cuda_runtime.h>

#include "axis_mma.cuh"
#include "phi_schedule.h"

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
    pdl_wait();  // everything above reads only the operators
    pdl_launch_dependents();

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
        if (u == blockIdx.x) {
            cp_async_wait_but_newest();
            __syncthreads();  // the operators
        }
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
                f[k] = __ldcg(reinterpret_cast<const double2*>(w + at * gs + col));
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
                    if (other_w) f1 = __ldcg(reinterpret_cast<const double2*>(w1 + at * gs + col));
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
                const double2 f = __ldcg(reinterpret_cast<const double2*>(w1 + r * gs + ch));
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

// ---------------------------------------------------------------------------
// The same phase for grids whose axes all have at most 64 points: any sizes, odd and unequal ones
// among them, one CTA a unit of each chain.
//
// Waiting for the previous launch costs these grids as much as their work, so
//   - two CTAs fit an SM (128 registers): those of phase k copy the operators and wait beside
//     those of phase k - 1;
//   - phi is summed in that time.  Phase k - 2 has completed when phase k starts to run (phase
//     k - 1 lets it start only after its own wait), so the slots that phase finished are multiplied
//     with the other chain's, stored long ago (second half of the contour).  The sums alternate
//     between two accumulators with the parity of k, because those of phase k - 1 may still be on
//     their way.
// The first launch of a contour is not dispatched early: the CTAs of a phase take the SMs that those
// of the phase before leave least occupied, so a first phase that is spread one CTA an SM stays so,
// while one that was fitted in beside the tail of another kernel puts two of its CTAs on some SMs,
// and every phase after it does the same (64^3: 5.9 against 10 us a phase).
// Per iteration on one B200 against what ran these grids before: 16^3 0.173 ms (persistent kernel
// 0.331), 24^3 0.31, 32^3 0.25 (0.46), 64^3 1.30 (1.46; P1 1.18 against 1.66), 200 steps of 45^3 P1
// 1.16 (three passes a step 2.13; 1.40 with run-time trip counts in the K loops).  A 64^3 phase takes
// 5.7 us, 0.55 of it from a launch's last store to the next one's first load.  Of the 9.4 thousand
// cycles in the CTA 4.6 are DMMA at the peak rate, 1.2 the rows' fetch, 1.3 the epilogue of the
// finishing operation, the rest latencies and sums around the MMAs.  The same phases as one
// persistent launch with a release flag per unit pair took 9.1 us (4.5 of them until the last of a
// CTA's 64 flags was seen), and so did holding back the q stores behind the release.
// ---------------------------------------------------------------------------
constexpr int kStepMaxN = 64;
constexpr int kStepThreads = 256;
constexpr int kStepResults = 16;  // results of a lane in one operation

struct ContourAnyArgs {
    const double* in[2];   // k = 0: the initial slice; else the exchange buffer of the other layout
    double* q[2];          // k >= 1: the finished slice
    double* xout[2];       // k < U: this layout's exchange buffer, [x][y][zpad]
    const double* w0[2];   // k >= 1: Boltzmann factor of the finished step
    const double* w1[2];   // k < U: of the started step
    const double* opz;     // packed blocks of A_z and of the layout's column axis
    const double* opc;
    int opz_count, opc_count;
    int n[3];
    int nchain, plane, finish, start;
    int vec;               // 1: nz even and every array 16-byte aligned
    PhiStep<double> phi;
};

__host__ __device__ inline int step_zpad(int nz) { return (nz + 1) & ~1; }
// leading dimension of a tile: of the fixed cubic sides their own, else that of the largest
__host__ __device__ constexpr int step_ld(int side) { return (side ? side : kStepMaxN) + 4; }

// Axis operations of a unit in block form MODE: kEo1 with run-time lengths (NC = 0) or on a cubic
// grid of side NC; kEo2 / kCirc4 with NC = 64.
template <int MODE, int NC>
struct StepOp {
    static constexpr int VPI = MODE == kEo1 ? 2 : 4;
    static constexpr int NMAX = NC ? NC : kStepMaxN;
    static constexpr int G = (NMAX + 8 * VPI - 1) / (8 * VPI);
    static constexpr int ACC = MODE == kEo1 ? 2 : 4;
    static_assert(G * 2 * VPI <= kStepResults, "results of a lane");
    using Acc = double[ACC][G][1][2];

    // kEo1 with GR groups of 8 pair indices: every trip count known
    template <bool ROW, int GR>
    __device__ __forceinline__ static void run_eo1(const double* T, const double* op, int n, int line0, Acc& acc) {
        constexpr int HP = 8 * GR, LD = HP + 4, LF = step_ld(NC);
        const int nn = NC ? NC : n, h = (nn + 1) / 2;
        const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
        for (int r = 0; r < GR; ++r)
            acc[0][r][0][0] = acc[0][r][0][1] = acc[1][r][0][0] = acc[1][r][0][1] = 0.0;
        const double* f = ROW ? T + (line0 + g) * LF : T + line0 + g;
        constexpr int KS = ROW ? 1 : LF;
        const double* B = op + g * LD + t;
#pragma unroll
        for (int k0 = 0; k0 < HP; k0 += 4) {
            const int j = k0 + t, jc = NC || j < h ? j : h - 1;  // padding columns of the operator are 0
            const double x0 = f[jc * KS], x1 = f[(nn - 1 - jc) * KS];
            const double u = x0 + x1, v = x0 - x1;
#pragma unroll
            for (int r = 0; r < GR; ++r) {
                const double e = B[8 * r * LD + k0], o = B[HP * LD + 8 * r * LD + k0];
                if (ROW) {
                    dmma884(acc[0][r][0], u, e);
                    dmma884(acc[1][r][0], v, o);
                } else {
                    dmma884(acc[0][r][0], e, u);
                    dmma884(acc[1][r][0], o, v);
                }
            }
        }
    }
    template <bool ROW>
    __device__ __forceinline__ static void run(const double* T, const double* op, int n, int line0, Acc& acc) {
        if constexpr (MODE != kEo1) {
            warp_axis_mma<MODE, NC, 1, ROW>(T, op, line0, acc);
        } else if constexpr (NC != 0) {
            run_eo1<ROW, G>(T, op, n, line0, acc);
        } else {
            switch ((n + 15) / 16) {
                case 1: run_eo1<ROW, 1>(T, op, n, line0, acc); break;
                case 2: run_eo1<ROW, 2>(T, op, n, line0, acc); break;
                case 3: run_eo1<ROW, 3>(T, op, n, line0, acc); break;
                default: run_eo1<ROW, 4>(T, op, n, line0, acc); break;
            }
        }
    }
    // groups of an axis of n points (kEo1), a bound on those with results
    __device__ __forceinline__ static bool has_group(int r, int n) { return NC || r < (n + 15) / 16; }
    // results of group r, accumulator element e
    __device__ __forceinline__ static void results(const Acc& acc, int r, int e, double (&y)[VPI]) {
        if constexpr (MODE == kEo1) {
            y[0] = acc[0][r][0][e] + acc[1][r][0][e];
            y[1] = acc[0][r][0][e] - acc[1][r][0][e];
        } else {
            pair_results<MODE>(acc[0][r][0][e], acc[1][r][0][e], acc[2][r][0][e], acc[3][r][0][e], y);
        }
    }
    // position k of pair index i; -1: none (padding, or the middle point a second time)
    __device__ __forceinline__ static int position(int i, int k, int n) {
        const int nn = NC ? NC : n;
        if constexpr (MODE == kEo1) {
            if (!NC && (2 * i > nn - 1 || (k == 1 && 2 * i == nn - 1))) return -1;
            return k == 0 ? i : nn - 1 - i;
        } else {
            return k == 0 ? i : (k == 1 ? nn - 1 - i : (k == 2 ? nn / 2 - 1 - i : nn / 2 + i));
        }
    }
};

// acc += q qc over all points, by the whole grid
template <typename T>
__device__ __forceinline__ void phi_step(const PhiStep<T>& p, long long M) {
    if (!p.acc[0] && !p.acc[1]) return;
    const bool one = p.acc[0] == p.acc[1];  // both slots in one block of the copolymer
    const long long stride = (long long)gridDim.x * blockDim.x;
#pragma unroll 4
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < M; i += stride) {
        const double a = p.acc[0] ? (double)__ldcg(p.q[0] + i) * (double)__ldcg(p.qc[0] + i) : 0.0;
        const double b = p.acc[1] ? (double)__ldcg(p.q[1] + i) * (double)__ldcg(p.qc[1] + i) : 0.0;
        if (one) {
            __stcg(p.acc[0] + i, (p.add[0] ? __ldcg(p.acc[0] + i) : 0.0) + a + b);
        } else {
            if (p.acc[0]) __stcg(p.acc[0] + i, (p.add[0] ? __ldcg(p.acc[0] + i) : 0.0) + a);
            if (p.acc[1]) __stcg(p.acc[1] + i, (p.add[1] ? __ldcg(p.acc[1] + i) : 0.0) + b);
        }
    }
}

// One unit of one phase: an x-plane or y-slab tile of R rows and nz columns (z) in T.  All pointers
// are at the unit's first element.
struct UnitIO {
    const double* in;   // finish: the exchange buffer of the other layout (row stride xgs); else the initial slice (gs)
    double* q;          // finish: the finished slice
    double* x;          // start: this layout's exchange buffer
    const double* w0;   // finish: Boltzmann factor of the finished step (also in the tile W, see stage_factors)
    const double* w1;   // start: of the started step (the same pointer within a block)
    long long gs, xgs;  // row strides of a field and of an exchange buffer
    int R, nz;
    bool finish, start, vec;
    bool active;        // false: this warp has no unit
};

// Copies the 8 rows of warp lw (NC values each, row stride gs) into a tile, asynchronously: 8 lanes
// on 128 bytes of a row, which fill whole lines and all banks.  (4 lanes a row, as where rows may
// be short and odd, are two lanes a bank.)
template <int NC>
__device__ __forceinline__ void copy_rows(double* tile, const double* x, long long gs, int lw) {
    const int lane = threadIdx.x & 31, ch = 2 * (lane & 7);
    if (lw * 8 >= NC) return;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int r = lw * 8 + 4 * h + (lane >> 3);
#pragma unroll
        for (int e = 0; e < NC; e += 16) cp_async16(tile + r * step_ld(NC) + e + ch, x + r * gs + e + ch);
    }
}

// Copies the factors w (row stride gs) of this warp's rows into the tile W, asynchronously: the
// caller commits, and contour_unit waits for it with its rows.  The factors are older than the
// exchange, so their latency passes while a phase waits for its rows; loaded into registers in
// front of the column operation they held it up (64^3: 2.4 against 1.8 thousand cycles, 16^3 0.7
// against 0.2).
template <int NC>
__device__ __forceinline__ void stage_factors(double* W, const double* w, long long gs, int R_, int nz_, bool vec, int lw) {
    constexpr int LF = step_ld(NC);
    const int R = NC ? NC : R_, nz = NC ? NC : nz_;
    if (NC) {
        copy_rows<NC>(W, w, gs, lw);
        return;
    }
    const int lane = threadIdx.x & 31, r = lw * 8 + (lane >> 2), t = lane & 3;
    if (r >= R) return;
    if (vec) {
#pragma unroll 4
        for (int ch = t; ch < nz / 2; ch += 4) cp_async16(W + r * LF + 2 * ch, w + r * gs + 2 * ch);
    } else {
        for (int z = t; z < nz; z += 4) cp_async8(W + r * LF + z, w + r * gs + z);
    }
}

// Copies this warp's rows of the exchange buffer (row stride xgs) into the tile T, asynchronously.
template <int NC>
__device__ __forceinline__ void stage_rows(double* T, const double* x, long long xgs, int R_, int nz_, int lw) {
    constexpr int LF = step_ld(NC);
    if (NC) {
        copy_rows<NC>(T, x, xgs, lw);
        return;
    }
    const int R = R_, zpad = step_zpad(nz_);
    const int lane = threadIdx.x & 31, r = lw * 8 + (lane >> 2), t = lane & 3;
    if (r >= R) return;
#pragma unroll 4
    for (int ch = t; ch < zpad / 2; ch += 4) cp_async16(T + r * LF + 2 * ch, x + r * xgs + 2 * ch);
}

// Called by all threads of the block, warp lw of those that share the unit taking lines 8 lw.. of T.
// The results are complete, and T free, after a block barrier.
template <int MODE, int NC>
__device__ __forceinline__ void contour_unit(double* T, const double* W, const double* opz, const double* opc,
                                             const UnitIO& u, int lw) {
    using Op = StepOp<MODE, NC>;
    constexpr int VPI = Op::VPI, G = Op::G, LF = step_ld(NC);
    const int R = NC ? NC : u.R, nz = NC ? NC : u.nz, zpad = step_zpad(nz);
    const long long gs = u.gs, xgs = u.xgs;
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3, line0 = lw * 8;
    const bool warp_rows = u.active && line0 < R, warp_cols = u.active && line0 < nz;
    const int col = line0 + 2 * t;  // this lane's columns: col, col + 1
    const bool vec = NC || u.vec;
    // The row of this lane's result (r, k) of a column operation.  Rows are 32 bytes past a multiple
    // of 128, which the operand loads need, so the 16-byte accesses of two neighbouring rows share
    // banks; lanes of odd g take the mirrored results of a pair in the other order, whose rows lie
    // 64 bytes apart (NC a multiple of 16).  Shared memory bounds the epilogue: with this and whole
    // rows in copy_rows a 64^3 PMMM iteration takes 1.302 instead of 1.349 ms, 32^3 0.2535 / 0.2563, 16^3
    // 0.1733 / 0.1755, a batch of 24 instances 5.6 / 6.0.  (The same exchange in contour_step_kernel:
    // 256^3 PMMM 11.63 against 11.49 ms.)
    const bool swap = NC && (g & 1);
    auto row_of = [&](int r, int k) { return Op::position(8 * r + g, swap ? k ^ 1 : k, R); };
    auto ld2 = [&](const double* s) {
        if (vec) return __ldcg(reinterpret_cast<const double2*>(s));
        return make_double2(__ldcg(s), col + 1 < nz ? __ldcg(s + 1) : 0.0);
    };
    // factors at this lane's column results, (group, point) order
    double2 f[G * VPI];
    auto factors = [&](const double* w) {
#pragma unroll
        for (int r = 0; r < G; ++r)
#pragma unroll
            for (int k = 0; k < VPI; ++k) {
                const int row = row_of(r, k);
                f[r * VPI + k] = row >= 0 && col < nz ? ld2(w + row * gs + col) : make_double2(0.0, 0.0);
            }
    };
    typename Op::Acc acc;
    if (u.finish) {
        // this warp's rows, A_z on them
        if (warp_rows) {
            stage_rows<NC>(T, u.in, xgs, R, nz, lw);
            cp_async_commit();
            cp_async_wait_all();
            __syncwarp();
            Op::template run<true>(T, opz, nz, line0, acc);
            __syncwarp();
#pragma unroll
            for (int r4 = 0; r4 < G; ++r4) {
                if (!Op::has_group(r4, nz)) break;
                double y0[VPI], y1[VPI];
                Op::results(acc, r4, 0, y0);
                Op::results(acc, r4, 1, y1);
                double* row = T + (line0 + g) * LF;
                const int i = 8 * r4 + 2 * t;
#pragma unroll
                for (int k = 0; k < VPI; ++k) {
                    const int p0 = Op::position(i, k, nz), p1 = Op::position(i + 1, k, nz);
                    if (NC) {
                        *reinterpret_cast<double2*>(row + (p0 < p1 ? p0 : p1)) =
                            p0 < p1 ? make_double2(y0[k], y1[k]) : make_double2(y1[k], y0[k]);
                    } else {
                        if (p0 >= 0) row[p0] = y0[k];
                        if (p1 >= 0) row[p1] = y1[k];
                    }
                }
            }
        }
        __syncthreads();  // every row is through A_z, the factors are in
        if (!warp_cols) return;
        Op::template run<false>(T, opc, R, line0, acc);
        __syncwarp();
        const bool same_w = u.w1 == u.w0;
        double v[G * VPI][2];
#pragma unroll
        for (int r = 0; r < G; ++r) {
            if (!Op::has_group(r, R)) break;
            double y0[VPI], y1[VPI];
            Op::results(acc, r, 0, y0);
            Op::results(acc, r, 1, y1);
#pragma unroll
            for (int k = 0; k < VPI; ++k) {
                const int id = r * VPI + k, row = row_of(r, k);
                if (row < 0) continue;
                const double2 w = *reinterpret_cast<const double2*>(W + row * LF + col);
                v[id][0] = (swap ? y0[k ^ 1] : y0[k]) * w.x;
                v[id][1] = (swap ? y1[k ^ 1] : y1[k]) * w.y;
                if (u.start && same_w)
                    *reinterpret_cast<double2*>(T + row * LF + col) = make_double2(v[id][0] * w.x, v[id][1] * w.y);
                if (col >= nz) continue;
                if (vec) {
                    __stcg(reinterpret_cast<double2*>(u.q + row * gs + col), make_double2(v[id][0], v[id][1]));
                } else {
                    __stcg(u.q + row * gs + col, v[id][0]);
                    if (col + 1 < nz) __stcg(u.q + row * gs + col + 1, v[id][1]);
                }
            }
        }
        if (!u.start) return;
        if (!same_w) {  // the step that starts is the first of the other block
            factors(u.w1);
#pragma unroll
            for (int r = 0; r < G; ++r) {
                if (!Op::has_group(r, R)) break;
#pragma unroll
                for (int k = 0; k < VPI; ++k) {
                    const int id = r * VPI + k, row = row_of(r, k);
                    if (row >= 0)
                        *reinterpret_cast<double2*>(T + row * LF + col) =
                            make_double2(v[id][0] * f[id].x, v[id][1] * f[id].y);
                }
            }
        }
        __syncwarp();
    } else {
        // the first phase: D q(0), each warp its columns
        if (!warp_cols) return;
        factors(u.w1);
#pragma unroll
        for (int r = 0; r < G; ++r)
#pragma unroll
            for (int k = 0; k < VPI; ++k) {
                const int id = r * VPI + k, row = row_of(r, k);
                if (row < 0) continue;
                const double2 x = col < nz ? ld2(u.in + row * gs + col) : make_double2(0.0, 0.0);
                *reinterpret_cast<double2*>(T + row * LF + col) = make_double2(x.x * f[id].x, x.y * f[id].y);
            }
        __syncwarp();
    }
    Op::template run<false>(T, opc, R, line0, acc);
#pragma unroll
    for (int r = 0; r < G; ++r) {
        if (!Op::has_group(r, R)) break;
        double y0[VPI], y1[VPI];
        Op::results(acc, r, 0, y0);
        Op::results(acc, r, 1, y1);
#pragma unroll
        for (int k = 0; k < VPI; ++k) {
            const int row = Op::position(8 * r + g, k, R);
            if (row >= 0 && col < zpad)  // the padding column takes a dead value
                __stcg(reinterpret_cast<double2*>(u.x + row * xgs + col), make_double2(y0[k], y1[k]));
        }
    }
}

template <int MODE, int NC>
__global__ void __launch_bounds__(kStepThreads, 2) contour_any_kernel(const ContourAnyArgs a) {
    const int nx = NC ? NC : a.n[0], ny = NC ? NC : a.n[1], nz = NC ? NC : a.n[2];
    constexpr int LF = step_ld(NC);
    const int zpad = step_zpad(nz);
    const bool plane = a.plane != 0;
    const int R = plane ? ny : nx;  // rows of the tile; its columns are z
    extern __shared__ __align__(16) double any[];
    double* T = any;
    double* W = T + ((R + 7) & ~7) * LF;
    double* opz = W + ((R + 7) & ~7) * LF;
    double* opc = a.opc == a.opz ? opz : opz + a.opz_count;
    const int units = nx > ny ? nx : ny;
    const int c = (int)blockIdx.x >= units ? 1 : 0, p = (int)blockIdx.x - c * units;
    const bool has_unit = NC || p < (plane ? nx : ny);  // in this layout
    const long long psz = (long long)ny * nz, xpsz = (long long)ny * zpad;
    const long long off = plane ? p * psz : (long long)p * nz, xoff = plane ? p * xpsz : (long long)p * zpad;
    UnitIO u;
    u.gs = plane ? nz : psz;
    u.xgs = plane ? zpad : xpsz;
    u.in = (c ? a.in[1] : a.in[0]) + (a.finish ? xoff : off);
    u.q = (c ? a.q[1] : a.q[0]) + off;
    u.x = (c ? a.xout[1] : a.xout[0]) + xoff;
    u.w0 = (c ? a.w0[1] : a.w0[0]) + off;
    u.w1 = (c ? a.w1[1] : a.w1[0]) + off;
    u.R = R;
    u.nz = nz;
    u.finish = a.finish != 0;
    u.start = a.start != 0;
    u.vec = a.vec != 0;
    u.active = true;
    for (int i = threadIdx.x; i < a.opz_count / 2; i += kStepThreads) cp_async16(opz + 2 * i, a.opz + 2 * i);
    if (opc != opz)
        for (int i = threadIdx.x; i < a.opc_count / 2; i += kStepThreads) cp_async16(opc + 2 * i, a.opc + 2 * i);
    // phase 0 waits for the kernel that writes the factors; they are older than any other launch
    if (a.finish && has_unit) stage_factors<NC>(W, u.w0, u.gs, R, nz, u.vec, (int)threadIdx.x >> 5);
    cp_async_commit();
    phi_step(a.phi, (long long)nx * psz);
    cp_async_wait_all();
    pdl_wait();
    pdl_launch_dependents();
    __syncthreads();  // the operators
    if (!has_unit) return;
    contour_unit<MODE, NC>(T, W, opz, opc, u, (int)threadIdx.x >> 5);
}

}  // namespace crysscft
