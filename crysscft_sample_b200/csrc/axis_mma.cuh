// FP64 axis passes on the tensor cores (DMMA) for axes of up to 128 points: any grid, any
// of the three solvers, one persistent launch per pass (z, y or x) over both contour chains.
//
//   out[line][i] = sum_j A[i][j] in[line][j], lines along z (contiguous), y or x (strided),
// with the Boltzmann factor of the contour step on the z pass's input (pre) and the x pass's
// output (post), and an optional accumulation (multi-term 3m operators).
//
// The axis operator is applied in the block form its symmetry allows (AxisMode), and the sums
// and differences of mirrored points that the blocks act on are formed once, in registers, on
// the way from global to shared memory.  (Forming them from the raw tile inside the MMA loops
// repeats them in every warp that shares the lines: twice the shared-memory reads, which were
// the limit there, and FP64 adds that take the pipe the DMMAs run on.)  The results go from
// the MMA accumulators straight to global memory.
//
//   kFull  A itself                                                      n   multiply-adds a point
//   kEo1   A[n-1-i][n-1-j] = A[i][j] (PMMM, P1, any n):                  n/2
//          u = x_j + x_{n-1-j}, v = x_j - x_{n-1-j}, p = E u, r = O v,
//          y_i = p + r, y_{n-1-i} = p - r
//   kEo2   the even half E splits once more (PMMM, n a multiple of 32):  3n/8
//          [EE u+ | EO u-] and the odd half O dense
//   kCirc4 symmetric circulant (P1, n a multiple of 32): the cyclic shift n/4
//          by n/2 splits A into a circulant and a skew-circulant of n/2
//          points, and both are centrosymmetric: four blocks of n/4
//
// 3m with zero translations stores the even points of a mirror-symmetric line: its operator
// is the PMMM one in another order of the points (position j of the half line is stored at
// j/2 for even j and at n-1-(j-1)/2 for odd j), so `perm` is the only difference.
//
// Two CTAs of 8 warps share an SM (up to 227 KB: operator + one tile each), so one's loads,
// barriers and stores run under the other's MMAs; the next tile is in flight in registers
// during the current one's MMAs.  The passes are launched with programmatic stream
// serialization: the operator of the next pass is copied while this one drains.
#pragma once
#include <cuda_runtime.h>

#include "contour_kernel.cuh"

namespace crysscft {

enum AxisMode { kFull = 0, kEo1 = 1, kEo2 = 2, kCirc4 = 3 };

constexpr int kMmaThreads = 256;
constexpr int kMmaLines = 32;    // lines of a tile
constexpr int kMmaMaxN = 128;

struct AxisMmaPass {
    const double* in[2];
    double* out[2];
    const double* pre[2];    // input *= pre (nullptr: none)
    const double* post[2];   // output *= post (nullptr: none)
    const double* op;        // packed blocks (AxisBlocks)
    int op_count;
    int n;
    int perm;                // 1: 3m order of the points
    int accum;               // 1: add to what out holds (before post)
    int nchain;
    int discard_in;          // 1: the input is dead once read (a triplet intermediate): drop its L2 lines
    long long outer, inner;  // element j of line (o, r) at (o n + j) inner + r; inner 1: contiguous lines
};

// Sizes of the packed operator and of a transformed line.
struct AxisBlocks {
    int h;    // pair indices: n, ceil(n/2), n/4, n/4
    int hp;   // ... padded to the 8 of an MMA tile
    int kt;   // values of a transformed line
    int ld;   // leading dimension of the hp x hp blocks
    int ldo;  // kEo2: leading dimension of O (n/2 x n/2)
    int count;
    __host__ __device__ AxisBlocks(int mode, int n) {
        h = mode == kFull ? n : (mode == kEo1 ? (n + 1) / 2 : n / 4);
        hp = (h + 7) & ~7;
        ld = hp + 4;
        ldo = n / 2 + 4;
        kt = mode == kFull ? hp : (mode == kEo1 ? 2 * hp : n);
        count = mode == kFull ? hp * ld
                              : (mode == kEo1 ? 2 * hp * ld
                                              : (mode == kEo2 ? 2 * hp * ld + (n / 2) * ldo : 4 * hp * ld));
    }
};

// shared memory of a pass: the operator, then the transformed tile (16-byte aligned parts)
__host__ __device__ constexpr int axis_mma_row_ld(int kt) { return (kt % 16 == 0 || kt % 16 == 8) ? kt + 4 : kt + 12; }
inline size_t axis_mma_smem(int mode, int n, bool row) {
    const AxisBlocks b(mode, n);
    const int tile = row ? kMmaLines * axis_mma_row_ld(b.kt) : b.kt * (kMmaLines + 4);
    return (size_t)(((b.count + 1) & ~1) + tile) * sizeof(double);
}

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// storage index of position j
__device__ __forceinline__ int axis_at(int j, int n, int perm) {
    return !perm ? j : ((j & 1) ? n - 1 - (j >> 1) : (j >> 1));
}

// ROW: contiguous lines (tile = 32 rows x line), else strided (tile = line x 32 columns).
// NC: the axis length, or 0 for any length up to NMAX.  ML: 8-line groups per warp tile.
template <int MODE, bool ROW, int NC, int NMAX, int ML>
__global__ void __launch_bounds__(kMmaThreads, 2) axis_mma_kernel(const AxisMmaPass p) {
    constexpr int VPI = MODE == kFull ? 1 : (MODE == kEo1 ? 2 : 4);  // points of one pair index
    constexpr int HMAX = NMAX / VPI;
    constexpr int ITEMS = ROW ? (kMmaLines / 8) * ((HMAX + 31) / 32) : (HMAX + 7) / 8;
    constexpr int NJ = (HMAX + 31) / 32;
    constexpr int ACC = MODE == kFull ? 1 : (MODE == kEo1 ? 2 : 4);
    const int n = NC ? NC : p.n;
    const AxisBlocks b(MODE, n);
    const int h = b.h, hp = b.hp, ld = b.ld, kt = b.kt;
    const int LF = ROW ? axis_mma_row_ld(kt) : kMmaLines + 4;
    const int half = n / 2;
    extern __shared__ __align__(16) double axm[];
    __shared__ long long s_base[2][kMmaLines];  // offset of each line of the tile (-1: none), by tile parity
    double* sop = axm;
    double* F = axm + ((b.count + 1) & ~1);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;

    op_copy_async(sop, p.op, b.count);
    if (h != hp)  // the padding columns stay zero
        for (int e = threadIdx.x; e < (ROW ? kMmaLines : kt) * LF; e += kMmaThreads) F[e] = 0.0;
    cp_async_wait_all();
    pdl_wait();  // everything above reads only the operator
    pdl_launch_dependents();

    const long long inner = ROW ? 1 : p.inner;
    const long long lines = ROW ? p.outer : p.outer * inner;
    const long long tpc = (lines + kMmaLines - 1) / kMmaLines;
    const long long tiles = tpc * p.nchain;
    auto line_base = [&](long long L) -> long long {
        if (L >= lines) return -1;
        if (ROW) return L * n;
        const long long o = L / inner;
        return o * n * inner + (L - o * inner);
    };

    double v[ITEMS * VPI], w[ROW ? ITEMS * VPI : 1];
    // positions of the points of pair index j, in the order the transforms below use
    auto pos = [&](int j, int k) -> int {
        int q;
        if (MODE == kFull) q = j;
        else if (MODE == kEo1) q = k == 0 ? j : n - 1 - j;
        else q = k == 0 ? j : (k == 1 ? n - 1 - j : (k == 2 ? half - 1 - j : half + j));
        return axis_at(q, n, p.perm);
    };
    auto fetch = [&](long long tile, int par) {
        const int c = tile >= tpc ? 1 : 0;
        const long long L0 = (tile - c * tpc) * kMmaLines;
        const double* in = c ? p.in[1] : p.in[0];
        const double* pre = !ROW ? nullptr : (c ? p.pre[1] : p.pre[0]);
        if (warp == 0) s_base[par][lane] = line_base(L0 + lane);
        const long long cb = ROW ? 0 : line_base(L0 + lane);
#pragma unroll
        for (int q = 0; q < ITEMS; ++q) {
            const int l = ROW ? warp + 8 * (q / NJ) : lane;
            const int j = ROW ? lane + 32 * (q % NJ) : warp + 8 * q;
            const long long base = ROW ? line_base(L0 + l) : cb;
            const bool ok = j < h && base >= 0;
#pragma unroll
            for (int k = 0; k < VPI; ++k) {
                const long long a = base + (long long)pos(j, k) * inner;
                v[q * VPI + k] = ok ? __ldcg(in + a) : 0.0;
                if (ROW) w[ROW ? q * VPI + k : 0] = (ok && pre) ? __ldcg(pre + a) : 1.0;
            }
        }
    };
    // transform the fetched points and put them into the tile
    auto put = [&]() {
#pragma unroll
        for (int q = 0; q < ITEMS; ++q) {
            const int l = ROW ? warp + 8 * (q / NJ) : lane;
            const int j = ROW ? lane + 32 * (q % NJ) : warp + 8 * q;
            if (j >= h) continue;
            double x[VPI];
#pragma unroll
            for (int k = 0; k < VPI; ++k) x[k] = ROW ? v[q * VPI + k] * w[ROW ? q * VPI + k : 0] : v[q * VPI + k];
            auto st = [&](int kpos, double val) { F[ROW ? l * LF + kpos : kpos * LF + l] = val; };
            if constexpr (MODE == kFull) {
                st(j, x[0]);
            } else if constexpr (MODE == kEo1) {
                st(j, x[0] + x[1]);
                st(hp + j, x[0] - x[1]);
            } else if constexpr (MODE == kEo2) {
                const double s = x[0] + x[1], d = x[2] + x[3];  // u_j, u_{half-1-j}
                st(j, s + d);
                st(hp + j, s - d);
                st(2 * hp + j, x[0] - x[1]);              // v_j
                st(2 * hp + half - 1 - j, x[2] - x[3]);  // v_{half-1-j}
            } else {
                // shift pairs (j, half + j) and (half-1-j, n-1-j)
                const double u0 = x[0] + x[3], v0 = x[0] - x[3];
                const double u1 = x[2] + x[1], v1 = x[2] - x[1];
                st(j, u0 + u1);
                st(hp + j, u0 - u1);
                st(2 * hp + j, v0 + v1);
                st(3 * hp + j, v0 - v1);
            }
        }
    };

    long long tile = blockIdx.x;
    int par = 0;
    if (tile < tiles) fetch(tile, par);
    for (; tile < tiles; tile += gridDim.x, par ^= 1) {
        const int c = tile >= tpc ? 1 : 0;
        __syncthreads();  // the previous tile's MMAs have read F (first tile: the operator is in)
        put();
        __syncthreads();
        if (!ROW && NC && p.discard_in) {
            // every load of this tile has returned: its 256-byte row pieces are dead
            const long long b0 = s_base[par][0];
            for (int e = threadIdx.x; e < 2 * n; e += kMmaThreads) {
                const double* a = (c ? p.in[1] : p.in[0]) + b0 + (long long)(e >> 1) * inner + (e & 1) * 16;
                asm volatile("discard.global.L2 [%0], 128;" ::"l"(a) : "memory");
            }
        }
        if (tile + gridDim.x < tiles) fetch(tile + gridDim.x, par ^ 1);
        const double* post = c ? p.post[1] : p.post[0];
        double* out = c ? p.out[1] : p.out[0];
        const int groups = hp / 8;
        constexpr int LG = kMmaLines / (8 * ML);
#pragma unroll 1
        for (int unit = warp; unit < LG * groups; unit += kMmaThreads / 32) {
            const int lg = unit % LG, i0 = (unit / LG) * 8;
            double acc[ACC][ML][2];
#pragma unroll
            for (int a = 0; a < ACC; ++a)
#pragma unroll
                for (int m = 0; m < ML; ++m) acc[a][m][0] = acc[a][m][1] = 0.0;
            const double* Fl = ROW ? F + (lg * 8 * ML + g) * LF + t : F + t * LF + lg * 8 * ML + g;
            const int ks = ROW ? 1 : LF, ms = ROW ? 8 * LF : 8;  // strides of k and of an 8-line group
            // one block: acc[a] += rows i0.. of `blk` times the tile's values from kpos on
            auto mma = [&](int a, double o, const double* f) {
#pragma unroll
                for (int m = 0; m < ML; ++m) {
                    const double x = f[m * ms];
                    if (ROW) dmma884(acc[a][m], x, o);
                    else dmma884(acc[a][m], o, x);
                }
            };
            if constexpr (MODE == kEo2) {
                const double* EE = sop + (i0 + g) * ld + t;
                const double* EO = EE + hp * ld;
                const double* OA = sop + 2 * hp * ld + (i0 + g) * b.ldo + t;
                const double* OB = sop + 2 * hp * ld + (half - 1 - i0 - g) * b.ldo + t;
#pragma unroll(NC ? 8 : 2)
                for (int k0 = 0; k0 < hp; k0 += 4) {
                    mma(0, EE[k0], Fl + k0 * ks);
                    mma(1, EO[k0], Fl + (hp + k0) * ks);
                }
#pragma unroll(NC ? 8 : 2)
                for (int k0 = 0; k0 < half; k0 += 4) {
                    const double oa = OA[k0], ob = OB[k0];
                    const double* f = Fl + (2 * hp + k0) * ks;
#pragma unroll
                    for (int m = 0; m < ML; ++m) {
                        const double x = f[m * ms];
                        if (ROW) {
                            dmma884(acc[2][m], x, oa);
                            dmma884(acc[3][m], x, ob);
                        } else {
                            dmma884(acc[2][m], oa, x);
                            dmma884(acc[3][m], ob, x);
                        }
                    }
                }
            } else {
                const double* B = sop + (i0 + g) * ld + t;
#pragma unroll(NC ? 8 : 2)
                for (int k0 = 0; k0 < hp; k0 += 4)
#pragma unroll
                    for (int a = 0; a < ACC; ++a) mma(a, B[a * hp * ld + k0], Fl + (a * hp + k0) * ks);
            }
            // results: (line, pair index) of this lane's two accumulator values e = 0, 1
#pragma unroll
            for (int m = 0; m < ML; ++m)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int l = (lg * ML + m) * 8 + (ROW ? g : 2 * t + e);
                    const int i = i0 + (ROW ? 2 * t + e : g);
                    const long long base = s_base[par][l];
                    if (i >= h || base < 0) continue;
                    double y[VPI];
                    if constexpr (MODE == kFull) {
                        y[0] = acc[0][m][e];
                    } else if constexpr (MODE == kEo1) {
                        y[0] = acc[0][m][e] + acc[1][m][e];
                        y[1] = acc[0][m][e] - acc[1][m][e];
                    } else if constexpr (MODE == kEo2) {
                        const double p1 = acc[0][m][e] + acc[1][m][e], p2 = acc[0][m][e] - acc[1][m][e];
                        y[0] = p1 + acc[2][m][e];
                        y[1] = p1 - acc[2][m][e];
                        y[2] = p2 + acc[3][m][e];
                        y[3] = p2 - acc[3][m][e];
                    } else {
                        const double u0 = acc[0][m][e] + acc[1][m][e], u1 = acc[0][m][e] - acc[1][m][e];
                        const double v0 = acc[2][m][e] + acc[3][m][e], v1 = acc[2][m][e] - acc[3][m][e];
                        y[0] = u0 + v0;
                        y[3] = u0 - v0;
                        y[2] = u1 + v1;
                        y[1] = u1 - v1;
                    }
#pragma unroll
                    for (int k = 0; k < VPI; ++k) {
                        if (MODE == kEo1 && k == 1 && 2 * i == n - 1) continue;  // the middle point
                        const long long a = base + (long long)pos(i, k) * inner;
                        double r = y[k];
                        if (p.accum) r = r + out[a];
                        if (post) r = r * __ldcg(post + a);
                        __stcg(out + a, r);
                    }
                }
        }
    }
}

}  // namespace crysscft
