// Field kernels of one SCFT iteration (FP64 fields; contour slices of type T).
//
//  prep    : calc_ksi (src/crysSCFT_sample.cpp:341-346), array_exp (:315-322) for the
//            two Boltzmann factors, and the initial slices q(0) = 1, q+(end) = 1 (:483)
//  Q       : array_average of q+_A(0) (:324-331, :494)
//  phi     : integrate_phi, trapezoid weights (:348-360), both blocks
//  energy  : the sums of print_energy (:398-424) and the max incompressibility
//  update  : calc_new_fields, simple mixing (:362-371)
//  anderson: Anderson mixing in place of calc_new_fields (no counterpart in the reference)
//
// Reductions are deterministic: a fixed grid writes per-block partials, the last
// block to finish (atomic ticket, no waiting) reduces them in a fixed order.
//
// On small grids these kernels are launch latency and reduction barriers, nothing else, so they are
// launched programmatically (each starts with the wait for the one before it, and the next is
// dispatched meanwhile), several sums share one pair of barriers (block_sums), and the mixing is in
// the energy kernel.  The kernels around the contour of a 32^3 Anderson iteration (10 iterates): 110
// us before, 70 after.  A kernel starts while the one that writes its inputs still runs, so no pointer
// is __restrict__: that would let the compiler load through it ahead of the wait.
#pragma once
#include <cuda_runtime.h>

#include "axis_mma.cuh"
#include "phi_schedule.h"

namespace crysscft {

constexpr int kRedThreads = 256;
constexpr int kRedMaxBlocks = 592;  // 4 x 148 SMs

// Layout of the per-iteration record written by energy_kernel (doubles).
// HIST_RES: rms of the mixing residual r = (xN phiB + ksi - wA, xN phiA + ksi - wB) over both fields
enum { HIST_F = 0, HIST_EH, HIST_E0, HIST_E1, HIST_EK, HIST_MAXINC, HIST_Q, HIST_FLAGS, HIST_RES, HIST_STRIDE };

struct IterState {
    double Q;            // partition function of the current iteration
    unsigned ticket_q;   // last-block tickets
    unsigned ticket_e;
    unsigned iteration;  // iterations completed since the counter was reset
    int error;           // bit 0: Q <= 0 or not finite, bit 1: F not finite
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}
// block-wide sums (maxima where max_mask has the bit) of K values over kRedThreads threads; results
// valid in thread 0.  sh: K x kRedThreads / 32 doubles.
template <int K>
__device__ __forceinline__ void block_sums(double (&v)[K], double* sh, unsigned max_mask = 0) {
    constexpr int W = kRedThreads / 32;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = (max_mask >> k) & 1 ? warp_max(v[k]) : warp_sum(v[k]);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k)
        if (lane == 0) sh[k * W + w] = v[k];
    __syncthreads();
    if (w == 0) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const double r = lane < W ? sh[k * W + lane] : 0.0;
            v[k] = (max_mask >> k) & 1 ? warp_max(r) : warp_sum(r);
        }
    }
}
__device__ __forceinline__ double block_sum(double v, double* sh) {
    double x[1] = {v};
    block_sums(x, sh);
    return x[0];
}

// Point order of the contour (slices and Boltzmann factors).  The fields are always in the
// solver's storage order; the FP64 contour of a 3m solver without translations is kept in the
// order of positions along the half lines, in which its operators are the PMMM ones (on = 1):
// storage index s of an axis of n points is position 2 s, or 2 (n - 1 - s) + 1 beyond the middle.
struct PointOrder {
    int on = 0, nx = 0, ny = 0, nz = 0;
    __device__ __forceinline__ static int position(int s, int n) { return 2 * s < n ? 2 * s : 2 * (n - 1 - s) + 1; }
    __device__ __forceinline__ static int storage(int j, int n) { return (j & 1) ? n - 1 - (j >> 1) : (j >> 1); }
    // contour index of field point i, and the reverse
    __device__ __forceinline__ long long to_contour(long long i) const {
        if (!on) return i;
        const int z = (int)(i % nz), y = (int)((i / nz) % ny), x = (int)(i / ((long long)ny * nz));
        return ((long long)position(x, nx) * ny + position(y, ny)) * nz + position(z, nz);
    }
    __device__ __forceinline__ long long to_field(long long i) const {
        if (!on) return i;
        const int z = (int)(i % nz), y = (int)((i / nz) % ny), x = (int)(i / ((long long)ny * nz));
        return ((long long)storage(x, nx) * ny + storage(y, ny)) * nz + storage(z, nz);
    }
};

template <typename T>
__global__ void prep_kernel(const double* wA, const double* wB,
                            double* ksi, T* wAds, T* wBds,
                            T* q_first, T* qc_last, double xN, double ds,
                            long long M, PointOrder po) {
    pdl_wait();
    pdl_launch_dependents();
    const double index = -ds / 2;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < M;
         i += (long long)gridDim.x * blockDim.x) {
        const double a = wA[i], b = wB[i];
        ksi[i] = 0.5 * (a + b - xN);
        const long long j = po.to_contour(i);
        wAds[j] = (T)(1. * exp(index * a));
        wBds[j] = (T)(1. * exp(index * b));
        q_first[i] = T(1);
        qc_last[i] = T(1);
    }
}

template <typename T>
__global__ void __launch_bounds__(kRedThreads)
q_reduce_kernel(const T* qc0, long long M, double* partials,
                IterState* st) {
    pdl_wait();
    pdl_launch_dependents();
    __shared__ double sh[kRedThreads / 32];
    __shared__ bool last;
    double s = 0.0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < M;
         i += (long long)gridDim.x * blockDim.x)
        s += (double)qc0[i];
    s = block_sum(s, sh);
    if (threadIdx.x == 0) {
        partials[blockIdx.x] = s;
        __threadfence();
        const unsigned t = atomicAdd(&st->ticket_q, 1u);
        last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double r = 0.0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) r += __ldcg(&partials[i]);
    r = block_sum(r, sh);
    if (threadIdx.x == 0) {
        const double Q = r / (double)M;
        st->Q = Q;
        st->ticket_q = 0;
        if (!(Q > 0.0) || !isfinite(Q)) st->error |= 1;
    }
}

// phi_A = sum_{u=0}^{NsA} w_u fA/(NsA Q) q[u] q+[u];  phi_B over u = NsA..NsA+NsB.
// q (forward chain) and qc (backward chain) hold U+1 = NsA+NsB+1 slices of M.  Each thread
// takes two neighbouring points (16-byte loads for FP64) and the slice loop is unrolled so
// several slices' loads are in flight; the sum runs over the slices in order.  The stored
// contour is read once, with streaming loads (it is larger than L2).
template <typename T>
struct Pair;
template <>
struct Pair<double> {
    using type = double2;
};
template <>
struct Pair<float> {
    using type = float2;
};

template <typename T>
__device__ __forceinline__ void phi_point_pair(const T* q, const T* qc, long long M,
                                               long long i, long long s0, long long ns, double c, double& a0,
                                               double& a1) {
    using P = typename Pair<T>::type;
#pragma unroll 4
    for (long long s = 0; s <= ns; ++s) {
        double factor = s == 0 ? 0.5 : (s == ns ? 0.5 : 1);
        factor *= c;
        const long long o = (s0 + s) * M + i;
        const P x = __ldcs(reinterpret_cast<const P*>(q + o));
        const P y = __ldcs(reinterpret_cast<const P*>(qc + o));
        a0 += factor * (double)x.x * (double)y.x;
        a1 += factor * (double)x.y * (double)y.y;
    }
}

template <typename T>
__global__ void phi_kernel(const T* q, const T* qc, double* phiA,
                           double* phiB, const IterState* st, double fA, long long NsA,
                           long long NsB, long long M, PointOrder po) {
    pdl_wait();
    pdl_launch_dependents();
    const double Q = st->Q;
    const double fB = 1 - fA;
    const double cA = fA / (NsA * Q);
    const double cB = fB / (NsB * Q);
    if (M & 1) {  // odd M: pairs would straddle slices unaligned; one point per thread
        for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < M;
             i += (long long)gridDim.x * blockDim.x) {
            double a = 0.0, b = 0.0;
            for (long long s = 0; s <= NsA; ++s) {
                double factor = s == 0 ? 0.5 : (s == NsA ? 0.5 : 1);
                factor *= cA;
                a += factor * (double)q[s * M + i] * (double)qc[s * M + i];
            }
            for (long long s = 0; s <= NsB; ++s) {
                double factor = s == 0 ? 0.5 : (s == NsB ? 0.5 : 1);
                factor *= cB;
                const long long u = NsA + s;
                b += factor * (double)q[u * M + i] * (double)qc[u * M + i];
            }
            const long long f = po.to_field(i);
            phiA[f] = a;
            phiB[f] = b;
        }
        return;
    }
    const long long pairs = M / 2;
    for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < pairs;
         j += (long long)gridDim.x * blockDim.x) {
        const long long i = 2 * j;
        double a0 = 0.0, a1 = 0.0, b0 = 0.0, b1 = 0.0;
        phi_point_pair<T>(q, qc, M, i, 0, NsA, cA, a0, a1);
        phi_point_pair<T>(q, qc, M, i, NsA, NsB, cB, b0, b1);
        if (po.on) {
            const long long f0 = po.to_field(i), f1 = po.to_field(i + 1);
            phiA[f0] = a0;
            phiA[f1] = a1;
            phiB[f0] = b0;
            phiB[f1] = b1;
        } else {
            *reinterpret_cast<double2*>(phiA + i) = make_double2(a0, a1);
            *reinterpret_cast<double2*>(phiB + i) = make_double2(b0, b1);
        }
    }
}

// phi from the alternating contour kernel's fused sums (cubic grid n^3, U = NsA + NsB even).
// acc[c][block][layout][tile][panel element] holds, for chain c, the sum of q(s) q+(s) over
// the slots s of the block that the chain finished in that layout, except slots 0, NsA,
// U/2 and U; those are added here with the trapezoid weights of integrate_phi
// (src/crysSCFT_sample.cpp:348-360: 1/2 at both ends of each block, 1 inside).  The panel
// element of grid point (x, y, z) is (z / 8) * 8n + row * 8 + z % 8, with row y in plane
// tile x and row x in slab tile y.
template <typename T>
__global__ void phi_fused_finish_kernel(const double* acc, const T* q,
                                        const T* qc, double* phiA,
                                        double* phiB, const IterState* st, double fA, long long NsA,
                                        long long NsB, int n, PointOrder po) {
    pdl_wait();
    pdl_launch_dependents();
    const long long n2 = (long long)n * n, M = n2 * n, U = NsA + NsB;
    const double Q = st->Q;
    const double cA = fA / (NsA * Q), cB = (1 - fA) / (NsB * Q);
    long long sp[4] = {0, NsA, U / 2, U};
    int nsp = 4;
    if (U / 2 == NsA) {  // the midpoint is the block boundary
        sp[2] = U;
        nsp = 3;
    }
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < M; i += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(i / n2), y = (int)((i / n) % n), z = (int)(i % n);
        const long long zp = (long long)(z >> 3) * 8 * n + (z & 7);
        const long long ep = x * n2 + zp + y * 8;  // plane tile x, row y
        const long long es = y * n2 + zp + x * 8;  // slab tile y, row x
        double a = 0.0, b = 0.0;
        for (int c = 0; c < 2; ++c) {
            const double* t = acc + (size_t)c * 4 * M;
            a += t[ep] + t[M + es];
            b += t[2 * M + ep] + t[3 * M + es];
        }
        for (int j = 0; j < nsp; ++j) {
            const long long s = sp[j];
            const double w = (double)q[s * M + i] * (double)qc[s * M + i];
            if (s <= NsA) a += (s == 0 || s == NsA ? 0.5 : 1.0) * w;
            if (s >= NsA) b += (s == NsA || s == U ? 0.5 : 1.0) * w;
        }
        const long long f = po.to_field(i);
        phiA[f] = cA * a;
        phiB[f] = cB * b;
    }
}

// phi from the sums of the step launches and the slots that they leave out, with the trapezoid
// weights of integrate_phi.
template <typename T>
__global__ void phi_step_finish_kernel(const T* q, const T* qc,
                                       double* phiA, double* phiB, const IterState* st,
                                       double fA, long long NsA, long long NsB, long long M, PhiSlots sp, PointOrder po) {
    pdl_wait();
    pdl_launch_dependents();
    const long long U = NsA + NsB;
    const double Q = st->Q;
    const double cA = fA / (NsA * Q), cB = (1 - fA) / (NsB * Q);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < M; i += (long long)gridDim.x * blockDim.x) {
        double s[2] = {0.0, 0.0};
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (sp.acc[h][b]) s[b] += sp.acc[h][b][i];
        for (int j = 0; j < sp.count; ++j) {
            const long long u = sp.s[j];
            const double w = (double)q[u * M + i] * (double)qc[u * M + i];
            if (u <= NsA) s[0] += (u == 0 || u == NsA ? 0.5 : 1.0) * w;
            if (u >= NsA) s[1] += (u == NsA || u == U ? 0.5 : 1.0) * w;
        }
        const long long f = po.to_field(i);
        phiA[f] = cA * s[0];
        phiB[f] = cB * s[1];
    }
}

// mix: calc_new_fields with acceptance acc in the same pass (simple mixing); else the fields are left
// to the Anderson kernels, which count the iteration.
__global__ void __launch_bounds__(kRedThreads)
energy_kernel(double* wA, double* wB,
              const double* phiA, const double* phiB,
              const double* ksi, double xN, long long M, double* partials,
              IterState* st, double* hist, unsigned hist_cap, int mix, double acc) {
    __shared__ double sh[5 * (kRedThreads / 32)];
    __shared__ bool last;
    pdl_wait();
    pdl_launch_dependents();
    double s[5] = {0.0, 0.0, 0.0, 0.0, 0.0};  // e1, eh, ek, max incompressibility, |r|^2
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < M;
         i += (long long)gridDim.x * blockDim.x) {
        const double pa = phiA[i], pb = phiB[i];
        const double a = wA[i], b = wB[i], x = ksi[i];
        s[0] += -a * pa - b * pb;
        s[1] += xN * pa * pb;
        const double temp = 1 - pa - pb;
        s[2] += -x * temp;
        s[3] = fmax(s[3], fabs(temp));
        const double ra = xN * pb + x - a, rb = xN * pa + x - b;
        s[4] += ra * ra + rb * rb;
        if (mix) {
            wA[i] = a + acc * ra;
            wB[i] = b + acc * rb;
        }
    }
    block_sums(s, sh, 8u);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < 5; ++k) partials[5 * blockIdx.x + k] = s[k];
        __threadfence();
        const unsigned t = atomicAdd(&st->ticket_e, 1u);
        last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
#pragma unroll
    for (int k = 0; k < 5; ++k) s[k] = 0.0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) {
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            const double v = __ldcg(&partials[5 * i + k]);
            s[k] = k == 3 ? fmax(s[k], v) : s[k] + v;
        }
    }
    block_sums(s, sh, 8u);
    if (threadIdx.x == 0) {
        const double Q = st->Q;
        const double fe_entropic_0 = -log(Q);
        const double fe_entropic_1 = s[0] / (double)M;
        const double fe_enthalpic = s[1] / (double)M;
        const double fe_ksi = s[2] / (double)M;
        const double F = fe_entropic_0 + fe_entropic_1 + fe_enthalpic + fe_ksi;
        if (!isfinite(F)) st->error |= 2;
        double* h = hist + (size_t)(st->iteration % hist_cap) * HIST_STRIDE;
        h[HIST_F] = F;
        h[HIST_EH] = fe_enthalpic;
        h[HIST_E0] = fe_entropic_0;
        h[HIST_E1] = fe_entropic_1;
        h[HIST_EK] = fe_ksi;
        h[HIST_MAXINC] = s[3];
        h[HIST_Q] = Q;
        h[HIST_FLAGS] = (double)st->error;
        h[HIST_RES] = sqrt(s[4] / (2.0 * (double)M));
        st->ticket_e = 0;
        if (mix) st->iteration += 1;
    }
}

// ---------------------------------------------------------------------------
// Anderson mixing (replaces calc_new_fields when enabled; no counterpart in the
// reference).  The iterate w = (wA, wB) and residual r = (xN phiB + ksi - wA,
// xN phiA + ksi - wB) of every iteration go into a ring of history + 1 slots of 2M
// doubles; gram[a][b] = <r_a, r_b> is kept per ring slot.  With D_j = r_0 - r_j
// (0 the current iterate, j the j-th previous) the update solves
// sum_j <D_i, D_j> c_j = <D_i, r_0> and sets
// w <- w_0 + sum_j c_j (w_j - w_0) + beta (r_0 + sum_j c_j (r_j - r_0)).
// ---------------------------------------------------------------------------
constexpr int kAndersonMax = 32;

struct AndersonState {
    int count;    // previous iterates in the ring (<= history)
    int head;     // ring slot of the current iterate
    int k;        // previous iterates this iteration's update uses
    int restart;  // the last solve was singular: history restarted
    int slot[kAndersonMax + 1];  // slot[0] current, slot[j] the j-th previous
    double c[kAndersonMax];
    double gram[(kAndersonMax + 1) * (kAndersonMax + 1)];
    unsigned ticket;
};

// W[head] <- (wA, wB), R[head] <- residual, and
// gram[head][s_j] = gram[s_j][head] = <R[head], R[s_j]>, j = 0..count (deterministic:
// per-block partials, the last block reduces them in block order).  kDots products share a pass
// and its barriers.
constexpr int kDots = 8;

__global__ void __launch_bounds__(kRedThreads)
anderson_record_kernel(const double* wA, const double* wB,
                       const double* phiA, const double* phiB,
                       const double* ksi, double xN, long long M, double* W,
                       double* R, int slots, double* partials, AndersonState* as) {
    __shared__ double sh[kDots * (kRedThreads / 32)];
    __shared__ bool last;
    pdl_wait();
    pdl_launch_dependents();
    const int head = as->head, count = as->count;
    const long long n2 = 2 * M;
    double* r0 = R + (long long)head * n2;
    double* w0 = W + (long long)head * n2;
    for (int j0 = 0; j0 <= count; j0 += kDots) {
        double d[kDots];
#pragma unroll
        for (int k = 0; k < kDots; ++k) d[k] = 0.0;
        for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n2;
             i += (long long)gridDim.x * blockDim.x) {
            double r;
            if (j0 == 0) {
                const bool b = i >= M;
                const long long m = b ? i - M : i;
                const double w = b ? wB[m] : wA[m];
                r = xN * (b ? phiA[m] : phiB[m]) + ksi[m] - w;
                w0[i] = w;
                r0[i] = r;
            } else {
                r = r0[i];
            }
#pragma unroll
            for (int k = 0; k < kDots; ++k)
                if (j0 + k <= count)
                    d[k] += r * (j0 + k == 0 ? r : R[(long long)((head - j0 - k + slots) % slots) * n2 + i]);
        }
        block_sums(d, sh);
        if (threadIdx.x == 0) {
#pragma unroll
            for (int k = 0; k < kDots; ++k)
                if (j0 + k <= count) partials[(size_t)blockIdx.x * (kAndersonMax + 1) + j0 + k] = d[k];
        }
    }
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned t = atomicAdd(&as->ticket, 1u);
        last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int j0 = 0; j0 <= count; j0 += kDots) {
        double d[kDots];
#pragma unroll
        for (int k = 0; k < kDots; ++k) d[k] = 0.0;
        for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) {
#pragma unroll
            for (int k = 0; k < kDots; ++k)
                if (j0 + k <= count) d[k] += __ldcg(&partials[(size_t)b * (kAndersonMax + 1) + j0 + k]);
        }
        block_sums(d, sh);
        if (threadIdx.x == 0) {
#pragma unroll
            for (int k = 0; k < kDots; ++k)
                if (j0 + k <= count) {
                    const int sj = (head - j0 - k + slots) % slots;
                    as->gram[head * (kAndersonMax + 1) + sj] = d[k];
                    as->gram[sj * (kAndersonMax + 1) + head] = d[k];
                }
        }
    }
    if (threadIdx.x == 0) as->ticket = 0;
}

// One block: the k x k normal equations by Gaussian elimination with partial pivoting (the first of
// equal pivots); a pivot below 1e-13 of the largest diagonal entry restarts the history (simple
// step).  Then advances the ring.  A row per thread of the first warp, the columns of a row shared
// by the block's warps: one thread took 18 us for 10 iterates.
__global__ void __launch_bounds__(kRedThreads) anderson_solve_kernel(AndersonState* as, int history) {
    pdl_wait();
    pdl_launch_dependents();
    constexpr int G = kAndersonMax + 1;
    __shared__ double U[kAndersonMax][G];  // odd row stride: lanes of a column on distinct banks
    __shared__ double V[kAndersonMax], f[kAndersonMax], c[kAndersonMax];
    __shared__ int s[G], piv, singular;
    const int slots = history + 1;
    const int n = as->head, k = as->count;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = kRedThreads / 32;
    if (threadIdx.x <= k) s[threadIdx.x] = (n - (int)threadIdx.x + slots) % slots;
    if (threadIdx.x == 0) singular = 0;
    __syncthreads();
    const double* g = as->gram;
    const double g00 = g[n * G + n];
    for (int e = threadIdx.x; e < k * k; e += kRedThreads) {
        const int i = e / k, j = e - i * k;
        U[i][j] = g00 - g[n * G + s[j + 1]] - g[s[i + 1] * G + n] + g[s[i + 1] * G + s[j + 1]];
    }
    if (threadIdx.x < k) V[threadIdx.x] = g00 - g[n * G + s[threadIdx.x + 1]];
    __syncthreads();
    double scale = lane < k ? fabs(U[lane][lane]) : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) scale = fmax(scale, __shfl_xor_sync(0xffffffffu, scale, o));
    for (int col = 0; col < k; ++col) {
        if (warp == 0) {
            // largest |U[r][col]|, r >= col, the first of equals
            double best = lane >= col && lane < k ? fabs(U[lane][col]) : -1.0;
            int at = lane;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const double ob = __shfl_xor_sync(0xffffffffu, best, o);
                const int oa = __shfl_xor_sync(0xffffffffu, at, o);
                if (ob > best || (ob == best && oa < at)) {
                    best = ob;
                    at = oa;
                }
            }
            if (lane == 0) {
                piv = at;
                if (!(best > 1e-13 * scale)) singular = 1;
            }
        }
        __syncthreads();
        if (singular) break;
        if (piv != col) {
            if (threadIdx.x < k) {
                const double x = U[col][threadIdx.x];
                U[col][threadIdx.x] = U[piv][threadIdx.x];
                U[piv][threadIdx.x] = x;
            } else if (threadIdx.x == 32 * (warps - 1)) {
                const double x = V[col];
                V[col] = V[piv];
                V[piv] = x;
            }
            __syncthreads();
        }
        if (warp == 0 && lane > col && lane < k) f[lane] = U[lane][col] / U[col][col];
        __syncthreads();
        for (int r = col + 1 + warp; r < k; r += warps) {
            if (lane >= col && lane < k) U[r][lane] -= f[r] * U[col][lane];
            if (lane == 0) V[r] -= f[r] * V[col];
        }
        __syncthreads();
    }
    if (!singular && warp == 0) {
        double acc = 0.0;  // of row `lane`
        for (int r = k - 1; r >= 0; --r) {
            if (lane == r) c[r] = (V[r] - acc) / U[r][r];
            __syncwarp();
            if (lane < r) acc += U[lane][r] * c[r];
        }
        if (lane < k) as->c[lane] = c[lane];
    }
    if (threadIdx.x <= k) as->slot[threadIdx.x] = s[threadIdx.x];
    if (threadIdx.x == 0) {
        as->k = singular ? 0 : k;
        as->restart = singular;
        const int kept = singular ? 0 : k;
        as->count = kept + 1 < history ? kept + 1 : history;
        as->head = (n + 1) % slots;
    }
}

// (wA, wB) <- w_0 + sum_j c_j (w_j - w_0) + beta (r_0 + sum_j c_j (r_j - r_0))
__global__ void anderson_update_kernel(double* wA, double* wB,
                                       const double* W, const double* R,
                                       long long M, const AndersonState* as, double beta, IterState* st) {
    pdl_wait();
    pdl_launch_dependents();
    const int k = as->k;
    const long long n2 = 2 * M;
    const double* w0 = W + (long long)as->slot[0] * n2;
    const double* r0 = R + (long long)as->slot[0] * n2;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n2;
         i += (long long)gridDim.x * blockDim.x) {
        const double w = w0[i], r = r0[i];
        double dw = 0.0, dr = 0.0;
        for (int j = 1; j <= k; ++j) {
            const long long o = (long long)as->slot[j] * n2 + i;
            const double c = as->c[j - 1];
            dw += c * (W[o] - w);
            dr += c * (R[o] - r);
        }
        const double out = (w + dw) + beta * (r + dr);
        if (i < M) wA[i] = out;
        else wB[i - M] = out;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) st->iteration += 1;
}

}  // namespace crysscft
