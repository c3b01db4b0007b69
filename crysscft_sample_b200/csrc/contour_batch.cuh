// Batch contour kernel (FP64): the propagator chains of many SCFT instances in ONE
// persistent cooperative launch.
//
// Each chain (forward q or backward q+ of one instance, src/crysSCFT_sample.cpp:483-491)
// runs on a team of T CTAs with the schedule of contour_any_kernel (contour_step.cuh: plane phase
// [A_z A_y] D store D [A_y], slab phase [A_z A_x] D store D [A_x], one exchange per step through
// the chain's exchange buffers).  Where contour_any_kernel gives every unit (x-plane or y-slab)
// its own CTA, a team CTA owns P = n / T units (rank, rank + T, ...) and runs them one after the
// other in every phase, so a chain occupies T CTAs instead of n and one exchange latency per step
// is shared by P units of work.  Synchronisation is per phase and CTA pair: a CTA waits once per
// phase for one flag of every producer CTA of its team, and releases its own flags once, after
// its last unit.  Every unit is contour_any_kernel's (contour_unit), so the results are
// bit-identical to the per-instance launches.
//
// Two CTAs share an SM.  A unit is a chain of latencies (fetch, a barrier, three short MMA loops,
// stores) and a phase ends in a flag round trip, so a second team fills what the first leaves idle.
// Units of sides below 64 run side by side in a CTA (a warp owns 8 lines, and 8 warps are there).
// ms an iteration of the seeded mixture of 4 / 8 / 12 / 16 / 24 / 32 / 64 instances: 1.38 / 2.34 / 2.52 /
// 2.39 / 5.59 / 9.37 / 13.2, where one CTA an SM fetching W and X panels by TMA, the kernel before, took
// 1.51 / 2.65 / 3.81 / 2.98 / 7.37 / 9.86 / 15.3.  One CTA an SM with the next unit's tile prefetched was
// slower than two (24 instances 6.4 against 6.0, 64 16.2 against 14.3, before contour_unit's last gain).
//
// Scheduling: the host (team_schedule in scft.cu) gives every CTA an ordered task list
// (chain, rank, team size).  CTAs are grouped in columns of one team size; every CTA of a
// column runs the same chains in the same order, so a team never waits for a member busy
// with another task and the launch cannot deadlock.  Every wait is bounded; a CTA that
// gives up sets the batch's abort word, which every other wait polls, and leaves.
#pragma once

#include "contour_step.cuh"

namespace crysscft {

// One chain of one instance as the batch kernel sees it (device memory).
struct TeamChain {
    double* q;                           // contour store (slot0 is the chain's input)
    const double* wds[2];                // Boltzmann factors exp(-w ds/2) of blocks A and B
    double* xbuf;                        // 2 x space_size_phy: plane-phase then slab-phase exchange buffer
    const double* op[3];                 // packed blocks of each axis (equal pointers: one copy)
    unsigned* flags;                     // [layout][consumer CTA][producer CTA], room for 2 n^2; zeroed before the launch
    unsigned* error;                     // the instance's error word (same bits as contour_alt_kernel)
    long long slot0;                     // first input slot
    long long NsA;                       // segments < NsA use block A's factors
    int op_count;                        // doubles of one axis' blocks
    int mode;                            // AxisMode: kEo1, or kEo2 / kCirc4 at n = 64
    int dir;                             // +1 forward, -1 backward
    int U;                               // contour steps
    int n;                               // cubic physical grid side
};

// (chain, rank in team, team size) of one CTA's task
struct TeamTask {
    int chain;
    int rank;
    int size;
    int pad;
};

struct BatchContourArgs {
    const TeamChain* chains;
    const TeamTask* tasks;   // CTA b runs tasks[task_begin[b] .. task_begin[b + 1]) in order
    const int* task_begin;   // gridDim.x + 1 entries
    unsigned* abort;         // nonzero once any CTA gave up (zeroed before the launch)
    long long spin_limit;
};

__device__ __forceinline__ unsigned ld_relaxed_u32(const unsigned* p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_relaxed_u32(unsigned* p, unsigned v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Units a CTA of the batch kernel runs at a time on a grid of side n.
__host__ __device__ inline int team_side_by_side(int n) { return n >= 64 ? 1 : (kStepThreads / 32) / (n / 8); }

// Run one task: this CTA's units of chain ch, as rank `rank` of a team of T CTAs.
// Returns false after an error (the CTA then stops taking tasks).
template <int MODE, int NC>
__device__ bool team_chain(const BatchContourArgs& a, const TeamChain* ch, int rank, int T, double* smem, int* s_fail) {
    const int n = NC ? NC : ch->n, U = ch->U, dir = ch->dir;
    const long long PLANE = (long long)n * n, M = PLANE * n, slot0 = ch->slot0, NsA = ch->NsA;
    // units side by side in the CTA, n / 8 warps and a tile each
    const int side = team_side_by_side(n);
    const int warp = (int)threadIdx.x >> 5, group = warp / (n / 8), lw = warp - group * (n / 8);
    // this group's tiles: rows and factors
    const int words = n * step_ld(NC);
    double* tile = smem + min(group, side - 1) * 2 * words;
    double* op[3];
    __syncthreads();  // every thread is done with the previous task's operators
    {
        double* o = smem + 2 * side * words;
        const int cnt = ch->op_count;
        for (int ax = 2; ax >= 0; --ax) {
            int like = -1;
            for (int b = 2; b > ax; --b)
                if (ch->op[b] == ch->op[ax]) like = b;
            if (like >= 0) {
                op[ax] = like == 2 ? op[2] : op[1];
                continue;
            }
            op[ax] = o;
            for (int i = threadIdx.x; i < cnt / 2; i += kStepThreads) cp_async16(o + 2 * i, ch->op[ax] + 2 * i);
            o += cnt;
        }
        cp_async_commit();
        cp_async_wait_all();
    }
    __syncthreads();
    double* XP = ch->xbuf;  // written by plane phases
    double* XS = XP + M;    // written by slab phases
    // flags[layout][consumer CTA][producer CTA] (T x T each): phase + 1 once the producer's
    // units of that phase are in the exchange buffer
    unsigned* fl_plane = ch->flags;        // written after plane phases
    unsigned* fl_slab = fl_plane + T * T;  // written after slab phases
    auto factor = [&](int s) -> const double* {
        const long long in_slot = slot0 + (long long)dir * s;
        return ch->wds[(dir > 0 ? in_slot : in_slot - 1) < NsA ? 0 : 1];
    };
    for (int k = 0; k <= U; ++k) {
        const bool plane = (k & 1) == 0;
        if (k >= 1) {
            // every CTA of the team has finished phase k-1 (all its units written to the
            // exchange buffer): one flag per producer CTA, polled by thread t
            if ((int)threadIdx.x < T) {
                const unsigned* f = (plane ? fl_slab : fl_plane) + (size_t)rank * T + threadIdx.x;
                long long spins = 0;
                while (ld_acquire_u32(f) < (unsigned)k) {
                    if (++spins > a.spin_limit) {
                        *s_fail = 1;
                        break;
                    }
                    if (spins > 64) {
                        if ((spins & 255) == 0 && ld_relaxed_u32(a.abort)) {
                            *s_fail = 1;
                            break;
                        }
                        __nanosleep(20);
                    }
                }
            }
            __syncthreads();
            if (*s_fail) {
                if (threadIdx.x == 0) {
                    atomicOr(ch->error, 1u);
                    atomicOr(a.abort, 1u);
                }
                return false;
            }
        }
        const double* w0 = k >= 1 ? factor(k - 1) : nullptr;
        const double* w1 = k < U ? factor(k) : w0;
        double* slice = ch->q + (slot0 + (long long)dir * k) * M;
        const long long gs = plane ? n : PLANE;
        for (int p0 = rank; p0 < n; p0 += T * side) {
            const int p = p0 + group * T;
            const long long off = plane ? (long long)p * PLANE : (long long)p * n;
            UnitIO u;
            u.gs = u.xgs = gs;
            u.in = (k == 0 ? slice : (plane ? XS : XP)) + off;
            u.q = slice + off;
            u.x = (plane ? XP : XS) + off;
            u.w0 = w0 + off;
            u.w1 = w1 + off;
            u.R = u.nz = n;
            u.active = group < side && p < n;
            u.finish = k >= 1;
            u.start = k < U;
            u.vec = true;  // n is even, the buffers are the library's
            if (u.finish && u.active) stage_factors<NC>(tile + words, u.w0, gs, n, n, true, lw);
            contour_unit<MODE, NC>(tile, tile + words, op[2], plane ? op[1] : op[0], u, lw);
            __syncthreads();
        }
        if (k < U && (int)threadIdx.x < T) {  // tell CTA threadIdx.x that this CTA's units of phase k are out
            // one fence (the barrier above put the block's stores before it), then the flag
            asm volatile("fence.acq_rel.gpu;" ::: "memory");
            st_relaxed_u32((plane ? fl_plane : fl_slab) + (size_t)threadIdx.x * T + rank, (unsigned)(k + 1));
        }
    }
    return true;
}

__global__ void __launch_bounds__(kStepThreads, 2) batch_contour_kernel(const BatchContourArgs a) {
    extern __shared__ __align__(16) double team_smem[];
    __shared__ int s_fail;
    if (threadIdx.x == 0) s_fail = 0;
    const int t0 = a.task_begin[blockIdx.x], t1 = a.task_begin[blockIdx.x + 1];
    for (int t = t0; t < t1; ++t) {
        const TeamTask task = a.tasks[t];
        const TeamChain* ch = a.chains + task.chain;
        bool ok = false;
        switch (ch->mode) {
            case kEo2: ok = team_chain<kEo2, 64>(a, ch, task.rank, task.size, team_smem, &s_fail); break;
            case kCirc4: ok = team_chain<kCirc4, 64>(a, ch, task.rank, task.size, team_smem, &s_fail); break;
            default:
                ok = ch->n == 16   ? team_chain<kEo1, 16>(a, ch, task.rank, task.size, team_smem, &s_fail)
                     : ch->n == 32 ? team_chain<kEo1, 32>(a, ch, task.rank, task.size, team_smem, &s_fail)
                     : ch->n == 48 ? team_chain<kEo1, 48>(a, ch, task.rank, task.size, team_smem, &s_fail)
                                   : team_chain<kEo1, 0>(a, ch, task.rank, task.size, team_smem, &s_fail);
                break;
        }
        if (!ok) break;
    }
}

// Whether the batch kernel takes a cubic grid of side n; dynamic shared memory it needs for
// `ops` distinct operators of `count` doubles.
inline bool team_side(int n) { return n >= 8 && n <= kStepMaxN && n % 8 == 0; }
inline size_t team_smem_bytes(int n, int ops, int count) {
    return ((size_t)2 * team_side_by_side(n) * n * step_ld(0) + (size_t)ops * count) * sizeof(double);
}

}  // namespace crysscft
