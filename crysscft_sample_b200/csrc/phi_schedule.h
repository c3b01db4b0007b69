// Which launch of a contour sums which slots for phi (contour_any_kernel, contour_step_kernel_f32,
// contour_simt_kernel_f32).  Host code without CUDA.
#pragma once
#include <cstddef>
#include <vector>

namespace crysscft {

// phi work of one phase: acc += q qc of up to two slots (null pointers: none)
template <typename T>
struct PhiStep {
    const T* q[2];
    const T* qc[2];
    double* acc[2];
    int add[2];  // 0: the first term of this accumulator
};

// What is left for phi_step_finish_kernel: the sums acc[parity][block][point], contour order (null: no
// slot went there), and the slots `s` that the sums leave out.
struct PhiSlots {
    const double* acc[2][2];
    int count;
    long long s[8];
};

// The launch of phase k sums the slots that phase k - 2 finished, if the other chain has them too;
// slot NsA and the ones that no phase takes go to `sums` for the finishing kernel (at most 8: 0, 1,
// U - 1, U, NsA and the middle one or two).
template <typename T>
struct PhiSchedule {
    const T* q;
    const T* qc;
    double* acc;  // 4 fields [parity of k][block]; null: phi is not summed
    long long U, NsA, M;
    PhiSlots sums{};
    std::vector<char> summed;
    PhiSchedule(const T* q_, const T* qc_, double* acc_, long long U_, long long NsA_, long long M_)
        : q(q_), qc(qc_), acc(acc_), U(U_), NsA(NsA_), M(M_), summed((size_t)U_ + 1, 0) {}
    PhiStep<T> of(long long k) {
        PhiStep<T> p{};
        const long long kf = k - 2;
        if (!acc || kf < 1 || 2 * kf - U < 2) return p;
        const int h = (int)(k & 1);
        for (int c = 0; c < 2; ++c) {
            const long long s = c == 0 ? kf : U - kf;
            if (s == NsA) continue;
            p.q[c] = q + s * M;
            p.qc[c] = qc + s * M;
            p.acc[c] = acc + (size_t)(2 * h + (s < NsA ? 0 : 1)) * M;
            p.add[c] = sums.acc[h][s < NsA ? 0 : 1] != nullptr;
            summed[(size_t)s] = 1;
        }
        for (int b = 0; b < 2; ++b)
            for (int c = 0; c < 2; ++c)
                if (p.acc[c] == acc + (size_t)(2 * h + b) * M) sums.acc[h][b] = p.acc[c];
        return p;
    }
    void finish() {
        for (long long s = 0; acc && s <= U; ++s)
            if (!summed[(size_t)s]) sums.s[sums.count++] = s;
    }
};

}  // namespace crysscft
