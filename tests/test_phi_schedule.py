"""Which launch sums which slots of phi (csrc/phi_schedule.h), compiled and run on the CPU.

Every slot is counted once; a launch takes only slots that both chains have stored two launches
earlier or more; the first term of an accumulator replaces what it held; the finishing kernel's
list holds at most eight slots.
"""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "crysscft_sample_b200", "csrc")

PROGRAM = """
#include <cstdio>
#include <cstdlib>
#include "phi_schedule.h"
// arguments: first phase, then pairs U NsA; pointers stand for slots (q: 1000 apart) and accumulators
int main(int argc, char** argv) {
    const long long first = atoll(argv[1]);
    static float q[1], qc[1];
    static double acc[1];
    for (int i = 2; i + 1 < argc; i += 2) {
        const long long U = atoll(argv[i]), NsA = atoll(argv[i + 1]), M = 1000;
        crysscft::PhiSchedule<float> ps(q, qc, acc, U, NsA, M);
        printf("case %lld %lld\\n", U, NsA);
        for (long long k = first; k <= U; ++k) {
            const auto p = ps.of(k);
            for (int c = 0; c < 2; ++c)
                if (p.acc[c])
                    printf("phase %lld %lld %lld %lld %d\\n", k, (long long)(p.q[c] - q) / M, (long long)(p.qc[c] - qc) / M,
                           (long long)(p.acc[c] - acc) / M, p.add[c]);
        }
        ps.finish();
        for (int h = 0; h < 2; ++h)
            for (int b = 0; b < 2; ++b)
                if (ps.sums.acc[h][b]) printf("held %lld\\n", (long long)(ps.sums.acc[h][b] - acc) / M);
        for (int j = 0; j < ps.sums.count; ++j) printf("left %lld\\n", ps.sums.s[j]);
    }
}
"""


@pytest.fixture(scope="module")
def schedules(tmp_path_factory):
    d = tmp_path_factory.mktemp("phi")
    (d / "phi.cpp").write_text(PROGRAM)
    exe = str(d / "phi")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-o", exe, str(d / "phi.cpp")], check=True)

    def run(first, pairs):
        args = [str(v) for p in pairs for v in p]
        out = subprocess.run([exe, str(first)] + args, check=True, capture_output=True, text=True).stdout
        cases = []
        for line in out.splitlines():
            word, *v = line.split()
            v = [int(x) for x in v]
            if word == "case":
                cases.append({"case": tuple(v), "phase": [], "held": [], "left": []})
            else:
                cases[-1][word].append(v)
        return cases

    return run


PAIRS = [(U, NsA) for U in range(2, 25) for NsA in range(1, U)] + \
        [(U, NsA) for U in (97, 100, 199, 200) for NsA in (1, 2, U // 4, U // 2, U // 2 + 1, U - 2, U - 1)]


# first: 0 for one launch a phase, 1 for two launches a step (which ask from the second phase on)
@pytest.mark.parametrize("first", [0, 1])
def test_every_slot_is_summed_once_and_in_time(schedules, first):
    for s in schedules(first, PAIRS):
        U, NsA = s["case"]
        counted = {left[0]: 1 for left in s["left"]}
        assert len(s["left"]) == len(counted) <= 8 and {0, NsA, U} <= set(counted)
        started, by_phase = set(), {}
        for k, slot, slot_c, acc, add in s["phase"]:
            assert slot == slot_c and slot != NsA
            counted[slot] = counted.get(slot, 0) + 1
            # chain 0 stores slot s in phase s, chain 1 in phase U - s
            assert max(slot, U - slot) <= k - 2
            # the accumulator of this parity and block: launches k - 1 and k write different ones
            assert acc == 2 * (k % 2) + (0 if slot < NsA else 1)
            by_phase.setdefault((k, acc), []).append(add)
        for (k, acc), adds in sorted(by_phase.items()):
            assert set(adds) == {1 if acc in started else 0}
            started.add(acc)
        assert {h[0] for h in s["held"]} == started
        assert counted == {slot: 1 for slot in range(U + 1)}
