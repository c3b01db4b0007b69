"""The persistent contour kernels, which wait on flags and barriers inside.

Iterations launch one kernel per contour step by default; a poll limit of the caller's own asks for
these instead (scft_diblock_set_wait_limit).  Their results against the numpy oracle, with phi summed
inside and in the separate pass: every block form (dense, even/odd, two-level), the two-phase kernel
of unequal sides, and 3m, whose operators and contour are in position order.  The FP32 kernels against
the step launches, which do the same arithmetic.
"""
import numpy as np
import pytest

from crysscft_sample_b200 import batch, fields, scft, solvers
from oracle import scft_oracle as O

pytestmark = pytest.mark.gpu

LIMIT = 20_000_001  # not the default
CELL, XN, FA, DS = (4.2, 4.2, 4.2), 18.0, 0.3, 0.1


def _fields(kind, N):
    return [fields.to_physical(kind, w) for w in fields.seed_fields(N, CELL[0])]


def _run(kind, N, w, precision="fp64", limit=LIMIT, fused=True, ds=DS):
    G = solvers.make_solver(kind, N)
    G.set_cell_para(CELL)
    run = scft.DiblockSCFT(G, FA, ds, XN, 0.1)
    run.set_precision(precision)
    run.set_wait_limit(limit)
    run.set_phi_form(fused)
    run.set_fields(*w)
    got = run.iterate(2)
    got.update(run.get_fields())
    got["launches"] = run.launches_per_iteration()
    run.close()
    G.close()
    return got


# sides of the alternating kernel: 8, 24, 40, 56 dense, 16, 32, 48, 64 even/odd, 64 two-level (PMMM, 3M)
@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("kind,N", [("P1", (8,) * 3), ("P1", (16,) * 3), ("PMMM", (48,) * 3), ("P1", (32,) * 3),
                                    ("PMMM", (80,) * 3), ("P1", (48,) * 3), ("PMMM", (112,) * 3), ("P1", (64,) * 3),
                                    ("PMMM", (128,) * 3), ("3M", (32,) * 3), ("3M", (48,) * 3), ("3M", (128,) * 3),
                                    ("PMMM", (96, 64, 32)), ("3M", (96, 64, 32)), ("3M", (48, 16, 80))])
def test_fp64_iterations_equal_oracle(gpu, kind, N, fused):
    w = _fields(kind, N)
    want = O.scft_iterations(O.OracleSolver(kind, N), FA, DS, XN, CELL, 0.1, 2, *w)
    got = _run(kind, N, w, fused=fused)
    assert got["launches"] == 5  # prep, contour, Q, phi, energy and mixing
    assert np.abs(got["F"] - want["F"]).max() <= 1e-10 * np.abs(want["F"]).max()
    for k in ("phiA", "phiB"):
        assert np.abs(got[k] - want[k].ravel()).max() <= 1e-12


# the separate pass on both sides: the same bits; the kernel's own sums: another order of FP64 sums of
# the steps' slots (ds = 0.1: 8 of them, even; 0.07: 13, odd)
@pytest.mark.parametrize("ds", [0.1, 0.07])
@pytest.mark.parametrize("kind,N", [("PMMM", (32,) * 3), ("P1", (32,) * 3), ("P1", (48,) * 3), ("PMMM", (128,) * 3),
                                    ("3M", (64,) * 3), ("P1", (64,) * 3)])
def test_fp32_iterations_equal_the_step_launches(gpu, kind, N, ds):
    w = _fields(kind, N)
    step = _run(kind, N, w, "fp32", 20_000_000, False, ds)
    wait = _run(kind, N, w, "fp32", LIMIT, False, ds)
    assert wait["launches"] == 5 < step["launches"]
    for k in ("F", "phiA", "phiB", "wA", "wB"):
        assert np.array_equal(wait[k], step[k])
    for limit in (20_000_000, LIMIT):
        own = _run(kind, N, w, "fp32", limit, True, ds)
        assert np.abs(own["F"] - step["F"]).max() <= 1e-13 * np.abs(step["F"]).max()
        for k in ("phiA", "phiB"):
            assert np.abs(own[k] - step[k]).max() <= 1e-13


# phi summed in the contour's launches: one launch an iteration is the same, the bits of phi are not
# (a grid on which both forms are the separate pass would not show a wrong sum)
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("kind,N", [("PMMM", (32,) * 3), ("P1", (40,) * 3), ("P1", (17, 24, 33)), ("3M", (36, 50, 30))])
def test_step_launches_sum_phi_themselves(gpu, kind, N, precision):
    w = _fields(kind, N) if all(v % 2 == 0 for v in N) else list(np.random.default_rng(5).standard_normal((2,) + N))
    a, b = (_run(kind, N, w, precision, 20_000_000, fused, 0.03) for fused in (True, False))
    assert any(not np.array_equal(a[k], b[k]) for k in ("phiA", "phiB"))
    assert np.abs(a["F"] - b["F"]).max() <= 1e-13 * np.abs(b["F"]).max()
    for k in ("phiA", "phiB"):
        assert np.abs(a[k] - b[k]).max() <= 1e-13


# the buffer of the sums is there before the batch is captured
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("form", [0, 1])
def test_a_batch_with_its_own_limit(gpu, precision, form):
    N = (32, 32, 32)
    w, h = _fields("PMMM", N), []
    for limit in (20_000_000, LIMIT):
        B = batch.BatchSCFT("PMMM", [{"N": N, "L": CELL[0], "fA": FA, "xN": XN}], ds=DS, precision=precision)
        B.configure(1, form)
        B.set_wait_limit(limit)
        B.set_fields(0, *w)
        h.append(B.iterate(2)["F"])
        B.close()
    assert np.abs(h[1] - h[0]).max() <= 1e-12 * np.abs(h[0]).max()
