"""What a launch plan must not outlive: the point order of a stored contour."""
import numpy as np
import pytest

from crysscft_sample_b200 import scft, solvers

pytestmark = pytest.mark.gpu

CELL = (4.2, 4.0, 5.1)


# 3m without translations keeps its FP64 contour in another point order than the fields; the slice a
# caller gets is in storage order whatever has happened to the cell since
@pytest.mark.parametrize("kind,N", [("3M", (36, 50, 30)), ("3M", (128, 128, 128)), ("3M", (300, 16, 8)),
                                    ("PMMM", (32, 32, 32)), ("P1", (13, 22, 9))])
def test_a_stored_slice_is_the_same_after_a_new_cell(gpu, kind, N):
    G = solvers.make_solver(kind, N)
    G.set_cell_para(CELL)
    run = scft.DiblockSCFT(G, 0.3, 0.1, 18.0, 0.1)
    rng = np.random.default_rng(1)
    run.set_fields(*(rng.standard_normal(G.get_space_size_phy()) for _ in range(2)))
    run.iterate(1)
    want = [run.get_contour(c, s) for c in (0, 1) for s in (1, 4)]
    G.set_cell_para((4.1, 4.1, 5.0))
    got = [run.get_contour(c, s) for c in (0, 1) for s in (1, 4)]
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
    G.set_contour_step(0.1)
    assert np.array_equal(run.get_contour(0, 4), want[1])
    run.close()
    G.close()
