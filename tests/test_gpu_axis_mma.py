"""FP64 tensor-core axis passes and the one-launch-per-step kernel at the edges of their tiles:
triplets and chains against the dense per-axis operators, iterations against the numpy oracle."""
import numpy as np
import pytest

from crysscft_sample_b200 import batch, fields, scft, solvers
from oracle import scft_oracle as O

pytestmark = pytest.mark.gpu

L = (4.2, 3.9, 5.1)
U64 = 2.0**-53


def _solver(kind, N, cell=None, ds=0.01):
    G = solvers.make_solver(kind, N)
    G.set_cell_para(cell if cell is not None else ((L[0],) * 3 if kind == "PMMM" else L))
    G.set_contour_step(ds)
    return G


def _operators(kind, N, cell=None, ds=0.01):
    cell = cell if cell is not None else ((L[0],) * 3 if kind == "PMMM" else L)
    return solvers.operator_terms(kind, N, cell, ds)[0]


def _apply(A, q):
    q = np.einsum("xyj,zj->xyz", q, A[2])
    q = np.einsum("xjz,yj->xyz", q, A[1])
    return np.einsum("jyz,xj->xyz", q, A[0])


def _bound(n, q):
    # dot products of n terms on each axis: gamma_n with row sums of |A| below 1.3, twice for the
    # sums and differences of mirrored points, on both sides of the comparison
    return 2 * 2 * 1.3**3 * sum(n) * U64 * np.abs(q).max()


# lengths around the 8-wide tiles, the 32-line tiles and the block forms (n % 32), odd, tiny and
# mixed; 64, 96 and 128 have kernels of their own
GRIDS = [("P1", n) for n in [(1, 2, 3), (7, 9, 5), (8, 16, 24), (31, 33, 32), (63, 65, 64), (96, 64, 128), (127, 17, 97),
                             (129, 8, 15), (128, 40, 1)]] + \
        [(k, n) for k in ("PMMM", "3M") for n in [(2, 4, 6), (14, 18, 10), (62, 66, 64), (128, 192, 30), (90, 256, 34)]]


@pytest.mark.parametrize("kind,N", GRIDS)
def test_triplet_equals_dense_operators(gpu, kind, N):
    G = _solver(kind, N)
    n = G.get_grid_size_phy()
    q = np.random.default_rng(1).standard_normal(n)
    G.get_iomat_for_diffusion()[:] = q.ravel()
    G.diffusion()
    got = G.get_iomat_for_diffusion().reshape(n)
    assert np.abs(got - _apply(_operators(kind, N), q)).max() <= _bound(n, q)


# one launch per step (cubic 64, 96, 128; at 128 only with equal axes for PMMM), both directions,
# and a 16-byte misaligned store, which takes the three passes
# and grids up to 64 at the edges of the 8-line tiles, odd, unequal and tiny
@pytest.mark.parametrize("kind,n,cell", [("P1", (64,) * 3, L), ("P1", (96,) * 3, L), ("P1", (128,) * 3, L),
                                         ("PMMM", (64,) * 3, None), ("PMMM", (96,) * 3, None), ("PMMM", (128,) * 3, None),
                                         ("3M", (64,) * 3, L), ("PMMM", (16,) * 3, None), ("PMMM", (32,) * 3, None),
                                         ("PMMM", (48,) * 3, None), ("P1", (30,) * 3, L), ("P1", (33,) * 3, L),
                                         ("P1", (5, 9, 7), L), ("P1", (8, 64, 33), L), ("P1", (64, 17, 64), L),
                                         ("P1", (63, 1, 2), L), ("P1", (1, 2, 65), L), ("PMMM", (7, 31, 24), None)])
@pytest.mark.parametrize("direction,offset", [(1, 0), (-1, 0), (1, 1)])
def test_chain_equals_dense_operators(gpu, kind, n, cell, direction, offset):
    import torch

    N = n if kind == "P1" else tuple(2 * v for v in n)
    G, A, steps = _solver(kind, N, cell), _operators(kind, N, cell), 3
    rng = np.random.default_rng(2)
    init, w = 1 + 0.1 * rng.standard_normal(n), np.exp(0.01 * rng.standard_normal(n))
    store = torch.zeros((steps + 1) * init.size + offset, dtype=torch.float64, device="cuda")
    q = store[offset:]
    G.propagate_device(q, torch.from_numpy(init).cuda().ravel(), torch.from_numpy(w).cuda().ravel(), steps, direction)
    torch.cuda.synchronize()
    got = q.cpu().numpy().reshape((steps + 1,) + n)[::direction]
    want = init
    for k in range(1, steps + 1):
        want = w * _apply(A, w * want)
        assert np.abs(got[k] - want).max() <= k * 1.1 * _bound(n, want)


# iterations on the step kernel (96, 128), the whole-contour kernel in position order (3m, 64) and
# the passes (ragged, anisotropic), with stress and a stored slice
# one-launch-per-step kernels for sides up to 64 with the fewest steps, odd and even counts and the
# block boundary on both sides of the middle (the phi sums start two phases behind the middle)
@pytest.mark.parametrize("kind,N,fA,ds", [("P1", (96, 96, 96), 0.3, 0.1), ("PMMM", (256, 256, 256), 0.3, 0.1),
                                          ("3M", (192, 192, 192), 0.3, 0.1), ("3M", (128, 128, 128), 0.3, 0.1),
                                          ("3M", (36, 50, 30), 0.3, 0.1), ("P1", (33, 20, 15), 0.3, 0.1),
                                          ("P1", (70, 20, 15), 0.3, 0.1), ("PMMM", (32, 32, 32), 0.5, 0.4),
                                          ("PMMM", (32, 32, 32), 0.3, 0.3), ("PMMM", (30, 32, 34), 0.5, 0.21),
                                          ("PMMM", (30, 32, 34), 0.75, 0.2), ("P1", (48, 48, 48), 0.3, 0.12),
                                          ("PMMM", (64, 64, 64), 0.75, 0.07), ("P1", (13, 22, 9), 0.25, 0.03)])
def test_iterations_equal_oracle(gpu, kind, N, fA, ds):
    cell, xN = (4.2, 4.2, 4.2), 18.0
    rng = np.random.default_rng(3)
    if all(v % 2 == 0 for v in N):
        a, b = (fields.to_physical(kind, w) for w in fields.seed_fields(N, cell[0]))
    else:
        a, b = rng.standard_normal(N), rng.standard_normal(N)
    S = O.OracleSolver(kind, N)
    want = O.scft_iterations(S, fA, ds, xN, cell, 0.1, 2, a, b)
    G = solvers.make_solver(kind, N)
    G.set_cell_para(cell)
    run = scft.DiblockSCFT(G, fA, ds, xN, 0.1)
    run.set_fields(a, b)
    got = run.iterate(2)
    got.update(run.get_fields())
    assert np.abs(got["F"] - want["F"]).max() <= 1e-10 * np.abs(want["F"]).max()
    for k in ("phiA", "phiB"):
        assert np.abs(got[k] - want[k].ravel()).max() <= 1e-12
    if run.NsA < 2:
        return
    # a stored slice in the solver's own point order: one step from the one before it
    S.set_cell_para(cell)
    S.set_contour_step(ds)
    run.set_fields(a, b)
    run.iterate(1)
    w = np.exp(-ds / 2 * np.asarray(a).ravel())
    q0, q1 = run.get_contour(0, 1), run.get_contour(0, 2)
    step = w * np.asarray(S.diffusion((w * q0).reshape(S.grid_phy))).ravel()
    assert np.abs(q1 - step).max() <= 1e-13 * np.abs(step).max() * 10


# FP32 steps of grids off the tensor-core sizes: the triplets of the per-axis passes, bit for bit
# (batch form 3 runs those), at sides around the 4 x 4 results of a thread, unequal and tiny
@pytest.mark.parametrize("kind,N", [("P1", (45, 45, 45)), ("P1", (64, 63, 1)), ("P1", (7, 9, 5)), ("PMMM", (34, 62, 18)),
                                    ("3M", (36, 50, 30)), ("P1", (3, 64, 33))])
def test_fp32_steps_equal_the_passes(gpu, kind, N):
    from crysscft_sample_b200 import batch

    rng = np.random.default_rng(4)
    inst = [{"N": N, "L": (4.2, 4.2, 4.2), "fA": 0.3, "xN": 18.0}]
    B = batch.BatchSCFT(kind, inst, ds=0.06, precision="fp32")
    a, b = rng.standard_normal(B.M[0]), rng.standard_normal(B.M[0])
    B.configure(1, 3)
    B.set_fields(0, a, b)
    want = B.iterate(1)["F"][0, 0]
    G = solvers.make_solver(kind, N)
    G.set_cell_para((4.2, 4.2, 4.2))
    run = scft.DiblockSCFT(G, 0.3, 0.06, 18.0, 0.1)
    run.set_precision("fp32")
    run.set_fields(a, b)
    got = run.iterate(1)
    assert abs(got["F"][0] - want) <= 1e-12 * abs(want)  # FP64 sums in another order
    w = B.get_fields(0)
    for k, v in run.get_fields().items():
        assert np.abs(v - w[k]).max() <= 1e-12 * (1 + np.abs(w[k]).max())
    B.close()


# the one-launch batch: every side it takes and block form (reflection, two-level, circulant; equal and
# different axes; the permuted store of 3M), against one launch per step of each instance, bit for bit
@pytest.mark.parametrize("teams", [None, {8: 2, 40: 5, 56: 7, 64: 2}])
@pytest.mark.parametrize("kind,sides,cell", [("PMMM", (8, 40, 56, 64), 4.1), ("3M", (8, 40, 64), list(L)),
                                             ("P1", (8, 40, 56, 64), list(L)), ("P1", (16, 48, 64), 4.4)])
def test_batch_sides_equal_step_launches(gpu, kind, sides, cell, teams):
    m = 1 if kind == "P1" else 2
    inst = [{"N": (m * s,) * 3, "xN": 16.0 + i, "fA": 0.25 + 0.02 * i, "L": cell, "seed": 7 + i}
            for i, s in enumerate(sides)]
    runs = []
    for form in (1, 4):
        B = batch.BatchSCFT(kind, inst, ds=0.02)
        B.configure(4, form)
        if form == 4:
            B.set_team_sizes({s: t for s, t in (teams or {}).items() if s in sides})
        rng = np.random.default_rng(5)
        for i in range(len(inst)):
            B.set_fields(i, 16.0 * rng.random(B.M[i]), 16.0 * rng.random(B.M[i]))
        h = B.iterate(2)
        if form == 4:
            assert B.team_plan()["instances"] == len(inst)
        runs.append((h, [B.get_fields(i) for i in range(len(inst))]))
        B.close()
    (h1, f1), (h4, f4) = runs
    assert np.array_equal(h1["F"], h4["F"]) and np.array_equal(h1["maxinc"], h4["maxinc"])
    for a, b in zip(f1, f4):
        assert all(np.array_equal(a[k], b[k]) for k in a)
