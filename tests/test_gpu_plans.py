"""What a launch plan must not outlive: the point order of a stored contour, the form a batch was
configured to, and the buffers a captured call relies on."""
import ctypes

import numpy as np
import pytest

from crysscft_sample_b200 import _lib, batch, scft, solvers

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


def _batch(kind, N, precision, first, cell=CELL, U=(0.3, 0.06)):
    """A batch of one instance that has iterated once in form `first` (None: not at all)."""
    B = batch.BatchSCFT(kind, [{"N": N, "L": cell, "fA": U[0], "xN": 18.0}], ds=U[1], precision=precision)
    rng = np.random.default_rng(2)
    B.w = [rng.standard_normal(B.M[0]) for _ in range(2)]
    if first is not None:
        B.configure(1, first)
        B.set_fields(0, *B.w)
        B.iterate(1)
    B.set_fields(0, *B.w)
    return B


# form 3 is the three axis passes a step, whatever ran before it: 4 launches beside 3 a step
@pytest.mark.parametrize("first", [None, 0, 1, 4])
@pytest.mark.parametrize("kind,N,precision", [("PMMM", (32, 32, 32), "fp64"), ("P1", (13, 22, 9), "fp64"),
                                              ("PMMM", (64, 64, 64), "fp32"), ("P1", (13, 22, 9), "fp32")])
def test_batch_form_3_is_the_axis_passes_after_any_form(gpu, kind, N, precision, first):
    B, want = _batch(kind, N, precision, first), _batch(kind, N, precision, None)
    steps = int(0.3 / 0.06) + int(0.7 / 0.06)
    for b in (B, want):
        b.configure(1, 3)
        assert b.launches_per_iteration() == 3 * steps + 4
    assert np.array_equal(B.iterate(2)["F"], want.iterate(2)["F"])
    a, b = B.get_fields(0), want.get_fields(0)
    assert all(np.array_equal(a[k], b[k]) for k in a)
    B.close()
    want.close()


# a plan keeps nothing of the operators that a new cell frees
@pytest.mark.parametrize("first", [0, 1, 4])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_batch_form_3_after_a_new_cell(gpu, precision, first):
    new = (3.7, 4.6, 4.9)
    B, want = _batch("P1", (13, 22, 9), precision, first), _batch("P1", (13, 22, 9), precision, None, cell=new)
    B.configure(1, 3)
    B.iterate(1)
    lib, d, s = _lib.load(), ctypes.c_void_p(), ctypes.c_void_p()
    _lib.check(lib.scft_batch_instance(B._h, 0, ctypes.byref(d)))
    _lib.check(lib.scft_diblock_get_solver(d, ctypes.byref(s)))
    _lib.check(lib.scft_solver_set_cell_para(s, _lib.dptr(np.array(new + (0.0, 0.0, 0.0)))))
    B.set_fields(0, *B.w)
    want.configure(1, 3)
    assert np.array_equal(B.iterate(2)["F"], want.iterate(2)["F"])
    B.close()
    want.close()


# forms 2 and 3 where form 2 has no kernel: cubic 96 and 128, and FP32 off the tensor-core sizes
@pytest.mark.parametrize("form", [2, 3])
@pytest.mark.parametrize("kind,N,precision", [("P1", (96, 96, 96), "fp64"), ("PMMM", (256, 256, 256), "fp64"),
                                              ("P1", (13, 22, 9), "fp32")])
def test_forms_without_step_launches_keep_the_axis_passes(gpu, kind, N, precision, form):
    B = _batch(kind, N, precision, None, cell=4.2, U=(0.3, 0.1))
    B.configure(1, 0)
    steps = int(0.3 / 0.1) + int(0.7 / 0.1)
    assert B.launches_per_iteration() < 3 * steps
    want = B.iterate(1)["F"]
    B.configure(1, form)
    assert B.launches_per_iteration() == 3 * steps + 4
    B.set_fields(0, *B.w)
    assert np.abs(B.iterate(1)["F"] - want).max() <= 1e-10 * np.abs(want).max()
    B.close()


# a chain enqueues and nothing else once a triplet has run: its work buffers are the triplet's
@pytest.mark.parametrize("kind,n", [("PMMM", (16, 16, 16)), ("P1", (45, 40, 54)), ("P1", (13, 22, 9)), ("P1", (96,) * 3),
                                    ("3M", (18, 25, 15))])
def test_a_chain_is_capturable_after_one_triplet(gpu, kind, n):
    import torch

    G = solvers.make_solver(kind, n if kind == "P1" else tuple(2 * v for v in n))
    G.set_cell_para(CELL)
    G.set_contour_step(0.01)
    M, steps = G.get_space_size_phy(), 5
    gen = torch.Generator(device="cuda").manual_seed(3)
    init, w = (torch.rand(M, dtype=torch.float64, device="cuda", generator=gen) for _ in range(2))
    q = torch.zeros((steps + 1) * M, dtype=torch.float64, device="cuda")
    G.diffusion_device(init.clone(), torch.cuda.current_stream())
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        G.propagate_device(q, init, w, steps, 1, torch.cuda.current_stream())
    graph.replay()
    torch.cuda.synchronize()
    want = torch.zeros_like(q)
    G.propagate_device(want, init, w, steps, 1, torch.cuda.current_stream())
    torch.cuda.synchronize()
    assert torch.equal(q, want)
    G.close()
