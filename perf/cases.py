"""Timed workloads of the library: what its users have it do, over the sizes they use.

An operation (`op`) is one call, or one short sequence of calls, of the public Python API:

  triplet        diffusion_device: one triplet on a device field (a driver that keeps its own
                 contour arrays on the GPU calls this once per contour step)
  triplet_host   diffusion on the solver's host iomat: the reference's own driver, unchanged,
                 calls this once per contour step
  propagate      propagate_device: one whole chain (solve_diffusion_equation) on device arrays,
                 forward or backward
  iterate        DiblockSCFT.iterate on resident fields, the SCFT loop itself
  iterate_host   the same for a driver that keeps wA, wB on the host between calls
  polished       iterate_polished: FP32 iterations finished by FP64 ones
  relax          one evaluation of a cell relaxation: new cell, fields in, Anderson-mixed
                 iterations, the stress of the converged contour, fields out
  batch          a batch of independent PMMM instances of mixed size, advanced together

Sizes are logical (full-cell) grids; PMMM and 3M store an eighth of the points.  Parameters are
those of the repository's benchmark and tests: BCC or FCC seed fields, fA 0.2 .. 0.35,
chiN 14 .. 30, L 3.8 .. 5.5, ds 0.005 or 0.01.
"""
import math

import numpy as np
import torch

from crysscft_sample_b200 import scft, solvers
from crysscft_sample_b200.batch import BatchSCFT, batch_config

ACCEPTANCE = 0.1  # simple mixing
BETA = 0.5        # Anderson mixing


def _case(name, op, kind, grid, L, fA, ds, n=0, xN=20.0, history=0, direction=1, phase="BCC"):
    lx, ly, lz = (L, L, L) if isinstance(L, float) else L
    c = {"op": op, "kind": kind, "nx": grid[0], "ny": grid[1], "nz": grid[2], "lx": lx, "ly": ly, "lz": lz,
         "fA": fA, "xN": xN, "ds": ds, "n": n, "history": history, "direction": direction, "phase": phase}
    return {"name": name, **c} if name else c


def listed():
    return [
        # the smallest call there is: one triplet of a 32^3 cell, launch latency and little else
        _case("triplet_pmmm_32", "triplet", "PMMM", (32, 32, 32), 4.2, 0.25, 0.01),
        # the drop-in path of the reference's driver at the benchmark's size
        _case("triplet_host_pmmm_128", "triplet_host", "PMMM", (128, 128, 128), 4.2, 0.25, 0.005),
        # one A-block chain of the benchmark system, as solve_diffusion_equation runs it
        _case("propagate_pmmm_128", "propagate", "PMMM", (128, 128, 128), 4.2, 0.25, 0.005, n=50),
        # an orthorhombic P1 cell with odd, ragged sides, backward
        _case("propagate_p1_ragged", "propagate", "P1", (45, 40, 54), (4.2, 3.7, 5.1), 0.25, 0.01, n=75, direction=-1),
        # the small test system, fields on the host between calls, ten iterations a call (the
        # driver prints every tenth)
        _case("iterate_host_pmmm_32", "iterate_host", "PMMM", (32, 32, 32), 4.2, 0.25, 0.01, n=10),
        # the benchmark: 128^3 BCC, Ns = 200
        _case("iterate_pmmm_128", "iterate", "PMMM", (128, 128, 128), 4.2, 0.25, 0.005, n=10),
        # the same system with the other two solvers
        _case("iterate_3m_128", "iterate", "3M", (128, 128, 128), 4.2, 0.25, 0.005, n=5),
        _case("iterate_p1_128", "iterate", "P1", (128, 128, 128), 4.2, 0.25, 0.005, n=2),
        # the largest grid of the benchmark
        _case("iterate_pmmm_256", "iterate", "PMMM", (256, 256, 256), 4.2, 0.25, 0.005, n=2),
        # the precision form at the benchmark's 9 : 1
        _case("polished_pmmm_128", "polished", "PMMM", (128, 128, 128), 4.2, 0.25, 0.005, n=10),
        # a cell-relaxation step at 64^3
        _case("relax_pmmm_64", "relax", "PMMM", (64, 64, 64), 4.0, 0.25, 0.01, n=12, history=10),
        # sixteen instances of the batch benchmark's distribution
        _case("batch_pmmm_16", "batch", "PMMM", (16, 20261203, 0), 0.0, 0.0, 0.01, n=2),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _side(rng, kind, lo, hi):
    """A logical side: PMMM and 3M need even ones; two in three are multiples of 16 (8 for P1)."""
    v = _log(rng, lo, hi)
    step = (8 if kind == "P1" else 16) if rng.random() < 2 / 3 else (1 if kind == "P1" else 2)
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    op = rng.choice(["triplet", "triplet_host", "propagate", "iterate", "iterate", "iterate_host", "polished", "relax",
                     "batch"])
    ds = rng.choice([0.005, 0.01])
    fA, xN, phase = round(rng.uniform(0.2, 0.35), 3), round(rng.uniform(14.0, 30.0), 2), rng.choice(["BCC", "FCC"])
    if op == "batch":
        return _case("", op, "PMMM", (rng.randint(4, 24), rng.randint(1, 9999), 0), 0.0, 0.0, 0.01, n=rng.randint(1, 3))
    kind = rng.choice(["PMMM", "3M", "P1"])
    hi = {"iterate": 128, "triplet": 128, "relax": 48}.get(op, 64)
    lo, hi = (16, hi) if kind == "P1" else (32, 2 * hi)
    a = _side(rng, kind, lo, hi)
    cubic = rng.random() < 0.5
    grid = (a, a, a) if cubic else (a, _side(rng, kind, lo, hi), _side(rng, kind, lo, hi))
    L = round(rng.uniform(3.8, 5.5), 3)
    Ls = L if cubic or kind == "PMMM" else (L, round(rng.uniform(3.8, 5.5), 3), round(rng.uniform(3.8, 5.5), 3))
    n = {"triplet": 0, "triplet_host": 0, "propagate": int(_log(rng, 10, 150)), "iterate": int(_log(rng, 1, 10)),
         "iterate_host": int(_log(rng, 1, 10)), "polished": rng.randint(4, 10), "relax": rng.randint(5, 12)}[op]
    if op == "relax":  # ordered phases: in the disordered ones the stress that is asked for vanishes
        fA, xN = max(fA, 0.25), max(xN, 20.0)
    c = _case("", op, kind, grid, Ls, fA, ds, n=n, xN=xN, history=rng.randint(4, 10) if op == "relax" else 0,
              direction=rng.choice([1, -1]) if op == "propagate" else 1, phase=phase)
    if op == "iterate":  # no more work than two iterations of the largest grid
        c["n"] = max(1, min(n, int(2.0**21 * 200 * 2 / (math.prod(_phys(c)) / ds))))
    return c


# ---- inputs -------------------------------------------------------------------------
def _grid(case):
    return case["nx"], case["ny"], case["nz"]


def _phys(case):
    return _grid(case) if case["kind"] == "P1" else tuple(v // 2 for v in _grid(case))


def _fields(case, seed):
    """Host wA, wB on the physical grid: a BCC or FCC modulation and a little noise."""
    rng = np.random.default_rng(seed)
    n = _phys(case)
    amp = rng.uniform(1.8, 2.2)
    cs = []
    for d in range(3):
        i = np.arange(n[d])
        x = 2 * i + 0.5 if case["kind"] == "3M" else i + 0.5  # 3M: the even sub-lattice
        cs.append(np.cos(2 * np.pi * x / _grid(case)[d]))
    x, y, z = cs[0][:, None, None], cs[1][None, :, None], cs[2][None, None, :]
    S = x * y + y * z + z * x if case["phase"] == "BCC" else x * y * z
    wA = amp * S + 0.01 * rng.standard_normal(n)
    wB = -amp * S + 0.01 * rng.standard_normal(n)
    return wA.ravel(), wB.ravel()


def _solver(case):
    G = solvers.make_solver(case["kind"], _grid(case))
    G.set_cell_para((case["lx"], case["ly"], case["lz"]))
    G.set_contour_step(case["ds"])
    return G


class _Resident:
    """A field in the library's own memory, as an array that keeps its owner alive."""

    def __init__(self, owner, ptr, size, device):
        self.owner = owner
        face = {"shape": (size,), "typestr": "<f8", "data": (ptr, False), "version": 3}
        setattr(self, "__cuda_array_interface__" if device else "__array_interface__", face)


def _device_array(owner, ptr, size):
    return torch.as_tensor(_Resident(owner, ptr, size, True), device="cuda")


def _host_array(owner, a):
    return np.asarray(_Resident(owner, a.ctypes.data, a.size, False))


def _instances(case):
    """The batch's systems: nx of them, drawn with the case's own number ny; their fields are the seed's."""
    return batch_config(case["nx"], seed=case["ny"])


def prepare(case, seed):
    op = case["op"]
    if op == "batch":
        its = _instances(case)
        b = BatchSCFT("PMMM", its, ds=case["ds"], acceptance=ACCEPTANCE)
        for i, it in enumerate(its):
            b.set_fields(i, *_fields(_instance_case(case, it), seed + i))
        b.configure(8, 4)
        total = sum(b.M)
        out = {k: torch.empty(total, dtype=torch.float64).pin_memory().numpy() for k in ("phiA", "phiB", "wA", "wB")}
        return {"case": case, "batch": b, "out": out}
    G = _solver(case)
    wA, wB = _fields(case, seed)
    s = {"case": case, "solver": G}
    if op == "triplet":
        s["q"] = torch.from_numpy(np.exp(0.1 * wA)).cuda()
    elif op == "triplet_host":
        s["iomat"] = _host_array(G, G.get_iomat_for_diffusion())
        s["iomat"][:] = np.exp(0.1 * wA)
    elif op == "propagate":
        s["init"] = torch.from_numpy(np.exp(0.02 * wB)).cuda()
        s["wds"] = torch.from_numpy(np.exp(-case["ds"] / 2 * wA)).cuda()
        s["q"] = torch.empty((case["n"] + 1) * wA.size, dtype=torch.float64, device="cuda")
    else:
        run = scft.DiblockSCFT(G, case["fA"], case["ds"], case["xN"], ACCEPTANCE)
        s["run"] = run
        if op == "iterate_host":
            s["host"] = [torch.from_numpy(v).pin_memory().numpy() for v in (wA, wB, np.empty_like(wA), np.empty_like(wB))]
        elif op == "relax":
            s["w"] = (wA, wB)
            run.set_mixing("anderson", history=case["history"], beta=BETA)
        else:
            run.set_fields(wA, wB)
            s["fields"] = {k: _device_array(run, p, run.M)
                           for k, p in zip(("phiA", "phiB", "wA", "wB"), run.device_fields())}
    return s


def run(s):
    case, op = s["case"], s["case"]["op"]
    if op == "triplet":
        s["solver"].diffusion_device(s["q"])
        return s["q"]
    if op == "triplet_host":
        s["solver"].diffusion()
        return s["iomat"]
    if op == "propagate":
        s["solver"].propagate_device(s["q"], s["init"], s["wds"], case["n"], case["direction"])
        return s["q"]
    if op == "iterate":
        return {**s["run"].iterate(case["n"]), **s["fields"]}
    if op == "polished":
        return {**s["run"].iterate_polished(case["n"], 1), **s["fields"]}
    if op == "iterate_host":
        wA, wB, phiA, phiB = s["host"]
        return {**s["run"].iterate_host(wA, wB, case["n"], phiA, phiB), "wA": wA, "wB": wB}
    if op == "relax":
        s["solver"].set_cell_para((case["lx"], case["ly"], case["lz"]))
        s["run"].set_fields(*s["w"])
        h = s["run"].iterate(case["n"])
        return {**h, "residuals": s["run"].residuals(), **s["run"].stress(), **s["run"].get_fields()}
    b, out = s["batch"], s["out"]
    h = b.iterate(case["n"])
    o = 0
    for i, m in enumerate(b.M):
        b.get_fields(i, out=[out[k][o:o + m] for k in ("phiA", "phiB", "wA", "wB")])
        o += m
    return {**h, **out}


# ---- what a pass cannot do without ------------------------------------------------------
def _instance_case(case, it):
    return dict(case, kind="PMMM", nx=it["N"][0], ny=it["N"][1], nz=it["N"][2], lx=it["L"], ly=it["L"], lz=it["L"],
                fA=it["fA"], xN=it["xN"], phase=it["phase"])


def _triplet_flops(M):
    return 5.0 * M * math.log2(M) + 3.0 * M  # two fast transforms, K and the Boltzmann factors


def work(case):
    op = case["op"]
    if op == "batch":
        parts = [work(dict(_instance_case(case, it), op="iterate")) for it in _instances(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    M = math.prod(_phys(case))
    if op in ("triplet", "triplet_host"):
        return {"bytes": 16.0 * M, "flops": _triplet_flops(M)}
    if op == "propagate":
        return {"bytes": 8.0 * M * (case["n"] + 3), "flops": case["n"] * _triplet_flops(M)}
    U = sum(scft.contour_counts(case["fA"], case["ds"]))
    # per iteration both contour stores are written (get_contour returns them, phi and the
    # stress come from them), wA and wB are read, phiA, phiB, wA and wB written
    contour = 2.0 * (U + 1) * M
    w = {"bytes": case["n"] * (8.0 * contour + 48.0 * M), "flops": case["n"] * (2 * U * _triplet_flops(M) + 2 * contour)}
    if op == "polished":
        w["bytes"] -= (case["n"] - 1) * 4.0 * contour  # FP32 stores
    if op == "relax":
        w["bytes"] += 8.0 * contour                    # the stress reads them once
        w["flops"] += 3 * U * _triplet_flops(M)
    return w


# ---- the same in plain torch, 64 bits -----------------------------------------------------
def _axis(kind, N, L, ds, derivative=False):
    """The operator of one axis on its physical grid, and if asked its derivative by L."""
    k = np.arange(N)
    k = np.minimum(k, N - k) * (2 * np.pi / L)
    g = np.exp(-ds * k * k)
    if derivative:
        g = g * 2 * ds * k * k / L
    if kind == "P1":
        d = (np.arange(N)[:, None] - np.arange(N)[None, :]) % N
        c = np.cos(2 * np.pi / N * np.arange(N))
        return torch.from_numpy((c[(np.arange(N)[:, None] * np.arange(N)[None, :]) % N] @ g / N)[d]).cuda()
    n = N // 2
    i = np.arange(n)
    pos = 2 * i if kind == "3M" else i  # PMMM and 3M keep points of one mirror-symmetric line
    c = np.cos(np.pi / N * ((np.arange(n)[:, None] * (2 * pos + 1)[None, :]) % (2 * N)))
    s = np.where(np.arange(n) == 0, 1.0, 2.0) / n
    return torch.from_numpy(c.T @ ((g[:n] * s)[:, None] * c)).cuda()


class _Exact:
    def __init__(self, case):
        self.n = _phys(case)
        Ls = (case["lx"],) * 3 if case["kind"] == "PMMM" else (case["lx"], case["ly"], case["lz"])
        self.A = [_axis(case["kind"], N, L, case["ds"]) for N, L in zip(_grid(case), Ls)]
        self.dA = [_axis(case["kind"], N, L, case["ds"], True) for N, L in zip(_grid(case), Ls)]

    def apply(self, ops, q):
        nx, ny, nz = self.n
        t = q.reshape(nx * ny, nz) @ ops[2].T
        t = torch.matmul(ops[1], t.reshape(nx, ny, nz))
        return (ops[0] @ t.reshape(nx, ny * nz)).reshape(-1)

    def chain(self, init, wds):
        q = [init]
        for w in wds:
            q.append(w * self.apply(self.A, w * q[-1]))
        return q


def _exact_iterations(case, wA, wB, history, stress):
    E = _Exact(case)
    NsA, NsB = scft.contour_counts(case["fA"], case["ds"])
    fA, xN, ds = case["fA"], case["xN"], case["ds"]
    wA, wB = torch.from_numpy(wA).cuda(), torch.from_numpy(wB).cuda()
    rows, past = [], []
    for _ in range(case["n"]):
        ksi = 0.5 * (wA + wB - xN)
        eA, eB = torch.exp(-ds / 2 * wA), torch.exp(-ds / 2 * wB)
        one = torch.ones_like(wA)
        w = [eA] * NsA + [eB] * NsB
        q = E.chain(one, w)
        qc = E.chain(one, w[::-1])[::-1]
        Q = qc[0].mean()
        prod = [a * b for a, b in zip(q, qc)]
        phiA = fA / (NsA * Q) * (sum(prod[1:NsA], torch.zeros_like(one)) + 0.5 * (prod[0] + prod[NsA]))
        phiB = (1 - fA) / (NsB * Q) * (sum(prod[NsA + 1:-1], torch.zeros_like(one)) + 0.5 * (prod[NsA] + prod[-1]))
        rest = 1 - phiA - phiB
        parts = torch.stack([xN * (phiA * phiB).mean(), -torch.log(Q), -(wA * phiA + wB * phiB).mean(), -(ksi * rest).mean()])
        rA, rB = xN * phiB + ksi - wA, xN * phiA + ksi - wB
        rms = torch.sqrt((rA.square().sum() + rB.square().sum()) / (2 * wA.numel()))
        rows.append((parts.sum(), parts, rest.abs().max(), Q, rms))
        if not history:
            wA, wB = wA + ACCEPTANCE * rA, wB + ACCEPTANCE * rB
            continue
        W, R = torch.cat([wA, wB]), torch.cat([rA, rB])
        dw, dr = torch.zeros_like(W), torch.zeros_like(R)
        if past:
            D = torch.stack([R - r for _, r in past])
            c = torch.linalg.solve(D @ D.T, D @ R)
            for cj, (pw, pr) in zip(c, past):
                dw += cj * (pw - W)
                dr += cj * (pr - R)
        past = ([(W, R)] + past)[:history]
        wA, wB = torch.chunk(W + dw + BETA * (R + dr), 2)
    out = {k: np.array([r[i].cpu().numpy() for r in rows]) for i, k in enumerate(("F", "parts", "maxinc", "Q"))}
    out |= {"phiA": phiA, "phiB": phiB, "wA": wA, "wB": wB}
    if stress:
        grad = []
        for a in range(3):
            ops = [E.dA[b] if b == a else E.A[b] for b in range(3)]
            grad.append(sum(torch.dot(w_ * qc[t + 1], E.apply(ops, w_ * q[t])) for t, w_ in enumerate(w)) / wA.numel() / Q)
        out["residuals"] = np.array([r[4].item() for r in rows])
        out["dlnQ_dL"] = np.array([g.item() for g in grad])
        out["dF_dxN"] = ((phiA * phiB).mean() + 0.5 * (1 - phiA - phiB).mean()).item()
        out["Q"] = Q.item()  # stress() reports the last iteration's
    return out


def exact(case, seed):
    op = case["op"]
    if op == "batch":
        per = []
        for i, it in enumerate(_instances(case)):
            c = _instance_case(case, it)
            per.append(_exact_iterations(c, *_fields(c, seed + i), 0, False))
        out = {k: np.stack([p[k] for p in per], axis=1) for k in ("F", "maxinc")}
        out |= {k: torch.cat([p[k] for p in per]).cpu().numpy() for k in ("phiA", "phiB", "wA", "wB")}
        return out
    wA, wB = _fields(case, seed)
    if op in ("triplet", "triplet_host"):
        E = _Exact(case)
        return E.apply(E.A, torch.from_numpy(np.exp(0.1 * wA)).cuda())
    if op == "propagate":
        init = torch.from_numpy(np.exp(0.02 * wB)).cuda()
        wds = torch.from_numpy(np.exp(-case["ds"] / 2 * wA)).cuda()
        q = _Exact(case).chain(init, [wds] * case["n"])
        return torch.cat(q if case["direction"] == 1 else q[::-1])
    out = _exact_iterations(case, wA, wB, case["history"], op == "relax")
    return {k: v.cpu().numpy() if isinstance(v, torch.Tensor) and op in ("iterate_host", "relax") else v
            for k, v in out.items()}
