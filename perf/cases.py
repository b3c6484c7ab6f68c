"""Timed cases of the GFN2-xTB engine: what a user's program has it compute, through the public entry points.

Two families of molecules, built by the package's own rules (axtb_b200.structures): water clusters
(compact, many fragments, 6 basis functions per molecule) and alkane chains (covalent, 6k + 2 basis
functions), from one water to 2400 basis functions. Kinds of use:

* ``single``   one molecule through ``Calculator.singlepoint``: energy, gradient, charges, moments and orbital
               levels, from the start guess (the command line's job, a geometry given once);
* ``md``       the same, started from the moments of a neighbouring geometry: a molecular-dynamics or
               optimisation step of a molecule that stays loaded;
* ``batch``    many molecules through ``Batch.run`` with host arrays (conformer and data-set screening),
               the small ones bound by launches, with implicit solvation as an option;
* ``device``   the mixed batch through ``Batch.run_device`` with positions already on the GPU: data-set
               labelling at full throughput;
* ``autograd`` energies and backward pass through ``GFN2Energy`` inside a PyTorch program;
* ``hessian``  ``numerical_hessian`` of a small molecule: a batch of displaced copies, set up in the call;
* ``density``  the allocation-free density from given Fock and overlap matrices (a caller that brings its own).
"""
import ctypes
import functools
import math

import numpy as np
import torch

from axtb_b200 import Batch, Calculator, _lib, numerical_hessian, structures
from axtb_b200.torch_ops import GFN2Energy

KT = 300.0 * 3.1668115634564e-6
NOISE = 0.02 * structures.AATOAU  # thermal-like displacement of every coordinate, bohr


def listed():
    return [
        # the smallest call there is: one water, where launches and host work are everything
        {"name": "single_water_1", "kind": "single", "family": "water", "size": 1, "accuracy": 1.0},
        # (H2O)32, 96 atoms: the ordinary single point
        {"name": "single_water_32", "kind": "single", "family": "water", "size": 32, "accuracy": 1.0},
        # C200H402, 602 atoms: a long chain, dense matrices of an even but not round size (1202)
        {"name": "single_alkane_200", "kind": "single", "family": "alkane", "size": 200, "accuracy": 1.0},
        # (H2O)400, 1200 atoms: the largest single point of the range
        {"name": "single_water_400", "kind": "single", "family": "water", "size": 400, "accuracy": 1.0},
        # split precision, the option for the dense products of a larger molecule
        {"name": "split_water_67", "kind": "single", "family": "water", "size": 67, "accuracy": 1.0, "precision": "split"},
        # one step of a trajectory of C25H52, started from the previous step's moments
        {"name": "md_alkane_25", "kind": "md", "family": "alkane", "size": 25, "accuracy": 1.0},
        # screening of small molecules (up to 62 basis functions)
        {"name": "batch_small_300", "kind": "batch", "count": 300, "lo": 1, "hi": 10, "accuracy": 0.1},
        # solvated conformers of middling size
        {"name": "batch_alpb_48", "kind": "batch", "count": 48, "lo": 6, "hi": 30, "accuracy": 1.0, "solvent": "water"},
        # the mixed batch: half water clusters of 5 to 100, half alkanes of 5 to 60, positions on the GPU
        {"name": "device_mixed_1024", "kind": "device", "count": 1024, "lo": 5, "hi": 100, "accuracy": 0.1},
        # training on energies and forces: alkanes and water clusters of 10 to 60
        {"name": "autograd_96", "kind": "autograd", "count": 96, "lo": 10, "hi": 60, "accuracy": 0.1},
        # vibrations of the water trimer: 54 displaced copies
        {"name": "hessian_water_3", "kind": "hessian", "family": "water", "size": 3},
        # a density from a caller's own matrices, an odd size
        {"name": "density_201", "kind": "density", "size": 201},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["single", "single", "split", "md", "batch", "alpb", "device", "autograd", "hessian", "density"])
    family = rng.choice(["water", "alkane"])
    if kind == "single":
        return {"kind": "single", "family": family, "size": log(1, 340) if family == "water" else log(2, 240),
                "accuracy": rng.choice([0.01, 0.1, 1.0])}
    if kind == "split":
        return {"kind": "single", "family": family, "size": log(10, 120), "accuracy": 1.0, "precision": "split"}
    if kind == "md":
        return {"kind": "md", "family": family, "size": log(2, 90), "accuracy": rng.choice([0.1, 1.0])}
    if kind == "batch":
        return {"kind": "batch", "count": log(20, 800), "lo": 1, "hi": rng.randint(4, 16), "accuracy": rng.choice([0.1, 1.0])}
    if kind == "alpb":
        return {"kind": "batch", "count": log(5, 90), "lo": 3, "hi": rng.randint(10, 40), "accuracy": 1.0,
                "solvent": rng.choice(["water", "toluene", "dmso"])}
    if kind == "device":
        return {"kind": "device", "count": log(40, 900), "lo": 5, "hi": rng.randint(20, 100), "accuracy": 0.1}
    if kind == "autograd":
        return {"kind": "autograd", "count": log(8, 200), "lo": 5, "hi": rng.randint(20, 60), "accuracy": 0.1}
    if kind == "hessian":
        return {"kind": "hessian", "family": family, "size": rng.randint(2, 5), "step": round(rng.uniform(0.003, 0.01), 4)}
    return {"kind": "density", "size": log(7, 256)}


# ---------------------------------------------------------------------------------------- molecules
@functools.lru_cache(maxsize=None)
def template(family, size):
    """Numbers and positions of one molecule of the rule; a case's seed displaces them."""
    if family == "water":
        return structures.water_cluster(size, seed=size)
    return structures.alkane(size, seed=size, gauche=0.1 if size > 60 else 0.3)


def sizes(case):
    """(family, size) of a batch's molecules: water clusters and alkanes in turn, fixed by the case."""
    rng = np.random.default_rng(case["count"] * 1009 + case["hi"])
    lo, hi = case["lo"], case["hi"]
    return [("water", int(rng.integers(lo, hi + 1))) if i % 2 == 0 else
            ("alkane", int(rng.integers(max(lo, 2), min(hi, 60) + 1))) for i in range(case["count"])]


def displaced(family, size, rng):
    z, x = template(family, size)
    return z, x + rng.normal(0.0, NOISE, x.shape)


def molecules(case, seed):
    rng = np.random.default_rng(seed)
    if "count" not in case:
        return [displaced(case["family"], case["size"], rng)]
    return [displaced(f, s, rng) for f, s in sizes(case)]


def matrices(case, seed):
    """Overlap and Fock matrix of a caller's own: Gaussians on a jittered lattice, extended-Hueckel elements."""
    n = case["size"]
    rng = np.random.default_rng(seed)
    side = math.ceil(n ** (1.0 / 3.0))
    grid = np.array([(i, j, k) for i in range(side) for j in range(side) for k in range(side)][:n], dtype=float)
    r = 2.8 * grid + rng.uniform(-0.2, 0.2, (n, 3))
    s = np.exp(-((r[:, None] - r[None]) ** 2).sum(-1) / 4.0)
    e = np.where(np.arange(n) % 2 == 0, -0.75, -0.25) + rng.uniform(-0.05, 0.05, n)
    f = 0.875 * (e[:, None] + e[None]) * s
    f[np.arange(n), np.arange(n)] = e
    return f, s, float((n + 1) // 2)


# ---------------------------------------------------------------------------------------- the cases
def options(case):
    o = {"accuracy": case.get("accuracy", 1.0)}
    if "precision" in case:
        o["precision"] = case["precision"]
    if "solvent" in case:
        o["solvation"] = ("alpb", case["solvent"])
    return o


def prepare(case, seed):
    kind = case["kind"]
    if kind == "density":
        f, s, nocc = matrices(case, seed)
        n = case["size"]
        new = functools.partial(torch.empty, dtype=torch.float64, device="cuda")
        return {"kind": kind, "n": n, "nocc": nocc, "f": torch.tensor(f, device="cuda"), "s": torch.tensor(s, device="cuda"),
                "emo": new(n), "focc": new(n), "p": new(n, n), "status": torch.zeros(1, dtype=torch.int32, device="cuda")}
    mols = molecules(case, seed)
    if kind == "hessian":
        return {"kind": kind, "mol": mols[0], "step": case.get("step", 0.005)}
    if kind in ("single", "md"):
        calc = Calculator(mols[0][0], **options(case))
        state = {"kind": kind, "calc": calc, "x": mols[0][1], "moments": None}
        if kind == "md":  # the trajectory's previous point
            step = np.random.default_rng(seed + 1).normal(0.0, NOISE, mols[0][1].shape)
            calc.set_history(None)
            calc.singlepoint(mols[0][1] + 0.2 * step, levels=False)
            state["moments"] = calc.wavefunction()
        return state
    batch = Batch(mols, **options(case))
    state = {"kind": kind, "batch": batch}
    if kind == "batch":
        state["x"] = [x for _, x in mols]
    else:
        state["x"] = torch.tensor(np.concatenate([x for _, x in mols]), device="cuda")
        if kind == "device":
            state["energy"] = torch.empty(len(mols), dtype=torch.float64, device="cuda")
            state["gradient"] = torch.empty_like(state["x"])
        else:
            g = torch.Generator(device="cuda").manual_seed(int(seed))
            state["weights"] = torch.rand(len(mols), dtype=torch.float64, device="cuda", generator=g) + 0.5
    return state


def fields(r):
    return {"energy": r.energy, "gradient": r.gradient, "charges": r.charges, "dipole": r.dipole, "qsh": r.qsh,
            "dpat": r.dpat, "qpat": r.qpat}


def run(state):
    kind = state["kind"]
    if kind == "single":
        state["calc"].set_history(None)  # a geometry of its own: from the start guess
        r = state["calc"].singlepoint(state["x"])
        return {**fields(r), "emo": r.emo, "focc": r.focc}
    if kind == "md":
        state["calc"].set_wavefunction(state["moments"])
        return fields(state["calc"].singlepoint(state["x"], levels=False))
    if kind == "batch":
        rs = [fields(r) for r in state["batch"].run(state["x"])]
        return {k: np.concatenate([np.asarray(r[k]).reshape(-1) for r in rs]) for k in rs[0]}
    if kind == "device":
        b = state["batch"]
        status = b.run_device(state["x"].data_ptr(), state["energy"].data_ptr(), state["gradient"].data_ptr())
        return {"energy": state["energy"], "gradient": state["gradient"], "status": status}
    if kind == "autograd":
        x = state["x"].detach().requires_grad_(True)
        e = GFN2Energy.apply(x, state["batch"])
        (e * state["weights"]).sum().backward()
        return {"energy": e.detach(), "gradient": x.grad}
    if kind == "hessian":
        h = numerical_hessian(*state["mol"], step=state["step"])
        return {"hessian": h.hessian, "dipole_derivatives": h.dipole_derivatives, "energy": h.reference.energy}
    p = ctypes.c_void_p
    rc = _lib.load().axtb_gpu_density_static(
        p(state["f"].data_ptr()), p(state["s"].data_ptr()), state["n"], state["nocc"], state["nocc"], KT,
        p(state["emo"].data_ptr()), p(state["focc"].data_ptr()), p(state["p"].data_ptr()),
        p(state["status"].data_ptr()), p(torch.cuda.current_stream().cuda_stream))
    if rc != 0:
        raise RuntimeError(_lib.last_error())
    return {"emo": state["emo"], "focc": state["focc"], "p": state["p"]}


def work(case):
    """Dense algebra of one eigenproblem per SCF iteration (reduction to standard form, tridiagonal form,
    occupied vectors, density: 7/3 n^3 + 4 n^2 k) for ten iterations (four from given moments), the
    weighted density, and the ATM and integral terms left out; positions in, results out."""
    if case["kind"] == "density":
        n = case["size"]
        return {"bytes": 8.0 * (3 * n * n + 2 * n), "flops": 10.0 / 3.0 * n ** 3 + 2.0 * n ** 3}
    mols = sizes(case) if "count" in case else [(case["family"], case["size"])]
    iterations = {"md": 4}.get(case["kind"], 10)
    flops = byte = 0.0
    for family, size in mols:
        nat = 3 * size if family == "water" else 3 * size + 2
        n = 6 * size if family == "water" else 6 * size + 2
        copies = 6 * nat + 1 if case["kind"] == "hessian" else 1
        k = (4 if family == "water" else 3) * size + (0 if family == "water" else 1)
        flops += copies * (n ** 3 + iterations * (7.0 / 3.0 * n ** 3 + 4.0 * n * n * k) + 2.0 * n * n * k)
        byte += copies * 8.0 * 16.0 * nat
    return {"bytes": byte, "flops": flops}


def exact(case, seed):
    """The density's values from a plain generalized eigensolve; the SCF cases have no plain form."""
    if case["kind"] != "density":
        return None
    f, s, nocc = matrices(case, seed)
    linv = np.linalg.inv(np.linalg.cholesky(s))
    e, u = np.linalg.eigh(linv @ f @ linv.T)
    c = linv.T @ u
    lo, hi = e[0] - 1.0, e[-1] + 1.0
    for _ in range(200):
        mu = 0.5 * (lo + hi)
        if (1.0 / (1.0 + np.exp(np.clip((e - mu) / KT, -700, 700)))).sum() > nocc:
            hi = mu
        else:
            lo = mu
    occ = 2.0 / (1.0 + np.exp(np.clip((e - 0.5 * (lo + hi)) / KT, -700, 700)))
    return {"emo": e, "focc": occ, "p": (c * occ) @ c.T}
