"""Performance cases: what a program that uses chemps2_gb300 has it do.

The work of a DMRG program is the sweep, and that of a sweep is the Heff matvec inside its
Davidson solver, so most cases are one matvec through DMRG.heff_apply_device or
DMRG.heff_apply_precision, from a chain of eight sites to the D = 2000 state of the
benchmark, in the three arithmetics. The others are whole calls: a small ground state from
scratch, a sweep of a converged chain, the density matrices, and a batch of small problems.

Matvec cases run on a state loaded from a checkpoint (DMRG(makechkpt=True), as a restarted
program does) whose sector dimensions have the shape that sweeps give: Gaussian in the
particle number, (2S + 1) exp(-S(S + 1) / 1.9) in the spin, about D multiplets in all, as
fitted to the swept L = 30, D = 2000 state (140 live sectors of up to 47 states in the
middle). One DMRG object per chain is kept, as a Davidson solver keeps it; the seed makes
the vectors.
"""
import os
import struct
import tempfile

import numpy as np
import torch

import chemps2_gb300 as c2g
from chemps2_gb300 import models

GROUPS = {"c1": 0, "c2v": 5, "d2h": 7}
NIRREPS = {"c1": 1, "c2v": 4, "d2h": 8}


# ---------------------------------------------------------------- cases


def listed():
    return [
        # the smallest calls: one matvec of a chain that takes microseconds
        {"name": "matvec hubbard L8 D64 fp64", "kind": "matvec", "model": "hubbard", "group": "c1", "L": 8, "N": 8,
         "two_s": 0, "D": 64, "site": 3, "precision": "fp64"},
        # the everyday chain of the reference's own CPU runs
        {"name": "matvec hubbard L16 D200 fp64", "kind": "matvec", "model": "hubbard", "group": "c1", "L": 16, "N": 16,
         "two_s": 0, "D": 200, "site": 7, "precision": "fp64"},
        # an odd electron number, a ragged site and bond dimension, four irreps
        {"name": "matvec abinitio L17 D389 fp64", "kind": "matvec", "model": "abinitio", "group": "c2v", "L": 17,
         "N": 17, "two_s": 1, "D": 389, "site": 6, "precision": "fp64"},
        # the mid-size molecule
        {"name": "matvec abinitio L24 D1000 fp64", "kind": "matvec", "model": "abinitio", "group": "d2h", "L": 24,
         "N": 24, "two_s": 0, "D": 1000, "site": 11, "precision": "fp64"},
        # the mixed solver's two arithmetics where blocks are large
        {"name": "matvec hubbard L20 D512 fp32", "kind": "matvec", "model": "hubbard", "group": "c1", "L": 20, "N": 20,
         "two_s": 0, "D": 512, "site": 9, "precision": "fp32"},
        # the headline chain: FP64, and the tensor-core form through host buffers
        {"name": "matvec abinitio L30 D2000 fp64", "kind": "matvec", "model": "abinitio", "group": "d2h", "L": 30,
         "N": 30, "two_s": 0, "D": 2000, "site": 14, "precision": "fp64"},
        {"name": "matvec abinitio L30 D2000 tc", "kind": "matvec", "model": "abinitio", "group": "d2h", "L": 30,
         "N": 30, "two_s": 0, "D": 2000, "site": 14, "precision": "tc"},
        # a small ground state from scratch: what an orbital optimisation calls many times
        {"name": "solve hubbard L8 D128", "kind": "solve", "L": 8, "N": 8, "D": 128, "sweeps": 4},
        # one more left and right sweep of a chain that has settled
        {"name": "sweep hubbard L12 D128", "kind": "sweep", "L": 12, "N": 12, "D": 128, "sweeps": 3},
        # the density matrices and correlations of a converged state
        {"name": "rdm hubbard L8 D128", "kind": "rdm", "L": 8, "N": 8, "D": 128, "sweeps": 6},
        # independent small problems on one GPU
        {"name": "batch hubbard 6 problems", "kind": "batch", "count": 6, "Lmin": 5, "Lmax": 8, "D": 128, "sweeps": 2},
    ]


def draw(rng):
    kind = rng.choice(["matvec"] * 7 + ["solve", "sweep", "rdm", "batch"])

    def log_int(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    if kind == "matvec":
        if rng.random() < 0.45:
            model, group, L = "hubbard", "c1", rng.randint(8, 20)
            D = min(log_int(48, 512), 8 << L // 2)
        else:
            model, group, L = "abinitio", rng.choice(["c2v", "d2h"]), rng.randint(10, 30)
            D = min(log_int(100, 2000 if group == "d2h" else 1000), 40 * (L - 6))
        N = L - rng.randint(0, 2)
        return {"kind": kind, "model": model, "group": group, "L": L, "N": N, "two_s": N % 2 + 2 * rng.randint(0, 1),
                "D": D, "site": rng.randint(L // 3, 2 * L // 3 - 1), "precision": rng.choice(["fp64", "fp64", "fp32", "tc"])}
    if kind == "batch":
        lo = rng.randint(4, 6)
        return {"kind": kind, "count": rng.randint(3, 8), "Lmin": lo, "Lmax": lo + 2, "D": rng.randint(90, 160), "sweeps": 2}
    L = rng.randint(9, 12) if kind == "sweep" else rng.randint(5, 8)
    D = rng.randint(64, 128) if kind == "sweep" else rng.randint(110, 200)
    return {"kind": kind, "L": L, "N": L - L % 2, "D": D, "sweeps": {"solve": 4, "sweep": 3, "rdm": 6}[kind]}


# ---------------------------------------------------------------- problems


def problem(model, two_s, n):
    ham = c2g.Hamiltonian(model.L, model.group, model.irreps)
    for i in range(model.L):
        for j in range(i, model.L):
            if model.tmat[i, j] != 0.0:
                ham.setTmat(i, j, float(model.tmat[i, j]))
    for i, j, k, l in np.argwhere(model.vmat != 0.0):
        if i <= k and j <= l:  # one of each pair that the setter mirrors
            ham.setVmat(int(i), int(j), int(k), int(l), float(model.vmat[i, j, k, l]))
    return c2g.Problem(ham, two_s, n, 0)


def scheme(D, sweeps, rtol):
    s = c2g.ConvergenceScheme(sweeps)
    for k in range(sweeps):  # one sweep an instruction: their number does not depend on the energies
        s.set_instruction(k, D, 1e-10, 1, 0.0, rtol)
    return s


def chain(L, seed):
    """A Hubbard chain with a random U and random site energies: its ground state is a
    non-degenerate singlet for an even number of electrons."""
    rng = np.random.default_rng([seed, L, 11])
    model = models.hubbard(L, float(rng.uniform(2.0, 6.0)))
    model.tmat[np.arange(L), np.arange(L)] = rng.uniform(-0.3, 0.3, L)
    return model


# ---------------------------------------------------------------- the state of the matvec cases


def sector_dims(rows, b, L, N, D):
    """About D states over the sectors of boundary b, in the shape that sweeps give."""
    fci = rows[:, 3].astype(np.float64)
    if fci.sum() <= D:
        return rows[:, 3]
    n, s = rows[:, 0].astype(np.float64), 0.5 * rows[:, 1]
    w = np.where(fci > 0, np.exp(-((n - N * b / L) ** 2) / 4.5) * (2 * s + 1) * np.exp(-s * (s + 1) / 1.9), 0.0)
    lo, hi = 0.0, 8.0 * D / w.sum()
    while hi / max(w.sum(), 1e-300) < 1e12 and np.minimum(fci, np.rint(hi * w)).sum() < D:
        hi *= 2.0
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if np.minimum(fci, np.rint(mid * w)).sum() < D else (lo, mid)
    return np.minimum(fci, np.rint(hi * w)).astype(np.int32)


def write_checkpoint(path, prob, case):
    """A checkpoint of a random state: the header, the sector dimensions of every boundary,
    and the tensor of every site, with entries scaled so that it is normalised on average."""
    L, N, D = case["L"], case["N"], case["D"]
    nirr = NIRREPS[case["group"]]
    rng = np.random.default_rng([L, N, D, nirr])
    rows = [prob.bookkeeper_sectors(D, b) for b in range(L + 1)]
    dims = [r[:, 3] if b in (0, L) else sector_dims(r, b, L, N, D) for b, r in enumerate(rows)]
    at = [{(int(r[0]), int(r[1]), int(r[2])): int(d) for r, d in zip(rows[b], dims[b])} for b in range(L + 1)]
    with open(path, "wb") as f:
        f.write(b"C2GMPS01" + struct.pack("7i", L, N, case["two_s"], 0, nirr, 0, 0))
        for d in dims:
            f.write(np.ascontiguousarray(d, dtype=np.int32).tobytes())
        for site in range(L):
            ip = prob._ham.getOrbitalIrrep(site)
            size = 0
            for (n, s, i), dl in at[site].items():
                for key in ((n, s, i), (n + 1, s - 1, i ^ ip), (n + 1, s + 1, i ^ ip), (n + 2, s, i)):
                    size += dl * at[site + 1].get(key, 0)
            rows_of_a_column = max(1.0, size / max(1, sum(at[site + 1].values())))
            f.write(struct.pack("q", size) + (rng.standard_normal(size) / np.sqrt(rows_of_a_column)).tobytes())


_kept = {}  # the one DMRG object that the matvec cases hold


def matvec_dmrg(case):
    key = tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "precision")))
    if key not in _kept:
        for old in _kept.values():
            old.close()
        _kept.clear()
        L, group = case["L"], GROUPS[case["group"]]
        model = models.hubbard(L, 4.0) if case["model"] == "hubbard" else models.synthetic_ab_initio(L, group, 1234)
        prob = problem(model, case["two_s"], case["N"])
        here = os.getcwd()
        with tempfile.TemporaryDirectory() as folder:
            os.chdir(folder)  # checkpoints are read from the working directory
            try:
                write_checkpoint("CheMPS2_MPS0.c2g", prob, case)
                dmrg = c2g.DMRG(prob, scheme(case["D"], 1, 1e-8), makechkpt=True)
            finally:
                os.chdir(here)
        for site in range(L - 2, case["site"], -1):  # the right-hand operators, down to the pair
            dmrg.update(site, False)
        _kept[key] = dmrg
    return _kept[key]


# ---------------------------------------------------------------- the interface


def prepare(case, seed):
    kind = case["kind"]
    if kind == "matvec":
        dmrg = matvec_dmrg(case)
        n = dmrg.sobject_size(case["site"])
        x = np.random.default_rng(seed).standard_normal(n)
        x /= np.linalg.norm(x)
        if case["precision"] == "tc":
            return {"case": case, "dmrg": dmrg, "x": x}
        x = torch.from_numpy(x).cuda()
        torch.cuda.current_stream().synchronize()
        return {"case": case, "dmrg": dmrg, "x": x, "y": torch.empty_like(x), "stream": torch.cuda.Stream()}
    if kind == "batch":
        rng = np.random.default_rng([seed, 5])
        Ls = [int(v) for v in rng.permutation(np.resize(np.arange(case["Lmin"], case["Lmax"] + 1), case["count"]))]
        return {"case": case, "seeds": [int(v) for v in rng.integers(1, 2**31 - 1, len(Ls))],
                "problems": [problem(chain(L, seed + 1000 * k), 0, L - L % 2) for k, L in enumerate(Ls)],
                "schemes": [scheme(case["D"], case["sweeps"], 1e-8) for _ in Ls]}
    prob = problem(chain(case["L"], seed), 0, case["N"])
    state = {"case": case, "seed": seed % (2**31 - 1) + 1, "problem": prob}
    if kind == "solve":
        state["scheme"] = scheme(case["D"], case["sweeps"], 1e-8)
        return state
    c2g.srand(state["seed"])
    if kind == "sweep":
        state["dmrg"] = c2g.DMRG(prob, scheme(case["D"], 1, 1e-8))
        for _ in range(case["sweeps"]):
            state["dmrg"].Solve()
    else:
        state["dmrg"] = c2g.DMRG(prob, scheme(case["D"], case["sweeps"], 1e-11))
        state["dmrg"].Solve()
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "matvec":
        d, x, site = state["dmrg"], state["x"], case["site"]
        if case["precision"] == "tc":  # the product is good to 16 bits or so: FP32 holds it
            return d.heff_apply_precision(site, x, "tc").astype(np.float32)
        y, s = state["y"], state["stream"]
        d.heff_apply_device(site, x.data_ptr(), y.data_ptr(), y.numel(), case["precision"], s.cuda_stream)
        if case["precision"] == "fp64":
            return y
        with torch.cuda.stream(s):
            return y.float()
    if kind == "solve":
        c2g.srand(state["seed"])
        d = c2g.DMRG(state["problem"], state["scheme"])
        energy = d.Solve()
        steps = d.step_energies()
        d.close()
        return {"energy": energy, "step_energies": steps}
    if kind == "sweep":
        # the tensors of a truncated state are defined up to rotations of its bonds only
        energy = state["dmrg"].Solve()
        return {"energy": energy, "step_energies": state["dmrg"].step_energies()[-2 * (case["L"] - 2):]}
    if kind == "rdm":
        state["dmrg"].calc_rdms_and_correlations()
        dm, corr = state["dmrg"].get2DM(), state["dmrg"].getCorrelations()
        return {"A": dm.A, "B": dm.B, "energy": dm.energy(), "mutinfo": corr["MutInfo"], "cdens": corr["Cdens"]}
    out = c2g.solve_batch(state["problems"], state["schemes"], state["seeds"], workers=4)
    return {"energies": np.array([r["energy"] for r in out])}


def work(case):
    kind, D = case["kind"], case.get("D", 0)
    if kind == "matvec":  # the operators of the two boundaries and both vectors; the compiler's ledger of products
        led = matvec_dmrg(case).bench_heff(case["site"], 0, 0, 0, "fp64")
        scale = 1.0 if case["precision"] == "fp64" else 0.5
        return {"bytes": scale * led["bytes"], "flops": led["flops"]}

    def steps(L, n):  # n two-site steps of four matvecs: L^2 operator pairs on blocks of about D / 8
        m = min(D, 4 ** (L // 2) / 3) / 8.0
        return {"bytes": n * 8.0 * L * L * 16 * m * m, "flops": n * 4 * 4.0 * L * L * 64 * m**3}

    if kind == "batch":
        Ls = np.resize(np.arange(case["Lmin"], case["Lmax"] + 1), case["count"])
        w = [steps(int(L), 2 * case["sweeps"] * (int(L) - 2)) for L in Ls]
        return {k: sum(v[k] for v in w) for k in ("bytes", "flops")}
    L = case["L"]
    return steps(L, {"solve": 2 * case.get("sweeps", 1), "sweep": 2, "rdm": 2}[kind] * (L - 2))


# ---------------------------------------------------------------- exact results


def singles(L, n):
    """<I| a+_p a_q |J> over the determinants of n electrons in L orbitals, as [p, q, I, J]."""
    dets = [m for m in range(1 << L) if bin(m).count("1") == n]
    index = {m: k for k, m in enumerate(dets)}
    out = np.zeros((L, L, len(dets), len(dets)))
    for j, m in enumerate(dets):
        for q in range(L):
            if m >> q & 1:
                m1, sq = m ^ 1 << q, bin(m & (1 << q) - 1).count("1")
                for p in range(L):
                    if not m1 >> p & 1:
                        out[p, q, index[m1 | 1 << p], j] = (-1) ** (sq + bin(m1 & (1 << p) - 1).count("1"))
    return out


def ground_state(model, n_up, n_down):
    """(energy, state as [up determinant, down determinant], single excitations of either
    spin) of a Hubbard model by diagonalisation."""
    L = model.L
    eu, ed = singles(L, n_up), singles(L, n_down)
    iu, idn = np.eye(eu.shape[2]), np.eye(ed.shape[2])
    H = np.kron(np.einsum("pq,pqij->ij", model.tmat, eu), idn) + np.kron(iu, np.einsum("pq,pqij->ij", model.tmat, ed))
    occ_u, occ_d = np.einsum("ppii->pi", eu), np.einsum("ppii->pi", ed)
    U = np.array([model.vmat[p, p, p, p] for p in range(L)])
    H[np.diag_indices_from(H)] += np.einsum("p,pi,pj->ij", U, occ_u, occ_d).ravel()
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    w, v = torch.linalg.eigh(torch.from_numpy(H).to(dev))
    return float(w[0]), v[:, 0].cpu().numpy().reshape(len(iu), len(idn)), eu, ed


def exact(case, seed):
    kind = case["kind"]
    if kind in ("matvec", "sweep"):
        # a matvec's value needs the whole many-body embedding of the state, and a truncated
        # sweep's depends on its path: neither is had from plain linear algebra
        return None
    if kind == "batch":
        rng = np.random.default_rng([seed, 5])
        Ls = [int(v) for v in rng.permutation(np.resize(np.arange(case["Lmin"], case["Lmax"] + 1), case["count"]))]
        es = [ground_state(chain(L, seed + 1000 * k), L // 2, L // 2)[0] for k, L in enumerate(Ls)]
        return {"energies": np.array(es)}
    L, half = case["L"], case["N"] // 2
    energy, c, eu, ed = ground_state(chain(L, seed), half, half)
    if kind == "solve":
        return {"energy": energy, "step_energies": None}
    up, dn = np.einsum("pqij,jk->pqik", eu, c), np.einsum("pqij,kj->pqki", ed, c)
    out = {"energy": energy, "mutinfo": None, "cdens": None}
    one = np.einsum("pqij,ij->pq", up + dn, c)
    for name, v in (("A", up + dn), ("B", up - dn)):
        f = v.reshape(L * L, -1)
        # <E_ac E_bd> - delta_bc <E_ad>, with <E_ac = <(E_ca c)|
        g = (f @ f.T).reshape(L, L, L, L).transpose(1, 2, 0, 3)
        out[name] = np.ascontiguousarray(g - np.einsum("bc,ad->abcd", np.eye(L), one))
    return out
