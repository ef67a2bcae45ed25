"""The work that users of this engine have it do, as cases that can be timed and compared.

Every case goes through the public calls (``dmrg``, ``tdvp_twosite``, ``makeEnv``, ``Lupdate`` /
``Rupdate``, ``DeviceState.heff``, ``expect``, ``correlationmatrix``, ``Server``) on the models of
the benchmark's configurations: the dense Heisenberg chain, the U(1) Heisenberg chain of 100 sites,
the U(1)xU(1) Hubbard chain, the Heisenberg cylinder and the served transverse-field Ising chains.

States are random matrix product states with the sector sizes of a solved state of that bond
dimension and Schmidt weights falling from 1 to about 1e-7 inside every charge sector, in the
right-canonical form (or mixed, where a centre inside the chain is asked for), so that the bond
dimension a truncation keeps is set by ``maxm`` as it is in the ramp of a run. Site tensors are
defined only up to a rotation of their bond states, so a solve's outputs are what does not depend
on that choice: the energy, the per-sweep records and the correlation matrix of the state that the
solve left on the device, which a program measures after it. A state truncated at a discarded
weight of 1e-8 gives correlations to about six digits, and the split-precision products carry
32-bit accuracy, so the correlations after a solve, and all that a split-precision solve gives,
are handed on as 32-bit numbers.
"""
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]


def package():
    """The repository's package (its folder's name is not an identifier)."""
    if "dmrjtensor_b200" not in sys.modules:
        where = ROOT / "dmrjtensor.jl_b200"
        spec = importlib.util.spec_from_file_location(
            "dmrjtensor_b200", where / "__init__.py", submodule_search_locations=[str(where)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["dmrjtensor_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["dmrjtensor_b200"]


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # one effective-Hamiltonian product through the environment API on a small dense chain:
        # the smallest call, where launches and planning are everything
        dict(name="heff_small", kind="heff", model="heisenberg", L=14, m=45, precision="fp64"),
        # the same product on a U(1) state of several hundred states in the split form, as a
        # program with its own eigensolver calls it
        dict(name="heff_u1_split", kind="heff", model="heisenberg_u1", L=40, m=320,
             precision="3xtf32"),
        # Lupdate and Rupdate on dense tensors of odd sizes (host arrays in and out)
        dict(name="env_step", kind="env_step", ml=151, mr=203, d=2, w=5),
        # makeEnv of a resident dense state with its centre inside the chain, and the two
        # environments at the centre
        dict(name="make_env", kind="make_env", model="heisenberg", L=26, m=384),
        # the dense L=20 chain of the small configuration: bond 10 start, maxm 100, eight Krylov
        # vectors
        dict(name="chain_dense", kind="dmrg", model="heisenberg", L=20, m=10, maxm=100, sweeps=3,
             cutoff=1e-10, krylov=8, precision="fp64", half=False),
        # one sweep of the L=100 U(1) chain at a step of its bond-dimension ramp, then its
        # spin correlations
        dict(name="chain_u1", kind="dmrg", model="heisenberg_u1", L=100, m=135, maxm=173, sweeps=1,
             cutoff=1e-8, krylov=2, precision="fp64", half=False),
        # the half-filled Hubbard chain, L=32, with the split-precision products it is meant to be
        # run with
        dict(name="hubbard_split", kind="dmrg", model="hubbard", L=32, m=400, maxm=450, sweeps=1,
             cutoff=1e-8, krylov=2, precision="3xtf32", half=False),
        # the 4 x 16 cylinder in FP64 at the bond dimension its cutoff keeps: the heaviest of the
        # configurations
        dict(name="cylinder", kind="dmrg", model="cylinder", L=64, m=450, maxm=500, sweeps=1,
             cutoff=1e-8, krylov=2, precision="fp64", half=False),
        # a dense chain at the largest bond dimension of the served requests, one half sweep with
        # eight Krylov vectors: density matrices of 1024 states
        dict(name="dense_large", kind="dmrg", model="heisenberg", L=22, m=512, maxm=512, sweeps=1,
             cutoff=1e-8, krylov=8, precision="fp64", half=True),
        # measurements on a resident U(1) state: the energy and two correlation matrices
        dict(name="measure", kind="measure", model="heisenberg_u1", L=100, m=150),
        # imaginary-time evolution: one two-site TDVP call on the U(1) chain
        dict(name="tdvp", kind="tdvp", model="heisenberg_u1", L=60, m=120, maxm=120, krylov=4,
             prefactor=-2.0, cutoff=1e-8, precision="fp64"),
        # serving: transverse-field Ising chains of mixed length and maxm, submitted at once to a
        # running server
        dict(name="serve", kind="serve", requests=16, slots=8, sweeps=4, cutoff=1e-8,
             precision="fp64"),
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["heff", "env_step", "make_env", "dmrg", "dmrg", "dmrg", "dmrg", "3s",
                       "measure", "tdvp", "serve"])
    prec = rng.choice(["fp64", "fp64", "3xtf32", "bf16x9"])
    if kind == "heff":
        model = rng.choice(["heisenberg", "heisenberg_u1", "tfi"])
        return dict(kind=kind, model=model, L=rng.randint(12, 40), m=log(16, 400), precision=prec)
    if kind == "env_step":
        return dict(kind=kind, ml=log(16, 400), mr=log(16, 400), d=rng.choice([2, 2, 3, 4]),
                    w=rng.choice([3, 5, 6, 14]))
    if kind == "make_env":
        return dict(kind=kind, model=rng.choice(["heisenberg", "heisenberg_u1", "hubbard"]),
                    L=rng.randint(12, 32), m=log(24, 384))
    if kind == "measure":
        return dict(kind=kind, model=rng.choice(["heisenberg", "heisenberg_u1"]),
                    L=rng.randint(16, 100), m=log(24, 160))
    if kind == "tdvp":
        m = log(24, 140)
        return dict(kind=kind, model=rng.choice(["heisenberg", "heisenberg_u1"]),
                    L=rng.randint(10, 60), m=m, maxm=m + rng.randint(0, 20),
                    krylov=rng.randint(2, 8), prefactor=-round(rng.uniform(0.5, 3.0), 3),
                    cutoff=1e-8, precision="fp64")
    if kind == "3s":
        m = log(16, 120)
        return dict(kind=kind, model=rng.choice(["heisenberg", "heisenberg_u1"]),
                    L=rng.randint(10, 60), m=m, maxm=m + rng.randint(1, 30), sweeps=1,
                    cutoff=1e-8, krylov=2, precision="fp64", half=False)
    if kind == "serve":
        return dict(kind=kind, requests=rng.randint(2, 16), slots=rng.randint(2, 8), sweeps=4,
                    cutoff=1e-8, precision="fp64")
    model = rng.choice(["heisenberg", "heisenberg_u1", "hubbard", "cylinder", "tfi"])
    L, m = {"heisenberg": (rng.randint(8, 22), log(16, 400)),
            "tfi": (rng.randint(8, 40), log(16, 256)),
            "heisenberg_u1": (rng.randint(12, 100), log(32, 300)),
            "hubbard": (rng.randint(8, 32), log(32, 400)),
            "cylinder": (4 * rng.randint(4, 16), log(32, 450))}[model]
    return dict(kind="dmrg", model=model, L=L, m=m, maxm=m + rng.randint(1, 1 + m // 4),
                sweeps=rng.randint(1, 2) if m < 128 else 1, cutoff=1e-8,
                krylov=rng.choice([2, 2, 4, 8]) if model != "cylinder" else 2,
                precision=prec, half=rng.random() < 0.25)


# ------------------------------------------------------------------ states

SPIN = [(1,), (-1,)]
FERMION = [(0, 0), (1, 1), (1, -1), (2, 0)]


def physical(model):
    """(charges of the site's basis states, whether the state conserves them)."""
    if model == "hubbard":
        return FERMION, True
    return SPIN, model in ("heisenberg_u1", "cylinder")


def charges_of(model):
    """The charges of the site's basis states, empty where none are conserved."""
    phys, conserved = physical(model)
    return phys if conserved else [()] * len(phys)


def add(a, b, sign=1):
    return tuple(x + sign * y for x, y in zip(a, b))


def sectors(model, L, m):
    """Per bond, the (charge, states) list of a half-filled (Sz = 0) state of about m states: a
    normal distribution of the charge around its mean, limited by what either side can reach.
    A dense bond is one sector without charges."""
    phys, conserved = physical(model)
    if not conserved:
        d = len(phys)
        return [[((), int(min(d ** min(b, 30), d ** min(L - b, 30), m)))] for b in range(L + 1)]
    pairs = model == "hubbard"
    end = (L, L % 2) if pairs else (L % 2,)
    from_left = [{(0,) * len(end): 1}]
    for _ in range(L):
        nxt = {}
        for q, n in from_left[-1].items():
            for p in phys:
                nxt[add(q, p)] = min(nxt.get(add(q, p), 0) + n, 10 ** 9)
        from_left.append(nxt)
    from_right = [{end: 1}]
    for _ in range(L):
        nxt = {}
        for q, n in from_right[-1].items():
            for p in phys:
                nxt[add(q, p, -1)] = min(nxt.get(add(q, p, -1), 0) + n, 10 ** 9)
        from_right.append(nxt)
    from_right.reverse()
    out = []
    for b in range(L + 1):
        most = {q: min(n, from_right[b].get(q, 0)) for q, n in from_left[b].items()}
        if pairs:
            w = {q: math.exp(-(q[0] - b) ** 2 / 2.5 - q[1] ** 2 / 2.5) for q in most}
        else:
            w = {q: math.exp(-q[0] ** 2 / 7.0) for q in most}
        tot = sum(w[q] for q in most if most[q])
        dims = {q: min(most[q], int(round(m * w[q] / tot))) for q in most}
        out.append({q: n for q, n in dims.items() if n > 0})
    out[0], out[L] = {(0,) * len(end): 1}, {end: 1}
    for _ in range(2):          # no sector larger than its neighbours can carry
        for b in range(L - 1, -1, -1):
            out[b] = {q: min(n, sum(out[b + 1].get(add(q, p), 0) for p in phys))
                      for q, n in out[b].items()}
            out[b] = {q: n for q, n in out[b].items() if n > 0}
        for b in range(1, L + 1):
            out[b] = {q: min(n, sum(out[b - 1].get(add(q, p, -1), 0) for p in phys))
                      for q, n in out[b].items()}
            out[b] = {q: n for q, n in out[b].items() if n > 0}
    return [sorted(s.items()) for s in out]


class Blocks:
    """A matrix product state in block form: per site and left sector one matrix [dim, columns],
    its column blocks in the order of the physical states (the block order of the package)."""

    def __init__(self, model, L, m, seed, centre=0):
        self.phys, self.conserved = physical(model)
        self.charges = charges_of(model)
        self.bonds = sectors(model, L, m)
        self.L, self.oc = L, centre
        rng = np.random.default_rng(seed)
        self.site = []
        for i in range(L):
            groups = []
            for q, n in self.bonds[i]:
                cols = [np.zeros((n, 0))]
                for _, k in self.targets(i, q):
                    D = self.bonds[i + 1][k][1]
                    # Schmidt weights falling from 1 to about 1e-7 inside the sector
                    scale = np.exp(-8.0 * (np.arange(D) + 0.5) / max(D, 8))
                    cols.append(rng.standard_normal((n, D)) * scale)
                groups.append(np.concatenate(cols, axis=1))
            self.site.append(groups)
        for i in range(L - 1, 0, -1):
            self.to_left(i)
        for i in range(centre):
            self.to_right(i)
        norm = math.sqrt(sum(float(np.sum(g * g)) for g in self.site[centre]))
        self.site[centre] = [g / norm for g in self.site[centre]]

    def targets(self, i, q):
        """(physical state, right sector) of every block of left charge q at site i."""
        where = {c: k for k, (c, _) in enumerate(self.bonds[i + 1])}
        return [(s, where[add(q, p)]) for s, p in enumerate(self.charges) if add(q, p) in where]

    def to_left(self, i):
        """Site i right-canonical, its remainder into site i-1."""
        rest = []
        for k, g in enumerate(self.site[i]):
            Q, R = np.linalg.qr(g.T)
            self.site[i][k] = Q.T
            rest.append(R.T)
        for k, (q, _) in enumerate(self.bonds[i - 1]):
            g, o = self.site[i - 1][k], 0
            for _, t in self.targets(i - 1, q):
                D = self.bonds[i][t][1]
                g[:, o:o + D] = g[:, o:o + D] @ rest[t]
                o += D

    def to_right(self, i):
        """Site i left-canonical, its remainder into site i+1."""
        parts = {}
        for k, (q, n) in enumerate(self.bonds[i]):
            o = 0
            for _, t in self.targets(i, q):
                D = self.bonds[i + 1][t][1]
                parts.setdefault(t, []).append((k, o, self.site[i][k][:, o:o + D]))
                o += D
        for t, ps in parts.items():
            Q, R = np.linalg.qr(np.concatenate([p[2] for p in ps], axis=0))
            r = 0
            for k, o, blk in ps:
                self.site[i][k][:, o:o + blk.shape[1]] = Q[r:r + blk.shape[0]]
                r += blk.shape[0]
            self.site[i + 1][t] = R @ self.site[i + 1][t]

    def dense(self, i):
        ml = sum(n for _, n in self.bonds[i])
        mr = sum(n for _, n in self.bonds[i + 1])
        A = np.zeros((ml, len(self.phys), mr))
        start = np.cumsum([0] + [n for _, n in self.bonds[i + 1]])
        r = 0
        for k, (q, n) in enumerate(self.bonds[i]):
            o = 0
            for s, t in self.targets(i, q):
                D = self.bonds[i + 1][t][1]
                A[r:r + n, s, start[t]:start[t] + D] = self.site[i][k][:, o:o + D]
                o += D
            r += n
        return A

    def labels(self):
        """The charge of every state of every bond."""
        return [[q for q, n in bond for _ in range(n)] for bond in self.bonds]

    def host(self):
        """What a program holds on the host: the block form of a charged state, plain tensors
        otherwise."""
        if not self.conserved:
            return [np.asfortranarray(self.dense(i)) for i in range(self.L)]
        out = []
        for i in range(self.L):
            out.append(np.concatenate([g.ravel(order="F") for g in self.site[i]]))
        return out


def as_mps(state):
    """A fresh MPS object on the state's host data."""
    pkg = package()
    if not state["conserved"]:
        return pkg.MPS(state["host"], oc=state["oc"])
    psi = pkg.MPS(oc=state["oc"])
    psi.sectors, psi.blocks = state["bonds"], state["host"]
    psi.phys = [list(state["phys"])] * len(state["host"])
    return psi


def operator(case, seed):
    """The case's MPO: the model in a random field along z (a disorder realisation)."""
    pkg = package()
    model, L = case["model"], case["L"]
    if model == "hubbard":
        mpo = pkg.makeMPO(pkg.hubbardMPO(t=1.0, mu=0.0, HubU=4.0), 4, L).with_qn(pkg.HUBBARD_QN)
    elif model == "cylinder":
        mpo = pkg.heisenbergCylinderMPO(4, L // 4).with_qn(pkg.SPIN_QN)
    elif model == "tfi":
        mpo = pkg.makeMPO(pkg.tfiMPO(h=0.9), 2, L)
    else:
        mpo = pkg.makeMPO(pkg.heisenbergMPO, 2, L)
        mpo = mpo.with_qn(pkg.SPIN_QN) if model == "heisenberg_u1" else mpo
    field = np.random.default_rng(seed + 7919).uniform(-0.2, 0.2, L)
    for i in range(L):                   # the on-site slot: last row, first column
        mpo.W[i][-1, :, :, 0] += field[i] * spin_z(model)
    return mpo


def spin_z(model):
    return np.diag([0.0, 0.5, -0.5, 0.0]) if model == "hubbard" else np.diag([0.5, -0.5])


def requests(case, seed):
    """The served requests: transverse-field Ising chains, h in [0.5, 1.5], in a weak random field
    along z, from the |+...+> state."""
    pkg = package()
    rng = np.random.default_rng(seed)
    shape = np.random.default_rng(case["requests"])      # lengths and maxm belong to the case
    out = []
    for _ in range(case["requests"]):
        L = int(shape.choice([16, 32, 64, 128]))
        m = int(shape.choice([64, 128, 256, 512]))
        mpo = pkg.makeMPO(pkg.tfiMPO(h=float(rng.uniform(0.5, 1.5))), 2, L)
        for w, b in zip(mpo.W, rng.uniform(-0.1, 0.1, L)):
            w[-1, :, :, 0] += b * np.diag([1.0, -1.0])
        psi = pkg.MPS([np.full((1, 2, 1), 1 / math.sqrt(2)) for _ in range(L)], oc=0)
        out.append((psi, mpo, m))
    return out


def env_step_inputs(case, seed):
    rng = np.random.default_rng(seed)
    ml, mr, d, w = case["ml"], case["mr"], case["d"], case["w"]
    A = rng.standard_normal((ml, d, mr)) / math.sqrt(d * max(ml, mr))
    W = np.zeros((w, d, d, w))           # lower triangular in the MPO states, as every MPO here
    W[0, :, :, 0] = W[w - 1, :, :, w - 1] = np.eye(d)
    W[1:w - 1, :, :, 0] = rng.standard_normal((w - 2, d, d))
    W[w - 1, :, :, 1:w - 1] = rng.standard_normal((d, d, w - 2))
    return A, W, rng.standard_normal((ml, w, ml)), rng.standard_normal((mr, w, mr))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "serve":
        return dict(case=case, requests=requests(case, seed),
                    server=package().Server(slots=case["slots"], hbm_budget=150 * 10 ** 9))
    if kind == "env_step":
        A, W, Lenv, Renv = env_step_inputs(case, seed)
        return dict(case=case, A=A, W=W, Lenv=Lenv, Renv=Renv)
    centre = case["L"] // 2 if kind in ("heff", "make_env") else 0
    b = Blocks(case["model"], case["L"], case["m"], seed, centre)
    state = dict(case=case, mpo=operator(case, seed), host=b.host(), bonds=b.bonds, phys=b.charges,
                 conserved=b.conserved, oc=centre, sz=spin_z(case["model"]))
    if kind == "heff":
        pkg = package()
        dev = pkg.DeviceState(as_mps(state), state["mpo"].device())
        dev.env_build()
        state["dev"] = dev
        state["x"] = np.asfortranarray(np.tensordot(b.dense(centre), b.dense(centre + 1), (2, 0)))
    elif kind in ("make_env", "measure"):
        state["psi"] = as_mps(state)
        package().makeEnv(state["psi"], state["mpo"])       # resident on the device from here on
    return state


def records(stats):
    """The per-sweep records of a solve as one array: energy, truncation error, entropy and the
    largest singular values at the centre bond."""
    return np.array([[s["energy"], s["max_truncerr"], s["entropy"], *s["d_top"]] for s in stats])


def correlations(state, psi):
    return package().correlationmatrix(psi, state["sz"], state["sz"]).astype(np.float32)


def run(state):
    case, pkg = state["case"], package()
    kind = case["kind"]
    if kind == "heff":
        return state["dev"].heff(state["oc"], state["x"], precision=case["precision"])
    if kind == "env_step":
        return [pkg.Lupdate(state["Lenv"], state["A"], state["A"], state["W"]),
                pkg.Rupdate(state["Renv"], state["A"], state["A"], state["W"])]
    if kind == "make_env":
        Lenv, Renv = pkg.makeEnv(state["psi"], state["mpo"])
        return [Lenv[state["oc"]], Renv[state["oc"]]]
    if kind == "measure":
        sp = np.array([[0.0, 1.0], [0.0, 0.0]])
        return [pkg.expect(state["psi"], state["mpo"]),
                pkg.correlationmatrix(state["psi"], state["sz"], state["sz"]),
                pkg.correlationmatrix(state["psi"], sp, sp.T)]
    if kind == "serve":
        srv = state["server"]
        tickets = [srv.submit(psi, mpo, m=m, sweeps=case["sweeps"], cutoff=case["cutoff"],
                              precision=case["precision"])
                   for psi, mpo, m in state["requests"]]
        out = []
        for t in tickets:
            st, psi = srv.result(t)
            srv.release(t)
            out.append([st["energy"], st["max_truncerr"], st["entropy"]])
        return np.array(out)
    psi = as_mps(state)
    if kind == "tdvp":
        pkg.tdvp_twosite(psi, state["mpo"], m=case["maxm"], cutoff=case["cutoff"],
                         r=case["krylov"], prefactor=case["prefactor"],
                         precision=case["precision"])
        last = psi.sweep_stats[-1]
        return [np.array([last["energy"], last["max_truncerr"]]),
                correlations(state, psi)]
    pkg.dmrg(psi, state["mpo"], m=case["maxm"], sweeps=case["sweeps"], cutoff=case["cutoff"],
             method="3S" if kind == "3s" else "twosite", krylov=case["krylov"],
             precision=case["precision"], halfsweep=case["half"])
    recs = records(psi.sweep_stats)
    if case["precision"] != "fp64":
        recs = recs.astype(np.float32)
    return [recs, correlations(state, psi)]


# ------------------------------------------------------------------ work

MPO_STATES = {"heisenberg": 5, "heisenberg_u1": 5, "hubbard": 6, "cylinder": 14, "tfi": 3}


def blocks_of(case):
    """Per site, the (left, right) sector sizes of the blocks that the charges allow."""
    charges = charges_of(case["model"])
    bonds = sectors(case["model"], case["L"], case["m"])
    out = []
    for i in range(case["L"]):
        right = dict(bonds[i + 1])
        out.append([(n, right[add(q, p)]) for q, n in bonds[i] for p in charges
                    if add(q, p) in right])
    return bonds, charges, out


def work(case):
    kind = case["kind"]
    if kind == "env_step":
        ml, mr, d, w = case["ml"], case["mr"], case["d"], case["w"]
        one = 2.0 * w * d * (ml * ml * mr + ml * mr * mr)
        n = 2 * ml * d * mr + w * (ml * ml + mr * mr) * 2 + 2 * w * d * d * w
        return {"bytes": 8.0 * n, "flops": 2 * one}
    if kind == "serve":
        n = f = 0.0
        for psi, mpo, m in requests(case, 0):
            L, m = len(mpo), 16                   # the cutoff keeps about 16 states
            f += case["sweeps"] * 2 * (L - 1) * 2 * (2 * 3 * 4 * 2 * m ** 3)
            n += 8.0 * L * (2 + 2 * m * m + 3 * m * m)
        return {"bytes": n, "flops": f}
    L, w = case["L"], MPO_STATES[case["model"]]
    d = len(physical(case["model"])[0])
    bonds, charges, site = blocks_of(case)
    vals = [sum(n * k for n, k in blocks) for blocks in site]
    env = [w * sum(n * n for _, n in b) for b in bonds]
    # a product with an environment on one side and on the other, per block
    env_f = [2.0 * w * sum(n * k * (n + k) for n, k in blocks) for blocks in site]
    corr_f = sum(4.0 * (i + 1) * sum(n * k * (n + k) for n, k in site[i]) for i in range(L))
    if kind == "make_env":
        return {"bytes": 8.0 * (sum(vals) + env[L // 2] + env[L // 2 + 1]), "flops": sum(env_f)}
    if kind == "measure":
        return {"bytes": 8.0 * (sum(vals) + 2 * L * L), "flops": sum(env_f) + 2 * corr_f}
    heff_f, two, eig_f = [], [], []
    for i in range(L - 1):
        last = dict(bonds[i + 2])
        pairs = [(n, last[add(add(q, p), r)]) for q, n in bonds[i] for p in charges
                 for r in charges if add(add(q, p), r) in last]
        two.append(sum(n * k for n, k in pairs))
        heff_f.append(2.0 * w * sum(n * k * (n + k) for n, k in pairs))
        # the density matrix of a centre sector has about d times its states
        eig_f.append(sum(4.0 / 3 * min(d * n, d * sum(x for _, x in bonds[i])) ** 3
                         for _, n in bonds[i + 1]))
    if kind == "heff":
        c = L // 2
        return {"bytes": 8.0 * (2 * two[c] + env[c] + env[c + 2]), "flops": heff_f[c]}
    steps = 1.0 if kind == "tdvp" or case["half"] else 2.0
    steps *= case.get("sweeps", 1)
    f = steps * (case["krylov"] * sum(heff_f) + sum(eig_f) + sum(env_f)) + corr_f
    n = 8.0 * (2 * sum(vals) + sum(env) * steps + L * L)
    return {"bytes": n, "flops": f}


# ------------------------------------------------------------------ the same in plain torch, 64 bits

DEV = "cuda" if torch.cuda.is_available() else "cpu"


def on(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=DEV)


def next_left(E, A, W):
    T = torch.tensordot(E, A, ([2], [0]))                   # a w s b'
    T = torch.tensordot(T, W, ([1, 2], [0, 1]))             # a b' t w'
    return torch.tensordot(A, T, ([0, 1], [0, 2])).permute(0, 2, 1)


def next_right(E, A, W):
    T = torch.tensordot(A, E, ([2], [0]))                   # b s w' a'
    T = torch.tensordot(T, W, ([1, 2], [1, 3]))             # b a' w t
    return torch.tensordot(T, A, ([1, 3], [2, 1]))


def two_site(E, F, x, V, W):
    T = torch.tensordot(E, x, ([2], [0]))                   # a w s1 s2 d
    T = torch.tensordot(T, V, ([1, 2], [0, 1]))             # a s2 d t1 w'
    T = torch.tensordot(T, W, ([4, 1], [0, 1]))             # a d t1 t2 w''
    return torch.tensordot(T, F, ([1, 4], [0, 1]))


def one_site(E, F, x, W):
    T = torch.tensordot(E, x, ([2], [0]))                   # a w s b
    T = torch.tensordot(T, W, ([1, 2], [0, 1]))             # a b t w'
    return torch.tensordot(T, F, ([1, 3], [0, 1]))


def environments(A, W, oc):
    L = len(A)
    left, right = [None] * L, [None] * L
    left[0] = right[L - 1] = torch.ones((1, 1, 1), dtype=torch.float64, device=DEV)
    for i in range(oc):
        left[i + 1] = next_left(left[i], A[i], W[i])
    for i in range(L - 1, oc, -1):
        right[i - 1] = next_right(right[i], A[i], W[i])
    return left, right


def krylov(apply, x, k):
    """Orthonormal Krylov vectors from x and the projected matrix."""
    V = [x / x.norm()]
    T = np.zeros((k, k))
    for j in range(k):
        y = apply(V[j])
        T[j, j] = float((V[j] * y).sum())
        if j == k - 1:
            break
        for _ in range(2):
            for v in V:
                y = y - (v * y).sum() * v
        b = float(y.norm())
        if b <= 1e-10:
            T = T[:j + 1, :j + 1]
            break
        T[j, j + 1] = T[j + 1, j] = b
        V.append(y / b)
    return V, T


def cut(weights, maxm, cutoff, mag):
    """How many of the (descending) weights a truncation keeps, and the discarded weight."""
    tail = np.concatenate([np.cumsum(weights[::-1])[::-1], [0.0]])
    tot = tail[0] if mag == 0 else mag
    k = next((n for n in range(1, len(weights) + 1) if tail[n] <= cutoff * tot), len(weights))
    k = max(1, min(max(k, 2), maxm, len(weights)))
    return k, float(tail[k] / tot)


def split(x, j, maxm, cutoff, mag, q, phys):
    """The two-site tensor as two sites, the centre moved on in direction j; q: the charges of
    the states of the bonds on its left, between the sites and on its right."""
    a, s, t, b = x.shape
    M = x.reshape(a * s, t * b)
    if j > 0:
        side = [add(c, p) for c in q[0] for p in phys]
    else:
        M = M.T
        side = [add(c, p, -1) for p in phys for c in q[2]]
    values, vectors = [], []
    for c in sorted(set(side)):
        at = torch.tensor([n for n, e in enumerate(side) if e == c], device=x.device)
        m = M[at]
        lam, U = torch.linalg.eigh(m @ m.T)
        values += [(float(v), c, n) for n, v in enumerate(lam.cpu().numpy())]
        vectors.append((c, at, U))
    values.sort(key=lambda v: -v[0])
    lam = np.array([v[0] for v in values])
    k, err = cut(lam, maxm, cutoff, mag)
    Q = torch.zeros((M.shape[0], k), dtype=x.dtype, device=x.device)
    q[1], o = [], 0
    for c, at, U in vectors:
        keep = torch.tensor([n for _, e, n in values[:k] if e == c], device=x.device, dtype=torch.long)
        Q[at, o:o + len(keep)] = U[:, keep]
        q[1] += [c] * len(keep)
        o += len(keep)
    rest = Q.T @ M
    if j > 0:
        return Q.reshape(a, s, k), rest.reshape(k, t, b), err, lam[:k]
    return rest.T.reshape(a, s, k), Q.T.reshape(k, t, b), err, lam[:k]


def moved(A, l, x, j, case, mag, q):
    """Sites l, l+1 and the charges of the bond between them replaced by the split of x."""
    three = q[l:l + 3]
    A[l], A[l + 1], err, kept = split(x, j, case["maxm"], case["cutoff"], mag, three,
                                      charges_of(case["model"]))
    q[l + 1] = three[1]
    return err, kept


def exact_sweeps(A, W, q, case):
    L, oc, j = len(A), 0, 1
    left, right = environments(A, W, 0)
    recs = []
    S, top = 0.0, np.zeros(8)
    for _ in range(case["sweeps"]):
        worst = 0.0
        if case["half"]:
            S, top = 0.0, np.zeros(8)
        for _ in range((L - 1) * (1 if case["half"] else 2)):
            l, r = (oc, oc + 1) if j > 0 else (oc - 1, oc)
            A[oc] = A[oc] / A[oc].norm()
            x = torch.tensordot(A[l], A[r], ([2], [0]))
            V, T = krylov(lambda v: two_site(left[l], right[r], v, W[l], W[r]), x, case["krylov"])
            lam, U = np.linalg.eigh(T)
            x = sum(float(U[n, 0]) * V[n] for n in range(len(V)))
            err, kept = moved(A, l, x, j, case, 1.0, q)
            worst = max(worst, err)
            if j < 0 and oc == min(max(2, (L + 1) // 2 + 1), L) - 1:
                kept = kept[kept > 0]
                S = float(-np.sum(kept * np.log(kept)))
                top = np.zeros(8)
                top[:min(8, len(kept))] = np.sqrt(kept[:8])
            if j > 0:
                left[oc + 1] = next_left(left[oc], A[oc], W[oc])
            else:
                right[oc - 1] = next_right(right[oc], A[oc], W[oc])
            oc += j
            if (j > 0 and oc == L - 1) or (j < 0 and oc == 0):
                j = -j
        recs.append([float(lam[0]), worst, S, *top])
    return np.array(recs), A


def exact_tdvp(A, W, q, case):
    L, oc, worst = len(A), 0, 0.0
    left, right = environments(A, W, 0)
    tau = case["prefactor"] / (L - 1) / 2

    def evolve(apply, x):
        V, T = krylov(apply, x, max(2, case["krylov"]))
        lam, U = np.linalg.eigh(T)
        c = U @ (np.exp(tau * lam) * U[0])
        x = sum(float(c[n]) * V[n] for n in range(len(V)))
        return x / x.norm(), float(lam[0])

    for _ in range(L - 1):
        l, r = oc, oc + 1
        x = torch.tensordot(A[l], A[r], ([2], [0]))
        x, E = evolve(lambda v: two_site(left[l], right[r], v, W[l], W[r]), x)
        err, _ = moved(A, l, x, 1, case, 0.0, q)
        worst = max(worst, err)
        left[r] = next_left(left[l], A[l], W[l])
        A[r], E = evolve(lambda v: one_site(left[r], right[r], v, W[r]), A[r])
        oc += 1
    return np.array([E, worst]), A


def exact_correlations(A, C, D):
    """<C_i D_j> / <psi|psi>, mirrored below the diagonal."""
    L = len(A)
    C, D = on(C), on(D)

    def through(E, B, K):
        T = torch.matmul(E, B.reshape(B.shape[0], -1))                    # .. a (s b')
        T = T.reshape(*E.shape[:-1], *B.shape[1:]).flatten(-3, -2)        # .. (a s) b'
        return torch.matmul(K.reshape(-1, K.shape[2]).T, T)

    right = [None] * (L + 1)
    one = torch.ones((1, 1), dtype=torch.float64, device=DEV)
    right[L] = one
    for i in range(L - 1, -1, -1):
        T = torch.tensordot(A[i], right[i + 1], ([2], [0]))
        right[i] = torch.tensordot(T, A[i], ([1, 2], [1, 2]))             # b(ket) a(bra)
    norm = float(right[0][0, 0])
    rho = np.zeros((L, L))
    E, X = one, None
    for j in range(L):
        DA = torch.einsum("ts,asb->atb", D, A[j])
        if X is not None:
            v = (through(X, DA, A[j]) * right[j + 1].T).sum((-2, -1)) / norm
            rho[:j, j] = rho[j, :j] = v.cpu().numpy()
        CD = torch.einsum("ts,asb->atb", C @ D, A[j])
        rho[j, j] = float((through(E, CD, A[j]) * right[j + 1].T).sum()) / norm
        new = through(E, torch.einsum("ts,asb->atb", C, A[j]), A[j])[None]
        X = new if X is None else torch.cat([through(X, A[j], A[j]), new])
        E = through(E, A[j], A[j])
    return rho


def exact(case, seed):
    kind = case["kind"]
    if kind in ("serve", "3s"):       # many whole solves; a noise schedule of its own
        return None
    if kind == "dmrg" and case["precision"] != "fp64":
        return None                   # a trajectory of 32-bit products has no 64-bit one
    if kind == "env_step":
        A, W, E, F = (on(a) for a in env_step_inputs(case, seed))
        return [next_left(E, A, W).cpu().numpy(), next_right(F, A, W).cpu().numpy()]
    centre = case["L"] // 2 if kind in ("heff", "make_env") else 0
    b = Blocks(case["model"], case["L"], case["m"], seed, centre)
    A = [on(b.dense(i)) for i in range(b.L)]
    W = [on(w) for w in operator(case, seed).W]
    if kind == "heff":
        left, right = environments(A, W, centre)
        right_of = right[centre + 1]
        x = torch.tensordot(A[centre], A[centre + 1], ([2], [0]))
        return two_site(left[centre], right_of, x, W[centre], W[centre + 1]).cpu().numpy()
    if kind == "make_env":
        left, right = environments(A, W, centre)
        return [left[centre].cpu().numpy(), right[centre].cpu().numpy()]
    sz = spin_z(case["model"])
    if kind == "measure":
        E = torch.ones((1, 1, 1), dtype=torch.float64, device=DEV)
        for a, w in zip(A, W):
            E = next_left(E, a, w)
        sp = np.array([[0.0, 1.0], [0.0, 0.0]])
        return [float(E[0, 0, 0]), exact_correlations(A, sz, sz),
                exact_correlations(A, sp, sp.T)]
    if kind == "tdvp":
        recs, A = exact_tdvp(A, W, b.labels(), case)
    else:
        recs, A = exact_sweeps(A, W, b.labels(), case)
    return [recs, exact_correlations(A, sz, sz)]
