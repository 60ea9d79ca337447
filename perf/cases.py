"""Performance cases of the exact-diagonalization engine.

Each case is one call (or one short sequence of calls) that a user's program
makes through the public entry points of ``lsquantumed_gb300``:

    hv      y = H x for one vector (what MatMult is in the reference's drivers)
    dots    Gram-Schmidt projection h = V^T w of a Krylov expansion
    combine Krylov-Schur restart combination V Y
    solve   eigensolve of one Hamiltonian with random fields, eigenvectors read
    batch   eigensolve of several field realisations at once
    pairs   <O_ij> of one state for every pair of sites
    dsf     dynamical-structure-factor coefficients <v_n| S_i |psi>
    egrad   Hellmann-Feynman gradient of an energy over every bond and field
    mixed   <lambda| dH/dtheta |psi> over every bond and field (adjoint gradients)

Sizes are those of the repository's benchmark workloads and tests: chains,
square and honeycomb lattices from 12 to 30 sites.
"""
import math

import numpy as np
import torch

import lsquantumed_gb300 as ed

SOLVE_TOL = 1e-10


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------
def listed():
    return [
        # smallest product: the plain chain of 16 sites, complex vector, one launch chain per call
        dict(name="hv_chain16", kind="hv", lattice="chain", lx=1, ly=16, sz=0, j2=0.0, form="complex"),
        # ordinary product of a real-storage program: 4x6 frustrated square lattice with fields
        dict(name="hv_square24", kind="hv", lattice="square", lx=4, ly=6, sz=0, j2=0.5, form="real"),
        # largest product: 6x5, with x.y and |y|^2 as a Lanczos step wants them
        dict(name="hv_square30", kind="hv", lattice="square", lx=6, ly=5, sz=0, j2=0.55, form="real_dot"),
        # projection of the new vector on 13 Krylov vectors of the 4x6 lattice
        dict(name="dots_13x2704156", kind="dots", n=2704156, m=13),
        # restart of ncv = 16 vectors of the 4x7 lattice, nine of them kept
        dict(name="combine_16to9x40116600", kind="combine", n=40116600, m=16, keep=9),
        # smallest solve: ground state of the 16-site chain, latency of every step counts
        dict(name="solve_chain16", kind="solve", lattice="chain", lx=1, ly=16, sz=0, j2=0.0, width=0.3, nev=1, ncv=0),
        # large solve: ground state of the 4x7 lattice, vectors far beyond the L2 cache
        dict(name="solve_square28", kind="solve", lattice="square", lx=4, ly=7, sz=0, j2=0.55, width=0.3, nev=1, ncv=16),
        # disorder sweep: 64 realisations of the 20-site chain in the Sz = 1 sector
        dict(name="batch_chain20", kind="batch", lattice="chain", lx=1, ly=20, sz=1, j2=0.2, width=2.0, nev=2, count=64),
        # all S_i.S_j of a real state of the 4x7 lattice
        dict(name="pairs_square28", kind="pairs", lattice="square", lx=4, ly=7, sz=0, op="SiSj", values="real"),
        # S^z_i matrix elements to ten states of the 4x6 lattice
        dict(name="dsf_square24", kind="dsf", lattice="square", lx=4, ly=6, sz=0, op="Sqz", nev=10),
        # energy gradient over the 96 bonds and 24 fields of the 4x6 lattice
        dict(name="egrad_square24", kind="egrad", lattice="square", lx=4, ly=6, sz=0),
        # adjoint contraction of a correlation gradient on the 4x4 lattice: 64 bonds twice, 16 fields
        dict(name="mixed_square16", kind="mixed", lattice="square", lx=4, ly=4, sz=0),
    ]


_SHAPES = {"chain": [(1, n) for n in range(12, 27, 2)],
           "square": [(3, 4), (2, 7), (4, 4), (3, 6), (4, 5), (2, 11), (4, 6), (6, 4), (2, 13)],
           "honeycomb": [(2, 6), (4, 4), (2, 10), (4, 6), (6, 4)]}


def _shape(rng, most):
    lattice = rng.choice(sorted(_SHAPES))
    lx, ly = rng.choice([s for s in _SHAPES[lattice] if s[0] * s[1] <= most])
    return dict(lattice=lattice, lx=lx, ly=ly, sz=rng.choice([0, 0, 0, 1, 2]))


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["hv", "hv", "dots", "combine", "solve", "solve", "batch", "pairs", "dsf", "egrad", "mixed"])
    case = dict(kind=kind)
    j2 = rng.choice([0.0, 0.2, round(rng.uniform(0.1, 1.0), 3)])
    if kind == "hv":
        case.update(_shape(rng, 26), j2=j2, form=rng.choice(["complex", "real", "real_dot"]))
    elif kind == "dots":
        case.update(n=_log_int(rng, 5_000, 40_000_000), m=rng.randint(1, 32))
    elif kind == "combine":
        m = rng.randint(4, 32)
        case.update(n=_log_int(rng, 5_000, 40_000_000), m=m, keep=rng.randint(1, m - 1))
    elif kind == "solve":
        case.update(_shape(rng, 24), j2=j2, width=round(rng.uniform(0.2, 2.0), 3), nev=rng.randint(1, 4),
                    ncv=rng.choice([0, 0, 16, 24]))
    elif kind == "batch":
        case.update(_shape(rng, 18), j2=j2, width=round(rng.uniform(0.5, 3.0), 3), nev=rng.randint(1, 2),
                    count=rng.randint(3, 48))
    elif kind == "pairs":
        case.update(_shape(rng, 26), op=rng.choice(["SiSj", "SiSj", "SzSz", "SpSm", "SmSp"]),
                    values=rng.choice(["real", "real", "real", "complex"]))
    elif kind == "dsf":
        case.update(_shape(rng, 24), op=rng.choice(["Sqz", "Sqp"]), nev=rng.randint(1, 12))
    elif kind == "egrad":
        case.update(_shape(rng, 26))
    else:
        case.update(_shape(rng, 24))
    return case


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
_LATTICES = {"chain": ed.chain1D, "square": ed.square2D, "honeycomb": ed.honeycomb2D}


def _sites(case):
    return case["lx"] * case["ly"]


def _dim(case, more=0):
    return math.comb(_sites(case), _sites(case) // 2 + case["sz"] + more)


def _lattice(env, case):
    make = _LATTICES[case["lattice"]]
    return make(env) if case["lattice"] == "chain" else make(env, case["lx"], case["ly"])


def _system(case, seed):
    env = ed.Environment(nspins=_sites(case))
    basis = ed.Basis(env, case["sz"])
    return env, basis, _lattice(env, case)


def _fields(case, seed):
    w = case.get("width", 0.5)
    return np.random.default_rng(seed).uniform(-w, w, _sites(case))


def _hamiltonian(env, basis, lattice, case, seed, fields=True):
    j2 = case.get("j2", 0.0)
    h = ed.Hamiltonian(env, basis, lattice, 1.0, 1.0, j2, j2)
    h.build_diag(env)
    h.build_off_diag(env)
    if fields:
        h.build_disorder(env, _fields(case, seed))
    return h


def _rng(seed):
    return torch.Generator(device="cuda").manual_seed(1000 + seed)


def _unit_vector(g, n):
    """A Krylov vector: centred entries, unit norm."""
    v = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
    return v / v.norm()


def _state(g, n, values="real"):
    """An eigenvector-like state: amplitudes over a few decades, mostly of one sign, unit norm."""
    a = torch.exp(1.5 * torch.randn(n, dtype=torch.float64, device="cuda", generator=g))
    a *= torch.randn(n, dtype=torch.float64, device="cuda", generator=g) + 1.0
    a /= a.norm()
    if values == "real":
        return torch.complex(a, torch.zeros_like(a))
    phase = 2.0 * math.pi * torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
    return torch.polar(a.abs(), 0.25 * phase)


def _pairs(lattice):
    return np.concatenate([lattice.nn_pairs, lattice.nnn_pairs])


def prepare(case, seed):
    kind = case["kind"]
    g = _rng(seed)
    if kind in ("dots", "combine"):
        env = ed.Environment(nspins=2)
        V = [_unit_vector(g, case["n"]) for _ in range(case["m"])]
        if kind == "dots":
            return dict(kind=kind, env=env, V=V, w=_unit_vector(g, case["n"]))
        q, _ = np.linalg.qr(np.random.default_rng(seed).standard_normal((case["m"], case["m"])))
        return dict(kind=kind, env=env, V=V, Y=np.ascontiguousarray(q[:, :case["keep"]]))
    env, basis, lattice = _system(case, seed)
    state = dict(kind=kind, env=env, basis=basis, lattice=lattice)
    if kind == "hv":
        state.update(h=_hamiltonian(env, basis, lattice, case, seed), form=case["form"])
        if case["form"] == "complex":
            x = torch.complex(_unit_vector(g, basis.size), _unit_vector(g, basis.size)) / math.sqrt(2.0)
        else:
            x = _unit_vector(g, basis.size)
        state.update(x=x)
    elif kind == "solve":
        state.update(h=_hamiltonian(env, basis, lattice, case, seed), nev=case["nev"],
                     ncv=case["ncv"] or ed.PETSC_DEFAULT)
    elif kind == "batch":
        h = _hamiltonian(env, basis, lattice, case, seed, fields=False)
        w = case["width"]
        f = np.random.default_rng(seed).uniform(-w, w, (case["count"], _sites(case)))
        state.update(h=h, batch=ed.DisorderBatch(h, f), nev=case["nev"], count=case["count"])
    elif kind == "pairs":
        state.update(op=getattr(ed, case["op"])(env, basis), psi=_state(g, basis.size, case["values"]))
    elif kind == "dsf":
        target = basis if case["op"] == "Sqz" else ed.Basis(env, case["sz"] + 1)
        vecs = torch.stack([_state(g, target.size) for _ in range(case["nev"])])
        state.update(target=target, op=0 if case["op"] == "Sqz" else 1, psi=_state(g, basis.size), vecs=vecs)
    elif kind == "egrad":
        state.update(bonds=_pairs(lattice), psi=_state(g, basis.size))
    else:
        bonds = [tuple(map(int, b)) for b in _pairs(lattice)]
        terms = [(ed.Adjoint.XY, i, j) for i, j in bonds] + [(ed.Adjoint.ZZ, i, j) for i, j in bonds]
        terms += [(ed.Adjoint.Z, i, i) for i in range(_sites(case))]
        state.update(terms=terms, lam=_state(g, basis.size), psi=_state(g, basis.size))
    return state


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
def _fixed_sign(v):
    """Eigenvectors (rows) with their largest entry positive: a level of a disordered sample is single, so
    this fixes what an eigensolver leaves open."""
    at = v.real.abs().argmax(dim=1, keepdim=True)
    return v * torch.sign(torch.gather(v.real, 1, at))


def run(state):
    kind, env = state["kind"], state["env"]
    if kind == "hv":
        h, x = state["h"], state["x"]
        if state["form"] == "complex":
            return h.apply(x)
        return h.apply_real(x) if state["form"] == "real" else h.apply_real_dot(x)
    if kind == "dots":
        return ed.bv_dot_real(env, state["V"], state["w"])
    if kind == "combine":
        return ed.bv_mult_real(env, state["V"], state["Y"])
    if kind == "solve":
        eps = ed.Solver.SolverInit(state["h"], state["nev"], state["ncv"])
        ed.Solver.EPSSetTolerances(eps, SOLVE_TOL)
        ed.Solver.solve(env, eps)
        values, vectors = [], []
        for i in range(state["nev"]):
            e, v, _ = ed.Solver.solution(eps, i)
            values.append(e)
            vectors.append(v)
        ed.Solver.SolverClean(eps)
        return np.array(values), _fixed_sign(torch.stack(vectors))
    if kind == "batch":
        r = state["batch"].solve(nev=state["nev"], tol=SOLVE_TOL)
        v = [state["batch"].eigenvector(b, i) for b in range(state["count"]) for i in range(state["nev"])]
        return r["evals"], _fixed_sign(torch.stack(v))
    if kind == "pairs":
        return state["op"].AllPairs(state["psi"])
    if kind == "dsf":
        return ed.Phys.dsf_coefficients(env, state["basis"], state["target"], state["op"], state["psi"], state["vecs"])
    if kind == "egrad":
        return ed.Adjoint.energy_gradient(state["basis"], state["bonds"], state["psi"])
    return ed.Adjoint.expect_mixed(state["basis"], state["terms"], state["lam"], state["psi"])


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------
def _bond_counts(case):
    """Distinct nearest- and next-nearest-neighbour bonds (0 where the coupling is zero)."""
    n = _sites(case)
    per_site = {"chain": (1, 1), "square": (2, 2), "honeycomb": (1.5, 3)}[case["lattice"]]
    return n * per_site[0], (n * per_site[1] if case.get("j2", 0.0) else 0)


def _hv_flops(case):
    """Two operations per bond that flips, in the mean over the rows."""
    n, up = _sites(case), _sites(case) // 2 + case["sz"]
    p = 2.0 * math.comb(n - 2, up - 1) / math.comb(n, up)
    return 2.0 * sum(_bond_counts(case)) * p * _dim(case)


def work(case):
    kind = case["kind"]
    if kind == "dots":
        return dict(bytes=8 * case["n"] * (case["m"] + 1), flops=2 * case["n"] * case["m"])
    if kind == "combine":
        return dict(bytes=8 * case["n"] * (case["m"] + case["keep"]), flops=2 * case["n"] * case["m"] * case["keep"])
    dim, n = _dim(case), _sites(case)
    if kind == "hv":
        c = 2 if case["form"] == "complex" else 1
        return dict(bytes=dim * (16 * c + 8), flops=c * _hv_flops(case))
    if kind in ("solve", "batch"):
        # one expansion to ncv vectors: a product and two passes over the basis per step; the vectors out
        count = case.get("count", 1)
        ncv = case.get("ncv") or max(2 * case["nev"], case["nev"] + 15)
        return dict(bytes=count * dim * (24 * ncv + 8 * ncv * (ncv + 1) + 16 * case["nev"]),
                    flops=count * (ncv * _hv_flops(case) + 2.0 * dim * ncv * (ncv + 1)))
    if kind == "pairs":
        c = 1 if case["values"] == "real" else 2
        return dict(bytes=16 * dim, flops=c * dim * n * (n - 1) / 2)
    if kind == "dsf":
        more = 0 if case["op"] == "Sqz" else 1
        return dict(bytes=16 * (dim + case["nev"] * _dim(case, more)), flops=2.0 * dim * n * case["nev"])
    flops = 2.0 * dim * sum(_bond_counts(dict(case, j2=1.0)))
    return dict(bytes=16 * dim * (1 if kind == "egrad" else 2), flops=flops)


# --------------------------------------------------------------------------
# the same results in plain FP64
# --------------------------------------------------------------------------
_HALF = 15


class _Sector:
    """States of one sector in ascending order, and the rank of a state."""

    def __init__(self, n, up):
        self.n, self.up = n, up
        low = np.arange(1 << _HALF, dtype=np.int64)
        pop = np.zeros(1 << _HALF, dtype=np.int64)
        for b in range(_HALF):
            pop += (low >> b) & 1
        within = np.zeros(1 << _HALF, dtype=np.int64)  # position among the low parts of equal popcount
        groups = {}
        for k in range(_HALF + 1):
            groups[k] = low[pop == k]
            within[groups[k]] = np.arange(len(groups[k]))
        if n <= _HALF:
            self.states = torch.from_numpy(groups[up][groups[up] < (1 << n)]).cuda()
            start = np.zeros(1, dtype=np.int64)
        else:
            high = np.arange(1 << (n - _HALF), dtype=np.int64)
            k = up - pop[high]
            size = np.array([math.comb(_HALF, int(v)) if 0 <= v <= _HALF else 0 for v in k], dtype=np.int64)
            start = np.concatenate([[0], np.cumsum(size)[:-1]])
            self.states = torch.empty(int(size.sum()), dtype=torch.int64, device="cuda")
            dev = {k: torch.from_numpy(v).cuda() for k, v in groups.items()}
            for c1 in high[size > 0]:
                s = int(start[c1])
                self.states[s:s + int(size[c1])] = dev[int(k[c1])] + (int(c1) << _HALF)
        self.within = torch.from_numpy(within).cuda()
        self.start = torch.from_numpy(start).cuda()

    def rank(self, s):
        return self.start[s >> _HALF] + self.within[s & ((1 << _HALF) - 1)]

    def bit(self, i):
        return (self.states >> i) & 1


def _bond_lists(case):
    """Nearest and next-nearest neighbour bonds of the periodic lattices."""
    lx, ly = case["lx"], case["ly"]
    n = lx * ly
    if case["lattice"] == "chain":
        return [(i, (i + 1) % n) for i in range(n)], [(i, (i + 2) % n) for i in range(n)]

    def at(x, y):
        return (x % lx) * ly + y % ly

    nn, nnn = [], []
    for x in range(lx):
        for y in range(ly):
            c = at(x, y)
            nn.append((c, at(x, y + 1)))
            if case["lattice"] == "square" or c % 2 == x % 2:
                nn.append((c, at(x + 1, y)))
            if case["lattice"] == "honeycomb":
                nnn.append((c, at(x, y + 2)))
            nnn += [(c, at(x + 1, y + 1)), (c, at(x + 1, y - 1))]
    return nn, nnn


def _exact_hv(case, state):
    sec = _Sector(_sites(case), _sites(case) // 2 + case["sz"])
    x = state["x"]
    y = torch.zeros_like(x)
    diag = torch.zeros(len(sec.states), dtype=torch.float64, device="cuda")
    nn, nnn = _bond_lists(case)
    for bonds, j in ((nn, 1.0), (nnn, case["j2"])):
        if j == 0.0:
            continue
        for a, b in bonds:
            m = (1 << a) | (1 << b)
            if a == b:
                diag += 0.25 * j
                continue
            anti = (sec.bit(a) ^ sec.bit(b)).bool()
            diag += 0.25 * j - 0.5 * j * anti.double()
            at = torch.nonzero(anti).squeeze(1)
            y[at] += 0.5 * j * x[sec.rank(sec.states[at] ^ m)]
    for i, h in enumerate(_fields(case, state["seed"])):
        diag += (sec.bit(i).double() - 0.5) * float(h)
    y += diag * x
    if case["form"] == "real_dot":
        return y, float(torch.dot(x, y)), float(torch.dot(y, y))
    return y


def _flip_sum(sec, psi, a, b):
    """sum over the states with a up and b down of conj(psi(flipped)) psi."""
    at = torch.nonzero((sec.bit(a) == 1) & (sec.bit(b) == 0)).squeeze(1)
    return complex((psi[at] * psi[sec.rank(sec.states[at] ^ ((1 << a) | (1 << b)))].conj()).sum())


def _exact_pairs(case, state):
    n, psi, op = _sites(case), state["psi"], case["op"]
    sec = _Sector(n, n // 2 + case["sz"])
    w = psi.abs() ** 2
    total = float(w.sum())
    out = np.zeros((n, n), dtype=np.complex128)
    for a in range(n):
        up = float((w * sec.bit(a)).sum())
        out[a, a] = {"SzSz": 0.25 * total, "SiSj": 0.75 * total, "SpSm": up, "SmSp": total - up}[op]
        for b in range(a + 1, n):
            v = 0.0
            if op in ("SzSz", "SiSj"):
                anti = float((w * (sec.bit(a) ^ sec.bit(b))).sum())
                v = 0.25 * (total - 2.0 * anti)
            if op != "SzSz":
                f = _flip_sum(sec, psi, a, b)
                v += {"SiSj": f.real, "SpSm": f.conjugate(), "SmSp": f}[op]
            out[a, b], out[b, a] = v, np.conj(v)
    return out


def _exact_dsf(case, state):
    n, psi, vecs = _sites(case), state["psi"], state["vecs"]
    sec = _Sector(n, n // 2 + case["sz"])
    out = np.zeros((n, case["nev"]), dtype=np.complex128)
    target = sec if case["op"] == "Sqz" else _Sector(n, n // 2 + case["sz"] + 1)
    for i in range(n):
        if case["op"] == "Sqz":
            out[i] = ((sec.bit(i).double() - 0.5) * psi * vecs.conj()).sum(dim=1).cpu().numpy()
        else:
            at = torch.nonzero(sec.bit(i) == 0).squeeze(1)
            to = target.rank(sec.states[at] | (1 << i))
            out[i] = (psi[at] * vecs[:, to].conj()).sum(dim=1).cpu().numpy()
    return out


def _exact_egrad(case, state):
    n, psi = _sites(case), state["psi"]
    sec = _Sector(n, n // 2 + case["sz"])
    w = psi.abs() ** 2
    total = float(w.sum())
    dj, dd = [], []
    for bonds in _bond_lists(case):
        for a, b in bonds:
            dj.append(0.5 if a == b else _flip_sum(sec, psi, a, b).real / total)
            dd.append(0.25 * (1.0 - 2.0 * float((w * (sec.bit(a) ^ sec.bit(b))).sum()) / total))
    dh = [float((w * (sec.bit(i).double() - 0.5)).sum()) / total for i in range(n)]
    return np.array(dj), np.array(dd), np.array(dh)


def _exact_mixed(case, state):
    n, psi, lam = _sites(case), state["psi"], state["lam"].conj()
    sec = _Sector(n, n // 2 + case["sz"])
    out = []
    for kind, a, b in state["terms"]:
        if kind == ed.Adjoint.Z:
            out.append(complex((lam * psi * (sec.bit(a).double() - 0.5)).sum()))
            continue
        anti = (sec.bit(a) ^ sec.bit(b)).double()
        if kind == ed.Adjoint.ZZ:
            out.append(complex((lam * psi * (0.25 - 0.5 * anti)).sum()))
        elif a == b:
            out.append(0.5 * complex((lam * psi).sum()))
        else:
            at = torch.nonzero(anti).squeeze(1)
            out.append(0.5 * complex((lam[at] * psi[sec.rank(sec.states[at] ^ ((1 << a) | (1 << b)))]).sum()))
    return np.array(out)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "batch"):
        return None
    state = prepare(case, seed)
    state["seed"] = seed
    if kind == "dots":
        return np.array([float(torch.dot(v, state["w"])) for v in state["V"]])
    if kind == "combine":
        out = []
        for c in range(case["keep"]):
            y = torch.zeros_like(state["V"][0])
            for v, f in zip(state["V"], state["Y"][:, c]):
                y += v * float(f)
            out.append(y)
        return out
    return {"hv": _exact_hv, "pairs": _exact_pairs, "dsf": _exact_dsf, "egrad": _exact_egrad,
            "mixed": _exact_mixed}[kind](case, state)
