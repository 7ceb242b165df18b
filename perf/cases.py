"""The work that users of this framework have it do, as timed cases.

A case is one call (or one short chain of calls) through the package's public
entry points: products H * psi, ground states, all momentum sectors or a
disorder ensemble in one batch, quenches, block Lanczos and entanglement
spectra.  ``listed()`` holds the named cases, ``draw()`` makes more of the same
ranges, ``prepare()`` builds what a program has in hand before the call (basis,
operator, start vectors), ``run()`` is one pass, ``work()`` what the pass
cannot do without and ``exact()`` its result in plain 64-bit torch.
"""
import math

import numpy as np
import torch

from __graft_entry__ import load_package

ek = load_package()
DEV = "cuda" if torch.cuda.is_available() else "cpu"
DTYPES = {"f64": torch.float64, "c128": torch.complex128, "f32": torch.float32,
          "c64": torch.complex64}


def _case(name, kind, basis, L, **kw):
    case = {"name": name, "kind": kind, "basis": basis, "L": L}
    case.update(kw)
    return case


def listed():
    return [
        # the smallest products (interactive work, small-system checks): one
        # complex vector on the full space of ten sites
        _case("product_small", "product", "tensor", 10, model="xxz", dtype="c128", nvec=1),
        # transverse-field Ising on the full space: operators that are not
        # charge-conserving flip-flops
        _case("product_ising", "product", "tensor", 20, model="ising", dtype="f64", nvec=1),
        # the framework's headline: half filling, zero momentum, real vector,
        # rank search as its benchmark sets it
        _case("product_momentum", "product", "momentum", 28, N=14, k=0, model="xxz",
              dtype="f64", nvec=1, search="rank"),
        # an odd chain off half filling at a complex momentum, everything else
        # left at its default
        _case("product_momentum_odd", "product", "momentum", 25, N=11, k=7, model="xxz",
              dtype="c128", nvec=1, search="hash"),
        # basis(k, p, z): the symmetry-group sectors of level statistics
        _case("product_group", "product", "group", 22, N=11, k=0, p=1, z=1, model="xxz",
              dtype="f64", nvec=1),
        # random fields (many-body localisation), a ragged block of single
        # precision columns
        _case("product_block", "product", "charge", 18, N=9, model="fields", dtype="f32",
              nvec=13),
        # ground state and its vector, double precision
        _case("ground_state", "ground", "momentum", 26, N=13, k=0, model="xxz", search="rank"),
        # the lowest levels of all momentum sectors of one chain, one mixed
        # precision batch
        _case("sectors_mixed", "sectors", "momentum", 22, N=11, model="xxz", nev=4,
              precision="mixed"),
        # a disorder ensemble of uneven chains, one batch
        _case("ensemble", "ensemble", "charge", 20, instances=96, model="fields", nev=1,
              precision="fp64"),
        # a quench from a product state, every state kept on the GPU
        _case("quench", "quench", "momentum", 26, N=13, k=0, model="j1j2", search="rank",
              times=101, dt=0.1),
        # block Lanczos over the momentum sectors
        _case("block_lanczos", "block", "momentum", 18, N=9, model="xxz", block=16, steps=60,
              nev=4),
        # entanglement spectrum of a sector vector across half the chain
        _case("entanglement", "entropy", "momentum", 20, N=10, k=0, cut=10, dtype="f64"),
    ]


def draw(rng):
    kind = rng.choice(["product"] * 5 + ["ground", "sectors", "ensemble", "quench", "block",
                                         "entropy"])
    if kind == "product":
        return _draw_product(rng)
    if kind == "ground":
        L = rng.randint(14, 26)
        return {"kind": kind, "basis": "momentum", "L": L, "N": L // 2 - rng.choice([0, 0, 1]),
                "k": 0, "model": rng.choice(["xxz", "j1j2"]),
                "search": rng.choice(["hash", "rank"])}
    if kind == "sectors":
        L = rng.randint(12, 21)
        return {"kind": kind, "basis": "momentum", "L": L, "N": L // 2, "model": "xxz",
                "nev": rng.randint(1, 4), "precision": rng.choice(["fp64", "mixed"])}
    if kind == "ensemble":
        return {"kind": kind, "basis": "charge", "L": rng.choice([12, 14, 16, 18]),
                "instances": rng.randint(4, 96), "model": "fields", "nev": rng.choice([1, 4]),
                "precision": rng.choice(["fp64", "mixed"])}
    if kind == "quench":
        L = rng.randint(14, 24)
        return {"kind": kind, "basis": "momentum", "L": L, "N": L // 2, "k": 0,
                "model": rng.choice(["xxz", "j1j2"]), "search": rng.choice(["hash", "rank"]),
                "times": rng.randint(2, 101), "dt": rng.choice([0.05, 0.1, 0.25])}
    if kind == "block":
        L = rng.randint(16, 18)
        return {"kind": kind, "basis": "momentum", "L": L, "N": L // 2, "model": "xxz",
                "block": rng.choice([8, 16]), "steps": rng.randint(30, 45),
                "nev": rng.randint(1, 4)}
    L = rng.randint(12, 20)
    return {"kind": kind, "basis": "momentum", "L": L, "N": L // 2, "k": 0,
            "cut": rng.randint(L // 2 - 2, L // 2), "dtype": rng.choice(["f64", "c128"])}


def _draw_product(rng):
    basis = rng.choice(["tensor", "charge", "momentum", "momentum", "group"])
    real = rng.choice(["f64", "f64", "f32"])
    case = {"kind": "product", "basis": basis}
    if basis == "tensor":
        case.update(L=rng.randint(8, 20), model=rng.choice(["xxz", "ising"]))
    elif basis == "charge":
        L = rng.randint(10, 22)
        case.update(L=L, N=L // 2 - rng.choice([0, 0, 1, 2]), model="fields")
    elif basis == "momentum":
        L = rng.randint(14, 28)
        k = rng.choice([0, rng.randint(1, L - 1)])
        search = rng.choice(["hash", "rank"])
        case.update(L=L, N=L // 2 - rng.choice([0, 1, 2]), k=k,
                    model=rng.choice(["xxz", "j1j2"]), search=search)
        if k and 2 * k != L:
            real = {"f64": "c128", "f32": "c64"}[real]
    else:
        L = 2 * rng.randint(6, 12)
        case.update(L=L, N=L // 2, k=0, p=rng.choice([1, -1]), z=rng.choice([1, -1]),
                    model="xxz")
    case["dtype"] = real if rng.random() < 0.6 else {"f64": "c128", "f32": "c64"}.get(real, real)
    case["nvec"] = rng.choice([1, 1, 1, 2, 5, 16, 33]) if case["L"] <= 22 else 1
    if rng.random() < 0.2 and case["L"] <= 24:
        case["sparse"] = True  # the program called sparse!() on the operator
    return case


# ---------------------------------------------------------------------------
# what a program has in hand before the call
# ---------------------------------------------------------------------------
def _basis(case, L=None, k=None):
    L = case["L"] if L is None else L
    if case["basis"] == "tensor":
        return ek.TensorBasis(L=L)
    if case["basis"] == "charge":
        return ek.ProjectedBasis(L=L, N=case.get("N", L // 2))
    if case["basis"] == "group":
        return ek.basis(L=L, N=case["N"], k=case["k"], p=case["p"], z=case["z"])
    B = ek.TranslationalBasis(L=L, N=case["N"], k=case.get("k", 0) if k is None else k)
    if case.get("search", "rank") == "rank":
        B.set_search("rank")
    return B


def _fields(seed, L, q=0):
    return np.random.default_rng([seed, q, L]).uniform(-3.0, 3.0, L)


def _operator(case, B, seed, q=0):
    L, model = B.L, case["model"]
    bond = ek.spin((1.0, "xx"), (1.0, "yy"), (1.0, "zz"))
    open_bonds = [[i, i + 1] for i in range(1, L)]
    sites = [[i] for i in range(1, L + 1)]
    if model == "ising":
        return ek.operator([-ek.spin("zz")] * (L - 1) + [-0.8 * ek.spin("x")] * L,
                           open_bonds + sites, B)
    if model == "fields":
        h = _fields(seed, L, q)
        return ek.operator([bond] * (L - 1) + [v * ek.spin("z") for v in h],
                           open_bonds + sites, B)
    if case["basis"] == "tensor":
        return ek.operator([bond] * (L - 1), open_bonds, B)
    H = ek.trans_inv_operator(bond, 2, B)
    if model == "j1j2":
        H = H + ek.trans_inv_operator(0.5 * bond, [1, 3], B)
    return H


def _columns(case, D, seed):
    """nvec normalised columns (a column-major block), or one vector."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    nvec = case.get("nvec", 1)
    x = torch.randn((nvec, D), dtype=DTYPES[case["dtype"]], device=DEV, generator=g)
    x /= torch.linalg.vector_norm(x, dim=1, keepdim=True)
    return x[0] if nvec == 1 else x.t()


def _digits(case, seed):
    dg = np.zeros(case["L"], dtype=np.int64)
    up = np.random.default_rng(seed).permutation(case["L"])[: case["L"] - case["N"]]
    dg[up] = 1
    return dg


def _lengths(case, seed):
    """Chain lengths of the ensemble: even, spread below the longest."""
    top = case["L"]
    some = np.random.default_rng(seed).integers(0, 5, case["instances"])
    return [max(12, top - 2 * int(v)) for v in some]


def _start(seed, D, q=0):
    return np.random.default_rng([seed, q]).standard_normal(D)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("product", "entropy"):
        B = _basis(case)
        state = {"case": case, "B": B, "x": _columns(case, B.size(1), seed)}
        if kind == "product":
            state["H"] = _operator(case, B, seed)
            if case.get("sparse"):
                state["H"].sparse_()
        return state
    if kind in ("ground", "quench"):
        B = _basis(case)
        state = {"case": case, "H": _operator(case, B, seed)}
        if kind == "ground":
            state["v0"] = _start(seed, B.size(1))
        else:
            psi = ek.productstate(_digits(case, seed), B)
            state["psi"] = torch.from_numpy(psi).to(DEV, torch.complex128)
            state["ts"] = np.arange(case["times"]) * case["dt"]
        return state
    if kind == "ensemble":
        lengths = _lengths(case, seed)
        bases = {L: _basis(case, L=L) for L in sorted(set(lengths))}
        ops = [_operator(case, bases[L], seed, q) for q, L in enumerate(lengths)]
    else:
        ops = [_operator(case, _basis(case, k=k), seed) for k in range(case["L"])]
    state = {"case": case, "ops": ops}
    if kind == "block":
        state["seed"] = seed
    else:
        state["v0s"] = [_start(seed, op.size(1), q) for q, op in enumerate(ops)]
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "product":
        return state["H"] * state["x"]
    if kind == "ground":
        E0, psi, _ = ek.ground_state(state["H"], state["v0"])
        return {"E0": E0, "psi": psi}
    if kind == "quench":
        return ek.timeevolve(state["H"], state["psi"], state["ts"])
    if kind == "block":
        return ek.block_lanczos(state["ops"], block=case["block"], m=case["steps"],
                                nev=case["nev"], seed=state["seed"])[0]
    if kind == "entropy":
        return ek.ent_spec(state["x"], list(range(1, case["cut"] + 1)), state["B"])
    return ek.batch_lanczos_e0(state["ops"], state["v0s"], m=200, nev=case["nev"], tol=1e-12,
                               precision=case["precision"])[0]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _dim(case, L=None, N=None):
    """States of the sector (of one momentum sector: an average)."""
    L = case["L"] if L is None else L
    N = case.get("N", L // 2) if N is None else N
    D = {"tensor": 2.0 ** L, "charge": float(math.comb(L, N))}.get(case["basis"])
    if D is None:
        D = math.comb(L, N) / L / (4 if case["basis"] == "group" else 1)
    return max(1.0, D)


def _hits(case, L=None):
    """Off-diagonal entries per row."""
    L = case["L"] if L is None else L
    if case["model"] == "ising":
        return float(L)
    anti = 0.5 if case["basis"] == "tensor" else \
        2.0 * case.get("N", L // 2) * (L - case.get("N", L // 2)) / (L * (L - 1))
    return (2 if case["model"] == "j1j2" else 1) * L * anti


def work(case):
    kind, D = case["kind"], _dim(case)
    cx = 16.0 if case.get("dtype") in ("c128", "c64") or case.get("k", 0) else 8.0
    # the state list and the norms of a sector are read by every product
    table = {"tensor": 0.0, "charge": 8.0}.get(case["basis"], 16.0)
    if kind == "product":
        s = {"f64": 8, "c128": 16, "f32": 4, "c64": 8}[case["dtype"]]
        n = case["nvec"]
        return {"bytes": D * (2 * s * n + table), "flops": 2.0 * D * (_hits(case) + 1) * n * (cx / 8)}
    if kind == "entropy":
        a, b = 2.0 ** case["cut"], 2.0 ** (case["L"] - case["cut"])
        lo, hi = min(a, b), max(a, b)
        return {"bytes": D * (table + cx) + a * b * cx,
                "flops": (2.0 * lo * lo * hi + 4.0 / 3.0 * lo ** 3) * (cx / 8)}
    if kind == "quench":
        # per 1.2 time units one basis of 40 vectors: two reads of what is
        # there per new vector, one read for the states served, the states out
        spans = max(1.0, math.ceil(case["times"] * case["dt"] / 1.2))
        m = 40
        return {"bytes": 16.0 * D * (spans * (m * m + m) + case["times"]) + spans * m * D * table,
                "flops": 8.0 * D * (spans * (2 * m * m + m * _hits(case)) + m * case["times"])}
    if kind == "block":
        p, m, D = case["block"], case["steps"], D * case["L"]
        return {"bytes": 16.0 * D * p * m * 6, "flops": m * (32.0 * p * p * D + 8 * p * D * _hits(case))}
    # Lanczos with full reorthogonalisation: two reads of the basis per step
    m = {"ground": 60, "sectors": 90, "ensemble": 90}[kind]
    rows = [(D, _hits(case))]
    if kind == "sectors":
        rows = rows * case["L"]
    elif kind == "ensemble":
        tops = [max(12, case["L"] - 2 * v) for v in range(5)]
        rows = [(_dim(case, L, L // 2) * case["instances"] / 5, _hits(case, L)) for L in tops]
    s = 16.0 if kind == "sectors" else 8.0
    s /= 2 if case.get("precision") == "mixed" else 1
    return {"bytes": sum(d * (s * m * m + m * (3 * s + table)) for d, _ in rows),
            "flops": sum(d * (4.0 * m * m + 2 * m * h) for d, h in rows) * (4 if kind == "sectors" else 1)}


# ---------------------------------------------------------------------------
# the same results in plain 64-bit torch
# ---------------------------------------------------------------------------
def _popcount(s):
    c = torch.zeros_like(s)
    for b in range(32):
        c += (s >> b) & 1
    return c


class _Reference:
    """A sector's states, and H as one target row and one value per bond and
    row, from the group elements alone."""

    def __init__(self, case, seed, L=None, k=None, q=0):
        L = case["L"] if L is None else L
        k = case.get("k", 0) if k is None else k
        self.L, full = L, (1 << L) - 1
        rot = lambda s, r: ((s << r) | (s >> (L - r))) & full  # noqa: E731

        def rev(s):
            o = torch.zeros_like(s)
            for b in range(L):
                o |= ((s >> b) & 1) << (L - 1 - b)
            return o

        group = [(lambda s: s, 1.0)]  # (action, amplitude of the image)
        if case["basis"] in ("momentum", "group"):
            group = []
            for r in range(L):
                ph = complex(math.cos(2 * math.pi * k * r / L), -math.sin(2 * math.pi * k * r / L))
                ph = ph.real if (2 * k) % L == 0 else ph
                group.append((lambda s, r=r: rot(s, r), ph))
        if case["basis"] == "group":
            p, z = case["p"], case["z"]
            group = [e for a, c in group for e in (
                (a, c), (lambda s, a=a: a(rev(s)), c * p), (lambda s, a=a: a(s) ^ full, c * z),
                (lambda s, a=a: a(rev(s)) ^ full, c * p * z))]
        self.cx = any(isinstance(c, complex) for _, c in group)
        amp_t = torch.complex128 if self.cx else torch.float64
        reps = []
        for s0 in range(0, 1 << L, 1 << 24):
            s = torch.arange(s0, min(1 << L, s0 + (1 << 24)), device=DEV)
            if case["basis"] != "tensor":
                ones = L - case.get("N", L // 2)
                s = s[_popcount(s) == ones]
            keep = torch.ones_like(s, dtype=torch.bool)
            for act, _ in group:
                keep &= act(s) >= s
            reps.append(s[keep])
        s = torch.cat(reps)
        fixed = torch.zeros(len(s), dtype=amp_t, device=DEV)
        for act, c in group:
            fixed += c * (act(s) == s)
        s = s[fixed.abs() > 0.5]
        self.reps, self.D = s, len(s)
        self.idx = torch.full((1 << L,), -1, dtype=torch.int32, device=DEV)
        self.amp = torch.zeros(1 << L, dtype=amp_t, device=DEV)
        row = torch.arange(self.D, device=DEV, dtype=torch.int32)
        orbit = torch.zeros(self.D, device=DEV, dtype=torch.float64)
        for act, c in group:
            orbit += act(s) == s
        orbit = len(group) / orbit  # images of each representative
        for act, c in reversed(group):
            self.idx[act(s)] = row
            self.amp[act(s)] = (c / orbit.sqrt()).to(amp_t)
        if "model" in case:
            self._terms(case, seed, q)

    def _terms(self, case, seed, q):
        L, s, model = self.L, self.reps, case["model"]
        bit = lambda i: (s >> (L - 1 - i % L)) & 1  # noqa: E731  (site i = 0 .. L-1)
        mask = lambda i: 1 << (L - 1 - i % L)  # noqa: E731
        closed = case["basis"] in ("momentum", "group")
        bonds = [(i, i + 1, 1.0) for i in range(L if closed else L - 1)]
        if model == "j1j2":
            bonds += [(i, i + 2, 0.5) for i in range(L)]
        self.diag = torch.zeros(self.D, dtype=torch.float64, device=DEV)
        cols, vals = [], []

        def hit(target, weight):
            t = self.idx[target].long()
            v = torch.where(t >= 0, weight, torch.zeros_like(weight)) * self.amp[target] / \
                self.amp[s]
            cols.append(t.clamp(min=0))
            vals.append(v)

        for i, j, w in bonds:
            anti = bit(i) != bit(j)
            w = -w if model == "ising" else w
            self.diag += w * (0.25 - 0.5 * anti.double())
            if model != "ising":
                hit(torch.where(anti, s ^ (mask(i) | mask(j)), s), 0.5 * w * anti.double())
        if model == "ising":
            for i in range(L):
                hit(s ^ mask(i), torch.full((self.D,), -0.4, dtype=torch.float64, device=DEV))
        if model == "fields":
            for i, h in enumerate(_fields(seed, L, q)):
                self.diag += float(h) * (0.5 - bit(i).double())
        self.cols, self.vals = torch.stack(cols), torch.stack(vals)

    def mul(self, x):
        return self.diag * x + (self.vals * x[self.cols]).sum(0)

    def krylov(self, v, steps, stop=None):
        """Orthonormal Krylov rows, alpha, beta; `stop(a, b)` ends it early."""
        V = torch.zeros((steps + 1, self.D), dtype=v.dtype, device=DEV)
        V[0] = v / torch.linalg.vector_norm(v)
        a, b = [], []
        for j in range(steps):
            w = self.mul(V[j])
            c = V[: j + 1].conj() @ w
            a.append(float(c[j].real))
            w = w - V[: j + 1].T @ c
            w = w - V[: j + 1].T @ (V[: j + 1].conj() @ w)
            b.append(float(torch.linalg.vector_norm(w)))
            if b[-1] < 1e-12 or (stop is not None and j % 10 == 9 and stop(a, b)):
                break
            V[j + 1] = w / b[-1]
        return V[: len(a)], np.array(a), np.array(b)

    def lowest(self, nev, seed):
        seen = [np.full(nev, np.inf)]

        def stop(a, b):
            w = np.linalg.eigvalsh(_tridiagonal(a, b))[:nev]
            done = len(w) == nev and np.all(np.abs(w - seen[0][: len(w)]) <= 1e-14 * np.abs(w))
            if len(w) == nev:
                seen[0] = w
            return done

        g = torch.Generator(device=DEV).manual_seed(seed + 1)
        v = torch.randn(self.D, dtype=self.amp.dtype, device=DEV, generator=g)
        _, a, b = self.krylov(v, min(self.D, 400), stop)
        w = np.linalg.eigvalsh(_tridiagonal(a, b))[:nev]
        return np.concatenate([w, np.full(nev - len(w), np.nan)])


def _tridiagonal(a, b):
    b = np.asarray(b)[: len(a) - 1]
    return np.diag(a) + np.diag(b, 1) + np.diag(b, -1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "product":
        ref = _Reference(case, seed)
        x = _columns(case, ref.D, seed)
        x = x.to(torch.complex128 if x.is_complex() else torch.float64)
        return ref.mul(x) if x.ndim == 1 else \
            torch.stack([ref.mul(x[:, c]) for c in range(x.shape[1])], dim=1)
    if kind == "ground":
        # the vector is as converged as the energy's stop rule leaves it
        return {"E0": float(_Reference(case, seed).lowest(1, seed)[0]), "psi": None}
    if kind == "quench":
        ref = _Reference(case, seed)
        start = int("".join(str(v) for v in _digits(case, seed)), 2)
        v = torch.zeros(ref.D, dtype=torch.complex128, device=DEV)
        v[ref.idx[start].long()] = 1.0
        out = [v]
        for _ in range(case["times"] - 1):
            V, a, b = ref.krylov(v, min(ref.D, 20))
            w, Q = np.linalg.eigh(_tridiagonal(a, b))
            c = Q @ (np.exp(-1j * case["dt"] * w) * Q[0]) * float(torch.linalg.vector_norm(v))
            v = V.T @ torch.from_numpy(c).to(DEV)
            out.append(v)
        return torch.stack(out, dim=1)
    if kind == "entropy":
        ref = _Reference(case, seed)
        x = _columns(case, ref.D, seed)
        full = torch.where(ref.idx >= 0, ref.amp * x[ref.idx.long().clamp(min=0)], 0)
        return torch.linalg.svdvals(full.reshape(2 ** case["cut"], -1).cpu()).numpy()
    if kind == "ensemble":
        lengths = _lengths(case, seed)
        if sum(math.comb(L, L // 2) for L in lengths) > 6_000_000:
            return None
        return np.stack([_Reference(case, seed, L=L, q=q).lowest(case["nev"], seed)
                         for q, L in enumerate(lengths)])
    return np.stack([_Reference(case, seed, k=k).lowest(case["nev"], seed)
                     for k in range(case["L"])])
