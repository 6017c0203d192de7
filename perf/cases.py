"""What a user of this framework has it do, as cases that can be timed and checked.

A case names an operation, a periodic torus with its couplings, a sector
(Sz, kx, ky) and a precision.  The operations are the framework's public entry
points, as a program calls them:

  hv       w = H v on device vectors (GpuSector.hv), with the rows stored in
           HBM and perhaps tuned, or matrix-free: the step of every Krylov method
  host     the drop-in call on host arrays (GpuSector.sHv)
  block    H on 2 or 4 vectors at once (GpuSector.hv_block)
  first    a new sector up to its first H v: basis, stored rows, one hv (what a
           request of the serving loop pays before its first step)
  dense    solve_plain below its dense threshold: the full spectrum in FP64
  plain    solve_plain: the reference's FP64 Lanczos with its defaults
  mixed    solve_mixed with partial reorthogonalisation
  batch    many small sectors' solves together (BatchSolver)

Couplings of the sectors that are solved or built are drawn from the seed, as
are all vectors, so every seed is another Hamiltonian or another vector.
exact() states the same quantities in 64 bits with torch alone.
"""
import math

import numpy as np
import torch

from ed_code_gb300 import lattice as L
from ed_code_gb300.batch import BatchSolver
from ed_code_gb300.sector import GpuSector


def _case(name, op, lattice, Lx, Ly, k=(0, 0), Sz=0, Jz=1.0, J2=0.0, Ch=0.0, dtype="c128", **more):
    return {"name": name, "op": op, "lattice": lattice, "Lx": Lx, "Ly": Ly, "kx": k[0], "ky": k[1], "Sz": Sz,
            "Jz": Jz, "J2": J2, "Ch": Ch, "dtype": dtype, **more}


def listed():
    return [
        # The smallest real sector (4x4 Heisenberg, 822 states): what one H v costs when only latency counts.
        _case("hv_16_f64", "hv", "square", 4, 4, stored=True, tuned=False),
        # A sector used without stored rows (a single H v, an observable, rows that do not fit), FP64, chirality.
        _case("hv_28_free_f64", "hv", "triangular", 7, 4, (1, 2), Jz=0.8, Ch=0.2, stored=False, tuned=False),
        # Stored rows in FP64 at a general momentum with chirality: the plain form's H v and the Rayleigh quotients'.
        _case("hv_28_f64", "hv", "triangular", 7, 4, (1, 2), Jz=0.8, Ch=0.2, stored=True, tuned=False),
        # One sector of the precision benchmark, FP32 vectors, tuned: the H v of the mixed solver.
        _case("hv_30_f32", "hv", "triangular", 6, 5, (2, 3), Jz=0.8, Ch=0.2, dtype="c64", stored=True, tuned=True),
        # The headline sector: 36 sites, 2.5e8 states, FP32 vectors, tuned.
        _case("hv_36_f32", "hv", "triangular", 6, 6, Ch=0.15, dtype="c64", stored=True, tuned=True),
        # The reference's own call on host arrays in FP64: vectors go in and come back.
        _case("host_24_f64", "host", "square", 6, 4, J2=0.3, stored=True, tuned=False),
        # Four vectors at once on a serving-size sector with one up spin more (Sz = 1), FP32.
        _case("block4_32_f32", "block", "square", 8, 4, (0, 2), Sz=1, Jz=1.2, dtype="c64", nv=4, tuned=True),
        # A new 32-site sector up to its first H v: the construction that each large request pays.
        _case("first_32_f32", "first", "triangular", 8, 4, (3, 1), Jz=1.1, Ch=0.1, dtype="c64"),
        # The full spectrum of a small sector (2,700 states).
        _case("dense_18", "dense", "triangular", 6, 3, (1, 1), Jz=0.9, Ch=0.2),
        # The reference's Lanczos in FP64 with its defaults (112,750 states, two levels).
        _case("plain_24", "plain", "triangular", 6, 4, (1, 0), Jz=0.9, Ch=0.1, n_ev=2),
        # The mixed-precision solver, four levels of a 1.4-million-state sector.
        _case("mixed_28", "mixed", "square", 7, 4, (2, 1), Jz=1.1, n_ev=4, iterations=300),
        # Eight random Hamiltonians, every momentum at Sz = 0, three levels each: the batched small sectors.
        _case("batch_20", "batch", "triangular", 5, 4, Jz=1.0, J2=0.2, Ch=0.2, n_ev=3, iterations=150, models=8),
    ]


_TORI = [(4, 3), (4, 4), (6, 3), (5, 4), (6, 4), (8, 3), (9, 3), (7, 4), (6, 5), (10, 3), (8, 4)]


def draw(rng):
    """One more case: any operation on any torus of its range (odd row lengths
    and column counts among them), any momentum, couplings and precision."""
    op = rng.choice(["hv", "hv", "hv", "host", "block", "first", "dense", "plain", "mixed", "batch"])
    lo, hi = {"hv": (12, 32), "host": (12, 28), "block": (16, 32), "first": (16, 32), "dense": (12, 18),
              "plain": (16, 24), "mixed": (18, 28), "batch": (16, 20)}[op]
    Lx, Ly = rng.choice([t for t in _TORI if lo <= t[0] * t[1] <= hi and t[0] * t[1] % 2 == 0])
    lattice = rng.choice(["square", "triangular"])
    j2 = round(rng.uniform(0.05, 0.5), 3) if Lx >= 4 and Ly >= 4 and rng.random() < 0.4 else 0.0
    ch = round(rng.uniform(0.05, 0.4), 3) if lattice == "triangular" and rng.random() < 0.6 else 0.0
    k = (0, 0) if rng.random() < 0.3 else (rng.randrange(Lx), rng.randrange(Ly))
    c = _case(None, op, lattice, Lx, Ly, k, rng.choice([0, 0, 1]), round(rng.uniform(0.5, 1.5), 3), j2, ch,
              rng.choice(["c64", "c128"]))
    del c["name"]
    if op == "hv":
        c.update(stored=rng.random() < 0.75, tuned=rng.random() < 0.5)
    elif op == "host":
        c.update(stored=rng.random() < 0.75, tuned=False)
    elif op == "block":
        c.update(nv=rng.choice([2, 4]), tuned=rng.random() < 0.5)
    elif op in ("dense", "plain", "mixed", "batch"):
        c.update(dtype="c128")
        if op == "plain":
            c.update(n_ev=rng.choice([1, 2]))
        elif op == "mixed":
            c.update(n_ev=rng.choice([1, 2, 4]))
            c.update(iterations=300 if c["n_ev"] > 2 else 200)
        elif op == "batch":
            c.update(n_ev=rng.choice([1, 3]), iterations=150, models=rng.choice([1, 2, 4]))
    return c


def _couplings(case, seed):
    """The couplings of one Hamiltonian: the case's own where a vector is the
    input, drawn around them where the Hamiltonian is."""
    if case["op"] in ("hv", "host", "block"):
        return case["Jz"], case["J2"], case["Ch"]
    r = np.random.default_rng([seed, 7])
    return tuple(float(x * f) for x, f in zip((case["Jz"], case["J2"], case["Ch"]), r.uniform(0.8, 1.2, 3)))


def _model(case, seed, k=None):
    Jz, J2, Ch = _couplings(case, seed)
    spec = L.TorusSpec(case["lattice"], case["Lx"], case["Ly"], Jz=Jz, J2=J2, Ch=Ch)
    kx, ky = (case["kx"], case["ky"]) if k is None else k
    return L.make_model(spec, case["Sz"], kx, ky, bowties=False)


def _dtype(case):
    return torch.complex64 if case["dtype"] == "c64" else torch.complex128


def _vector(n, seed, nv=None):
    """A normalised complex Gaussian vector (or nv of them side by side): the
    start vector of a Krylov run, in 64 bits."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = (n,) if nv is None else (n, nv)
    v = torch.randn(shape, dtype=torch.complex64, device="cuda", generator=g)
    return v / math.sqrt(n)


def prepare(case, seed):
    op = case["op"]
    s = {"op": op}
    if op == "batch":
        s["sectors"] = []
        for q in range(case["models"]):
            for kx in range(case["Lx"]):
                for ky in range(case["Ly"]):
                    sec = GpuSector(_model(case, seed * 1000 + q, (kx, ky)))
                    sec.build_targets()
                    s["sectors"].append(sec)
        s.update(n_ev=case["n_ev"], iterations=case["iterations"], seed=seed)
        return s
    model = _model(case, seed)
    if op == "first":
        sec = GpuSector(model)
        s["model"] = model
        s["v"] = _vector(sec.n_p, seed).to(_dtype(case))
        s["w"] = torch.empty_like(s["v"])
        sec.close()
        return s
    sec = s["sec"] = GpuSector(model)
    if case.get("stored", True):
        sec.build_targets()
        if case.get("tuned"):
            sec.tune()
    if op in ("hv", "host", "block"):
        v = _vector(sec.n_p, seed, case.get("nv")).to(_dtype(case))
        if op == "host":
            s["v"] = v.cpu().numpy()
        else:
            s["v"], s["w"] = v, torch.empty_like(v)
    else:
        s.update({k: case[k] for k in ("n_ev", "iterations") if k in case}, seed=seed)
    return s


def run(s):
    op = s["op"]
    if op == "hv":
        s["sec"].hv(s["v"], s["w"])
        return s["w"]
    if op == "host":
        return s["sec"].sHv(s["v"], dtype=s["v"].dtype)
    if op == "block":
        s["sec"].hv_block(s["v"], s["w"], stream=torch.cuda.current_stream())
        return s["w"]
    if op == "first":
        sec = GpuSector(s["model"])
        sec.build_targets()
        sec.hv(s["v"], s["w"])
        sec.close()
        return s["w"]
    if op == "dense":
        return s["sec"].solve_plain()[0]
    if op == "plain":
        return list(s["sec"].solve_plain(n_ev=s["n_ev"], seed=s["seed"], dense_threshold=-1)[0])
    if op == "mixed":
        return s["sec"].solve_mixed(n_ev=s["n_ev"], iterations=s["iterations"], reorth_every=-1, seed=s["seed"])["eigs"]
    batch = BatchSolver(reorth=1)
    for q, sec in enumerate(s["sectors"]):
        batch.add(sec, n_ev=s["n_ev"], max_iterations=s["iterations"], tol=0.0, seed=s["seed"] + q, tag=q)
    out = np.full((len(s["sectors"]), s["n_ev"]), np.nan)
    for r in batch.run():
        out[r["tag"], : r["n_found"]] = r["eigs"]
    batch.close()
    return out


def _counts(case):
    """(states, flipped pairs, nonzeros) of the sector, to about a percent."""
    n = case["Lx"] * case["Ly"]
    up = n // 2 + case["Sz"]
    states = math.comb(n, up) / n
    bonds = n * ((2 if case["lattice"] == "square" else 3) + ((2 if case["lattice"] == "square" else 3) if case["J2"] else 0))
    return states, bonds, states * bonds * 2 * up * (n - up) / (n * (n - 1))


def work(case):
    """Bytes: vectors once in and once out, and a stored row's nonzeros as one
    32-bit word each.  Flops: 8 for each nonzero and vector.  The solvers take
    their steps' H v and the vectors that a step reads and writes."""
    op = case["op"]
    n, bonds, nnz = _counts(case)
    elem = 8 if case["dtype"] == "c64" else 16
    nv = case.get("nv", 1)
    rows = 4 * nnz if case.get("stored", True) else 8 * n
    if op in ("hv", "block", "host"):
        return {"bytes": rows + 2 * elem * n * nv, "flops": 8 * nnz * nv}
    if op == "first":  # the basis and the rows are written, then read once
        return {"bytes": 2 * (8 * n + 4 * nnz) + 2 * elem * n, "flops": 8 * nnz}
    if op == "dense":  # Householder reduction of a complex Hermitian matrix
        return {"bytes": 16 * n * n, "flops": 16 / 3 * n ** 3}
    steps = {"plain": 200 * case.get("n_ev", 1), "mixed": case.get("iterations", 0)}.get(op, 150)
    each = 8 if op != "plain" else 16
    many = case.get("models", 0) * case["Lx"] * case["Ly"] if op == "batch" else 1
    return {"bytes": many * steps * (4 * nnz + 8 * each * n), "flops": many * steps * 8 * (nnz + 6 * n)}


# ---- the same quantities in 64 bits, with torch alone -----------------------------------------

def _pairs(case):
    Lx, Ly = case["Lx"], case["Ly"]
    tri = case["lattice"] == "triangular"
    near = [(1, 0), (0, 1)] + ([(-1, 1)] if tri else [])
    far = [(1, 1), (-1, 2), (2, -1)] if tri else [(1, 1), (1, -1)]

    def site(x, y):
        return x % Lx + Lx * (y % Ly)

    def bonds(vectors):
        return [(site(x, y), site(x + dx, y + dy)) for y in range(Ly) for x in range(Lx) for dx, dy in vectors]

    triangles = []
    for y in range(Ly):
        for x in range(Lx):
            triangles.append((site(x, y), site(x + 1, y), site(x, y + 1)))
            triangles.append((site(x + 1, y), site(x + 1, y + 1), site(x, y + 1)))
    return bonds(near), bonds(far), triangles


def _translate(t, a, b, Lx, Ly):
    n = Lx * Ly
    full = (1 << n) - 1
    if b:
        t = ((t << (Lx * b)) | (t >> (n - Lx * b))) & full
    if a:
        high = sum(1 << s for s in range(n) if s % Lx >= a)
        t = ((t << a) & high) | ((t >> (Lx - a)) & (full ^ high))
    return t


class _Exact:
    """One sector's basis and H in 64 bits: representatives by the smallest
    translate, amplitudes by the orbit sizes, every target by search."""

    def __init__(self, case, k, couplings):
        self.case, self.k = case, k
        self.Jz, self.J2, self.Ch = couplings
        Lx, Ly = self.Lx, self.Ly = case["Lx"], case["Ly"]
        n = Lx * Ly
        up = n // 2 + int(case["Sz"])
        h = n // 2
        low = torch.arange(1 << h, device="cuda", dtype=torch.int64)
        ones = sum(((low >> s) & 1) for s in range(h))
        by = [low[ones == q] for q in range(h + 1)]
        parts, held, states = [], 0, []

        def keep():
            t = torch.cat(parts)
            for a in range(Lx):
                for b in range(Ly):
                    if a or b:
                        t = t[t <= _translate(t, a, b, Lx, Ly)]
            states.append(t)

        for left in range(1 << (n - h)):
            q = up - bin(left).count("1")
            if 0 <= q <= h:
                parts.append(by[q] | (left << h))
                held += len(by[q])
                if held > 1 << 25:
                    keep()
                    parts, held = [], 0
        if parts:
            keep()
        t = torch.cat(states)
        size = torch.zeros(len(t), device="cuda", dtype=torch.float64)
        sums = torch.zeros(len(t), device="cuda", dtype=torch.complex128)
        for a in range(Lx):
            for b in range(Ly):
                same = _translate(t, a, b, Lx, Ly) == t
                size += same
                sums += same.to(torch.complex128) * self._phase(a, b)
        ok = sums.abs() > 1e-8
        self.t = t[ok]
        self.norm = torch.sqrt(n / size[ok])
        self.n = len(self.t)

    def _phase(self, a, b):
        x = -2 * math.pi * (self.k[0] * ((-a) % self.Lx) / self.Lx + self.k[1] * ((-b) % self.Ly) / self.Ly)
        return complex(math.cos(x), math.sin(x))

    def terms(self):
        """(flip mask, coefficient of each state) of every pair, and the diagonal."""
        near, far, triangles = _pairs(self.case)
        diag = torch.zeros(self.n, device="cuda", dtype=torch.float64)
        flips = {}
        for pairs, J in ((near, 1.0), (far, self.J2)):
            for x, y in pairs if J else []:
                anti = ((self.t >> x) ^ (self.t >> y)) & 1
                diag += 0.25 * self.Jz * J * (1 - 2 * anti).double()
                flips.setdefault((min(x, y), max(x, y)), []).append(("J", J))
        if self.Ch and self.case["lattice"] == "triangular":
            for i, j, k in triangles:
                for x, y, z in ((i, j, k), (j, k, i), (k, i, j)):
                    flips.setdefault((min(x, y), max(x, y)), []).append((y, z))
        return flips, diag

    def entries(self):
        """Per flipped pair: rows, columns and values of H."""
        flips, self.diag = self.terms()
        phases = torch.tensor([self._phase(a, b) for b in range(self.Ly) for a in range(self.Lx)],
                              device="cuda", dtype=torch.complex128)
        step = 1 << 23
        for (x, y), what in flips.items():
            for at in range(0, self.n, step):
                t = self.t[at: at + step]
                rows = torch.nonzero(((t >> x) ^ (t >> y)) & 1).flatten()
                s = t[rows]
                c = torch.zeros(len(s), device="cuda", dtype=torch.complex128)
                for kind, v in what:
                    if kind == "J":
                        c += 0.5 * v
                    else:
                        sign = (2 * ((s >> kind) & 1) - 1) * (2 * ((s >> v) & 1) - 1)
                        c += 0.25j * self.Ch * sign.to(torch.complex128)
                s = s ^ ((1 << x) | (1 << y))
                best, g = s.clone(), torch.zeros_like(s)
                for b in range(self.Ly):
                    for a in range(self.Lx):
                        if a or b:
                            m = _translate(s, a, b, self.Lx, self.Ly)
                            less = m < best
                            best = torch.where(less, m, best)
                            g = torch.where(less, a + self.Lx * b, g)
                cols = torch.searchsorted(self.t, best).clamp_(max=self.n - 1)
                ok = self.t[cols] == best
                rows, cols = rows[ok] + at, cols[ok]
                yield rows, cols, (c[ok] * phases[g[ok]]) * (self.norm[rows] / self.norm[cols])

    def apply(self, v):
        w = torch.zeros_like(v)
        for rows, cols, val in self.entries():
            w.index_add_(0, rows, (val if v.dim() == 1 else val[:, None]) * v[cols])
        return w + (self.diag if v.dim() == 1 else self.diag[:, None]) * v

    def matrix(self):
        got = [(r.clone(), c.clone(), v.clone()) for r, c, v in self.entries()]
        at = torch.arange(self.n, device="cuda")
        r = torch.cat([x[0] for x in got] + [at])
        c = torch.cat([x[1] for x in got] + [at])
        v = torch.cat([x[2] for x in got] + [self.diag.to(torch.complex128)])
        return torch.sparse_coo_tensor(torch.stack([r, c]), v, (self.n, self.n)).coalesce().to_sparse_csr()

    def lowest(self, how_many, steps):
        """Lowest levels by Lanczos with every vector kept and used twice."""
        H = self.matrix()
        steps = min(steps, self.n)
        g = torch.Generator(device="cuda").manual_seed(1)
        v = torch.randn(self.n, dtype=torch.complex128, device="cuda", generator=g)
        V = torch.empty((steps, self.n), dtype=torch.complex128, device="cuda")
        V[0] = v / v.norm()
        a, b = [], []
        for j in range(steps):
            w = H @ V[j]
            a.append(torch.vdot(V[j], w).real)
            for _ in range(2):
                w = w - V[: j + 1].T @ (V[: j + 1].conj() @ w)
            size = w.norm()
            if j + 1 == steps or float(size) < 1e-10:
                break
            b.append(size)
            V[j + 1] = w / size
        T = torch.diag(torch.stack(a))
        if b:
            e = torch.stack(b)[: len(a) - 1]
            T = T + torch.diag(e, 1) + torch.diag(e, -1)
        return torch.linalg.eigvalsh(T.cpu())[:how_many]


def exact(case, seed):
    op = case["op"]
    n = case["Lx"] * case["Ly"]
    if op == "batch" or n > 32 or (op in ("mixed", "plain") and n > 28):
        return None  # a thousand spectra, or a sector beyond a generic evaluation in seconds
    x = _Exact(case, (case["kx"], case["ky"]), _couplings(case, seed))
    if op in ("hv", "host", "block", "first"):
        v = _vector(x.n, seed, case.get("nv")).to(_dtype(case)).to(torch.complex128)
        w = x.apply(v)
        return w.cpu().numpy() if op == "host" else w
    if op == "dense":
        return torch.linalg.eigvalsh(x.matrix().to_dense().cpu() if x.n < 600 else x.matrix().to_dense()).cpu().numpy()
    found = x.lowest(case["n_ev"], 300 if op == "mixed" else 250).numpy()
    if op == "plain":
        # deflation finds a level as often as it occurs, this Lanczos once: the first is the same for both
        return [float(found[0])] + [None] * (case["n_ev"] - 1)
    return found
