"""The work that users of this library have it do, as cases for timing and comparison.

A case is one crystal on one q-mesh with the options of a run.  The crystals are the benchmark suite's:
fcc Lennard-Jones argon (3 bands), rock-salt Morse (6 bands), Lennard-Jones mass superlattices of p conventional
cells (12 p bands) and the 64-atom rock-salt cell (192 bands).  The seed draws the atomic masses.

What a case does, `do`:
  job1        the whole three-phonon conductivity run, kappa_pipeline.  `phonons` says where the eigenpairs come
              from: "own" has the library diagonalise again (get_frequencies on the device), "given" hands it the
              host program's own (set_phonons, then the pipeline), the two ways in which a host program calls it.
  job3        the iterative solution, kappa_iterative, on given eigenpairs.
  job2        the self-energy along a band path, self_energy_bs.
  frequencies get_frequencies with its arrays on the host.
  files       a run as a command-line user has it: context from the input files, pipeline, context closed.

Results of the FP64 path are double precision.  The mixed path contracts and weighs in single precision and hands
single-precision numbers out in double-precision arrays; they are taken as single precision here.
"""
import functools
import math
import os
import shutil
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "anharmonic-lattice-dynamics_b200", "python"))
import ald  # noqa: E402
from ald import inputs  # noqa: E402

THZ = inputs.THZ_TO_CM


def listed():
    job1 = {"do": "job1", "tempk": 300.0, "width_thz": 0.1, "cg_tol": 0.0}
    return [
        # a first look at a material: one atom, a coarse mesh; launches and latency count
        dict(job1, name="argon-10-gauss-mixed", crystal="argon", mesh="10x10x10", delta="gauss", precision="mixed",
             phonons="own"),
        # the everyday run: two atoms, 16^3, tetrahedra, in both precisions
        dict(job1, name="rocksalt-16-tetra-mixed", crystal="rocksalt", mesh="16x16x16", delta="tetra",
             precision="mixed", phonons="own"),
        dict(job1, name="rocksalt-16-tetra-fp64", crystal="rocksalt", mesh="16x16x16", delta="tetra",
             precision="fp64", phonons="given"),
        # a converged mesh of one atom, solved to a residual (FP64 one mesh step below, an odd mesh in draw())
        dict(job1, name="argon-32-gauss-mixed", crystal="argon", mesh="32x32x32", delta="gauss", precision="mixed",
             phonons="given", width_thz=0.05, cg_tol=1e-8),
        dict(job1, name="argon-26-gauss-fp64", crystal="argon", mesh="26x26x26", delta="gauss", precision="fp64",
             phonons="given", width_thz=0.05, cg_tol=1e-8),
        # superlattices: 4 and 8 atoms, anisotropic meshes
        dict(job1, name="superlattice-1-gauss-fp64", crystal="superlattice 1", mesh="8x8x8", delta="gauss",
             precision="fp64", phonons="given"),
        dict(job1, name="superlattice-2-gauss-mixed", crystal="superlattice 2", mesh="6x12x12", delta="gauss",
             precision="mixed", phonons="given"),
        # the largest cell
        dict(job1, name="rocksalt-192-tetra-mixed", crystal="supercell", mesh="4x4x4", delta="tetra",
             precision="mixed", phonons="given"),
        # harmonic phonons of the largest cell alone (dispersion, density of states)
        {"do": "frequencies", "name": "frequencies-192", "crystal": "supercell", "mesh": "4x4x4"},
        # the iterative solution
        {"do": "job3", "name": "rocksalt-12-iterative-fp64", "crystal": "rocksalt", "mesh": "12x12x12",
         "delta": "tetra", "precision": "fp64", "tempk": 300.0},
        # linewidths along a band path
        {"do": "job2", "name": "rocksalt-14-self-energy", "crystal": "rocksalt", "mesh": "14x14x14",
         "tempk": 300.0, "gauss": False, "points": 20},
        # from the files to the conductivity, everything new
        {"do": "files", "name": "rocksalt-12-files", "crystal": "rocksalt", "mesh": "12x12x12", "delta": "tetra",
         "precision": "mixed", "tempk": 300.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["job1"] * 7 + ["job3", "job2", "frequencies", "files"])
    tempk = float(rng.randrange(100, 601, 20))
    if what == "frequencies":
        if rng.random() < 0.5:
            p, m = rng.randrange(1, 9), rng.choice([4, 6])
            return {"do": what, "crystal": "superlattice %d" % p,
                    "mesh": "%dx%dx%d" % (m if p == 1 else rng.choice([2, 4]), m, m)}
        e = rng.randrange(6, 31)
        return {"do": what, "crystal": rng.choice(["argon", "rocksalt"]), "mesh": "%dx%dx%d" % (e, e, e)}
    if what == "job2":
        e = rng.randrange(6, 17)
        return {"do": what, "crystal": rng.choice(["argon", "rocksalt"]), "mesh": "%dx%dx%d" % (e, e, e),
                "tempk": tempk, "gauss": rng.random() < 0.5, "points": rng.randrange(3, 24)}
    delta, precision = rng.choice(["tetra", "gauss"]), rng.choice(["fp64", "mixed"])
    if what in ("job3", "files"):
        e = 2 * _log_int(rng, 3, 7)
        return {"do": what, "crystal": rng.choice(["argon", "rocksalt"]), "mesh": "%dx%dx%d" % (e, e, e),
                "delta": delta, "precision": precision, "tempk": tempk}
    crystal = rng.choice(["argon", "rocksalt", "superlattice"])
    phonons = "given"
    if crystal == "superlattice":
        # p cells along x (one cell is cubic, and so is its mesh); an even number of points along each axis, where
        # the reference's test for the zone centre finds it
        p = rng.randrange(1, 5)
        crystal = "superlattice %d" % p
        m = 2 * rng.randrange(2, 7 if p <= 2 else 5)
        mesh = (m if p == 1 else 2 * rng.randrange(1, 4 if p == 2 else 3), m, m)
    else:
        # odd meshes in FP64 only: there the acoustic modes at the zone centre enter every row, and single
        # precision leaves rounding noise in them that no two orders of summation share
        top = {"argon": {"fp64": 26, "mixed": 32}, "rocksalt": {"fp64": 14, "mixed": 16}}[crystal][precision]
        e = _log_int(rng, 6, top)
        if e % 2 and precision == "mixed":
            e += 1
        mesh = (e, e, e)
        if e % 2 == 0:
            phonons = rng.choice(["own", "given"])
    return {"do": "job1", "crystal": crystal, "mesh": "%dx%dx%d" % mesh, "delta": delta, "precision": precision,
            "phonons": phonons, "tempk": tempk, "width_thz": rng.choice([0.05, 0.1]),
            "cg_tol": rng.choice([0.0, 0.0, 1e-8])}


# ---------------------------------------------------------------------------- inputs


def _mesh(case):
    return tuple(int(x) for x in case["mesh"].split("x"))


def _sentinel(k):
    return 1001.0 + k


@functools.lru_cache(maxsize=None)
def _crystal(kind):
    """The structure with a recognisable mass in the place of each free one, and its force constants."""
    if kind == "argon":
        st, n = inputs.lj_argon(mass=_sentinel(0)), 1
    elif kind == "rocksalt":
        st, n = inputs.rocksalt_morse(mA=_sentinel(0), mB=_sentinel(1)), 2
    elif kind == "supercell":
        st, n = inputs.rocksalt_supercell(inputs.BASE_SEED), 64
        st.atom_masses = [_sentinel(k) for k in range(n)]
    else:
        p = int(kind.split()[1])
        st, n = inputs.lj_superlattice(p, inputs.BASE_SEED), 4 * p
        st.atom_masses = [_sentinel(k) for k in range(n)]
    return st, n, inputs.build_force_constants(st)


@functools.lru_cache(maxsize=None)
def _template(kind):
    """The input files of a crystal with the recognisable masses, by name."""
    st, _, _ = _crystal(kind)
    with tempfile.TemporaryDirectory() as d:
        inputs.write_inputs(st, inputs.RunParams(mesh=(2, 2, 2)), d)
        return {f: open(os.path.join(d, f)).read() for f in os.listdir(d)}


def _masses(kind, seed):
    """Masses as the suites draw them: one per species, per superlattice layer, or (supercell) per atom as in a
    disordered alloy."""
    rng = np.random.default_rng([int(seed) % (1 << 32), 7])
    n = _crystal(kind)[1]
    if kind == "argon":
        return [float(m) for m in rng.uniform(30.0, 50.0, 1)]
    if kind == "rocksalt":
        return [float(m) for m in (rng.uniform(18.0, 28.0), rng.uniform(30.0, 45.0))]
    if kind == "supercell":
        return [float(m) for m in rng.uniform(20.0, 60.0, n)]
    return [float(m) for m in np.repeat(rng.uniform(20.0, 80.0, n // 4), 4)]


def _write(case, seed):
    """The directory of input files of a case."""
    kind = case["crystal"]
    d = tempfile.mkdtemp(prefix="ald_case_")
    files = dict(_template(kind))
    for k, m in enumerate(_masses(kind, seed)):
        for f in ("structure.params", "lat_fc.dat"):
            files[f] = files[f].replace(repr(_sentinel(k)), repr(m))
    run = files["latdyn.params"].split("\n")
    run[0] = "%d %d %d .false.   mesh, dos_bs_only" % _mesh(case)
    run[4] = "%r 1.0   width, etaz" % (case.get("width_thz", 0.1) * THZ)
    run[6] = "%r %r 1   tmin tmax ntemp" % (case.get("tempk", 300.0), case.get("tempk", 300.0))
    files["latdyn.params"] = "\n".join(run)
    if case["do"] == "job2":
        # between points of no symmetry, off the mesh
        files["kpbs.params"] = "0\n%d\n2\nA 0.03 0.07 0.11\nB 0.21 0.05 0.47\nC 0.41 0.33 0.13\n" % case["points"]
    for f, text in files.items():
        with open(os.path.join(d, f), "w") as out:
            out.write(text)
    return d


def _options(case):
    o = ald.default_options(precision=ald.MIXED if case.get("precision") == "mixed" else ald.FP64,
                            delta=ald.DELTA_GAUSS if case.get("delta") == "gauss" else ald.DELTA_TETRA)
    if case.get("cg_tol"):
        o.cg_stop, o.cg_tol = ald.CG_RESIDUAL, case["cg_tol"]
    return o


class _State:
    """A context with its input files, or the files alone."""

    def __init__(self, case, seed):
        self.case = case
        self.dir = _write(case, seed)
        self.opt = _options(case)
        self.ctx = self.given = None

    def __del__(self, rmtree=shutil.rmtree):
        if self.ctx is not None:
            self.ctx.close()
        rmtree(self.dir, ignore_errors=True)


def prepare(case, seed):
    s = _State(case, seed)
    if case["do"] != "files":
        s.ctx = ald.Context(s.dir, s.opt)
    if case["do"] == "job3" or case.get("phonons") == "given":
        p = _Phonons(case, seed)
        s.given = (p.lam, p.vec, p.vel)
    elif case["do"] == "job2":
        s.ctx.invalidate_phonons()
    return s


def _held(case, v):
    """The mixed path's numbers in the precision that they have."""
    if case.get("precision") != "mixed":
        return v
    return np.asarray(v, dtype=np.float32)


JOB1 = ("Q", "QN", "QU", "kappa_rta_modes", "kappa_cg_modes", "x")


def run(state):
    c, ctx = state.case, state.ctx
    if c["do"] == "frequencies":
        lam, vec, vel = ctx.get_frequencies()
        return {"eigenval": lam, "eigenvec": vec, "veloc": vel}
    if c["do"] == "job2":
        r = ctx.self_energy_bs(state.dir, c["tempk"], gauss=c["gauss"])
        return {k: r[k] for k in ("omega0", "nself", "uself")}
    if c["do"] == "files":
        with ald.Context(state.dir, state.opt) as ctx:
            r = ctx.kappa_pipeline(c["tempk"])
        return {k: _held(c, r[k]) for k in JOB1}
    if state.given is not None:
        ctx.set_phonons(*state.given)
    else:
        ctx.invalidate_phonons()
    if c["do"] == "job3":
        r = ctx.kappa_iterative(c["tempk"])
        return {k: _held(c, r[k]) for k in ("Q", "kappa_rta_modes", "kappa_iter_modes", "F")}
    r = ctx.kappa_pipeline(c["tempk"])
    return {k: _held(c, r[k]) for k in JOB1}


# ---------------------------------------------------------------------------- what a pass cannot do without


@functools.lru_cache(maxsize=None)
def _sizes(kind, mesh):
    """Bands, mesh points and irreducible points."""
    d = _write({"do": "files", "crystal": kind, "mesh": mesh}, 0)
    info, _ = ald.read_mesh(d)
    shutil.rmtree(d, ignore_errors=True)
    return info.ndyn, info.nkc, info.nibz


def work(case):
    """Bytes: eigenpairs in, results out, and for the linear solve its matrix once.  Flops: for each pair of mesh
    points the two complex mode products (8 b^4 each) and for each band triplet about 20 for the two processes'
    delta weights; for the harmonic problem 10 b^3 complex multiply-adds for each of seven stencil points."""
    b, nk, ni = _sizes(case["crystal"], case["mesh"])
    eig = nk * (b + 2 * b * b + 3 * b) * 8
    harmonic = 7 * nk * 80.0 * b ** 3
    if case["do"] == "frequencies":
        return {"bytes": eig, "flops": harmonic}
    if case["do"] == "job2":
        n = 2 * case["points"]
        return {"bytes": eig + n * b * 40, "flops": n * nk * (80.0 * b ** 3 + 16.0 * b ** 4 + 40.0 * b ** 3)}
    word = 4 if case["precision"] == "mixed" else 8
    n = 3 * b * ni
    three = ni * nk * (16.0 * b ** 4 + 20.0 * b ** 3)
    matrix = 0 if case["do"] == "job3" else n * n * word
    own = harmonic if case["do"] == "files" or case.get("phonons") == "own" else 0.0
    return {"bytes": eig + 8 * (3 * n // 3 + n) + matrix, "flops": own + three}


# ---------------------------------------------------------------------------- the same in 64 bits, in numpy and torch

CNST = float(np.float32(521.1098918))  # the reference keeps this constant in single precision
HBAR, UMA, EE, H, C_LIGHT, K_B = 1.054571628e-34, 1.66053878e-27, 1.60217653e-19, 6.62606896e-34, 2.99792458e8, \
    1.3806504e-23
CONST33 = 1e30 * (HBAR / UMA) ** 1.5 / math.sqrt(EE * 1e20 / UMA) ** 1.5 * EE / H / 100 / C_LIGHT
# acoustic modes at the zone centre have no frequency, and what multiplies 1/frequency there is 0/0; the given
# eigenpairs keep them at this share of the largest eigenvalue
FLOOR = 1e-10


class _Phonons:
    """The mesh and the harmonic eigenpairs of a case, on the exact mesh fractions as a host program hands them over,
    or (reference_mesh) on the reference's, which are single-precision quotients."""

    def __init__(self, case, seed, reference_mesh=False):
        st, _, fc = _crystal(case["crystal"])
        masses = _masses(case["crystal"], seed)
        self.fc, self.nc = fc, _mesh(case)
        self.mass = np.array(masses if len(masses) == fc["nat0"] else [masses[t - 1] for t in st.atom_types])
        nc, nat0 = self.nc, fc["nat0"]
        self.b, self.nk = 3 * nat0, nc[0] * nc[1] * nc[2]
        self.even = all(x % 2 == 0 for x in nc)
        self.m = np.stack(np.meshgrid(*(np.arange(x) for x in nc), indexing="ij"), -1).reshape(-1, 3)
        g = 2 * np.pi * np.linalg.inv(np.asarray(fc["r"], dtype=float)).T  # rows: reciprocal vectors
        word = np.float32 if reference_mesh else np.float64
        frac = (self.m.astype(word) / np.array(nc, dtype=word)).astype(float) - (0.5 if self.even else 0.0)
        self.kpc, self.pairs = frac @ g, not reference_mesh
        self.cell = np.array([np.array(a[2:5], dtype=float) @ np.asarray(fc["r"], dtype=float) for a in fc["atoms"]])
        self.home = np.array([a[1] - 1 for a in fc["atoms"]])
        self.lam, self.vec, self.vel = self._solve()

    def index(self, m):
        return np.ravel_multi_index(tuple((m % np.array(self.nc)).T), self.nc)

    def _solve(self):
        b, nk = self.b, self.nk
        t = np.array([x[:4] for x in self.fc["fc2"]]) - 1
        w = np.array([x[4] for x in self.fc["fc2"]]) / np.sqrt(self.mass[t[:, 0]] * self.mass[self.home[t[:, 2]]])
        atoms = np.unique(t[:, 2])
        M = np.zeros((len(atoms), b * b))
        np.add.at(M, (np.searchsorted(atoms, t[:, 2]), (3 * t[:, 0] + t[:, 1]) * b + 3 * self.home[t[:, 2]] + t[:, 3]), w)
        half = np.flatnonzero(self.index(-self.m) >= np.arange(nk)) if self.pairs else np.arange(nk)
        neg = self.index(-self.m[half])
        R = self.cell[atoms]
        lam, vec = np.zeros((nk, b)), np.zeros((nk, b, b), dtype=complex)
        vel = np.zeros((nk, b, 3))
        for at in np.array_split(half, max(1, len(half) * b * b // 4_000_000)):
            ph = np.exp(1j * (self.kpc[at] @ R.T))
            D = (ph @ M).reshape(-1, b, b)
            l, v = np.linalg.eigh((D + D.conj().transpose(0, 2, 1)) / 2)
            lam[at], vec[at] = l, v
            for x in range(3):
                G = ((1j * R[:, x] * ph) @ M).reshape(-1, b, b)
                vel[at, :, x] = np.einsum("qil,qil->ql", v.conj(), (G + G.conj().transpose(0, 2, 1)) / 2 @ v).real
        if self.pairs:  # e(-q) is the conjugate of e(q)
            lam[neg], vec[neg], vel[neg] = lam[half], vec[half].conj(), -vel[half]
        self.raw = lam.copy()
        lam = np.maximum(np.abs(lam), FLOOR * np.abs(lam).max())
        vel *= (1e-10 * math.sqrt(EE * 1e20 / UMA) / C_LIGHT / 2 / np.sqrt(lam))[:, :, None]
        centre = self.index(np.array([[x // 2 for x in self.nc]]) if self.even else np.zeros((1, 3), dtype=int))
        vel[centre, :3] = 0.0
        # in the reference's layouts: (b, nk), (b, b, nk), (3, b, nk)
        return (np.asfortranarray(lam.T), np.asfortranarray(vec.transpose(1, 2, 0)),
                np.asfortranarray(vel.transpose(2, 1, 0)))


def _v3_row(P, T, q1, q2s):
    """|V3|^2 (q2, l1, l2, l3) of one row for the mesh points q2s."""
    q3 = T["i3"](q1)[q2s]
    b, nat0 = P.b, P.b // 3
    ph = T["eiqr"][q2s][:, T["j"]] * T["eiqr"][q3][:, T["k"]]
    e1 = T["vec"][q1].T.reshape(b, nat0, 3)[:, T["i"]]  # (l1, triple, alpha)
    Hs = torch.einsum("tabc,lta->tlbc", T["w"], e1)
    A = torch.zeros((len(q2s), b, b, b), dtype=torch.complex128, device="cuda")
    for j0, k0, sel in T["blocks"]:
        A[:, :, 3 * j0:3 * j0 + 3, 3 * k0:3 * k0 + 3] = (ph[:, sel] @ Hs[sel].reshape(len(sel), -1)).reshape(-1, b, 3, 3)
    A = torch.matmul(T["vec"][q2s].transpose(1, 2)[:, None], A)  # (q2, l1, l2, k gamma)
    A = torch.matmul(A, T["vec"][q3][:, None])
    lam = T["lam"]
    den = 8 * torch.sqrt(lam[q1][None, :, None, None] * lam[q2s][:, None, :, None] * lam[q3][:, None, None, :])
    return (A.real ** 2 + A.imag ** 2) / den * CONST33 ** 2


def _corner_weights(E, e):
    """Linear-tetrahedron weights of the corners, E (n, 4) ascending, at energies e (n)."""
    E1, E2, E3, E4 = E.unbind(1)
    d = lambda a, b: torch.clamp(a - b, min=1e-10)  # noqa: E731
    D21, D31, D41, D32, D42, D43 = d(E2, E1), d(E3, E1), d(E4, E1), d(E3, E2), d(E4, E2), d(E4, E3)
    x = e - E1
    low = torch.stack([((E2 - e) / D21 + (E3 - e) / D31 + (E4 - e) / D41) * x * x / (D41 * D31 * D21),
                       x ** 3 / (D21 ** 2 * D31 * D41), x ** 3 / (D21 * D31 ** 2 * D41),
                       x ** 3 / (D21 * D31 * D41 ** 2)], 1)
    y = E4 - e
    high = torch.stack([y ** 3 / (D41 ** 2 * D42 * D43), y ** 3 / (D41 * D42 ** 2 * D43), y ** 3 / (D41 * D42 * D43 ** 2),
                        ((e - E3) / D43 + (e - E2) / D42 + (e - E1) / D41) * y * y / (D41 * D42 * D43)], 1)
    a, b, c, f = E3 - e, E4 - e, e - E1, e - E2
    b11 = a * f / (D42 * D32) + b * c / (D41 * D42) + a * c / (D32 * D41)
    b12 = b * c / (D42 * D31) + b * f / (D42 * D32) + a * c / (D31 * D32)
    b21 = a * f / (D42 * D31) + b * f / (D42 * D41) + a * c / (D31 * D41)
    b22 = a * f / (D32 * D31) + b * c / (D41 * D31) + b * f / (D32 * D41)
    mid = 0.5 * torch.stack([a / D31 ** 2 * b11 + b / D41 ** 2 * b12, a / D32 ** 2 * b21 + b / D42 ** 2 * b22,
                             f / D32 ** 2 * b21 + c / D31 ** 2 * b11, f / D42 ** 2 * b22 + c / D41 ** 2 * b12], 1)
    return torch.where((e <= E2)[:, None], low, torch.where((e <= E3)[:, None], mid, high))


def _exact_q(case, seed):
    """The linewidths Q (irreducible point, band) of a run on given eigenpairs."""
    P = _Phonons(case, seed)
    d = _write(case, seed)
    _, tables = ald.read_mesh(d)  # the rows that the run computes
    shutil.rmtree(d, ignore_errors=True)
    rows = tables["mapinv"] - 1
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    b, nk, nc = P.b, P.nk, np.array(P.nc)
    half = nc // 2 if P.even else 0 * nc
    m = torch.from_numpy(P.m).cuda()
    N, h = torch.from_numpy(nc).cuda(), torch.from_numpy(half).cuda()

    def at(x):
        x = x % N
        return (x[:, 0] * int(nc[1]) + x[:, 1]) * int(nc[2]) + x[:, 2]

    t = np.array([x[:6] for x in P.fc["fc3"]]) - 1  # i a j b k c
    val = np.array([x[6] for x in P.fc["fc3"]]) / np.sqrt(
        P.mass[t[:, 0]] * P.mass[P.home[t[:, 2]]] * P.mass[P.home[t[:, 4]]])
    trip, which = np.unique(t[:, [0, 2, 4]], axis=0, return_inverse=True)
    W = np.zeros((len(trip), 3, 3, 3))
    np.add.at(W, (which.reshape(-1), t[:, 1], t[:, 3], t[:, 5]), val)
    home = P.home[trip[:, 1]], P.home[trip[:, 2]]
    blocks = [(int(j0), int(k0), dev(np.flatnonzero((home[0] == j0) & (home[1] == k0))))
              for j0, k0 in np.unique(np.stack(home, 1), axis=0)]
    T = {"eiqr": torch.exp(1j * dev(P.kpc @ P.cell.T)), "i": dev(trip[:, 0]), "j": dev(trip[:, 1]),
         "k": dev(trip[:, 2]), "w": dev(W).to(torch.complex128), "blocks": blocks, "lam": dev(P.lam.T),
         "vec": dev(P.vec.transpose(2, 0, 1)), "i3": lambda q: at(h - m[q] - m)}
    freq = torch.sqrt(T["lam"]) * CNST
    temp = case["tempk"] * K_B / (100 * H * C_LIGHT)
    z = freq / temp
    n = torch.where(z > 60, torch.zeros_like(z), 1 / torch.expm1(z))
    # where the reference's zone-centre test holds, the first three bands are left out
    centre = torch.zeros(nk, 3, dtype=torch.bool, device="cuda")
    centre[at(torch.from_numpy(nc // 2).cuda()[None])] = True
    keep = torch.ones(nk, b, device="cuda", dtype=torch.float64)
    keep[:, :3][centre] = 0.0
    neg = at(-m)
    sigma = case.get("width_thz", 0.1) * THZ
    scale = (2 * math.pi) ** 2 / nk
    step = max(1, int(1.2e10 / (16 * b ** 3)))
    corner = None
    if case["delta"] == "tetra":
        off = torch.tensor([[0, 0, 0], [1, 0, 0], [0, 1, 0], [1, 1, 0], [0, 0, 1], [1, 0, 1], [0, 1, 1], [1, 1, 1]],
                           device="cuda")
        six = torch.tensor([[1, 2, 3, 6], [2, 3, 4, 6], [1, 3, 5, 6], [3, 4, 6, 8], [3, 5, 6, 7], [3, 6, 7, 8]],
                           device="cuda") - 1
        box = torch.stack([at(m + o) for o in off], 1)
        corner = box[:, six].reshape(-1, 4)
    Q = torch.zeros(len(rows), b, dtype=torch.float64, device="cuda")
    for r, q1 in enumerate(int(x) for x in rows):
        plus, minus = at(m[q1] + m + h), at(m[q1] - m + h)
        v = torch.cat([_v3_row(P, T, q1, s) for s in torch.arange(nk, device="cuda").split(step)]) * scale
        w1 = freq[q1]
        # process 1 at q2, process 2 at -q2
        f1 = v * keep[:, None, :, None] * keep[plus][:, None, None, :]
        f2 = torch.empty_like(v)
        f2[neg] = v * keep[neg][:, None, :, None] * keep[plus][:, None, None, :]
        del v
        for f, three, sign, half_of, occ in ((f1, plus, -1.0, 1.0, n), (f2, minus, 1.0, 0.5, n + 1)):
            f = f * occ[:, None, :, None] * (n[three] + 1)[:, None, None, :]
            E = sign * freq[:, :, None] + freq[three][:, None, :]  # (w, l2, l3)
            if corner is None:
                x = w1[None, :, None, None] - E[:, None]
                Q[r] += half_of * (f * torch.exp(-x * x / 2 / sigma / sigma)).sum((0, 2, 3)) / math.sqrt(
                    2 * math.pi) / sigma
                continue
            for l2 in range(b):
                Es, order = E[:, l2][corner].sort(1)  # (tetrahedron, corner, l3)
                inside = (w1[:, None, None] >= Es[None, :, 0]) & (w1[:, None, None] <= Es[None, :, 3])
                l1, tet, l3 = inside.nonzero(as_tuple=True)
                c = _corner_weights(Es[tet, :, l3], w1[l1])
                wts = corner[tet].gather(1, order[tet, :, l3])
                Q[r].index_add_(0, l1, half_of * (c / 6 * f[wts, l1[:, None], l2, l3[:, None]]).sum(1))
        Q[r] *= n[q1]
    return Q.cpu().numpy()


def exact(case, seed):
    """Given eigenpairs: the linewidths.  The conductivities and the solution have no such value: the operation that
    stands for an arm of a star is the reference's choice, and the normal and umklapp shares go by which side of the
    zone boundary single precision puts a point.  Own eigenpairs: the eigenvalues; what follows from the eigenvectors
    depends on the basis that a solver leaves in degenerate levels."""
    if case["do"] == "frequencies":
        P = _Phonons(case, seed, reference_mesh=True)
        return {"eigenval": np.asfortranarray(np.abs(P.raw).T), "eigenvec": None, "veloc": None}
    if case["do"] == "job3" or case.get("phonons") == "given":
        return {"Q": _exact_q(case, seed)}
    return None
