"""The work a user of this library has it do, as timed cases.

A case is one call (or one step's calls) through the public entry points, on a
seeded synthetic molecule of the repository's own workload rules
(lio_b200/workloads.py): H:C:N:O clusters, the H 2s1p / C,N,O 3s2p1d contracted
Cartesian basis, 30 or 40 radial shells x 194 or 302 directions per atom, and
densities from random orthonormal orbitals. Fields of a case:

  call      what is called (see `prepare` and `run`):
              scf     g2g_solve_groups_(0): energy and Kohn-Sham update of an SCF or TD step
              energy  g2g_solve_groups_(1): energy alone
              forces  g2g_solve_groups_(2): energy and XC forces
              md      a molecular-dynamics step: g2g_reload_atom_positions_, then type 2
              device  g2g_solve_device_noalloc_: device arrays in and out, FP64 form
              batch   lio_batch_solve: many molecules, half LDA, half PBE
              serve   lio_srv: one request for each of the resident molecules in flight at once
  atoms     atoms of the molecule (batch, serve: of the largest one)
  molecules batch, serve: how many molecules
  iexch     3 LDA (Slater + VWN), 9 PBE
  open      open shell (alpha and beta densities)
  rad, ang  radial shells and directions per atom
  form      "default" (what a caller that sets nothing gets) or "fp64" (g2g_set_precision_(0))

The grid, its device arrays and the caller's vectors are what a program keeps
from one step to the next, so `prepare` builds them; the Kohn-Sham vectors are
added into, as the ABI says. The g2g ABI holds one molecule per loaded library,
so each state has a private copy of the library, kept for later states.
"""
import atexit
import ctypes as C
import functools
import math
import os
import shutil
import tempfile

import numpy as np
import torch

from lio_b200 import g2g, serve
from lio_b200 import workloads as W


# ------------------------------------------------------------------ the cases
def _case(name, call, atoms, iexch=9, open_=False, rad=40, ang=194, form="default", molecules=1):
    c = dict(call=call, atoms=atoms, molecules=molecules, iexch=iexch, open=open_, rad=rad, ang=ang, form=form)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a water-sized molecule on the small grid: launches and host latency are all there is
        _case("scf 3 atoms PBE", "scf", 3, rad=30),
        # the 8-atom LDA cluster, the repository's smallest configuration
        _case("scf 8 atoms LDA", "scf", 8, iexch=3),
        # an ordinary radical, odd sizes, open shell
        _case("scf 27 atoms PBE open", "scf", 27, open_=True),
        # the 64-atom closed-shell configuration on the 302-point grid
        _case("scf 64 atoms PBE 302", "scf", 64, ang=302),
        # the large LDA molecule: no gradient kinds, F alone
        _case("scf 121 atoms LDA", "scf", 121, iexch=3),
        # the 256-atom open-shell configuration, the largest
        _case("scf 256 atoms PBE open 302", "scf", 256, open_=True, ang=302),
        # the plain FP64 form, for callers that ask for it
        _case("scf 45 atoms PBE fp64", "scf", 45, form="fp64"),
        # FP64, device arrays, no allocation: a host program that owns the GPU's memory
        _case("device 14 atoms PBE open fp64", "device", 14, open_=True, form="fp64"),
        # forces of a geometry optimisation step
        _case("forces 64 atoms PBE open 302", "forces", 64, open_=True, ang=302),
        # a molecular-dynamics step: new grid, energy and forces
        _case("md 100 atoms PBE", "md", 100),
        # many small molecules per launch (conformers, fragments)
        _case("batch 36 molecules", "batch", 40, rad=30, molecules=36),
        # a service with molecules of different sizes, one request of each at once
        _case("serve 10 molecules 302", "serve", 90, ang=302, molecules=10),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["scf", "scf", "scf", "scf", "energy", "forces", "md", "device", "batch", "serve"])
    iexch = 9 if rng.random() < 0.75 else 3
    open_ = iexch == 9 and rng.random() < 0.45  # open-shell LDA has no potential in LIO
    ang, rad = rng.choice([194, 194, 302]), rng.choice([30, 40, 40])
    if call == "batch":
        return _case(None, call, _log(rng, 8, 40), rad=rad, molecules=_log(rng, 4, 48))
    if call == "serve":
        return _case(None, call, _log(rng, 12, 110), open_=open_, rad=rad, ang=ang, molecules=_log(rng, 3, 12))
    if call == "device":
        return _case(None, call, _log(rng, 3, 40), iexch, open_, rad, 194, "fp64")
    if call == "md":
        return _case(None, call, _log(rng, 6, 130), 9, open_, rad, ang)
    fp64 = rng.random() < 0.25
    return _case(None, call, _log(rng, 3, 60 if fp64 else 240), iexch, open_, rad, ang, "fp64" if fp64 else "default")


# ----------------------------------------------------------- molecules, densities
def _counts(atoms):
    c, n = atoms // 4, atoms // 16
    o = n if atoms > 3 else 1
    return {"C": c if atoms > 3 else 0, "N": n, "O": o, "H": atoms - (c if atoms > 3 else 0) - n - o}


def _molecule(atoms, iexch, open_, rad, ang, box, seed):
    mol = W.random_cluster(_counts(atoms), box, seed)
    return W.Workload("case", mol, W.build_basis(mol, seed + 1), iexch, open_, ang, rad, np.zeros(0), None, None, seed)


def _cuda():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _occupied(M, n, gen):
    """Packed P = C C^T (lower triangle, off-diagonals doubled) of n random orthonormal orbitals."""
    q, _ = torch.linalg.qr(torch.randn(M, max(1, n), dtype=torch.float64, device=gen.device, generator=gen))
    r, c = torch.triu_indices(M, M, device=gen.device)
    v = (q @ q.T)[r, c]
    return torch.where(r == c, v, 2.0 * v).cpu().numpy()


def _with_density(wl, seed):
    gen = torch.Generator(_cuda()).manual_seed(seed + 2)
    M, electrons = wl.basis.M, int(sum(wl.mol.Z))
    if wl.open_shell:
        wl.nco, wl.nunp = (electrons - 2) // 2, 2
        wl.rho_a = _occupied(M, wl.nco + 2, gen)
        wl.rho_b = _occupied(M, wl.nco, gen)
        wl.rho = wl.rho_a + wl.rho_b
    else:
        wl.nco = electrons // 2
        wl.rho = 2.0 * _occupied(M, wl.nco, gen)
    return wl


def _box(atoms):
    """Box (angstrom) of the repository's 8-, 64- and 256-atom clusters' density."""
    return max(3.0, 3.46 * atoms ** (1.0 / 3.0))


def _sizes(case):
    """Atoms of each molecule of a batch or a service: log-spaced up to the largest, the smallest 3 or 4."""
    n, lo = case["molecules"], 3 if case["call"] == "batch" else 4
    return [int(round(lo * (case["atoms"] / lo) ** (i / max(1, n - 1)))) for i in range(n)]


def _molecules(case, seed, density=True):
    """The case's molecules for a seed, with their densities."""
    if case["call"] in ("batch", "serve"):
        out = []
        for i, atoms in enumerate(_sizes(case)):
            iexch = (3 if i % 2 else 9) if case["call"] == "batch" else case["iexch"]
            box = max(3.0, 2.2 * atoms ** (1.0 / 3.0) + 1.5)
            out.append(_molecule(atoms, iexch, case["open"], case["rad"], case["ang"], box, 1000 * seed + 10 * i))
    else:
        out = [_molecule(case["atoms"], case["iexch"], case["open"], case["rad"], case["ang"], _box(case["atoms"]),
                         1000 * seed)]
    return [_with_density(wl, wl.seed) if density else wl for wl in out]


# ------------------------------------------------------------- states and passes
_free_libraries = []
_copies = []


def _library():
    if _free_libraries:
        return _free_libraries.pop()
    if not _copies:
        _copies.append(tempfile.mkdtemp(prefix="g2g_copy_"))
        atexit.register(shutil.rmtree, _copies[0], ignore_errors=True)
    fd, path = tempfile.mkstemp(suffix=".so", dir=_copies[0])
    os.close(fd)
    shutil.copyfile(g2g.DEFAULT_LIB, path)
    lib = g2g.G2GLibrary(path)
    lib.init()
    lib.check("g2g_init_")
    return lib


class _Single:
    """One molecule bound to its own copy of the g2g library, with its grid built."""

    def __init__(self, case, wl):
        self.case, self.wl = case, wl
        self.lib = _library()
        lib = self.lib
        e, w = g2g.angular_tables(wl.n_ang)
        lib.set_options(eai=True)
        if wl.n_ang == 194:
            lib.bind_workload(wl, {2: (e, w)})
            self.grid_type = 2
        else:
            lib.bind_workload(wl, {})
            lib.set_angular_grid(3, e, w)
            self.grid_type = 3
        if case["form"] == "fp64" or hasattr(lib, "perf_mode_set"):
            lib.set_precision(0 if case["form"] == "fp64" else 3)  # 3: the mode of a caller that sets none
            lib.perf_mode_set = True  # a later state of this copy sets its mode again
        self.reload()
        if case["call"] == "device":
            up = lambda v: torch.from_numpy(v).cuda()  # noqa: E731
            dens = [wl.rho_a, wl.rho_b] if wl.open_shell else [wl.rho]
            self.rho = [up(d) for d in dens]
            self.fock = [torch.zeros_like(d) for d in self.rho]
            self.energy = torch.zeros(1, dtype=torch.float64, device="cuda")
            self.stream = torch.cuda.Stream()
            torch.cuda.synchronize()

    def reload(self):
        msg = self.lib.reload_atom_positions(self.grid_type)
        if msg:
            raise RuntimeError(msg)

    def run(self):
        lib, call = self.lib, self.case["call"]
        if call == "scf":
            e = lib.solve_groups(0)
            out = {"energy": np.array([e]), "fock": lib.fock}
            return dict(out, fock_b=lib.fockb) if self.wl.open_shell else out
        if call == "energy":
            return {"energy": np.array([lib.solve_groups(1)])}
        if call == "device":
            p = [C.c_void_p(t.data_ptr()) for t in self.rho + self.fock]
            n = len(self.rho)
            rc = lib.lib.g2g_solve_device_noalloc_(p[0], p[1] if n == 2 else None, p[n], p[n + 1] if n == 2 else None,
                                                   C.c_void_p(self.energy.data_ptr()),
                                                   C.c_void_p(self.stream.cuda_stream))
            if rc:
                lib.check("g2g_solve_device_noalloc_")
            out = {"energy": self.energy, "fock": self.fock[0]}
            return dict(out, fock_b=self.fock[1]) if n == 2 else out
        if call == "md":  # the integrator's new positions, then the grid and the gradients
            lib._arrays["r"][...] = self.wl.mol.pos
            self.reload()
        e, forces = lib.solve_forces(2)
        return {"energy": np.array([e]), "forces": forces}

    def __del__(self):
        if getattr(self, "lib", None) is not None:
            self.lib.deinit()
            _free_libraries.append(self.lib)


class _Batch:
    def __init__(self, wls):
        self.batch = serve.XCBatch(wls)
        self.dens = [(wl.rho_a, wl.rho_b) if wl.open_shell else (wl.rho, None) for wl in wls]

    def run(self):
        energies, fock, _, _ = self.batch.solve(self.dens)
        return {"energies": energies, "fock": fock}


class _Serve:
    def __init__(self, wls):
        self.server = serve.XCServer(budget_bytes=40 << 30)
        self.ids = [self.server.add(wl) for wl in wls]
        self.dens = [(wl.rho_a, wl.rho_b) if wl.open_shell else (wl.rho, None) for wl in wls]
        self.run()  # every molecule resident, as in a service that has been up for a while

    def run(self):
        reqs = [self.server.submit(i, *d) for i, d in zip(self.ids, self.dens)]
        got = [self.server.wait(r, i) for r, i in zip(reqs, self.ids)]
        out = {"energies": np.array([g[0] for g in got]), "fock": [g[1] for g in got]}
        return dict(out, fock_b=[g[2] for g in got]) if got[0][2] is not None else out


def prepare(case, seed):
    wls = _molecules(case, seed)
    if case["call"] == "batch":
        return _Batch(wls)
    if case["call"] == "serve":
        return _Serve(wls)
    return _Single(case, wls[0])


def run(state):
    return state.run()


# ------------------------------------------------------------- work and tolerance
@functools.lru_cache(maxsize=None)
def _grid_sums(case_items):
    """Sums over the molecules of points, points x functions^2 and packed elements, of one seed's geometry."""
    n = nmm = packed = 0
    for wl in _molecules(dict(case_items), 1, density=False):
        for g in _groups(wl, weights=False):
            m = sum((1, 3, 6)[t] for t in g["types"])
            n += len(g["atom"])
            nmm += len(g["atom"]) * m * m
        packed += wl.basis.M * (wl.basis.M + 1) // 2
    return n, nmm, packed


def work(case):
    """Bytes: each grid point (position, weight), the densities and the results once. Flops: the two
    contractions, G = F D (and, for a gradient functional, the three derivatives of F) and K = F^T f F."""
    n, nmm, packed = _grid_sums(tuple(sorted((k, v) for k, v in case.items() if k != "name")))
    spins = 2 if case["open"] else 1
    fock = case["call"] in ("scf", "device", "batch", "serve")
    kinds = 2.5 if case["call"] == "batch" else (1 if case["iexch"] == 3 else 4)
    return {"bytes": 32.0 * n + 8.0 * packed * spins * (2 if fock else 1), "flops": 2.0 * nmm * spins * (kinds + fock)}


def tolerance(case):
    # relative 2-norm, about four times the largest difference seen from `exact`. Points of very low density
    # set it: there the gradient functional magnifies the error of the density. The default form keeps 42-bit
    # operands (Kohn-Sham matrices mostly 2e-12 off, up to 1.5e-9 with such points; forces 1.2e-9); the FP64
    # form's sums in another order (1e-15 off) meet the same points with 2^10 to 2^11 smaller errors
    if case["form"] == "fp64":
        return {"rel": 1e-11}
    return {"rel": 1e-8}


# ------------------------------------------------- the same result in plain torch, 64 bits
def _f32(x):
    return float(np.float32(x))


def _groups(wl, weights=True):
    """The grid's point groups (8-bohr cubes, atom spheres of the innermost 60 % of the shells) with their
    points, significant shells and Becke weights: g2g's default options."""
    dev = _cuda()
    pos = torch.tensor(wl.mol.pos, dtype=torch.float64, device=dev)
    bas, natom = wl.basis, wl.mol.natom
    nuc = bas.nuc.astype(np.int64) - 1
    lcs, frac, mfe, ns = 8.0, 0.6, 10, wl.n_rad
    rm = torch.tensor(W.rm_table()[wl.mol.Z], device=dev)
    e, wang = (torch.tensor(np.ascontiguousarray(v), device=dev) for v in g2g.angular_tables(wl.n_ang))
    a = np.where(np.arange(bas.a.shape[1])[None] < bas.ncont[:, None], bas.a, np.inf)
    amin = a.min(axis=1)  # smallest exponent of each function
    amin_z = {z: min(amin[i] for i in range(bas.M) if wl.mol.Z[nuc[i]] == z) for z in set(wl.mol.Z.tolist())}
    reach = torch.tensor([2.0 * math.sqrt(mfe / amin_z[z]) for z in wl.mol.Z.tolist()], device=dev)[:, None]
    x0, x1 = (pos - reach).min(0).values, (pos + reach).max(0).values
    size = torch.ceil((x1 - x0) / lcs).long()
    # points: Gauss-Chebyshev radial shells on Becke's mapping times the directions
    t0 = math.pi / (ns + 1)
    x = torch.cos(t0 * torch.arange(1, ns + 1, dtype=torch.float64, device=dev))
    r = rm[:, None] * (1.0 + x) / (1.0 - x)
    wr = t0 * torch.sin(t0 * torch.arange(1, ns + 1, dtype=torch.float64, device=dev)) * r * r * rm[:, None] * 2.0 / (1.0 - x) ** 2
    p = pos[:, None, None] + e[None, None] * r[:, :, None, None]
    w = wr[:, :, None] * wang[None, None]
    inc = math.ceil(frac * ns)
    sphere = (torch.arange(ns, device=dev) >= ns - inc)[None, :, None].expand(natom, ns, wl.n_ang)
    atom = torch.arange(natom, device=dev)[:, None, None].expand(natom, ns, wl.n_ang)
    inside = ((p >= x0) & (p <= x1)).all(-1)
    p, w, atom, sphere = p[inside], w[inside], atom[inside], sphere[inside]
    cube = torch.floor((p - x0) / lcs).long()
    ncubes = int(size.prod())
    key = torch.where(sphere, ncubes + atom, (cube[:, 0] * size[1] + cube[:, 1]) * size[2] + cube[:, 2])
    key, order = torch.sort(key, stable=True)
    p, w, atom = p[order], w[order], atom[order]
    keys, counts = torch.unique_consecutive(key, return_counts=True)
    # squared distance of every group's box or sphere to every atom
    idx = torch.stack([keys // (size[1] * size[2]), (keys // size[2]) % size[1], keys % size[2]], 1)
    lo = (x0 + idx * lcs)[:, None]
    gap = torch.clamp(lo - pos[None], min=0) + torch.clamp(pos[None] - (lo + lcs), min=0)
    xs = math.cos(t0 * (ns - inc + 1))
    sr = rm * (1.0 + xs) / (1.0 - xs)
    own = torch.clamp(keys - ncubes, min=0)
    sgap = torch.clamp(torch.linalg.norm(pos[None] - pos[own][:, None], dim=-1) - sr[own][:, None], min=0)
    d2 = torch.where((keys >= ncubes)[:, None], sgap * sgap, (gap * gap).sum(-1)).cpu().numpy()
    # shells and the bound of each: exponent times squared distance (s), a distance (p, d)
    first = np.array([f for f in range(bas.M) if f < bas.nshell[0]
                      or (f < bas.nshell[0] + bas.nshell[1] and (f - bas.nshell[0]) % 3 == 0)
                      or (f >= bas.nshell[0] + bas.nshell[1] and (f - bas.nshell[0] - bas.nshell[1]) % 6 == 0)])
    types = bas.lmom[first]
    keep = np.empty((len(keys), len(first)), bool)
    for q, f in enumerate(first):
        z = amin[f]
        dist2 = d2[:, nuc[f]]
        if types[q] == 0:
            keep[:, q] = z * dist2 < mfe - math.log((2.0 * z / math.pi) ** 3) / 4
            continue
        norm = math.sqrt((2.0 * z / math.pi) ** 3 * 4.0 * z)
        if types[q] == 1:
            norm = math.sqrt(norm)
        s, delta = 1.0, 1.0
        while delta > 0.1:
            s1 = math.sqrt((mfe - math.log(norm) + types[q] * math.log(s)) / z)
            delta, s = abs(s - s1), s1
        keep[:, q] = np.sqrt(dist2) < s
    adj = rm[:, None] / rm[None]
    adj = (adj - 1.0) / (adj + 1.0)
    adj = adj / (adj * adj - 1.0)
    apart = torch.cdist(pos, pos, compute_mode="donot_use_mm_for_euclid_dist")
    out, at = [], 0
    for g, n in enumerate(counts.tolist()):
        sel = slice(at, at + n)
        at += n
        shells = np.nonzero(keep[g])[0]
        if len(shells) == 0 and int(keys[g]) < ncubes:
            continue
        grp = dict(p=p[sel], w=w[sel], atom=atom[sel], first=first[shells], types=types[shells])
        if weights:
            grp["w"] = grp["w"] * _becke(grp["p"], grp["atom"], np.unique(nuc[grp["first"]]), pos, adj, apart)
        out.append(grp)
    return out


def _becke(p, atom, nucs, pos, adj, apart):
    """Fuzzy-cell weight of each point's atom over the group's nuclei, with the atomic-size adjustment."""
    nl = torch.tensor(nucs, device=p.device)
    out = torch.empty(len(p), dtype=torch.float64, device=p.device)
    step = max(1, int(2e7) // max(1, len(nucs) ** 2))

    def cut(u, aa):
        u = u + aa * (1.0 - u * u)
        for _ in range(3):
            u = 1.5 * u - 0.5 * (u * u * u)
        return 0.5 * (1.0 - u)

    for i in range(0, len(p), step):
        q, at = p[i:i + step], atom[i:i + step]
        d = torch.linalg.norm(q[:, None] - pos[nl][None], dim=-1)
        ap = apart[nl][:, nl] + torch.eye(len(nucs), device=p.device)
        s = cut((d[:, :, None] - d[:, None, :]) / ap, adj[nl][:, nl])
        s[:, torch.arange(len(nucs)), torch.arange(len(nucs))] = 1.0
        cells = s.prod(-1)
        mine = at[:, None] == nl[None]
        da = torch.linalg.norm(q - pos[at], dim=-1)
        far = torch.where(mine, torch.ones_like(d), apart[at][:, nl])
        alone = cut((da[:, None] - d) / far, adj[at][:, nl]).prod(-1)
        pa = torch.where(mine.any(-1), (cells * mine).sum(-1), alone)
        total = cells.sum(-1)
        out[i:i + step] = torch.where(total == 0, torch.zeros_like(pa), pa / total)
    return out


_COMP = {0: [(0, 0, 0)], 1: [(1, 0, 0), (0, 1, 0), (0, 0, 1)],
         2: [(2, 0, 0), (1, 1, 0), (0, 2, 0), (1, 0, 1), (0, 1, 1), (0, 0, 2)]}
_HESS = [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]


def _basis(wl, pos, q, first, types):
    """(F, gradient, second derivatives) of a group's functions at points q, their indices and atoms."""
    bas, dev = wl.basis, q.device
    f = torch.tensor(first, device=dev)
    nuc = torch.tensor(bas.nuc.astype(np.int64) - 1, device=dev)[f]
    a, c = (torch.tensor(v, device=dev)[f] for v in (bas.a, bas.c))
    nc = torch.tensor(bas.ncont.astype(np.int64), device=dev)[f]
    r = q[:, None] - pos[nuc][None]
    d2 = (r * r).sum(-1)
    t, tg, th = (torch.zeros_like(d2) for _ in range(3))
    for k in range(int(nc.max())):
        z = a[:, k] * d2
        v = torch.where((z > 70.0) | (k >= nc), torch.zeros_like(z), torch.exp(-z) * c[:, k])
        t, tg, th = t + v, tg + v * a[:, k], th + v * a[:, k] ** 2
    shell, lx, scale, glob = [], [], [], []
    for s, (f0, ty) in enumerate(zip(first, types)):
        for k, l in enumerate(_COMP[int(ty)]):
            shell.append(s)
            lx.append(l)
            scale.append(1.0 / math.sqrt(3.0) if max(l) == 2 else 1.0)
            glob.append(int(f0) + k)
    sh, l = torch.tensor(shell, device=dev), torch.tensor(lx, device=dev)
    sc = torch.tensor(scale, dtype=torch.float64, device=dev)
    r, t, tg, th = r[:, sh], t[:, sh] * sc, tg[:, sh] * sc, th[:, sh] * sc
    one = torch.ones_like(r)
    pw = torch.where(l == 0, one, torch.where(l == 1, r, r * r))
    dp = torch.where(l == 0, 0 * one, torch.where(l == 1, one, 2 * r))
    d2p = torch.where(l == 2, 2 * one, 0 * one)

    def mono(which):  # product over the axes of x^l, its first (1) or second (2) derivative
        m = torch.ones_like(t)
        for ax in range(3):
            m = m * (pw, dp, d2p)[which[ax]][..., ax]
        return m

    P = mono((0, 0, 0))
    Pa = [mono(tuple(int(b == ax) for b in range(3))) for ax in range(3)]
    F = P * t
    dF = [Pa[ax] * t - 2.0 * r[..., ax] * P * tg for ax in range(3)]
    H = []
    for x, y in _HESS:
        Pab = mono(tuple(int(b == x) + int(b == y) for b in range(3)))
        cross = r[..., y] * Pa[x] + r[..., x] * Pa[y] + (P if x == y else 0.0)
        H.append(Pab * t - 2.0 * cross * tg + 4.0 * r[..., x] * r[..., y] * P * th)
    return F, dF, H, torch.tensor(glob, device=dev), nuc[sh]


def _lda(rho):
    """Slater exchange with Vosko-Wilk-Nusair correlation: energy per electron and potential."""
    ok = rho != 0
    y = torch.where(ok, rho, torch.ones_like(rho)).abs().pow(1 / 3) * torch.sign(torch.where(ok, rho, torch.ones_like(rho)))
    A1, B1, X0, Q, A16, T4 = 0.03109205, 3.72744, -0.10498, 6.15199066246304849, 0.005182008333, -0.0311676086789438
    rs = 0.620350490899400087 / y
    x = torch.sqrt(rs)
    X, t1 = rs + B1 * x + 12.9352, 2.0 * x + B1
    t2, t3, t5 = torch.log(X), torch.atan(Q / t1), (B1 * x + 25.8704) / x
    ec = A1 * (2.0 * torch.log(x) - t2 + 1.21178337371132 * t3
               - T4 * (2.0 * torch.log(x - X0) - t2 + 1.14352579286644 * t3))
    vc = ec - A16 * x * (t5 / X - 14.90976 / (t1 * t1 + 37.8469891110325) * 1.0329232240928
                         - T4 * (2.0 / (x - X0) - t1 / X))
    z = torch.zeros_like(rho)
    return torch.where(ok, -0.738558766382022447 * y + ec, z), torch.where(ok, -0.984745021842697 * y + vc, z)


_PW = {1: (0.0310907, 0.21370, 7.5957, 3.5876, 1.6382, 0.49294),
       2: (0.01554535, 0.20548, 14.1189, 6.1977, 3.3662, 0.62517),
       3: (0.0168869, 0.11125, 10.357, 3.6231, 0.88026, 0.49671)}
_AX, _UM, _UK, _UL = (_f32(v) for v in (-0.738558766382022405884230032680836, 0.2195149727645171, 0.804, 0.273028573090195))
_BETA, _PI32 = _f32(0.06672455060314922), _f32(29.608813203268075856503472999628)
_F43, _F13, _FM16 = _f32(4.0 / 3.0), _f32(1.0 / 3.0), _f32(-1.0 / 6.0)


def _pw92(which, rtrs):
    """G(rs) and its derivative of Perdew and Wang's interpolation, with single-precision parameters."""
    a0, a1, b1, b2, b3, b4 = (_f32(v) for v in _PW[which])
    q0 = -2.0 * a0 * (1.0 + a1 * rtrs * rtrs)
    q1 = 2.0 * a0 * rtrs * (b1 + rtrs * (b2 + rtrs * (b3 + b4 * rtrs)))
    q2 = torch.log(1.0 + 1.0 / q1)
    q3 = a0 * (b1 / rtrs + 2.0 * b2 + rtrs * (3.0 * b3 + 4.0 * b4 * rtrs))
    return q0 * q2, -2.0 * a0 * a1 * q2 - q0 * q3 / (q1 * (1.0 + q1))


def _invariants(g, h):
    """|grad rho|, grad rho . H grad rho / |grad rho| and the Laplacian."""
    n2 = torch.clamp((g * g).sum(0), min=np.finfo(np.float64).tiny)
    d = torch.sqrt(n2)
    dg = (g[0] ** 2 * h[0] + g[1] ** 2 * h[1] + g[2] ** 2 * h[2]
          + 2 * (g[0] * g[1] * h[3] + g[0] * g[2] * h[4] + g[1] * g[2] * h[5])) / d
    return d, dg, h[0] + h[1] + h[2]


def _pbe_x(rho13, s, u, v):
    ex, p0 = _AX * rho13, 1.0 + _UL * s * s
    fx = 1.0 + _UK - _UK / p0
    Fs = 2.0 * _UM / (p0 * p0)
    Fss = -4.0 * _UL * s * Fs / p0
    return ex * fx, ex * (_F43 * fx - (u - _F43 * s ** 3) * Fss - v * Fs)


def _pbe_h(t, B, G3, bd, DELTA):
    """The gradient correction H and the derivatives both spin cases share (times G^3)."""
    t2, B2 = t * t, B * B
    t4, t6 = t2 * t2, t2 ** 3
    Q4, Q5, Q9 = 1.0 + B * t2, 1.0 + B * t2 + B2 * t2 * t2, 1.0 + 2.0 * B * t2
    Q8 = Q5 * Q5 + DELTA * Q4 * Q5 * t2
    H = G3 * bd * torch.log(1.0 + DELTA * Q4 * t2 / Q5)
    hB = -_BETA * G3 * B * (t6 / Q8) * (2.0 + B * t2)
    f0, f1 = 2.0 * DELTA - 6.0 * B, Q5 * Q9 + Q4 * Q9 * Q9
    hBT = 2.0 * _BETA * G3 * t4 * ((Q4 * Q5 * f0 - DELTA * f1) / Q8) / Q8
    hT = 2.0 * _BETA * G3 * (Q9 / Q8)
    f2 = Q4 * Q5 + B * t2 * (Q4 * Q9 + Q5)
    f3 = 2.0 * B * Q5 * Q9 + DELTA * f2
    hTT = 4.0 * _BETA * G3 * t * (2.0 * B / Q8 - ((Q9 / Q8) * f3) / Q8)
    return H, hB, hBT, hT, hTT


def _pbe_closed(rho0, g, h):
    ok = rho0 >= 1e-18
    rho = torch.where(ok, rho0, torch.ones_like(rho0))
    d, dg, lap = _invariants(g, h)
    rho13 = rho.pow(1 / 3)
    fk = _PI32 ** (1 / 3) * rho13
    k2 = 2.0 * fk
    ex, vx = _pbe_x(rho13, d / (k2 * rho), dg / (k2 ** 3 * rho * rho), lap / (k2 * k2 * rho))
    z = torch.zeros_like(rho)
    has_x = rho * rho > 1e-18
    ex, vx = torch.where(has_x, ex, z), torch.where(has_x, vx, z)
    rs = (3.0 / (4.0 * math.pi * rho)).pow(1 / 3)
    ks = 2.0 * torch.sqrt(4.0 * fk / math.pi)
    t, uu, vv = d / (ks * rho), dg / (rho * rho * ks ** 3), lap / (rho * ks * ks)
    ec, ers = _pw92(1, torch.sqrt(rs))
    DELTA = _f32(2.14612633996736)
    B = DELTA / (torch.exp(-ec * _f32(32.1639684429148)) - 1.0)
    H, hB, hBT, hT, hTT = _pbe_h(t, B, 1.0, _BETA / DELTA, DELTA)
    bec = B * B * (DELTA / B + 1.0) / _BETA
    comm = H - rs / 3.0 * hB * bec * ers + rs / 3.0 * t * t * hBT * bec * ers + t * t * hT / 6.0 + 7.0 * t ** 3 * hTT / 6.0
    vc = ec - rs * _F13 * ers + comm - uu * hTT - vv * hT
    has_c = rho >= 1e-12
    e = ex + torch.where(has_c, ec + H, z)
    return torch.where(ok, e, z), torch.where(ok, vx + torch.where(has_c, vc, z), z)


def _pbe_open(ra0, rb0, ga, gb, ha, hb):
    ok = (ra0 > 1e-18) | (rb0 > 1e-18)
    one, z = torch.ones_like(ra0), torch.zeros_like(ra0)
    ra, rb = torch.where(ok, ra0, one), torch.where(ok, rb0, one)
    ex, vx, inv = [], [], []
    for r, g, h in ((ra, ga, ha), (rb, gb, hb)):
        d, dg, lap = _invariants(g, h)
        inv.append((d, dg, lap))
        has = 2.0 * r > 1e-18
        two = torch.where(has, 2.0 * r, one)
        k2 = 2.0 * _PI32 ** (1 / 3) * two.pow(1 / 3)
        e, v = _pbe_x(two.pow(1 / 3), 2.0 * d / (two * k2), 4.0 * dg / (two * two * k2 ** 3), 2.0 * lap / (two * k2 * k2))
        ex.append(torch.where(has, e, z))
        vx.append(torch.where(has, v, z))
    rho = ra + rb
    e = ex[0] * (ra / rho) + ex[1] * (rb / rho)
    has_c = rho >= 1e-13
    d, dg, _ = _invariants(ga + gb, ha + hb)
    zet = torch.clamp((ra - rb) / rho, -1.0, 1.0)
    zp, zm = 1.0 + zet, 1.0 - zet
    cp, cm = zp.pow(1 / 3), zm.pow(1 / 3)
    G = (cp * cp + cm * cm) / 2.0
    pi = _f32(math.pi)
    fk = _PI32 ** (1 / 3) * rho.pow(1 / 3)
    rs = (9.0 * pi / 4.0) ** (1 / 3) / fk
    ks = 2.0 * torch.sqrt(4.0 * fk / pi) * G
    t, uu = d / (ks * rho), dg / (rho * rho * ks ** 3)
    vv = (inv[0][2] + inv[1][2]) / (rho * ks * ks)
    ww = (inv[0][0] ** 2 - inv[1][0] ** 2 - zet * d * d) / (rho * rho * ks * ks)
    rt = torch.sqrt(rs)
    (eu, eurs), (ep, eprs), (al, alrs) = (_pw92(k, rt) for k in (1, 2, 3))
    z2, z3, z4 = zet ** 2, zet ** 3, zet ** 4
    gam = 2.0 ** (4.0 / 3.0) - 2.0
    F = (zp * cp + zm * cm - 2.0) / gam
    fzz = 8.0 / (9.0 * gam)
    ec = eu * (1.0 - F * z4) + ep * F * z4 - al * F * (1.0 - z4) / fzz
    ecrs = eurs * (1.0 - F * z4) + eprs * F * z4 - alrs * F * (1.0 - z4) / fzz
    fz = _F43 * (cp - cm) / gam
    ecz = 4.0 * z3 * F * (ep - eu + al / fzz) + fz * (z4 * ep - z4 * eu - (1.0 - z4) * al / fzz)
    comm = ec - rs * ecrs / 3.0 - zet * ecz
    vca, vcb = comm + ecz, comm - ecz
    GAMMA = _f32(0.03109069086965489503494086371273)
    DELTA, eta, G3 = _BETA / GAMMA, _f32(1e-12), G ** 3
    B = DELTA / (torch.exp(-ec / (G3 * GAMMA)) - 1.0)
    H, hB, hBT, hT, hTT = _pbe_h(t, B, G3, _BETA / DELTA, DELTA)
    gz = ((zp * zp + eta).pow(_FM16) - (zm * zm + eta).pow(_FM16)) / 3.0
    fac = DELTA / B + 1.0
    bg, bec = -3.0 * B * B * ec * fac / (_BETA * G3 * G), B * B * fac / (_BETA * G3)
    hz = 3.0 * gz * H / G + hB * (bg * gz + bec * ecz)
    hzt = 3.0 * gz * hT / G + hBT * (bg * gz + bec * ecz)
    comm = (H - rs / 3.0 * hB * bec * ecrs + rs / 3.0 * t * t * hBT * bec * ecrs + t * t * hT / 6.0
            + 7.0 * t ** 3 * hTT / 6.0)
    pref = hz - gz * t * t * hT / G
    comm = comm - pref * zet - uu * hTT - vv * hT - ww * (hzt - gz * (2.0 * hT + t * hTT) / G)
    e = e + torch.where(has_c, ec + H, z)
    va, vb = vx[0] + torch.where(has_c, vca + comm + pref, z), vx[1] + torch.where(has_c, vcb + comm - pref, z)
    return torch.where(ok, e, z), torch.where(ok, va, z), torch.where(ok, vb, z)


def _build(wl, forces):
    """(E_xc, packed Kohn-Sham matrices, forces) of one molecule in FP64."""
    dev, M = _cuda(), wl.basis.M
    pos = torch.tensor(wl.mol.pos, dtype=torch.float64, device=dev)
    r, c = torch.triu_indices(M, M, device=dev)
    dens = []
    for v in ([wl.rho_a, wl.rho_b] if wl.open_shell else [wl.rho]):
        D = torch.zeros(M, M, dtype=torch.float64, device=dev)
        D[r, c] = torch.tensor(v, device=dev) / 2.0
        dens.append(D + D.T)
    K = [torch.zeros(M, M, dtype=torch.float64, device=dev) for _ in dens]
    frc = torch.zeros(wl.mol.natom, 3, dtype=torch.float64, device=dev)
    energy = torch.zeros((), dtype=torch.float64, device=dev)
    for grp in _groups(wl):
        if len(grp["first"]) == 0:
            continue
        step = 8192
        for i in range(0, len(grp["w"]), step):
            w = grp["w"][i:i + step]
            F, dF, H, f, at = _basis(wl, pos, grp["p"][i:i + step], grp["first"], grp["types"])
            rho, grad, hess, G = [], [], [], []
            for D in dens:
                d = D[f][:, f]
                g0 = F @ d
                G.append(g0)
                rho.append((F * g0).sum(1))
                if wl.iexch != 3:
                    ga = [x @ d for x in dF]
                    grad.append(torch.stack([2.0 * (x * g0).sum(1) for x in dF]))
                    hess.append(torch.stack([2.0 * (H[k] * g0 + dF[x] * ga[y]).sum(1) for k, (x, y) in enumerate(_HESS)]))
            if wl.iexch == 3:
                e, *v = _lda(rho[0])
            elif wl.open_shell:
                e, *v = _pbe_open(rho[0], rho[1], grad[0], grad[1], hess[0], hess[1])
            else:
                e, *v = _pbe_closed(rho[0], grad[0], hess[0])
            energy += (sum(rho) * w * e).sum()
            for s in range(len(dens)):
                wv = (w * v[s])[:, None]
                K[s][f[:, None], f[None]] += F.T @ (wv * F)
                if forces:
                    x = torch.stack([(wv * G[s] * d).sum(0) for d in dF], 1)
                    frc.index_add_(0, at, -2.0 * x)
    return energy.item(), [k[r, c].cpu().numpy() for k in K], frc.cpu().numpy()


def exact(case, seed):
    wls = _molecules(case, seed)
    if case["call"] in ("batch", "serve"):
        got = [_build(wl, False) for wl in wls]
        out = {"energies": np.array([g[0] for g in got]), "fock": [g[1][0] for g in got]}
        return dict(out, fock_b=[g[1][1] for g in got]) if len(got[0][1]) == 2 else out
    e, K, forces = _build(wls[0], case["call"] in ("forces", "md"))
    if case["call"] in ("forces", "md"):
        return {"energy": np.array([e]), "forces": forces}
    out = {"energy": np.array([e])}
    if case["call"] != "energy":
        out["fock"] = K[0]
        if len(K) == 2:
            out["fock_b"] = K[1]
    return out
