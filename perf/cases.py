"""Workloads that a program on this engine runs, with the means to time and check them.

Every case is one wave-function set (or a batch of them) of a synthetic system
of the kinds that the tests, the benchmark and the serving workload use: bulk
silicon from 2 to 128 atoms, water clusters and the 32-molecule water box, on
the FFT grids of the reference's rule or the fixed ones of the benchmark.

  step         CP steps with moving nuclei between two outputs of the wave functions
  hpsi         WAVES$HPSI, as a host that steps routine by routine calls it
  projections  WAVES$PROJECTIONS with PROJ read back for the one-centre densities
  force        WAVES$FORCE
  density      WAVES$RHO with the density read back
  single       a single point: new coefficients and positions, Gram-Schmidt, energies, forces
  batch        two CP steps of many small systems by one graph launch

listed() are the timed cases, draw() gives more of the same ranges, prepare()
what a program holds before the call, run() one pass through the public entry
points, exact() the same outputs from plain torch in 64 bits.
"""
import ctypes
import functools
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "cp-paw_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import cuwaves  # noqa: E402
from cuwaves import systems  # noqa: E402

PRECISION = {"fp64": cuwaves.CUW_PREC_FP64, "mixed": cuwaves.CUW_PREC_MIXED}
FRICTION = 0.05  # damped run: wave functions relax while the nuclei move
_D = ctypes.POINTER(ctypes.c_double)


def _case(name, op, kind, size, precision, ry=30.0, grid="reference", nb=0, steps=0, sets=1):
    """kind Si: `size` is the number of cubic cells along each axis, e.g. "2x2x4",
    or the number of atoms of a small cell; kind H2O: molecules of a cluster, or
    "box32".  nb: bands, 0 = all valence bands.  grid: "reference" rule, "sphere"
    (the smallest that holds the wave-function sphere) or points per axis."""
    c = dict(op=op, kind=kind, size=size, precision=precision, ry=ry, grid=grid, nb=nb, steps=steps, sets=sets)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a two-atom cell: every launch is tiny, the step is latency
        _case("step_si2_fp64", "step", "Si", "2", "fp64", grid="sphere", steps=4),
        # the cubic Si8 cell of the CPU-runnable configuration
        _case("step_si8_mixed", "step", "Si", "1x1x1", "mixed", grid="32", steps=4),
        # the benchmark's system, on either precision path
        _case("step_si64_fp64", "step", "Si", "2x2x2", "fp64", grid="64", steps=4),
        _case("step_si64_mixed", "step", "Si", "2x2x2", "mixed", grid="64", steps=4),
        # 32 water molecules: two species, fewer projectors per band, a 72^3 grid
        _case("step_h2o32_mixed", "step", "H2O", "box32", "mixed", ry=40.0, grid="72", steps=4),
        # the largest system of the serving mix
        _case("step_si128_fp64", "step", "Si", "2x2x4", "fp64", steps=2),
        # a host that steps routine by routine; reference-rule 56^3 grid
        _case("hpsi_si64_mixed", "hpsi", "Si", "2x2x2", "mixed"),
        # ragged: 4 molecules in vacuum, many plane waves for 16 bands and 48 projectors
        _case("projections_h2o4_fp64", "projections", "H2O", "4", "fp64", ry=40.0),
        # forces of an uneven cell with 118 of its 192 valence bands
        _case("force_si96_fp64", "force", "Si", "2x2x3", "fp64", nb=118),
        # the density that the host's potential needs once per step
        _case("density_h2o32_fp64", "density", "H2O", "box32", "fp64", ry=40.0, grid="72"),
        # a serving request's single point
        _case("single_h2o8_mixed", "single", "H2O", "8", "mixed", ry=40.0),
        # many small systems of uneven size by one launch
        _case("batch16_mixed", "batch", "mix", "16", "mixed", grid="sphere", steps=2, sets=16),
    ]


def draw(rng):
    largest = max(_weight(c) for c in listed())
    while True:
        op = rng.choice(["step", "step", "step", "hpsi", "projections", "force", "density", "single", "batch"])
        precision = rng.choice(["fp64", "mixed"])
        if op == "batch":
            n = rng.randint(2, 24)
            return _case(None, "batch", "mix", str(n), precision, grid="sphere", steps=2, sets=n)
        if rng.random() < 0.65:
            ry = round(rng.uniform(22.0, 36.0), 1)
            if rng.random() < 0.4:
                c = _case(None, op, "Si", str(2 * rng.randint(1, 8)), precision, ry=ry)
            else:
                cells = sorted(rng.choice([1, 1, 2, 2, 3]) for _ in range(3))
                atoms = 8 * cells[0] * cells[1] * cells[2]
                nb = 0 if rng.random() < 0.5 else 2 * rng.randint(max(1, atoms // 2), atoms)
                c = _case(None, op, "Si", "x".join(map(str, cells)), precision, ry=ry, nb=nb)
        else:
            n = max(1, int(round(math.exp(rng.uniform(0.0, math.log(16.0))))))
            c = _case(None, op, "H2O", str(n), precision, ry=round(rng.uniform(30.0, 45.0), 1))
        if op == "step":
            c["steps"] = rng.choice([1, 2, 4])
        if _weight(c) <= largest:
            return c


# -- systems ------------------------------------------------------------------


@functools.lru_cache(maxsize=None)
def _mix():
    return systems.config_batch_mix(64)


@functools.lru_cache(maxsize=64)
def _system(kind, size, ry, grid, nb, index=0):
    """The geometry and tables of a case: what does not depend on the seed."""
    if kind == "mix":
        sy = _mix()[index]
    elif kind == "Si" and "x" in size:
        sy = systems.si_supercell(*(int(k) for k in size.split("x")), disp=0.05, seed=1, epw_psi_ry=ry)
    elif kind == "Si":
        sy = systems.si_small(int(size), epw_psi_ry=ry)
    elif size == "box32":
        sy = systems.water_box(32, epw_psi_ry=ry)
    else:
        sy = systems.water_cluster(int(size), epw_psi_ry=ry)
    if kind != "mix":
        sy.grid = (0, 0, 0) if grid == "reference" else systems.psi_grid(sy) if grid == "sphere" else (int(grid),) * 3
        sy.nb = nb or sy.nb
    return systems.build_inputs(sy, psi_init="zero")


def _systems(case):
    return [_system(case["kind"], case["size"] if case["op"] != "batch" else "", case["ry"], case["grid"], case["nb"],
                    i if case["op"] == "batch" else 0) for i in range(case["sets"])]


def _inputs(case, seed):
    """Seeded inputs of every set: displaced positions, one-centre Hamiltonians,
    Lagrange multipliers for the single routines, and coefficients: orthonormal
    ones, as a run reads them from its restart file, or raw ones for a single point."""
    out = []
    for i, base in enumerate(_systems(case)):
        rng = np.random.default_rng([seed, i])
        inp = dict(base)
        shape = (inp["nbh"], inp["ngl"])
        inp["psi"] = rng.standard_normal(shape + (2,)).view(np.complex128)[..., 0] * np.exp(-inp["g2"] / 8.0)
        inp["r0"] = inp["r0"] + rng.uniform(-0.02, 0.02, inp["r0"].shape)
        n = rng.uniform(-0.02, 0.02, inp["dh"].shape)
        inp["dh"] = inp["dh"] + 0.5 * (n + n.transpose(0, 2, 1)) * (inp["dh"] != 0)
        lam = rng.standard_normal((inp["nb"],) * 2)
        inp["rlam0"] = -0.2 * np.eye(inp["nb"]) + 0.01 * (lam + lam.T)
        inp["annee"] = FRICTION
        if case["op"] != "single":
            s = _Plain(inp)
            s.orthonormalise()
            inp["psi"] = s.super(s.phi).numpy()
        out.append(inp)
    return out


def _sizes(inp):
    npro = sum(sum(2 * l + 1 for l in inp["lox"][s - 1]) for s in inp["isp"].tolist())
    return inp["ngl"], inp["nb"], npro, inp["grid"][0] * inp["grid"][1] * inp["grid"][2]


def _work_of(inp, op, steps):
    """Bytes and flops of one set at the Gamma point, where each +-G pair of a
    band is one real contraction index twice: <p|psi> costs 2 NGL NPRO NB."""
    ngl, nb, npro, nr = _sizes(inp)
    psi = 8.0 * ngl * nb
    contract, overlap, fft = 2.0 * ngl * npro * nb, 2.0 * ngl * nb * nb, 2.5 * nr * math.log2(nr) * nb
    small = 16.0 * npro * nb / 2
    if op == "projections":
        return psi + small, contract
    if op == "hpsi":
        return 2 * psi + small + 8.0 * nr, contract + 2 * fft
    if op == "force":
        return psi + small + 8.0 * nb * nb, contract
    if op == "density":
        return psi + 8.0 * nr, fft
    if op == "single":  # Gram-Schmidt: projections, half a Gram matrix, rotation; then the single point
        return 2 * psi + 8.0 * nr, 4 * contract + 1.5 * overlap + 2 * fft
    # step: H and O back-projections, two projections, force; three Gram matrices
    # (two symmetric) and the rotation; PSI0 and PSIM read, PSI(+) written
    return steps * (3 * psi + 8.0 * nr) + psi, steps * (5 * contract + 3 * overlap + 2 * fft)


def work(case):
    parts = [_work_of(inp, case["op"], case["steps"]) for inp in _systems(case)]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


def _weight(case):
    """Relative cost of a case, for draw()."""
    return work(case)["flops"] * (2.0 if case["precision"] == "fp64" else 1.0)


def tolerance(case):
    """Four times what the path differs by from exact(), at most, over the ranges."""
    step = case["op"] in ("step", "batch", "single")
    if case["precision"] == "fp64":
        # single routines 7e-15; a step stops at 1e-8 in the overlap, which moves
        # the Lagrange multipliers and with them the forces by up to 8e-8
        return {"rel": 3e-7 if step else 3e-14}
    # single routines 4e-7 (forces of many bands), a step's forces 2.5e-6
    return {"rel": 1e-5 if step else 2e-6}


# -- one pass -------------------------------------------------------------------


def prepare(case, seed):
    inps = _inputs(case, seed)
    prec = PRECISION[case["precision"]]
    sets = [cuwaves.open_waves(inp, precision=prec).setup() for inp in inps]
    state = {"op": case["op"], "steps": case["steps"], "sets": sets, "inputs": inps,
             "psi": [torch.empty((i["nbh"], i["ngl"]), dtype=torch.complex128, pin_memory=True) for i in inps]}
    if case["op"] == "single":
        state["new"] = torch.from_numpy(np.ascontiguousarray(inps[0]["psi"])).pin_memory()
        return state
    for w in sets:
        w.projections()
        if case["op"] in ("step", "batch"):
            w.cp_step(move_atoms=True)  # a run under way: eigenbasis and Lagrange history exist
    if case["op"] == "batch":
        share = max(16, torch.cuda.get_device_properties(0).multi_processor_count // len(sets))
        for w in sets:
            w.set_option(cuwaves.CUW_OPT_SM_SHARE, share)
        state["batch"] = cuwaves.Batch(sets)
    elif case["op"] in ("hpsi", "projections", "force", "density"):
        sets[0].set_rlam0(inps[0]["rlam0"])
    return state


def _psi(state, which=cuwaves.CUW_PSI0):
    """The wave functions of every set in page-locked host buffers."""
    download = cuwaves.engine()["download_psi"]
    for w, buf in zip(state["sets"], state["psi"]):
        if download(w.h, which, ctypes.cast(buf.data_ptr(), _D)):
            raise RuntimeError("download_psi failed")
    return list(state["psi"])


def run(state):
    op, w = state["op"], state["sets"][0]
    if op == "step":
        for _ in range(state["steps"]):
            out, force = w.cp_step(move_atoms=True)
        return {"energies": out[:4], "force": force, "psi": _psi(state)}
    if op == "batch":
        out = state["batch"].step(move_atoms=True)
        return {"energies": out[:, :, :4], "psi": _psi(state)}
    if op == "hpsi":
        w.hpsi()
        return {"hpsi": _psi(state, cuwaves.CUW_HPSI)}
    if op == "projections":
        w.projections()
        return {"proj": w.get_proj()}
    if op == "force":
        return {"force": w.force()}
    if op == "density":
        return {"rho": w.density()}
    inp = state["inputs"][0]
    if cuwaves.engine()["upload_psi"](w.h, cuwaves.CUW_PSI0, ctypes.cast(state["new"].data_ptr(), _D)):
        raise RuntimeError("upload_psi failed")
    w.reset_atoms(inp["r0"])
    w.gramschmidt(cuwaves.CUW_PSI0, inp["r0"])
    w.projections()
    out, force = w.etot()
    return {"energies": out, "force": force, "proj": w.get_proj()}


# -- the same in 64 bits --------------------------------------------------------


class _Plain:
    """One set in plain torch: the bands as real functions of r, phi (NGL, NB)
    complex with phi(-G) = conj(phi(G)), two per super wave function."""

    def __init__(self, inp):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.t = lambda x: torch.as_tensor(np.ascontiguousarray(x), device=dev)
        self.inp, self.omega = inp, inp["omega"]
        self.g, self.g2, self.mpsi = self.t(inp["gvec"]), self.t(inp["g2"]), self.t(inp["mpsi"])
        self.minus = self.t(inp["minusg"].astype(np.int64) - 1)
        self.f = self.t(inp["occ"])
        self.mass = self.t(inp["masses"])[:, None]
        isp = [s - 1 for s in inp["isp"].tolist()]
        first = np.cumsum([0] + inp["lnx"]).tolist()
        bare, ylm = self.t(inp["pro"]), self.t(inp["ylm"])
        table = []  # the radial and angular factors of a species' projectors
        for s in range(inp["nsp"]):
            cols = [bare[first[s] + ln] * ylm[l * l + m] * (-1j) ** l
                    for ln, l in enumerate(inp["lox"][s]) for m in range(2 * l + 1)]
            table.append(torch.stack(cols))
        self.radial = torch.cat([table[s] for s in isp])
        self.atom = self.t(np.concatenate([np.full(len(table[s]), a) for a, s in enumerate(isp)]))
        n = len(self.atom)
        self.dh = torch.zeros((n, n), dtype=torch.float64, device=dev)
        self.do = torch.zeros_like(self.dh)
        at = 0
        for a, s in enumerate(isp):
            k = len(table[s])
            self.dh[at:at + k, at:at + k] = self.t(inp["dh"][a, :k, :k].real.T)
            lm = [(ln, l, m) for ln, l in enumerate(inp["lox"][s]) for m in range(2 * l + 1)]
            for i, (n1, l1, m1) in enumerate(lm):
                for j, (n2, l2, m2) in enumerate(lm):
                    if (l1, m1) == (l2, m2):
                        self.do[at + i, at + j] = float(inp["dover"][s, n2, n1])
            at += k
        self.r0 = self.t(inp["r0"])
        self.rm = self.r0.clone()
        self.lam = torch.zeros((inp["nb"],) * 2, dtype=torch.float64, device=dev)
        self.lam_old = None
        psi = self.t(inp["psi"]).T
        back = psi[self.minus].conj()
        self.phi = torch.stack([(psi + back) / 2, (psi - back) / 2j], 2).reshape(len(self.g2), -1)
        self.old = self.phi

    def super(self, phi):
        return (phi[:, 0::2] + 1j * phi[:, 1::2]).T.contiguous().cpu()

    def projectors(self, r):
        return self.radial * torch.exp(-1j * (self.g @ r.T)).T[self.atom]

    def project(self, p, phi):
        return self.omega * (p.conj() @ phi).real

    def overlap(self, a, pa, b, pb):
        return self.omega * (a.real.T @ b.real + a.imag.T @ b.imag) + pa.T @ self.do @ pb

    def orthonormalise(self):
        p = self.projectors(self.r0)
        for _ in range(2):
            pr = self.project(p, self.phi)
            low = torch.linalg.cholesky(self.overlap(self.phi, pr, self.phi, pr))
            low = torch.linalg.inv(low).T
            self.phi = torch.complex(self.phi.real @ low, self.phi.imag @ low)

    def wave_on_grid(self, phi):
        nr = self.inp["grid"]
        ig = self.t(self.inp["igvec"].astype(np.int64))
        box = torch.zeros((phi.shape[1], nr[2], nr[1], nr[0]), dtype=torch.complex128, device=phi.device)
        self.at = (ig[:, 2] % nr[2], ig[:, 1] % nr[1], ig[:, 0] % nr[0])
        box[:, self.at[0], self.at[1], self.at[2]] = phi.T
        return torch.fft.ifftn(box, dim=(1, 2, 3), norm="forward")

    def density(self):
        rho = 0.0
        for k in range(0, self.phi.shape[1], 16):
            w = self.wave_on_grid(self.phi[:, k:k + 16]).real
            rho = rho + (self.f[k:k + 16, None, None, None] * w * w).sum(0)
        return rho

    def hamilton(self, p, pr):
        v = self.t(self.inp["v"])
        parts = []
        for k in range(0, self.phi.shape[1], 16):
            w = torch.fft.fftn(self.wave_on_grid(self.phi[:, k:k + 16]) * v, dim=(1, 2, 3), norm="forward")
            parts.append(w[:, self.at[0], self.at[1], self.at[2]].T)
        return torch.cat(parts, 1) + 0.5 * self.g2[:, None] * self.phi + p.T @ (self.dh @ pr).to(p.dtype)

    def force(self, p, pr, lam):
        d = self.f * (self.dh @ pr) - (self.do @ pr) @ (lam * (self.f[:, None] + self.f[None, :]) / 2)
        s = (1j * p * (self.phi @ d.T.to(p.dtype)).T.conj()).real
        out = torch.zeros_like(self.r0)
        return 2.0 * self.omega * out.index_add_(0, self.atom, s @ self.g)

    def energies(self, p, pr, h):
        etot = self.omega * (self.f * (self.phi.conj() * h).real.sum(0)).sum()
        return etot, 0.5 * self.omega * (self.g2[:, None] * self.f * self.phi.abs() ** 2).sum()

    def fictitious(self, dphi):
        return self.omega * (self.mpsi[:, None] * self.f * dphi.abs() ** 2).sum() / self.inp["delt"] ** 2

    def step(self):
        dt, fric = self.inp["delt"], 1.0 + self.inp["annee"]
        p = self.projectors(self.r0)
        pr = self.project(p, self.phi)
        f = self.force(p, pr, self.lam)
        h = self.hamilton(p, pr)
        etot, ekin = self.energies(p, pr, h)
        fict = self.fictitious(self.phi - self.old)
        rp = 2.0 * self.r0 - self.rm + dt * dt * f / self.mass
        scale = (dt * dt / fric / self.mpsi)[:, None]
        bar = 2.0 / fric * self.phi + (1.0 - 2.0 / fric) * self.old - scale * h
        chi = scale * (self.phi + p.T @ (self.do @ pr).to(p.dtype))
        p = self.projectors(rp)
        pb, pc = self.project(p, bar), self.project(p, chi)
        bb, cb, cc = self.overlap(bar, pb, bar, pb), self.overlap(chi, pc, bar, pb), self.overlap(chi, pc, chi, pc)
        lam = self.lam.clone()
        one = torch.eye(len(lam), dtype=lam.dtype, device=lam.device)
        e, u = torch.linalg.eigh(0.5 * (cb + cb.T))
        last = math.inf
        for _ in range(200):
            w = lam.T @ (cc @ lam + 2.0 * cb)
            w = 0.5 * (w + w.T) + bb - one
            off = float(w.abs().max())
            if off < 1e-14 or (off < 1e-11 and off >= last):
                break
            last = off
            lam = lam - u @ ((u.T @ w @ u) / (e[:, None] + e[None, :])) @ u.T
        new = bar + torch.complex(chi.real @ lam, chi.imag @ lam)
        fict = 0.5 * (fict + self.fictitious(self.phi - new))
        vel = (rp - self.rm) / (2.0 * dt)
        ion = 0.5 * (self.mass * vel * vel).sum()
        self.lam, self.lam_old = (lam if self.lam_old is None else 2.0 * lam - self.lam_old), lam
        self.old, self.phi = self.phi, new
        self.rm, self.r0 = self.r0, rp
        return [float(x) for x in (etot, ekin, fict, ion)], f.cpu()


def exact(case, seed):
    op = case["op"]
    sets = [_Plain(inp) for inp in _inputs(case, seed)]
    s = sets[0]
    if op == "single":
        s.orthonormalise()
    if op in ("step", "batch"):
        energies = []
        for x in sets:
            x.step()
            energies.append([])
            for _ in range(case["steps"]):
                e, f = x.step()
                energies[-1].append(e)
        psi = [x.super(x.phi) for x in sets]
        if op == "batch":
            return {"energies": np.array(energies), "psi": psi}
        return {"energies": np.array(energies[0][-1]), "force": f, "psi": psi}
    if op == "density":
        return {"rho": s.density().cpu()}
    p = s.projectors(s.r0)
    pr = s.project(p, s.phi)
    proj = torch.complex(pr[:, 0::2], pr[:, 1::2]).cpu()
    if op == "projections":
        return {"proj": proj}
    if op == "force":
        return {"force": s.force(p, pr, s.t(s.inp["rlam0"])).cpu()}
    h = s.hamilton(p, pr)
    if op == "hpsi":
        return {"hpsi": [s.super(h)]}
    etot, ekin = s.energies(p, pr, h)
    return {"energies": np.array([float(etot), float(ekin)]), "force": s.force(p, pr, s.lam).cpu(), "proj": proj}
