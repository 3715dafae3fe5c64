"""The folded contractions (fold.cu, and tc.cu on the mixed path) at the edges
of their tiles, and the complex kernels that take a G set whose tables lack the
parity of real-valued projectors, against the oracle."""
import numpy as np
import pytest

import cuwaves
from cuwaves import CUW_HPSI, CUW_PSI0, CUW_PSIM, systems

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(np.ravel(a - b)) / max(np.linalg.norm(np.ravel(b)), 1e-300))


def system(atoms, nb, ry):
    s = systems.si_small(atoms, epw_psi_ry=ry)
    s.nb = nb
    s.grid = systems.psi_grid(s)
    return systems.build_inputs(s)


def pair(inp, oracle, precision=cuwaves.CUW_PREC_FP64):
    gpu = cuwaves.open_waves(inp, precision=precision).setup().initialize()
    cpu = oracle.open_oracle(inp).setup()
    for which in (CUW_PSI0, CUW_PSIM):
        cpu.upload_psi(which, gpu.download_psi(which))
    cpu.set_proj(gpu.get_proj())
    return gpu, cpu


# bands below, at and past the 32-, 64- and 128-column tiles (a step's fused tile
# holds each band twice); cutoffs give sphere sizes of every remainder
EDGES = [(2, 2, 9.0), (2, 8, 14.0), (6, 16, 11.0), (8, 18, 10.0), (10, 32, 12.0), (12, 34, 9.5), (16, 64, 8.0),
         (16, 66, 10.5), (16, 130, 13.0)]


@pytest.mark.parametrize("atoms,nb,ry", EDGES)
def test_tile_edges_fp64(atoms, nb, ry, oracle):
    inp = system(atoms, nb, ry)
    gpu, cpu = pair(inp, oracle)
    # products of K terms in FP64: K * 2^-53 of the sums of magnitudes, far below 1e-11
    gpu.projections()
    cpu.projections()
    assert rel(gpu.get_proj(), cpu.get_proj()) < 1e-11
    assert rel(gpu.force(), cpu.force()) < 1e-10
    gpu.hpsi()
    cpu.hpsi()
    assert rel(gpu.download_psi(CUW_HPSI), cpu.download_psi(CUW_HPSI)) < 1e-11
    m, dev = gpu.overlap_check()
    mo, _ = cpu.overlap_check()
    assert np.abs(m - mo).max() < 1e-11
    for _ in range(2):
        og, fg = gpu.cp_step(move_atoms=True)
        oc, fc = cpu.cp_step(move_atoms=True)
        assert og[4] == oc[4]
        assert abs(og[0] - oc[0]) < 1e-8
        assert np.abs(fg - fc).max() < 1e-6
    # two solves stopped at 1e-8 in the overlap, with equal iteration counts
    assert rel(gpu.download_psi(CUW_PSI0), cpu.download_psi(CUW_PSI0)) < 1e-8


@pytest.mark.parametrize("atoms,nb,ry", EDGES)
def test_tile_edges_mixed(atoms, nb, ry, oracle):
    inp = system(atoms, nb, ry)
    gpu, cpu = pair(inp, oracle, cuwaves.CUW_PREC_MIXED)
    # split-tf32 products carry about 21 bits: 2^-21 = 5e-7, four times that
    gpu.projections()
    cpu.projections()
    assert rel(gpu.get_proj(), cpu.get_proj()) < 2e-6
    assert rel(gpu.force(), cpu.force()) < 2e-6
    gpu.hpsi()
    cpu.hpsi()
    assert rel(gpu.download_psi(CUW_HPSI), cpu.download_psi(CUW_HPSI)) < 2e-6
    gpu.propagate()
    cpu.propagate()
    gpu.orthogonalize()
    cpu.orthogonalize()
    assert rel(gpu.download_psi(CUW_PSIM), cpu.download_psi(CUW_PSIM)) < 2e-6
    assert gpu.overlap_check()[1] < 1e-4


@pytest.mark.parametrize("precision", [cuwaves.CUW_PREC_FP64, cuwaves.CUW_PREC_MIXED])
@pytest.mark.parametrize("table", ["ylm", "pro"])
def test_tables_without_parity(table, precision, oracle):
    """One table value changed at one G: the G set has no parity, and the
    projector contractions follow the tables as they are."""
    inp = dict(system(8, 16, 10.0))
    t = inp[table].copy()
    t[0, 7] *= 1.25
    inp[table] = t
    gpu, cpu = pair(inp, oracle, precision)
    gpu.projections()
    cpu.projections()
    assert rel(gpu.get_proj(), cpu.get_proj()) < 1e-11
    gpu.hpsi()
    cpu.hpsi()
    tol = 1e-11 if precision == cuwaves.CUW_PREC_FP64 else 2e-6  # FP32 transforms
    assert rel(gpu.download_psi(CUW_HPSI), cpu.download_psi(CUW_HPSI)) < tol
    og, fg = gpu.cp_step()
    oc, fc = cpu.cp_step()
    assert abs(og[0] - oc[0]) < (1e-8 if precision == cuwaves.CUW_PREC_FP64 else 1e-4)


@pytest.mark.parametrize("precision", [cuwaves.CUW_PREC_FP64, cuwaves.CUW_PREC_MIXED])
def test_tables_with_parity_to_rounding(precision, oracle):
    """Tables that a host's arithmetic leaves a few units in the last place off
    parity take the same kernels as exact ones, and the results stay the oracle's
    for those tables to the rounding of the products."""
    exact = dict(system(8, 16, 10.0))
    inp = dict(exact)
    rng = np.random.default_rng(3)
    for name, scale in (("ylm", 1.0), ("pro", None), ("gvec", None)):
        t = inp[name]
        inp[name] = t + rng.integers(-2, 3, t.shape) * 2.0**-52 * (np.abs(t) if scale is None else scale)
    ref, _ = pair(exact, oracle, precision)
    gpu, cpu = pair(inp, oracle, precision)
    count = []
    for w in (ref, gpu):
        before = w.get_timing()[1]
        w.projections()
        w.force()
        w.hpsi()
        count.append(w.get_timing()[1] - before)
    assert count[0] == count[1]  # the complex kernels take fewer launches
    cpu.projections()
    tol = 1e-11 if precision == cuwaves.CUW_PREC_FP64 else 2e-6
    assert rel(gpu.get_proj(), cpu.get_proj()) < tol
    cpu.hpsi()
    assert rel(gpu.download_psi(CUW_HPSI), cpu.download_psi(CUW_HPSI)) < tol
    assert rel(gpu.force(), cpu.force()) < 10 * tol
