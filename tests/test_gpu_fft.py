"""z transforms of every length with a two-step kernel, on xy planes whose
columns do not fill the last block, and of a length without one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import cuwaves  # noqa: E402
from cuwaves import CUW_PREC_FP64, CUW_PREC_MIXED, systems  # noqa: E402

LENGTHS = (18, 20, 22, 24, 28, 30, 32, 36, 40, 42, 44, 48, 50, 54, 56, 60, 64, 66, 70, 72, 80, 84, 88, 90, 96, 100, 108,
           110, 120, 126, 128)


@pytest.mark.parametrize("prec", [CUW_PREC_FP64, CUW_PREC_MIXED])
@pytest.mark.parametrize("nr3", LENGTHS)
def test_z_lengths(nr3, prec, oracle):
    """H|psi> and the density against the oracle.  Both are sums of a few
    transforms' outputs: each step of a transform rounds by half an ulp of its
    values' norm, at most ~10 steps and 4 operations a step on one path, so the
    largest error stays below 40 ulp (2^-53 or 2^-24) of the largest value."""
    inp = systems.build_inputs(systems.water_box(1, box=8.0, lattice=(1, 1, 1), epw_psi_ry=9.0, grid=(21, 20, nr3)))
    w = cuwaves.open_waves(inp, precision=prec).setup().initialize()
    cpu = oracle.open_oracle(inp).setup()
    for which in (cuwaves.CUW_PSI0, cuwaves.CUW_PSIM):
        cpu.upload_psi(which, w.download_psi(which))
    cpu.set_proj(w.get_proj())
    occ = np.array(inp["occ"], dtype=np.float64)
    occ[-1] = 0.5
    for b in (w, cpu):
        b.set_occ(occ)
        b.hpsi()
    tol = 40 * (2.0**-53 if prec == CUW_PREC_FP64 else 2.0**-24)
    ref, got = cpu.download_psi(cuwaves.CUW_HPSI), w.download_psi(cuwaves.CUW_HPSI)
    assert np.abs(got - ref).max() < tol * np.abs(ref).max()
    ref, got = cpu.density(), w.density()
    assert np.abs(got - ref).max() < 2 * tol * np.abs(ref).max()  # squares
    w.close()
    cpu.close()
