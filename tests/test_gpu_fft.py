"""z transforms of every length with a two-step kernel, on xy planes whose
columns do not fill the last block, and of a length without one; every plan
variant of the grids with compiled xy planes."""
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
    check((21, 20, nr3), prec, oracle, 9.0)


GRIDS = ((18, 18, 18), (18, 18, 36), (24, 24, 24), (28, 28, 28), (28, 28, 56), (28, 56, 56), (32, 32, 32), (36, 36, 36),
         (48, 48, 48), (56, 56, 56), (56, 56, 110), (64, 64, 64), (72, 72, 72), (80, 80, 80), (96, 96, 96))


@pytest.mark.parametrize("prec", [CUW_PREC_FP64, CUW_PREC_MIXED])
@pytest.mark.parametrize("grid", GRIDS)
def test_plane_variants(grid, prec, oracle):
    check(grid, prec, oracle, 9.0, range(4 if grid == (64, 64, 64) else 3))
    if min(grid) >= 48:  # a sphere that fills more of the rows
        check(grid, prec, oracle, 60.0, (0,))


# every length with Stockham stages of its own, and run-time lengths beside them, on
# planes that are not in the table; the last three differ from table grids in NR3 only
OTHER = ((16, 20, 24), (24, 28, 24), (32, 36, 24), (40, 48, 24), (56, 64, 24), (72, 80, 24), (96, 16, 24), (42, 84, 24),
         (24, 24, 48), (28, 28, 84), (28, 56, 80))


@pytest.mark.parametrize("prec", [CUW_PREC_FP64, CUW_PREC_MIXED])
@pytest.mark.parametrize("grid", OTHER)
def test_planes_off_the_table(grid, prec, oracle):
    check(grid, prec, oracle, 9.0)


def check(grid, prec, oracle, ry, variants=(0,)):
    """H|psi> and the density against the oracle.  Both are sums of a few
    transforms' outputs: each step of a transform rounds by half an ulp of its
    values' norm, at most ~10 steps and 4 operations a step on one path, so the
    largest error stays below 40 ulp (2^-53 or 2^-24) of the largest value."""
    inp = systems.build_inputs(systems.water_box(1, box=8.0, lattice=(1, 1, 1), epw_psi_ry=ry, grid=grid))
    w = cuwaves.open_waves(inp, precision=prec).setup().initialize()
    cpu = oracle.open_oracle(inp).setup()
    for which in (cuwaves.CUW_PSI0, cuwaves.CUW_PSIM):
        cpu.upload_psi(which, w.download_psi(which))
    cpu.set_proj(w.get_proj())
    occ = np.array(inp["occ"], dtype=np.float64)
    occ[-1] = 0.5
    for b in (w, cpu):
        b.set_occ(occ)
    cpu.hpsi()
    tol = 40 * (2.0**-53 if prec == CUW_PREC_FP64 else 2.0**-24)
    ref, rho = cpu.download_psi(cuwaves.CUW_HPSI), cpu.density()
    for v in variants:
        w.set_option(cuwaves.CUW_OPT_FFT_VARIANT, v)
        w.hpsi()
        got = w.download_psi(cuwaves.CUW_HPSI)
        assert np.abs(got - ref).max() < tol * np.abs(ref).max(), v
        assert np.abs(w.density() - rho).max() < 2 * tol * np.abs(rho).max(), v  # squares
    w.close()
    cpu.close()
