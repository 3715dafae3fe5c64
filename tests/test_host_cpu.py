"""The engine's host side on a runtime without a device (fake_cuda.cpp): what it
allocates, launches and refuses.  No kernel runs, so no result is looked at."""
import numpy as np
import pytest

from cuwaves import CUW_PREC_FP64, CUW_PREC_MIXED, WavesError, systems

PRECISIONS = [CUW_PREC_FP64, CUW_PREC_MIXED]


def inputs(sy):
    return systems.build_inputs(sy, psi_init="zero")


def every_routine(w):
    w.projections()
    w.force()
    w.hpsi()
    w.density()
    w.cp_step(move_atoms=True)


@pytest.mark.parametrize("prec", PRECISIONS)
def test_failed_gset_leaves_no_set(fake_engine, prec):
    """A set_gset that runs out of memory leaves the handle without a G set: later
    calls are refused, nothing is launched with the buffers that are gone, and the
    handle takes a G set again."""
    inp = inputs(systems.si_small(2, epw_psi_ry=12.0))
    other = dict(inp, minusg=np.arange(1, inp["ngl"] + 1, dtype=np.int32))  # every G its own partner
    before = fake_engine.lib.fake_in_use()
    w = fake_engine.open(inp, prec).setup()
    every_routine(w)
    gsets = (other, inp)
    refused = 0
    for n in range(1, 100):
        w.inp = gsets[n % 2]
        fake_engine.lib.fake_fail_malloc(n)
        try:
            w.setup()
            break
        except WavesError:
            refused += 1
        finally:
            fake_engine.lib.fake_fail_malloc(-1)
        fake_engine.launches()
        for call in (w.projections, w.force, w.hpsi, w.density, w.cp_step, w.ekin):
            with pytest.raises(WavesError, match="(?i)not loaded"):
                call()
        assert fake_engine.launches() == []
        assert fake_engine.lib.fake_misuse() == 0
        if n % 3 == 0:  # the same set again, and a change between two good ones
            w.setup()
            every_routine(w)
    assert refused > 8  # the buffers of a G set, one after the other
    every_routine(w)
    w.close()
    assert fake_engine.lib.fake_misuse() == 0
    assert fake_engine.lib.fake_in_use() == before


@pytest.mark.parametrize("nb", [2, 34])
def test_launches_of_long_cells(fake_engine, nb):
    """More plane waves than 65535 row tiles of the folded products hold (32 rows
    each, two rows a pair): every launch stays within the grid limits."""
    n = 2_200_000
    base = inputs(systems.si_small(2, epw_psi_ry=12.0))
    g = np.arange(n, dtype=np.int32)
    igvec = np.stack([g % 100, g // 100 % 100, g // 10000], axis=1).astype(np.int32)
    inp = dict(base, ngl=n, nb=nb, nbh=nb // 2, grid=(100, 100, 720), igvec=igvec, minusg=(g ^ 1) + 1, gvec=np.zeros((n, 3)),
               g2=np.ones(n), pro=np.ones((len(base["pro"]), n)), ylm=np.ones((len(base["ylm"]), n)), mpsi=np.ones(n),
               v=np.zeros(100 * 100 * 720), occ=np.full(nb, 2.0), psi=np.zeros((nb // 2, n), dtype=np.complex128))
    w = fake_engine.open(inp).setup()
    w.gramschmidt(0, inp["r0"])
    w.projections()
    w.force()
    w.hpsi()
    w.propagate()
    w.orthogonalize()
    w.cp_step(move_atoms=True)
    w.close()
    assert fake_engine.lib.fake_misuse() == 0


SETS = {
    "Si2": lambda: systems.si_small(2, epw_psi_ry=12.0),
    "Si8": lambda: systems.si_supercell(1, 1, 1),
    "H2O8": lambda: systems.water_cluster(8),  # many plane waves for few bands
    "Si64": lambda: systems.si_supercell(2, 2, 2),
}


@pytest.mark.parametrize("prec", PRECISIONS)
@pytest.mark.parametrize("name", SETS)
def test_set_up_allocates_for_every_routine(fake_engine, prec, name):
    """The first calls of a new set allocate nothing: what the contractions need is
    known with the G set."""
    w = fake_engine.open(inputs(SETS[name]()), prec).setup()
    before = fake_engine.lib.fake_mallocs()
    w.gramschmidt(0, w.inp["r0"])
    w.projections()
    w.hpsi()
    w.etot()
    w.overlap_check()
    for _ in range(2):
        w.cp_step(move_atoms=True)
    assert fake_engine.lib.fake_mallocs() == before
    w.close()


@pytest.mark.parametrize("prec", PRECISIONS)
@pytest.mark.parametrize("name", SETS)
def test_admission_estimate_bounds_the_memory(fake_engine, prec, name, monkeypatch):
    """The serving runtime admits a set by an estimate of its device memory: never
    below what the set allocates, and not far above it."""
    from cuwaves import serve

    monkeypatch.setattr(serve, "load_library", lambda: fake_engine.lib)
    monkeypatch.setattr(serve, "_fns", None)
    inp = inputs(SETS[name]())
    srv = serve.Server(hbm_budget=1 << 40, workers=1)
    before = fake_engine.lib.fake_in_use()
    fake_engine.lib.fake_reset_peak()
    for nsteps in (0, 2):
        srv.submit(inp, nsteps=nsteps, precision=prec)
        srv.wait_all()
    held = fake_engine.lib.fake_peak() - before
    est = srv.stats()["peak_bytes"]
    srv.close()
    print(f"{name}: {held / 1e6:.1f} MB held, {est / 1e6:.1f} MB estimated")
    assert held <= est <= 1.1 * held + (24 << 20)
