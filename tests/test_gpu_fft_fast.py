"""The line-pass FFTs (fft_pencil.cuh) on the configurations' cubic grids
against the runtime-radix kernels of fft.cu, against FP64 and against the
oracle, through the C ABI.

QBX_FAST_FFT=0 at qbx_set_cell selects the runtime-radix kernels for a context.
Tolerances: FP64 1e-12 of the largest value (the same arithmetic in another
order); mixed precision 2e-6 of the largest value.
"""
import os

import numpy as np
import pytest

from qbx import capi, systems
from oracle import qbox_np

pytestmark = pytest.mark.gpu


def _ctx(s, precision, fast):
    os.environ["QBX_FAST_FFT"] = "1" if fast else "0"
    try:
        return capi.from_system(s, precision=precision)
    finally:
        os.environ.pop("QBX_FAST_FFT", None)


def _system(name):
    return systems.si512().band_sample(32) if name == "si512_32" else systems.get(name)


def _run(ctx):
    ctx.update_density()
    rho = ctx.density()
    ctx.update_vhxc()
    e = ctx.energy(hpsi=True)
    return rho, ctx.get_hpsi(), e


@pytest.mark.parametrize("name", ["si8", "si64", "h2o32", "si512_32"])
@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED])
def test_fast_matches_generic(name, precision):
    s = _system(name)
    a = _ctx(s, precision, True)
    b = _ctx(s, precision, False)
    ra, ha, ea = _run(a)
    rb, hb, eb = _run(b)
    tol = 1e-12 if precision == capi.FP64 else 2e-6
    np.testing.assert_allclose(ra, rb, rtol=0, atol=tol * np.abs(rb).max())
    np.testing.assert_allclose(ha, hb, rtol=0, atol=tol * np.abs(hb).max())
    etol = (1e-9 if precision == capi.FP64 else 1e-6) * len(s.atoms)
    assert abs(ea["etotal"] - eb["etotal"]) < etol
    a.close()
    b.close()


def test_fast_fp64_matches_oracle_si64():
    s = systems.si64()
    es = qbox_np.ElectronicStep(s)
    es.update_density()
    es.update_vhxc()
    es.energy(True)
    ctx = _ctx(s, capi.FP64, True)
    rho, hc, e = _run(ctx)
    np.testing.assert_allclose(rho, es.rhor, rtol=0, atol=1e-12 * np.abs(es.rhor).max())
    np.testing.assert_allclose(hc, es.hc, rtol=0, atol=1e-11)
    assert abs(e["etotal"] - es.etotal) < 1e-8
    ctx.close()


@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED])
def test_autotune_keeps_results(precision):
    """qbx_autotune times the transforms and names their kernels; the density and
    H psi stay the same."""
    s = systems.si64()
    a = _ctx(s, precision, True)
    ra, ha, ea = _run(a)
    report = a.autotune()
    assert "chosen:" in report
    rb, hb, eb = _run(a)
    tol = 1e-12 if precision == capi.FP64 else 2e-6
    np.testing.assert_allclose(rb, ra, rtol=0, atol=tol * np.abs(ra).max())
    np.testing.assert_allclose(hb, ha, rtol=0, atol=tol * np.abs(ha).max())
    a.close()


@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED])
@pytest.mark.parametrize("bands", [31, 34, 68])
def test_last_chunk_of_slots_is_smaller(bands, precision):
    """140^3: 16, 17 and 34 slots a line in one, two and three CTAs, the last of
    them with fewer (and an odd band alone in its pair) against the runtime-radix
    kernels."""
    s = systems.si512().band_sample(bands)
    a, b = _ctx(s, precision, True), _ctx(s, precision, False)
    ra, ha, _ = _run(a)
    rb, hb, _ = _run(b)
    a.close()
    b.close()
    tol = 1e-12 if precision == capi.FP64 else 2e-6
    np.testing.assert_allclose(ra, rb, rtol=0, atol=tol * np.abs(rb).max())
    np.testing.assert_allclose(ha, hb, rtol=0, atol=tol * np.abs(hb).max())


@pytest.mark.parametrize("name", ["si8", "si64", "h2o32", "si512_32"])
def test_mixed_matches_fp64(name):
    """The FP32 passes against the FP64 ones from the same coefficients: density
    and H psi to 2e-6 of the largest value, the energy to 1e-6 Ha per atom, and a
    two-step trajectory's energies to the same."""
    s = _system(name)
    a, b = _ctx(s, capi.MIXED, True), _ctx(s, capi.FP64, True)
    a.set_coeffs(b.get_coeffs())
    ra, ha, ea = _run(a)
    rb, hb, eb = _run(b)
    np.testing.assert_allclose(ra, rb, rtol=0, atol=2e-6 * np.abs(rb).max())
    np.testing.assert_allclose(ha, hb, rtol=0, atol=2e-6 * np.abs(hb).max())
    assert abs(ea["etotal"] - eb["etotal"]) < 1e-6 * len(s.atoms)
    for _ in range(2):
        ea, eb = a.scf_step(), b.scf_step()
        assert abs(ea["etotal"] - eb["etotal"]) < 1e-6 * len(s.atoms)
    a.close()
    b.close()


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("name", ["si64", "si512_32"])
def test_kept_tiles_give_the_recomputed_step(name, graph, monkeypatch):
    """The tiles kept in HBM from the density pass and reused by the H psi pass
    of the same step (QBX_PSIR=1) give the step that transforms every band
    pair backward twice (QBX_PSIR=0): energies to 1e-12 relative and the
    coefficients after three steps to 1e-12, eager and captured."""
    s = _system(name)
    ctxs = []
    for mode in ("1", "0"):
        monkeypatch.setenv("QBX_PSIR", mode)
        c = _ctx(s, capi.MIXED, True)
        c.set_step_graph(graph)
        ctxs.append(c)
    monkeypatch.delenv("QBX_PSIR")
    a, b = ctxs
    for _ in range(3):
        ea, eb = a.scf_step(), b.scf_step()
        for k in ("ekin", "enl", "etotal", "eigenvalue_sum"):
            assert abs(ea[k] - eb[k]) <= 1e-12 * abs(eb[k]) + 1e-12, (k, ea[k], eb[k])
    np.testing.assert_allclose(a.get_coeffs(), b.get_coeffs(), rtol=0, atol=1e-12)
    a.close()
    b.close()
