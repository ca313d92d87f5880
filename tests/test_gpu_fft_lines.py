"""The line-pass FFTs (fft_pencil.cuh) against the runtime-radix kernels
(QBX_FAST_FFT=0) where the passes can go wrong: grids of three different
lengths, the shortest and longest register factorisations, odd band counts,
line counts that are no multiple of a CTA's lines, k points, and the tiles
kept from the density pass against transforming twice (QBX_PSIR=0).

FP64: the same sums in another order, 1e-12 of the largest value.  FP32: one
rounding of 6e-8 per butterfly level on three axes, 2e-6 of the largest
value; the charge, whose systematic part the passes take out, 1e-7 of the
electrons (the FP32 sum of at most 16 bands and the FFT's rounding average
out over the grid).
"""
import os

import numpy as np
import pytest

from qbx import capi, systems

pytestmark = pytest.mark.gpu


def _cell(nx, ny, nz, ecut_ry, bands, xc="LDA", name="box"):
    pos = systems.diamond_supercell(10.26, 1, 0.0, 1)[:4] % 5.0 + 0.3
    return systems.System(name, np.diag([nx, ny, nz]).astype(float), [systems.SI],
                          [(0, p) for p in pos], ecut_ry, bands, xc, 7)


def _run(s, precision, fast, psir="1", kpoints=None, steps=0):
    os.environ["QBX_FAST_FFT"] = fast
    os.environ["QBX_PSIR"] = psir
    try:
        ctx = capi.from_system(s if kpoints is None else s.with_kpoints(kpoints),
                               precision=precision)
        if steps:
            out = [ctx.scf_step()["etotal"] for _ in range(steps)]
            c = [ctx.get_kpoint_coeffs(i) for i in range(len(kpoints))] if kpoints else \
                [ctx.get_coeffs()]
            return np.array(out), c, 0.0
        q = ctx.update_density()
        rho = ctx.density()
        ctx.update_vhxc()
        ctx.energy(hpsi=True)
        h = [ctx.get_kpoint_hpsi(i) for i in range(len(kpoints))] if kpoints else [ctx.get_hpsi()]
        return rho, h, q
    finally:
        os.environ.pop("QBX_FAST_FFT")
        os.environ.pop("QBX_PSIR")
        if "ctx" in locals():
            ctx.close()


# grids: (22, 30, 40), (40, 28, 60), (84, 18, 20), (144, 16, 16), (16, 192, 16),
# (18, 18, 220)
CASES = [((6.0, 9.0, 11.0), 22.0, 5), ((12.0, 7.5, 19.0), 20.0, 8), ((25.5, 5.2, 5.8), 20.0, 3),
         ((46.0, 4.4, 4.0), 21.0, 1), ((4.0, 61.0, 4.4), 20.5, 6), ((5.0, 4.6, 73.0), 20.0, 35)]


@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_lines_match_runtime_radix(case, precision):
    cell, ecut, bands = CASES[case]
    s = _cell(*cell, ecut, bands)
    ra, ha, qa = _run(s, precision, "1")
    rb, hb, qb = _run(s, precision, "0")
    tol = 1e-12 if precision == capi.FP64 else 2e-6
    np.testing.assert_allclose(ra, rb, rtol=0, atol=tol * np.abs(rb).max())
    np.testing.assert_allclose(ha[0], hb[0], rtol=0, atol=tol * np.abs(hb[0]).max())
    assert abs(qa - 2 * bands) <= (1e-12 if precision == capi.FP64 else 1e-7) * 2 * bands


@pytest.mark.parametrize("case", [0, 2, 5])
def test_lines_at_k_points(case):
    cell, ecut, bands = CASES[case]
    s = _cell(*cell, ecut, bands)
    k = [((0.25, 0.25, 0.25), 0.5), ((0.0, 0.5, 0.4), 0.5)]
    ra, ha, _ = _run(s, capi.FP64, "1", kpoints=k)
    rb, hb, _ = _run(s, capi.FP64, "0", kpoints=k)
    np.testing.assert_allclose(ra, rb, rtol=0, atol=1e-12 * np.abs(rb).max())
    for a, b in zip(ha, hb):
        np.testing.assert_allclose(a, b, rtol=0, atol=1e-12 * np.abs(b).max())


@pytest.mark.parametrize("kpoints", [None, [((0.25, 0.25, 0.25), 0.5), ((0.0, 0.5, 0.4), 0.5)]])
@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED])
def test_kept_tiles_give_the_recomputed_step(precision, kpoints):
    """Three steps, the same arithmetic in both (1e-11 for the order of the
    density's atomic sums through the orthonormalisation)."""
    if kpoints and precision == capi.MIXED:
        pytest.skip("k points run in FP64")
    s = _cell(11.0, 12.5, 9.0, 20.0, 9)
    ea, ca, _ = _run(s, precision, "1", "1", kpoints, steps=3)
    eb, cb, _ = _run(s, precision, "1", "0", kpoints, steps=3)
    np.testing.assert_allclose(ea, eb, rtol=1e-12)
    for a, b in zip(ca, cb):
        np.testing.assert_allclose(a, b, rtol=0, atol=1e-11)
