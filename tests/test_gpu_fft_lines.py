"""The line-pass FFTs (fft_pencil.cuh) against the runtime-radix kernels
(QBX_FAST_FFT=0) where the passes can go wrong: grids of three different
lengths, the shortest and longest register factorisations, odd band counts,
line counts that are no multiple of a CTA's lines, k points, and the tiles
kept from the density pass against transforming twice (QBX_PSIR=0).

FP64: the same sums in another order, 1e-12 of the largest value.  FP32: one
rounding of 6e-8 per butterfly level on three axes, 2e-6 of the largest
value; the charge, whose systematic part the passes take out, 1e-7 of the
electrons (the FFT's rounding averages out over the grid).  In FP32 too the
density's weights, products and sums are FP64 and V(r) keeps its FP64 value.
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


def _mixed_box(bands):
    """64 x 32 x 64 points: the sums of a constant are exact in FP32, and a
    CTA of the x passes takes 16 slots of 320 bands."""
    return _cell(20.0, 9.75, 19.75, 20.0, bands)


def _constant(ctx, values):
    """Band n constant in r: its G = 0 coefficient alone."""
    c = np.zeros((ctx.nst, ctx.ngw), complex)
    g0 = int(np.flatnonzero(~ctx.miller().any(axis=1))[0])
    c[:, g0] = values
    ctx.set_coeffs(c)
    return g0


@pytest.mark.parametrize("fast", ["1", "0"])
def test_mixed_density_sums_in_fp64(fast, tmp_path):
    """Constant bands whose values FP32 holds: the density is sum_n f_n c_n^2 /
    Omega times one factor (the gain that the passes take out), for fractional
    occupations too.  A product, weight or sum of 16 slots in FP32 shows at
    1e-8; FP64 leaves 320 roundings, 1e-13."""
    bands = 320
    os.environ["QBX_FAST_FFT"] = fast
    try:
        ctx = capi.from_system(_mixed_box(bands), precision=capi.MIXED, gram=False)
    finally:
        os.environ.pop("QBX_FAST_FFT")
    assert tuple(ctx.grid) == (64, 32, 64)
    rng = np.random.default_rng(4)
    values = 1.0 + rng.integers(0, 1 << 12, bands) / (1 << 12)
    # occupations come with a sample's <wavefunction>
    path = str(tmp_path / "wf.xml")
    ctx.write_wavefunction(path)
    text = open(path).read()
    a = text.index(">", text.index("<density_matrix")) + 1
    b = text.index("</density_matrix>")
    factor = []
    for occ in (np.full(bands, 2.0), rng.uniform(0.1, 2.0, bands), rng.uniform(0.1, 2.0, bands)):
        with open(path, "w") as f:
            f.write(text[:a] + "\n" + "\n".join(repr(float(o)) for o in occ) + "\n" + text[b:])
        ctx.read_wavefunction(path)
        _constant(ctx, values)
        ctx.update_density()
        rho = ctx.density()
        factor += [rho.min() / np.dot(occ, values ** 2), rho.max() / np.dot(occ, values ** 2)]
    ctx.close()
    np.testing.assert_allclose(factor, factor[0], rtol=1e-13)


@pytest.mark.parametrize("fast", ["1", "0"])
def test_mixed_product_with_the_fp64_potential(fast):
    """A constant band times a constant V: FP32 rounds the product with the
    FP64 value of V, which here is one unit off the product with V rounded to
    FP32 first."""
    os.environ["QBX_FAST_FFT"] = fast
    try:
        ctx = capi.from_system(_mixed_box(4), precision=capi.MIXED, gram=False)
    finally:
        os.environ.pop("QBX_FAST_FFT")
    x = np.float32([1.9, 1.99, 1.75, 1.95]).astype(float)
    g0 = _constant(ctx, x)
    out = []
    v = 1.0 + 0.98 * 2.0 ** -24
    for pot in (1.0, v):
        dc = np.zeros((ctx.nst, ctx.ngw), complex)
        ctx.rs_mul_add(np.full(int(np.prod(ctx.grid)), pot), dc)
        out.append(dc[:, g0].real.copy())
    ctx.close()
    want = (x * v).astype(np.float32).astype(float)
    assert np.float32(v) == 1.0 and np.all(want > x)
    np.testing.assert_allclose(out[1] / out[0], want / x, rtol=1e-12)


def test_mixed_density_of_long_slot_chunks():
    """320 bands, 16 slots a CTA, against FP64 point by point: the transforms'
    rounding (17 butterfly levels of 6e-8 in each of 320 bands, independent),
    2e-7 of the largest value."""
    s = _mixed_box(320)
    rho = []
    for precision in (capi.FP64, capi.MIXED):
        ctx = capi.from_system(s, precision=precision)
        ctx.update_density()
        rho.append(ctx.density())
        ctx.close()
    np.testing.assert_allclose(rho[1], rho[0], rtol=0, atol=2e-7 * np.abs(rho[0]).max())


@pytest.mark.parametrize("fast", ["1", "0"])
def test_precision_switch(fast):
    """qbx_set_precision on either route and back: the buffers of the new
    precision are there (the runtime-radix kernels' only where they run)."""
    os.environ["QBX_FAST_FFT"] = fast
    try:
        ctx = capi.from_system(_cell(12.0, 7.5, 19.0, 20.0, 9), precision=capi.FP64)
    finally:
        os.environ.pop("QBX_FAST_FFT")
    rho, h = [], []
    for precision in (capi.FP64, capi.MIXED, capi.FP64):
        ctx.set_precision(precision)
        ctx.update_density()
        ctx.update_vhxc()
        ctx.energy(hpsi=True)
        rho.append(ctx.density())
        h.append(ctx.get_hpsi())
    ctx.close()
    for i, tol in ((1, 2e-6), (2, 1e-12)):
        np.testing.assert_allclose(rho[i], rho[0], rtol=0, atol=tol * np.abs(rho[0]).max())
        np.testing.assert_allclose(h[i], h[0], rtol=0, atol=tol * np.abs(h[0]).max())
