"""The n x n algebra of ortho_align and polar in one kernel (up to 128 bands)
against the library chain (QBX_ORTHO_SMALL=0): the panel remainders, one and
eight panels, both branches of the polar iteration in both precisions, captured
and eager, and a factorisation that fails.

Both are FP64 throughout; they differ in the order of sums and in forming L^-1
explicitly, so to some n eps times the condition of the overlap (10 here):
1e-11.
"""
import os

import numpy as np
import pytest

from qbx import capi, systems

pytestmark = pytest.mark.gpu

BANDS = [1, 7, 15, 16, 17, 40, 97, 127, 128]


def _ctx(bands, precision, small, xc="LDA", edges=(11.0, 10.0, 12.5)):
    pos = systems.diamond_supercell(10.26, 1, 0.03, 4)[:5]
    s = systems.System("box", np.diag(edges), [systems.SI], [(0, p) for p in pos],
                       20.0, bands, xc, 13)
    os.environ["QBX_ORTHO_SMALL"] = small
    try:
        return capi.from_system(s, precision=precision)
    finally:
        os.environ.pop("QBX_ORTHO_SMALL")


@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED])
@pytest.mark.parametrize("n", BANDS)
def test_polar(n, precision):
    rng = np.random.default_rng(n)
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    near = q @ (np.eye(n) + 0.02 / n * rng.standard_normal((n, n)))
    far = q @ np.diag(np.linspace(0.4, 2.5, n)) @ np.linalg.qr(rng.standard_normal((n, n)))[0]
    ctx = _ctx(n, precision, "1")
    for x in (near, far):
        u, _, vt = np.linalg.svd(x)
        for graph in (False, True):
            f, it = ctx.polar(x, 1e-6, 20, graph)
            np.testing.assert_allclose(f, u @ vt, rtol=0, atol=1e-11)
            assert 1 <= it <= 12
    ctx.close()


@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED])
@pytest.mark.parametrize("n", BANDS)
def test_step_matches_library_chain(n, precision):
    out = []
    for small in ("1", "0"):
        ctx = _ctx(n, precision, small)
        e = [ctx.scf_step()["etotal"] for _ in range(2)]
        ctx.set_step_graph(True)
        e += [ctx.scf_step()["etotal"] for _ in range(2)]
        out.append((np.array(e), ctx.get_coeffs()))
        ctx.close()
    (ea, ca), (eb, cb) = out
    np.testing.assert_allclose(ea, eb, rtol=1e-11)
    np.testing.assert_allclose(ca, cb, rtol=0, atol=1e-10 if precision == capi.FP64 else 1e-7)


@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED])
def test_singular_overlap_is_an_error(precision):
    ctx = _ctx(20, precision, "1")
    c = ctx.get_coeffs()
    bad = c.copy()
    bad[7] = 0.0
    ctx.set_coeffs(bad)
    with pytest.raises(capi.QbxError):
        ctx.ortho_align(c)
    # the context goes on
    ctx.set_coeffs(c)
    ctx.ortho_align(c)
    np.testing.assert_allclose(ctx.get_coeffs(), c, rtol=0,
                               atol=1e-11 if precision == capi.FP64 else 1e-6)
    ctx.close()


@pytest.mark.parametrize("n", [16, 45, 128])
def test_pivots_over_their_range(n):
    """Bands scaled by powers of two, the pivots of their overlap between 1e-35 and
    1e35 (past both ends of the range in which the kernel takes its own
    reciprocal square root): every other operation scales exactly, so the aligned
    bands are those of the unscaled ones to the roundings of the pivots, a few
    eps each over n of them."""
    ctx = _ctx(n, capi.FP64, "1")
    c = ctx.get_coeffs()
    rng = np.random.default_rng(n)
    near = c + 0.01 * rng.standard_normal((n, 1)) * np.roll(c, 1, axis=0)
    scale = np.concatenate([[58, -58, 50, 49, -49, -50], np.linspace(-58, 58, n)])[:n]
    scale = 2.0 ** rng.permutation(np.round(scale))
    out = []
    for f in (np.ones(n), scale):
        ctx.set_coeffs(near * f[:, None])
        ctx.ortho_align(c)
        out.append(ctx.get_coeffs())
    ctx.close()
    np.testing.assert_allclose(out[1], out[0], rtol=0, atol=8 * n * np.finfo(float).eps)


@pytest.mark.parametrize("n", [1, 31, 33, 65, 200, 432])
def test_lower_inverse_with_smaller_last_blocks(n):
    """L^-1 by blocks whose last ones are not whole: n eps times the factor's
    condition number (4)."""
    rng = np.random.default_rng(n)
    l = np.tril(0.5 / np.sqrt(n) * rng.standard_normal((n, n)), -1) + np.diag(rng.uniform(1, 2, n))
    bad = l.copy()
    bad[np.triu_indices(n, 1)] = np.nan
    ctx = _ctx(4, capi.MIXED, "1")
    got, _ = ctx.lower_inverse(bad)
    np.testing.assert_allclose(got @ l, np.eye(n), rtol=0, atol=64 * n * np.finfo(float).eps)
    assert np.all(got[np.triu_indices(n, 1)] == 0.0)
    ctx.close()


@pytest.mark.parametrize("n,edges", [(130, (11.0, 10.0, 12.5)), (520, (15.0, 14.0, 15.0)),
                                     (1024, (11.0, 10.0, 12.5)), (1025, (11.0, 10.0, 12.5))])
def test_overlap_and_polar_products(n, edges):
    """The overlap as one product (130 bands), by blocks of columns of which the
    last is smaller (520) and as a triangle (1024: a contraction short against
    the bands), and the polar iteration's products on both sides of their lines:
    C orthonormal to n eps times the overlap's condition (10) after gram, and
    polar's factor that of the SVD to n eps times the matrix's condition (6)."""
    ctx = _ctx(n, capi.FP64, "1", edges=edges)
    c = ctx.get_coeffs()
    s = 2 * (c.conj() @ c.T).real - np.outer(c[:, 0].real, c[:, 0].real)
    tol = 10 * n * np.finfo(float).eps
    np.testing.assert_allclose(s, np.eye(n), rtol=0, atol=tol)
    rng = np.random.default_rng(n)
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    w, _ = np.linalg.qr(rng.standard_normal((n, n)))
    x = q @ np.diag(np.linspace(0.4, 2.5, n)) @ w
    for precision in (capi.FP64, capi.MIXED):
        if precision == capi.MIXED:
            ctx.close()
            ctx = _ctx(n, precision, "1", edges=edges)
        f, _ = ctx.polar(x, 1e-6, 20, False)
        np.testing.assert_allclose(f, q @ w, rtol=0, atol=tol)
    ctx.close()


@pytest.mark.parametrize("n", [255, 257, 513, 700])
def test_complex_overlap_by_blocks(n):
    pos = systems.diamond_supercell(10.26, 1, 0.03, 4)[:5]
    s = systems.System("box", np.diag([11.0, 10.0, 12.5]), [systems.SI], [(0, p) for p in pos],
                       20.0, n, "LDA", 13).with_kpoints([((0.25, 0.1, 0.3), 1.0)])
    ctx = capi.from_system(s, precision=capi.FP64)
    c = ctx.get_kpoint_coeffs(0)
    np.testing.assert_allclose(c.conj() @ c.T, np.eye(n), rtol=0, atol=10 * n * np.finfo(float).eps)
    ctx.close()
