"""Contexts whose real-space grids are kept x fastest (fft.cu, grid_zfast)
against contexts that keep them z fastest: the runtime-radix kernels
(QBX_FAST_FFT=0), and the line passes with a stick buffer (QBX_FAST_ZBUF_MB)
that holds a slot of the wavefunctions but none of the density basis, so that
the passes transpose the density and V(r).
"""
import numpy as np
import pytest

from qbx import capi, systems

pytestmark = pytest.mark.gpu

ZBUF_MB = 1
# the routes that keep the grids x fastest
ROUTES = [{"QBX_FAST_FFT": "0"}, {"QBX_FAST_ZBUF_MB": str(ZBUF_MB)}]


def _cell(edges=(12.0, 7.5, 19.0), ecut=20.0, bands=8, xc="LDA"):
    pos = systems.diamond_supercell(10.26, 1, 0.0, 1)[:4] % 5.0 + 0.3
    return systems.System("box", np.diag(edges).astype(float), [systems.SI],
                          [(0, p) for p in pos], ecut, bands, xc, 7)


def _ctx(s, monkeypatch, env=(), precision=capi.FP64):
    with monkeypatch.context() as m:
        for k, v in dict(env).items():
            m.setenv(k, v)
        return capi.from_system(s, precision=precision)


def _slot_bytes(hkl, grid, stick_per_rod, size=16):
    """Sticks and tile of one slot: the (h, k) rods of a sphere's half, one or
    two sticks each, and the columns -h ... h."""
    rods = len({(int(h), int(k)) for h, k, _ in hkl})
    cols = len({int(h) for h, _, _ in hkl} | {-int(h) for h, _, _ in hkl})
    sticks = rods if stick_per_rod == 1 else 2 * rods - 1
    return size * grid[2] * (sticks + cols * grid[1])


def test_small_stick_buffer_takes_wavefunctions_only():
    """What the QBX_FAST_ZBUF_MB route relies on."""
    s = _cell()
    _, _, grid, hkl = capi.host_basis(s.cell, s.ecut)
    _, _, _, dense = capi.host_basis(s.cell, 4 * s.ecut)
    assert _slot_bytes(hkl, grid, 2) < ZBUF_MB << 20 < _slot_bytes(dense, grid, 2)


@pytest.mark.parametrize("xc", ["LDA", "PBE"])
@pytest.mark.parametrize("route", range(len(ROUTES)))
def test_stress_parts(route, xc, monkeypatch):
    """Every part of the stress, of a step and of a separate call, in either
    order of the grids (FP64: the same sums in another order, 1e-12 of the
    largest)."""
    s = _cell(xc=xc)
    out = []
    for env in ({}, ROUTES[route]):
        ctx = _ctx(s, monkeypatch, env)
        _, step = ctx.scf_step(stress=True), ctx.last_stress()[1]
        ctx.update_density()
        ctx.update_vhxc()
        ctx.energy()
        out.append((step, ctx.stress()[1]))
        ctx.close()
    for a, b in zip(*out):
        for k in a:
            np.testing.assert_allclose(b[k], a[k], rtol=0, atol=1e-12 * max(1e-3, np.abs(a[k]).max()),
                                       err_msg=k)


def _after_k_points(s, monkeypatch, env, k):
    """The stress at Gamma from the fields of a step at k points, and the
    density and V(r) before and after the return to Gamma."""
    ctx = _ctx(s, monkeypatch, env)
    ctx.scf_step()
    sk = s.with_kpoints([(k, 1.0)])
    ctx.set_kpoints([k], [1.0])
    reach = np.abs(ctx.kpoint_miller(0)).max(0)
    ctx.set_kpoint_coeffs(0, sk.kcoefficients(0, sk.kmiller(0)))
    ctx.gram()
    ctx.scf_step()
    before = ctx.density(), ctx.vr()
    ctx.set_kpoints([], [])
    after = ctx.density(), ctx.vr()
    parts = ctx.stress()[1]
    ctx.close()
    return reach, before, after, parts


@pytest.mark.parametrize("xc", ["LDA", "PBE"])
def test_fields_follow_the_order_of_the_grids(xc, monkeypatch):
    """A k point whose sphere reaches beyond the line kernels' points takes the
    grids to x fastest and the return to Gamma takes them back: every field
    moves with them (FP64, as above)."""
    s = _cell(xc=xc)
    k = (2.0, 0.0, 0.0)
    _, _, grid, _ = capi.host_basis(s.cell, s.ecut)
    reach, before, after, parts = _after_k_points(s, monkeypatch, {}, k)
    assert reach[0] > (grid[0] - 1) // 4            # not a line kernel's sphere
    _, _, _, want = _after_k_points(s, monkeypatch, ROUTES[0], k)
    for a, b in zip(before, after):
        np.testing.assert_array_equal(a, b)
    for q in want:
        np.testing.assert_allclose(parts[q], want[q], rtol=0,
                                   atol=1e-12 * max(1e-3, np.abs(want[q]).max()), err_msg=q)
