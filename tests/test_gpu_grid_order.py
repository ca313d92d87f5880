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


def _fields(ctx):
    ctx.update_density()
    ctx.update_vhxc()
    e = ctx.energy(hpsi=True)
    return ctx.density(), ctx.vr(), ctx.get_hpsi(), e


@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED])
@pytest.mark.parametrize("xc,edges", [("LDA", (12.0, 7.5, 19.0)), ("PBE", (12.0, 7.5, 19.0)),
                                      ("PBE", (9.0, 16.5, 6.0))])
@pytest.mark.parametrize("psir", ["0", "1"])
def test_line_passes_on_x_fastest_grids(psir, xc, edges, precision, monkeypatch):
    """The passes that transpose the density and V(r) against those that read and
    write them in place, in one and in several batches of slots; at 30 x 56 x 22
    the small buffer takes one slot of the density basis and the GGA's components go
    through one transform at a time (FP64: the same arithmetic, 1e-12 of the largest
    value; mixed: V(r) differs in its last bits, 2e-6)."""
    s = _cell(edges=edges, bands=9, xc=xc)
    out = []
    for env in ({}, dict(ROUTES[1], QBX_PSIR=psir)):
        ctx = _ctx(s, monkeypatch, env, precision)
        f = _fields(ctx)
        steps = [ctx.scf_step()["etotal"] for _ in range(2)]
        out.append((f, steps))
        ctx.close()
    (fa, sa), (fb, sb) = out
    tol = 1e-12 if precision == capi.FP64 else 2e-6
    for a, b in zip(fa[:3], fb[:3]):
        np.testing.assert_allclose(b, a, rtol=0, atol=tol * np.abs(a).max())
    etol = 1e-11 if precision == capi.FP64 else 1e-7
    for k in fa[3]:
        if isinstance(fa[3][k], float):
            assert abs(fa[3][k] - fb[3][k]) <= etol * max(1.0, abs(fa[3][k])), k
    np.testing.assert_allclose(sb, sa, rtol=etol)


@pytest.mark.parametrize("mb", [40, 100])
@pytest.mark.parametrize("psir", ["0", "1"])
@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED])
def test_smaller_stick_buffers(precision, psir, mb, monkeypatch):
    """140^3, 16 band pairs (FP64 30 MB a pair): buffers that take the slots in
    several batches, no slot of the density basis (40 MB) or one instead of the two
    of the GGA's components (100 MB)."""
    s = systems.si512().band_sample(32)
    out = []
    for env in ({}, {"QBX_FAST_ZBUF_MB": str(mb), "QBX_PSIR": psir}):
        ctx = _ctx(s, monkeypatch, env, precision)
        out.append((_fields(ctx), [ctx.scf_step()["etotal"] for _ in range(2)]))
        ctx.close()
    (fa, sa), (fb, sb) = out
    tol = 1e-12 if precision == capi.FP64 else 2e-6
    for a, b in zip(fa[:3], fb[:3]):
        np.testing.assert_allclose(b, a, rtol=0, atol=tol * np.abs(a).max())
    np.testing.assert_allclose(sb, sa, rtol=1e-11 if precision == capi.FP64 else 1e-7)


@pytest.mark.parametrize("route", ["buffer", "sphere"])
def test_k_points_on_x_fastest_grids(route, monkeypatch):
    """k points through the passes that transpose: the stick buffer too small for
    the density basis, or another k point of the set whose sphere reaches beyond
    the line kernels' points; against the runtime-radix kernels (FP64)."""
    far = (2.0, 0.0, 0.0) if route == "sphere" else (0.0, 0.5, 0.4)
    s = _cell().with_kpoints([((0.25, 0.25, 0.25), 0.5), (far, 0.5)])
    out = []
    for env in ({"QBX_FAST_FFT": "0"}, ROUTES[1] if route == "buffer" else {}):
        ctx = _ctx(s, monkeypatch, env)
        ctx.update_density()
        ctx.update_vhxc()
        e = ctx.energy(hpsi=True)
        out.append((ctx.density(), ctx.vr(), [ctx.get_kpoint_hpsi(i) for i in range(2)],
                    e["ekin"], [ctx.scf_step()["etotal"] for _ in range(2)]))
        ctx.close()
    (ra, va, ha, ka, ea), (rb, vb, hb, kb, eb) = out
    for a, b in [(ra, rb), (va, vb)] + list(zip(ha, hb)):
        np.testing.assert_allclose(b, a, rtol=0, atol=1e-12 * np.abs(a).max())
    assert abs(ka - kb) <= 1e-11 * abs(ka)
    np.testing.assert_allclose(eb, ea, rtol=1e-11)
