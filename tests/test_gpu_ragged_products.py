"""Split products of band and projector counts that fill no whole 128 x 128 tile
(and fewer than one, and just over one and two), on the tcgen05 kernel: E_nl, H
psi and one step of the mixed path against the cuBLAS split products
(QBX_GEMM_BACKEND=0) from the same coefficients.

Both form hi*hi + hi*lo + lo*hi of the same BF16 splits (16 significant bits);
they differ in the FP32 sums only: 2^-24 per addition of a chain, 2e-6 of the
largest value after some hundred blocks.  The step's rotation is split TF32 in
both, cuBLAS accumulating in one FP32 chain: 2e-5.
"""
import os

import numpy as np
import pytest

from qbx import capi, systems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bands", [1, 15, 33, 65, 97, 130, 257])
def test_ragged_products(bands):
    pos = systems.diamond_supercell(10.26, 1, 0.03, 4)[:7]
    s = systems.System("box", np.diag([15.0, 12.0, 13.0]), [systems.SI], [(0, p) for p in pos],
                       20.0, bands, "LDA", 11)
    out = []
    for backend in ("1", "0"):
        os.environ["QBX_GEMM_BACKEND"] = backend
        try:
            ctx = capi.from_system(s, precision=capi.MIXED)
        finally:
            os.environ.pop("QBX_GEMM_BACKEND")
        ctx.update_density()
        ctx.update_vhxc()
        e = ctx.energy(hpsi=True, forces=True)
        h = ctx.get_hpsi()
        ctx.scf_step()
        out.append((e["enl"], e["fion"], h, ctx.get_coeffs()))
        ctx.close()
    (ea, fa, ha, ca), (eb, fb, hb, cb) = out
    assert abs(ea - eb) <= 2e-6 * abs(eb)
    np.testing.assert_allclose(fa, fb, rtol=0, atol=2e-6 * max(1.0, np.abs(fb).max()))
    np.testing.assert_allclose(ha, hb, rtol=0, atol=2e-6 * np.abs(hb).max())
    np.testing.assert_allclose(ca, cb, rtol=0, atol=2e-5 * np.abs(cb).max())


@pytest.mark.parametrize("batch", [False, True])
def test_captured_ragged_steps(batch):
    """Captured steps of ragged band counts, with and without forces and in any
    order, take the workspaces that their first, eager run sized: the eager
    steps' energies and forces (1e-7 of them: atomic sums through three steps)."""
    systems_ = []
    for bands, edge in ((33, 11.0), (130, 12.5)):
        pos = systems.diamond_supercell(10.26, 1, 0.03, 4)[:7]
        systems_.append(systems.System("box", np.diag([edge, 11.5, 12.0]), [systems.SI],
                                       [(0, p) for p in pos], 20.0, bands, "PBE", 11))
    order = [False, False, False, True, True, True, False, True]
    runs = []
    for graph in (False, True):
        ctxs = [capi.from_system(s, precision=capi.MIXED) for s in systems_]
        rows = []
        for c in ctxs:
            c.set_step_graph(graph)
        for forces in order:
            if batch and graph:
                rows.append([e["etotal"] for e in capi.scf_step_batch(ctxs, forces=forces)])
            else:
                e = [c.scf_step(forces=forces) for c in ctxs]
                rows.append([x["etotal"] for x in e])
        runs.append(np.array(rows))
        for c in ctxs:
            c.close()
    np.testing.assert_allclose(runs[1], runs[0], rtol=1e-7)
