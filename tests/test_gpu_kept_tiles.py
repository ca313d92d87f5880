"""When the tiles of the density pass are kept for the H psi pass (fft.cu,
tile_area): a step that keeps them launches fewer kernels than one that
transforms every band again.  Device memory is taken by a tensor of the test's
own, so that the library finds as much room as a case says.
"""
import gc

import numpy as np
import pytest

from qbx import capi, systems

pytestmark = pytest.mark.gpu

GB = 1 << 30


def _load(ctx, s):
    """The system's cell, atoms and coefficients into a context."""
    ctx.set_cell(s.cell, s.ecut, s.nbands, s.xc)
    hkl = s.miller()
    if not np.array_equal(ctx.miller(), hkl):
        ctx.set_coeff_order(hkl)
    for sp in s.species:
        ctx.add_species(sp.zval, sp.mesh_spacing, sp.local_potential(), sp.projectors(),
                        [d for _, d in sp.dmatrix()])
    counts = [len(s.positions(i)) for i in range(len(s.species))]
    ctx.set_atoms(counts, np.concatenate([s.positions(i) for i in range(len(s.species))]))
    ctx.set_coeffs(s.coefficients(hkl))
    ctx.gram()


def _launches(ctx):
    """Kernels of an eager step, after one that allocates."""
    ctx.scf_step()
    n = ctx.launch_count()
    ctx.scf_step()
    return ctx.launch_count() - n


class _Full:
    """All device memory but `left` bytes taken."""

    def __init__(self, left):
        import torch
        gc.collect()
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        self.block = torch.empty(max(0, free - left), dtype=torch.uint8, device="cuda")

    def release(self):
        import torch
        self.block = None
        torch.cuda.empty_cache()


@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED])
def test_room_is_looked_for_again_with_each_cell(precision):
    """A cell that found no room does not keep later cells of its context from
    keeping their tiles."""
    s = systems.si8()
    ctx = capi.Context(0, precision)
    _load(ctx, s)
    kept = _launches(ctx)
    full = _Full(3 * GB)
    try:
        _load(ctx, s)
        again = _launches(ctx)
    finally:
        full.release()
    assert again > kept
    _load(ctx, s)
    assert _launches(ctx) == kept
    ctx.close()


def test_as_much_room_is_left_as_the_tiles_take():
    """256 bands of the 512-atom cell in FP64, 2.9 GB of tiles: kept where 12 GB are
    free, not where 8 GB are, so that a context made next still finds its memory."""
    s = systems.si512().band_sample(256)
    ctx = capi.Context(0, capi.FP64)
    _load(ctx, s)
    _, _, grid, hkl = capi.host_basis(s.cell, s.ecut)
    need = s.nbands // 2 * 16 * (2 * int(hkl[:, 0].max()) + 1) * grid[1] * grid[2]
    assert 2 * need + 4 * GB < 12 * GB and need + 4 * GB < 8 * GB < 2 * need + 4 * GB
    used = []
    for left in (8 * GB, 12 * GB):
        _load(ctx, s)
        full = _Full(left)
        try:
            used.append(_launches(ctx))
        finally:
            full.release()
    ctx.close()
    assert used[0] > used[1]
