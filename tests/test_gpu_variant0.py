"""Tile variant 0 gives the same fields from either of its kernels, one cell or two cells per
thread: which one runs depends on the number of cells in all, so a case alone and the same case
in a batch may take different ones. Both kernels name every fused operation in their source."""
import numpy as np
import pytest

import mcb

pytestmark = pytest.mark.gpu

FIELDS = ("phi", "rho", "ux", "uy", "uz")
STORAGES = ["f32", "f16", "bf16"]
MODES = [mcb.BC_PERIODIC, mcb.BC_WALLS_Z, mcb.BC_REF]
STEPS = 25


def _config(dims, bc, storage, **kw):
    return mcb.default_config(nx=dims[0], ny=dims[1], nz=dims[2], bc=bc, storage=storage,
                              tau=0.65, sigma=0.3, sharp_c=0.0,
                              gravity=0.0 if bc == mcb.BC_REF else 1e-3, **kw)


def _start(dims, bc):
    phi = mcb.fill_phi_bubbles(*dims, bc, 4.0, [(dims[0] * 0.47, dims[1] * 0.52, dims[2] * 0.4,
                                                 min(dims) * 0.2)])
    rng = np.random.default_rng(11)
    return phi, [(2e-2 * rng.standard_normal(phi.shape)).astype(np.float32) for _ in range(3)]


def _alone(dims, bc, storage, **kw):
    phi, u = _start(dims, bc)
    with mcb.Solver(_config(dims, bc, storage, **kw)) as s:
        s.set_fields(phi, *u)
        s.step(STEPS)
        return [s.get(k).copy() for k in FIELDS] + [s.get_phi_q30().copy()]


@pytest.mark.parametrize("bc", MODES)
@pytest.mark.parametrize("storage", STORAGES)
@pytest.mark.parametrize("dims", [(66, 33, 30), (30, 50, 40)])
def test_two_cells_per_thread_give_the_fields_of_one(dims, storage, bc):
    one_cell = _alone(dims, bc, storage, variant=3)
    for zchunk in (0, 7, -1):
        two_cells = _alone(dims, bc, storage, variant=0, zchunk=zchunk)
        for a, b in zip(one_cell, two_cells):
            assert np.array_equal(a, b), zchunk


@pytest.mark.parametrize("bc", MODES)
@pytest.mark.parametrize("storage", STORAGES)
def test_a_case_gives_the_same_fields_alone_and_in_a_batch(storage, bc):
    all_dims = [(30, 28, 26), (34, 17, 40), (20, 24, 16)]  # each below 2^15 cells, not in all
    assert max(x * y * z for x, y, z in all_dims) < 2 ** 15 < sum(x * y * z for x, y, z in all_dims)
    for zchunk in (6, -1):
        with mcb.Batch([_config(d, bc, storage, variant=0, zchunk=zchunk)
                        for d in all_dims]) as b:
            for i, d in enumerate(all_dims):
                phi, u = _start(d, bc)
                b.set_fields(i, phi, *u)
            b.step(STEPS)
            for i, d in enumerate(all_dims):
                for k, want in zip(FIELDS, _alone(d, bc, storage, variant=0)):
                    assert np.array_equal(want, b.get(i, k)), (d, k, zchunk)
