"""The default work split and the chained launches that go with it: every plane is covered once
whatever the lattice, and an update sees the whole of the one before it, so the fields depend
neither on the split nor on graph replay (bit for bit)."""
import numpy as np
import pytest

import mcb

pytestmark = pytest.mark.gpu

# one tile column, ragged columns, grids of one, two and three blocks per SM, several waves,
# fewer planes than a chunk
LATTICES = [(8, 8, 4), (32, 32, 32), (34, 9, 33), (64, 64, 64), (97, 75, 61), (128, 100, 37),
            (256, 256, 24)]


def _run(cfg, steps=40):
    d = (cfg.nx, cfg.ny, cfg.nz)
    phi = mcb.fill_phi_bubbles(*d, cfg.bc, 4.0, [(d[0] * 0.47, d[1] * 0.52, d[2] * 0.4, 5.0)])
    with mcb.Solver(cfg) as s:
        s.set_fields(phi)
        s.step(steps)
        return s.schedule, s.get_phi_q30().copy(), s.get("ux").copy()


@pytest.mark.parametrize("dims", LATTICES)
@pytest.mark.parametrize("tau_g", [1.0, 0.8])
def test_default_split_gives_the_fields_of_any_split(dims, tau_g):
    kw = dict(nx=dims[0], ny=dims[1], nz=dims[2], bc=mcb.BC_PERIODIC, tau=0.7, tau_g=tau_g,
              sharp_c=0.0)
    (_, zc), phi, ux = _run(mcb.default_config(**kw))
    assert 1 <= zc <= dims[2]
    for other, graph in ((dims[2], 1), (3, 1), (-1, 1), (0, 0)):
        _, phi2, ux2 = _run(mcb.default_config(zchunk=other, use_graph=graph, **kw))
        assert np.array_equal(phi, phi2) and np.array_equal(ux, ux2), (other, graph)


def test_small_batch_runs_balanced_and_keeps_the_fields():
    cfgs = [mcb.default_config(nx=e, ny=e, nz=e, bc=mcb.BC_PERIODIC, storage="f16", tau=0.7,
                               sharp_c=0.0) for e in (12, 20, 28)]
    phis = [mcb.fill_phi_bubbles(c.nx, c.ny, c.nz, c.bc, 4.0,
                                 [(c.nx / 2 - 0.3, c.ny / 2, c.nz / 2 + 0.2, 4.0)])
            for c in cfgs]
    out = []
    for zc in (0, 5):
        for c in cfgs:
            c.zchunk = zc
        with mcb.Batch(cfgs) as b:
            for i, p in enumerate(phis):
                b.set_fields(i, p)
            b.step(5)
            assert b.schedule(0)[1] == (-1 if zc == 0 else 5)
            out.append([b.get(i, "phi") for i in range(len(cfgs))])
    for a, c in zip(*out):
        assert np.array_equal(a, c)


# above and below the size where tile variant 0 takes two cells per thread; ragged in x and y,
# one tile wide, wall and shell planes in the first and the last chunk
@pytest.mark.parametrize("dims", [(34, 33, 30), (96, 30, 12), (30, 50, 40), (32, 32, 32)])
@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("bc", [mcb.BC_PERIODIC, mcb.BC_WALLS_Z, mcb.BC_REF])
def test_tile_0_with_two_cells_per_thread_rounds_as_the_one_cell_tiles(dims, storage, bc):
    kw = dict(nx=dims[0], ny=dims[1], nz=dims[2], bc=bc, storage=storage, tau=0.65, sigma=0.3,
              sharp_c=0.0, gravity=0.0 if bc == mcb.BC_REF else 1e-3)
    ref = _run(mcb.default_config(variant=3, **kw))
    got = _run(mcb.default_config(variant=0, **kw))
    assert got[0][0] == 0 and ref[0][0] == 3
    assert np.array_equal(ref[1], got[1]) and np.array_equal(ref[2], got[2])
