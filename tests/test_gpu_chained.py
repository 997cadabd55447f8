"""Chained updates against updates that cannot overlap.

Consecutive collide kernels may overlap (the next one starts under the last blocks of the one
before it, and waits before it touches the lattice). The control runs the same updates one call
at a time and waits for the GPU after each. Every field has to be the same bit for bit, on grids
below and above one wave of blocks, for every form of the kernels."""
import numpy as np
import pytest

import mcb

pytestmark = pytest.mark.gpu

FIELDS = ("phi", "rho", "ux", "uy", "uz")
STEPS = 37  # the first update, two graph replays of 16, four single launches

CASES = {
    "one-cell-32": ((32, 32, 32), {}),
    "one-cell-f16-30": ((30, 26, 28), dict(storage="f16")),
    "odd": ((97, 75, 61), {}),
    "two-cells-as-0": ((96, 48, 40), dict(storage="f16")),
    "pair": ((128, 100, 37), {}),
    "pair-bf16": ((64, 64, 64), dict(storage="bf16")),
    "pair-waves": ((256, 256, 48), dict(storage="f16")),
    "pair-balanced": ((64, 60, 50), dict(zchunk=-2)),
    "walls": ((64, 40, 44), dict(bc=mcb.BC_WALLS_Z, gravity=1e-5)),
    "shell": ((64, 48, 52), dict(bc=mcb.BC_REF)),
    "relaxed": ((64, 64, 64), dict(tau_g=0.8)),
    "relaxed-f16": ((34, 33, 47), dict(tau_g=0.8, storage="f16")),
    "relaxed-f16-pair": ((64, 64, 72), dict(tau_g=0.8, storage="f16")),
    "populations": ((48, 44, 40), dict(g_mode=mcb.G_POPULATIONS)),
    "d3q27": ((60, 45, 50), dict(velocity_set=27)),
    "d3q27-f16": ((60, 45, 50), dict(velocity_set=27, storage="f16")),
    "ratio": ((48, 48, 48), dict(rho_in=10.0, sigma=0.01)),
}


def _start(dims, bc, seed=3):
    nx, ny, nz = dims
    phi = mcb.fill_phi_bubbles(nx, ny, nz, bc, 4.0,
                               [(nx * 0.47, ny * 0.52, nz * 0.45, min(dims) * 0.25)])
    if bc == mcb.BC_REF:
        return phi, None
    rng = np.random.default_rng(seed)
    return phi, [(1e-2 * rng.standard_normal(phi.shape)).astype(np.float32) for _ in range(3)]


def _fields(s):
    return {k: s.get(k).copy() for k in FIELDS} | {"q30": s.get_phi_q30().copy()}


@pytest.mark.parametrize("name", CASES)
def test_chained_updates_equal_updates_run_one_at_a_time(name):
    dims, kw = CASES[name]
    cfg = mcb.default_config(**(dict(nx=dims[0], ny=dims[1], nz=dims[2], bc=mcb.BC_PERIODIC,
                                     tau=0.7, sigma=0.05, width=4.0, sharp_c=0.0) | kw))
    phi, u = _start(dims, cfg.bc)
    with mcb.Solver(cfg) as s:
        s.set_fields(phi, *(u or (None,) * 3))
        for _ in range(STEPS):
            s.step(1)
            s.synchronize()
        want = _fields(s)
        for graph in (True, False):
            s.set_fields(phi, *(u or (None,) * 3))
            if graph:
                s.step(STEPS)
            else:
                for _ in range(STEPS):
                    s.step(1)
            got = _fields(s)
            for k in want:
                assert np.array_equal(want[k], got[k]), (k, graph)


@pytest.mark.parametrize("kw", [dict(zchunk=0), dict(zchunk=5), dict(zchunk=-1),
                                dict(zchunk=0, tau_g=0.8), dict(zchunk=0, storage="f32")])
def test_chained_batch_updates_equal_updates_run_one_at_a_time(kw):
    cfgs = [mcb.default_config(**(dict(nx=e, ny=e, nz=e, bc=mcb.BC_PERIODIC, storage="f16",
                                       tau=0.7, sigma=0.05, width=4.0, sharp_c=0.0) | kw))
            for e in (20, 36, 52, 28)]
    starts = [_start((c.nx, c.ny, c.nz), c.bc, i) for i, c in enumerate(cfgs)]

    def run(apart):
        with mcb.Batch(cfgs) as b:
            for i, (phi, u) in enumerate(starts):
                b.set_fields(i, phi, *u)
            if apart:
                for _ in range(STEPS):
                    b.step(1)
                    b.get(0, "phi")  # waits for the update
            else:
                b.step(STEPS)
            return [b.get(i, k) for i in range(len(cfgs)) for k in FIELDS]

    for a, c in zip(run(True), run(False)):
        assert np.array_equal(a, c)
