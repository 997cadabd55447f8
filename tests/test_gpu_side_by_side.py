"""Several handles stepped side by side, each on its own stream, against each one alone.

`step` returns before the updates have run, so the blocks of all handles share the GPU, chained
blocks that wait for their own handle's update among them. Fields must not depend on it."""
import numpy as np
import pytest

import mcb

pytestmark = pytest.mark.gpu

# one plane per block, a fraction of a wave, a whole wave, relaxed g, a shell
HANDLES = [((24, 24, 24), {}), ((48, 44, 40), {}), ((64, 64, 64), dict(tau_g=0.8)),
           ((97, 75, 61), dict(storage="f16")), ((40, 40, 40), dict(bc=mcb.BC_REF))]


def _solver(dims, kw):
    cfg = mcb.default_config(**(dict(nx=dims[0], ny=dims[1], nz=dims[2], bc=mcb.BC_PERIODIC,
                                     tau=0.7, sigma=0.05, width=4.0, sharp_c=0.0) | kw))
    s = mcb.Solver(cfg)
    s.set_fields(mcb.fill_phi_bubbles(*dims, cfg.bc, 4.0,
                                      [tuple(n * 0.48 for n in dims) + (min(dims) * 0.25,)]))
    return s


def test_handles_side_by_side_give_the_fields_of_each_alone():
    want = []
    for dims, kw in HANDLES:
        with _solver(dims, kw) as s:
            s.step(120)
            want.append((s.get_phi_q30().copy(), s.get("rho").copy()))
    solvers = [_solver(*h) for h in HANDLES]
    for _ in range(6):
        for s in solvers:
            s.step(20)
    for s, (phi, rho) in zip(solvers, want):
        assert np.array_equal(phi, s.get_phi_q30()) and np.array_equal(rho, s.get("rho"))
        s.close()
