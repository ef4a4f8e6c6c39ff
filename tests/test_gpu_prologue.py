"""What precedes a step's stages against the oracle, bit for bit: the ghost fill of every
axis in one launch (and axis by axis where an axis has 5 cells, whose ghosts copy ghosts),
every mix of boundary methods with NONE among them, and the timestep from each axis's
largest wave speed on axes of different cell sizes."""
import itertools

import pytest

from _cases import describe_diff, random_state, same
from hydrodynamicsgpu_gb300 import _abi

pytestmark = pytest.mark.gpu

SIZES = [(5,), (6,), (7,), (6, 6), (6, 9), (5, 7), (7, 5), (41, 6), (6, 7, 8), (5, 6, 6), (6, 6, 5), (9, 6, 7)]
MIXES = [("PERIODIC", "PERIODIC"), ("MIRROR", "FREEFLOW"), ("NONE", "MIRROR"), ("FREEFLOW", "NONE"),
         ("PERIODIC", "MIRROR")]


@pytest.mark.parametrize("solver,prec", itertools.product(["EulerRoe", "EulerHLLC"], [_abi.FP64, _abi.FP32]))
@pytest.mark.parametrize("size", SIZES)
def test_ghosts_and_timestep(hg, oracle_mod, size, solver, prec):
    for k in range(len(MIXES)):
        boundary = [MIXES[(k + a) % len(MIXES)] for a in range(3)]
        cfg = _abi.make_config(solver=solver, size=size, boundary=boundary, limiter="MinMod", precision=prec,
                               integrator="RungeKutta2", xmax=(.5, .125, 2.))
        init = random_state(cfg, seed=10 * k + len(size))
        s, o = hg.Solver(cfg), oracle_mod.Oracle(cfg)
        try:
            s.resetState(init)
            o.set_state(init)
            for step in range(3):
                assert s.update(1) == o.update(1), "%s: dt of step %d" % (boundary, step)
                a, b = s.getState(), o.get_state()
                assert same(a, b), "%s, step %d: %s" % (boundary, step, describe_diff(a, b))
        finally:
            s.close()
