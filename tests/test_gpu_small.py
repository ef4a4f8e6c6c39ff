"""EulerRoe steps of small grids in few launches (roe_small.cu) against the oracle, bit for
bit: sizes below, at and past the edges of the tiles (29 cells in 1D, 8 x 8 in 2D), every
boundary method with NONE, limiters with kernels of their own and without, tableaus with
fractional alphas, ForwardEuler, states with flat regions, FP32."""
import pytest

from _cases import describe_diff, random_state, same
from hydrodynamicsgpu_gb300 import _abi

pytestmark = pytest.mark.gpu

BOUNDARIES = ["PERIODIC", "MIRROR", "FREEFLOW", [("NONE", "MIRROR"), ("FREEFLOW", "NONE")]]
SCHEMES = [("ForwardEuler", "Superbee"), ("RungeKutta2", "MinMod"), ("RungeKutta3TVD", "Koren"),
           ("RungeKutta4", "MonotizedCentral"), ("RungeKutta4NonTVD", "MinMod")]


@pytest.mark.parametrize("prec", [_abi.FP64, _abi.FP32])
@pytest.mark.parametrize("size", [(6,), (28,), (29,), (30,), (58,), (59,), (500,), (6, 6), (8, 8), (9, 7), (16, 17),
                                  (33, 24), (50, 61)])
def test_small_steps(hg, oracle_mod, size, prec):
    for k, boundary in enumerate(BOUNDARIES):
        for integrator, limiter in SCHEMES:
            cfg = _abi.make_config(solver="EulerRoe", size=size, boundary=boundary, limiter=limiter, precision=prec,
                                   integrator=integrator, xmax=(.5, .25, .5))
            init = random_state(cfg, seed=k + sum(size), blocky=k % 2 == 1)
            s, o = hg.Solver(cfg), oracle_mod.Oracle(cfg)
            try:
                s.resetState(init)
                o.set_state(init)
                for step in range(3):
                    what = "%s %s %s, step %d" % (boundary, integrator, limiter, step)
                    assert s.update(1) == o.update(1), "%s: dt" % what
                    a, b = s.getState(), o.get_state()
                    assert same(a, b), "%s: %s" % (what, describe_diff(a, b))
            finally:
                s.close()
