"""The grouped arithmetic of the Roe kernels (fp64ops.cuh GroupPlain, GroupZeros and the
dense sums) against the oracle, bit for bit: states whose values, differences and zeros put
the lanes of one warp in different groups -- gas at rest, exact zeros beside noise, tiny
velocities down to subnormal numbers, and states scaled out of the window of ordinary
magnitudes."""
import numpy as np
import pytest

from _cases import describe_diff, same
from hydrodynamicsgpu_gb300 import _abi
from hydrodynamicsgpu_gb300 import initconds as ic

pytestmark = pytest.mark.gpu

KINDS = ["rest", "stripes", "tiny", "subnormal", "small", "large"]


def state(size, kind):
    shape = tuple(reversed(list(size) + [1] * (3 - len(size))))
    rng = np.random.default_rng(len(size))
    rho = 1. + .5 * (rng.uniform(size=shape) > .7)
    p = np.ones(shape)
    v = [rng.uniform(-.3, .3, shape) for _ in range(3)]
    if kind in ("rest", "stripes"):
        moving = rng.uniform(size=shape) > (.9 if kind == "rest" else .5)
        v = [x * moving for x in v]
    if kind == "tiny":
        v = [x * 10. ** rng.uniform(-200, 0, shape) for x in v]
    if kind == "subnormal":
        v = [x * 10. ** rng.uniform(-320, -300, shape) for x in v]
    u = ic.build_state_euler(len(size), 1.4, rho, v[0], v[1], v[2], p)
    if kind == "small":
        u = u * 2. ** -500
    if kind == "large":
        u = u * 2. ** 490
    return u.reshape(-1)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("size,solver", [((70,), "EulerRoe"), ((37, 21), "EulerRoe"), ((37, 21), "EulerHLLC"),
                                         ((37, 21), "EulerHLL"), ((12, 11, 9), "EulerRoe"), ((12, 11, 9), "EulerHLLC")])
def test_mixed_magnitudes(hg, oracle_mod, size, solver, kind):
    for integrator, limiter in (("ForwardEuler", "Superbee"), ("RungeKutta2", "MinMod"), ("RungeKutta3TVD", "Koren")):
        cfg = _abi.make_config(solver=solver, size=size, boundary="FREEFLOW", limiter=limiter, integrator=integrator)
        u = state(size, kind)
        s, o = hg.Solver(cfg), oracle_mod.Oracle(cfg)
        try:
            s.resetState(u)
            o.set_state(u)
            for step in range(3):
                assert s.update(1) == o.update(1), "%s, dt of step %d" % (integrator, step)
                a, b = s.getState(), o.get_state()
                assert same(a, b), "%s, step %d: %s" % (integrator, step, describe_diff(a, b))
        finally:
            s.close()
