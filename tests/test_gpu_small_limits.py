"""The line between the few-launch step of small EulerRoe grids and the kernels for large
ones: both sides of each size limit against the oracle, bit for bit, captured and launched
one by one (grids of thousands of blocks, whose last block forms the timestep), and one
solver that goes from one path to the other and back."""
import numpy as np
import pytest

from _cases import describe_diff, random_state, same
from hydrodynamicsgpu_gb300 import _abi

pytestmark = pytest.mark.gpu

# the largest small grid and the smallest large one, and the launches of a step on each
LIMITS = [((200000,), "RungeKutta2", _abi.FP64, True), ((200001,), "RungeKutta2", _abi.FP64, False),
          ((200000,), "RungeKutta2", _abi.FP32, True), ((200001,), "RungeKutta2", _abi.FP32, False),
          ((256, 128), "ForwardEuler", _abi.FP64, True), ((241, 136), "ForwardEuler", _abi.FP64, False),
          ((400, 250), "RungeKutta3TVD", _abi.FP32, True), ((273, 367), "RungeKutta3TVD", _abi.FP32, False)]


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("size,integrator,prec,small", LIMITS)
def test_size_limits(hg, oracle_mod, size, integrator, prec, small, graphs):
    cfg = _abi.make_config(solver="EulerRoe", size=size, boundary=[("PERIODIC", "PERIODIC"), ("MIRROR", "FREEFLOW")],
                           limiter="Superbee", integrator=integrator, precision=prec)
    init = random_state(cfg, seed=sum(size), blocky=True)
    s, o = hg.Solver(cfg), oracle_mod.Oracle(cfg)
    try:
        s.set_graphs(graphs)
        s.resetState(init)
        o.set_state(init)
        for step in range(2):
            assert s.update(1) == o.update(1), "dt of step %d" % step
        a, b = s.getState(), o.get_state()
        assert same(a, b), describe_diff(a, b)
        # small: prologue, a kernel a stage (ForwardEuler: and its end), state check; large:
        # ghosts, eigenbasis and timestep before the stages, three or four kernels each
        stages = {"ForwardEuler": 1, "RungeKutta2": 2, "RungeKutta3TVD": 3}[integrator]
        few = 2 + stages + (integrator == "ForwardEuler")
        assert (s.kernels_per_step() == few) == small, s.kernels_per_step()
    finally:
        s.close()


@pytest.mark.parametrize("prec", [_abi.FP64, _abi.FP32])
@pytest.mark.parametrize("size,integrator", [((31, 26), "ForwardEuler"), ((90,), "ForwardEuler"),
                                             ((90,), "RungeKutta3TVD")])
def test_paths_alternate_on_one_solver(hg, oracle_mod, size, integrator, prec):
    cfg = _abi.make_config(solver="EulerRoe", size=size, boundary=[("MIRROR", "FREEFLOW"), ("PERIODIC", "PERIODIC")],
                           limiter="MinMod", integrator=integrator, precision=prec)
    init, other = random_state(cfg, seed=3), random_state(cfg, seed=4, blocky=True)
    pot = (.1 * np.sin(np.arange(int(np.prod(size))))).astype(init.dtype)
    s, o = hg.Solver(cfg), oracle_mod.Oracle(cfg)

    def check(what):
        a, b = s.getState(), o.get_state()
        assert same(a, b), "%s: %s" % (what, describe_diff(a, b))

    def step(what):
        assert s.update(1) == o.update(1), what
        check(what)

    def host_step(what, state):
        out, dt = s.update_host(state)
        o.set_state(state)
        assert dt == o.update(1), what
        assert same(out, o.get_state()), what

    try:
        for round_ in range(2):
            s.resetState(init)
            o.set_state(init)
            step("few launches")
            step("few launches again")
            host_step("host step on the large-grid kernels", s.getState())
            step("few launches after a host step")
            s.resetState(other, pot)
            o.set_state(other, pot)
            step("static potential")
            step("static potential again")
            s.resetState(other)
            o.set_state(other)
            step("few launches after a potential")
            host_step("host step after a reset", init)
            s.set_graphs(round_ == 1)
    finally:
        s.close()
