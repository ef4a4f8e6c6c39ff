"""bench.py's FP64 roofline with the table that the measurement uses: the RK4 step's launches
as the solver now profiles them, every kernel known to the table; and the reference arm, which
runs the reference's kernels or says that it cannot."""
import importlib.util
import json
import os
import types

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
STEP = {"boundary": 1, "roe_eigenbasis": 1, "cfl_min_reduce": 1, "roe_delta_q_tilde": 4, "roe_flux": 4,
        "flux_divergence_combine": 4, "state_check": 1}


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench_roofline", os.path.join(REPO, "bench.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


@pytest.mark.parametrize("steps", [1, 2, 5])
def test_current_table(bench, steps):
    prof = {k: (n * steps, .1) for k, n in STEP.items()}
    per_update, achieved, frac = bench.fp64_roofline(prof, 7.8e8, 5.3e11, bench.FP64_PIPE_NOW)
    # 49.97 + 3.97 + 1.98 + 4 (29.79 + 87.39 + 25.80), each within .005 of its count
    assert per_update == pytest.approx(627.84, abs=.01)
    assert achieved == pytest.approx(per_update * 7.8e8) and frac == pytest.approx(achieved / 5.3e11)
    assert bench.uncounted_kernels(prof) == []


def test_a_kernel_missing_from_the_table_is_named(bench):
    prof = {k: (n, .1) for k, n in STEP.items()}
    table = {k: v for k, v in bench.FP64_PIPE_NOW.items() if k != "roe_flux"}
    assert bench.uncounted_kernels(prof, table) == ["roe_flux"]


def test_reference_arm_is_the_reference_or_unavailable(bench, monkeypatch, capsys):
    import pyoracle

    def no_source(*a, **k):
        raise RuntimeError("no reference\nsources")

    monkeypatch.setattr(pyoracle, "refcl_available", lambda cfg=None: False)
    monkeypatch.setattr(pyoracle, "build_refcl", no_source)
    assert bench.run_reference(types.SimpleNamespace(size=128, steps=1, warmup=3, gpus=1)) == 0
    line = json.loads(capsys.readouterr().out)
    assert line == {"impl": "reference",
                    "unavailable": "the reference's kernels cannot be built here: no reference sources"}


@pytest.mark.gpu
def test_profiled_step_is_counted(bench, hg):
    from hydrodynamicsgpu_gb300 import _abi
    from hydrodynamicsgpu_gb300 import initconds as ic
    cfg = _abi.make_config(solver="EulerRoe", size=(128, 128), boundary="PERIODIC", limiter="MinMod",
                           integrator="RungeKutta4")
    s = hg.Solver(cfg)
    s.resetState(ic.kelvin_helmholtz(size=(128, 128), seed=0).reshape(-1))
    prof = s.profile(2)
    s.close()
    assert {k: v[0] // 2 for k, v in prof.items()} == STEP
    assert bench.uncounted_kernels(prof) == []
