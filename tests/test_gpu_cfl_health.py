"""The CFL kernels' health bit: a NaN quotient, which needs an infinite cell size (a domain
wider than the largest number) and an infinite wave speed (an infinite energy at rest), is
reported by hgpu_health and by hgpu_synchronize; either one alone gives no NaN and no bit.
1D and small 2D EulerRoe grids take the few-launch step, the others the kernels for large
grids."""
import numpy as np
import pytest

from hydrodynamicsgpu_gb300 import _abi

pytestmark = pytest.mark.gpu

LIMIT = {_abi.FP64: 1e308, _abi.FP32: 3e38}


def uniform(size, prec, energy):
    u = np.zeros((int(np.prod(size)), len(size) + 2), dtype=np.float64 if prec == _abi.FP64 else np.float32)
    u[:, 0] = 1
    u[:, -1] = energy
    return u.reshape(-1)


@pytest.mark.parametrize("prec", [_abi.FP64, _abi.FP32])
@pytest.mark.parametrize("size", [(40,), (40, 36), (12, 10, 8)])
@pytest.mark.parametrize("solver,integrator", [("EulerRoe", "ForwardEuler"), ("EulerRoe", "RungeKutta2"),
                                               ("EulerHLLC", "RungeKutta2"), ("EulerHLL", "RungeKutta2")])
def test_nan_timestep_is_reported(hg, solver, integrator, size, prec):
    big = LIMIT[prec]
    for wide, energy, expect in ((True, np.inf, _abi.HEALTH_NONFINITE_DT), (False, np.inf, 0), (True, 2.5, 0)):
        x = (big if wide else .5,) * 3
        cfg = _abi.make_config(solver=solver, size=size, xmin=tuple(-v for v in x), xmax=x, boundary="FREEFLOW",
                               limiter="MinMod", integrator=integrator, precision=prec)
        s = hg.Solver(cfg)
        try:
            s.set_health_mode(_abi.HEALTH_OFF)               # only the CFL kernels write the word
            s.resetState(uniform(size, prec, energy))
            s.update(1, want_dt=False)
            if expect:
                with pytest.raises(hg.HgpuError) as e:
                    s.synchronize()
                assert e.value.status == _abi.ERR_NONFINITE
            else:
                s.synchronize()
            assert s.health() & _abi.HEALTH_NONFINITE_DT == expect, (wide, energy)
        finally:
            s.close()
