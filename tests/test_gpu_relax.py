"""The relaxation's stored quotients against the oracle, bit for bit: one, two and more
sweeps a callback (first, storing and plain sweeps in every combination), one plane of
quotients (equal dx) and one per axis, single interior rows, ragged rows."""
import pytest

from test_gpu_gravity import compare
from hydrodynamicsgpu_gb300 import _abi
from hydrodynamicsgpu_gb300 import initconds as ic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sweeps", [1, 2, 3])
@pytest.mark.parametrize("size", [(9,), (24, 24), (21, 5), (35, 19), (11, 11, 11), (13, 6, 10)])
def test_stored_quotients(hg, oracle_mod, size, sweeps):
    cfg = _abi.make_config(solver="EulerRoe", size=size, integrator="RungeKutta2Heun", use_gravity=True,
                           boundary="FREEFLOW", limiter="MinMod", gauss_seidel_max_iter=sweeps)
    compare(hg, oracle_mod, cfg, ic.gravity_blobs(size=size, seed=sweeps), steps=2)
