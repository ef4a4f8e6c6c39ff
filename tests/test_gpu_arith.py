"""The kernels' other replacements for the FP64 unit against it, bit for bit, over seeded
operands of every class: the square root, quotients by a divisor whose reciprocal was formed
on the device and on the host, the grouped products, quotients and roots, the sum of two
equal numbers, and the FP32 flux's product-difference beside midpoints of two floats."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_forms_match_the_fp64_unit(hg, seed):
    bad = hg.arith_selftest(cases=1 << 25, seed=seed)
    assert bad == dict.fromkeys(bad, 0)
