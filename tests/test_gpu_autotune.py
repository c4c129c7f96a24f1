"""The autotuner of the fused 3D sweep times each launch once: shapes that differ in name only
share their time, every other offered shape has its own, and the model runs the fastest."""
import pytest

from helpers import Pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_same_launch_is_timed_once(dtype):
    slip = ("slip", (0.0, 0.0, 0.0))
    p = Pair((70, 40, 36), ((slip, slip),) * 3, dtype=dtype, library="strict")
    best, ms = p.model.autotune(iters=2)
    names = list(ms)
    timed = {n: t for n, t in ms.items() if t > 0}
    assert ms["tile32x8_zb32_trim"] == ms["tile32x8_zb32"] > 0
    assert ms["tile64x8_zb32_trim"] == ms["tile64x8_zb32"] and (ms["tile64x8_zb32"] > 0) == (dtype == "f32")
    assert timed[names[best]] == min(timed.values())
    shapes = len(timed) - len([n for n in timed if n.endswith("_trim")])
    p.oracle.advance(3 * shapes)  # a warm-up and two timed iterations of each launch
    bad = p.bitwise_equal()
    p.close()
    assert not bad, bad
