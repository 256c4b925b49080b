"""Count, plan and scatter in one call against the three calls: around a round of 1024 slots and the one-launch limit."""
import numpy as np
import pytest

from helpers import dev, host

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 4, 31, 1023, 1024, 1025, 2048, 2049, 5000])
def test_route_equals_steps(lkb, n):
    lkb.init(0)
    rng = np.random.default_rng(n)
    idx = dev((64 * rng.random(n) ** 2).astype(np.int32))
    z = lambda k: torch.full((k,), -7, dtype=torch.int32, device="cuda")
    a, b = ([z(64), z(64), z(4 * (n // 64 + 65)), z(1), z(n)] for _ in range(2))
    lkb.zero_i32(a[0], 64)
    lkb.k_pf_moe_count(idx, n, a[0])
    lkb.k_pf_moe_plan(a[0], a[1], a[2], a[3])
    lkb.k_pf_moe_scatter(idx, n, a[1], a[4])
    lkb.k_pf_moe_route(idx, n, b[0], b[1], b[2], b[3], b[4])
    for x, y in zip(a, b):
        assert np.array_equal(host(x), host(y))
