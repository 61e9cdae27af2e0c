"""The sums behind the adaptive speed: float32, in an order that neither the
grid nor the block's size changes.  The walk's swing and traction terms are
restated here operation by operation (each correctly rounded), so the speed
after one step is known to the last bit.

Start speed and previous forces are chosen so that the rule sets the speed to
its target, jt * efficiency * traction / swing."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F = np.float32


def _tree_sum(v):
    """The sum over the last axis of 32, as a warp's shuffles form it."""
    for o in (16, 8, 4, 2, 1):
        v = v + v[..., np.arange(32) ^ o]
    return v[..., 0]


def _chain(v):
    s = np.zeros(v.shape[1:], F)
    for row in v:
        s = s + row
    return s


def _total(terms):
    groups = -(-len(terms) // 32)
    v = np.zeros((groups, 32), F)
    v.reshape(-1)[:len(terms)] = terms
    part = _tree_sum(v)
    rows = np.zeros((-(-groups // 1024), 1024), F)
    rows.reshape(-1)[:groups] = part
    return _chain(_tree_sum(_chain(rows).reshape(32, 32))[:, None])[0]


def _norm(d):
    x, y = d[:, 0].astype(np.float64), d[:, 1]
    return np.sqrt((x * x + (y * y).astype(np.float64)).astype(F))


@pytest.mark.parametrize("n", [40, 8193, 40000, 100001])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_speed_sums_are_in_the_stated_order(n, seed):
    from gpugraphlayout_b200 import Engine
    rng = np.random.default_rng(seed)
    ids = np.arange(n, dtype=np.uint32)
    e = Engine(n, ids, np.roll(ids, -1), scale=2.0)
    xy = rng.uniform(-1e3, 1e3, (n, 2)).astype(F)
    e.set_positions(xy)
    e.step(1)
    f = e.forces()[0]
    prev = (f * F(0.5) + rng.normal(0, 0.1 * np.abs(f).mean(), f.shape)).astype(F)
    order = e.sort_order()
    fs, ps = f[order], prev[order]
    mass = F(3.0)
    swing = _total(mass * _norm(fs - ps))
    traction = _total(mass * (_norm(fs + ps) * F(0.5)))
    jitter = F(0.05 * np.float64(np.sqrt(F(n))))
    jt = max(np.sqrt(jitter), min(F(10.0), jitter * traction / F(n) ** F(2)))
    target = jt * traction / swing
    e.set_positions(xy)
    e.set_speed_state(float(F(1.5) * target), 1.0, prev)
    e.step(1)
    assert np.array_equal(e.forces()[0], f)
    assert F(e.speed_state()[0]) == target
