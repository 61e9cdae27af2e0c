"""The tree build at the sizes and crowdings where its paths change.

One block sorts in shared memory up to 512 bodies; more blocks by buckets up
to 1024 bodies each, and beyond that, or where more than 128 bodies share one
of the buckets' squares, by radix passes with a fix-up.  The choice looks at
the tree before, so each layout is built first after a fresh start and again
after another one.  The body order is the oracle's exactly on every path; the
repulsion sums the same terms in another order (float32: under 1e-4 relative
for sums of up to 1500 terms, the suite's bar).
"""
import numpy as np
import pytest

from conftest import rel_rmse

pytestmark = pytest.mark.gpu

TOL = 1e-4


def _graph(n):
    from oracle import oracle as O
    s = np.arange(n, dtype=np.uint32)
    return O.Graph(s, np.roll(s, -1)) if n > 2 else O.Graph(s[:1], s[1:2])


def _uniform(n, seed):
    """Two bodies at opposite corners pin the root box to [-1024, 1024]^2; the
    others keep out of the level-6 cell [0, 32)^2."""
    rng = np.random.default_rng(seed)
    xy = rng.uniform(-1000, 1000, (n, 2))
    xy[:, 0] = np.where((xy >= 0).all(1) & (xy < 32).all(1), xy[:, 0] - 500, xy[:, 0])
    xy[0], xy[1] = (-1024, -1024), (1024, 1024)
    return xy.astype(np.float32)


def _crowd(n, count, seed, kind):
    """`count` bodies in that cell: spread over it, or in one cell of level 24;
    "equal": some of them share all 64 bits of their keys."""
    xy = _uniform(n, seed)
    rng = np.random.default_rng(seed + 1)
    w = 30.0 if kind == "spread" else 2048.0 / 2 ** 24
    side = int(np.ceil(np.sqrt(count)))
    grid = rng.permutation(side * side)[:count]
    xy[2:2 + count, 0] = (grid % side + 0.5) * (w / side)
    xy[2:2 + count, 1] = (grid // side + 0.5) * (w / side)
    if kind == "equal":
        xy[2:5] = [(1e-9, 1e-9), (3e-9, 1e-9), (2e-9, 4e-9)]
    return xy


def _check(e, xy, mass, forces):
    from oracle import oracle as O
    e.set_positions(xy)
    e.step(1)
    st = e.stats()
    assert st["device_error"] == 0
    t = O.Tree(xy, mass)
    assert np.array_equal(e.sort_order(), t.sort().astype(np.uint32))
    if forces:
        tot, ga = e.forces()
        ref, overflow, _ = t.repulsion(10.0)
        assert overflow or rel_rmse(tot - ga, ref) <= TOL


# 1 and 2 blocks; the edges of 148 blocks' tiles of 512 and 1024 bodies
@pytest.mark.parametrize("n", [2, 31, 33, 511, 512, 513, 1025, 4737, 75776, 75777, 151552, 151553])
def test_order_at_tile_edges(n):
    from gpugraphlayout_b200 import Engine
    g = _graph(n)
    e = Engine(g.n, g.sources, g.targets, scale=10.0)
    for seed in (1, 2):
        _check(e, _uniform(n, seed), g.mass, n <= 5000)


@pytest.mark.parametrize("kind", ["spread", "tight", "equal"])
@pytest.mark.parametrize("n,count", [(500, 127), (500, 128), (500, 129), (500, 400),
                                     (3000, 128), (3000, 129), (3000, 1500)])
def test_order_of_crowded_bodies(n, count, kind):
    from gpugraphlayout_b200 import Engine
    g = _graph(n)
    e = Engine(g.n, g.sources, g.targets, scale=10.0)
    for seed in (1, 3):  # the second build knows that the first one's were crowded
        _check(e, _crowd(n, count, seed, kind), g.mass, kind == "spread")
    _check(e, _uniform(n, 5), g.mass, True)
    _check(e, _crowd(n, count, 7, kind), g.mass, kind == "spread")


@pytest.mark.parametrize("threads", [None, 256])
def test_batch_order_at_team_edges(threads):
    """The teams' sizes (1, 4 and 8 blocks) and a block's staging; 256 threads:
    one block per graph, whatever its size."""
    from gpugraphlayout_b200 import BatchEngine
    from oracle import oracle as O
    sizes = [2, 512, 513, 2048, 2049, 2304, 2305, 8192, 8193]
    graphs = [_graph(n) for n in sizes]
    b = BatchEngine([(g.n, g.sources, g.targets) for g in graphs], scale=10.0)
    if threads:
        b.configure(0, threads, threads)
    for seed in (1, 2):
        xys = [_crowd(n, n // 8, seed, "spread") if i % 3 == 2 else _uniform(n, seed)
               for i, n in enumerate(sizes)]
        b.set_positions(np.concatenate(xys))
        b.step(1)
        order = b.sort_order()
        tot, ga = b.forces()
        for i, (g, xy) in enumerate(zip(graphs, xys)):
            t = O.Tree(xy, g.mass)
            assert np.array_equal(b.part(order, i), t.sort().astype(np.uint32)), i
            ref, overflow, _ = t.repulsion(10.0)
            assert overflow or rel_rmse(b.part(tot - ga, i), ref) <= TOL, i


@pytest.mark.parametrize("n", [300, 3000])
def test_one_call_of_many_iterations_equals_one_call_per_iteration(n):
    """Calls replay four iterations at a time and the rest one by one: the
    same arithmetic bit for bit."""
    from gpugraphlayout_b200 import Engine
    g = _graph(n)
    out = []
    for calls in ([9], [1] * 9, [3, 6]):
        e = Engine(g.n, g.sources, g.targets, scale=10.0)
        e.set_positions(_uniform(n, 4))
        for k in calls:
            e.step(k)
        out.append(e.get_positions())
    assert np.array_equal(out[0], out[1])
    assert np.array_equal(out[0], out[2])


@pytest.mark.parametrize("n", [2, 33, 512, 513, 4737, 20000])
def test_quadrupole_moments_at_tile_edges(n):
    """The build's prefix sums of the second moments, through the walk that
    uses them."""
    from gpugraphlayout_b200 import Engine
    from oracle import oracle as O
    g = _graph(n)
    e = Engine(g.n, g.sources, g.targets, scale=10.0, theta=1.5, multipole=2)
    for seed in (1, 2):
        xy = _uniform(n, seed)
        e.set_positions(xy)
        e.step(1)
        tot, ga = e.forces()
        ref, overflow, _ = O.Tree(xy, g.mass).repulsion(10.0, itolsq=1 / 1.5 ** 2, multipole=2)
        assert not overflow
        assert rel_rmse(tot - ga, ref) <= TOL


@pytest.mark.parametrize("n", [3, 511, 512, 513])
def test_order_after_a_displacement(n):
    """The root box that the displacement leaves, by one block (up to 512
    bodies) and by more: the next step's order is the oracle's of the
    positions then."""
    from gpugraphlayout_b200 import Engine
    from oracle import oracle as O
    g = _graph(n)
    e = Engine(g.n, g.sources, g.targets, scale=10.0)
    e.set_positions(_uniform(n, 6))
    for _ in range(3):
        e.step(1)
        xy = e.get_positions()
        e.step(1)
        assert np.array_equal(e.sort_order(), O.Tree(xy, g.mass).sort().astype(np.uint32))


@pytest.mark.parametrize("n,count", [(500, 255), (500, 256), (500, 257), (500, 480), (3000, 129),
                                     (3000, 255), (3000, 256), (3000, 257), (3000, 600),
                                     (3000, 1100)])
def test_long_runs_are_sorted_again(n, count):
    """After a tree of thin cells the sort leaves out the levels past 12.  A
    level-12 cell of up to 256 bodies is put in order by the fix-up; one of
    more sorts on every digit, which counts as one of perturb_rounds."""
    from gpugraphlayout_b200 import Engine
    g = _graph(n)
    e = Engine(g.n, g.sources, g.targets, scale=10.0)
    _check(e, _uniform(n, 1), g.mass, False)
    xy = _uniform(n, 2)
    at = np.random.default_rng(3).permutation(64 * 64)[:count]  # in (0, 0.5)^2, 2048 / 4096 wide
    xy[2:2 + count, 0] = (at % 64 + 0.5) / 128
    xy[2:2 + count, 1] = (at // 64 + 0.5) / 128
    _check(e, xy, g.mass, False)
    assert e.stats()["perturb_rounds"] == (count > 256)
    _check(e, xy, g.mass, False)  # the plan knows the cell now
    assert e.stats()["perturb_rounds"] == 0


def _cell_counts(xy, levels):
    """Bodies in the fullest cell of each level under the box [-1024, 1024]^2."""
    out = []
    for lvl in levels:
        c = np.ceil((xy.astype(np.float64) + 1024) * (2.0 ** lvl / 2048)).astype(np.int64)
        out.append(int(np.unique(c, axis=0, return_counts=True)[1].max()))
    return out


def _nested(n, level, low, seed):
    """More than 128 bodies in one level-6 cell (no bucket sort next time), 40
    of them in one cell of `level`, apart four levels down; and 60 bodies in
    one cell of the last level that a sort without its `low` lowest digits
    tells apart."""
    xy = _crowd(n, 200, seed, "spread")
    rng = np.random.default_rng(seed)
    w = 2048.0 / 2 ** level
    at = rng.permutation(49)[:40]
    xy[202:242, 0] = (at % 7 + 0.5) * (w / 7)
    xy[202:242, 1] = (at // 7 + 0.5) * (w / 7)
    if low:
        w = 2048.0 / 2 ** (32 - 4 * low)
        at = rng.permutation(64)[:60]
        xy[242:302, 0] = -(at % 8 + 0.5) * (w / 8)
        xy[242:302, 1] = -(at // 8 + 0.5) * (w / 8)
    return xy


# one block's sort in shared memory, and a team's through global memory
@pytest.mark.parametrize("n", [500, 3000])
@pytest.mark.parametrize("low", [5, 4, 3, 2, 1, 0])
def test_order_with_each_number_of_digits_left_out(n, low):
    """The sort leaves out the digits below the first of the levels 12, 16, ..,
    28 at which the last tree's cells hold at most 32 bodies: every number of
    moves, odd ones from the other buffer, and a run for the fix-up."""
    from gpugraphlayout_b200 import Engine
    g = _graph(n)
    e = Engine(g.n, g.sources, g.targets, scale=10.0)
    level = 28 - 4 * low
    xy = _nested(n, level, 0, 1)
    counts = _cell_counts(xy, [6, 12, 16, 20, 24, 28])
    assert counts[0] > 128
    assert next((5 - i for i in range(5) if counts[1 + i] <= 32), 0) == low
    _check(e, xy, g.mass, False)
    xy = _nested(n, level, low, 2)
    if low:
        assert _cell_counts(xy, [32 - 4 * low])[0] >= 60
    _check(e, xy, g.mass, False)
    assert e.stats()["perturb_rounds"] == 0


@pytest.mark.parametrize("threads", [None, 256])
@pytest.mark.parametrize("n", [1500, 2048, 2304])
def test_batch_order_when_a_block_sorts_again(n, threads):
    """A batch graph's first iteration knows no tree: 1100 bodies in one
    level-24 cell are a run too long for the fix-up of the block's own sort."""
    from gpugraphlayout_b200 import BatchEngine
    from oracle import oracle as O
    g = _graph(n)
    b = BatchEngine([(g.n, g.sources, g.targets)], scale=10.0)
    if threads:
        b.configure(0, threads, threads)
    xy = _crowd(n, 1100, 4, "tight")
    assert _cell_counts(xy, [24])[0] > 1024
    b.set_positions(xy)
    b.step(1)
    assert np.array_equal(b.sort_order(), O.Tree(xy, g.mass).sort().astype(np.uint32))


@pytest.mark.parametrize("n", [2049, 4608, 4609, 6001])
def test_batch_order_when_single_blocks_fill_the_gpu(n):
    """As many graphs as fill the GPU with one 512-thread block each: more
    nodes than a cluster's line, either side of what a block's sort stages."""
    from gpugraphlayout_b200 import BatchEngine
    from oracle import oracle as O
    g = _graph(n)
    k = 224
    b = BatchEngine([(g.n, g.sources, g.targets)] * k, scale=10.0)
    xys = [_uniform(n, s) if s % 2 else _crowd(n, n // 8, s, "spread") for s in range(k)]
    b.set_positions(np.concatenate(xys))
    b.step(1)
    order = b.sort_order()
    tot, ga = b.forces()
    for i in (0, 1, 112, 223):
        t = O.Tree(xys[i], g.mass)
        assert np.array_equal(b.part(order, i), t.sort().astype(np.uint32)), i
        ref, overflow, _ = t.repulsion(10.0)
        assert overflow or rel_rmse(b.part(tot - ga, i), ref) <= TOL, i


def test_batch_order_of_a_few_small_graphs():
    """Few enough graphs for four blocks each: the line lies at 768 nodes."""
    from gpugraphlayout_b200 import BatchEngine
    from oracle import oracle as O
    sizes = [767, 768, 769, 1024, 3072, 3073]
    graphs = [_graph(n) for n in sizes]
    b = BatchEngine([(g.n, g.sources, g.targets) for g in graphs], scale=10.0)
    for crowd in (False, True):
        xys = [_crowd(n, 300, 5, "tight") if crowd else _uniform(n, 4) for n in sizes]
        b.set_positions(np.concatenate(xys))
        b.step(1)
        order = b.sort_order()
        for i, (g, xy) in enumerate(zip(graphs, xys)):
            assert np.array_equal(b.part(order, i), O.Tree(xy, g.mass).sort().astype(np.uint32)), i
