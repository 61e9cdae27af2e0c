"""The traversal at the sizes where its groups, lists and stacks have edges.

The repulsion (fa2_repulsion_noalloc, which gives it alone) against the
oracle's walk of the reference rule on the same positions.  The terms are the
same set (the accept test is bit-exact); only their order of summation
differs.  With T terms a body's float32 sum is off by at most T 2^-24 of the
sum of the terms' magnitudes: under 1e-4 for T <= 1500, the suite's bar
(relative RMSE).  The engine's cell centres are exact sums rounded once and the
oracle's are float sums, so they differ by an ulp of the coordinate; the
positions keep that far below the distances (the dense cluster sits at the
origin, where an ulp is small), and no two coincide.
"""
import ctypes as C

import numpy as np
import pytest

from conftest import rel_rmse

pytestmark = pytest.mark.gpu

TOL = 1e-4


def _positions(kind, n, seed):
    rng = np.random.default_rng(seed)
    xy = rng.uniform(-1000, 1000, (n, 2))
    if kind == "clustered":  # deep chains of one-child cells, groups far apart inside
        half = rng.random(n) < 0.5
        xy[half] = rng.normal(0, 0.02, (int(half.sum()), 2))
    return xy.astype(np.float32)


def _check(kind, n, theta, seed=3):
    import torch
    from gpugraphlayout_b200 import _native
    from oracle import oracle as O
    xy = _positions(kind, n, seed)
    mass = np.full(n, 2.0 if n < 3 else 3.0, np.float32)
    prm = _native.Params()
    _native.lib().fa2_default_params(C.byref(prm))
    prm.scale, prm.theta = 10.0, theta
    d_xy, d_mass = torch.from_numpy(xy).cuda(), torch.from_numpy(mass).cuda()
    out = torch.full((n, 2), float("nan"), device="cuda")
    assert _native.lib().fa2_repulsion_noalloc(
        C.c_void_p(d_xy.data_ptr()), C.c_void_p(d_mass.data_ptr()), n, C.byref(prm), None,
        C.c_void_p(out.data_ptr())) == 0
    itolsq = float(np.float32(1.0) / (np.float32(theta) * np.float32(theta)))
    ref, overflow, _ = O.Tree(xy, mass).repulsion(10.0, itolsq=itolsq)
    assert not overflow
    assert rel_rmse(out.cpu().numpy(), np.asarray(ref).reshape(-1, 2)) <= TOL


@pytest.mark.parametrize("n", [2, 3, 5, 31, 32, 33, 63, 64, 65, 97, 1000, 1500])
def test_group_edges(n):
    _check("uniform", n, 1.0)


@pytest.mark.parametrize("kind", ["uniform", "clustered"])
@pytest.mark.parametrize("theta", [0.2, 0.6, 1.0, 2.0])
def test_opening_angles(kind, theta):
    """From nearly every cell opened (full lists and stacks) to few."""
    _check(kind, 1201, theta)


@pytest.mark.parametrize("n", [75776, 75777])
def test_either_side_of_loading_ahead(n):
    """Up to half of the resident warps (148 x 16 groups) a walk loads ahead."""
    from gpugraphlayout_b200 import Engine
    from oracle import oracle as O
    s = np.arange(n, dtype=np.uint32)
    g = O.Graph(s, np.roll(s, -1))
    xy = _positions("uniform", n, 5)
    e = Engine(g.n, g.sources, g.targets, scale=10.0)
    e.set_positions(xy)
    e.step(1)
    tot, ga = e.forces()
    ref, overflow, _ = O.Tree(xy, g.mass).repulsion(10.0)
    assert not overflow
    assert rel_rmse(tot - ga, np.asarray(ref).reshape(-1, 2)) <= TOL


def _noalloc(xy, mass, theta, eps):
    import torch
    from gpugraphlayout_b200 import _native
    prm = _native.Params()
    _native.lib().fa2_default_params(C.byref(prm))
    prm.scale, prm.theta, prm.epssq = 1.0, theta, eps
    d_xy, d_m = torch.tensor(xy, device="cuda"), torch.tensor(mass, device="cuda")
    out = torch.empty_like(d_xy)
    torch.cuda.synchronize()
    _native.check(_native.lib().fa2_repulsion_noalloc(
        C.c_void_p(d_xy.data_ptr()), C.c_void_p(d_m.data_ptr()), len(xy), C.byref(prm), None,
        C.c_void_p(out.data_ptr())), "fa2_repulsion_noalloc")
    return out.cpu().numpy()


@pytest.mark.parametrize("n", [2, 40, 3000])
def test_a_softening_below_the_normal_numbers(n):
    """epssq under 2^-126 walks without flushing: a body and itself, and two
    bodies 1e-20 apart, have a subnormal d^2 + eps.  (mass / epssq has to be
    finite, so epssq is just below 2^-126.)  The pair's force is d / (d^2 + eps),
    the others' terms vanish beside it."""
    xy = _positions("even", n, n)
    xy[0] = (0.0, 0.0)
    xy[1] = (1e-20, 0.0)
    mass = np.ones(n, np.float32)
    eps = np.float32(1e-38)
    f = _noalloc(xy, mass, 1.0, eps)
    assert np.isfinite(f).all()
    d = np.float64(xy[1, 0])
    pull = d / (d * d + np.float64(eps))
    assert np.abs(f[:2] - [[-pull, 0.0], [pull, 0.0]]).max() <= 1e-5 * pull


@pytest.mark.parametrize("n", [2, 33, 5000])
def test_a_tiny_softening_in_every_walk(n):
    """The same on the engine's walks (a group's loads ahead of its test or
    not), with the quadrupole term, and in the batch; the scale keeps the
    repulsion, read as total less attraction and gravity, the larger part."""
    from gpugraphlayout_b200 import BatchEngine, Engine
    from oracle import oracle as O
    ids = np.arange(n, dtype=np.uint32)
    g = O.Graph(ids, np.roll(ids, -1)) if n > 2 else O.Graph(ids[:1], ids[1:])
    xy = _positions("even", n, n)
    eps = float(np.float32(1e-38))
    for multipole in (1, 2, 0):
        if multipole:
            e = Engine(n, g.sources, g.targets, scale=1e4, epssq=eps, theta=1.2,
                       multipole=multipole)
        else:
            e = BatchEngine([(n, g.sources, g.targets)], scale=1e4, epssq=eps, theta=1.2)
        e.set_positions(xy)
        e.step(1)
        tot, ga = e.forces()
        ref, overflow, _ = O.Tree(xy, g.mass).repulsion(
            1e4, itolsq=1 / 1.2 ** 2, epssq=np.float32(eps), multipole=max(1, multipole))
        assert not overflow
        assert rel_rmse(tot - ga, ref) <= TOL
