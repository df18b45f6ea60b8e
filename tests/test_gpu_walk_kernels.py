"""The walk kernels that a call's size chooses between give the bits of the
one-warp walk (pipeline 0): the same batches, in the same order, with the same
arithmetic.  Sizes lie on both sides of every switch, plus the smallest trees,
groups of one target per lane, and shapes that fill the walk's queues: bodies
with equal keys (ranges above 16 bodies), large leaves, a wide shallow tree and
a deep one whose stack leaves its shared-memory window."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _forces(m, q, **kw):
    from hierarquicos_b200.system import BHSystem

    s = BHSystem()
    f = s.forces(m, q[:, 0], q[:, 1], q[:, 2], **kw).cpu().numpy()
    s.close()
    return f


def _same(m, q, **kw):
    a, b = _forces(m, q, pipeline=0, **kw), _forces(m, q, pipeline=1, **kw)
    assert np.isfinite(a).all()
    assert np.array_equal(a.view(np.uint64), b.view(np.uint64))


def _cloud(n, seed, cusp=False):
    rng = np.random.default_rng(seed)
    q = rng.normal(size=(n, 3))
    if cusp:
        q *= rng.uniform(size=(n, 1)) ** 4
    return rng.uniform(0.5, 1.5, n) / n, q


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("order", [1, 4, 8])
@pytest.mark.parametrize("n", [1, 2, 33, 65, 1500])
def test_small_trees(n, order, precision):
    _same(*_cloud(n, n), order=order, precision=precision, theta=0.5, eps=0.01)


@pytest.mark.parametrize("n,order,precision", [
    (20480, 4, 0), (20481, 4, 0), (65536, 1, 0), (65537, 1, 0), (49152, 8, 0), (49153, 8, 0),
    (24576, 4, 1), (24577, 1, 1), (196608, 1, 1), (196609, 8, 1), (262144, 4, 1), (262145, 4, 1)])
def test_both_sides_of_a_switch(n, order, precision):
    _same(*_cloud(n, 3), order=order, precision=precision, theta=0.8, eps=0.0)


@pytest.mark.parametrize("n", [3000, 30000, 70000])
@pytest.mark.parametrize("kw", [dict(group_size=32), dict(leaf_cap=64), dict(theta=0.15),
                                dict(mac=0), dict(depth=4), dict(out_kind=1)])
def test_shapes(n, kw):
    kw = dict(dict(order=4, theta=0.6, eps=0.01), **kw)
    if n > 30000 and kw["theta"] < 0.5:
        n = 66000
    _same(*_cloud(n, 7, cusp=True), **kw)


@pytest.mark.parametrize("precision", [0, 1])
def test_equal_keys(precision):
    """Buckets of 1..200 coincident bodies: leaf ranges of every length."""
    rng = np.random.default_rng(11)
    sizes = rng.integers(1, 200, 60)
    q = np.repeat(rng.normal(size=(60, 3)), sizes, axis=0)
    m = np.full(len(q), 1.0 / len(q))
    _same(m, q, order=4, precision=precision, theta=0.5, eps=0.05)


def test_softening_beyond_any_distance():
    """FP64: eps^2 past the reciprocal series' range gives zero forces."""
    m, q = _cloud(500, 1)
    assert (_forces(m, q, order=4, precision=1, eps=1e160) == 0.0).all()


# batches of equal systems on both sides of the choice's lines: (systems, bodies)
BATCHES = [(150, 10), (700, 30), (2, 100), (120, 100), (300, 64), (37, 500), (40, 500), (80, 500),
           (20, 1000), (60, 1000), (4, 4000), (9, 4000), (20, 4000), (1, 2047), (1, 2048)]


def _batch_walks(systems, n, **kw):
    """The walk of one built batch, one warp a group and by choice."""
    from hierarquicos_b200._lib import default_params
    from hierarquicos_b200.system import BHSystem, offsets_of

    m, q = _cloud(systems * n, 5)
    s = BHSystem()
    params = [default_params(**dict(kw, pipeline=p)) for p in (0, 1)]
    s.build_batch(m, q[:, 0], q[:, 1], q[:, 2], offsets_of([n] * systems), params[0])
    s.sync()
    return s, params, [torch.empty(3 * systems * n, dtype=torch.float64, device="cuda") for _ in params]


@pytest.mark.parametrize("order,precision,group_size", [
    (1, 0, 64), (4, 0, 64), (8, 0, 64), (8, 0, 32), (4, 1, 64), (8, 1, 64)])
def test_batches_on_both_sides_of_a_line(order, precision, group_size):
    for systems, n in BATCHES:
        s, params, outs = _batch_walks(systems, n, order=order, precision=precision, theta=0.6,
                                       eps=0.01, group_size=group_size)
        for p, out in zip(params, outs):
            s.walk(p, out)
            s.sync()
        assert torch.equal(*outs), (systems, n)
        s.close()


@pytest.mark.parametrize("systems,n,order,precision", [
    (6000, 10, 4, 0), (1600, 30, 8, 0), (1000, 200, 4, 1), (1900, 100, 8, 1)])
def test_many_small_systems_do_not_wait_for_producers(systems, n, order, precision):
    """The walk that is chosen for many groups of short walks takes no more than
    half as long again as one warp a group (blocks of one producer took 1.7 to 2.1
    times as long; the chosen walk at most 1.2)."""
    s, params, outs = _batch_walks(systems, n, order=order, precision=precision, theta=0.5,
                                   eps=0.01, group_size=64)
    best = [np.inf, np.inf]
    for _ in range(7):
        for k in (0, 1):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            s.walk(params[k], outs[k])
            a.record()
            for _ in range(10):
                s.walk(params[k], outs[k])
            b.record()
            torch.cuda.synchronize()
            best[k] = min(best[k], a.elapsed_time(b) / 10)
    s.close()
    assert best[1] <= 1.5 * best[0], best


@pytest.mark.parametrize("n,order,precision,group_size", [
    (153600, 1, 1, 64), (153601, 1, 1, 64), (320000, 4, 1, 64), (320001, 4, 1, 64),
    (185600, 8, 1, 64), (185601, 8, 1, 64), (12800, 8, 0, 32), (12801, 8, 0, 32),
    (44800, 8, 0, 32), (44801, 8, 0, 32), (10240, 4, 0, 32), (10241, 4, 0, 32)])
def test_both_sides_of_a_line_in_groups(n, order, precision, group_size):
    _same(*_cloud(n, 3), order=order, precision=precision, group_size=group_size, theta=0.9, eps=0.0)


@pytest.mark.parametrize("groups", [1, 319, 320, 321, 1024, 1025])
def test_ranges_of_groups(groups):
    """A range of a large system's groups goes to the kernel of that many groups."""
    from hierarquicos_b200._lib import default_params
    from hierarquicos_b200.system import BHSystem

    m, q = _cloud(150000, 8)
    s = BHSystem()
    params = [default_params(order=4, theta=0.7, eps=0.01, pipeline=p) for p in (0, 1)]
    s.build(m, q[:, 0], q[:, 1], q[:, 2], params[0])
    s.sync()
    outs = [torch.zeros(3 * len(m), dtype=torch.float64, device="cuda") for _ in params]
    for p, out in zip(params, outs):
        s.walk(p, out, groups=(700, 700 + groups))
        s.sync()
    s.close()
    assert torch.equal(*outs) and 0 < int((outs[0] != 0).sum()) <= 3 * 64 * groups
