"""The build's size-dependent paths: keys, permutation, octree records and
moments against the oracle's Morton tree on both sides of every switch (sort by
counting / radix passes, one or four binary nodes a thread, staged / per-level
upward pass), at the edges of their tiles, and with shapes that stress them
(equal keys, one long chain of nested nodes, shallow trees, odd pass counts)."""
import numpy as np
import pytest

from conftest import xyz
from refcompact import compact_from_reference

pytestmark = pytest.mark.gpu


def _cloud(n, seed=0):
    rng = np.random.default_rng(seed)
    return rng.uniform(0.5, 1.5, n) / n, rng.normal(size=(n, 3))


def _check(oracle_mod, m, q, depth=21, order=4):
    from hierarquicos_b200.system import BHSystem

    s = BHSystem()
    s.build(m, *xyz(q), order=order, depth=depth)
    s.sync()
    keys, perm = s.keys()
    ref = oracle_mod.MortonTree(m, *xyz(q), L=depth, ssa=1.2, use_quadrupole=True, fma_mode=1)
    rkeys, rperm = ref.sorted()
    assert np.array_equal(keys, rkeys) and np.array_equal(perm, rperm)
    nodes = s.nodes()
    _, meta, children, nch = compact_from_reference(ref.nodes())
    assert np.array_equal(nodes["meta"], meta)
    used = np.arange(8)[None, :] < nch[:, None]
    assert np.array_equal(np.where(used, nodes["child"], 0), children)
    return s, nodes, perm


def _moments(m, q, nodes, perm):
    """Masses, centres and quadrupoles summed over each node's bodies (relative
    to the sum of the terms' absolute values: n u of rounding on either side)."""
    ms, qs = m[perm], q[perm]
    for j in range(len(nodes["meta"])):
        f, c = nodes["meta"][j][:2]
        w, r = ms[f:f + c], qs[f:f + c]
        tol = 4 * (c + 64) * 2.0 ** -53
        assert abs(nodes["com"][j][3] - w.sum()) <= tol * w.sum()
        com = (w[:, None] * r).sum(0) / w.sum()
        assert (np.abs(nodes["com"][j][:3] - com) <= tol * np.abs(w[:, None] * r).sum(0) / w.sum() + 1e-300).all()
        d = r - com
        ref = np.array([(w * d[:, a] * d[:, b]).sum() for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))])
        size = w.sum() * (np.abs(r - com).max() + np.abs(com).max() * 2.0 ** -20) ** 2
        assert (np.abs(nodes["quad"][j] - ref) <= 1e-9 * size).all()


@pytest.mark.parametrize("n", [1, 2, 3, 63, 64, 65, 255, 256, 257, 1023, 1025, 2049, 4097])
def test_small_builds(oracle_mod, n):
    m, q = _cloud(n, n)
    if n < 2:
        from hierarquicos_b200.system import BHSystem

        f = BHSystem().forces(m, *xyz(q)).cpu().numpy()
        assert (f == 0.0).all()
        return
    s, nodes, perm = _check(oracle_mod, m, q)
    _moments(m, q, nodes, perm)
    s.close()


@pytest.mark.parametrize("n", [12000, 12001, 32769, 65536, 65537, 262144, 262145])
def test_switches(oracle_mod, n):
    s, _, _ = _check(oracle_mod, *_cloud(n, 1))
    s.close()


@pytest.mark.parametrize("depth", [1, 2, 3, 5, 8, 16])
@pytest.mark.parametrize("n", [3000, 20000])
def test_depths(oracle_mod, n, depth):
    """Odd and even numbers of radix passes, and buckets of equal keys."""
    s, _, _ = _check(oracle_mod, *_cloud(n, 2), depth=depth)
    s.close()


def test_nested_chain(oracle_mod):
    """Bodies that halve their distance to a corner: every level holds a node
    that spans almost all bodies (the longest lists of the staged pass)."""
    rng = np.random.default_rng(4)
    n = 40000
    q = rng.uniform(0.5, 1.0, size=(n, 3)) * 2.0 ** -rng.integers(0, 20, size=(n, 1))
    q = np.concatenate([q, q[:300]])  # and some exact duplicates
    m = np.full(len(q), 1.0 / len(q))
    s, nodes, perm = _check(oracle_mod, m, q)
    s.close()


@pytest.mark.parametrize("order", [1, 4, 8])
def test_batch_equals_lone_systems(order):
    """Both sorts of a batch, with systems of one body and sizes off every tile:
    each system's keys and moments are its own build's, bit for bit."""
    from hierarquicos_b200.system import BHSystem, offsets_of

    for sizes in ([1, 2, 300, 1, 4097, 65], [1, 30000, 257, 2, 25000, 700], [37] * 300 + [22000]):
        m, q = _cloud(sum(sizes), 9)
        off = offsets_of(sizes)
        b = BHSystem()
        f = b.forces_batch(m, *xyz(q), off, order=order, theta=0.6, eps=0.01).cpu().numpy()
        lone = BHSystem()
        for s in range(len(sizes)) if len(sizes) < 10 else [0, 150, 300]:
            a, e = int(off[s]), int(off[s + 1])
            g = lone.forces(m[a:e], *xyz(q[a:e]), order=order, theta=0.6, eps=0.01).cpu().numpy()
            assert np.array_equal(f[3 * a:3 * e], g), (sizes[s], s)
        b.close()
        lone.close()


@pytest.mark.parametrize("sizes", [[20001, 7, 20000, 1, 33], [1, 2, 3] * 90 + [30001, 31, 17, 45],
                                   [257, 1, 2000, 63] * 300 + [5, 9001]])
def test_batch_radix_places(sizes):
    """Batches above the counting sort's limit, one and two digits of the system:
    every body has its own place, in its system's range and in that system's key
    order (a lone build's, by the counting sort where it is small).  Half of the
    bodies lie on cell edges, so that the lanes of a warp take different ways
    through the keys kernel before they count their systems."""
    from hierarquicos_b200.system import BHSystem, offsets_of

    n = sum(sizes)
    assert sum(k * k for k in sizes) > 5e8
    rng = np.random.default_rng(6)
    q = rng.uniform(-1, 1, size=(n, 3))
    edge = rng.random(n) < 0.5
    q[edge] = np.round(q[edge] * 32) / 32
    m = np.full(n, 1.0 / n)
    off = offsets_of(sizes)
    b, lone = BHSystem(), BHSystem()
    b.build_batch(m, *xyz(q), off, strict_keys=0)
    b.sync()
    keys, perm = b.keys()
    assert np.array_equal(np.sort(perm), np.arange(n))
    system_of = np.repeat(np.arange(len(sizes)), sizes)
    assert np.array_equal(system_of[perm], system_of)
    for s in range(0, len(sizes), max(1, len(sizes) // 40)):
        a, e = int(off[s]), int(off[s + 1])
        if e - a < 2:
            continue
        lone.build(m[a:e], *xyz(q[a:e]), strict_keys=0)
        lone.sync()
        k1, p1 = lone.keys()
        assert np.array_equal(keys[a:e], k1) and np.array_equal(perm[a:e] - a, p1), s
    b.close()
    lone.close()


@pytest.mark.parametrize("sizes", [[6700] * 2, [6760] * 2, [5750] * 4, [5840] * 4, [4850] * 16,
                                   [4920] * 16, [2330] * 128, [2345] * 128])
def test_batches_on_both_sides_of_the_sorts_line(sizes):
    """Just below and above the sum of n_s^2 up to which a batch is sorted by
    counting: the same places as lone builds (counting up to 12,000 bodies)."""
    from hierarquicos_b200.system import BHSystem, offsets_of

    m, q = _cloud(sum(sizes), 12)
    off = offsets_of(sizes)
    b, lone = BHSystem(), BHSystem()
    b.build_batch(m, *xyz(q), off)
    b.sync()
    keys, perm = b.keys()
    for s in sorted({0, 1, len(sizes) - 1}):
        a, e = int(off[s]), int(off[s + 1])
        lone.build(m[a:e], *xyz(q[a:e]))
        lone.sync()
        k1, p1 = lone.keys()
        assert np.array_equal(keys[a:e], k1) and np.array_equal(perm[a:e] - a, p1), s
    b.close()
    lone.close()


def _chain(n):
    """Bodies that halve their distance to a corner, and some exact duplicates."""
    rng = np.random.default_rng(4)
    q = rng.uniform(0.5, 1.0, size=(n, 3)) * 2.0 ** -rng.integers(0, 20, size=(n, 1))
    q = np.concatenate([q, q[:300]])
    return rng.uniform(0.5, 1.5, len(q)) / len(q), q


def _all_moments(m, q, nodes, perm, order):
    """Every node's mass, centre, second and third moments from its bodies, level by
    level (the nodes of a level hold disjoint ranges).  The second and third moments
    are taken about the node's own centre; a child's centre is off by a few roundings
    of |r| a level, at most 21 levels, and the translation takes its dipole for zero:
    3 * 40 u |r| / size, with |r| / size below 2^20 (below that the moments are
    measured against |r| 2^-20): 1.4e-8."""
    ms, qs = m[perm], q[perm]
    n = len(ms)
    for level in np.unique(nodes["meta"][:, 2]):
        j = np.flatnonzero(nodes["meta"][:, 2] == level)
        f, c = nodes["meta"][j, 0].astype(int), nodes["meta"][j, 1].astype(int)
        ends = np.stack([f, f + c], 1).ravel()

        def total(v):
            return np.add.reduceat(np.append(v, 0.0), np.minimum(ends, n))[::2]

        body = np.repeat(np.arange(len(j)), c)
        at = np.concatenate([np.arange(a, b) for a, b in zip(f, f + c)])
        tol = 4 * (c + 64) * 2.0 ** -53
        mass = total(ms)
        assert (np.abs(nodes["com"][j, 3] - mass) <= tol * mass).all(), level
        com = nodes["com"][j, :3]
        for k in range(3):
            ref, size = total(ms * qs[:, k]) / mass, total(np.abs(ms * qs[:, k])) / mass
            assert (np.abs(com[:, k] - ref) <= tol * size + 1e-300).all(), level
        if order < 4:
            continue
        d = np.zeros((n, 3))
        d[at] = qs[at] - com[body]
        r = np.zeros(len(j))
        np.maximum.at(r, body, np.abs(d[at]).max(1))
        size = r + np.abs(com).max(1) * 2.0 ** -20
        for k, (a, b) in enumerate(((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))):
            got = nodes["quad"][j, k]
            assert (np.abs(got - total(ms * d[:, a] * d[:, b])) <= 2e-8 * mass * size ** 2).all(), (level, k)
        if order < 8:
            continue
        third = ((0, 0, 0), (0, 1, 1), (0, 2, 2), (0, 0, 1), (1, 1, 1), (1, 2, 2), (0, 0, 2), (1, 1, 2),
                 (2, 2, 2), (0, 1, 2))
        for k, (a, b, e) in enumerate(third):
            got = nodes["oct"][j, k]
            assert (np.abs(got - total(ms * d[:, a] * d[:, b] * d[:, e])) <= 2e-8 * mass * size ** 3).all(), (level, k)


@pytest.mark.parametrize("order", [1, 4, 8])
@pytest.mark.parametrize("n", [257, 32768, 32769, 65536, 65537, -40000, -65236, -70000])
def test_moments_of_every_stage(n, order):
    """One chunk and one list, both list stages, and level by level; n < 0: the
    nested chain, whose nodes span chunks on every level (65,536 bodies the most
    that go in stages)."""
    from hierarquicos_b200.system import BHSystem

    m, q = _cloud(n, 3) if n > 0 else _chain(-n)
    s = BHSystem()
    s.build(m, *xyz(q), order=order)
    s.sync()
    _all_moments(m, q, s.nodes(), s.keys()[1], order)
    s.close()


@pytest.mark.parametrize("order", [4, 8])
def test_staged_and_levelled_moments_are_the_same(order):
    """Systems of a batch of more than 65,536 bodies go level by level, alone in
    stages: the same centres, moments and forces, bit for bit."""
    from hierarquicos_b200.system import BHSystem, offsets_of

    parts = [_cloud(40000, 1), _chain(20000), _cloud(300, 2), _cloud(33000, 3)]
    m, q = np.concatenate([p[0] for p in parts]), np.concatenate([p[1] for p in parts])
    off = offsets_of([len(p[0]) for p in parts])
    b, lone = BHSystem(), BHSystem()
    f = b.forces_batch(m, *xyz(q), off, order=order, theta=0.6, eps=0.01).cpu().numpy()
    all_nodes = b.nodes()
    for s in range(len(parts)):
        a, e = int(off[s]), int(off[s + 1])
        g = lone.forces(m[a:e], *xyz(q[a:e]), order=order, theta=0.6, eps=0.01).cpu().numpy()
        nodes = lone.nodes()
        first = all_nodes["meta"][:, 0]
        j = np.flatnonzero((first >= a) & (first < e))
        for name in ("com", "quad", "oct")[:2 if order < 8 else 3]:
            assert np.array_equal(all_nodes[name][j], nodes[name]), (s, name)
        assert np.array_equal(f[3 * a:3 * e], g), s
    b.close()
    lone.close()
