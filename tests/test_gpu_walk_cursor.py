"""Walks that do not directly follow the build they use: after a replay of a
recorded graph, in a capture of the walk alone, after a capture of the build
alone, and a repeated walk when a replay ran out of stack.  Each must walk every
group, whatever moved the group cursor before it: the bits of a plain call."""
import numpy as np
import pytest
import torch

from conftest import xyz

pytestmark = pytest.mark.gpu


def _cloud(n, seed=0):
    rng = np.random.default_rng(seed)
    m = torch.from_numpy(rng.uniform(0.5, 1.5, n) / n).cuda()
    q = torch.from_numpy(rng.normal(size=(3, n))).cuda()
    return m, q[0].contiguous(), q[1].contiguous(), q[2].contiguous()


def _plain(args, p):
    from hierarquicos_b200.system import BHSystem

    s = BHSystem()
    f = s.forces(*args, p).clone()
    s.close()
    return f


def _params(**kw):
    from hierarquicos_b200._lib import default_params

    return default_params(**dict(dict(eps=0.01, order=4), **kw))


@pytest.fixture
def system():
    from hierarquicos_b200.system import BHSystem

    s = BHSystem()
    yield s
    torch.cuda.synchronize()
    s.close()


# teams / three consumers / seven consumers, and the one-warp walk
SHAPES = [(70000, 0, 1), (30000, 0, 1), (5000, 0, 1), (5000, 0, 0), (5000, 1, 1)]


@pytest.mark.parametrize("n,precision,pipeline", SHAPES)
def test_walk_after_a_replay(system, n, precision, pipeline):
    args = _cloud(n)
    kw = dict(precision=precision, pipeline=pipeline)
    pa, pb = _params(theta=0.5, **kw), _params(theta=0.8, **kw)
    ga = torch.empty(3 * n, dtype=torch.float64, device="cuda")
    system.build(*args, pa)
    system.capture(pa, ga)
    system.build(*args, pa)  # the same layout keeps the graph
    system.replay()
    out = torch.full_like(ga, float("nan"))
    system.walk(pb, out)
    system.sync()
    assert torch.equal(ga, _plain(args, pa))
    assert torch.equal(out, _plain(args, pb))


@pytest.mark.parametrize("n,precision,pipeline", SHAPES)
def test_capture_of_the_walk_alone(system, n, precision, pipeline):
    args = _cloud(n, 1)
    p = _params(theta=0.6, precision=precision, pipeline=pipeline)
    ref = _plain(args, p)
    out = torch.empty_like(ref)
    system.build(*args, p)
    system.sync()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        system.walk(p, out)
    for _ in range(2):
        out.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, ref)


def test_walk_after_a_capture_of_the_build_alone(system):
    args = _cloud(5000, 2)
    p = _params(theta=0.6)
    ref = _plain(args, p)
    system.build(*args, p)
    out = torch.empty_like(ref)
    system.walk(p, out)
    system.sync()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        system.build(*args, p)  # recorded, not run: the tree is still the first build's
    out.zero_()
    system.walk(p, out)
    system.sync()
    assert torch.equal(out, ref)


def wide_deep_bodies():
    """Bodies of which the last 32 nodes of every level from the second to the
    twentieth have eight children each: a walk that opens everything (theta 0)
    pushes 256 entries for the 32 it takes, and holds 4,320 at the end -- more
    than the 4,096 that a stack starts with.  The corners make the root cube the
    unit cube."""
    rng = np.random.default_rng(3)
    cells, q = np.zeros((1, 3)), [np.zeros((1, 3)), np.ones((1, 3))]
    octants = np.array([[d >> 2, (d >> 1) & 1, d & 1] for d in range(8)])
    for level in range(1, 22):
        kids = (2 * cells[:, None] + octants).reshape(-1, 3)  # in key order
        cells = kids[-32:] if level < 21 else kids[:0]
        rest = kids[:len(kids) - len(cells)]
        # two bodies in opposite eighths of the cell (the same cell at level 21)
        for e in (0.25, 0.75):
            q.append((rest + e + rng.uniform(-0.1, 0.1, rest.shape)) / 2.0 ** level)
    q = np.concatenate(q)
    return np.full(len(q), 1.0 / len(q)), q


def test_replay_that_runs_out_of_stack(system):
    m, q = wide_deep_bodies()
    args = [torch.from_numpy(a).cuda() for a in (m, *xyz(q))]
    p = _params(theta=0.0, eps=0.01, leaf_cap=1, amp=1.0 + 2.0 ** -23, strict_keys=0)
    out = torch.full((3 * len(m),), float("nan"), dtype=torch.float64, device="cuda")
    ref = _plain(args, p)
    system.build(*args, p)
    system.capture(p, out)
    system.build(*args, p)
    system.replay()
    system.sync()  # repeats the walk with a larger stack
    assert torch.equal(out, ref)


def test_replay_repeats_its_own_walk(system):
    """The walk that is repeated because a replay ran out of stack is the graph's:
    its parameters, output, inputs and all groups, whatever was built and walked
    between the capture and the replay."""
    m, q = wide_deep_bodies()
    args = [torch.from_numpy(a).cuda() for a in (m, *xyz(q))]
    kw = dict(leaf_cap=1, amp=1.0 + 2.0 ** -23, strict_keys=0)
    p, other = _params(theta=0.0, **kw), _params(theta=0.9, order=1, **kw)
    ref = _plain(args, p)
    out = torch.full_like(ref, float("nan"))
    mine = torch.full_like(ref, 7.0)
    system.build(*args, p)
    system.walk(p, torch.empty_like(ref), groups=(0, 1))
    system.capture(p, out)
    system.build(args[0] * 2.0, *args[1:], other)
    system.walk(other, mine, groups=(0, 1))
    system.sync()
    kept = mine.clone()
    system.replay()
    system.sync()
    assert torch.equal(out, ref)
    assert torch.equal(mine, kept)
