"""The FP64 direct sum at the edges of its tiles, slices and groups.

Tolerance: every term m d / r^3 is formed with at most 8 roundings and 2 ulp of
the reciprocal power, and a sum of n terms in any order adds at most n
roundings, on either side, so |f - f_ref| <= 2 (n + 10) u sum_j |f_j| per
component, u = 2^-53."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def _terms(m, q, eps):
    d = q[None, :, :] - q[:, None, :]
    r2 = (d ** 2).sum(-1) + eps * eps
    np.fill_diagonal(r2, 1.0)
    return (m[:, None] * m[None, :] / (r2 * np.sqrt(r2)))[..., None] * d


def _direct(m, q, targets=None, eps=0.0, kind=0):
    from hierarquicos_b200.system import direct_targets

    return direct_targets(m, q[:, 0], q[:, 1], q[:, 2], targets, 1.0, eps, kind).T.cpu().numpy()


@pytest.mark.parametrize("eps", [0.0, 0.02])
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 63, 64, 65, 257, 511, 513, 2047, 2049])
def test_direct_sum_edges(n, eps):
    rng = np.random.default_rng(n)
    m, q = rng.uniform(0.5, 1.5, n) / n, rng.normal(size=(n, 3))
    t = _terms(m, q, eps)
    bound = 2 * (n + 10) * U * np.abs(t).sum(1) + 1e-300
    assert (np.abs(_direct(m, q, eps=eps) - t.sum(1)) <= bound).all()
    tg = np.arange(n)[::3]
    assert (np.abs(_direct(m, q, tg, eps, 1) * m[tg, None] - t.sum(1)[tg]) <= bound[tg]).all()


def test_direct_sum_special_values():
    """Coincident unsoftened bodies give NaN for the pair and leave the others
    finite; an index out of range gives NaN; distances whose cube overflows add
    nothing, those whose cube underflows give an infinite force."""
    rng = np.random.default_rng(5)
    m, q = np.full(100, 0.01), rng.normal(size=(100, 3))
    q[70] = q[3]
    f = _direct(m, q)
    assert np.isnan(f[[3, 70]]).all()
    rest = np.delete(np.arange(100), [3, 70])
    assert np.isfinite(f[rest]).all()
    f = _direct(m, q, np.array([5, -1, 100, 99]), 0.01)
    assert np.isfinite(f[[0, 3]]).all() and np.isnan(f[[1, 2]]).all()
    far = np.array([[0.0, 0.0, 0.0], [1e120, 0.0, 0.0]])
    assert (_direct(m[:2], far) == 0.0).all()
    near = np.array([[0.0, 0.0, 0.0], [1e-120, 0.0, 0.0]])
    f = _direct(m[:2], near)
    assert f[0, 0] == np.inf and f[1, 0] == -np.inf
