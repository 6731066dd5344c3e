"""The cluster test by bounds (bounds_factor_one, tc_classify.cu) restated in
float32: wherever it accepts a cluster, every edge factor is 1."""
import numpy as np
import pytest

f32 = np.float32


def _dot(a, b):
    return (a[..., 0] * b[..., 0] + a[..., 1] * b[..., 1]) + a[..., 2] * b[..., 2]


def _len(a):
    return np.sqrt(_dot(a, a))


def _bounds(p):
    """k_cluster_bounds for vertices p (N, V, 3), every pair of them an edge."""
    mid = f32(0.5) * (p.min(1) + p.max(1))
    d = p - mid[:, None]
    r = np.sqrt(_dot(d, d).max(1)) * f32(1 + 1e-5)
    e = p[:, :, None] - p[:, None, :]
    edge = np.sqrt(_dot(e, e).max((1, 2))) * f32(1 + 1e-5)
    return mid, r, edge, (_len(mid) + r) * f32(1 + 1e-5)


def _world(m, p):
    """xform_point, columns m[c] of the affine matrix."""
    return ((m[:, 0, None] * p[..., 0:1] + m[:, 1, None] * p[..., 1:2]) + m[:, 2, None] * p[..., 2:3]) + m[:, 3, None]


@pytest.mark.parametrize("seed", range(4))
@pytest.mark.parametrize("spread", [1.0, 1e-3])
def test_accepted_clusters_have_factors_of_one(seed, spread):
    """Rotations with even, uneven and sheared scales, translations and view points up to 1e4 times the cluster's size,
    clusters far from their object's origin, distances packed around the bound."""
    rng = np.random.default_rng(seed)
    n, accepted, tight = 20000, 0, 0
    for near, rate in ((0.01, 0.25), (0.5, 1.0), (0.01, 0.0)):
        p = (rng.normal(size=(n, 5, 3)) * spread + rng.normal(size=(n, 1, 3)) * rng.choice([0, 1, 100], (n, 1, 1))).astype(f32)
        q, _ = np.linalg.qr(rng.normal(size=(n, 3, 3)))
        scale = np.exp(rng.normal(size=(n, 3)) * rng.choice([0, 0.7], (n, 1)))
        a = q * scale[:, None, :] + rng.normal(size=(n, 3, 3)) * rng.choice([0, 0, 0.5], (n, 1, 1))
        t = rng.normal(size=(n, 3)) * rng.choice([1, 30, 1000], (n, 1))
        m = np.concatenate([np.swapaxes(a, 1, 2), t[:, None]], 1).astype(f32)  # (n, column, row)
        mid, r, edge, size = _bounds(p)
        k = f32(f32(1080.0) * f32(rate))
        # the view at about the distance where the bound just holds
        s = np.linalg.norm(a, 2, axis=(1, 2))
        dist = s * r + s * edge * float(k) / 1.5 * rng.uniform(0.98, 1.3, n) + 1e-6
        dirs = rng.normal(size=(n, 3))
        centre = _world(m, mid[:, None])[:, 0]
        view = (centre + dirs / np.linalg.norm(dirs, axis=1, keepdims=True) * dist[:, None]).astype(f32)
        # the test
        g = [_dot(m[:, i], m[:, j]) for i, j in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))]
        g01, g02, g12 = np.abs(g[3]), np.abs(g[4]), np.abs(g[5])
        s2 = np.maximum((g[0] + g01) + g02, np.maximum((g[1] + g01) + g12, (g[2] + g02) + g12))
        sv = np.sqrt(s2) * f32(1 + 1e-5)
        err = f32(2e-6) * (sv * size + _len(m[:, 3]))
        d = _len(centre - view) - sv * r - err
        claim = (sv * edge + err) * k < f32(1.4999) * np.maximum(f32(near), d * f32(1 - 1e-5))
        # every edge's factor, as tess_factors evaluates it
        w = _world(m[:, None].repeat(5, 1).reshape(-1, 4, 3), p.reshape(-1, 1, 3)).reshape(n, 5, 3)
        far = _len(w - view[:, None])
        spl = f32(1) / np.maximum(f32(near), np.minimum(far[:, :, None], far[:, None, :]))
        x = ((_len(w[:, :, None] - w[:, None, :]) * spl) * f32(1080.0)) * f32(rate)
        f = np.clip(np.rint(x), 1, 32768).max((1, 2))
        assert not np.any(claim & (f != 1))
        accepted += int(claim.sum())
        tight += int((claim & (x.max((1, 2)) > 1.2)).sum())
    assert accepted > n and tight > 100  # it answers, also close to the threshold
