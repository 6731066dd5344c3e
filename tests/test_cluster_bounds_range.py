"""The cluster test by bounds (k_cluster_bounds, bounds_factor_one, tc_classify.cu) where squares leave the range of a
float: restated in float32, and on the GPU against the oracle."""
import dataclasses

import numpy as np
import pytest

from tests.conftest import cuda_available

f32 = np.float32
TINY = f32(1.17549435e-38)  # kBoundsTiny


def _dot(a, b):
    return (a[..., 0] * b[..., 0] + a[..., 1] * b[..., 1]) + a[..., 2] * b[..., 2]


def _len(a):
    return np.sqrt(_dot(a, a))


def _false_claims(mesh, scale, tiny, n=4000):
    """Clusters of meshes about `mesh` in size under matrices about `scale`, near the view: how many are accepted that
    have an edge of another factor than 1, and how many are accepted."""
    rng = np.random.default_rng(9)
    p = (rng.normal(size=(n, 5, 3)) * mesh).astype(f32)
    q, _ = np.linalg.qr(rng.normal(size=(n, 3, 3)))
    m = (q * scale * np.exp(rng.normal(size=(n, 1, 3)))).astype(f32)  # rows: the matrix' columns
    # (world coordinates about the view, edges from far below to far above the bound)
    k, near = f32(1080.0), f32(1e-3 * mesh * scale)
    view = (rng.normal(size=(n, 3)) * mesh * scale * 10.0 ** rng.uniform(0, 5, (n, 1))).astype(f32)
    mid = f32(0.5) * (p.min(1) + p.max(1))
    d = p - mid[:, None]
    r = np.sqrt(_dot(d, d).max(1) + tiny) * f32(1 + 1e-5)
    e = p[:, :, None] - p[:, None, :]
    edge = np.sqrt(_dot(e, e).max((1, 2)) + tiny) * f32(1 + 1e-5)
    size = (_len(mid) + r) * f32(1 + 1e-5)
    g = [_dot(m[:, i], m[:, j]) for i, j in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))]
    g01, g02, g12 = np.abs(g[3]), np.abs(g[4]), np.abs(g[5])
    s2 = np.maximum((g[0] + g01) + g02, np.maximum((g[1] + g01) + g12, (g[2] + g02) + g12))
    s = np.sqrt(s2 + tiny) * f32(1 + 1e-5)
    world = lambda x: (m[:, 0, None] * x[..., 0:1] + m[:, 1, None] * x[..., 1:2]) + m[:, 2, None] * x[..., 2:3]  # noqa: E731
    err = f32(2e-6) * (s * size)
    dist = _len(world(mid[:, None])[:, 0] - view) - s * r - err
    claim = (s * edge + err) * k < f32(1.4999) * np.maximum(near, dist * f32(1 - 1e-5))
    w = world(p)
    far = _len(w - view[:, None])
    per = f32(1) / np.maximum(near, np.minimum(far[:, :, None], far[:, None, :]))
    x = (_len(w[:, :, None] - w[:, None, :]) * per) * k
    f = np.clip(np.rint(x), 1, 32768).max((1, 2))
    return int((claim & (f != 1)).sum()), int(claim.sum())


@pytest.mark.parametrize("mesh,scale", [(1.0, 1.0), (1e-18, 1e18), (1e-23, 1e18), (1e-24, 1e24), (1e-30, 1e30),
                                        (1e18, 1e-18), (1e19, 1e-19), (1e18, 1e-23)])
def test_squares_out_of_range(mesh, scale):
    with np.errstate(over="ignore", under="ignore", invalid="ignore"):
        false, accepted = _false_claims(mesh, scale, TINY)
        assert false == 0
        if mesh == 1.0:
            assert accepted > 100  # it answers
        if mesh == 1e-23 or scale == 1e-23:
            assert _false_claims(mesh, scale, f32(0))[0] > 0  # without kBoundsTiny it answers wrongly


@pytest.mark.gpu
@pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")
@pytest.mark.parametrize("mesh,scale", [(1.0, 1.0), (1e-23, 1e18), (1e18, 1e-23)])
def test_meshes_and_matrices_of_extreme_scales(oracle, mesh, scale):
    """96 instances in four groups, their meshes and matrices scaled, the places and the view with both: integers
    bit-exact and positions to the vertex tolerance."""
    from tests.parity import assert_same, vertex_tolerance
    from vk_tessellated_clusters_gb300 import layouts as L
    from vk_tessellated_clusters_gb300 import scene as S
    from vk_tessellated_clusters_gb300.pipeline import TessellationPipeline
    sc = S.scene_batched(num_instances=96, map_size=64)
    tolerance = vertex_tolerance(sc) * mesh  # (its squares, too, would leave the range of the meshes' floats)
    for g in sc.geometries:
        for a in (g.positions, g.lo, g.hi):
            a *= a.dtype.type(mesh)
        for f in g.bboxes.dtype.names[:2]:
            g.bboxes[f] = g.bboxes[f] * f32(mesh)
    for inst in sc.instances:
        inst.displacement_index = -1
        inst.world = np.array(inst.world, np.float64)
        inst.world[:3, :3] *= scale
        inst.world[:3, 3] *= mesh * scale
    assert sc.total_clusters >= 16384
    flags = L.FLAG_CULLING | L.FLAG_WRITE_FULLCLUSTERS
    caps = L.default_caps(vertex_bits=22)
    cam, at = S.camera_orbit(5), mesh * scale
    cam = dataclasses.replace(cam, eye=tuple(at * np.array(cam.eye)), center=tuple(at * np.array(cam.center)),
                              near=at * cam.near, far=at * cam.far)
    ref_state, _ = oracle.frame(sc, cam, caps, flags)
    want = ref_state.outputs(oracle.entries)
    assert len(want["partTriangles"]) > 1000
    pipe = TessellationPipeline(sc, caps, flags)
    pipe.set_cameras(cam)
    pipe.build("graph")
    assert_same(pipe.outputs(), want, "graph", vertex_tol=tolerance)
    pipe.close()
