"""Sizes at which a count, a table or a rule of the frame changes."""
import numpy as np
import pytest

from tests.conftest import cuda_available
from vk_tessellated_clusters_gb300 import layouts as L
from vk_tessellated_clusters_gb300 import scene as S

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]

FLAGS = L.FLAG_CULLING | L.FLAG_WRITE_FULLCLUSTERS


def _first_level(mesh, instances, capacity, every_pass):
    """(split items of the first level, split items and parts written or refused) of a frame whose instances lie on
    one another, split once (or in all passes)."""
    from vk_tessellated_clusters_gb300.pipeline import TessellationPipeline
    sc = S.Scene("stacked", [mesh], [S.Instance(0, np.eye(4), 0, 0.01, 0.0) for _ in range(instances)],
                 [S.Texture(np.zeros((4, 4), np.float32), L.TEXEL_F32)])
    caps = dict(L.default_caps(visible_bits=20, part_bits=18, vertex_bits=18, megs=64, split_factor=11),
                maxSplitTriangles=capacity)
    pipe = TessellationPipeline(sc, caps, FLAGS)
    pipe.set_cameras(S.Camera(eye=(0.0, 0.8, -2.2), center=(0.0, 0.0, 0.0), tess_rate_pixels=0.04))
    pipe.stage("frame_begin")
    pipe.stage("instances_classify")
    pipe.stage("clusters_cull", 0, instances)
    pipe.stage("build_setup", L.BUILD_SETUP_CLASSIFY)
    pipe.stage("cluster_classify", 0, instances)
    pipe.stage("build_setup", L.BUILD_SETUP_SPLIT)
    items = int(pipe.state.scene_building()["splitWriteCounter"])
    if every_pass:
        pipe.stage("triangle_split_all")
    else:
        pipe.stage("triangle_split", 0, instances)
    b = pipe.state.scene_building()
    assert pipe.device_errors() == 0
    pipe.close()
    return items, int(b["splitWriteCounter"]), int(b["partTriangleCounter"])


def test_level_of_more_than_2_to_the_32_children():
    """112 instances of a mesh of 524,288 triangles, each split in 75 on average: 4.4e9 children in one level. Each
    instance's are those of one instance alone, so the counters are 112 times that frame's."""
    n = 112
    mesh = S.clusterize(S.grid(512, 512, 4.0, 4.0), 0)
    items, splits, parts = _first_level(mesh, 1, 1 << 20, False)
    assert items == 524288 and splits > items and parts > 0
    assert n * (splits - items + parts) > 1 << 32 > n * splits
    got = _first_level(mesh, n, 59000000, False)
    assert got == (n * items, n * splits, n * parts)
    # every pass in one launch: the later levels only add split items
    got = _first_level(mesh, n, 59000000, True)
    assert got[0] == n * items and got[1] >= n * splits


def _many(instances, apart, seed=3):
    """Small meshes in many places; each instance with a key of its own (apart) or one of six."""
    rng = np.random.default_rng(seed)
    meshes = [S.clusterize(S.icosphere(3), 0), S.clusterize(S.torus(1.0, 0.3, 64, 16), 1)]
    insts = []
    for i in range(instances):
        world = S.translate_rotate_scale(rng.random(3) * 40.0, S.random_unit_quaternion(rng), 0.5 + rng.random())
        offset = 0.0001 * (i + 1) if apart else 0.01 * (i % 3)
        insts.append(S.Instance(i % 2, world, i % 2, 0.03, offset))
    textures = [S.Texture(rng.random((37, 53), np.float32), L.TEXEL_F32) for _ in range(2)]
    return S.Scene("many", meshes, insts, textures)


# the instances one round of the grouping block takes (1,024, also the most whose first clusters classify keeps in
# shared memory), one more, the most that are grouped, one more
@pytest.mark.parametrize("instances", [1024, 1025, 4096, 4097])
@pytest.mark.parametrize("apart", [False, True])
def test_groups_of_many_instances(oracle, instances, apart):
    """Integers bit-exact against the oracle and positions to the vertex tolerance, from the graph, the direct launches
    and the graph with its host traffic; the same bytes from all."""
    import torch
    from tests.parity import assert_same, vertex_tolerance
    from vk_tessellated_clusters_gb300.pipeline import TessellationPipeline
    sc = _many(instances, apart)
    assert sc.total_clusters >= 16384
    caps = L.default_caps(part_bits=19, vertex_bits=23)
    fc = S.frame_constants(S.camera_orbit(5, tess_rate_pixels=6.0))
    ref_state, _ = oracle.frame(sc, fc, caps, FLAGS)
    want = ref_state.outputs(oracle.entries)
    assert len(want["partTriangles"]) > 0 and len(want["fullClusters"]) > 16384 // 2
    pipe = TessellationPipeline(sc, caps, FLAGS)
    pipe.set_cameras(fc)
    block = np.concatenate([np.frombuffer(fc.tobytes(), np.uint8), np.frombuffer(fc.tobytes(), np.uint8),
                            pipe.state.res.instance_records.view(np.uint8).reshape(-1)])
    host = torch.empty(block.size, dtype=torch.uint8, pin_memory=True)
    host.numpy()[:] = block
    readback = torch.zeros(L.Readback.itemsize, dtype=torch.uint8, pin_memory=True)
    device = torch.zeros(block.size, dtype=torch.uint8, device="cuda")
    first = None
    for mode in ("graph", "batched", "host"):
        pipe.state.gen_vertices.handle.zero_()
        if mode == "host":
            a = pipe.args
            a.view, a.viewLast = device.data_ptr(), device.data_ptr() + fc.nbytes
            a.instances = device.data_ptr() + 2 * fc.nbytes
            pipe.build_host(host.data_ptr(), device.data_ptr(), block.size, readback.data_ptr())
        else:
            pipe.build(mode)
        got = pipe.outputs()
        assert_same(got, want, mode, vertex_tol=vertex_tolerance(sc))
        first = first or got
        assert got["genVertices"].tobytes() == first["genVertices"].tobytes()
    assert readback.numpy().tobytes() == got["readback"].tobytes()
    assert pipe.device_errors() == 0
    pipe.close()


# the most instances whose full clusters the adjoint takes by groups, and one more
@pytest.mark.parametrize("instances", [1024, 1025])
@pytest.mark.parametrize("apart", [False, True])
def test_adjoint_of_many_instances(oracle, instances, apart):
    """Each gradient against the FP64 adjoint: relative error of its norm within 1e-4, as for fewer instances."""
    import ctypes
    import torch
    from oracle.binding import lib as olib
    from vk_tessellated_clusters_gb300.autograd import FrozenFrame
    from vk_tessellated_clusters_gb300.pipeline import TessellationPipeline
    sc = _many(instances, apart)
    assert sc.total_clusters >= 12288
    caps = L.default_caps(part_bits=18, vertex_bits=23)
    cam = S.camera_orbit(5, tess_rate_pixels=6.0)
    pipe = TessellationPipeline(sc, caps, FLAGS)
    pipe.set_cameras(cam)
    pipe.build("graph")
    frozen = FrozenFrame(pipe)
    g = np.random.default_rng(1).normal(0, 1, (frozen.num_vertices, 3)).astype(np.float32)
    dP, dN, dT = frozen.scatter_gradients(torch.from_numpy(g).cuda())
    ref_state, _ = oracle.frame(sc, cam, caps, FLAGS)
    want = [[np.zeros(tuple(x.shape)) for x in xs] for xs in (dP, dN, dT)]
    mesh = [i.geometry for i in sc.instances]
    ptr = lambda a: (ctypes.c_void_p * len(a))(*[x.ctypes.data for x in a])
    g64 = g.astype(np.float64)
    olib().tco_backward_f64(ctypes.byref(oracle.table), ctypes.byref(ref_state.args), g64.ctypes.data,
                            ptr([want[0][m] for m in mesh]), ptr([want[1][m] for m in mesh]), ptr(want[2]))
    for got, ref in zip([*dP, *dN, *dT], [*want[0], *want[1], *want[2]]):
        part, norm = got.double().cpu().numpy(), np.linalg.norm(ref)
        assert norm > 0 and np.linalg.norm(part - ref) <= 1e-4 * norm, np.linalg.norm(part - ref) / norm
    assert pipe.device_errors() == 0
    pipe.close()


@pytest.mark.parametrize("call", ["raster", "frame", "frame_pn", "plain", "frozen"])
def test_map_of_more_than_2_to_the_32_texels(call):
    """A map of 65,536 x 65,600 texels, ones in its last 64 rows and zeros elsewhere, read in the middle of those rows:
    the same bits as from a small map of ones."""
    import torch
    from vk_tessellated_clusters_gb300.autograd import FrozenFrame
    from vk_tessellated_clusters_gb300.pipeline import TessellationPipeline
    wide, high = 65536, 65600
    sc = S.scene_icosphere(subdivisions=3, map_size=64)
    sc.textures[0] = S.Texture(np.full((4, 4), 65535, np.uint16), L.TEXEL_UNORM16)
    rng = np.random.default_rng(2)
    for g in sc.geometries:
        g.texcoords[:, 0] = rng.random(len(g.texcoords))
        g.texcoords[:, 1] = (high - 32) / high
    caps = L.default_caps(visible_bits=12, part_bits=17, split_bits=14, vertex_bits=20, megs=64)
    pipe = TessellationPipeline(sc, caps, FLAGS | (L.FLAG_PN if call == "frame_pn" else 0))
    # whole clusters and parts
    pipe.set_cameras(S.Camera(eye=(0.0, 0.0, 3.6), center=(0.0, 0.0, 0.0), tess_rate_pixels=40.0))
    texels = torch.zeros(wide * high * 2, dtype=torch.uint8, device="cuda")
    texels[-64 * wide * 2:] = 255
    record = np.zeros(1, L.DisplacementTexture)
    got = []
    for large in (False, True):
        if large:
            record[0] = (texels.data_ptr(), wide, high, L.TEXEL_UNORM16, 0)
            pipe.state.res.textures.write(record)
        pipe.state.gen_vertices.handle.zero_()
        pipe.build("plain" if call == "plain" else "graph")
        out = pipe.outputs()
        assert len(out["fullClusters"]) > 0 and len(out["partTriangles"]) > 0
        if call == "raster":
            got.append(pipe.raster_batches()["worldPositions"])
        elif call == "frozen":
            frozen = FrozenFrame(pipe)
            pipe.state.gen_vertices.handle.zero_()
            got.append(frozen.generate().cpu().numpy())
        else:
            got.append(out["genVertices"])
    assert np.abs(got[0]).max() > 1.04  # displaced
    assert got[0].tobytes() == got[1].tobytes()
    assert pipe.device_errors() == 0
    pipe.close()


def test_adjoint_adds_a_part_once(oracle):
    """224,000 parts of 54 vertices on 320 triangles: the positions' gradients are sums of thousands of parts' terms, and
    their error is that of adding each part once. Adding n terms of random sign in float32 makes an error of
    c sqrt(n / 2) of the sum, c <= 2^-24 / sqrt(3); each part in as many pieces as the walk cuts it into (2.7 here) makes
    1.6 times as much."""
    import ctypes
    import torch
    from oracle.binding import lib as olib
    from vk_tessellated_clusters_gb300.autograd import FrozenFrame
    from vk_tessellated_clusters_gb300.pipeline import TessellationPipeline
    sc = S.scene_icosphere(subdivisions=2, map_size=64)
    sc.instances[0].displacement_index = -1
    caps = L.default_caps(visible_bits=12, part_bits=18, split_bits=16, vertex_bits=24, megs=1024)
    cam = S.Camera(eye=(0.0, 0.0, 1.5), center=(0.0, 0.0, 0.0), tess_rate_pixels=1.0, near=0.01, far=10.0)
    pipe = TessellationPipeline(sc, caps, FLAGS)
    pipe.set_cameras(cam)
    pipe.build("graph")
    frozen = FrozenFrame(pipe)
    out = pipe.outputs()
    g = np.random.default_rng(1).normal(0, 1, (frozen.num_vertices, 3)).astype(np.float32)
    got = frozen.scatter_gradients(torch.from_numpy(g).cuda())[0][0].double().cpu().numpy()
    ref_state, _ = oracle.frame(sc, cam, caps, FLAGS)
    want = [np.zeros(x.shape) for x in (sc.geometries[0].positions, sc.geometries[0].normals)]
    texels = np.zeros(sc.textures[0].texels.shape)
    g64 = g.astype(np.float64)
    ptr = lambda a: (ctypes.c_void_p * 1)(a.ctypes.data)
    olib().tco_backward_f64(ctypes.byref(oracle.table), ctypes.byref(ref_state.args), g64.ctypes.data, ptr(want[0]),
                            ptr(want[1]), ptr(texels))
    # parts on each base vertex
    parts, geo = out["partTriangles"], sc.geometries[0]
    assert len(parts) > 200000
    cluster = geo.clusters[parts["clusterID"]]
    first = cluster["firstLocalTriangle"].astype(np.int64) + 3 * (parts["triangleID_config"] & 0xFFFF).astype(np.int64)
    n = np.zeros(len(geo.positions))
    for k in range(3):
        np.add.at(n, cluster["firstLocalVertex"].astype(np.int64) + geo.local_triangles.reshape(-1)[first + k], 1)
    bound = 2.0 ** -24 / 3 ** 0.5 * np.sqrt((n * n / 2).sum() / n.sum())
    error = np.linalg.norm(got - want[0]) / np.linalg.norm(want[0])
    assert error <= bound, (error, bound)
    assert pipe.device_errors() == 0
    pipe.close()
