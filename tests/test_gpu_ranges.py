"""Kernels whose mapping depends on sizes or alignment, at the edges of each
form, against the CPU oracle."""
import ctypes

import numpy as np
import pytest

from tests.conftest import cuda_available
from tests.parity import assert_same, vertex_tolerance
from vk_tessellated_clusters_gb300 import layouts as L
from vk_tessellated_clusters_gb300 import scene as S

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]

FLAGS = L.FLAG_CULLING | L.FLAG_WRITE_FULLCLUSTERS


# part counts at which k_raster_write's warps (4 per block, 8 blocks per SM, 152 SMs: 4,864; with PN or the ripple
# half of that) share a group four ways, two ways and not at all
@pytest.mark.parametrize("instances,pixels,flags,parts", [(24, 4.0, 0, (1, 38912)), (170, 4.0, 0, (38913, 77824)),
                                                          (256, 3.0, 0, (77825, 1 << 20)),
                                                          (170, 4.0, L.FLAG_PN, (38913, 1 << 20))])
def test_raster_group_sharing(oracle, instances, pixels, flags, parts):
    """Whole outputs against the oracle (positions to the vertex tolerance times the largest instance scale), then
    the same call on outputs one float off 16-byte alignment and too small by a few vertices and triangles: the same
    values up to the capacity, nothing past it, and the capacity bit."""
    import torch
    from vk_tessellated_clusters_gb300.pipeline import TessellationPipeline
    sc = S.scene_batched(num_instances=instances, map_size=64)
    cam = S.camera_orbit(5, tess_rate_pixels=pixels)
    caps = L.default_caps(vertex_bits=23)
    ref_state, _ = oracle.frame(sc, cam, caps, FLAGS | flags)
    want = oracle.raster_batches(ref_state)
    pipe = TessellationPipeline(sc, caps, FLAGS | flags)
    pipe.set_cameras(cam)
    pipe.build("graph")
    got = pipe.raster_batches()
    n = int(pipe.state.scene_building()["partTriangleCounter"])
    assert parts[0] <= n <= parts[1], n
    assert pipe.device_errors() == 0 and got["counts"] == want["counts"]
    for f in ("batches", "indices", "primitiveIDs"):
        assert got[f].tobytes() == want[f].tobytes(), f
    scale = max(float(np.abs(np.asarray(i.world)[:3, :3]).sum(axis=1).max()) for i in sc.instances)
    assert np.abs(got["worldPositions"].astype(np.float64) - want["worldPositions"]).max() <= vertex_tolerance(sc) * scale
    nv, nt = got["counts"][1] - 5, got["counts"][2] - 7
    ro, bufs = pipe.state.raster_outputs()
    small = type(ro).from_buffer_copy(ro)
    clip = torch.full((4 * nv + 64,), -7.0, device="cuda")
    small.clipPositions, small.maxVertices, small.maxTriangles = clip.data_ptr() + 4, nv, nt
    for b in ("worldPositions", "indices", "primitiveIDs"):
        bufs[b].handle.fill_(0xAB)
    pipe.stage("raster_batches", ctypes.byref(small))
    assert pipe.device_errors() == 8  # TC_DEVERR_CAPACITY
    c = clip.cpu().numpy()
    assert c[1:1 + 4 * nv].tobytes() == got["clipPositions"][:nv].tobytes()
    assert c[0] == -7.0 and (c[1 + 4 * nv:] == -7.0).all()
    cut = {"worldPositions": (np.float32, 3 * nv), "indices": (np.uint8, 3 * nt), "primitiveIDs": (np.uint32, nt)}
    for f, (dtype, count) in cut.items():
        raw = bufs[f].read(np.uint8, min(bufs[f].nbytes, count * dtype().itemsize + 64))
        size = count * dtype().itemsize
        assert raw[:size].tobytes() == got[f].reshape(-1)[:count].tobytes() and (raw[size:] == 0xAB).all(), f
    pipe.close()


# 80 to 20,480 parts on grids of 608 and 152 blocks: chunks of 1, 2, 4, 8, 16 and 32 parts, some cut by the end
@pytest.mark.parametrize("subdivisions,pixels", [(1, 6.0), (2, 5.0), (3, 8.0), (4, 5.0), (5, 8.0)])
@pytest.mark.parametrize("grid", [0, 1])
def test_vertex_chunk_widths(oracle, subdivisions, pixels, grid):
    """Frame graph and stage entry points against the oracle, integers bit-exact and positions to the vertex
    tolerance, whatever number of parts a warp takes at a time."""
    from vk_tessellated_clusters_gb300.pipeline import TessellationPipeline
    sc = S.scene_icosphere(subdivisions=subdivisions, map_size=64)
    cam = S.Camera(eye=(0.3, 0.2, 2.5), center=(0.0, 0.0, 0.0), tess_rate_pixels=pixels)
    caps = L.default_caps(visible_bits=12, part_bits=17, split_bits=14, vertex_bits=21, megs=256)
    ref_state, _ = oracle.frame(sc, cam, caps, FLAGS)
    want = ref_state.outputs(oracle.entries)
    pipe = TessellationPipeline(sc, caps, FLAGS, schedule={"vertexGridPerSM": grid})
    pipe.set_cameras(cam)
    pipe.build("graph")
    assert_same(pipe.outputs(), want, "graph", vertex_tol=vertex_tolerance(sc))
    pipe.state.gen_vertices.handle.zero_()
    pipe.build("plain")  # k_instantiate_parts, one launch per instance and run
    assert_same(pipe.outputs(), want, "stages", vertex_tol=vertex_tolerance(sc))
    assert pipe.device_errors() == 0
    pipe.close()


# every map kind the vertex walk is specialised for, and chunks that mix them
@pytest.mark.parametrize("dtype,fmt", [(np.float32, L.TEXEL_F32), (np.float16, L.TEXEL_F16), (np.uint16, L.TEXEL_UNORM16)])
@pytest.mark.parametrize("size", [(37, 53), (64, 32), (1, 1), "mixed"])
@pytest.mark.parametrize("deform", [0, L.FLAG_PN | L.FLAG_RIPPLE])
def test_map_kinds(oracle, dtype, fmt, size, deform):
    """Frame graph, stage entry points and raster batches against the oracle, integers bit-exact and positions to the
    vertex tolerance (times the largest instance scale); the frozen frame's forward gives the same bits."""
    from vk_tessellated_clusters_gb300.autograd import FrozenFrame
    from vk_tessellated_clusters_gb300.pipeline import TessellationPipeline
    sc = S.scene_batched(num_instances=12, map_size=64)
    rng = np.random.default_rng(3)
    for i in range(len(sc.textures)):
        if size != "mixed" or i % 2:
            shape = (37, 53) if size == "mixed" else size
            texels = rng.random(shape) * (65535 if dtype == np.uint16 else 1)
            sc.textures[i] = S.Texture(texels.astype(dtype), fmt)
    cam = S.camera_orbit(40, tess_rate_pixels=6.0)
    cam = _ripple(cam) if deform else cam
    caps = L.default_caps(vertex_bits=21)
    ref_state, _ = oracle.frame(sc, cam, caps, FLAGS | deform)
    want = ref_state.outputs(oracle.entries)
    pipe = TessellationPipeline(sc, caps, FLAGS | deform)
    pipe.set_cameras(cam)
    for mode in ("graph", "plain"):
        pipe.state.gen_vertices.handle.zero_()
        pipe.build(mode)
        assert_same(pipe.outputs(), want, mode, vertex_tol=vertex_tolerance(sc))
    built = pipe.outputs()["genVertices"]
    assert deform or FrozenFrame(pipe).generate().cpu().numpy().tobytes() == built.tobytes()
    got, ref = pipe.raster_batches(), oracle.raster_batches(ref_state)
    assert got["counts"] == ref["counts"] and got["indices"].tobytes() == ref["indices"].tobytes()
    scale = max(float(np.abs(np.asarray(i.world)[:3, :3]).sum(axis=1).max()) for i in sc.instances)
    assert np.abs(got["worldPositions"].astype(np.float64) - ref["worldPositions"]).max() <= vertex_tolerance(sc) * scale
    assert pipe.device_errors() == 0
    pipe.close()


def _ripple(cam):
    fc = S.frame_constants(cam)
    fc["animationRippleAmplitude"], fc["animationRippleFrequency"] = 0.02, 8.0
    fc["animationRippleSpeed"], fc["animationState"] = 1.5, 0.7
    return fc


# with PN or the ripple: 320 to 20,480 parts (chunks of 1 to 16 parts); 2X batches below and above one per warp
@pytest.mark.parametrize("case", ["ico2_pn", "ico4_pn_ripple", "ico5_ripple", "transient_24", "transient_256"])
def test_deform_chunk_widths(oracle, case):
    """Integers bit-exact against the oracle, positions to the vertex tolerance; an empty displacement map still
    displaces by the offsets (ico5_ripple)."""
    from vk_tessellated_clusters_gb300.pipeline import TessellationPipeline
    flags = FLAGS
    if case.startswith("ico"):
        sc = S.scene_icosphere(subdivisions=int(case[3]), map_size=64)
        cam = S.Camera(eye=(0.3, 0.2, 2.5), center=(0.0, 0.0, 0.0), tess_rate_pixels=6.0)
        flags |= (L.FLAG_PN if "pn" in case else 0) | (L.FLAG_RIPPLE if "ripple" in case else 0)
        if case == "ico5_ripple":
            sc.textures[0] = S.Texture(np.zeros((0, 0), np.float32), L.TEXEL_F32)
            sc.instances[0].displacement_offset = 0.125
    else:
        sc, cam = S.scene_batched(num_instances=int(case[10:]), map_size=64), S.camera_orbit(0)
        flags |= L.FLAG_TRANSIENT_1X | L.FLAG_TRANSIENT_2X | L.FLAG_PN | L.FLAG_RIPPLE
    fc = _ripple(cam)
    caps = L.default_caps(vertex_bits=22)
    ref_state, _ = oracle.frame(sc, fc, caps, flags)
    want = ref_state.outputs(oracle.entries)
    if case == "transient_256":
        assert len(want["transBuilds"]) > 152 * 7 * 4  # more builds than the kernel's warps: two per warp
    pipe = TessellationPipeline(sc, caps, flags)
    pipe.set_cameras(fc)
    pipe.build("graph")
    assert_same(pipe.outputs(), want, case, vertex_tol=vertex_tolerance(sc))
    assert pipe.device_errors() == 0
    pipe.close()


# split items of the first level, their children and the queue's capacity: indexed by every block for itself (320), by
# all (1,280 with 128 and 256 threads, 5,120), one chunk of children to a tile or, where a small queue's rows hold fewer
# tiles, up to 8 (320 and 512 places; what does not fit is dropped like the oracle's)
@pytest.mark.parametrize("subdivisions,eye,pixels,capacity,several", [(2, 1.08, 2.0, 320, True), (2, 1.08, 2.0, 512, True),
                                                                      (2, 1.08, 2.0, 17468, False),
                                                                      (3, 1.08, 1.5, 66984, False),
                                                                      (4, 1.3, 1.5, 32496, False)])
@pytest.mark.parametrize("block", [128, 256, 512])
def test_split_tiles(oracle, subdivisions, eye, pixels, capacity, several, block):
    """All passes in one launch, one per launch, and one per launch and instance window, against the oracle."""
    from vk_tessellated_clusters_gb300.pipeline import TessellationPipeline
    sc = S.scene_icosphere(subdivisions=subdivisions, map_size=64)
    cam = S.Camera(eye=(0.0, 0.0, eye), center=(0.0, 0.0, 0.0), tess_rate_pixels=pixels, near=0.01, far=10.0)
    caps = dict(L.default_caps(visible_bits=12, part_bits=18, vertex_bits=23, megs=256), maxSplitTriangles=capacity)
    ref_state, _ = oracle.frame(sc, cam, caps, FLAGS)
    want = ref_state.outputs(oracle.entries)
    items = want["splitTriangles"][:min(capacity, int(want["readback"]["numSplitTriangles"]))]
    first = np.isin(items["vtxEncoded"], (0, 1 << 15, 1 << 31)).all(axis=1)  # whole base triangles
    children = int(oracle.entries["numTriangles"][(items["triangleID_config"][first] >> 16) & 0x7FFF].sum())
    chunks = -(-children // block)
    assert (chunks > -(-capacity // 16)) == several
    pipe = TessellationPipeline(sc, caps, FLAGS, schedule={"splitBlockSize": block})
    pipe.set_cameras(cam)
    for mode, per_pass in (("graph", 0), ("graph", 1), ("plain", 0)):
        pipe.set_schedule({**pipe.schedule(), "splitPerPass": per_pass})
        pipe.state.gen_vertices.handle.zero_()
        pipe.build(mode)
        assert_same(pipe.outputs(), want, f"{mode} {per_pass}", vertex_tol=vertex_tolerance(sc))
    assert pipe.device_errors() == 0
    pipe.close()


# up to 8,192 hits without the staging, then partial and whole blocks of 256
@pytest.mark.parametrize("count", [1, 31, 256, 257, 1023, 8192, 8193, 8447, 8448, 8449])
@pytest.mark.parametrize("offset", [0, 4, 8])
def test_decode_counts_and_alignment(oracle, count, offset):
    """Partial blocks of hits at 4-, 8- and 16-byte aligned addresses: field-exact against the oracle, and nothing
    written past the results."""
    import torch
    from vk_tessellated_clusters_gb300.hits import sample_hits
    from vk_tessellated_clusters_gb300.pipeline import TessellationPipeline
    sc = S.scene_batched(num_instances=8, map_size=64)
    caps = L.default_caps(visible_bits=16, part_bits=18, split_bits=14, vertex_bits=21, megs=256)
    flags = FLAGS | L.FLAG_TRANSIENT_1X | L.FLAG_TRANSIENT_2X
    cam = S.frame_constants(S.camera_orbit(0))
    ref_state, _ = oracle.frame(sc, cam, caps, flags)
    pipe = TessellationPipeline(sc, caps, flags)
    pipe.set_cameras(cam)
    pipe.build("batched")
    hits = sample_hits(pipe.outputs(), sc, pipe.entries, count, seed=3, bad=0)
    want = oracle.decode_hits(ref_state, hits)
    src = torch.zeros(hits.nbytes + 16, dtype=torch.uint8, device="cuda")[offset:offset + hits.nbytes]
    src.copy_(torch.from_numpy(hits.view(np.uint8).reshape(-1).copy()))
    whole = torch.full((want.nbytes + 64,), 0xCD, dtype=torch.uint8, device="cuda")
    pipe.decode_hits_device(src, whole[offset:])
    got = whole.cpu().numpy()
    assert got[offset:offset + want.nbytes].tobytes() == want.tobytes()
    assert (got[:offset] == 0xCD).all() and (got[offset + want.nbytes:] == 0xCD).all()
    pipe.close()


# Frames of 16,384 clusters and more group their instances: groups of 24 and 25 (subgroups of 8 with and without a
# rest), a pair (grouped, but with too many distinct clusters for bounds), instances that share a mesh but not map,
# scale or offset, no sharing at all; capacities that refuse the last clusters, and an instance short of the limit
@pytest.mark.parametrize("case", ["groups24", "groups25", "pair", "mixed", "distinct", "vertices", "visible", "below",
                                  "mixed_transient"])
def test_instance_groups(oracle, case):
    """Integers bit-exact against the oracle and positions to the vertex tolerance, from the graph twice and from the
    direct launches; the per-instance launches, which use no groups, give the same bytes."""
    from vk_tessellated_clusters_gb300.pipeline import TessellationPipeline
    if case == "pair":
        mesh = S.clusterize(S.grid(512, 512, 4.0, 4.0), 0)
        sc = S.scene_batched(num_instances=2, map_size=64)
        sc.geometries = [mesh]
        for inst in sc.instances:
            inst.geometry, inst.displacement_index = 0, 1
    else:
        sc = S.scene_batched(num_instances={"groups25": 100, "below": 80}.get(case, 96), map_size=64)
    assert (sc.total_clusters >= 16384) == (case != "below")
    for i, inst in enumerate(sc.instances):
        if case.startswith("mixed"):
            # none, map 0, map 1; under the ripple maps only (it has no value at an undisplaced origin)
            inst.displacement_index = (i // 4) % 3 - (0 if case == "mixed_transient" else 1)
            inst.displacement_scale = 0.01 * (1 + i // 12 % 2)
            inst.displacement_offset = 0.005 * (i // 24)
        if case == "distinct":
            inst.displacement_scale = 0.001 * (i + 1)
    flags = FLAGS
    caps = L.default_caps(vertex_bits=22)
    if case == "mixed_transient":
        flags |= L.FLAG_TRANSIENT_1X | L.FLAG_TRANSIENT_2X | L.FLAG_RIPPLE
    if case == "vertices":
        caps = dict(caps, maxGeneratedVertices=700000)
    if case == "visible":
        caps = dict(caps, maxVisibleClusters=10000)
    fc = _ripple(S.camera_orbit(5))
    ref_state, _ = oracle.frame(sc, fc, caps, flags)
    want = ref_state.outputs(oracle.entries)
    if case == "vertices":
        assert int(want["readback"]["numGenVertices"]) > 700000
    pipe = TessellationPipeline(sc, caps, flags)
    pipe.set_cameras(fc)
    first = None
    for mode in ("graph", "graph", "batched", "plain"):
        pipe.state.gen_vertices.handle.zero_()
        pipe.build(mode)
        got = pipe.outputs()
        assert_same(got, want, f"{case} {mode}", vertex_tol=vertex_tolerance(sc))
        first = first or got
        assert got["genVertices"].tobytes() == first["genVertices"].tobytes()
    assert pipe.device_errors() == 0
    pipe.close()


# one instance; several below the instance groups' clusters; groups of 18 with some instances apart by offset or by
# their gradients' place; gradients 0 and 1 floats off 8-byte alignment, maps of odd width
@pytest.mark.parametrize("case", ["single", "few", "groups", "targets", "shared_map"])
@pytest.mark.parametrize("shift", [0, 1])
def test_backward_groups(oracle, case, shift):
    """Each gradient (positions and normals per mesh, texels per map) against the FP64 adjoint, twice with another
    frame in between: relative error of its norm within 1e-4, as for the frame the backward is specified on."""
    import torch
    from oracle.binding import lib as olib
    from vk_tessellated_clusters_gb300.autograd import FrozenFrame
    from vk_tessellated_clusters_gb300.pipeline import TessellationPipeline
    rng = np.random.default_rng(7)
    if case == "single":
        sc = S.scene_icosphere(subdivisions=4, map_size=64)
        cams = [S.Camera(eye=(0.0, 0.0, d), center=(0.0, 0.0, 0.0), tess_rate_pixels=8.0) for d in (8.0, 7.8)]
    else:
        sc = S.scene_batched(num_instances=8 if case == "few" else 72, map_size=64)
        cams = [S.camera_orbit(0), S.camera_orbit(40, tess_rate_pixels=6.0)]
        for i in (9, 30, 31):
            sc.instances[i % len(sc.instances)].displacement_offset = 0.01
        if case == "shared_map":  # one map for two meshes
            for i in sc.instances:
                i.displacement_index = min(i.displacement_index, 1)
    sc.textures[:] = [S.Texture(rng.random((37, 53), np.float32), L.TEXEL_F32) for _ in sc.textures]
    caps = L.default_caps(vertex_bits=22)
    pipe = TessellationPipeline(sc, caps, FLAGS)
    for cam in cams:
        pipe.set_cameras(cam)
        pipe.build("graph")
        frozen = FrozenFrame(pipe)
        ref_state, _ = oracle.frame(sc, cam, caps, FLAGS)
        full = pipe.outputs()["tempInstantiations"]["clusterIdOffset"] >> 30 == L.RT_CLUSTER_MODE_FULL_CLUSTER
        assert full.any() and (not full.all() or cam is cams[0])
        g = rng.normal(0, 1, (frozen.num_vertices, 3)).astype(np.float32)
        buf = torch.zeros(2 * frozen._grad_floats + 1, device="cuda")
        flat = buf[shift:shift + frozen._grad_floats]
        table = frozen._pointer_table(flat)
        own = [4, 13] if case == "targets" else []  # instances with gradients of their own, past the others
        apart = buf[frozen._grad_floats + shift:]
        for i in own:
            table[2 * i] = apart.data_ptr()
        frozen.launch_backward(torch.from_numpy(g).cuda(), table)
        dP = [np.zeros(m.positions.shape) for m in sc.geometries]
        dN = [np.zeros(m.normals.shape) for m in sc.geometries]
        dT = [np.zeros(t.texels.shape) for t in sc.textures]
        mesh = [i.geometry for i in sc.instances]
        assert not own or len({mesh[i] for i in own}) == 2
        ptr = lambda a: (ctypes.c_void_p * len(a))(*[x.ctypes.data for x in a])
        big = np.zeros((max(len(p) for p in dP), 3))
        g64 = g.astype(np.float64)
        olib().tco_backward_f64(ctypes.byref(oracle.table), ctypes.byref(ref_state.args), g64.ctypes.data,
                                ptr([big if i in own else dP[m] for i, m in enumerate(mesh)]),
                                ptr([dN[m] for m in mesh]), ptr(dT))
        got = flat.double().cpu().numpy()
        at = 0
        for name, want in [("positions", w) for w in dP] + [("normals", w) for w in dN] + [("texels", w) for w in dT]:
            part = got[at:at + want.size].reshape(want.shape)
            at += want.size
            norm = np.linalg.norm(want)
            assert np.linalg.norm(part - want) <= 1e-4 * norm, (name, np.linalg.norm(part - want) / norm)
        if own:
            part = apart[:big.size].double().cpu().numpy().reshape(big.shape)
            assert np.linalg.norm(part - big) <= 1e-4 * np.linalg.norm(big)
    assert pipe.device_errors() == 0
    pipe.close()
