"""The work that a program gives this framework, as cases to be timed.

A case is one frame of the tessellation chain (through the recorded graph, the
direct launches, the graph with its host traffic, or stage by stage), or one of
the calls on a built frame: a training step through autograd, the decode of ray
hits, and the raster batches. Scenes are the procedural ones of the test suite
and the benchmark; a seed gives the transforms, the camera, the displacement
maps and the upstream gradients or hits.
"""
import ctypes
import functools
import math

import numpy as np
import torch

from vk_tessellated_clusters_gb300 import layouts as L
from vk_tessellated_clusters_gb300 import scene as S
from vk_tessellated_clusters_gb300.autograd import FrozenFrame, tessellate
from vk_tessellated_clusters_gb300.pipeline import TessellationPipeline
from vk_tessellated_clusters_gb300.table import load_raw_table

FORMATS = {"fp32": L.TEXEL_F32, "fp16": L.TEXEL_F16, "unorm16": L.TEXEL_UNORM16}
TRANSIENT = L.FLAG_TRANSIENT_1X | L.FLAG_TRANSIENT_2X
OPTIONS = {"plain": 0, "pn": L.FLAG_PN, "ripple": L.FLAG_RIPPLE, "pn_ripple": L.FLAG_PN | L.FLAG_RIPPLE,
           "transient": TRANSIENT, "all": TRANSIENT | L.FLAG_PN | L.FLAG_RIPPLE}


def listed():
    return [
        # a single small object: the launches and their latency are the cost
        dict(name="icosphere_small", call="frame", mode="graph", scene="icosphere", size=3, map=256, format="fp32",
             pixels=8.0, distance=3.0, options="plain"),
        # one object of 20,480 triangles through build()'s default mode, each kernel launched by the host
        dict(name="icosphere_direct", call="frame", mode="batched", scene="icosphere", size=5, map=1024, format="fp32",
             pixels=8.0, distance=3.0, options="plain"),
        # an object that fills the screen: long edges that the split passes subdivide, on PN patches, odd map
        dict(name="close_up_pn", call="frame", mode="graph", scene="icosphere", size=4, map=517, format="unorm16",
             pixels=3.0, distance=1.15, options="pn"),
        # the ordinary frame: 256 instances of four meshes, culled, 1080p
        dict(name="batched_256", call="frame", mode="graph", scene="batched", size=256, map=512, format="fp32",
             pixels=4.0, distance=30.0, options="plain"),
        # the same scene with the renderer's ray-tracing defaults: transient builds, PN patches, ripple animation
        dict(name="batched_256_all", call="frame", mode="graph", scene="batched", size=256, map=512, format="fp32",
             pixels=4.0, distance=30.0, options="all"),
        # 1,024 moving instances: transforms and cameras uploaded, the statistics read back, every frame
        dict(name="animated_host_1024", call="frame", mode="host", scene="batched", size=1024, map=512, format="fp32",
             pixels=4.0, distance=30.0, options="plain"),
        # the large frame: 2 M base triangles, 4K, split passes, 26 M tessellated triangles
        dict(name="terrain_1024", call="frame", mode="graph", scene="terrain", size=1024, map=4096, format="fp16",
             pixels=4.0, distance=2.0, options="plain"),
        # a renderer that drives the stages itself, one call for each; map sizes that are no powers of two
        dict(name="terrain_stages_504", call="frame", mode="stages", scene="terrain", size=504, map=1500,
             format="unorm16", pixels=4.0, distance=2.0, options="plain"),
        # training steps with the frame's decisions held: one object, and the batched scene
        dict(name="train_icosphere", call="train", mode="graph", scene="icosphere", size=5, map=1024, format="fp32",
             pixels=8.0, distance=3.0, options="plain"),
        dict(name="train_batched_256", call="train", mode="graph", scene="batched", size=256, map=512, format="fp32",
             pixels=4.0, distance=30.0, options="plain"),
        # closest hits of one 1080p image of primary rays
        dict(name="decode_1080p", call="decode", mode="graph", scene="batched", size=256, map=512, format="fp32",
             pixels=4.0, distance=30.0, options="transient", hits=1920 * 1080, coherent=True),
        # the rasteriser's batches for a finely tessellated frame
        dict(name="raster_batched_256", call="raster", mode="graph", scene="batched", size=256, map=512, format="fp32",
             pixels=3.0, distance=30.0, options="plain"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    call = rng.choice(["frame", "frame", "frame", "frame", "train", "decode", "raster"])
    scene = rng.choice(["icosphere", "batched", "terrain"] if call in ("frame", "raster") else ["icosphere", "batched"])
    case = dict(call=call, scene=scene, mode="graph", options="plain", format="fp32")
    if scene == "icosphere":
        case.update(size=rng.randint(2, 5), map=round(_log(rng, 60, 1100)), distance=round(_log(rng, 1.15, 4.0), 3))
        case["pixels"] = round(_log(rng, 3.0, 12.0), 2)
    elif scene == "batched":
        case.update(size=round(_log(rng, 3, 1000)), map=round(_log(rng, 60, 600)), distance=round(rng.uniform(24, 40), 2))
        case["pixels"] = round(_log(rng, 3.0, 10.0), 2)
    else:
        case.update(size=8 * round(_log(rng, 8, 120)), map=round(_log(rng, 250, 4000)),
                    distance=round(rng.uniform(2.0, 6.0), 2), pixels=round(_log(rng, 4.5, 12.0), 2))
    if call != "train":  # only fp32 maps take gradients
        case["format"] = rng.choice(list(FORMATS))
    if call == "frame":
        case["mode"] = rng.choice(["graph", "graph", "batched", "host", "stages"])
        if case["mode"] != "stages" and scene != "terrain":
            case["options"] = rng.choice(list(OPTIONS))
    if call == "decode":
        case["options"] = rng.choice(["plain", "transient"])
        case.update(hits=round(_log(rng, 1000, 2 << 20)), coherent=rng.random() < 0.7)
    if call == "raster":
        case["options"] = rng.choice(["plain", "pn", "ripple", "pn_ripple"])
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _geometries(kind, size):
    """Clustered meshes; they don't depend on the seed."""
    if kind == "icosphere":
        return [S.clusterize(S.icosphere(size), 0)]
    if kind == "terrain":
        return [S.clusterize(S.grid(size, size, float(size), float(size)), 0)]
    meshes = [S.icosphere(4), S.torus(1.0, 0.3, 128, 48), S.grid(128, 128, 2.0, 2.0), S.subdivided_cube(16, 8)]
    return [S.clusterize(m, i) for i, m in enumerate(meshes)]


@functools.lru_cache(maxsize=8)
def _noise(size, octaves):
    return S.value_noise(size, octaves, 5)


def _texture(case, rng, octaves):
    """Tileable noise shifted by the seed, its width cut so that odd sizes are not square."""
    n = case["map"]
    img = np.roll(_noise(n, octaves), (int(rng.integers(n)), int(rng.integers(n))), (0, 1))
    if n & (n - 1):
        img = img[:, :n - n // 3]
    if case["format"] == "unorm16":
        img = np.round(img * 65535.0)
    dtype = {"fp32": np.float32, "fp16": np.float16, "unorm16": np.uint16}[case["format"]]
    return S.Texture(np.ascontiguousarray(img.astype(dtype)), FORMATS[case["format"]])


def _inputs(case, seed):
    """The scene, and the frame constants of this frame. Where the sizes of the outputs follow from the frame's
    decisions, the view and the transforms are the case's own and the seed gives the maps and the rest."""
    rng = np.random.default_rng(seed if case["call"] in ("frame", "decode") else 11)
    maps = np.random.default_rng(seed)
    kind, dist = case["scene"], case["distance"]
    geos = _geometries(kind, 0 if kind == "batched" else case["size"])
    turn = rng.random() * 2 * math.pi
    if kind == "icosphere":
        scene = S.Scene(kind, geos, [S.Instance(0, np.eye(4), 0, 0.05, 0.0)], [_texture(case, maps, 4)])
        tilt = rng.uniform(-0.4, 0.4)
        eye = (dist * math.cos(tilt) * math.sin(turn), dist * math.sin(tilt), dist * math.cos(tilt) * math.cos(turn))
        cam = S.Camera(eye=eye, center=(0.0, 0.0, 0.0), far=100.0, tess_rate_pixels=case["pixels"])
    elif kind == "batched":
        insts = []
        for i in range(case["size"]):
            world = S.translate_rotate_scale(rng.random(3) * 40.0, S.random_unit_quaternion(rng),
                                             0.5 + 1.5 * rng.random())
            insts.append(S.Instance(i % 4, world, i % 4, 0.03, 0.0))
        scene = S.Scene(kind, geos, insts, [_texture(case, maps, 4) for _ in range(4)])
        cam = S.camera_orbit(turn * 30.0 / math.pi, radius=dist, tess_rate_pixels=case["pixels"])
    else:
        n = float(case["size"])
        scene = S.Scene(kind, geos, [S.Instance(0, np.eye(4), 0, 0.1 * n, 0.0)], [_texture(case, maps, 8)])
        eye = np.array([rng.uniform(-0.1, 0.1) * n, dist, rng.uniform(-0.1, 0.1) * n])
        pitch = math.radians(10.0)
        ahead = np.array([math.cos(pitch) * math.sin(turn), -math.sin(pitch), math.cos(pitch) * math.cos(turn)])
        cam = S.Camera(eye=tuple(eye), center=tuple(eye + 10.0 * ahead), width=3840, height=2160, far=4 * n,
                       tess_rate_pixels=case["pixels"])
    fc = S.frame_constants(cam)
    fc["animationRippleAmplitude"], fc["animationRippleFrequency"] = 0.02, 8.0
    fc["animationRippleSpeed"], fc["animationState"] = 1.5, 0.1 * rng.random()
    return scene, fc, rng


def _caps(case):
    if case["scene"] == "terrain":
        return L.default_caps(visible_bits=16, part_bits=21, split_bits=18, vertex_bits=25, megs=2048)
    if case["scene"] == "batched":
        return L.default_caps(vertex_bits=23 if case["size"] < 512 else 24)
    return L.default_caps(visible_bits=12, part_bits=19, split_bits=16, vertex_bits=22, megs=512)


class State:
    def __init__(self, case, seed):
        self.case = case
        scene, fc, rng = _inputs(case, seed)
        flags = L.FLAG_CULLING | OPTIONS[case["options"]]
        if case["call"] in ("train", "decode"):
            flags |= L.FLAG_WRITE_FULLCLUSTERS
        self.pipe = pipe = TessellationPipeline(scene, _caps(case), flags)
        pipe.set_cameras(fc)
        if case["mode"] == "host":
            self._host_buffers(fc)
        if case["call"] == "frame":
            self.outputs = _frame_outputs(self)
            return
        pipe.build("graph")
        torch.cuda.synchronize()
        if case["call"] == "train":
            self.frozen = FrozenFrame(pipe)
            self.grad = _upstream(self.frozen.num_vertices, seed, "cuda")
        elif case["call"] == "decode":
            hits = _hits(case, pipe, scene, rng)
            self.hits = torch.from_numpy(hits.view(np.uint8).reshape(-1)).cuda()
            self.decoded = torch.zeros(len(hits) * L.BaseHit.itemsize, dtype=torch.uint8, device="cuda")
            rec = self.decoded.view(torch.int32).view(-1, 10)
            self.outputs = {"ids": rec[:, :5], "parts": rec[:, 8:], "barycentrics": rec.view(torch.float32)[:, 5:8]}
        else:
            self.raster, b = pipe.state.raster_outputs()
            self.outputs = {"counts": b["counts"].handle.view(torch.int32), "batches": _as(b["batches"], torch.int32, 6),
                            "clip": _as(b["clipPositions"], torch.float32, 4),
                            "world": _as(b["worldPositions"], torch.float32, 3),
                            "indices": b["indices"].handle, "primitives": b["primitiveIDs"].handle.view(torch.int32)}

    def _host_buffers(self, fc):
        """The frame's inputs as one pinned block, which the frame's arguments mirror on the device."""
        one = np.frombuffer(fc.tobytes(), np.uint8)
        records = self.pipe.state.res.instance_records.view(np.uint8).reshape(-1)
        self.inputs = np.concatenate([one, one, records])
        self.staging = torch.empty(self.inputs.size, dtype=torch.uint8, pin_memory=True)
        self.staging_np = self.staging.numpy()
        self.device_block = torch.zeros(self.inputs.size + 256, dtype=torch.uint8, device="cuda")
        self.base = (self.device_block.data_ptr() + 255) // 256 * 256
        self.readback = torch.zeros(L.Readback.itemsize, dtype=torch.uint8, pin_memory=True)
        a = self.pipe.args
        a.view, a.viewLast, a.instances = self.base, self.base + one.size, self.base + 2 * one.size


def _upstream(n, seed, device):
    """dL/dv as a renderer's loss would hand it back."""
    g = torch.from_numpy(np.random.default_rng(seed + 1000003).standard_normal((n, 3)).astype(np.float32))
    return g.to(device)


def _hits(case, pipe, scene, rng):
    """Closest hits on the built frame's instantiations and transient builds: uniformly spread over them, or, as
    primary rays come, in runs of neighbouring pixels on neighbouring ones."""
    out, n = pipe.outputs(), case["hits"]
    ti, full = out["tempInstantiations"], out["fullClusters"]
    inst = out["tempInstanceIDs"].astype(np.int64)
    cid = ti["clusterIdOffset"].astype(np.int64)
    tris = np.zeros(len(ti), np.int64)
    whole = (cid >> 30) == L.RT_CLUSTER_MODE_FULL_CLUSTER
    cid[whole] = full["clusterID"]
    geo = np.array([i.geometry for i in scene.instances])[inst]
    for g, data in enumerate(scene.geometries):
        at = whole & (geo == g)
        tris[at] = data.clusters["numTriangles"][cid[at]]
    config = out["partTriangles"]["triangleID_config"][cid[~whole] & 0x3FFFFFFF] >> 16
    tris[~whole] = pipe.entries["numTriangles"][config & 0x7FFF]
    if "transBuilds" in out:
        builds = out["transBuilds"]
        inst = np.concatenate([inst, out["transInstanceIDs"]])
        cid = np.concatenate([cid, builds["clusterID"].astype(np.int64)])
        tris = np.concatenate([tris, (builds["packed"] & 0x1FF).astype(np.int64)])
    if case["coherent"]:
        runs = -(-n // 64)
        slot = np.repeat(rng.integers(0, len(inst), runs), 64)[:n] + np.sort(rng.integers(0, 4, (runs, 64)), 1).reshape(-1)[:n]
        slot = np.minimum(slot, len(inst) - 1)
    else:
        slot = rng.integers(0, len(inst), n)
    uv = rng.random((n, 2), dtype=np.float32)
    over = uv.sum(1) > 1
    uv[over] = np.float32(1) - uv[over]
    hits = np.zeros(n, L.Hit)
    hits["instanceID"], hits["clusterID"] = inst[slot], cid[slot]
    hits["triangleID"] = (rng.random(n) * tris[slot]).astype(np.int64)
    hits["barycentrics"] = uv
    return hits


def prepare(case, seed):
    return State(case, seed)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _stages(pipe):
    n, passes = pipe.args.numInstances, pipe.split_passes()
    pipe.stage("frame_begin")
    pipe.stage("instances_classify")
    pipe.stage("clusters_cull", 0, n)
    pipe.stage("build_setup", L.BUILD_SETUP_CLASSIFY)
    pipe.stage("cluster_classify", 0, n)
    pipe.stage("build_setup", L.BUILD_SETUP_SPLIT)
    for p in range(passes):
        pipe.stage("triangle_split", 0, n)
        if p + 1 < passes:
            pipe.stage("build_setup", L.BUILD_SETUP_SPLIT_PASS)
    pipe.stage("build_setup", L.BUILD_SETUP_INSTANTIATE_TESS)
    pipe.stage("triangle_instantiate", 0, 0xFFFFFFFF)
    pipe.stage("build_setup", L.BUILD_SETUP_BUILD_BLAS)
    pipe.stage("blas_setup_insertion")
    pipe.stage("blas_clusters_insert")


def _as(buf, dtype, columns):
    return buf.handle.view(dtype).view(-1, columns)


def _frame_outputs(s):
    """Views of the frame's buffers. Addresses of the buffers themselves differ from program to program, so of those
    only the low 16 bits are given."""
    st = s.pipe.state
    out = {
        "vertices": _as(st.gen_vertices, torch.float32, 3),
        "parts": _as(st.part_triangles, torch.int32, 6),
        "splits": _as(st.split_triangles, torch.int32, 6),
        "visible": _as(st.visible_clusters, torch.int32, 2),
        "instance_states": st.instance_states.handle.view(torch.int32),
        "instantiation_ids": _as(st.temp_instantiations, torch.int64, 4)[:, 0],
        "instantiation_templates": _as(st.temp_instantiations, torch.int64, 4)[:, 1],
        "instantiation_vertices": _as(st.temp_instantiations, torch.int16, 16)[:, 8],
        "instantiation_strides": _as(st.temp_instantiations, torch.int64, 4)[:, 3],
        "instantiation_instances": st.temp_instance_ids.handle.view(torch.int32),
        "cluster_addresses": st.temp_cluster_addresses.handle.view(torch.int64),
        "blas_counts": _as(st.blas_build_infos, torch.int64, 2)[:, 0],
        "blas_lists": _as(st.blas_build_infos, torch.int16, 8)[:, 4],
        "blas_addresses": st.blas_cluster_addresses.handle.view(torch.int64),
        "counters": st.build.handle[:104].view(torch.int32),
        "dispatches": st.build.handle[144:224].view(torch.int32),
        "readback": st.readback.handle.view(torch.int32),
    }
    if st.transient:
        builds = _as(st.trans_builds, torch.int32, 16)
        out["builds"] = builds[:, :6]
        out["build_indices"] = _as(st.trans_builds, torch.int16, 32)[:, 12]
        out["build_vertices"] = _as(st.trans_builds, torch.int16, 32)[:, 16]
        out["build_instances"] = st.trans_instance_ids.handle.view(torch.int32)
        out["build_addresses"] = st.trans_cluster_addresses.handle.view(torch.int64)
    if s.case["mode"] == "host":
        out["host_readback"] = s.readback.view(torch.int32)
    return out


def run(s):
    pipe, call, mode = s.pipe, s.case["call"], s.case["mode"]
    if call == "train":
        v = tessellate(s.frozen)
        grads = torch.autograd.grad(v, s.frozen.parameters(), s.grad)
        return {"vertices": v.detach(), "grads": list(grads)}
    if call == "decode":
        pipe.decode_hits_device(s.hits, s.decoded)
        return s.outputs
    if call == "raster":
        pipe.stage("raster_batches", ctypes.byref(s.raster))
        return s.outputs
    if mode == "host":
        # the frame before has ended (the wait below), so its staging block is free to be written
        s.staging_np[:] = s.inputs
        pipe.build_host(s.staging.data_ptr(), s.base, s.inputs.size, s.readback.data_ptr())
        torch.cuda.current_stream().synchronize()
    elif mode == "stages":
        _stages(pipe)
    else:
        pipe.build(mode)
    return s.outputs


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def work(case):
    """Bytes: the scene's arrays, each read once (maps: at most four texels a vertex), and the frame's outputs, by the
    counts of a frame of these sizes. Flops: about 60 for each vertex and for each base triangle."""
    s = prepare(case, 1)
    if case["call"] == "frame":
        run(s)
    torch.cuda.synchronize()
    st, scene, caps = s.pipe.state, s.pipe.scene, s.pipe.caps
    rb = st.readback.read(L.Readback, 1)[0]
    verts = min(int(rb["numGenVertices"]), caps["maxGeneratedVertices"])
    parts = min(int(rb["numPartTriangles"]), caps["maxPartTriangles"])
    temps, builds = int(rb["numActualTempInstantiations"]), int(rb["numActualTransBuilds"])
    base_vertices = sum(len(g.positions) for g in scene.geometries)
    base_triangles = sum(g.num_triangles for g in scene.geometries)
    clusters = sum(g.num_clusters for g in scene.geometries)
    texel = scene.textures[0].texels.itemsize
    maps = texel * min(4 * verts, sum(t.texels.size for t in scene.textures))
    geometry = 32 * base_vertices + 3 * base_triangles + 28 * clusters + 192 * len(scene.instances)
    if case["call"] == "frame":
        written = (12 * verts + 24 * parts + 44 * temps + 76 * builds + 8 * (temps + builds)
                   + 8 * min(scene.total_clusters, caps["maxVisibleClusters"]) + 24 * caps["maxSplitTriangles"]
                   + 20 * len(scene.instances) + 880)
        return {"bytes": geometry + maps + written, "flops": 60 * verts + 60 * scene.total_triangles}
    if case["call"] == "train":
        # forward: attributes, parts and maps in, vertices out; backward: those and dL/dv in, the gradients out
        grads = sum(4 * p.numel() for p in s.frozen.parameters())
        return {"bytes": 2 * (geometry + maps + 24 * parts + 44 * temps) + 24 * verts + grads, "flops": 240 * verts}
    if case["call"] == "decode":
        return {"bytes": 64 * case["hits"] + 24 * parts + geometry - 32 * base_vertices, "flops": 40 * case["hits"]}
    run(s)
    batches, rv, rt = (int(x) for x in s.outputs["counts"][:3].cpu())
    return {"bytes": geometry + maps + 24 * parts + 24 * batches + 28 * rv + 7 * rt, "flops": 100 * rv}


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------

def _frustum_visible(scene, fc):
    """Frustum and size test of the instances' boxes, in single precision as the decisions are defined."""
    f32 = np.float32
    vp = fc["viewProjMatrix"].reshape(4, 4).astype(f32)  # [column][row]
    seen = np.zeros(len(scene.instances), bool)
    for i, inst in enumerate(scene.instances):
        w = inst.world.T.astype(f32)
        g = scene.geometries[inst.geometry]
        m = ((vp[0] * w[:, :1] + vp[1] * w[:, 1:2]) + vp[2] * w[:, 2:3]) + vp[3] * w[:, 3:4]
        corner = np.array([[(g.hi if n >> k & 1 else g.lo)[k] for k in range(3)] for n in range(8)], f32)
        h = ((m[0] * corner[:, :1] + m[1] * corner[:, 1:2]) + m[2] * corner[:, 2:]) + m[3]
        x, y, z, d = h.T
        outside = [x < -d, x > d, y < -d, y > d, z < 0, z > d, d <= 0]
        inside = not any(o.all() for o in outside)
        valid = not (np.abs(d) < f32(1.2e-07)).any()
        c = np.clip(h[:, :2] / np.abs(d)[:, None], f32(-1), f32(1))
        large = ((c.max(0) - c.min(0)) > f32(2) / fc["viewportf"].astype(f32)).any()
        seen[i] = inside and (not valid or large)
    return seen


def _edge_factors(scene, fc, inst, tri):
    """Segments of each edge of an instance's triangles (rows of vertex indices), in single precision likewise."""
    f32 = np.float32
    p = scene.geometries[inst.geometry].positions
    w = inst.world.T.astype(f32)
    p = ((w[0, :3] * p[:, :1] + w[1, :3] * p[:, 1:2]) + w[2, :3] * p[:, 2:]) + w[3, :3]

    def length(v):
        return np.sqrt((v[:, 0] * v[:, 0] + v[:, 1] * v[:, 1]) + v[:, 2] * v[:, 2])

    far = length(p - fc["viewPos"][:3].astype(f32))
    f = np.zeros((len(tri), 3), np.int64)
    for k in range(3):
        a, b = tri[:, k], tri[:, (k + 1) % 3]
        per = f32(1) / np.maximum(f32(fc["nearPlane"]), np.minimum(far[a], far[b]))
        e = ((length(p[a] - p[b]) * per) * f32(fc["viewportf"][1])) * f32(fc["tessRate"])
        f[:, k] = np.clip(np.rint(e), 1, 32768)
    return f


def _decisions(scene, fc):
    """The frame's vertices in their order, as (owner instance, three base vertices, their weights), how many of them
    belong to whole clusters, and the number of parts. None where an edge needs more segments than the table has."""
    raw = load_raw_table()
    configs = iter(raw.configs.reshape(-1, 4).astype(np.int64))
    record = np.zeros((12, 12, 12, 4), np.int64)
    for x in range(1, 12):
        for y in range(1, x + 1):
            for z in range(1, y + 1):
                record[x, y, z] = record[x, z, y] = next(configs)
    first = np.cumsum([0] + [len(g.positions) for g in scene.geometries])
    seen = _frustum_visible(scene, fc)
    whole, parts, corners, factors = [], [], [], []
    for i, inst in enumerate(scene.instances):
        g = scene.geometries[inst.geometry]
        nt, nv = g.clusters["numTriangles"].astype(np.int64), g.clusters["numVertices"].astype(np.int64)
        owner = np.repeat(np.arange(len(nt)), nt)
        tri = g.local_triangles.reshape(-1, 3).astype(np.int64) + g.clusters["firstLocalVertex"].astype(np.int64)[owner, None]
        f = _edge_factors(scene, fc, inst, tri) if seen[i] else np.ones((len(tri), 3), np.int64)
        if f.max() > 11:
            return None
        plain = np.ones(len(nt), bool)
        plain[owner[f.max(1) > 1]] = False
        at = np.flatnonzero(np.repeat(plain, nv)) + first[inst.geometry]
        whole.append(np.stack([np.full(len(at), i), at], 1))
        cut = ~plain[owner]
        parts.append(np.full(int(cut.sum()), i))
        corners.append(tri[cut] + first[inst.geometry])
        factors.append(f[cut])
    whole, parts, corners, f = (np.concatenate(v) for v in (whole, parts, corners, factors))
    # the largest factor goes first, and the corners turn with it
    m = f.max(1)
    turn = np.where(m == f[:, 1], 1, np.where(m == f[:, 2], 2, 0))
    order = (np.arange(3) + turn[:, None]) % 3
    f, corners = np.take_along_axis(f, order, 1), np.take_along_axis(corners, order, 1)
    r = record[f[:, 0], f[:, 1], f[:, 2]]
    part = np.repeat(np.arange(len(f)), r[:, 3])
    local = np.arange(len(part)) - np.repeat(np.cumsum(r[:, 3]) - r[:, 3], r[:, 3])
    word = raw.vertices[r[part, 1] + local].astype(np.int64)
    w = np.stack([32768 - (word & 0xFFFF) - (word >> 16), word & 0xFFFF, word >> 16], 1) / 32768.0
    flipped = (f[:, 2] > f[:, 1])[part]
    w[flipped] = w[flipped][:, [1, 0, 2]]
    owner = np.concatenate([whole[:, 0], parts[part]])
    base = np.concatenate([np.repeat(whole[:, 1:], 3, 1), corners[part]])
    weight = np.concatenate([np.tile([1.0, 0.0, 0.0], (len(whole), 1)), w])
    return owner, base, weight, len(whole), len(f)


def _displaced(scene, fc, owner, base, weight, positions, normals, texels):
    """Base attributes mixed by the weights, displaced by the bilinear, repeating map along the unit normal."""
    dev = positions.device
    on = lambda a: torch.as_tensor(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    uvs = on(np.concatenate([g.texcoords for g in scene.geometries]).astype(np.float64))
    owner, base, weight = on(owner), on(base), on(weight)[:, :, None]
    unit = normals / normals.norm(dim=1, keepdim=True)
    p, n, uv = ((a[base] * weight).sum(1) for a in (positions, unit, uvs))
    shape = np.array([t.texels.shape for t in scene.textures])
    start = np.cumsum([0] + [t.texels.size for t in scene.textures])
    tex = np.array([i.displacement_index for i in scene.instances])
    wide, high, begin = (on(a[tex].astype(np.int64))[owner] for a in (shape[:, 1], shape[:, 0], start))
    x, y = uv[:, 0] * wide - 0.5, uv[:, 1] * high - 0.5
    ix, iy = x.detach().floor().long(), y.detach().floor().long()
    fx, fy = x - ix, y - iy
    h = 0.0
    for dx, dy in ((0, 0), (1, 0), (0, 1), (1, 1)):
        at = begin + ((iy + dy) % high) * wide + (ix + dx) % wide
        h = h + texels[at] * (fx if dx else 1 - fx) * (fy if dy else 1 - fy)
    scale = on(np.array([i.displacement_scale for i in scene.instances]).astype(np.float32).astype(np.float64))[owner]
    offset = on(np.array([i.displacement_offset for i in scene.instances]).astype(np.float64))[owner]
    h = h * scale * float(fc["displacementScale"]) + offset + float(fc["displacementOffset"])
    return p + n / n.norm(dim=1, keepdim=True) * h[:, None]


def _padded(v, rows):
    out = torch.zeros((rows, v.shape[1]), dtype=torch.float64)
    out[:len(v)] = v.detach().cpu()
    return out


def exact(case, seed):
    """Positions and gradients in 64 bits, for frames without split triangles and the shader options. Every other
    output is a whole number or, for the decode, depends on the frame's own records."""
    if case["call"] == "decode" or case["options"] != "plain" or case["scene"] == "terrain":
        return None
    scene, fc, _ = _inputs(case, seed)
    got = _decisions(scene, fc)
    if got is None:
        return None
    owner, base, weight, whole, parts = got
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    put = lambda a: torch.as_tensor(np.concatenate(a).astype(np.float64)).to(dev).requires_grad_()  # noqa: E731
    positions, normals = put([g.positions for g in scene.geometries]), put([g.normals for g in scene.geometries])
    unit = 65535.0 if case["format"] == "unorm16" else 1.0
    texels = put([t.texels.reshape(-1) / unit if unit != 1.0 else t.texels.reshape(-1) for t in scene.textures])
    v = _displaced(scene, fc, owner, base, weight, positions, normals, texels)
    if case["call"] == "frame":
        return {"vertices": _padded(v, _caps(case)["maxGeneratedVertices"])}
    if case["call"] == "train":
        grads = torch.autograd.grad(v, [positions, normals, texels], _upstream(len(v), seed, dev).double())
        count = [len(g.positions) for g in scene.geometries]
        parted = [*grads[0].split(count), *grads[1].split(count)]
        parted += [t.view(s.texels.shape) for t, s in zip(grads[2].split([s.texels.size for s in scene.textures]),
                                                          scene.textures)]
        return {"vertices": v.detach().cpu(), "grads": [g.cpu() for g in parted]}
    v, owner = v[whole:].detach(), torch.as_tensor(owner[whole:]).to(dev)
    world = np.stack([i.world.astype(np.float32).astype(np.float64) for i in scene.instances])
    m = torch.as_tensor(world).to(dev)[owner]
    wp = torch.einsum("nij,nj->ni", m[:, :3, :3], v) + m[:, :3, 3]
    vp = torch.as_tensor(fc["viewProjMatrix"].reshape(4, 4).astype(np.float64)).to(dev)
    clip = torch.cat([wp, torch.ones_like(wp[:, :1])], 1) @ vp
    return {"clip": _padded(clip, 78 * parts), "world": _padded(wp, 78 * parts)}
