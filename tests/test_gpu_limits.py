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
