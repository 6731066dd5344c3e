"""The gradients that the autograd wrapper hands out have their parameters' shapes, also those without an element."""
import types

import numpy as np
import pytest

from tests.conftest import cuda_available


def _given_back_flat(flat, tensors):
    """torch._utils._unflatten_dense_tensors as in the versions that give an empty tensor back as a vector."""
    import torch
    out, at = [], 0
    for t in tensors:
        n = t.numel()
        out.append(flat.narrow(0, at, n).view(t.shape) if n else torch.empty(0, dtype=flat.dtype))
        at += n
    return tuple(out)


@pytest.mark.parametrize("own", [True, False])
def test_empty_parameters(monkeypatch, own):
    import torch
    from vk_tessellated_clusters_gb300.autograd import FrozenFrame, tessellate
    if own:
        monkeypatch.setattr(torch._utils, "_unflatten_dense_tensors", _given_back_flat)
    monkeypatch.setattr(torch, "device", lambda *a: "cpu")
    vertices = torch.arange(12.0).view(4, 3)
    frozen = object.__new__(FrozenFrame)
    frozen.torch, frozen.num_vertices = torch, 4
    frozen.pipe = types.SimpleNamespace(device=0, stage=lambda name: None, gen_vertices_tensor=lambda n: vertices,
                                        backward=lambda *a: None)
    frozen.positions = [torch.zeros(4, 3), torch.zeros(0, 3)]
    frozen.normals = [torch.ones(4, 3), torch.zeros(0, 3)]
    frozen.texels = [torch.zeros(0, 0), None, torch.zeros(5, 2)]
    frozen._inst_geo = np.array([0, 1])
    for p in frozen.parameters():
        p.requires_grad_(True)
    frozen._layout_gradients(None)
    tessellate(frozen).sum().backward()
    assert [p.grad.shape for p in frozen.parameters()] == [p.shape for p in frozen.parameters()]
    dP, dN, dT = frozen.scatter_gradients(torch.ones(4, 3))
    assert [g.shape for g in dP + dN] == [p.shape for p in frozen.positions + frozen.normals]
    assert dT[0].shape == (0, 0) and dT[1] is None and dT[2].shape == (5, 2)


@pytest.mark.gpu
@pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")
def test_empty_map_on_the_gpu():
    """An empty fp32 map is a parameter like any other: its gradient has its shape, the others are those of the frame
    without it (the map's instances are displaced by the offset alone)."""
    import torch
    from vk_tessellated_clusters_gb300 import layouts as L
    from vk_tessellated_clusters_gb300 import scene as S
    from vk_tessellated_clusters_gb300.autograd import FrozenFrame, tessellate
    from vk_tessellated_clusters_gb300.pipeline import TessellationPipeline
    sc = S.scene_icosphere(subdivisions=3, map_size=64)
    sc.textures[0] = S.Texture(np.zeros((0, 0), np.float32), L.TEXEL_F32)
    sc.textures.append(S.Texture(np.ones((4, 4), np.float32), L.TEXEL_F32))
    caps = L.default_caps(visible_bits=12, part_bits=17, split_bits=14, vertex_bits=20, megs=64)
    pipe = TessellationPipeline(sc, caps, L.FLAG_CULLING | L.FLAG_WRITE_FULLCLUSTERS)
    pipe.set_cameras(S.Camera(eye=(0.0, 0.0, 3.0), center=(0.0, 0.0, 0.0), tess_rate_pixels=8.0))
    pipe.build("graph")
    frozen = FrozenFrame(pipe)
    tessellate(frozen).sum().backward()
    assert [p.grad.shape for p in frozen.parameters()] == [p.shape for p in frozen.parameters()]
    # the barycentric weights of every vertex sum to one, so the positions' gradients sum to the vertices
    total = frozen.positions[0].grad.sum(0).cpu().numpy()
    assert np.abs(total - frozen.num_vertices).max() <= 1e-4 * frozen.num_vertices
    assert not frozen.texels[1].grad.any()
    assert pipe.device_errors() == 0
    pipe.close()
