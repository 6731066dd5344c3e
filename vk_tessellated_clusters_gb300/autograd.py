"""Differentiable displaced-vertex generation through torch.autograd.

The tessellation decisions of a built frame (segment counts, configs, split
tree, instantiation order) are piecewise constant in the inputs, so they are
held fixed: the differentiable function maps base positions, base normals and
displacement texels to the frame's generated vertices

    part triangle : v = P(w) + normalize(N(w)) * (bilinear(tex, uv(w)) * s + o)
    full cluster  : v = p + normalize(n) * (bilinear(tex, uv) * s + o)

(triangle_tess_template_instantiate.comp.glsl:343-371,
cluster_classify.comp.glsl:457-482), with forward tc_generate_vertices and
backward tc_instantiate_backward (CUDA kernels). The parameters are views of
the pipeline's own device buffers, so in-place updates (an optimiser step) are
seen by the next frame.

    frozen = FrozenFrame(pipe)               # after pipe.build(...) with FLAG_WRITE_FULLCLUSTERS
    v = tessellate(frozen)                    # (num_vertices, 3) float32
    loss = ((v - target) ** 2).sum(); loss.backward()
    frozen.positions[0].grad, frozen.normals[0].grad, frozen.texels[0].grad
"""
from __future__ import annotations

import numpy as np

from . import layouts as L


class FrozenFrame:
    def __init__(self, pipe):
        import torch
        self.torch = torch
        if not (pipe.state.flags & L.FLAG_WRITE_FULLCLUSTERS):
            raise ValueError("the frame must be built with FLAG_WRITE_FULLCLUSTERS")
        self.pipe = pipe
        torch.cuda.synchronize(pipe.device)
        out = pipe.state
        self.num_vertices = self._accepted_vertex_count()
        scene = pipe.scene
        res = out.res
        self.positions = [self._view(b["positions"], g.positions.shape) for b, g in zip(res.geo, scene.geometries)]
        self.normals = [self._view(b["normals"], g.normals.shape) for b, g in zip(res.geo, scene.geometries)]
        self.texels = []
        for buf, t in zip(res.tex, scene.textures):
            if t.format != L.TEXEL_F32:
                self.texels.append(None)  # only fp32 maps are differentiable parameters
            else:
                self.texels.append(buf.handle[:t.texels.nbytes].view(torch.float32).view(t.texels.shape))
        for p in self.parameters():
            p.requires_grad_(True)
        self._inst_geo = np.array([i.geometry for i in scene.instances], np.int64)
        self._layout_gradients(scene)

    def _layout_gradients(self, scene) -> None:
        """All gradients of one backward live in one flat float32 buffer, in
        parameter order; the kernel's pointer tables (per instance
        dPositions/dNormals, per map texels) are its address plus these
        offsets (0 where a gradient is not wanted), so a backward is a zeroed
        buffer, one addition for the table and the kernel, with no
        host-to-device transfer and no copy."""
        torch = self.torch
        sizes = [p.numel() for p in self.positions] + [n.numel() for n in self.normals]
        sizes += [t.numel() if t is not None else 0 for t in self.texels]
        starts = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
        self._grad_floats = int(starts[-1])
        # parameters without an element (an empty map): gradients() gives their gradients the shape
        self._empty = [(i, p.shape) for i, p in enumerate(self.parameters()) if p.numel() == 0]
        ng = len(self.positions)
        rel = np.zeros((len(self._inst_geo), 2), np.int64)
        rel[:, 0] = 4 * starts[self._inst_geo]
        rel[:, 1] = 4 * starts[ng + self._inst_geo]
        tex = np.array([4 * starts[2 * ng + i] if t is not None else -1 for i, t in enumerate(self.texels)] or [-1],
                       np.int64)
        self._num_targets = rel.size
        offsets = np.concatenate([rel.reshape(-1), tex])
        device = self.device = torch.device("cuda", self.pipe.device)
        self._offsets = torch.from_numpy(np.maximum(offsets, 0)).to(device)
        self._wanted = torch.from_numpy((offsets >= 0).astype(np.int64)).to(device)
        self._flat, self._table = None, None  # gradient_buffers()
        self._vertices = self.pipe.gen_vertices_tensor(self.num_vertices)

    def _view(self, buf, shape):
        n = int(np.prod(shape))
        return buf.handle[:4 * n].view(self.torch.float32).view(*shape)

    def _accepted_vertex_count(self) -> int:
        out = self.pipe.outputs()
        return len(out["genVertices"])

    def parameters(self) -> list:
        return [p for p in self.positions + self.normals + self.texels if p is not None]

    # ---- forward / backward on the C ABI ------------------------------------------------

    def generate(self):
        """Vertices of the frozen frame from the current parameters (a copy)."""
        self.pipe.stage("generate_vertices")
        return self._vertices.clone()

    def _pointer_table(self, flat):
        return self.torch.add(self._offsets, self._wanted, alpha=flat.data_ptr())

    def gradient_buffers(self, device=None):
        """A persistent flat float32 gradient buffer, zeroed (enqueued on the
        current stream), and the kernel's pointer table into it."""
        if self._flat is None:
            self._flat = self.torch.zeros(self._grad_floats, dtype=self.torch.float32, device=self.device)
            self._table = self._pointer_table(self._flat)
        self._flat.zero_()
        return self._flat, self._table

    def launch_backward(self, grad_vertices, table) -> None:
        """tc_instantiate_backward: accumulates dL/dv into the buffer `table` points at."""
        self.pipe.backward(grad_vertices.data_ptr(), table.data_ptr(), table.data_ptr() + 8 * self._num_targets)

    def gradients(self, grad_vertices):
        """dL/dv -> the gradients of parameters(), in their order; all enqueued
        on the current stream, no synchronisation."""
        flat = self.torch.empty(self._grad_floats, dtype=self.torch.float32, device=self.device).zero_()
        self.launch_backward(grad_vertices.contiguous().float(), self._pointer_table(flat))
        grads = list(self.torch._utils._unflatten_dense_tensors(flat, self.parameters()))
        for i, shape in self._empty:  # (given back as vectors of length 0 by some versions)
            grads[i] = grads[i].view(shape)
        return grads

    def scatter_gradients(self, grad_vertices):
        """dL/dv -> (dPositions, dNormals, dTexels), lists parallel to the
        parameters (None for a map without gradient)."""
        grads, ng = self.gradients(grad_vertices), len(self.positions)
        texels = iter(grads[2 * ng:])
        return (list(grads[:ng]), list(grads[ng:2 * ng]),
                [next(texels) if t is not None else None for t in self.texels])


class _Tessellate:
    """torch.autograd.Function, built lazily so importing this module needs no torch."""
    fn = None

    @classmethod
    def get(cls):
        if cls.fn is None:
            import torch

            class TessellateFunction(torch.autograd.Function):
                @staticmethod
                def forward(ctx, frozen, *params):
                    ctx.frozen = frozen
                    return frozen.generate()

                @staticmethod
                def backward(ctx, grad):
                    return (None, *ctx.frozen.gradients(grad))

            cls.fn = TessellateFunction
        return cls.fn


def tessellate(frozen: FrozenFrame):
    return _Tessellate.get().apply(frozen, *frozen.parameters())
