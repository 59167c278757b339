"""Scenes whose Nodes are not what arbor_buildBounds makes of P and Order go
through the block batch in a fixed order (csrc/orderbatch.cuh), whose results
tests/test_traversal_cpu.py pins; here the routes to it.

Bar: bit for bit equal to arbor_tracePixels / arbor_shadePixels on the same
scene alone.
"""
import ctypes

import numpy as np
import pytest
import torch

import arbor_b200 as ab
import workloads
from gpu_util import dev, dev_array, host, ok, render_buffers
from test_gpu_batch import Batch, single_image
from test_gpu_tight import Scene, state

pytestmark = pytest.mark.gpu


def cut(nodes):
    """Leaf boxes cut short: hits before their own box, so that the order
    decides which counts."""
    n = nodes.view(65536, 8)
    n[32768:, 0:3] += 0.04 * torch.rand((32768, 3), generator=torch.Generator().manual_seed(1)).to(n.device)


def bits(t):
    return host(t).view(np.uint32).reshape(-1, 4)


def test_one_irregular_species_among_regular_ones(cuda):
    """All instances on the irregular scene, of three resident ones."""
    w, h, n = 333, 187, 3
    s, one, C = Scene([7, 20, 33]), Scene([20]), dev(state(w, h, wind=0.6))
    cut(s.Nodes[65536 * 8:2 * 65536 * 8])
    one.Nodes.copy_(s.Nodes[65536 * 8:2 * 65536 * 8])
    of = (ctypes.c_int * 324)(*([1] * 324))
    a, b = render_buffers(w, h), render_buffers(w, h)
    ok(ab.call("arbor_traceSpeciesPixels", s.P, s.Nodes, s.Order, n, of, C, a["Hit"], w, h))
    ok(ab.call("arbor_shadeSpeciesPixels", s.P, s.Nodes, s.Order, n, of, C, a["Hit"], a["Linear"], a["Guide"], w, h))
    ok(ab.call("arbor_tracePixels", one.P, one.Nodes, one.Order, C, b["Hit"], w, h))
    ok(ab.call("arbor_shadePixels", one.P, one.Nodes, one.Order, C, b["Hit"], b["Linear"], b["Guide"], w, h))
    assert (host(b["Hit"]).reshape(-1, 4)[:, 1] >= 0).sum() > 1000
    for k in ("Hit", "Linear", "Guide"):
        assert np.array_equal(bits(a[k]), bits(b[k])), k


@pytest.mark.parametrize("queue", [16])
def test_batch_scene_changed_through_its_buffers(cuda, queue):
    import gpu_util

    views = [(v % 2, w, h, workloads.view_pose_state((7, 1788)[v % 2], w, h, 11.0, -23.0, 0.7, 0.12)) for v, (w, h) in
             enumerate(((320, 180), (97, 61), (160, 90)))]
    batch = Batch(views)
    try:
        p = batch.buffers(0).Nodes
        nodes = torch.from_numpy(dev_array(p, 65536 * 8)).cuda()
        cut(nodes)
        torch.cuda.synchronize()
        assert gpu_util._cudart().cudaMemcpy(p, nodes.data_ptr(), 65536 * 32, 3) == 0
        batch.configure(16, 2, 0, queue)
        batch.call("arbor_batch_render")
        for v in range(len(views)):
            got, want = batch.images(v), single_image(cuda, gpu_util, batch, v)
            for k in ("Hit", "Linear", "Guide", "Filtered", "Pixels"):
                assert np.array_equal(np.ascontiguousarray(got[k]).view(np.uint32), np.ascontiguousarray(want[k]).view(np.uint32)), f"view {v} {k}"
    finally:
        batch.close()


@pytest.mark.parametrize("wind", [3.0, 8.0, 30.0])
def test_batch_in_a_storm(cuda, wind):
    """Views whose wind sends the shadow pass, or both passes, to the fixed
    order, beside one in still air."""
    import gpu_util

    views = []
    for v, (w, h) in enumerate(((320, 180), (97, 61), (160, 90))):
        C = workloads.view_pose_state((7, 1788)[v % 2], w, h, 11.0, -23.0, 0.7, 0.12)
        C[8], C[11] = 3.25, 0.0 if v == 1 else wind
        views.append((v % 2, w, h, C))
    batch = Batch(views)
    try:
        batch.call("arbor_batch_render")
        for v in range(len(views)):
            got, want = batch.images(v), single_image(cuda, gpu_util, batch, v)
            for k in ("Hit", "Linear", "Guide", "Filtered", "Pixels"):
                assert np.array_equal(np.ascontiguousarray(got[k]).view(np.uint32), np.ascontiguousarray(want[k]).view(np.uint32)), f"view {v} {k}"
    finally:
        batch.close()
