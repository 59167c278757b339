"""The batched traversal over its own tight boxes (csrc/tight.cuh) against the
reference's traversal as written over Nodes (arbor_tracePixelsInOrder,
arbor_shadePixelsInOrder), on every route a call can take to its boxes: the
call's scratch, none during stream capture, none above the scratch's scene
limit, and none for a scene whose Nodes are not what buildBounds makes.

Bar: a hit that rounding puts before its own box can be kept by one traversal
order and pruned by the other; over 1080p frames that moves at most 1 pixel in
10^5 (test_gpu_order.py).  Here: at most 1 + pixels / 10^5 pixels differ.
"""
import ctypes

import numpy as np
import pytest

import arbor_b200 as ab
import workloads
from gpu_util import dev, host, ok, render_buffers, zeros_f, zeros_u

pytestmark = pytest.mark.gpu


class Scene:
    def __init__(self, seeds):
        n = len(seeds)
        self.n = n
        self.B, self.P, self.Nodes = zeros_f(2109 * 20), zeros_f(n * 32768 * 24), zeros_f(n * 65536 * 8)
        self.Keys, self.Order, scratch = zeros_u(32768), zeros_u(n * 32768), zeros_u(65536)
        for k, seed in enumerate(seeds):
            ok(ab.call("arbor_buildScene", seed, self.B, self.P[k * 32768 * 24:], self.Keys, self.Order[k * 32768:],
                       self.Nodes[k * 65536 * 8:], None, scratch))


def state(w, h, seed=7, wind=0.0, pitch=0.12):
    C = workloads.view_pose_state(seed, w, h, 11.0, -23.0, 0.7, pitch)
    C[8], C[11] = 3.25, wind
    return C


def differing(a, b, width=4):
    a, b = host(a).view(np.uint32).reshape(-1, width), host(b).view(np.uint32).reshape(-1, width)
    return int((a != b).any(axis=1).sum())


def in_order(s, C, w, h, tree=0):
    r = render_buffers(w, h)
    ok(ab.call("arbor_tracePixelsInOrder", s.P, s.Nodes, s.Order, C, r["Hit"], w, h, tree))
    ok(ab.call("arbor_shadePixelsInOrder", s.P, s.Nodes, s.Order, C, r["Hit"], r["Linear"], r["Guide"], w, h, tree))
    return r


def batched(s, C, w, h, tree=0, hit=None):
    form = "Tree" if tree else ""
    r = render_buffers(w, h)
    ok(ab.call(f"arbor_trace{form}Pixels", s.P, s.Nodes, s.Order, C, r["Hit"], w, h))
    ok(ab.call(f"arbor_shade{form}Pixels", s.P, s.Nodes, s.Order, C, r["Hit"] if hit is None else hit, r["Linear"], r["Guide"], w, h))
    return r


def close(a, b, w, h):
    bar = 1 + w * h // 100000
    for name in ("Hit", "Linear", "Guide"):
        n = differing(a[name], b[name])
        assert n <= bar, f"{name}: {n} of {w * h} pixels differ (at most {bar})"


@pytest.mark.parametrize("w,h", [(1, 1), (7, 5), (8, 4), (9, 33), (333, 187), (1201, 403)])
@pytest.mark.parametrize("wind", [0.0, 0.6])
def test_sizes_and_wind(cuda, w, h, wind):
    s, C = Scene([7]), dev(state(w, h, wind=wind))
    a = in_order(s, C, w, h)
    close(batched(s, C, w, h, hit=a["Hit"]), a, w, h)


@pytest.mark.parametrize("wind", [7.0, float("inf")])
def test_wind_beyond_the_breeze(cuda, wind):
    """Leaves turned by more than any box is widened for at the breeze, and an
    angle that is not finite."""
    w, h = 320, 200
    s, C = Scene([42]), dev(state(w, h, seed=42, wind=wind))
    a = in_order(s, C, w, h)
    close(batched(s, C, w, h, hit=a["Hit"]), a, w, h)


def test_single_tree(cuda):
    w, h = 250, 190
    C = workloads.single_tree_camera(w, h)
    C[22] = 1.0
    s, C = Scene([1]), dev(C)
    a = in_order(s, C, w, h, tree=1)
    close(batched(s, C, w, h, tree=1, hit=a["Hit"]), a, w, h)


@pytest.mark.parametrize("what", ["inner box", "emptied subtree", "top node"])
def test_nodes_that_are_not_the_records_bounds(cuda, what):
    """Nodes say what is hit: a moved or emptied node hides what lies under it,
    whatever the records' own bounds are.  (Boxes of leaves cut short are not
    here: hits then lie before their own boxes, and which of them counts
    depends on the order of the visits.)"""
    w, h = 400, 240
    s, C = Scene([7]), dev(state(w, h))
    N = s.Nodes.view(65536, 8)
    if what == "inner box":
        N[600, 4:7] -= 0.7
    elif what == "emptied subtree":
        N[65, 3] = 0.0
    else:
        N[5, 4] -= 1.5
    a = in_order(s, C, w, h)
    close(batched(s, C, w, h, hit=a["Hit"]), a, w, h)


def test_under_capture(cuda):
    """A captured call allocates nothing: its graph can be instantiated and
    replayed like any other, and gives what the call gives."""
    import torch

    w, h = 256, 144
    s, C = Scene([7]), dev(state(w, h))
    want, r = batched(s, C, w, h), render_buffers(w, h)
    g = torch.cuda.CUDAGraph()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(g, stream=side):
        ok(ab.call("arbor_tracePixels", s.P, s.Nodes, s.Order, C, r["Hit"], w, h, stream=side))
        ok(ab.call("arbor_shadePixels", s.P, s.Nodes, s.Order, C, r["Hit"], r["Linear"], r["Guide"], w, h, stream=side))
    for _ in range(2):
        for name in ("Hit", "Linear", "Guide"):
            r[name].zero_()
        g.replay()
        torch.cuda.synchronize()
        close(r, want, w, h)


@pytest.mark.parametrize("n", [2, 32, 33])
def test_species_scratch_limit(cuda, n):
    """n resident scenes, on both sides of the scratch's limit of 32, against
    one call per scene with every instance on it (pixels whose hit tree uses
    that scene in the mixed forest and that no nearer tree changes are covered
    by test_gpu_species.py; here all instances use scene n - 1)."""
    w, h = 320, 180
    s, C = Scene([7 + 13 * k for k in range(n)]), dev(state(w, h))
    of = (ctypes.c_int * 324)(*([n - 1] * 324))
    r = render_buffers(w, h)
    ok(ab.call("arbor_traceSpeciesPixels", s.P, s.Nodes, s.Order, n, of, C, r["Hit"], w, h))
    ok(ab.call("arbor_shadeSpeciesPixels", s.P, s.Nodes, s.Order, n, of, C, r["Hit"], r["Linear"], r["Guide"], w, h))
    one = Scene([7 + 13 * (n - 1)])
    close(r, batched(one, C, w, h), w, h)


def test_world_seed_the_host_never_registered(cuda):
    """A C record written by hand with a world seed no call has seen: the
    instance table comes from the call's scratch, during capture from shared
    memory, and is the one arbor_tracePixelsInOrder builds."""
    import torch

    w, h = 200, 120
    s = Scene([7])
    C = state(w, h)
    C[31] = 987653.0
    C = dev(C)
    a = in_order(s, C, w, h)
    close(batched(s, C, w, h, hit=a["Hit"]), a, w, h)
    r = render_buffers(w, h)
    g = torch.cuda.CUDAGraph()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(g, stream=side):
        ok(ab.call("arbor_tracePixels", s.P, s.Nodes, s.Order, C, r["Hit"], w, h, stream=side))
        ok(ab.call("arbor_shadePixels", s.P, s.Nodes, s.Order, C, a["Hit"], r["Linear"], r["Guide"], w, h, stream=side))
    g.replay()
    torch.cuda.synchronize()
    close(r, a, w, h)
