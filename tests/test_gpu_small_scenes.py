"""Scenes of a few records, small beside the distance they are seen from or
beside the swing of their leaves, through the batched passes against the
reference's traversal as written (arbor_tracePixelsInOrder,
arbor_shadePixelsInOrder); tests/test_traversal_cpu.py runs the same code on
the CPU with every load checked.

Bar: every pixel written and equal bit for bit.  No surface lies behind another
closely enough for the order of the tests to matter.
"""
import ctypes
import math

import numpy as np
import pytest
import torch

import arbor_b200 as ab
import workloads
from gpu_util import dev, host, ok, zeros_f
from pyoracle import Oracle
from test_traversal_cpu import CAPACITY, leaf, stone, wood

pytestmark = pytest.mark.gpu

LEAF = leaf(0.0, 1.0, 0.0, 0.15, 0.07)
# records, distance, wind, the angle the image spans (radians)
SCENES = {
    "stone of 1 cm at 5 m": ([stone(0.0, 1.0, 0.0, 0.005)], 5.0, 0.0, 0.006),
    "stone of 6 cm at 30 m": ([stone(0.0, 1.0, 0.0, 0.03)], 30.0, 0.0, 0.01),
    "stone of 9 cm at 45 m": ([stone(0.0, 1.0, 0.0, 0.045)], 45.0, 0.0, 0.01),
    "four stones at 35 m": ([stone(0.03 * k, 1.0, 0.02 * k, 0.02) for k in range(4)], 35.0, 0.0, 0.01),
    "leaf in a breeze": ([LEAF], 12.0, 0.6, 0.05),
    "leaf in a storm": ([LEAF], 12.0, 7.0, 0.05),
    "twig, leaf and stone in a storm": ([wood((0.0, 0.9, 0.0), (0.0, 1.0, 0.0), 0.02, 0.01), LEAF, stone(0.1, 0.95, 0.1, 0.03)], 8.0, 9.0, 0.08),
}


class Records:
    def __init__(self, records, n=1):
        P = np.zeros((n, CAPACITY, 24), np.float32)
        P[:, :, 3] = -1.0
        for k, rec in enumerate(records):
            P[:, k] = rec
        self.P, self.Nodes = dev(P.reshape(-1)), zeros_f(n * 65536 * 8)
        self.Order = dev(np.tile(np.arange(CAPACITY, dtype=np.uint32), n))
        for k in range(n):
            ok(ab.call("arbor_buildBounds", self.P[k * CAPACITY * 24:], self.Order[k * CAPACITY:], self.Nodes[k * 65536 * 8:]))


def camera(w, h, at, distance, angle, wind, shadows):
    C = workloads.base_state(7, w, h)
    C[4:7] = at
    C[0:3] = (at[0] + 0.6 * distance, at[1] + 0.5 * distance, at[2] + math.sqrt(0.39) * distance)
    C[14] = angle
    C[8], C[11], C[22] = 3.25, wind, 1.0 if shadows else 0.0
    C[9], C[10] = 0.0, 1.0
    return dev(C)


def forest_point(local, tree=171):
    """World position of a point near the trunk of an instance of world seed
    7's forest (the yaw of its few centimetres aside)."""
    i = Oracle("port").forest_instance(tree, 7)
    return float(i[0]), float(i[3]) * local[1], float(i[2])


def images(w, h):
    return {k: torch.full((w * h * 4,), float("nan"), device="cuda") for k in ("Hit", "Linear", "Guide")}


def same(a, b, w, h):
    for name in ("Hit", "Linear", "Guide"):
        x, y = host(a[name]).reshape(-1, 4), host(b[name]).reshape(-1, 4)
        assert np.isfinite(x).all(), f"{name}: {int((~np.isfinite(x)).any(1).sum())} pixels not written"
        n = int((x.view(np.uint32) != y.view(np.uint32)).any(1).sum())
        assert n == 0, f"{name}: {n} of {w * h} pixels differ"


@pytest.mark.parametrize("shadows", [False, True])
@pytest.mark.parametrize("single", [True, False])
@pytest.mark.parametrize("name", list(SCENES))
def test_few_records(cuda, name, single, shadows):
    records, distance, wind, angle = SCENES[name]
    w, h = 97, 61
    s = Records(records)
    at = (0.05, 1.0, 0.0) if records[0] is LEAF else tuple(records[0][0:3])
    if not single:  # from outside the instance's bounding sphere, within which the ground hides the tree (Arbor.cu:246)
        at, angle, distance = forest_point(at), 1.2 * angle, max(distance, 9.0)
    C = camera(w, h, at, distance, angle, wind, shadows)
    a, b = images(w, h), images(w, h)
    form = "Tree" if single else ""
    ok(ab.call(f"arbor_trace{form}Pixels", s.P, s.Nodes, s.Order, C, a["Hit"], w, h))
    ok(ab.call(f"arbor_shade{form}Pixels", s.P, s.Nodes, s.Order, C, a["Hit"], a["Linear"], a["Guide"], w, h))
    ok(ab.call("arbor_tracePixelsInOrder", s.P, s.Nodes, s.Order, C, b["Hit"], w, h, int(single)))
    ok(ab.call("arbor_shadePixelsInOrder", s.P, s.Nodes, s.Order, C, a["Hit"], b["Linear"], b["Guide"], w, h, int(single)))
    assert int((host(b["Hit"]).reshape(-1, 4)[:, 1] >= 0).sum()) >= 5, "the scene is in view"
    same(a, b, w, h)


def test_few_records_of_several_species(cuda):
    w, h = 97, 61
    records, distance, wind, _ = SCENES["twig, leaf and stone in a storm"]
    s, n = Records(records, 3), 3
    C = camera(w, h, forest_point((0.0, 1.0, 0.0)), distance, 0.12, wind, True)
    of = (ctypes.c_int * 324)(*[t % n for t in range(324)])
    a, b = images(w, h), images(w, h)
    ok(ab.call("arbor_traceSpeciesPixels", s.P, s.Nodes, s.Order, n, of, C, a["Hit"], w, h))
    ok(ab.call("arbor_shadeSpeciesPixels", s.P, s.Nodes, s.Order, n, of, C, a["Hit"], a["Linear"], a["Guide"], w, h))
    ok(ab.call("arbor_tracePixelsInOrder", s.P, s.Nodes, s.Order, C, b["Hit"], w, h, 0))
    ok(ab.call("arbor_shadePixelsInOrder", s.P, s.Nodes, s.Order, C, a["Hit"], b["Linear"], b["Guide"], w, h, 0))
    assert int((host(b["Hit"]).reshape(-1, 4)[:, 1] >= 0).sum()) >= 5, "the scene is in view"
    same(a, b, w, h)
