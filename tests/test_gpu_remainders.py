"""Images of one pixel, of one 8x4 block and of parts of blocks: every pixel is
written, and is the one of the reference's traversal as written.  Bar: bit for
bit (a tree whose answer depends on the order is one pixel in about a million)."""
import pytest

import arbor_b200 as ab
import workloads
from gpu_util import dev, ok
from test_gpu_small_scenes import images, same
from test_gpu_tight import Scene, state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("wind", [0.0, 0.6])
@pytest.mark.parametrize("w,h", [(1, 1), (7, 5), (8, 4), (9, 33), (33, 17), (5, 130)])
def test_parts_of_blocks(cuda, w, h, wind, single):
    s, C = Scene([7]), state(w, h, wind=wind)
    if single:
        C = workloads.single_tree_camera(w, h, 7)
        C[8], C[11], C[22] = 3.25, wind, 1.0
    C = dev(C)
    a, b, form = images(w, h), images(w, h), "Tree" if single else ""
    ok(ab.call(f"arbor_trace{form}Pixels", s.P, s.Nodes, s.Order, C, a["Hit"], w, h))
    ok(ab.call(f"arbor_shade{form}Pixels", s.P, s.Nodes, s.Order, C, a["Hit"], a["Linear"], a["Guide"], w, h))
    ok(ab.call("arbor_tracePixelsInOrder", s.P, s.Nodes, s.Order, C, b["Hit"], w, h, int(single)))
    ok(ab.call("arbor_shadePixelsInOrder", s.P, s.Nodes, s.Order, C, b["Hit"], b["Linear"], b["Guide"], w, h, int(single)))
    same(a, b, w, h)
