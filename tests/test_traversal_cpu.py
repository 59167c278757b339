"""The batched traversal's device code on the CPU (tests/emu) against the
reference's traversal as written, on scenes that no seed grows: a few records
that are small beside the viewing distance, leaves wider than they are long,
boxes that are inside out.

Bars: no load outside a scene's buffers, and the same hit (t, record and tree)
bit for bit.  The scenes have no two surfaces close enough along a ray for the
order of the tests to matter (one that rounding puts before its own box with
another between the two), so nothing else may differ.
"""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "arbor-cuda_b200", "csrc")
CAPACITY, NODE_COUNT, FAR = 32768, 65536, 100000.0


def _p(a):
    return None if a is None else a.ctypes.data_as(ctypes.c_void_p)


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    gxx, nvcc = shutil.which("g++"), shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    out = str(tmp_path_factory.mktemp("emu") / "traversal.so")
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I", include, "-I", CSRC,
                    os.path.join(HERE, "emu", "traversal.cpp"), "-o", out], check=True)
    lib = ctypes.CDLL(out)
    lib.emu_boxes.restype = lib.emu_trace.restype = lib.emu_loads.restype = ctypes.c_long
    return lib


class Scene:
    """Records in places 0 .. n - 1 of P (the rest unused), Nodes as
    arbor_buildBounds makes them."""

    def __init__(self, emu, records):
        self.emu = emu
        P = np.zeros((CAPACITY, 24), np.float32)
        P[:, 3] = -1.0
        for k, rec in enumerate(records):
            P[k] = rec
        self.P, self.Order = P.reshape(-1), np.arange(CAPACITY, dtype=np.uint32)
        self.Nodes = np.zeros(NODE_COUNT * 8, np.float32)
        emu.emu_leaf_nodes(_p(self.P), _p(self.Order), _p(self.Nodes))
        self.T = np.zeros(emu.emu_words(), np.uint32)
        assert emu.emu_boxes(_p(self.P), _p(self.Order), _p(self.Nodes), _p(self.T)) == 0

    def both(self, rays, wind=0.0, refine=True, inst=None, cone=1.0e-3, time=3.25, against="emu_reference"):
        """(t, id, tree) of every ray from the block batch and from the
        reference's traversal (or another); checks that no load left the
        buffers."""
        rays = np.ascontiguousarray(rays, np.float32)
        n, f = len(rays), ctypes.c_float
        got, want = np.full((n, 3), np.nan, np.float32), np.full((n, 3), np.nan, np.float32)
        regular = ctypes.c_int(-1)
        bad = self.emu.emu_trace(_p(self.P), _p(self.Order), _p(self.Nodes), _p(self.T), _p(inst), _p(rays), n, f(cone), f(time), f(wind),
                                 int(refine), _p(got), ctypes.byref(regular))
        getattr(self.emu, against)(_p(self.P), _p(self.Order), _p(self.Nodes), _p(inst), _p(rays), n, f(cone), f(time), f(wind), int(refine),
                                   _p(want))
        assert bad == 0, f"{bad} loads outside the scene's buffers"
        return got, want, regular.value


def same(got, want):
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), f"{(got != want).any(1).sum()} of {len(got)} rays differ"


def stone(x, y, z, a, b=None, c=None):
    r = np.zeros(24, np.float32)
    r[0:4], r[4:7] = (x, y, z, 2.0), (a, b or a, c or a)
    r[15] = 5.0
    return r


def wood(a, b, ra, rb):
    r = np.zeros(24, np.float32)
    r[0:3], r[3], r[4:7], r[7] = a, 0.0, b, ra
    r[8:11], r[11], r[15], r[18] = (0.0, 0.0, 1.0), rb, 11.0, ra
    return r


def leaf(x, y, z, length, width, stem=0.03, curl=0.02, twist=0.03, frame=((1, 0, 0), (0, 0, 1), (0, 1, 0))):
    r = np.zeros(24, np.float32)
    r[0:4], r[4:7], r[7] = (x, y, z, 1.0), frame[0], length
    r[8:11], r[11], r[12:15], r[15] = frame[1], width, frame[2], 9.0
    r[16:19] = stem, curl, twist
    return r


def rays_at(target, spread, distance, n, seed, best=FAR):
    """n rays from points `distance` away toward points within `spread` of the
    target."""
    r = np.random.RandomState(seed)
    d = r.standard_normal((n, 3))
    d[:, 1] = np.abs(d[:, 1]) + 0.3
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o = np.asarray(target) + distance * d
    at = np.asarray(target) + spread * (2.0 * r.random((n, 3)) - 1.0)
    v = at - o
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    return np.concatenate([o, v, np.full((n, 1), best)], 1)


# The scene of the far cases: 2 m high, a few surfaces far apart.
FAR_SCENE = [wood((0.0, 0.0, 0.0), (0.0, 2.0, 0.0), 0.1, 0.05), leaf(0.3, 1.5, 0.2, 0.2, 0.08), stone(-0.6, 0.2, 0.5, 0.3)]


@pytest.mark.parametrize("wind", [0.0, 0.6, 6.0])
@pytest.mark.parametrize("distance", [5.0, 60.0, 90.0, 400.0])
def test_single_tree_rays_that_miss_keep_their_distance(emu, distance, wind):
    """Beyond the tight boxes' line the pruning distance holds a slack; a ray
    that enters the root's box and meets nothing returns the distance it came
    with (the ground's, or the sky's), not one with the slack added."""
    s = Scene(emu, FAR_SCENE)
    rays = rays_at((0.0, 1.0, 0.0), 1.0, distance, 128, 4)
    rays[::2, 6] = distance + 30.0
    got, want, _ = s.both(rays, wind=wind)
    assert (want[:, 1] < 0).sum() >= 20 and (want[:, 1] >= 0).sum() >= 10
    same(got, want)


SMALL = {
    "stone of 1 cm at 5 m": ([stone(0.3, 0.5, -0.2, 0.005)], 5.0, 0.004),
    "stone of 9 cm at 45 m": ([stone(0.3, 0.5, -0.2, 0.045)], 45.0, 0.04),
    "stone of 12 cm at 60 m": ([stone(0.3, 0.5, -0.2, 0.06)], 60.0, 0.05),
    "four stones at 35 m": ([stone(0.03 * k, 0.5, 0.02 * k, 0.02) for k in range(4)], 35.0, 0.05),
    "twig and leaf at 75 m": ([wood((0.0, 0.5, 0.0), (0.0, 0.6, 0.0), 0.02, 0.01), leaf(0.0, 0.6, 0.0, 0.1, 0.04)], 75.0, 0.05),
}


@pytest.mark.parametrize("name", list(SMALL))
@pytest.mark.parametrize("refine", [True, False])
def test_small_scene_far_away(emu, name, refine):
    """The margin by which the boxes are widened is as large as the scene."""
    records, distance, spread = SMALL[name]
    s = Scene(emu, records)
    got, want, _ = s.both(rays_at(records[0][0:3], spread, distance, 96, 1), refine=refine)
    assert (want[:, 1] >= 0).sum() >= 10
    same(got, want)


@pytest.mark.parametrize("wind", [0.6, 7.0, 40.0])
def test_one_leaf_in_the_wind(emu, wind):
    """A shadow segment's margin with the leaf's swing: wider than the scene."""
    s = Scene(emu, [leaf(0.0, 1.0, 0.0, 0.15, 0.07)])
    got, want, _ = s.both(rays_at((0.1, 1.0, 0.0), 0.05, 20.0, 96, 2, best=36.0), wind=wind, refine=False)
    assert (want[:, 1] >= 0).sum() >= 10
    same(got, want)


def test_small_scene_in_a_forest(emu):
    inst = np.zeros(324 * emu.emu_instance_bytes(), np.uint8)
    emu.emu_instances(7, _p(inst))
    s = Scene(emu, [stone(0.2, 1.0, -0.1, 0.05), leaf(0.3, 1.2, 0.0, 0.1, 0.04)])
    f = inst.view(np.float32).reshape(324, -1)
    rays = [rays_at((f[t, 0], 1.0, f[t, 1]), 0.4, d, 64, t) for t, d in ((150, 12.0), (171, 40.0), (40, 70.0), (300, 25.0))]
    for refine in (True, False):
        got, want, _ = s.both(np.concatenate(rays), inst=inst, refine=refine, wind=0.6)
        assert (want[:, 1] >= 0).sum() >= 4
        same(got, want)


def test_rays_that_are_not_finite(emu):
    """Origins and directions with infinities and NaN: no load leaves the
    scene's buffers (what such a ray hits is not defined)."""
    s = Scene(emu, [stone(0.3, 0.5, -0.2, 0.045), leaf(0.0, 1.0, 0.0, 0.15, 0.07)])
    rays = rays_at((0.3, 0.5, -0.2), 0.05, 5.0, 64, 3)
    bad = [np.nan, np.inf, -np.inf, 1.0e30, 3.0e38]
    for k in range(60):
        rays[k, k % 6] = bad[k % 5]
    s.both(rays)
    s.both(rays, refine=False)


class Grown(Scene):
    """A grown scene whose Nodes, changed by `change`, are no longer the bounds
    of its records."""

    def __init__(self, emu, scene, change):
        self.emu = emu
        self.P, self.Order, self.Nodes = (np.array(scene[k]).reshape(-1) for k in ("P", "Order", "Nodes"))
        change(self.Nodes.reshape(NODE_COUNT, 8))
        self.T = np.zeros(emu.emu_words(), np.uint32)
        assert emu.emu_boxes(_p(self.P), _p(self.Order), _p(self.Nodes), _p(self.T)) == 0


def cut_leaf_boxes(N):
    N[CAPACITY:, 0:3] += 0.08 * np.random.RandomState(1).random((CAPACITY, 3)).astype(np.float32)


def pad_all(N):
    N[1:, 0:3] -= 0.01
    N[1:, 4:7] += 0.01


def empty_subtree(N):
    N[65, 3] = 0.0


@pytest.mark.parametrize("change", [cut_leaf_boxes, pad_all, empty_subtree])
@pytest.mark.parametrize("refine", [True, False])
def test_nodes_that_are_not_the_records_bounds(emu, scenes, change, refine):
    """The batch in the fixed order against one tree after another in that
    order (tree_in_order): with the leaves' boxes cut short, most hits lie
    before their own box and the order decides which one counts."""
    s = Grown(emu, scenes(7), change)
    inst = np.zeros(324 * emu.emu_instance_bytes(), np.uint8)
    emu.emu_instances(7, _p(inst))
    rays = np.concatenate([rays_at((0.0, 5.5, 0.0), 3.0, 12.0, 400, 1, best=FAR if refine else 36.0), rays_at((0.0, 3.0, 0.0), 2.0, 9.0, 400, 2)])
    rays[400:600, :3] = (0.3, 4.0, 0.2)  # from inside the crown
    for forest in (None, inst):
        got, want, regular = s.both(rays, wind=0.6, refine=refine, inst=forest, against="emu_in_order")
        assert regular == 0 and (want[:, 1] >= 0).sum() >= 60
        same(got, want)


@pytest.mark.parametrize("refine", [True, False])
def test_without_boxes(emu, scenes, refine):
    """A pass without scratch (under stream capture, above the scratch's scene
    limit): the fixed order, from the rays' own loads - no CTA looks through the
    scene first."""
    s = Grown(emu, scenes(7), lambda N: None)
    s.T = None
    rays = rays_at((0.0, 5.5, 0.0), 3.0, 12.0, 64, 5, best=FAR if refine else 36.0)
    got, want, _ = s.both(rays, refine=refine, against="emu_in_order")
    assert (want[:, 1] >= 0).sum() >= 10
    same(got, want)
    rays[:, 3:6] = (0.0, 1.0, 0.0)  # past the tree: its root's two loads a ray, no more
    rays[:, 0] = 50.0
    got, want, _ = s.both(rays, refine=refine, against="emu_in_order")
    same(got, want)
    assert emu.emu_loads() <= 2 * len(rays)


WIDE = {
    # half width far above the length: the blade reaches outside the cube that
    # bounds it in Nodes
    "wide leaf": [leaf(0.0, 1.0, 0.0, 0.1, 0.9, stem=0.0)],
    "wide leaf, turned": [leaf(0.0, 1.0, 0.0, 0.1, 0.9, stem=0.0, frame=((0.6, 0.8, 0.0), (0.0, 0.0, 1.0), (-0.8, 0.6, 0.0)))],
    "curled leaf": [leaf(0.0, 1.0, 0.0, 0.012, 0.01, stem=0.0, curl=0.06, twist=0.0)],
    "two wide leaves": [leaf(0.0, 1.0, 0.0, 0.1, 0.9, stem=0.0), leaf(0.4, 1.3, 0.2, 0.1, 0.7, stem=0.02, curl=-0.02)],
}


@pytest.mark.parametrize("wind", [0.0, 0.8])
@pytest.mark.parametrize("name", list(WIDE))
def test_leaf_that_reaches_outside_its_box(emu, name, wind):
    """A ray that passes the leaf's box in Nodes and meets the blade outside it
    has a hit."""
    s = Scene(emu, WIDE[name])
    rays = np.concatenate([rays_at((0.0, 1.0, 0.0), r, d, 128, k) for k, (r, d) in enumerate(((0.02, 4.0), (0.08, 4.0), (0.4, 6.0), (0.12, 1.5)))])
    rays[1::2, 1] -= 2.0 * (rays[1::2, 1] - 1.0) * 0.93  # half of them nearly along the blade
    v = np.array([0.0, 1.0, 0.0]) + 0.06 * (np.random.RandomState(8).random((len(rays), 3)) - 0.5) - rays[:, :3]
    rays[1::2, 3:6] = (v / np.linalg.norm(v, axis=1, keepdims=True))[1::2]
    for refine in (True, False):
        got, want, _ = s.both(rays, wind=wind, refine=refine, against="emu_in_order")
        assert (want[:, 1] >= 0).sum() >= 10
        same(got, want)


def test_record_whose_box_is_inside_out(emu):
    """A stone with a negative half-axis, wood with negative radii: their boxes
    in Nodes are inside out, and the slab test takes them as they are."""
    s = Scene(emu, [stone(0.0, 1.0, 0.0, 0.2, -0.2, 0.2), stone(1.0, 1.0, 0.0, 0.2), wood((0.5, 0.5, 0.0), (0.5, 0.9, 0.1), -0.1, -0.1)])
    for refine in (True, False):
        got, want, _ = s.both(np.concatenate([rays_at((0.0, 1.0, 0.0), 0.3, 5.0, 128, 1), rays_at((0.6, 0.8, 0.0), 0.5, 5.0, 128, 2)]), refine=refine)
        assert (want[:, 1] == 0).sum() >= 10
        same(got, want)

@pytest.mark.parametrize("kind", ["skewed frame", "negative length", "not a number", "unknown type"])
def test_records_without_a_bound(emu, kind):
    """Records whose surface their box says nothing about, among sound ones."""
    odd = leaf(0.0, 1.0, 0.0, 0.15, 0.07)
    if kind == "skewed frame":
        odd[4:7] = (0.5, 0.0, 0.0)
    elif kind == "negative length":
        odd[7] = -0.1
    elif kind == "not a number":
        odd[17] = np.nan
    else:
        odd = stone(0.0, 1.0, 0.0, 0.3)
        odd[3], odd[7] = 3.0, 0.05
    s = Scene(emu, [odd, stone(0.1, 1.05, 0.1, 0.05), leaf(0.05, 1.1, -0.05, 0.15, 0.07)])
    for refine in (True, False):
        got, want, _ = s.both(np.concatenate([rays_at((0.05, 1.0, 0.0), 0.15, 5.0, 192, 1), rays_at((0.1, 1.0, 0.0), 0.1, 3.0, 192, 2)]),
                              refine=refine, against="emu_in_order")
        assert (want[:, 1] >= 0).sum() >= 10
        same(got, want)


def test_grown_scenes_keep_their_tight_boxes(emu, scenes):
    s = Grown(emu, scenes(7), lambda N: None)
    _, _, regular = s.both(rays_at((0.0, 5.5, 0.0), 3.0, 12.0, 32, 5))
    assert regular == 1


@pytest.mark.parametrize("distance", [5.0, 90.0])
def test_ground_beyond_the_farthest_distance(emu, distance):
    """Rays just below the horizon meet the ground beyond t = 100000.  One that
    enters the single tree's root and passes every leaf box keeps that distance;
    one that meets a leaf box and misses the surface has the miss, at 100000
    (Arbor.cu:226)."""
    s = Scene(emu, FAR_SCENE)
    rays = rays_at((0.0, 1.0, 0.0), 1.0, distance, 256, 6)
    rays[:, 6] = np.linspace(9.0e4, 4.0e5, 256)
    for wind in (0.0, 6.0):
        got, want, _ = s.both(rays, wind=wind)
        assert (want[:, 0] > FAR).sum() >= 20 and ((want[:, 0] == FAR) & (want[:, 1] >= 0)).sum() >= 5
        same(got, want)


@pytest.mark.parametrize("distance", [9.0e4, 1.2e5, 3.0e5])
def test_surfaces_beyond_the_farthest_distance(emu, distance):
    """A scene 4 km across, farther away than t = 100000, before a ground that
    is farther still: its hits lie beyond the tests' "no hit" value."""
    s = Scene(emu, [stone(0.0, 500.0, 0.0, 2000.0), stone(1500.0, 900.0, 0.0, 900.0)])
    rays = rays_at((0.0, 500.0, 0.0), 2500.0, distance, 128, 7)
    rays[:, 6] = np.where(np.arange(128) % 2, FAR, distance + 1.0e5)
    for refine in (True, False):
        got, want, _ = s.both(rays, refine=refine, against="emu_in_order")
        assert (want[:, 1] >= 0).sum() >= 10
        same(got, want)


@pytest.mark.parametrize("kind", ["petioles", "wood"])
@pytest.mark.parametrize("refine", [True, False])
def test_steep_tapers(emu, kind, refine):
    """Petioles a hundredth as long as they are thick, wood whose radius falls
    faster than it is long: the cone's test reports hits far off the surface,
    and they count as they do in the fixed order."""
    r = np.random.RandomState(11)
    recs = []
    for _ in range(120):
        p = 0.06 * (r.random(3) - 0.5) + (0.0, 0.06, 0.0)
        if kind == "petioles":
            u, v, w = (x / np.linalg.norm(x) for x in np.linalg.qr(r.standard_normal((3, 3)))[0].T)
            recs.append(leaf(*p, 1.0e-3, 4.0e-4, stem=10.0 ** r.uniform(-5.5, -4.0), curl=1.0e-4, twist=0.1, frame=(u, v, w)))
        else:
            recs.append(wood(p, p + 1.0e-4 * r.standard_normal(3), 3.0e-3, 1.0e-3))
    s = Scene(emu, recs)
    got, want, _ = s.both(rays_at((0.0, 0.06, 0.0), 0.03, 6.0, 800, 12, best=FAR if refine else 36.0), refine=refine, against="emu_in_order")
    assert (want[:, 1] >= 0).sum() >= 50
    same(got, want)


def scaled(emu, scene, scale):
    """A grown scene with every length times `scale`."""
    s = Grown(emu, scene, lambda N: None)
    P = s.P.reshape(CAPACITY, 24)
    kind = P[:, 3].copy()
    P[:, [0, 1, 2, 7, 11]] *= np.float32(scale)
    P[kind != 1, 4:7] *= np.float32(scale)
    P[kind == 1, 16:18] *= np.float32(scale)
    P[kind == 0, 16] *= np.float32(scale)
    P[kind == 0, 18] *= np.float32(scale)
    emu.emu_leaf_nodes(_p(s.P), _p(s.Order), _p(s.Nodes))
    assert emu.emu_boxes(_p(s.P), _p(s.Order), _p(s.Nodes), _p(s.T)) == 0
    return s


@pytest.mark.parametrize("scale", [1.0, 0.1])
def test_small_trees_far_away_are_not_searched_whole(emu, scenes, scale):
    """A grown tree, and one a tenth as large, from as far as the margin is wide
    beside a leaf: the loads stay below twice the fixed order's, which tests the
    boxes of Nodes (a tenth as large, tight boxes widened by three leaves: 3
    times)."""
    s = scaled(emu, scenes(7), scale)
    rays = rays_at((0.0, 5.5 * scale, 0.0), 3.0 * scale, 70.0, 200, 1)
    got, want, regular = s.both(rays, against="emu_in_order")
    batch = emu.emu_loads()
    same(got, want)
    s.T = None
    s.both(rays, against="emu_in_order")
    print(f"[scale {scale}] {batch} loads, in order {emu.emu_loads()}")
    assert regular == 1 and batch < 2 * emu.emu_loads()


@pytest.mark.parametrize("scale,wind,distance,boxes", [
    (1.0, 0.0, None, 1), (1.0, 0.6, None, 1), (1.0, 3.0, None, 1), (1.0, 8.0, None, 0), (0.5, 0.0, None, 1), (0.2, 0.0, None, 0),
    (1.0, 0.0, 3.0, 1), (1.0, 0.0, 300.0, 1), (1.0, 8.0, 3.0, 1), (1.0, 8.0, 300.0, 0), (1.0, 0.0, 600.0, 0),
    (0.2, 0.0, 3.0, 1), (0.2, 3.0, 10.0, 1), (0.2, 0.0, 300.0, 0), (0.1, 0.0, 30.0, 1), (0.1, 0.0, 100.0, 0)])
def test_what_primary_rays_traverse(emu, scenes, scale, wind, distance, boxes):
    """The faster of tight boxes and fixed order, as measured (tight.cuh), for a
    forest (distance None) and the single tree."""
    s = scaled(emu, scenes(7), scale)
    eye = None if distance is None else np.array([0.0, 5.0 * scale, distance], np.float32)
    assert emu.emu_primary_takes_boxes(_p(s.T), ctypes.c_float(wind), _p(eye)) == boxes


@pytest.mark.parametrize("leaves,wind,boxes", [(1, 0.0, 1), (1, 0.6, 1), (1, -2.0, 1), (1, 3.0, 0), (1, -8.0, 0), (1, float("inf"), 0),
                                               (1, float("nan"), 0), (0, 8.0, 1)])
def test_what_shadow_segments_traverse(emu, leaves, wind, boxes):
    """The faster of tight boxes and fixed order, as measured (tight.cuh): the
    boxes in a breeze, or where nothing swings."""
    s = Scene(emu, [stone(0.0, 1.0, 0.0, 0.3), leaf(0.0, 1.0, 0.0, 0.15, 0.07) if leaves else stone(0.2, 1.0, 0.0, 0.1)])
    assert emu.emu_shadow_takes_boxes(_p(s.T), ctypes.c_float(wind)) == boxes
