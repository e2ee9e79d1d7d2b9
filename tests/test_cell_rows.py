"""The point-per-thread kernel's per-cell nodal sums at the sizes where they
can go wrong, against the oracle: items of one point, of a full and an
overfull bin, cells of many points, windows that are wide along every axis,
points that drift out of their item's tile, corners on the upper face of the
domain and point-sampled maps. Tolerances are the forms' own: 1e-10 per field
and step in FP64 (summation order only), 1e-4 in the mixed form."""
import numpy as np
import pytest

import bridge
from mpm_3d_b200 import inputs
from mpm_3d_b200.native import GPUBatch, GPUExplicitUSL
from util import FP64_TOL, assert_close, field_floor

pytestmark = pytest.mark.gpu

N = 16
H = 1.0 / N


@pytest.fixture(scope="module", autouse=True)
def restated_lib():
    bridge.build_restated()


def _cloud(x, v=(0.0, 0.0, 0.0), spin=2.0, E=1e4, dt=1e-4):
    """A body of the given positions with a velocity gradient, on an N^3 grid."""
    x = np.asarray(x, np.float64)
    n = x.shape[0]
    vol = (H / 2) ** 3
    xt = np.asarray(v) + (x - x.mean(0)) @ (spin * np.array([[0.3, -1.0, 0.2], [1.0, -0.2, 0.5], [-0.4, 0.1, 0.6]]))
    body = inputs.Body("cloud", np.full(n, 1000.0 * vol), np.full(n, vol), x, xt, np.ones(n, np.int32), E=E)
    return inputs.Case("cloud", 3, (1.0,) * 3, (N,) * 3, dt, 8, [body])


def _random(n, lo, hi, seed):
    return np.random.default_rng(seed).uniform(np.asarray(lo) * H, np.asarray(hi) * H, (n, 3))


def _faces():
    """Points whose upper corner lies on the domain's upper face, whose
    corners leave the domain (point-sampled), and ordinary ones beside them."""
    a = 0.25 * np.cbrt((H / 2) ** 3)   # half the extent
    x = _random(60, (12.3, 12.3, 12.3), (15.6, 15.6, 15.6), 5)
    x[:10, 0] = 1.0 - a
    x[10:20, 2] = 1.0 - 0.3 * a
    x[20:30, 1] = 1.0 - 0.1 * H * 0.3
    return x


CLOUDS = {
    "one_point": lambda: _cloud([[4.4 * H, 5.3 * H, 6.7 * H]], spin=0.0),
    "two_bins_33": lambda: _cloud(_random(33, (3.2, 4.1, 4.1), (4.9, 7.9, 7.9), 1)),
    "full_bin_512": lambda: _cloud(_random(512, (4.2, 4.2, 4.2), (7.8, 7.8, 7.8), 2)),
    "overfull_bin_1025": lambda: _cloud(_random(1025, (4.2, 4.2, 4.2), (7.8, 7.8, 7.8), 3)),
    "one_cell_300": lambda: _cloud(_random(300, (5.2, 5.2, 5.2), (5.8, 5.8, 5.8), 4)),
    "all_wide": lambda: _cloud(np.round(_random(200, (3.6, 3.6, 3.6), (9.4, 9.4, 9.4), 6) / H) * H + 0.01 * H),
    "faces": lambda: _cloud(_faces(), spin=0.5),
    "drift": lambda: _cloud(_random(400, (3.1, 3.1, 3.1), (6.9, 6.9, 6.9), 7), v=(0.45 * H / 1e-4, 0.3 * H / 1e-4, 0.0)),
    "drift_down": lambda: _cloud(_random(400, (8.1, 8.1, 8.1), (11.9, 11.9, 11.9), 8),
                                 v=(0.0, -0.4 * H / 1e-4, -0.4 * H / 1e-4)),
}


@pytest.mark.parametrize("cap", [128, 256, 512])
@pytest.mark.parametrize("name", sorted(CLOUDS))
def test_cell_sums(name, cap):
    case = CLOUDS[name]()
    gpu = GPUExplicitUSL(case, keep_debug=True, kernel=("point_per_thread", cap))
    ref = bridge.RestatedJob(case)
    for s in range(6):
        gpu.step(1)
        ref.step(1)
        for f in ("x", "x_t", "T", "v"):
            assert_close(gpu.points(0, f), ref.points(0, f), FP64_TOL, f"{name} step {s} {f}", field_floor(case, f))
        assert_close(gpu.nodes(0, "m"), ref.nodes(0, "m"), FP64_TOL, f"{name} step {s} nodal m")
    gpu.synchronize()
    gpu.close()


# "faces" places corners exactly on the upper face (the extent, H / 4, is an
# FP32 number too): such a corner has no element, so the point's weights sum to
# one half, and the reference velocity that the mixed form gathers against
# must go by that sum. Each kernel form has its own gather.
@pytest.mark.parametrize("kernel", [("point_per_thread", 128), ("point_per_thread", 512), ("staged", 512)],
                         ids=lambda k: f"{k[0]}{k[1]}")
@pytest.mark.parametrize("name", sorted(CLOUDS))
def test_cell_sums_mixed(name, kernel):
    case = CLOUDS[name]()
    gpu = GPUExplicitUSL(case, mode="mixed", kernel=kernel)
    ref = bridge.RestatedJob(case)
    gpu.step(6)
    ref.step(6)
    for f in ("x", "x_t", "T"):
        assert_close(gpu.points(0, f), ref.points(0, f), 1e-4, f"{name} {f}", field_floor(case, f))
    gpu.close()


# The same clouds as the first body of a contact (contact normals, the second
# body close by or out of reach) and, over the body table, as jobs of a batch of
# seven bodies with and without contact: the items of one kind are passed over
# by the other kind's launch, and tiles are loaded ahead across bodies.
def _with_contact(name):
    case = CLOUDS[name]()
    rng = np.random.default_rng(31)
    x = np.clip(case.bodies[0].x[:64] + rng.uniform(-0.4, 0.4, (min(64, case.bodies[0].n), 3)) * H, 0.05, 0.95)
    n, vol = len(x), (H / 2) ** 3
    other = inputs.Body("other", np.full(n, 1000.0 * vol), np.full(n, vol), x, -case.bodies[0].x_t[:n],
                        np.ones(n, np.int32), E=1e4)
    case.bodies.append(other)
    case.contacts.append(inputs.Contact(0, 1, 0.3))
    return case


# "one_point" is left out: a lone pair's contact normal divides two sums of
# rounding size, which no two orders agree on
@pytest.mark.parametrize("cap", [128, 512])
@pytest.mark.parametrize("name", sorted(set(CLOUDS) - {"one_point"}))
def test_cell_sums_in_contact_and_over_the_table(name, cap):
    both, alone = _with_contact(name), CLOUDS[name]()
    cases = [both, alone, both, CLOUDS["drift_down"](), alone]
    batch = GPUBatch(dim=3, mode="fp64", kernel=("point_per_thread", cap))
    ids = [batch.add(c, steps=4) for c in cases]
    solo = GPUExplicitUSL(both, kernel=("point_per_thread", cap))
    refs = {id(c): bridge.RestatedJob(c) for c in (both, alone, cases[3])}
    batch.step(4)
    solo.step(4)
    for ref in refs.values():
        ref.step(4)
    for f in ("x", "x_t", "T", "v"):
        for b in range(2):
            assert_close(solo.points(b, f), refs[id(both)].points(b, f), 4 * FP64_TOL, f"{name} contact body {b} {f}",
                         field_floor(both, f))
        for j, c in zip(ids, cases):
            for b in range(len(c.bodies)):
                assert_close(batch.points(j, b, f), refs[id(c)].points(b, f), 4 * FP64_TOL, f"{name} job {j} body {b} {f}",
                             field_floor(c, f))
    solo.close()
    batch.close()


# Both grid updates: from the flags (up to 16,384 node blocks) and from the list
# of active blocks (above), in 2D (blocks of 8 x 8 nodes) and 3D (4 x 4 x 4).
@pytest.mark.parametrize("dim,n", [(2, 1016), (2, 1040), (3, 96), (3, 104)])
def test_grid_update_on_either_side_of_the_block_limit(dim, n):
    h = 1.0 / n
    rng = np.random.default_rng(41)
    x, v = np.zeros((3000, 3)), np.zeros((3000, 3))
    x[:, :dim] = 0.5 + rng.uniform(-12, 12, (3000, dim)) * h
    v[:, :dim] = rng.uniform(-1.0, 1.0, (3000, dim))
    vol = (h / 2) ** dim
    body = inputs.Body("cloud", np.full(3000, 1000.0 * vol), np.full(3000, vol), x, v, np.ones(3000, np.int32), E=1e4)
    case = inputs.Case("cloud", dim, (1.0,) * dim, (n,) * dim, 1e-6, 4, [body])
    blocks = ((n + 1 + 7) // 8) ** 2 if dim == 2 else ((n + 1 + 3) // 4) ** 3
    assert (blocks <= 16384) == (n in (1016, 96))
    gpu = GPUExplicitUSL(case, keep_debug=True)
    ref = bridge.RestatedJob(case)
    for s in range(4):
        gpu.step(1)
        ref.step(1)
        for f in ("x", "x_t", "T", "v"):
            assert_close(gpu.points(0, f), ref.points(0, f), (s + 1) * FP64_TOL, f"step {s} {f}", field_floor(case, f))
    m = ref.nodes(0, "m")
    assert_close(gpu.nodes(0, "m"), m, FP64_TOL, "nodal m")
    assert gpu.active_nodes()[0] == int((m > 0).sum())
    gpu.close()


def _on_nodes(nodes, cpdi):
    """A body on a 20^3 grid whose h has no exact binary form: a cloud, and in
    it points whose x coordinate (cpdi 0) or lower corner in x (cpdi 1) is
    h * i, which is on node i up to the rounding of the product."""
    n, h = 20, 1.0 / 20
    vol = (h / 2) ** 3
    half = 0.25 * np.cbrt(vol)
    rng = np.random.default_rng(21)
    x = rng.uniform(0.11, 0.89, (2000, 3))
    for k, i in enumerate(nodes):
        x[8 * k:8 * k + 8, 0] = h * i + (half if cpdi else 0.0)
    x_t = (x - 0.5) @ np.array([[0.3, -1.0, 0.2], [1.0, -0.2, 0.5], [-0.4, 0.1, 0.6]])
    body = inputs.Body("nodes", np.full(2000, 1000.0 * vol), np.full(2000, vol), x, x_t, np.ones(2000, np.int32), E=1e4)
    return inputs.Case("nodes", 3, (1.0,) * 3, (n,) * 3, 1e-5, 8, [body], cpdi=cpdi)


# The offset of such a point from its node is rounding, and the sampled map's
# gradient follows its sign (1/h or -1/h) and is 0/0 where it is zero: both
# kernel forms must take it alike. Formed as (x - h i) / h it is zero at nodes
# 4, 8 and 16 and negative at 9, 13 and 18; formed as x N / L - i it is positive
# at all six. The same nodal sums in another order: 1e-10 in FP64, 1e-4 in the
# mixed form.
@pytest.mark.parametrize("mode,tol", [("fp64", FP64_TOL), ("mixed", 1e-4)])
@pytest.mark.parametrize("nodes,cpdi", [((9, 13, 18), 0), ((4, 8, 16), 0), ((5, 10, 15), 0),
                                        ((4, 5, 8, 9, 10, 13, 15, 16), 1)])
def test_points_on_nodes_as_in_the_staged_kernel(nodes, cpdi, mode, tol):
    case = _on_nodes(nodes, cpdi)
    runs = []
    for kernel in (("staged", 512), ("point_per_thread", 512), ("point_per_thread", 128)):
        gpu = GPUExplicitUSL(case, mode=mode, kernel=kernel)
        gpu.step(1)
        runs.append(([gpu.points(0, f) for f in ("x", "x_t", "v", "T")], gpu.active_nodes()[0]))
        gpu.close()
    for got, active in runs[1:]:
        assert active == runs[0][1], "nodes with mass"
        for f, g, r in zip(("x", "x_t", "v", "T"), got, runs[0][0]):
            assert np.array_equal(np.isnan(g), np.isnan(r)), f"{f}: NaN at other points"
            assert_close(np.nan_to_num(g), np.nan_to_num(r), tol, f, field_floor(case, f))


@pytest.mark.parametrize("name", sorted(CLOUDS))
def test_drift_is_counted_as_in_the_staged_kernel(name):
    """mpmgpu_active_nodes: visits that found a point outside its bin's tile.
    Points that take the general path for another reason (corners on the upper
    face) are none, and the two kernel forms share the bins."""
    counts = []
    for kernel in (("staged", 512), ("point_per_thread", 512), ("point_per_thread", 128)):
        gpu = GPUExplicitUSL(CLOUDS[name](), kernel=kernel)
        gpu.step(6)
        counts.append(gpu.active_nodes()[1])
        gpu.close()
    assert counts[1:] == counts[:1] * 2
    assert (counts[0] > 0) == name.startswith("drift")
