"""kami_sdf_bake on the GPU against the FP64 oracle bake, and a baked head driving the solver's
SDF pass."""
import numpy as np
import pytest

from kamisimulator_b200 import synth, vbd
from oracle import oracle as orc
from tests import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", ["icosphere", "torus"])
def test_gpu_bake_matches_the_oracle(mesh):
    V, T = synth.icosphere(4) if mesh == "icosphere" else synth.torus(0.06, 0.025, 48, 24)
    lo, hi = synth.mesh_bounds(V)
    pad = 0.15 * (np.asarray(hi) - np.asarray(lo))
    lo, hi = tuple(np.asarray(lo) - pad), tuple(np.asarray(hi) + pad)
    dims = (33, 40, 28)
    g = vbd.bake_sdf(V, T, dims, lo, hi)
    phi, grad = orc.sdf_bake(V, T, dims, g.grid_min, g.grid_max)
    assert np.abs(g.phi - phi).max() <= 2e-6
    clear = np.abs(phi) > 1e-5
    np.testing.assert_array_equal(np.sign(g.phi[clear]), np.sign(phi[clear]))
    # outside: the radial rule, deterministic
    out = phi > 1e-4
    assert np.abs(g.grad - grad)[out].max() <= 1e-5
    # inside: near the medial axis several triangles tie within float precision and the nearest
    # point is not unique, so check the property instead: x - phi * grad is a nearest surface point
    inside = phi < -1e-4
    nx, ny, nz = dims
    ds = (np.asarray(g.grid_max, np.float64) - np.asarray(g.grid_min, np.float64)) / np.asarray(dims)
    iz, iy, ix = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    x = np.stack([g.grid_min[0] + ds[0] * ix, g.grid_min[1] + ds[1] * iy, g.grid_min[2] + ds[2] * iz], -1)
    cp = x[inside] - g.phi[inside][:, None] * g.grad[inside]
    assert np.abs(orc.sdf_points(V, T, cp)).max() <= 1e-5
    np.testing.assert_allclose(np.linalg.norm(g.grad[inside], axis=-1), 1.0, atol=1e-5)


def test_baked_head_drives_the_solver_like_the_analytic_sphere():
    """Strands starting 2 mm inside a head: one step with the grid baked from an icosphere mesh
    against the same step with the analytic sphere sampled on the same nodes (synth.sphere_sdf).
    They differ by the mesh's tessellation (an inscribed icosphere of 2,562 vertices sits up to
    ~0.1 mm inside the sphere), and the solver agrees with the oracle on the baked grid."""
    V, T = synth.icosphere(4, radius=0.09)
    baked = vbd.bake_sdf(V, T, (96, 96, 96), (-0.12,) * 3, (0.12,) * 3, threshold=1e-3)
    analytic = synth.sphere_sdf(96, radius=0.09, half_extent=0.12, threshold=1e-3)
    assert np.abs(baked.phi - analytic.phi).max() <= 2e-4
    g = synth.groom(200, 24, seed=3)
    r = np.linalg.norm(g.positions, axis=1, keepdims=True)
    g.positions[:] = (g.positions * ((r - 0.002) / r)).astype(np.float32)
    xs = []
    for sdf in (baked, analytic):
        st = dict(num_itr=8, max_h=1 / 120, gravity=(0.0, 0.0, -9.81), radius=40e-6, sdf=sdf)
        s = helpers.gpu_solver(g, st, form="fused")
        s.step(1 / 120)
        xs.append(s.get_positions_velocities()[0])
        s.close()
        if sdf is baked:
            o = helpers.oracle_sim(g, st, np.float32)
            o.advance(1 / 120)
            assert np.abs(xs[0] - o.x).max() <= helpers.POS_TOL
    assert np.abs(xs[0] - xs[1]).max() <= 3e-4
    moved = np.abs(xs[1] - g.positions).max()
    assert moved > 1e-3  # the SDF pass pushed vertices out by millimetres


def _mesh_of(kind):
    rng = np.random.default_rng(11)
    if kind == "tetrahedron":  # fewer triangles than a cluster holds
        return np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]], np.float32) * np.float32(0.1), \
            np.array([[0, 2, 1], [0, 1, 3], [1, 2, 3], [0, 3, 2]], np.int32)
    V, T = synth.icosphere(3, 0.09)
    if kind == "slivers":  # clusters that may not be skipped beside clusters that may
        V = (V * np.array([1.0, 1.0, 1e-3])).astype(np.float32)
    elif kind == "away":
        V = (V + np.float32([3.0, -2.0, 1.0])).astype(np.float32)
    elif kind == "rough":
        V = (V + rng.normal(0, 2e-3, V.shape)).astype(np.float32)
    return V, T


@pytest.mark.parametrize("kind,dims,pad", [
    ("tetrahedron", (1, 1, 1), 0.05), ("tetrahedron", (5, 3, 7), 0.05), ("sphere", (9, 6, 3), 0.02),
    ("sphere", (8, 8, 4), 3.0), ("slivers", (13, 11, 10), 0.05), ("away", (10, 9, 5), 0.05), ("rough", (12, 7, 9), 0.1)])
def test_gpu_bake_skips_no_nearest_triangle(kind, dims, pad):
    """Clusters of triangles are skipped by a bound on their distance: the magnitudes still are the FP64
    distances over all triangles.  Tolerance: the node and the closest point are FP32 coordinates (a few units
    in the last place of the largest one, 6e-8 of it), and the weights of an interior closest point are off by
    up to 72 u (L D / 2A)^2 of the longest edge L, at a right angle to the distance; taken as 2e-6 + 1e-6 of
    the largest coordinate, and for a point displaced by s at distance d, s^2 / 2d is far below that here."""
    V, T = _mesh_of(kind)
    lo, hi = V.min(0) - np.float32(pad), V.max(0) + np.float32(pad)
    g = vbd.bake_sdf(V, T, dims, lo, hi)
    phi, _ = orc.sdf_bake(V, T, dims, g.grid_min, g.grid_max)
    big = max(np.abs(lo).max(), np.abs(hi).max())
    assert np.abs(np.abs(g.phi) - np.abs(phi)).max() <= 2e-6 + 1e-6 * big


def _scan_of_all(V, T, dims, lo, hi):
    """The bakes with nothing skipped: meshes of 16 consecutive triangles, which are one cluster each and tested
    whole."""
    for c in range(0, len(T), 16):
        used, local = np.unique(T[c:c + 16], return_inverse=True)
        yield vbd.bake_sdf(V[used], local.reshape(-1, 3).astype(np.int32), dims, lo, hi)


@pytest.mark.parametrize("kind,dims,pad", [
    ("tetrahedron", (5, 3, 7), 0.05), ("sphere", (15, 14, 13), 0.02), ("sphere", (8, 8, 4), 3.0),
    ("slivers", (13, 11, 10), 0.05), ("away", (10, 9, 5), 0.05), ("rough", (17, 12, 14), 0.0), ("tiny", (9, 9, 9), 2e-8)])
def test_gpu_bake_equals_a_scan_over_all_triangles(kind, dims, pad):
    """Skipping clusters changes no bit: the magnitude at every node, and the gradient where a node lies inside the
    mesh (there it points to the nearest triangle, so a wrong one shows; a patch of 16 triangles has no inside of
    its own, but its pseudonormals give the mesh's sign almost everywhere).  The sign is that
    of the FP64 distance, where that is clear of the coordinates' rounding (a few 6e-8 of the largest one)."""
    V, T = _mesh_of(kind) if kind != "tiny" else synth.icosphere(3, 1e-7)
    lo, hi = V.min(0) - np.float32(pad), V.max(0) + np.float32(pad)
    g = vbd.bake_sdf(V, T, dims, lo, hi)
    parts = list(_scan_of_all(V, T, dims, lo, hi))
    nearest = np.min([np.abs(p.phi) for p in parts], axis=0)
    np.testing.assert_array_equal(np.abs(g.phi).view(np.int32), nearest.view(np.int32))
    at = [(np.abs(p.phi) == nearest) & (p.phi < 0) for p in parts]  # (squares that differ may have one root)
    inside, shown = g.phi < 0, (g.phi < 0) & np.any(at, axis=0)
    if kind in ("sphere", "rough", "tiny") and pad < 1:
        assert shown.sum() >= 0.9 * inside.sum() > 50
    same = np.any([a & (p.grad == g.grad).all(-1) for a, p in zip(at, parts)], axis=0)
    assert same[shown].all()
    exact, _ = orc.sdf_bake(V, T, dims, g.grid_min, g.grid_max)
    clear = np.abs(exact) > 1e-6 * max(np.abs(lo).max(), np.abs(hi).max())
    np.testing.assert_array_equal(np.sign(g.phi[clear]), np.sign(exact[clear]))
