"""CPU tests of the prism walk records (hase_mesh_tables) and of the edge
windows that the walks read (hase_mesh_windows), both built on the host.

The records: the two triangles of an edge store exactly negated normals, so an
edge that a ray moves out through in one triangle it moves in through in the
next, to the last bit, and the neighbour codes are reciprocal.  The exported
copy marks mesh-boundary edges with NaN normals.

The windows: a triangle's two edges other than the one the walk entered
through, a code that is the window on the other side, and a boundary edge whose
exit parameter is negative for every ray.

Checked on the legacy fixtures and on the seeded workload meshes, with and
without consistently oriented triangles."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from conftest import legacy_mesh


def _desc(mesh):
    from haseongpu_b200 import _native as N

    pts = np.ascontiguousarray(mesh.points, np.float64)
    tri = np.ascontiguousarray(mesh.triangles, np.uint32)
    T = tri.shape[0]
    return (pts, tri), N.MeshDesc(mesh.numberOfPoints, T, mesh.numberOfLevels, N.ptr(pts, N._f64p), N.ptr(tri, N._u32p),
                                  mesh.thickness, None, None, None, 0, 0.0, 1.0, 1.0, None, None)


def _records(native, mesh):
    held, desc = _desc(mesh)
    T = held[1].shape[0]
    rec = np.zeros((T, 12), np.float32)
    walk = np.zeros((T, 12), np.float32)
    native.check(native.lib().hase_mesh_tables(C.byref(desc), rec.ctypes.data_as(C.POINTER(C.c_float)),
                                               walk.ctypes.data_as(C.POINTER(C.c_float))))
    return rec, walk


def _meshes():
    from haseongpu_b200.configs import disc_poly, disc_small

    out = [("cuboid", legacy_mesh("cuboid")), ("cylindrical", legacy_mesh("cylindrical")),
           ("disc_small", disc_small().mesh), ("disc_poly", disc_poly().mesh)]
    # the cylinder with every other triangle's vertex order reversed
    m = legacy_mesh("cylindrical")
    flipped = m.triangles.copy()
    flipped[::2] = flipped[::2, ::-1]
    m.triangles = flipped
    out.append(("cylindrical, mixed orientation", m))
    return out


NX, NY, C0, NB = (0, 3, 6), (1, 4, 7), (2, 5, 8), (9, 10, 11)


@pytest.mark.parametrize("name,mesh", _meshes(), ids=lambda v: v if isinstance(v, str) else "")
def test_shared_edges_store_exactly_negated_normals(native, name, mesh):
    rec, walk = _records(native, mesh)
    T = rec.shape[0]
    nb = rec[:, 9:12].copy().view(np.int32)
    shared = boundary = 0
    for t in range(T):
        for e in range(3):
            code = int(nb[t, e])
            if code < 0:
                boundary += 1
                assert np.isnan(walk[t, NX[e]]) and np.isnan(walk[t, NY[e]]), (t, e)
                assert walk[t, C0[e]] == rec[t, C0[e]]
                continue
            u, f = code >> 2, code & 3
            assert int(nb[u, f]) == (t << 2 | e), (t, e)
            # exact negation, bit for bit
            assert rec[u, NX[f]] == -rec[t, NX[e]] and rec[u, NY[f]] == -rec[t, NY[e]], (t, e, u, f)
            assert walk[t, NX[e]] == rec[t, NX[e]] and walk[t, NY[e]] == rec[t, NY[e]]
            shared += 1
    assert shared > 0 and boundary > 0
    # the copy differs from the records only in the boundary normals (columns
    # 9..11 are the neighbour codes, -1 reads as a NaN float there)
    assert np.array_equal(walk[:, 9:].view(np.int32), rec[:, 9:].view(np.int32))
    geo_w, geo_r = walk[:, :9], rec[:, :9]
    same = ~np.isnan(geo_w)
    assert np.array_equal(geo_w[same], geo_r[same])
    assert np.isnan(geo_w).sum() == 2 * boundary and not np.isnan(geo_r).any()


def test_entry_edge_fails_the_exit_test(native):
    """dd = -(n . u) of the edge a walk entered through is exactly minus the
    dd > 0 of the same edge in the triangle it left, for FP32 directions."""
    mesh = legacy_mesh("cylindrical")
    rec, _ = _records(native, mesh)
    nb = rec[:, 9:12].copy().view(np.int32)
    rng = np.random.default_rng(3)
    f32 = np.float32
    checked = 0
    for _ in range(2000):
        t, e = int(rng.integers(rec.shape[0])), int(rng.integers(3))
        code = int(nb[t, e])
        if code < 0:
            continue
        u, f = code >> 2, code & 3
        a = rng.uniform(0, 2 * np.pi)
        ux, uy = f32(np.cos(a)), f32(np.sin(a))
        dd_out = -np.float32(np.float32(rec[t, NX[e]] * ux) + np.float32(rec[t, NY[e]] * uy))
        dd_in = -np.float32(np.float32(rec[u, NX[f]] * ux) + np.float32(rec[u, NY[f]] * uy))
        assert dd_in == -dd_out
        if dd_out > 0:
            assert not dd_in > 0
        checked += 1
    assert checked > 1000


def _windows(native, mesh):
    held, desc = _desc(mesh)
    win = np.zeros((held[1].shape[0], 4, 4), np.float32)
    native.check(native.lib().hase_mesh_windows(C.byref(desc), win.ctypes.data_as(C.POINTER(C.c_float))))
    return win


FIRST_SLOT = (1, 2, 0)  # of the window entered through e0, e1, e2


@pytest.mark.parametrize("name,mesh", _meshes(), ids=lambda v: v if isinstance(v, str) else "")
def test_windows_hold_the_edges_a_ray_can_leave_by(native, name, mesh):
    """Slots e0 e1 e2 e0 of the records' edges; the code leads to the window of the neighbour's two other edges; a
    boundary edge is (0, 0, 1, 0)."""
    rec, _ = _records(native, mesh)
    win = _windows(native, mesh)
    T = rec.shape[0]
    nb = rec[:, 9:12].copy().view(np.int32)
    bits = win.view(np.uint32)
    code = bits[:, :, 3]
    np.testing.assert_array_equal(bits[:, 3], bits[:, 0])
    boundary = np.float32([0, 0, 1, 0]).view(np.uint32)
    edge_of_slot = (0, 1, 2, 0)
    for t in range(T):
        for e in range(3):
            if nb[t, e] < 0:
                assert np.array_equal(bits[t, e], boundary)
                continue
            assert np.array_equal(win[t, e, :3], rec[t, [NX[e], NY[e], C0[e]]])
            u, f = nb[t, e] >> 2, nb[t, e] & 3
            first = int(code[t, e]) & 3
            assert int(code[t, e]) >> 2 == u and first == FIRST_SLOT[f]
            assert {edge_of_slot[first], edge_of_slot[first + 1]} == {0, 1, 2} - {f}
    assert code.max() < 4 * T


def test_boundary_edges_are_never_exits(native):
    """The exit parameter of the walks' edge test, in FP32 as the kernels take it: negative on a boundary edge whatever
    the ray and the sample, and not positive on an edge that the ray moves in through."""
    mesh = legacy_mesh("cylindrical")
    win = _windows(native, mesh)
    rng = np.random.default_rng(3)
    f32 = np.float32

    def exit_parameter(edge, ux, uy, Sx, Sy):
        d = f32(f32(-edge[0] * ux) + f32(f32(-edge[1] * uy) + f32(-1e-30)))
        e = f32(f32(edge[0] * Sx) + f32(f32(edge[1] * Sy) - edge[2]))
        e = -abs(e) if np.signbit(d) else e
        return float(e) / abs(float(d)), d

    boundary = inward = 0
    for _ in range(6000):
        t, s = int(rng.integers(win.shape[0])), int(rng.integers(4))
        a = rng.uniform(0, 2 * np.pi)
        Sx, Sy = (f32(v) for v in mesh.points[rng.integers(mesh.numberOfPoints)])
        q, d = exit_parameter(win[t, s], f32(np.cos(a)), f32(np.sin(a)), Sx, Sy)
        if win[t, s, 2] == 1.0 and not win[t, s, :2].any():
            assert q < 0
            boundary += 1
        elif d < 0:
            assert q <= 0
            inward += 1
    assert boundary > 20 and inward > 1000


def test_mesh_tables_rejects_missing_arrays(native):
    from haseongpu_b200 import _native as N

    desc = N.MeshDesc()
    assert native.lib().hase_mesh_tables(C.byref(desc), None, None) == native.HASE_INVALID_ARGUMENT
    win = (C.c_float * 16)()
    assert native.lib().hase_mesh_windows(C.byref(desc), win) == native.HASE_INVALID_ARGUMENT
    held, full = _desc(legacy_mesh("cuboid"))
    assert native.lib().hase_mesh_windows(C.byref(full), None) == native.HASE_INVALID_ARGUMENT
