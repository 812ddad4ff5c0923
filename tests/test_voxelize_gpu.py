"""GPU: the device voxelizer (triangle mesh -> boundary ids and materials).

The reference's voxelizer is an external library that is not vendored, so its
output is not pinned; the voxelizer here follows the conventions of the
procedural rooms (rooms.py), and a grid-aligned box mesh must voxelize to
exactly the procedural room, ids and materials.
"""
import numpy as np
import pytest

from parallelfdtd_gb300 import rooms
from parallelfdtd_gb300.geometry import box_mesh, merge, voxelize

pytestmark = pytest.mark.gpu


def test_box_room_equals_procedural_room(gpu):
    room = box_mesh((0, 0, 0), (20, 16, 12), materials=(0, 1, 2, 3, 4, 5))
    a = box_mesh((5, 4, 3), (9, 8, 6), materials=(6,) * 6)
    b = box_mesh((10, 4, 3), (13, 8, 6), materials=(6,) * 6)   # 1-voxel slot to box a
    c = box_mesh((14, 10, 2), (17, 13, 9), materials=(3,) * 6)
    v, t, m = merge(room, a, b, c)
    bid, mat, dims, origin = voxelize(v, t, m, 1.0)
    assert dims == (22, 18, 14)
    assert np.allclose(origin, (-1.0, -1.0, -1.0))
    ref = rooms.build_room(dims, rooms.admittance_table(7, 0.1, 0.5, 1),
                           boxes=[(6, 5, 4, 10, 9, 7, 6), (11, 5, 4, 14, 9, 7, 6),
                                  (15, 11, 3, 18, 14, 10, 3)])
    assert np.array_equal(bid, ref.bid)
    assert np.array_equal(mat, ref.mat)


def test_scaled_room_and_node_coordinates(gpu):
    """A room of 7.875 x 5.125 x 3.25 m at dx = 0.125 m: node i of an axis sits
    at (i - 1) dx from the mesh's minimum, as the reference's element
    coordinates ROUND(p/dx) + 1 assume, so the room holds 63 x 41 x 26 air
    nodes with one solid layer around them."""
    room = box_mesh((2.0, -1.0, 0.5), (9.875, 4.125, 3.75))
    bid, mat, dims, origin = voxelize(*room, 0.125)
    X, Y, Z = dims
    assert (X, Y, Z) == (65, 43, 28)
    assert np.allclose(origin, (1.875, -1.125, 0.375))
    b = bid.reshape(Z, Y, X)
    inside = b > 0
    assert inside[1:27, 1:42, 1:64].all() and inside.sum() == 63 * 41 * 26
    assert (b[1:27, 1:42, 1] != 27).all() and (b[2:26, 2:41, 2] == 27).all()


def test_sphere_volume_and_ids(gpu):
    """A closed UV sphere (radius 10, dx 0.5): the air volume is the sphere's
    within a few per cent, ids are valid and every boundary node touches
    solid."""
    n_lat, n_lon, r = 48, 96, 10.0
    verts = [(0, 0, r)]
    for i in range(1, n_lat):
        th = np.pi * i / n_lat
        for j in range(n_lon):
            ph = 2 * np.pi * j / n_lon
            verts.append((r * np.sin(th) * np.cos(ph), r * np.sin(th) * np.sin(ph), r * np.cos(th)))
    verts.append((0, 0, -r))
    tris = []
    for j in range(n_lon):
        tris.append((0, 1 + j, 1 + (j + 1) % n_lon))
    for i in range(n_lat - 2):
        a0, b0 = 1 + i * n_lon, 1 + (i + 1) * n_lon
        for j in range(n_lon):
            j1 = (j + 1) % n_lon
            tris += [(a0 + j, b0 + j, b0 + j1), (a0 + j, b0 + j1, a0 + j1)]
    last = len(verts) - 1
    base = 1 + (n_lat - 2) * n_lon
    for j in range(n_lon):
        tris.append((base + j, last, base + (j + 1) % n_lon))
    v = np.array(verts, np.float32)
    t = np.array(tris, np.uint32)
    bid, mat, dims, origin = voxelize(v, t, np.zeros(len(t), np.uint8), 0.5)
    air = np.count_nonzero(bid) * 0.5 ** 3
    assert abs(air / (4 / 3 * np.pi * r ** 3) - 1) < 0.03
    assert bid.max() <= 27
    X, Y, Z = dims
    b = bid.reshape(Z, Y, X)
    solid = b == 0
    boundary = (b > 0) & (b < 27)
    nb = np.zeros_like(solid)
    nb[:, :, 1:] |= solid[:, :, :-1]
    nb[:, :, :-1] |= solid[:, :, 1:]
    nb[:, 1:] |= solid[:, :-1]
    nb[:, :-1] |= solid[:, 1:]
    nb[1:] |= solid[:-1]
    nb[:-1] |= solid[1:]
    assert np.array_equal(boundary, (b > 0) & nb)


def test_app_voxelizes_its_mesh(gpu):
    """libPyFDTD flow with a triangle mesh (initializeGeometryPy, one material
    row per triangle) gives the same responses as the same room given as
    voxels (initializeVoxels)."""
    from parallelfdtd_gb300 import libPyFDTD as pf
    fs = 4000
    dx = 344.0 / (fs * np.sqrt(1.0 / 3.0))   # the reference's dx = c / (fs * lambda)
    L_ = (24 * dx, 18 * dx, 14 * dx)
    v, t, m = merge(box_mesh((0, 0, 0), L_, materials=(0, 1, 2, 3, 4, 5)),
                    box_mesh((6 * dx, 5 * dx, 4 * dx), (10 * dx, 9 * dx, 7 * dx), materials=(6,) * 6))
    adm = np.linspace(0.1, 0.7, 7)
    coefs = np.repeat(adm[m][:, None], 20, axis=1)          # one row per triangle
    steps = 120

    def run(app):
        app.setSpatialFs(fs)
        app.setNumSteps(steps)
        app.setUpdateType(0)
        app.addSurfaceMaterials(coefs.flatten().tolist(), len(t), 20)
        app.addSource(12 * dx, 9 * dx, 7 * dx, 1, 0, 0)
        app.addReceiver(16 * dx, 12 * dx, 5 * dx)
        app.runSimulation()
        r = app.getResponse(0)
        app.close()
        return r

    a = pf.App()
    a.initializeDevices()
    a.initializeGeometryPy(t.flatten().tolist(), v.flatten().tolist())
    r_mesh = run(a)
    bid, mat, dims, _ = voxelize(v, t, m, dx)
    b = pf.App()
    b.initializeDevices()
    b.initializeGeometryPy(t.flatten().tolist(), v.flatten().tolist())  # materials per triangle
    b.initializeVoxels(bid, mat, dims)
    r_vox = run(b)
    assert np.abs(r_mesh).max() > 0
    assert np.array_equal(r_mesh, r_vox)


def _brute_force(v, t, m, dx, dims):
    """Ids and materials with every triangle tested for every column and every
    surface node, in double."""
    X, Y, Z = dims
    eps = (1.2345678901e-5, 3.1415926536e-5, 2.2360679775e-5)
    lo = v.astype(np.float64).min(axis=0)
    at = [lo[a] + (np.arange(n) - 1 + eps[a]) * dx for a, n in enumerate(dims)]
    tri = v.astype(np.float64)[t]

    def cross(k, ax, a0, a1):
        c0, c1 = [a for a in range(3) if a != ax]
        (x0, y0), (x1, y1), (x2, y2) = tri[k][:, [c0, c1]]
        e0 = (x1 - x0) * (a1 - y0) - (y1 - y0) * (a0 - x0)
        e1 = (x2 - x1) * (a1 - y1) - (y2 - y1) * (a0 - x1)
        e2 = (x0 - x2) * (a1 - y2) - (y0 - y2) * (a0 - x2)
        hit = ((e0 > 0) & (e1 > 0) & (e2 > 0)) | ((e0 < 0) & (e1 < 0) & (e2 < 0))
        area = np.where(hit, e0 + e1 + e2, 1.0)
        return hit, (e1 * tri[k][0, ax] + e2 * tri[k][1, ax] + e0 * tri[k][2, ax]) / area

    below = np.zeros((Z, Y, X), int)
    for k in range(len(t)):
        hit, z = cross(k, 2, at[0][None, :], at[1][:, None])
        below += hit[None] & (z[None] < at[2][:, None, None])
    solid = below % 2 == 0
    smat = np.full((Z, Y, X), 255, np.uint8)
    steps = [(0, 0, -1), (0, 0, 1), (0, -1, 0), (0, 1, 0), (-1, 0, 0), (1, 0, 0)]
    for z, y, x in np.argwhere(solid):
        for d, (dz, dy, dx_) in enumerate(steps):
            q = (z + dz, y + dy, x + dx_)
            if all(0 <= q[a] < solid.shape[a] for a in range(3)) and not solid[q]:
                ax, p = d >> 1, (at[0][x], at[1][y], at[2][z])
                best, c = 2.0, [a for a in range(3) if a != ax]
                for k in range(len(t)):
                    hit, w = cross(k, ax, p[c[0]], p[c[1]])
                    s = (w - p[ax]) * (1 if d & 1 else -1) / dx
                    if hit and 0 <= s <= 1 and s < best:
                        best, smat[z, y, x] = s, m[k]
                break
    while True:
        miss = rooms._neighbour_missing(solid)
        bad = ~solid & (rooms.BID_LUT[miss] == 0)
        if not bad.any():
            break
        smat = np.where(bad, rooms._first_solid_material(solid, smat), smat)
        solid = solid | bad
    bid = np.where(solid, 0, rooms.BID_LUT[miss]).astype(np.uint8)
    bmat = rooms._first_solid_material(solid, smat)
    mat = np.where((bid > 0) & (bid < 27) & (bmat != 255), bmat, 0)
    return bid.reshape(-1), mat.reshape(-1).astype(np.uint8)


@pytest.mark.parametrize("nodes,dx,origin", [
    ((33, 5, 9), 0.25, (0.0, 0.0, 0.0)),       # one node past a column tile and a cell
    ((32, 8, 16), 0.5, (-3.1, 2.7, 40.3)),     # whole tiles and cells
    ((65, 41, 23), 0.1, (1000.0, -500.0, 7.0)),  # far from the origin
    ((6, 5, 4), 1.0, (0.3, 0.3, 0.3)),         # smaller than a cell
])
def test_triangle_lists_lose_no_triangle(gpu, nodes, dx, origin):
    """Rooms with tilted obstacles (no face along an axis) equal a loop over
    every triangle, at sizes on either side of the list cells."""
    rng = np.random.default_rng(sum(nodes))
    size = (np.array(nodes) - 2.3) * dx
    parts = [box_mesh(origin, np.array(origin) + size, materials=(0, 1, 2, 3, 4, 5))]
    for k in range(3):  # octahedra of random corners along the axes
        c = np.array(origin) + size * rng.uniform(0.3, 0.7, 3)
        r = size * rng.uniform(0.15, 0.28, (2, 3))
        p = np.array([c - [r[0, 0], 0, 0], c + [r[1, 0], 0, 0], c - [0, r[0, 1], 0],
                      c + [0, r[1, 1], 0], c - [0, 0, r[0, 2]], c + [0, 0, r[1, 2]]])
        p += rng.uniform(-0.05, 0.05, (6, 3)) * size
        f = [(i, j, l) for i in (0, 1) for j in (2, 3) for l in (4, 5)]
        parts.append((p.astype(np.float32), np.array(f, np.uint32), np.full(8, 6 + k, np.uint8)))
    v, t, m = merge(*parts)
    bid, mat, dims, _ = voxelize(v, t, m, dx)
    ref_bid, ref_mat = _brute_force(v, t, m, dx, dims)
    assert np.array_equal(bid, ref_bid)
    assert np.array_equal(mat, ref_mat)


def _tilted_room(nodes, n_obstacles, seed):
    """A box with octahedra of random corners in it (8 triangles each)."""
    rng = np.random.default_rng(seed)
    size = np.array(nodes) - 2.3
    parts = [box_mesh((0, 0, 0), size, materials=(0, 1, 2, 3, 4, 5))]
    for k in range(n_obstacles):
        c, r = size * rng.uniform(0.3, 0.7, 3), size * rng.uniform(0.15, 0.28, (2, 3))
        p = np.array([c - [r[0, 0], 0, 0], c + [r[1, 0], 0, 0], c - [0, r[0, 1], 0],
                      c + [0, r[1, 1], 0], c - [0, 0, r[0, 2]], c + [0, 0, r[1, 2]]])
        p += rng.uniform(-0.05, 0.05, (6, 3)) * size
        f = [(i, j, l) for i in (0, 1) for j in (2, 3) for l in (4, 5)]
        parts.append((p.astype(np.float32), np.array(f, np.uint32), np.full(8, 6 + k, np.uint8)))
    return merge(*parts)


@pytest.mark.parametrize("nodes,n_obstacles,more", [
    ((33, 21, 13), 0, 0), ((33, 21, 13), 2, 0), ((33, 21, 13), 2, 36), ((33, 21, 13), 2, 37),
    ((33, 5, 9), 9, 0), ((32, 8, 16), 9, 0), ((65, 41, 23), 9, 0), ((6, 5, 4), 9, 0)])
def test_few_triangles_are_not_binned(gpu, nodes, n_obstacles, more):
    """Meshes of 12 and 28 triangles, 64 and 65 (with some that no line crosses)
    and 84, on both sides of where lists per cell start, the last at sizes on
    either side of the cells, equal a loop over every triangle."""
    v, t, m = _tilted_room(nodes, n_obstacles, 5)
    t = np.concatenate([t, np.array([[0, 0, 7]] * more, np.uint32).reshape(-1, 3)])
    m = np.concatenate([m, np.full(more, 99, np.uint8)])
    bid, mat, dims, _ = voxelize(v, t, m, 1.0)
    ref_bid, ref_mat = _brute_force(v, t, m, 1.0, dims)
    assert np.array_equal(bid, ref_bid) and np.array_equal(mat, ref_mat)


def test_lists_too_long_take_larger_cells(gpu):
    """500 triangles across the whole of a 3000 x 3000 x 5 grid would be in more
    lists than are kept of either kind, so both take larger cells.  No line
    crosses these triangles (two corners coincide), and the result is that of
    the mesh without them."""
    v, t, m = _tilted_room((3000, 3000, 5), 3, 6)
    far = np.argmax(v.sum(axis=1))
    near = np.argmin(v.sum(axis=1))
    more = np.array([[near, near, far]] * 500, np.uint32)
    want = voxelize(v, t, m, 1.0)
    got = voxelize(v, np.concatenate([t, more]), np.concatenate([m, np.full(500, 99, np.uint8)]), 1.0)
    assert want[2] == got[2] == (3000, 3000, 5) and np.count_nonzero(want[0]) > 10 ** 7
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
