"""GPU: FP64 updates of open air, which leave out products by 1 and (centred)
boundary neighbours times 0, against the CPU oracle: also where a field value is
infinite or not a number, so that 0 times it must still be done."""
import numpy as np
import pytest

from parallelfdtd_gb300 import _lib as L
from parallelfdtd_gb300 import rooms
from parallelfdtd_gb300.domain import Domain, default_params

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def O(built):
    from oracle import oracle
    return oracle


@pytest.mark.parametrize("dims", [(34, 19, 17), (66, 10, 21), (128, 9, 40)])
@pytest.mark.parametrize("scheme", ["forward", "centred"])
@pytest.mark.parametrize("kernel", ["auto", "zmarch", "tma"])
@pytest.mark.parametrize("bad", [None, np.inf, -np.inf, np.nan])
def test_f64(gpu, O, dims, scheme, kernel, bad):
    room = rooms.shoebox(dims, seed=4)
    rng = np.random.default_rng(dims[0])
    P0, Pp0 = rng.uniform(-1, 1, room.n_nodes), rng.uniform(-1, 1, room.n_nodes)
    if bad is not None:
        P0[room.flat(dims[0] // 2, dims[1] // 2, dims[2] // 2)] = bad
    steps = 3  # the value has not reached a wall
    with Domain(dims, "f64") as d:
        d.set_kernel(kernel)
        d.set_scheme(scheme)
        d.set_voxels(room.bid, room.mat, centred=scheme == "centred")
        d.set_materials(room.admittance)
        d.set_params()
        d.upload_field(L.FIELD_CURRENT, P0)
        d.upload_field(L.FIELD_PAST, Pp0)
        d.run(steps)
        P, Pp = d.download_field(L.FIELD_CURRENT), d.download_field(L.FIELD_PAST)
    pos, mat = O.encode_nodes(room.bid, room.mat, scheme == "centred")
    _, rP, rPp = O.run(pos, mat, dims, room.admittance, default_params(), [], [], np.zeros((0, steps)),
                       [], steps, scheme=2 if scheme == "centred" else 0, double=True, P0=P0, Pp0=Pp0)
    assert np.array_equal(P, rP, equal_nan=True)
    assert np.array_equal(Pp, rPp, equal_nan=True)


@pytest.mark.parametrize("dims", [(4, 4, 4), (24, 24, 24), (48, 40, 36), (35, 17, 60), (64, 64, 64),
                                  (100, 90, 80), (128, 96, 100), (130, 128, 128)])
@pytest.mark.parametrize("scheme", ["forward", "centred"])
@pytest.mark.parametrize("dif", [False, True])
def test_chunks(gpu, O, dims, scheme, dif):
    """Chunks of 1 to 8 planes, launched plainly or as programmatic dependents,
    with and without the pass of frequency-dependent walls behind them."""
    from parallelfdtd_gb300 import materials
    room = rooms.boxes_room(dims, n_boxes=3, edge=(4, 9), n_materials=4, seed=4) if min(dims) > 16 \
        else rooms.shoebox(dims, seed=4)
    n_mat, steps = len(room.admittance), 6
    rng = np.random.default_rng(dims[0])
    P0, Pp0 = rng.uniform(-1, 1, room.n_nodes), rng.uniform(-1, 1, room.n_nodes)
    flags = np.array([m % 2 for m in range(n_mat)], np.int32)
    filters = materials.dif_table(materials.positive_real_filters(n_mat, 3, seed=2), 3)
    at, pulse = tuple(n // 2 for n in dims), rng.uniform(-1, 1, (1, steps))
    with Domain(dims, "f64") as d:
        d.set_kernel("zmarch")
        d.set_scheme(scheme)
        d.set_voxels(room.bid, room.mat, centred=scheme == "centred")
        d.set_materials(room.admittance)
        d.set_params()
        if dif:
            d.set_dif_filters(flags, filters)
        d.set_sources([at], [1], pulse)
        d.set_receivers([at])
        d.upload_field(L.FIELD_CURRENT, P0)
        d.upload_field(L.FIELD_PAST, Pp0)
        got, _, _ = d.run(steps)
        P, Pp = d.download_field(L.FIELD_CURRENT), d.download_field(L.FIELD_PAST)
    pos, mat = O.encode_nodes(room.bid, room.mat, scheme == "centred")
    want, rP, rPp = O.run(pos, mat, dims, room.admittance, default_params(), [room.flat(*at)], [1], pulse,
                          [room.flat(*at)], steps, scheme=2 if scheme == "centred" else 0, double=True,
                          P0=P0, Pp0=Pp0, **({"dif": (flags, filters)} if dif else {}))
    assert np.array_equal(got, want) and np.array_equal(P, rP) and np.array_equal(Pp, rPp)


@pytest.mark.parametrize("dims,fields", [((8, 8, 8), 4), ((16, 12, 20), 8), ((160, 9, 12), 4), ((164, 9, 12), 4),
                                         ((80, 9, 14), 8), ((84, 20, 40), 8), ((96, 60, 50), 8), ((300, 8, 8), 4)])
@pytest.mark.parametrize("scheme", ["forward", "centred"])
@pytest.mark.parametrize("wide", [False, True])
def test_batched(gpu, O, dims, fields, scheme, wide):
    """Several fields, a few tile columns (5 and less) and more, short chunks and
    long, 8- and 16-bit class ids: every field equals the oracle's run of it
    alone, also with an infinity in the field."""
    room = rooms.shoebox(dims, seed=4)
    rng = np.random.default_rng(dims[0])
    mat, table = room.mat, room.admittance
    if wide:  # more than 256 classes
        table = rooms.admittance_table(100, 0.05, 0.9, 9)
        mat = np.where(room.bid > 0, rng.integers(0, 100, room.n_nodes), 0).astype(np.uint8)
    P0, Pp0 = rng.uniform(-1, 1, (2, room.n_nodes, fields))
    P0[room.flat(*(n // 2 for n in dims)), 1] = np.inf
    steps = 3  # the value reaches no wall
    with Domain(dims, "f64", fields=fields) as d:
        d.set_scheme(scheme)
        d.set_voxels(room.bid, mat, centred=scheme == "centred")
        d.set_materials(table)
        d.set_params()
        d.upload_field(L.FIELD_CURRENT, P0.reshape(-1))
        d.upload_field(L.FIELD_PAST, Pp0.reshape(-1))
        d.run(steps)
        P = d.download_field(L.FIELD_CURRENT).reshape(-1, fields)
        Pp = d.download_field(L.FIELD_PAST).reshape(-1, fields)
        assert d.kernel() == "tma"
    pos, m = O.encode_nodes(room.bid, mat, scheme == "centred")
    for f in (0, 1, fields - 1):
        _, rP, rPp = O.run(pos, m, dims, table, default_params(), [], [], np.zeros((0, steps)), [], steps,
                           scheme=2 if scheme == "centred" else 0, double=True,
                           P0=np.ascontiguousarray(P0[:, f]), Pp0=np.ascontiguousarray(Pp0[:, f]))
        assert np.array_equal(P[:, f], rP, equal_nan=True), f
        assert np.array_equal(Pp[:, f], rPp, equal_nan=True), f
