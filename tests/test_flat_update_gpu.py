"""GPU: the update of flat index runs (rows that are not 16-byte aligned) against
the CPU oracle, bit for bit.

A run holds 2048 indices of a plane: sizes lie on either side of one and two
runs and leave every remainder of the 16-byte boundaries.  Inside nodes on all
four side faces make the flat wrap across rows matter; materials drawn per node
give more than 256 classes (16-bit ids).  PFDTD_KERNEL_TMA keeps small rooms off
the resident path."""
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


def _values(rng, n, prec):
    v = rng.uniform(-1.0, 1.0, n).astype(np.float32)
    if prec == "bf16":
        return (v.view(np.uint32) >> 16).astype(np.uint16)
    return v.astype({"f32": np.float32, "f16": np.float16}[prec])


def _check(O, dims, prec="f32", scheme="forward", wide=False, fields=1, form="reference", steps=9):
    room = rooms.boxes_room(dims, n_boxes=2 if min(dims) > 16 else 0, edge=(4, 9), n_materials=5,
                            seed=sum(dims))
    X, Y, Z = dims
    rng = np.random.default_rng(X)
    bid, mat, table = room.bid.copy().reshape(Z, Y, X), room.mat.copy(), room.admittance
    bid[2:-2, :, [0, -1]] = 27
    bid[2:-2, [0, -1], :] = 27
    bid = bid.reshape(-1)
    if wide:
        table = rooms.admittance_table(200, 0.05, 0.9, 9)
        mat = np.where(bid > 0, rng.integers(0, 200, bid.size), 0).astype(np.uint8)
    inside = np.flatnonzero(bid)
    src, rec = rng.choice(inside, fields), rng.choice(inside, fields)
    pulses = rng.uniform(-1.0, 1.0, (fields, steps))
    P0, Pp0 = _values(rng, room.n_nodes * fields, prec), _values(rng, room.n_nodes * fields, prec)
    with Domain(dims, prec, fields=fields) as d:
        d.set_kernel("tma")
        d.set_scheme(scheme)
        d.set_voxels(bid, mat, centred=scheme == "centred")
        d.set_materials(table)
        d.set_params()
        if form != "reference":
            d.set_update_form(form)
        d.set_sources([room.coords(int(i)) for i in src], [1] * fields, pulses, fields=range(fields))
        d.set_receivers([room.coords(int(i)) for i in rec], fields=range(fields))
        d.upload_field(L.FIELD_CURRENT, P0)
        d.upload_field(L.FIELD_PAST, Pp0)
        got, _, st = d.run(steps)
        # (rows of 1023 leave no room for four stages: the z-march kernel)
        assert st == 0 and d.kernel() == ("tma" if X < 900 else "zmarch")
        P, Pp = (d.download_field(w).reshape(-1, fields) for w in (L.FIELD_CURRENT, L.FIELD_PAST))
    pos, m = O.encode_nodes(bid, mat, scheme == "centred")
    for f in range(fields):
        want, rP, rPp = O.run(pos, m, dims, table, default_params(), src[f:f + 1], [1], pulses[f:f + 1],
                              rec[f:f + 1], steps, scheme=2 if scheme == "centred" else 0,
                              storage=None if prec == "f32" else prec, form=form,
                              P0=P0.reshape(-1, fields)[:, f], Pp0=Pp0.reshape(-1, fields)[:, f])
        assert np.array_equal(got[f], want[0])
        assert np.array_equal(P[:, f], rP) and np.array_equal(Pp[:, f], rPp)


@pytest.mark.parametrize("dims", [(5, 4, 5), (33, 17, 9), (45, 46, 12), (683, 3, 6), (273, 15, 5),
                                  (203, 31, 12), (511, 9, 20), (18, 227, 7), (1023, 5, 5)])
@pytest.mark.parametrize("scheme", ["forward", "centred"])
def test_sizes(gpu, O, dims, scheme):
    _check(O, dims, scheme=scheme)


@pytest.mark.parametrize("prec", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("scheme", ["forward", "centred"])
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("dims", [(37, 29, 18), (70, 61, 11)])
def test_types(gpu, O, dims, prec, scheme, wide):
    _check(O, dims, prec, scheme, wide)


@pytest.mark.parametrize("dims", [(33, 40, 9), (41, 25, 12)])
def test_two_fields(gpu, O, dims):
    _check(O, dims, fields=2)


def test_difference_form(gpu, O):
    _check(O, (53, 40, 14), form="difference")


def test_expired_wait_is_reported(gpu):
    """A wait bound of a nanosecond runs out; the run fails and the next one,
    with the bound restored, works."""
    room = rooms.shoebox((203, 40, 60), seed=1)
    with Domain(room.dims) as d:
        d.set_kernel("tma")
        d.set_voxels(room.bid, room.mat, centred=False)
        d.set_materials(room.admittance)
        d.set_params()
        L.call("pfdtd_set_wait_limit", d.handle, 1)
        with pytest.raises(L.PfdtdError) as e:
            d.run(50)
        assert e.value.status == L.ERR_CUDA and "timed out" in str(e.value)
        L.call("pfdtd_set_wait_limit", d.handle, 0)
        d.reset_fields()
        assert d.run(50)[2] == 0


@pytest.mark.parametrize("dims,scheme,prec", [((160, 140, 140), "forward", "f32"), ((160, 140, 140), "centred", "f32"),
                                              ((160, 140, 140), "forward", "f16"), ((256, 200, 160), "forward", "f32"),
                                              ((160, 140, 140), "iwb", "f32"), ((109, 101, 97), "iwb", "f32")])
def test_large_aligned_rooms(gpu, dims, scheme, prec):
    """Rooms that the dispatch gives to the runs equal the z-march kernel."""
    room = rooms.boxes_room(dims, n_boxes=6, edge=(8, 40), n_materials=5, seed=3)
    P0 = _values(np.random.default_rng(1), room.n_nodes, prec)
    out = []
    for kernel in ("auto", "zmarch"):
        with Domain(dims, prec) as d:
            d.set_kernel(kernel)
            d.set_scheme(scheme)
            d.set_voxels(room.bid, room.mat, centred=scheme != "forward")
            d.set_materials(room.admittance)
            d.set_params(default_params(scheme="iwb" if scheme == "iwb" else "forward"))
            d.upload_field(L.FIELD_CURRENT, P0)
            d.run(5)
            out.append((d.download_field(L.FIELD_CURRENT), d.download_field(L.FIELD_PAST)))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("prec", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("dims,wide", [((5, 4, 5), False), ((45, 46, 12), False), ((683, 3, 6), False),
                                       ((37, 29, 18), True), ((64, 33, 20), False), ((203, 31, 12), True),
                                       ((100, 41, 24), True)])
def test_iwb(gpu, O, prec, dims, wide):
    """IWB by runs with the closure pass, inside nodes on the x and y faces,
    frequency-dependent walls in half of the materials; rows with and without
    16-byte alignment."""
    from parallelfdtd_gb300 import materials
    room = rooms.boxes_room(dims, n_boxes=2 if min(dims) > 16 else 0, edge=(4, 9), n_materials=6,
                            seed=sum(dims))
    X, Y, Z = dims
    rng = np.random.default_rng(X)
    bid, mat, table = room.bid.copy().reshape(Z, Y, X), room.mat.copy(), room.admittance
    bid[2:-2, :, [0, -1]] = 26
    bid[2:-2, [0, -1], :] = 26
    bid = bid.reshape(-1)
    if wide:
        table = rooms.admittance_table(100, 0.05, 0.9, 9)
        mat = np.where(bid > 0, rng.integers(0, 100, bid.size), 0).astype(np.uint8)
    flags = np.array([m % 2 for m in range(len(table))], np.int32)
    filters = materials.dif_table(materials.positive_real_filters(len(table), 3, seed=2), 3)
    inside, steps = np.flatnonzero(bid), 7
    src, rec = rng.choice(inside, 2), rng.choice(inside, 3)
    pulses = rng.uniform(-1.0, 1.0, (2, steps))
    P0, Pp0 = _values(rng, room.n_nodes, prec), _values(rng, room.n_nodes, prec)
    params = default_params(scheme="iwb")
    with Domain(dims, prec) as d:
        d.set_kernel("tma")
        d.set_scheme("iwb")
        d.set_voxels(bid, mat, centred=True)
        d.set_materials(table)
        d.set_params(params)
        d.set_dif_filters(flags, filters)
        d.set_sources([room.coords(int(i)) for i in src], [1, 1], pulses)
        d.set_receivers([room.coords(int(i)) for i in rec])
        d.upload_field(L.FIELD_CURRENT, P0)
        d.upload_field(L.FIELD_PAST, Pp0)
        got, _, st = d.run(steps)
        assert st == 0 and d.kernel() == "tma"
        P, Pp = d.download_field(L.FIELD_CURRENT), d.download_field(L.FIELD_PAST)
    pos, m = O.encode_nodes(bid, mat, True)
    want, rP, rPp = O.run(pos, m, dims, table, params, src, [1, 1], pulses, rec, steps, scheme=3,
                          storage=None if prec == "f32" else prec, dif=(flags, filters), P0=P0, Pp0=Pp0)
    assert np.array_equal(got, want) and np.array_equal(P, rP) and np.array_equal(Pp, rPp)


@pytest.mark.parametrize("dims,scheme,fields,dif,flat", [
    ((90, 91, 89), "forward", 1, False, False), ((97, 97, 97), "forward", 1, False, True),
    ((97, 97, 97), "centred", 1, False, True), ((13, 13, 5100), "centred", 1, False, False),
    ((96, 96, 96), "centred", 2, False, False), ((161, 120, 110), "centred", 1, False, True),
    ((80, 80, 66), "forward", 2, False, False), ((80, 80, 68), "forward", 2, False, True),
    ((90, 91, 89), "iwb", 1, True, False), ((101, 103, 99), "iwb", 1, True, True),
    ((101, 103, 99), "iwb", 1, False, False), ((131, 127, 101), "iwb", 1, False, True),
    ((13, 13, 9600), "iwb", 1, False, False)])
def test_rooms_by_size(gpu, dims, scheme, fields, dif, flat):
    """Rooms whose rows are not aligned (or with two fields) take the runs from
    where they pay, the z-march kernel below and where a plane fills too little of
    a run, and both give the z-march kernel's fields."""
    from parallelfdtd_gb300 import materials
    room = rooms.boxes_room(dims, n_boxes=3, edge=(8, 30), n_materials=5, seed=3) if min(dims) > 40 \
        else rooms.shoebox(dims, seed=3)
    P0 = _values(np.random.default_rng(1), room.n_nodes * fields, "f32")
    out, n_mat = [], len(room.admittance)
    for kernel in ("auto", "zmarch"):
        with Domain(dims, fields=fields) as d:
            d.set_kernel(kernel)
            d.set_scheme(scheme)
            d.set_voxels(room.bid, room.mat, centred=scheme != "forward")
            d.set_materials(room.admittance)
            d.set_params(default_params(scheme="iwb" if scheme == "iwb" else "forward"))
            if dif:
                d.set_dif_filters(np.array([m % 2 for m in range(n_mat)], np.int32),
                                  materials.dif_table(materials.positive_real_filters(n_mat, 3, seed=2), 3))
            d.upload_field(L.FIELD_CURRENT, P0)
            L.call("pfdtd_run_async", d.handle, 5)  # by single steps
            d.synchronize()
            assert d.kernel() == ("tma" if flat and kernel == "auto" else "zmarch")
            out.append((d.download_field(L.FIELD_CURRENT), d.download_field(L.FIELD_PAST)))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("prec", ["f16", "bf16"])
@pytest.mark.parametrize("scheme", ["forward", "centred"])
@pytest.mark.parametrize("dims,fields", [((37, 29, 18), 4), ((33, 31, 9), 2), ((9, 9, 30), 4)])
def test_fields_in_16_bits(gpu, O, prec, scheme, dims, fields):
    _check(O, dims, prec, scheme, fields=fields)


@pytest.mark.parametrize("dims", [(160, 128, 120), (256, 96, 101)])
def test_difference_form_of_tiles(gpu, O, dims):
    """The difference form in the tiled update, which aligned single-field rooms
    between the resident and the large ones take."""
    room = rooms.boxes_room(dims, n_boxes=3, edge=(8, 30), n_materials=5, seed=3)
    rng = np.random.default_rng(2)
    P0, Pp0 = _values(rng, room.n_nodes, "f32"), _values(rng, room.n_nodes, "f32")
    steps, at, pulse = 6, (40, 50, 60), rng.uniform(-1, 1, (1, 6))
    with Domain(dims) as d:
        d.set_voxels(room.bid, room.mat, centred=False)
        d.set_materials(room.admittance)
        d.set_params()
        d.set_update_form("difference")
        d.set_sources([at], [1], pulse)
        d.set_receivers([at])
        d.upload_field(L.FIELD_CURRENT, P0)
        d.upload_field(L.FIELD_PAST, Pp0)
        got, _, st = d.run(steps)
        assert st == 0 and d.kernel() == "tma"
        P, Pp = d.download_field(L.FIELD_CURRENT), d.download_field(L.FIELD_PAST)
    pos, mat = O.encode_nodes(room.bid, room.mat, False)
    want, rP, rPp = O.run(pos, mat, dims, room.admittance, default_params(), [room.flat(*at)], [1], pulse,
                          [room.flat(*at)], steps, P0=P0, Pp0=Pp0, form="difference")
    assert np.array_equal(got, want) and np.array_equal(P, rP) and np.array_equal(Pp, rPp)
