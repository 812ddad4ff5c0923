"""GPU: runs whose grid stays on the SMs, against the CPU oracle bit for bit.

Sizes lie around the brick splits: a brick's x vector of 4, bricks cut short on
each axis, one brick, one node of air, long and flat rooms, and the largest
number of planes a thread holds.  Fields start from random values, planes 0 and
Z-1 (never updated) included, and the step counts are odd, so that both buffers
of a halo exchange and both field roles are used."""
import os
import subprocess
import sys

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
    return v.astype({"f32": np.float32, "f64": np.float64, "f16": np.float16}[prec])


def _as_float(v):
    """Field values as numbers (BF16 comes as bit patterns): a zero on an x or y
    face may differ in sign, as in the temporally blocked runs."""
    return (v.astype(np.uint32) << 16).view(np.float32) if v.dtype == np.uint16 else v


def _check(O, dims, prec, scheme, steps, form="reference", runs=1, progress=None, captures=()):
    room = rooms.boxes_room(dims, n_boxes=3 if min(dims) > 16 else 0, edge=(4, 9), n_materials=5,
                            seed=sum(dims))
    rng = np.random.default_rng(steps)
    inside = np.flatnonzero(room.bid)
    some_air = inside.size > 0
    if not some_air:  # the closed room of 3 nodes across is all solid
        inside = np.array([room.flat(1, 1, 1)])
    pick = rng.choice(inside, 7)
    src, rec = [room.coords(int(i)) for i in pick[:3]], [room.coords(int(i)) for i in pick[3:]]
    src.append(src[0])  # a second source on one node: order matters
    types = [1, 0, 1, 1]
    pulses = rng.uniform(-1.0, 1.0, (4, steps))
    P0, Pp0 = _values(rng, room.n_nodes, prec), _values(rng, room.n_nodes, prec)
    with Domain(dims, prec) as d:
        d.set_scheme(scheme)
        d.set_voxels(room.bid, room.mat, centred=scheme == "centred")
        d.set_materials(room.admittance)
        d.set_params()
        if form != "reference":
            d.set_update_form(form)
        d.set_sources(src, types, pulses)
        d.set_receivers(rec)
        for _ in range(runs):  # the same start again: exchange tags go on
            d.upload_field(L.FIELD_CURRENT, P0)
            d.upload_field(L.FIELD_PAST, Pp0)
            if captures:
                got, slices = d.run_captures(steps, [(c, 0, dims[2] // 2) for c in captures])
            else:
                got, _, st = d.run(steps, progress=progress)
                assert st == 0
            P, Pp = d.download_field(L.FIELD_CURRENT), d.download_field(L.FIELD_PAST)
            if runs > 1 and steps % 2:
                d.flip()  # the same buffers' roles as at first
    pos, mat = O.encode_nodes(room.bid, room.mat, scheme == "centred")

    def oracle(n):
        return O.run(pos, mat, dims, room.admittance, default_params(),
                     [room.flat(*p) for p in src], types, pulses[:, :n], [room.flat(*p) for p in rec], n,
                     scheme=2 if scheme == "centred" else 0, double=prec == "f64",
                     storage=prec if prec in ("f16", "bf16") else None, P0=P0, Pp0=Pp0, form=form)
    want, rP, rPp = oracle(steps)
    assert (np.abs(want).max() > 0) == some_air
    assert np.array_equal(got, want)
    assert np.array_equal(_as_float(P), _as_float(rP))
    assert np.array_equal(_as_float(Pp), _as_float(rPp))
    if captures:
        X, Y, _ = dims
        for c, (p, _) in zip(captures, slices):
            z = oracle(c)[1].reshape(dims[2], Y, X)[dims[2] // 2]
            assert np.array_equal(p, z.astype(np.float32)), c


@pytest.mark.parametrize("dims", [(4, 4, 4), (5, 3, 7), (33, 17, 9), (64, 64, 64), (130, 31, 40),
                                  (21, 260, 12), (16, 18, 300), (301, 40, 33), (128, 120, 130)])
def test_sizes(gpu, O, dims):
    _check(O, dims, "f32", "forward", 61)


@pytest.mark.parametrize("prec", ["f32", "f64", "f16", "bf16"])
@pytest.mark.parametrize("scheme", ["forward", "centred"])
@pytest.mark.parametrize("dims", [(40, 37, 26), (90, 70, 61)])
def test_types(gpu, O, dims, prec, scheme):
    _check(O, dims, prec, scheme, 23)


def test_difference_form(gpu, O):
    _check(O, (75, 42, 31), "f32", "forward", 41, form="difference")


def test_largest_double(gpu, O):
    _check(O, (128, 100, 98), "f64", "forward", 21)


@pytest.mark.parametrize("prec", ["f32", "f16"])
def test_autotune_keeps_resident_runs(gpu, prec):
    """The autotuner times the resident launches that an automatic run of a
    small room makes (several times faster than the blocked updates of 64^3) and
    keeps them; fields and results are as before it."""
    room, steps = rooms.shoebox((64, 64, 64), seed=1), 60
    P0 = _values(np.random.default_rng(2), room.n_nodes, prec)
    with Domain(room.dims, prec) as d:
        d.set_voxels(room.bid, room.mat, centred=False)
        d.set_materials(room.admittance)
        d.set_params()
        d.set_receivers([(20, 30, 40)])
        out = []
        for tune in (False, True):
            d.upload_field(L.FIELD_CURRENT, P0)
            if tune:
                depth, _, ms = d.autotune(max_depth=4, iters=3)
                assert depth == 0 and ms > 0
                assert np.array_equal(d.download_field(L.FIELD_CURRENT), P0)
            before = L.load().pfdtd_kernel_launches()
            out.append(d.run(steps)[0])
            if tune:
                assert L.load().pfdtd_kernel_launches() - before == 1
            d.reset_fields()
    assert np.abs(out[0]).max() > 0 and np.array_equal(out[0], out[1])


@pytest.mark.parametrize("dims,resident", [((92, 90, 92), True), ((96, 96, 96), False)])
def test_double_rooms_by_size(gpu, dims, resident):
    """FP64 rooms beyond about 0.8 M nodes run faster by single steps and take
    them; on both sides of the line the run equals the z-march kernel."""
    room = rooms.boxes_room(dims, n_boxes=4, edge=(8, 30), n_materials=5, seed=3)
    P0 = _values(np.random.default_rng(1), room.n_nodes, "f64")
    out = []
    for kernel in ("auto", "zmarch"):
        with Domain(dims, "f64") as d:
            d.set_kernel(kernel)
            d.set_voxels(room.bid, room.mat, centred=False)
            d.set_materials(room.admittance)
            d.set_params()
            d.run(50)
            d.reset_fields()
            d.upload_field(L.FIELD_CURRENT, P0)
            before = L.load().pfdtd_kernel_launches()
            d.run(15)
            n = L.load().pfdtd_kernel_launches() - before
            assert (n <= 2) == (resident and kernel == "auto")
            out.append((d.download_field(L.FIELD_CURRENT), d.download_field(L.FIELD_PAST)))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


def test_repeated_run(gpu, O):
    _check(O, (52, 36, 45), "f32", "forward", 33, runs=3)


def test_chunks_with_progress(gpu, O):
    """With a callback the run is split into short launches: 120 steps in three."""
    seen = []
    _check(O, (52, 36, 45), "f32", "forward", 120, progress=lambda s, n, t: seen.append(s))
    assert seen == [0, 100]


def test_long_run_is_cut_into_launches(gpu, O):
    """A run of 2500 steps holds the SMs for about a millisecond at a time: it is
    several launches, and as the oracle has it."""
    launches = L.load().pfdtd_kernel_launches
    room, steps = rooms.shoebox((24, 24, 24), seed=2), 2500
    src, rec, pulse = (12, 12, 12), (5, 6, 7), rooms.gaussian_pulse(2500, 3.0)[None]
    with Domain(room.dims) as d:
        d.set_voxels(room.bid, room.mat, centred=False)
        d.set_materials(room.admittance)
        d.set_params()
        d.set_sources([src], [1], pulse)
        d.set_receivers([rec])
        d.run(50)
        d.reset_fields()
        before = launches()
        got, _, st = d.run(steps)
        assert st == 0 and 3 <= launches() - before <= 50
    pos, mat = O.encode_nodes(room.bid, room.mat, False)
    want, _, _ = O.run(pos, mat, room.dims, room.admittance, default_params(), [room.flat(*src)], [1],
                       pulse, [room.flat(*rec)], steps)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("dims,steps,resident", [((24, 24, 24), 2, False), ((24, 24, 24), 3, True),
                                                 ((128, 128, 128), 11, False), ((128, 128, 128), 12, True)])
def test_short_runs_take_single_steps(gpu, O, dims, steps, resident):
    """Filling and emptying the SMs costs some single steps' time: a run of fewer
    takes those, also between captures, and gives the same results."""
    launches = L.load().pfdtd_kernel_launches
    room, src, rec = rooms.shoebox(dims, seed=2), (12, 12, 12), (11, 12, 13)
    P0 = _values(np.random.default_rng(1), room.n_nodes, "f32")
    pulse = rooms.gaussian_pulse(5 * steps, 3.0)[None]
    caps = [(steps, 0, 12)] * 2 + [(2 * steps, 1, 12), (2 * steps, 2, 12)]  # three pieces
    with Domain(dims) as d:
        d.set_voxels(room.bid, room.mat, centred=False)
        d.set_materials(room.admittance)
        d.set_params()
        d.set_sources([src], [1], pulse)
        d.set_receivers([rec])
        d.run(50)  # classes, plan
        got = []
        for run in (lambda: d.run(steps)[0], lambda: d.run_captures(3 * steps, caps)[0]):
            d.reset_fields()
            d.upload_field(L.FIELD_CURRENT, P0)
            before = launches()
            got.append((run(), launches() - before, d.download_field(L.FIELD_CURRENT)))
    assert (got[0][1] == 1) == resident and (got[1][1] == 3 + len(caps)) == resident
    pos, mat = O.encode_nodes(room.bid, room.mat, False)
    for (r, _, P), n in zip(got, (steps, 3 * steps)):
        want, rP, _ = O.run(pos, mat, room.dims, room.admittance, default_params(), [room.flat(*src)],
                            [1], pulse[:, :n], [room.flat(*rec)], n, P0=P0)
        assert np.array_equal(r, want) and np.array_equal(P, rP)


def test_captures(gpu, O):
    _check(O, (52, 36, 45), "f32", "forward", 31, captures=(0, 4, 5, 31))


@pytest.mark.parametrize("place", [(0, 20, 10), (30, 20, 0)])
def test_other_rooms_take_the_general_path(gpu, O, place):
    """Inside nodes on an x face, or a source on plane 0: not resident, and as
    the oracle has it."""
    room = rooms.shoebox((48, 40, 36), seed=3)
    bid = room.bid.copy().reshape(36, 40, 48)
    if place[0] == 0:
        bid[5:30, 8:30, 0] = 27
    pulse = rooms.gaussian_pulse(40, 3.0)[None]
    with Domain(room.dims) as d:
        d.set_voxels(bid.reshape(-1), room.mat, centred=False)
        d.set_materials(room.admittance)
        d.set_params()
        d.set_sources([place], [1], pulse)
        d.set_receivers([(24, 20, 18)])
        got, _, _ = d.run(40)
        P = d.download_field(L.FIELD_CURRENT)
    pos, mat = O.encode_nodes(bid.reshape(-1), room.mat, False)
    want, rP, _ = O.run(pos, mat, room.dims, room.admittance, default_params(),
                        [room.flat(*place)], [1], pulse, [room.flat(24, 20, 18)], 40)
    assert np.array_equal(got, want) and np.array_equal(P, rP)


@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_expired_wait_is_reported(gpu, O, prec):
    """A wait bound of a nanosecond runs out in the exchange of faces: the run
    fails, with the context and the domain usable, and the next one, the bound
    restored, equals the oracle (its step tags go on after those of the run
    that broke off)."""
    room, steps = rooms.shoebox((64, 60, 56), seed=1), 40
    src, rec, pulse = (32, 30, 28), (20, 30, 40), rooms.gaussian_pulse(40, 3.0)[None]
    with Domain(room.dims, prec) as d:
        d.set_voxels(room.bid, room.mat, centred=False)
        d.set_materials(room.admittance)
        d.set_params()
        d.set_sources([src], [1], pulse)
        d.set_receivers([rec])
        L.call("pfdtd_set_wait_limit", d.handle, 1)
        for _ in range(3):
            with pytest.raises(L.PfdtdError) as e:
                d.run(2000)
            assert e.value.status == L.ERR_CUDA and "timed out" in str(e.value)
        L.call("pfdtd_set_wait_limit", d.handle, 0)
        d.reset_fields()
        got, _, st = d.run(steps)
        assert st == 0
        P = d.download_field(L.FIELD_CURRENT)
    pos, mat = O.encode_nodes(room.bid, room.mat, False)
    want, rP, _ = O.run(pos, mat, room.dims, room.admittance, default_params(), [room.flat(*src)], [1],
                        pulse, [room.flat(*rec)], steps, double=prec == "f64")
    assert np.abs(want).max() > 0 and np.array_equal(got, want) and np.array_equal(P, rP)


_REFUSED = """
import sys
import numpy as np
from tests.test_resident_gpu import _refusal_run
from parallelfdtd_gb300 import _lib
before = _lib.load().pfdtd_kernel_launches()
out = _refusal_run()
np.savez(sys.argv[1], *out, launches=_lib.load().pfdtd_kernel_launches() - before)
"""


def _refusal_run():
    room, steps = rooms.shoebox((48, 40, 36), seed=1), 70
    with Domain(room.dims) as d:
        d.set_voxels(room.bid, room.mat, centred=False)
        d.set_materials(room.admittance)
        d.set_params()
        d.set_sources([(24, 20, 18)], [1], rooms.gaussian_pulse(steps, 3.0)[None])
        d.set_receivers([(20, 10, 30)])
        a = d.run(steps)[0]
        P = d.download_field(L.FIELD_CURRENT)
        d.reset_fields()
        b, caps = d.run_captures(steps, [(0, 0, 18), (30, 1, 20), (70, 2, 24)])
        d.reset_fields()
        seen = []
        c = d.run(steps, progress=lambda s, n, t: seen.append(s))[0]
        assert seen == [0]
    return [a, P, b, c] + [p for p, _ in caps]


@pytest.mark.parametrize("code", [720, 701, 801])
def test_refused_cooperative_launch(gpu, tmp_path, code):
    """Where the runtime refuses a cooperative launch (a stand-in for the call
    answers with its error codes: too large, out of resources, not supported),
    runs take single steps and give the same results."""
    src, lib, out = tmp_path / "refuse.cpp", tmp_path / "refuse.so", tmp_path / "out.npz"
    src.write_text('extern "C" int cudaLaunchCooperativeKernel(...) { return %d; }\n' % code)
    subprocess.run(["g++", "-shared", "-fPIC", "-o", str(lib), str(src)], check=True)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, LD_PRELOAD=str(lib), PYTHONPATH=root)
    r = subprocess.run([sys.executable, "-c", _REFUSED, str(out)], cwd=root, env=env, timeout=120,
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    got = np.load(out)
    assert got["launches"] > 3 * 2 * 70  # update and step I/O of every step
    for i, v in enumerate(_refusal_run()):
        assert np.array_equal(got["arr_%d" % i], v), i


@pytest.mark.parametrize("scheme", ["forward", "centred"])
@pytest.mark.parametrize("prec,sample", [("f32", np.nan), ("f32", -np.inf), ("f64", np.inf), ("f16", 1e6)])
def test_values_not_finite_take_single_steps(gpu, O, scheme, prec, sample):
    """A source sample that is not finite (as the fields store it) reaches the
    faces, and from there the flat-index neighbours in the next rows and planes,
    where the reference has it: such a run takes single steps."""
    room, steps, src = rooms.shoebox((28, 20, 24), seed=2), 14, (26, 18, 4)
    recs = [(1, 3, 5), (2, 18, 4), (25, 1, 5), (13, 10, 12)]
    pulse = rooms.gaussian_pulse(steps, 3.0)[None].copy()
    pulse[0, 4] = sample
    with Domain(room.dims, prec) as d:
        d.set_scheme(scheme)
        d.set_voxels(room.bid, room.mat, centred=scheme == "centred")
        d.set_materials(room.admittance)
        d.set_params()
        d.set_sources([src], [1], pulse)
        d.set_receivers(recs)
        before = L.load().pfdtd_kernel_launches()
        got, _, _ = d.run(steps)
        assert L.load().pfdtd_kernel_launches() - before >= 2 * steps
        P = d.download_field(L.FIELD_CURRENT)
    pos, mat = O.encode_nodes(room.bid, room.mat, scheme == "centred")
    want, rP, _ = O.run(pos, mat, room.dims, room.admittance, default_params(), [room.flat(*src)], [1], pulse,
                        [room.flat(*r) for r in recs], steps, scheme=2 if scheme == "centred" else 0,
                        double=prec == "f64", storage="f16" if prec == "f16" else None)
    assert not np.isfinite(want).all()
    assert np.array_equal(got, want, equal_nan=True) and np.array_equal(P, rP, equal_nan=True)


@pytest.mark.parametrize("what", ["lambda", "material"])
def test_rooms_that_gain_energy_take_single_steps(gpu, O, what):
    """A lambda beyond the scheme's limit, or a material with a negative
    admittance, may end in values that are not finite: single steps, as the
    oracle has it to the overflow and beyond."""
    room, steps = rooms.shoebox((20, 18, 16), seed=2), 400
    table = room.admittance.copy()
    params = default_params(lam=0.75 if what == "lambda" else None)
    if what == "material":
        table[:] = -1.2
    src, rec, pulse = (10, 9, 8), [(3, 4, 5), (17, 2, 13)], rooms.gaussian_pulse(steps, 3.0)[None]
    with Domain(room.dims) as d:
        d.set_voxels(room.bid, room.mat, centred=False)
        d.set_materials(table)
        d.set_params(params)
        d.set_sources([src], [1], pulse)
        d.set_receivers(rec)
        before = L.load().pfdtd_kernel_launches()
        got, _, _ = d.run(steps)
        assert L.load().pfdtd_kernel_launches() - before >= 2 * steps
        P = d.download_field(L.FIELD_CURRENT)
    pos, mat = O.encode_nodes(room.bid, room.mat, False)
    want, rP, _ = O.run(pos, mat, room.dims, table, params, [room.flat(*src)], [1], pulse,
                        [room.flat(*r) for r in rec], steps)
    assert not np.isfinite(want).all()
    assert np.array_equal(got, want, equal_nan=True) and np.array_equal(P, rP, equal_nan=True)
