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
