"""GPU: sources and receivers between single steps, against the CPU oracle.

Source counts around the 32 that one warp injects at a time, with nodes that
carry several sources (their order decides: hard ones overwrite, soft ones
add), and receiver counts up to past one block's threads."""
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


@pytest.mark.parametrize("n_src,n_rec", [(1, 1), (2, 32), (32, 33), (33, 5), (70, 1100)])
@pytest.mark.parametrize("kernel", ["tma", "zmarch"])
@pytest.mark.parametrize("prec", ["f32", "f16"])
def test_many_sources_and_receivers(gpu, O, n_src, n_rec, kernel, prec):
    room = rooms.shoebox((32, 28, 24), seed=2)
    rng = np.random.default_rng(n_src)
    steps = 60
    air = room.air_nodes()
    nodes = rng.choice(air[:max(1, n_src // 3)], n_src)  # about three sources a node
    rec = rng.choice(air, n_rec)
    types = rng.integers(0, 2, n_src)
    pulses = rng.uniform(-1.0, 1.0, (n_src, steps))
    with Domain(room.dims, prec) as d:
        d.set_kernel(kernel)
        d.set_voxels(room.bid, room.mat, centred=False)
        d.set_materials(room.admittance)
        d.set_params()
        d.set_sources([room.coords(int(i)) for i in nodes], types, pulses)
        d.set_receivers([room.coords(int(i)) for i in rec])
        got, _, _ = d.run(steps)
        P = d.download_field(L.FIELD_CURRENT)
    pos, mat = O.encode_nodes(room.bid, room.mat, False)
    want, rP, _ = O.run(pos, mat, room.dims, room.admittance, default_params(), nodes, types, pulses,
                        rec, steps, storage=None if prec == "f32" else prec)
    assert np.abs(want).max() > 0
    assert np.array_equal(got, want)
    assert np.array_equal(P, rP)
