"""CPU: what a domain holds outside the library (no device needed)."""
import pytest

from parallelfdtd_gb300 import _lib as L
from parallelfdtd_gb300.domain import Domain


def test_captures_on_a_closed_domain_allocate_nothing(monkeypatch):
    """run_captures of a closed domain fails before it takes pinned memory,
    which nothing would give back."""
    d = Domain.__new__(Domain)
    d._h, d._pinned, d.dims, d.n_rec, d.precision = None, (None, 0), (8, 8, 8), 0, L.F32
    calls = []
    monkeypatch.setattr(L, "call", lambda name, *args: calls.append(name))
    with pytest.raises(RuntimeError):
        d.run_captures(10, [(5, 0, 4)])
    assert calls == [] and d._pinned == (None, 0)
