"""1-bit splits of states that hold bits of registers that are gone: they are
found once, and the note is dropped when the bits may have gone."""
from __future__ import annotations

import numpy as np
import pytest

import sparqsim_gb300 as ps

pytestmark = pytest.mark.gpu

U = ps.UnsignedInteger


def _state(n=70000, value=3):
    ps.System.add_register("q", ps.Boolean, 1)
    ps.System.add_register("r", U, 17)
    ps.System.add_register("g", U, 2)
    rng = np.random.default_rng(n)
    rows = np.stack([np.arange(n) & 1, np.arange(n) >> 1, np.full(n, value)], axis=1).astype(np.uint64)
    amps = rng.normal(size=n) + 1j * rng.normal(size=n)
    st = ps.SparseState()
    st.upload(rows, amps)
    ps.System.remove_register("g")
    return st, rows, amps


def _launches(st):
    """Kernels of a split and its inverse; the entries are as before."""
    keys, amps = st.download()
    op = ps.RY_Bool("q", 0, 0.7)
    before = ps.launch_count()
    op(st)
    n = ps.launch_count() - before
    op.dag(st)
    k2, a2 = st.download()
    o, o2 = (np.lexsort(k[:, :2].T) for k in (keys, k2))
    assert np.array_equal(keys[o, :2], k2[o2, :2]) and np.abs(amps[o] - a2[o2]).max() < 1e-14
    return n


def test_found_once():
    st, _, _ = _state(value=0)
    indexed = _launches(st)
    ps.System.clear()
    st, rows, amps = _state()
    first = _launches(st)
    again = _launches(st)
    assert indexed < again < first
    assert _launches(st.copy()) == again  # the copy holds the bits too
    ps.AddRegister("w", U, 1)(st)
    ps.RemoveRegister("w")(st)  # clears one of the two bits only
    assert _launches(st) == first
    assert _launches(st) == again


@pytest.mark.parametrize("how", ["upload", "reset", "cleared"])
def test_dropped_with_the_bits(how):
    st, _, _ = _state(value=0)
    indexed = _launches(st)
    ps.System.clear()
    st, rows, amps = _state()
    first = _launches(st)
    assert _launches(st) < first
    if how == "cleared":
        ps.AddRegister("w", U, 2)(st)
        ps.RemoveRegister("w")(st)
    elif how == "reset":
        st.reset()
        ps.Hadamard_Int("r", 12)(st)
    else:
        st.upload(rows[:, :2], amps)
    assert _launches(st) == indexed


def test_captured():
    st, rows, amps = _state()
    rots = [ps.RY_Bool("q", 0, 0.3 + i) for i in range(4)]

    def prepare():
        r = ps.System.add_register("g", U, 2)
        st.upload(rows, amps)
        ps.System.remove_register(r)

    def apply():
        for r in rots:
            r(st)

    prepare()
    ref = st.copy()
    for r in rots:
        r(ref)
    g = ps.Graph(st, apply, prepare)
    for _ in range(3):
        g.replay()
        ps.synchronize()
        assert st.to_dict() == ref.to_dict()
