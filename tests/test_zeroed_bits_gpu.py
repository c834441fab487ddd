"""Registers over reused bits that the call which made or moved their last
owner wrote itself: AddRegisterWithHadamard, CombineRegister that moves both
fields, and copies and sums of such states. The next register reads 0 in every
entry."""
from __future__ import annotations

import numpy as np
import pytest

import sparqsim_gb300 as ps

pytestmark = pytest.mark.gpu

U = ps.UnsignedInteger


def _state(n=300, width=10):
    ps.System.add_register("a", U, width)
    st = ps.SparseState()
    st.upload(np.arange(n, dtype=np.uint64)[:, None], np.full(n, 0.01 + 0j))
    return st


def _reads_zero(st, name, width):
    r = ps.AddRegister(name, U, width)(st)
    assert not st.download()[0][:, r].any()


@pytest.mark.parametrize("bits", [1, 3, 14])
def test_register_made_with_a_hadamard_and_dropped(bits):
    st = _state()
    ps.AddRegisterWithHadamard("k", U, bits)(st)
    assert st.size() == 300 << bits
    ps.System.remove_register("k")  # without a pass over the state
    _reads_zero(st, "v", bits)


def test_copy_of_a_state_after_the_hadamard():
    st = _state()
    ps.AddRegisterWithHadamard("k", U, 3)(st)
    d = st.copy()
    ps.RemoveRegister("k")(st)  # cleared in st only
    _reads_zero(d, "v", 3)


def _combined(st):
    """A register f = 150 over bits that an earlier removal cleared."""
    ps.AddRegister("s", U, 20)(st)
    ps.AddRegister("f", U, 4)(st)
    ps.RemoveRegister("s")(st)  # s's bits: cleared, free
    ps.AddRegister("p", U, 10)(st)
    ps.AddRegister("g", U, 4)(st)  # both over s's bits, so that f and g are not adjacent in order
    ps.Init_Unsafe("f", 9)(st)
    ps.Init_Unsafe("g", 6)(st)
    ps.RemoveRegister("p")(st)  # cleared, free: where the combined register lands
    ps.CombineRegister("f", "g")(st)


def test_combined_register_over_bits_cleared_before():
    st = _state()
    _combined(st)
    f = ps.System.resolve("f")
    assert (st.download()[0][:, f] == 150).all()
    ps.System.remove_register("f")
    _reads_zero(st, "v", 8)


def test_sum_with_such_a_state():
    st = _state()
    other = st.copy()
    ps.Add_ConstUInt_InPlace("a", 500)(st)
    ps.AddRegister("s", U, 20)(other)
    ps.RemoveRegister("s")(other)  # the bits are 0 in other
    _combined(st)
    ps.System.remove_register("f")
    ps.add_systems(other, st, 0.5)
    assert other.size() == 600
    _reads_zero(other, "v", 8)


def test_bits_stay_known_after_a_removal():
    """Removing with the state and adding again launches no clearing pass."""
    st = _state()
    ps.AddRegister("s", U, 12)(st)
    ps.RemoveRegister("s")(st)
    before = ps.launch_count()
    ps.AddRegister("s", U, 12)(st)
    assert ps.launch_count() == before
