"""Registers removed and added again over the same bits: the new register
reads 0 in every entry whether or not a clearing pass runs, also when the bits
were written in between by another register, an upload, another state or a
split, and after the table was cleared."""
from __future__ import annotations

import numpy as np
import pytest

import sparqsim_gb300 as ps

pytestmark = pytest.mark.gpu

U = ps.UnsignedInteger


def _start(dual, n=3000, pad=0):
    dual.reg("a", U, 16)
    for i in range(pad):
        dual.reg(f"pad{i}", U, 64)
    rng = np.random.default_rng(n)
    rows = np.concatenate([rng.permutation(1 << 16)[:n].astype(np.uint64)[:, None]]
                          + [rng.integers(0, 1 << 62, (n, 1), dtype=np.uint64) for _ in range(pad)], axis=1)
    amps = rng.normal(size=n) + 1j * rng.normal(size=n)
    dual.start(rows, amps / np.linalg.norm(amps))


@pytest.mark.parametrize("pad", [0, 1, 3])
def test_scratch_register_again_and_again(dual, pad):
    _start(dual, pad=pad)
    for i in range(4):
        dual.add_register("s", U, 20)
        dual.compare(exact_amp=True)
        dual.apply(ps.Assign("a", "s"))
        dual.compare(exact_amp=True)
        dual.remove_register("s")
        dual.apply(ps.RY_Bool("a", 1, 0.4))
        dual.compare()


def test_bits_written_by_a_wider_register_between(dual):
    _start(dual)
    dual.add_register("s", U, 8)
    dual.remove_register("s")
    dual.add_register("t", U, 30)
    dual.apply(ps.Add_ConstUInt_InPlace("t", 123456789))
    dual.apply(ps.RY_Bool("a", 0, 0.9))
    dual.remove_register("t")
    dual.add_register("s", U, 8)
    dual.apply(ps.Add_UInt_UInt_InPlace("a", "s"))
    dual.compare()


def test_unsynchronised_register_and_second_state(dual):
    """A register made without this state, then written here and dropped
    without a pass, leaves its bits set: the next one must clear them."""
    _start(dual)
    dual.add_register("s", U, 8)
    dual.remove_register("s")
    other = ps.SparseState()  # holds the register while this state never saw it zeroed
    r = ps.System.add_register("u", U, 8)
    assert r == dual.O.add_register(int(U), 8)
    dual.apply(ps.Init_Unsafe("u", 0xA5))
    ps.Init_Unsafe("u", 0x5A)(other)
    ps.System.remove_register(r)
    dual.O.remove_register_sync(dual.ora, r)  # the oracle clears it; the engine's next AddRegister has to
    ps.AddRegister("v", U, 8)(dual.gpu)
    dual.O.add_register_sync(dual.ora, int(U), 8)
    dual.compare(exact_amp=True)
    v = ps.System.resolve("v")
    assert not dual.gpu.download()[0][:, v].any()


def test_copies_sums_and_uploads():
    ps.System.add_register("a", U, 10)
    st = ps.SparseState()
    rows = np.arange(600, dtype=np.uint64)[:, None]
    st.upload(rows, np.full(600, 0.01 + 0j))
    s = ps.AddRegister("s", U, 12)(st)
    ps.Init_Unsafe("s", 7)(st)
    dirty = st.copy()            # s = 7 here
    ps.RemoveRegister("s")(st)   # cleared in st only
    ps.add_systems(st, dirty, 1.0)
    s = ps.AddRegister("s", U, 12)(st)
    assert not st.download()[0][:, s].any()
    ps.RemoveRegister("s")(st)
    c = st.copy()
    s = ps.AddRegister("s", U, 12)(c)
    assert not c.download()[0][:, s].any()
    # the table cleared and refilled: an older state's words are whatever they were
    ps.System.clear()
    for i in range(3):
        ps.System.add_register(f"w{i}", U, 64)
    st.upload(np.full((900, 3), 11, dtype=np.uint64) + np.arange(900, dtype=np.uint64)[:, None], np.full(900, 0.01 + 0j))
    ps.RemoveRegister("w2")(st)
    x = ps.AddRegister("x", U, 64)(st)
    assert not st.download()[0][:, x].any()
