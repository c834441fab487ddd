"""Elementwise programs where the kernel form changes: fields of at most 32
bits (32-bit arithmetic) and wider ones, one to eight key words in use (also
when a state has more words than the program touches), sizes around two
entries per thread, odd tails, and conditions that are merged per word. Every
operator bit-exact against the oracle, forward and undone."""
from __future__ import annotations

import numpy as np
import pytest

import sparqsim_gb300 as ps

pytestmark = pytest.mark.gpu

U = ps.UnsignedInteger
BIG = 152 * 2048 * 2  # entries from which a thread takes two


def _ops(theta):
    q = ps.QRAMCircuit_qutrit(6, 8, np.random.default_rng(3).integers(0, 256, 64, dtype=np.uint64))
    ops = [ps.Add_UInt_UInt("a", "b", "c"), ps.Sub_UInt_UInt("a", "b", "c"), ps.Mul_UInt_UInt("a", "b", "c"),
           ps.And_UInt_UInt("a", "b", "c"), ps.Or_UInt_UInt("a", "b", "c"), ps.Xor_UInt_UInt("a", "b", "c"),
           ps.Less_UInt_UInt("a", "b", "f"), ps.Add_UInt_UInt_InPlace("a", "c"), ps.Add_UInt_ConstUInt("a", 12345, "c"),
           ps.Add_ConstUInt_InPlace("c", 987654321987), ps.Mult_UInt_ConstUInt("a", 77, "c"),
           ps.Add_Mult_UInt_ConstUInt_InPlace("b", 0x123456789, "c"), ps.Neg_UInt("a", "c"), ps.IsZero_UInt("f", "g"),
           ps.Assign("a", "b"), ps.Swap_General_General("a", "b"), ps.X_Bool("c", 2), ps.FlipBools("c"),
           ps.ShiftLeft_InPlace("c", 3), ps.ShiftRight_InPlace("c", 5), ps.GetRowAddr("a", "b", 9, "c"),
           ps.GetDataAddr("a", "b", "f", 5, "c"), ps.Phase_Bool("c", 1, theta),
           ps.ZeroConditionalPhaseFlip(["f", "g"]), ps.Reflection_Bool(["f", "a"], True)]
    return ops, q


@pytest.mark.parametrize("w", [7, 8, 31, 32, 33, 60])
@pytest.mark.parametrize("n", [1, 2, 255, 1001])
def test_every_width(dual, w, n):
    rng = np.random.default_rng(w * 100 + n)
    for name, width in (("a", w), ("b", w), ("c", w), ("f", 1), ("g", 1), ("pad", 40), ("pad2", 64)):
        dual.reg(name, U, width)
    regs = np.stack([rng.integers(0, 1 << width, n, dtype=np.uint64) for width in (w, w, w, 1, 1, 40)]
                    + [np.arange(n, dtype=np.uint64)], axis=1)
    amps = rng.normal(size=n) + 1j * rng.normal(size=n)
    dual.start(regs, amps / np.linalg.norm(amps))
    ops, q = _ops(0.3)
    dual.O.register_qram(q)
    ops.append(ps.QRAMLoad(q, "a", "c") if w >= 8 else ps.Assign("b", "c"))
    for op in ops:
        dual.apply(op)
        dual.compare(exact_amp=True)
        dual.apply(op.conditioned_by_nonzeros("f"), dag=True)
        dual.compare(exact_amp=True)


@pytest.mark.parametrize("words", [1, 2, 3, 4, 6, 8])
def test_words_in_use(dual, words):
    """A chain touching one field in each key word, and one touching the first
    and last word only."""
    rng = np.random.default_rng(words)
    n = 777
    for i in range(words):
        dual.reg(f"x{i}", U, 60 if i % 2 else 64)
    regs = np.stack([rng.integers(0, 1 << 60, n, dtype=np.uint64) for _ in range(words)], axis=1)
    amps = rng.normal(size=n) + 1j * rng.normal(size=n)
    dual.start(regs, amps / np.linalg.norm(amps))
    chain = [ps.Add_ConstUInt_InPlace(f"x{i}", 3 + i) for i in range(words)]
    chain += [ps.Assign("x0", f"x{words - 1}")] if words > 1 else []
    for c in (chain, [chain[0], chain[-1]], [ps.GlobalPhase(1j)]):
        for op in c:
            dual.O.apply(dual.ora, op.spec(False))
        ps.Fused(c)(dual.gpu)
        dual.compare(exact_amp=True)


@pytest.mark.parametrize("n", [BIG - 1, BIG, BIG + 1])
def test_two_entries_per_thread(dual, n):
    rng = np.random.default_rng(n)
    for name, width in (("a", 30), ("b", 30), ("c", 20), ("f", 1)):
        dual.reg(name, U, width)
    regs = np.stack([np.arange(n, dtype=np.uint64)] + [rng.integers(0, 1 << w, n, dtype=np.uint64) for w in (30, 20, 1)],
                    axis=1)
    amps = rng.normal(size=n) + 1j * rng.normal(size=n)
    dual.start(regs, amps / np.linalg.norm(amps))
    for op in (ps.Mul_UInt_UInt("a", "b", "c"), ps.Phase_Bool("c", 3, 0.4).conditioned_by_all_ones("f"),
               ps.Add_UInt_UInt_InPlace("c", "b")):
        dual.apply(op)
    dual.compare(exact_amp=True)


@pytest.mark.parametrize("cond", ["value", "bit", "ones", "nonzero", "several", "never", "clash"])
def test_merged_conditions(dual, cond):
    rng = np.random.default_rng(5)
    n = 3000
    for name, width in (("a", 3), ("b", 2), ("c", 1), ("d", 50), ("e", 3)):
        dual.reg(name, U, width)
    regs = np.stack([rng.integers(0, 1 << w, n, dtype=np.uint64) for w in (3, 2, 1)]
                    + [np.arange(n, dtype=np.uint64), rng.integers(0, 8, n, dtype=np.uint64)], axis=1)
    amps = rng.normal(size=n) + 1j * rng.normal(size=n)
    dual.start(regs, amps / np.linalg.norm(amps))

    def with_cond(op):
        if cond == "value":
            op.conditioned_by_value([("a", 5), ("e", 2)])
        elif cond == "bit":
            op.conditioned_by_bit([("a", 2), ("a", 0), ("e", 1)])
        elif cond == "ones":
            op.conditioned_by_all_ones(["b", "c", "e"])
        elif cond == "nonzero":
            op.conditioned_by_nonzeros(["a", "b", "e"])
        elif cond == "several":
            op.conditioned_by_nonzeros("b").conditioned_by_bit("a", 1).conditioned_by_value("e", 6)
        elif cond == "never":
            op.conditioned_by_value("a", 9)
        else:
            op.conditioned_by_value("a", 5).conditioned_by_bit("a", 1)  # 5 has bit 1 clear
        return op

    for op in (with_cond(ps.Add_ConstUInt_InPlace("d", 1)), with_cond(ps.Phase_Bool("d", 0, 1.1))):
        dual.apply(op)
        dual.compare(exact_amp=True)
    dual.apply(with_cond(ps.Rot_Bool("d", 49, [0.6, -0.8, 0.8, 0.6])))
    dual.compare(exact_amp=True)
