"""1-bit splits of states whose registers span few enough bits of one key word
to index the partner table: edges of the rule, conditions (also on the target
bit), keys held twice, bits of registers that are gone, captured splits."""
from __future__ import annotations

import math

import numpy as np
import pytest

import sparqsim_gb300 as ps

pytestmark = pytest.mark.gpu

U = ps.UnsignedInteger


@pytest.mark.parametrize("n", [2049, 4096, 38913, 155648, 155649, 262143])
@pytest.mark.parametrize("fill", ["zero", "full", "some"])
@pytest.mark.parametrize("pad", [5, 6])  # 24 bits, and 25: the rule's edge
def test_against_oracle(dual, n, fill, pad):
    rng = np.random.default_rng(n + pad)
    dual.reg("r", U, 18)
    dual.reg("q", U, 1)
    dual.reg("pad", U, pad)
    if fill == "some":
        pick = rng.choice(1 << 19, n, replace=False)
    else:
        pick = np.arange(n) if fill == "full" else np.arange(n) << 1
    r, q = (pick >> 1) & 0x3FFFF, pick & 1
    p = pick >> 19
    rows = np.stack([r, q, p], axis=1).astype(np.uint64)[rng.permutation(n)]
    amps = rng.normal(size=n) + 1j * rng.normal(size=n)
    dual.start(rows, amps / np.linalg.norm(amps))
    rot = ps.Rot_Bool("q", 0, [math.cos(0.7), -math.sin(0.7), math.sin(0.7), math.cos(0.7)])
    dual.apply(rot)
    dual.compare(exact_amp=True)
    dual.apply(ps.Hadamard_Bool("q").conditioned_by_bit("r", 0))
    dual.compare(exact_amp=True)
    dual.apply(rot, dag=True)
    dual.compare(exact_amp=True)


def _sums(st):
    regs, amps = st.download()
    out = {}
    for r, a in zip(regs, amps):
        key = tuple(int(v) for v in r)
        out[key] = out.get(key, 0) + a
    return out


def test_condition_on_the_target_bit():
    """Entries failing through their target bit are copied and are no partners."""
    ps.System.add_register("q", ps.Boolean, 1)
    ps.System.add_register("r", U, 14)
    st = ps.SparseState()
    n = 1 << 14
    rows = np.array([[q, r] for q in (0, 1) for r in range(n)], dtype=np.uint64)
    rng = np.random.default_rng(3)
    amps = rng.normal(size=2 * n)
    st.upload(rows, amps.astype(np.complex128))
    ps.RY_Bool("q", 0, 0.6).conditioned_by_bit("q", 0)(st)
    got = _sums(st)
    c, s = math.cos(0.3), math.sin(0.3)
    for r in range(0, n, 37):
        assert got[(0, r)] == pytest.approx(amps[r] - s * amps[n + r], abs=1e-14 * 4)
        assert got[(1, r)] == pytest.approx(c * amps[n + r], abs=1e-14 * 4)


def test_keys_held_twice_stay_linear():
    """A key uploaded several times: the sum over its copies is what a split sees."""
    ps.System.add_register("q", ps.Boolean, 1)
    ps.System.add_register("r", U, 12)
    rng = np.random.default_rng(4)
    n = 20000
    rows = np.stack([rng.integers(0, 2, n), rng.integers(0, 1 << 12, n)], axis=1).astype(np.uint64)
    amps = rng.normal(size=n) + 1j * rng.normal(size=n)
    st = ps.SparseState()
    st.upload(rows, amps)
    before = np.zeros((2, 1 << 12), dtype=np.complex128)
    np.add.at(before, (rows[:, 0].astype(int), rows[:, 1].astype(int)), amps)
    ps.RY_Bool("q", 0, 0.6)(st)
    c, s = math.cos(0.3), math.sin(0.3)
    want = np.array([c * before[0] - s * before[1], s * before[0] + c * before[1]])
    after = np.zeros_like(before)
    for (q, r), a in _sums(st).items():
        after[q, r] = a
    # sums of at most 20 terms of size 5
    assert np.abs(after - want).max() < 20 * 5 * 8 * 2.0 ** -53


@pytest.mark.parametrize("stray", [False, True])
def test_bits_of_a_removed_register(stray):
    """Entries that differ only in a register that is gone are distinct; they
    have their own partners, as through the hashed table."""
    ps.System.add_register("q", ps.Boolean, 1)
    ps.System.add_register("r", U, 12)
    ps.System.add_register("g", U, 2)
    rows = np.array([[q, r, g if stray else 0] for g in range(4 if stray else 1) for r in range(1 << 12)
                     for q in (0, 1)], dtype=np.uint64)
    rng = np.random.default_rng(5)
    amps = rng.normal(size=len(rows)) + 1j * rng.normal(size=len(rows))
    st = ps.SparseState()
    st.upload(rows, amps)
    ps.System.remove_register("g")
    ps.Hadamard_Bool("q")(st)
    assert st.size() == len(rows)
    ps.Hadamard_Bool("q")(st)
    assert st.size() == len(rows)
    got = np.sort_complex(st.download()[1])
    assert np.abs(got - np.sort_complex(amps)).max() < 1e-14


def test_captured_splits():
    ps.System.add_register("q", U, 13)
    st = ps.SparseState()
    rots = [ps.RY_Bool("q", b, 0.3 + b) for b in range(13)] + [ps.RY_Bool("q", 3, 0.2)]

    def apply():
        for r in rots:
            r(st)

    g = ps.Graph(st, apply, st.reset)
    ref = ps.SparseState()
    for r in rots:
        r(ref)
    for _ in range(3):
        g.replay()
        ps.synchronize()
        assert st.to_dict() == ref.to_dict()
