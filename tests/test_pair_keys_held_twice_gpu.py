"""1-bit splits of states that hold keys several times (uploaded so), through
the one-CTA split, the hashed table (two key words, or bits of a register that
is gone) and the indexed table: the sum over a key's copies is what a split
sees, whichever copy meets which."""
from __future__ import annotations

import math

import numpy as np
import pytest

import sparqsim_gb300 as ps

pytestmark = pytest.mark.gpu

U = ps.UnsignedInteger


def _upload(n, keys, words, rng):
    ps.System.add_register("q", ps.Boolean, 1)
    ps.System.add_register("r", U, 13)
    for w in range(words - 1):
        ps.System.add_register(f"p{w}", U, 64)
    rows = np.stack([rng.integers(0, 2, n), rng.integers(0, keys, n)], axis=1).astype(np.uint64)
    pads = [(rows[:, 1] * np.uint64(0x9E3779B97F4A7C15 >> w))[:, None] for w in range(words - 1)]
    amps = rng.normal(size=n) + 1j * rng.normal(size=n)
    st = ps.SparseState()
    st.upload(np.concatenate([rows] + pads, axis=1), amps)
    return st, rows.astype(np.int64), amps


def _vector(rows, amps):
    v = np.zeros((2, 1 << 13), dtype=np.complex128)
    np.add.at(v, (rows[:, 0], rows[:, 1]), amps)
    return v


def _check(st, before, op, conditioned):
    op(st)
    regs, amps = st.download()
    got = _vector(regs[:, :2].astype(np.int64), amps)
    c, s = math.cos(0.3), math.sin(0.3)
    want = np.array([c * before[0] - s * before[1], s * before[0] + c * before[1]])
    if conditioned:
        odd = np.arange(1 << 13) & 1
        want = np.where(odd, want, before)
    # sums of at most 64 terms of size 5, each with a few roundings
    assert np.abs(got - want).max() < 64 * 5 * 8 * 2.0 ** -53


@pytest.mark.parametrize("words", [1, 2, 6])
@pytest.mark.parametrize("n,keys", [(3, 1), (60, 1), (200, 16), (256, 100), (300, 11), (2048, 300), (2049, 300),
                                    (20000, 4000), (70000, 8192)])
@pytest.mark.parametrize("conditioned", [False, True])
def test_sums_over_copies(words, n, keys, conditioned):
    st, rows, amps = _upload(n, keys, words, np.random.default_rng(n + words))
    op = ps.RY_Bool("q", 0, 0.6)
    if conditioned:
        op = op.conditioned_by_bit("r", 0)
    _check(st, _vector(rows, amps), op, conditioned)


@pytest.mark.parametrize("n,keys", [(5000, 300), (70000, 8192)])
def test_hashed_table_of_one_word(n, keys):
    """A bit of a register that is gone sends a one-word state to the hashed table."""
    ps.System.add_register("q", ps.Boolean, 1)
    ps.System.add_register("r", U, 13)
    ps.System.add_register("g", ps.Boolean, 1)
    rng = np.random.default_rng(n)
    rows = np.stack([rng.integers(0, 2, n), rng.integers(0, keys, n), np.ones(n, dtype=np.int64)], axis=1)
    amps = rng.normal(size=n) + 1j * rng.normal(size=n)
    st = ps.SparseState()
    st.upload(rows.astype(np.uint64), amps)
    ps.System.remove_register("g")
    _check(st, _vector(rows, amps), ps.RY_Bool("q", 0, 0.6), False)
