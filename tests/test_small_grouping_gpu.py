"""Grouping of small states in one CTA, now from one entry on: sizes around its
batches, lone groups only, mixed groups, entries failing the conditions, and
real and complex unitaries with amplitudes that are not finite."""
from __future__ import annotations

import numpy as np
import pytest

import sparqsim_gb300 as ps

pytestmark = pytest.mark.gpu

U = ps.UnsignedInteger


@pytest.mark.parametrize("n", [1, 2, 31, 1023, 1024, 1025, 4095, 4096, 8192, 8193])
@pytest.mark.parametrize("shape", ["lone", "mixed", "full"])
@pytest.mark.parametrize("cond", [False, True])
def test_small_states(dual, n, shape, cond):
    rng = np.random.default_rng(n + len(shape))
    dual.reg("q", U, 3)
    dual.reg("r", U, 13)
    dual.reg("c", U, 1)
    dual.reg("pad", U, 60)
    if shape == "lone":
        r, q = np.arange(n) % 8192, np.full(n, 5)
        c = np.arange(n) // 8192
    elif shape == "full":
        r, q, c = np.arange(n) // 8, np.arange(n) % 8, np.zeros(n, dtype=int)
    else:
        pick = rng.choice(3 * n, n, replace=False)
        r, q, c = pick // 8, pick % 8, (pick // 8) % 2
    pad = rng.integers(0, 1 << 60, 8192, dtype=np.uint64)
    rows = np.stack([q, r, c, pad[r]], axis=1).astype(np.uint64)[rng.permutation(n)]
    amps = rng.normal(size=n) + 1j * rng.normal(size=n)
    dual.start(rows, amps / np.linalg.norm(amps))
    m, _ = np.linalg.qr(rng.normal(size=(8, 8)))
    m2, _ = np.linalg.qr(rng.normal(size=(8, 8)) + 1j * rng.normal(size=(8, 8)))
    ops = [ps.Hadamard_Int("q", 3), ps.Rot_GeneralUnitary("q", m2), ps.Rot_GeneralUnitary("q", m)]
    for op in ops:
        dual.apply(op.conditioned_by_value("c", 0) if cond else op)
        dual.compare(exact_amp=True)
    dual.apply(ops[2], dag=True)
    dual.compare(exact_amp=True)


@pytest.mark.parametrize("bad", [np.inf, np.nan])
@pytest.mark.parametrize("op", ["unitary", "ry"])
def test_real_matrices_and_values_that_are_not_finite(bad, op):
    """inf * 0 is NaN: the shortcut for real matrices must not hide it."""
    ps.System.add_register("q", U, 1 if op == "ry" else 2)
    ps.System.add_register("r", U, 10)
    st = ps.SparseState()
    amps = np.ones(600, dtype=np.complex128)
    amps[0] = bad
    st.upload(np.stack([np.zeros(600), np.arange(600)], axis=1).astype(np.uint64), amps)
    if op == "ry":
        ps.RY_Bool("q", 0, 0.6)(st)
    else:
        ps.Rot_GeneralUnitary("q", np.kron([[0.6, -0.8], [0.8, 0.6]], np.eye(2)))(st)
    d = st.to_dict()
    assert np.isnan(d[(0, 0)].imag) and d[(0, 5)] == (np.cos(0.3) if op == "ry" else 0.6)
