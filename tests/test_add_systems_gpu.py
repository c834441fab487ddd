"""add_systems by hash join: sizes around its tiles, no / some / all keys in
common, cancelling sums, one to eight key words, a source with fewer key words
than the table now has, and states that hold a key twice, which take the sort
path. Keys and amplitudes bit-exact against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import sparqsim_gb300 as ps

pytestmark = pytest.mark.gpu

U = ps.UnsignedInteger


def _other(dual, rows, amps):
    from oracle import oracle as O
    g, o = ps.SparseState(), O.OracleState()
    g.upload(rows, amps)
    o.set(rows, amps)
    return g, o


def _amps(rng, n):
    return (rng.normal(size=n) + 1j * rng.normal(size=n)) / np.sqrt(max(n, 1))


@pytest.mark.parametrize("n0,n1", [(1, 1), (1, 3000), (2047, 1), (2048, 2048), (2049, 2047), (5000, 40)])
@pytest.mark.parametrize("common", ["none", "some", "all"])
@pytest.mark.parametrize("coef", [1.0, -1.0, 0.37])
def test_join(dual, n0, n1, common, coef):
    rng = np.random.default_rng(n0 * 7 + n1)
    dual.reg("a", U, 20)
    dual.reg("b", U, 64)
    keys = rng.permutation(1 << 16)[: n0 + n1]
    first = {"none": n0, "some": n0 // 2, "all": 0}[common]
    k0, k1 = keys[:n0], keys[first:first + n1]
    rows0 = np.array([[int(k), int(k) * 0x9E3779B97F4A7C15 % (1 << 64)] for k in k0], dtype=np.uint64)
    rows1 = np.array([[int(k), int(k) * 0x9E3779B97F4A7C15 % (1 << 64)] for k in rng.permutation(k1)], dtype=np.uint64)
    a0 = _amps(rng, n0)
    a1 = _amps(rng, n1)
    if coef == -1.0:  # common keys cancel exactly
        at = {int(k): v for k, v in zip(rows0[:, 0], a0)}
        a1 = np.array([at.get(int(k), v) for k, v in zip(rows1[:, 0], a1)])
    dual.start(rows0, a0)
    g, o = _other(dual, rows1, a1)
    ps.add_systems(dual.gpu, g, coef)
    dual.O.add_systems(dual.ora, o, coef)
    dual.compare(exact_amp=True)
    ps.Add_ConstUInt_InPlace("a", 1)(dual.gpu)  # the result is a state like any other
    dual.O.apply(dual.ora, ps.Add_ConstUInt_InPlace("a", 1).spec(False))
    dual.compare(exact_amp=True)


@pytest.mark.parametrize("where", ["current", "added", "both"])
def test_keys_held_twice(dual, where):
    rng = np.random.default_rng(3)
    dual.reg("a", U, 12)
    k0, k1 = rng.permutation(4096)[:900], rng.permutation(4096)[:700]
    if where != "added":
        k0 = np.concatenate([k0, k0[:5]])
    if where != "current":
        k1 = np.concatenate([k1, k1[100:103]])
    dual.start(k0.astype(np.uint64)[:, None], _amps(rng, k0.size))
    g, o = _other(dual, k1.astype(np.uint64)[:, None], _amps(rng, k1.size))
    ps.add_systems(dual.gpu, g, 0.5)
    dual.O.add_systems(dual.ora, o, 0.5)
    dual.compare(rel=1e-12)


@pytest.mark.parametrize("words", [1, 3, 8])
def test_key_words_and_late_registers(dual, words):
    rng = np.random.default_rng(words)
    dual.reg("a", U, 60)
    rows = rng.permutation(1 << 12)[:2500].astype(np.uint64)[:, None]
    dual.start(rows, _amps(rng, 2500))
    g, o = _other(dual, rows[::2], _amps(rng, 1250))  # made while the table had one word
    for w in range(words - 1):
        dual.add_register(f"p{w}", U, 62)
        dual.O.apply(dual.ora, ps.Add_ConstUInt_InPlace(f"p{w}", 0).spec(False))
    ps.add_systems(dual.gpu, g, 0.25)
    dual.O.add_systems(dual.ora, o, 0.25)
    dual.compare(exact_amp=True)
