"""1-bit splits by partner lookup at the sizes where their paths change: one
CTA in shared memory up to 2048 entries, the claim table above it; target bits
that are constant (no partners), partly and fully paired; entries failing the
conditions; every pair operator, one and several key words."""
from __future__ import annotations

import math
from decimal import Decimal, localcontext

import numpy as np
import pytest

import sparqsim_gb300 as ps

pytestmark = pytest.mark.gpu

U = ps.UnsignedInteger
SIZES = [1, 2, 255, 256, 257, 1025, 2048, 2049, 8193, 65536, 70001]


def _rows(rng, n, bits, fill):
    """n distinct rows (q, r, pad): r spans its groups, q is 0 ('zero'), 1
    ('one'), both ('full') or a random subset ('some')."""
    if fill in ("zero", "one"):
        r, q = np.arange(n), np.full(n, fill == "one")
    elif fill == "full":
        r, q = np.arange(n) >> 1, np.arange(n) & 1
    else:
        pick = rng.choice(2 * n, n, replace=False)
        r, q = pick >> 1, pick & 1
    pad = rng.integers(0, 1 << bits, 2 * n, dtype=np.uint64)[r]
    rows = np.stack([q.astype(np.uint64), r.astype(np.uint64), pad], axis=1)
    p = rng.permutation(n)
    amps = rng.normal(size=n) + 1j * rng.normal(size=n)
    return rows[p], amps / np.linalg.norm(amps)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("fill", ["zero", "one", "full", "some"])
def test_pair_split_paths(dual, n, fill):
    rng = np.random.default_rng(n * 7 + len(fill))
    pad = 16 if fill == "some" else 62  # one or two key words
    dual.reg("q", ps.Boolean, 1)
    dual.reg("r", U, 18)
    dual.reg("pad", U, pad)
    rows, amps = _rows(rng, n, pad, fill)
    dual.start(rows, amps)
    th = 0.7
    rot = ps.Rot_Bool("q", 0, [math.cos(th), -math.sin(th), math.sin(th), math.cos(th)])
    dual.apply(rot)
    dual.compare(exact_amp=True)
    dual.apply(ps.Hadamard_Bool("q").conditioned_by_bit("r", 0))
    dual.compare(exact_amp=True)
    dual.apply(rot, dag=True)
    dual.compare(exact_amp=True)


@pytest.mark.parametrize("n", [5, 2048, 2049, 40000])
@pytest.mark.parametrize("words", [1, 4, 8])
def test_pair_split_key_words(dual, n, words):
    rng = np.random.default_rng(n + words)
    dual.reg("q", ps.Boolean, 1)
    dual.reg("r", U, 18)
    dual.reg("x", ps.Rational, 30)
    for w in range(words - 1):
        dual.reg(f"p{w}", U, 64)
    base, amps = _rows(rng, n, 30, "some")
    rows = np.concatenate([base] + [rng.integers(0, 1 << 62, 2 * n, dtype=np.uint64)[base[:, 1].astype(np.int64)][:, None]
                                    for _ in range(words - 1)], axis=1)
    dual.start(rows, amps)
    dual.apply(ps.CondRot_Rational_Bool("x", "q"))
    dual.compare(rel=1e-12)  # device sin/cos
    dual.apply(ps.Hadamard_Bool("q").conditioned_by_nonzeros("x"))
    dual.compare(rel=1e-12)


def _cos_sin(v, w):
    """cos and sin of 2 pi v / 2^w, from the Taylor series in 60 digits."""
    with localcontext() as ctx:
        ctx.prec = 60
        pi = Decimal("3.14159265358979323846264338327950288419716939937510582097494459230781640628620899")
        x = 2 * pi * Decimal(v) / Decimal(1 << w)
        if x > pi:
            x -= 2 * pi
        s, c, t = Decimal(0), Decimal(0), Decimal(1)
        for k in range(0, 80, 2):
            c += t
            t = t * x / (k + 1)
            s += t
            t = -t * x / (k + 2)
        return c, s


@pytest.mark.parametrize("w", [1, 2, 3, 7, 32, 53, 63, 64])
def test_condrot_angles_are_correctly_rounded_to_an_ulp(w):
    """Rotations of a lone |0> give (cos, sin): within 2^-52 relative of the
    exact turn fraction (one rounding, 2^-53, and the series' 2^-61), also next
    to the zeros, where entries below the prune threshold are dropped."""
    rng = np.random.default_rng(w)
    vals = {int(rng.integers(0, 1 << 62)) * 4 + 3 >> (64 - w) for _ in range(300)} | {0}
    for e in range(8):  # the eighths of a turn and their neighbours
        for d in (-2, -1, 0, 1, 2):
            vals.add(((e << w) // 8 + d) % (1 << w))
    ps.System.add_register("x", ps.Rational, w)
    ps.System.add_register("q", ps.Boolean, 1)
    for dag in (False, True):
        st = ps.SparseState()
        st.upload(np.array([[v, 0] for v in sorted(vals)], dtype=np.uint64), np.ones(len(vals), dtype=np.complex128))
        op = ps.CondRot_Rational_Bool("x", "q")
        (op.dag if dag else op)(st)
        got = {(int(r[0]), int(r[1])): a for r, a in zip(*st.download())}
        for v in vals:
            for bit, e in enumerate(_cos_sin(v, w)):
                if bit and dag:
                    e = -e
                a = got.get((v, bit))
                if a is None:
                    assert abs(e) < Decimal("1.0001e-7")
                else:
                    assert a.imag == 0 and abs(Decimal(float(a.real)) - e) <= abs(e) * Decimal(2) ** -52


def test_small_split_in_a_graph():
    """A small split posts its size to the host directly; a captured one must not."""
    ps.System.add_register("q", U, 6)
    st = ps.SparseState()
    rots = [ps.RY_Bool("q", b, 0.3 + b) for b in range(6)]

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
