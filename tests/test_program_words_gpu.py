"""Fused programs over five to eight key words, each word's own instantiation,
around a block of 256 entries."""
from __future__ import annotations

import numpy as np
import pytest

import sparqsim_gb300 as ps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("words", [5, 6, 7, 8])
@pytest.mark.parametrize("n", [1, 256, 257, 5000])
def test_words_of_a_program(dual, words, n):
    """All words of the state, and all but the first of a wider state."""
    rng = np.random.default_rng(words * 10000 + n)
    total = min(words + 1, 8)
    for i in range(total):
        dual.reg(f"x{i}", ps.UnsignedInteger, 60 if i % 2 else 64)
    regs = np.stack([rng.integers(0, 1 << 60, n, dtype=np.uint64) for _ in range(total)], axis=1)
    amps = rng.normal(size=n) + 1j * rng.normal(size=n)
    dual.start(regs, amps / np.linalg.norm(amps))
    used = [f"x{total - words + i}" for i in range(words)]
    chain = [ps.Add_ConstUInt_InPlace(x, 3 + i) for i, x in enumerate(used)]
    chain += [ps.Mul_UInt_UInt(used[0], used[1], used[-1]), ps.Phase_Bool(used[-1], 2, 0.3).conditioned_by_bit(used[2], 0),
              ps.Reflection_Bool(used[:2])]
    for dag in (False, True):
        dual.apply(ps.Fused(chain), dag=dag)
        dual.compare(exact_amp=True)
