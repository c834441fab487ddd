"""Hash grouping with a table sized for fewer groups than there are: the
insert pass gives up early and the grouping is repeated with a table for every
entry; the results are those of a table that fitted."""
from __future__ import annotations

import numpy as np
import pytest

import sparqsim_gb300 as ps
from sparqsim_gb300 import predictor

pytestmark = pytest.mark.gpu

U = ps.UnsignedInteger


@pytest.mark.parametrize("hint", [1, 700, 40000, 140000, 300000])
@pytest.mark.parametrize("members", [1, 2])
def test_too_small_tables(dual, hint, members):
    n = 300001
    rng = np.random.default_rng(hint)
    dual.reg("q", U, 4)
    dual.reg("r", U, 40)
    i = np.arange(n)
    keys = rng.permutation(1 << 20)[:n].astype(np.uint64) * np.uint64(999983)
    r = keys[i // members]
    rows = np.stack([(i % members + 5).astype(np.uint64), r], axis=1)[rng.permutation(n)]
    amps = rng.normal(size=n) + 1j * rng.normal(size=n)
    dual.start(rows, amps / np.linalg.norm(amps))
    predictor.set_hash_groups_hint(hint)
    try:
        dual.apply(ps.Hadamard_Int("q", 4))
    finally:
        predictor.set_hash_groups_hint(0)
    dual.compare(exact_amp=True)
