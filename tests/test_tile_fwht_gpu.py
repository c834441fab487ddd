"""The 256-slot tile form of Hadamard_Int (exact-sum arithmetic, single pass)
at its edges: every width that it takes, groups that are empty, lone, partly
filled and full, last tiles and chunks that are not full, cached ranges after a
split, batched widths side by side; against the oracle, keys bit-exact and
amplitudes within the exact-sum bound (1e-12 of the largest)."""
from __future__ import annotations

import numpy as np
import pytest

import sparqsim_gb300 as ps

pytestmark = pytest.mark.gpu

U = ps.UnsignedInteger


@pytest.fixture(autouse=True)
def exact_sum(dual):
    ps.set_fwht_arithmetic("exact-sum")
    dual.relaxed = True


def _state(rng, n, groups, fill):
    S = 1 << n
    there = rng.random((groups, S)) < fill
    there[np.arange(groups), rng.integers(0, S, groups)] = True
    if groups > 2:
        there[1] = True  # a full group among the others
    r, q = np.nonzero(there)
    p = rng.permutation(r.size)
    amps = rng.normal(size=r.size) + 1j * rng.normal(size=r.size)
    return q[p].astype(np.uint64), r[p].astype(np.uint64), amps / np.linalg.norm(amps)


@pytest.mark.parametrize("n", [5, 6, 7, 8])
@pytest.mark.parametrize("groups", [1, 7, 33, 129, 1500])
@pytest.mark.parametrize("fill", [0.0, 0.1, 0.6, 1.0])
def test_tile_widths(dual, n, groups, fill):
    rng = np.random.default_rng(n * 1000 + groups + int(10 * fill))
    dual.reg("q", U, n)
    dual.reg("r", U, 11)
    q, r, amps = _state(rng, n, groups, fill)
    dual.start(np.stack([q, r], axis=1), amps)
    H = ps.Hadamard_Int("q", n)
    dual.apply(H)
    dual.compare()
    # back over the cached ranges, then once more over what that leaves
    dual.apply(ps.Phase_Bool("r", 0, 0.3))
    dual.apply(H)
    dual.compare()
    dual.apply(H)
    dual.compare()


@pytest.mark.parametrize("lo,hi,instances", [(1, 8, 300), (3, 5, 40), (8, 8, 9), (2, 2, 1000)])
def test_tile_batched_widths(dual, lo, hi, instances):
    """Instances of different widths: every width's groups share a chunk."""
    rng = np.random.default_rng(instances)
    dual.reg("q", U, 8)
    dual.reg("w", U, 4)
    dual.reg("t", U, 10)
    rows, amps = [], []
    for t in range(instances):
        n = int(rng.integers(lo, hi + 1))
        for q in rng.choice(1 << n, int(rng.integers(1, (1 << n) + 1)), replace=False):
            rows.append((int(q), n, t))
            amps.append(complex(rng.normal(), rng.normal()))
    amps = np.array(amps)
    dual.start(np.array(rows, dtype=np.uint64), amps / np.linalg.norm(amps))
    H = ps.Hadamard_Int_Batched("q", "w", 8)
    H(dual.gpu)
    for n in range(lo, hi + 1):  # the oracle: one conditioned Hadamard per width
        dual.O.apply(dual.ora, ps.Hadamard_Int("q", n).conditioned_by_value("w", n).spec(False))
    dual.compare()
    H(dual.gpu)
    for n in range(lo, hi + 1):
        dual.O.apply(dual.ora, ps.Hadamard_Int("q", n).conditioned_by_value("w", n).spec(False))
    dual.compare()
