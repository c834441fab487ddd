"""ClearZero with nothing, something and everything to drop, around its tile of
2048 entries; thresholds of 0 and below; infinities and NaN, which are kept;
a graph whose preparation ends with a ClearZero that drops nothing; norms whose
value does not depend on the launch."""
from __future__ import annotations

import numpy as np
import pytest

import sparqsim_gb300 as ps
from sparqsim_gb300 import _native

pytestmark = pytest.mark.gpu

U = ps.UnsignedInteger


@pytest.mark.parametrize("n", [1, 2047, 2048, 2049, 4096, 300001])
@pytest.mark.parametrize("drop", ["none", "one", "last", "most", "all"])
def test_drops(dual, n, drop):
    rng = np.random.default_rng(n)
    dual.reg("a", U, 20)
    dual.reg("b", U, 64)
    amps = (rng.normal(size=n) + 1j * rng.normal(size=n) + 1) / np.sqrt(n)
    amps[np.abs(amps) < 1e-3 / np.sqrt(n)] = 0.5
    if drop == "one":
        amps[n // 2] = 1e-9
    elif drop == "last":
        amps[-1] = 0
    elif drop == "most":
        amps[rng.random(n) < 0.9] *= 1e-12
    elif drop == "all":
        amps[:] = 1e-10j
    regs = np.stack([rng.permutation(1 << 20)[:n].astype(np.uint64), np.arange(n, dtype=np.uint64) << np.uint64(40)], axis=1)
    dual.start(regs, amps)
    first = dual.gpu.download()[0]
    for _ in range(2):
        dual.apply(ps.ClearZero())
        dual.compare(exact_amp=True)
    # the order is kept
    kept = regs[(amps.real * amps.real + amps.imag * amps.imag) >= 1e-14]
    assert np.array_equal(dual.gpu.download()[0], kept) and np.array_equal(first, regs)


@pytest.mark.parametrize("n", [10, 5000])
@pytest.mark.parametrize("eps", [0.0, -1.0, 1e-300])
def test_odd_thresholds_and_values(n, eps):
    ps.System.add_register("a", U, 20)
    st = ps.SparseState()
    amps = np.full(n, 1e-160 + 0j)
    amps[: 4] = [np.inf, np.nan, complex(0, -np.inf), complex(np.nan, 0)]
    st.upload(np.arange(n, dtype=np.uint64)[:, None], amps)
    ps.ClearZero(eps)(st)
    # x * x + y * y underflows to 0 for 1e-160, which is not below a threshold of 0 or less
    assert st.size() == (n if eps <= 0 else 4)


@pytest.mark.parametrize("idle", [0, 1, 2])
def test_graph_after_idle_clear_zeros(idle):
    """Graphs are bound to the buffers' roles. A ClearZero that drops nothing
    must count like any other: with an even number of them the preparation
    restores the roles and the replay runs, with an odd number it is refused."""
    n = 5000
    ps.System.add_register("a", U, 20)
    ps.System.add_register("q", U, 2)
    st = ps.SparseState()
    rows = np.stack([np.arange(n), np.zeros(n)], axis=1).astype(np.uint64)
    amps = np.full(n, 1 / np.sqrt(n) + 0j)
    H = ps.RY_Bool("q", 1, 0.4)

    def prepare():
        st.upload(rows, amps)
        for _ in range(idle):
            ps.ClearZero()(st)

    def apply():
        H(st)
        ps.ClearZero()(st)

    g = ps.Graph(st, apply, prepare)
    if idle == 1:
        prepare()
        with pytest.raises(_native.SparQInvalid):
            g.launch()
        return
    for _ in range(3):
        g.replay()
        ps.synchronize()
        got = st.to_dict()
        assert len(got) == 2 * n
        assert got[(7, 0)] == amps[7] * np.cos(0.2) and got[(7, 2)] == amps[7] * np.sin(0.2)


@pytest.mark.parametrize("n", [1, 255, 257, 100000, 1000003])
def test_norm(n):
    rng = np.random.default_rng(n)
    ps.System.add_register("a", U, 20)
    st = ps.SparseState()
    amps = rng.normal(size=n) + 1j * rng.normal(size=n)
    st.upload(np.arange(n, dtype=np.uint64)[:, None], amps)
    vals = {st.norm_sq() for _ in range(5)}
    assert len(vals) == 1
    want = float(np.sum(np.abs(amps.astype(np.clongdouble)) ** 2))
    # each thread's chain of n / threads sums, then 10 + 10 tree levels, all terms positive
    assert abs(vals.pop() - want) <= want * (2 * n / (256 * 608) + 24) * 2.0 ** -53 * 2
