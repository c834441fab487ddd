"""Entries read on another stream right after a call has returned: ClearZero,
1-bit splits, new and reset states have stored theirs by then. Elementwise
operators, which return no size, are not waited for."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

import sparqsim_gb300 as ps

pytestmark = pytest.mark.gpu

U = ps.UnsignedInteger


class _Array:
    def __init__(self, ptr, n, typestr):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (n,), "typestr": typestr, "version": 3}


def _read(st, stream):
    """Key words and amplitudes as `stream` sees them now."""
    import torch
    n = st.size()
    keys, amp = st.device_arrays()
    with torch.cuda.stream(stream):
        out = [torch.as_tensor(_Array(p, n, "<i8"), device="cuda").clone() for p in keys]
        out.append(torch.as_tensor(_Array(amp, n, "<c16"), device="cuda").clone())
    stream.synchronize()
    return out


def _same(st, stream):
    import torch
    now = _read(st, stream)
    ps.synchronize()
    for a, b in zip(now, _read(st, stream)):
        if a.is_complex():
            a, b = torch.view_as_real(a), torch.view_as_real(b)
        assert torch.equal(a, b)


@pytest.fixture
def other():
    import torch
    return torch.cuda.Stream()


@pytest.mark.parametrize("n", [1, 700, 2048, 2049, 100_000, 1 << 22])
def test_clear_zero(other, n):
    ps.System.add_register("a", U, 22)
    ps.System.add_register("p", U, 64)
    rng = np.random.default_rng(n)
    st = ps.SparseState()
    for step in range(6):
        amps = rng.normal(size=n) + 1j
        amps[rng.random(n) < 0.3] = 1e-9
        st.upload(np.stack([rng.permutation(n), rng.integers(0, 1 << 60, n)], axis=1).astype(np.uint64), amps)
        ps.ClearZero()(st)
        assert st.size() == (np.abs(amps) > 1e-3).sum()
        _same(st, other)
        ps.ClearZero()(st)  # nothing goes
        _same(st, other)


@pytest.mark.parametrize("words", [1, 5])
@pytest.mark.parametrize("n", [3, 256, 257, 2048, 5000, 300_000])
def test_splits(other, n, words):
    ps.System.add_register("q", U, 3)
    ps.System.add_register("a", U, 20)
    for w in range(words - 1):
        ps.System.add_register(f"p{w}", U, 64)
    rng = np.random.default_rng(n)
    st = ps.SparseState()
    st.upload(np.concatenate([np.zeros((n, 1)), rng.permutation(1 << 20)[:n, None]]
                             + [rng.integers(0, 1 << 50, (n, 1))] * (words - 1), axis=1).astype(np.uint64),
              rng.normal(size=n) + 0.5j)
    for step in range(12):
        ps.RY_Bool("q", step % 3, 0.3 + 0.1 * step)(st)
        _same(st, other)


@pytest.mark.parametrize("words", [1, 8])
def test_new_and_reset_states(other, words):
    for w in range(words):
        ps.System.add_register(f"p{w}", U, 64)
    st = ps.SparseState()
    for step in range(20):
        fresh = ps.SparseState()
        keys_amp = _read(fresh, other)
        assert all(int(k[0]) == 0 for k in keys_amp[:-1]) and complex(keys_amp[-1][0]) == 1
        for w in range(words):
            ps.Init_Unsafe(f"p{w}", step + 1)(st)
        ps.GlobalPhase(1j)(st)
        st.reset()
        keys_amp = _read(st, other)
        assert all(int(k[0]) == 0 for k in keys_amp[:-1]) and complex(keys_amp[-1][0]) == 1
