"""The Python copy of the register table against the engine's own answers, over
random additions, removals, type changes and clears, up to the most registers."""
from __future__ import annotations

from ctypes import byref, c_uint32

import numpy as np
import pytest

import sparqsim_gb300 as ps
from sparqsim_gb300._native import SQ_MAX_REGISTERS, call


def _engine():
    n = c_uint32()
    call("sq_system_register_count", byref(n))
    rows = []
    for i in range(n.value):
        v = [c_uint32() for _ in range(5)]
        call("sq_system_register_info", i, *map(byref, v))
        rows.append(tuple(x.value for x in v))
    return rows


@pytest.mark.parametrize("seed", range(4))
def test_copy_follows_the_table(seed):
    rng = np.random.default_rng(seed)
    names = {}
    for step in range(300):
        k = int(rng.integers(0, 10))
        if k < 6 and len(names) < SQ_MAX_REGISTERS:
            nm = f"r{int(rng.integers(0, 200))}"
            if nm not in names:
                names[nm] = ps.System.add_register(nm, ps.UnsignedInteger, int(rng.integers(0, 9)))
        elif k < 8 and names:
            nm = sorted(names)[int(rng.integers(0, len(names)))]
            ps.System.remove_register(nm if k == 6 else names[nm])
            del names[nm]
            with pytest.raises(ValueError):
                ps.System.get_id(nm)
        elif k == 8 and names:
            ps.System.set_register_type(sorted(names)[0], ps.Rational)
        elif rng.random() < 0.1:
            ps.System.clear()
            names = {}
        rows = _engine()
        assert ps.System.register_count() == len(rows)
        assert [tuple(map(int, ps.System._info(i))) for i in range(len(rows))] == rows
        assert sorted(ps.System.active_ids()) == sorted(names.values())
        for nm, rid in names.items():
            assert ps.System.get_id(nm) == rid == ps.System.resolve(nm) and ps.System.name_of(nm) == nm
        with pytest.raises(ps.SparQInvalid):
            ps.System.size_of(len(rows))
