"""Timed cases of the sparse-state engine, each one pass of a program as a user
writes it over the public operators: gate circuits, QRAM state preparation,
register circuits (eager and replayed as one CUDA graph), batched noisy
trajectories, the QDA and CKS linear-solver walks (tridiagonal and through
QRAM), fused register arithmetic and single multi-bit splits.

listed() names the cases, draw(rng) gives further ones of the same ranges,
prepare(case, seed) builds the inputs and what a program keeps between calls,
run(state) is one pass and returns its outputs, work(case) the bytes and
operations the pass cannot do without, exact(case, seed) its result in 64-bit
numpy where that is cheap.

The order of a state's entries is not fixed after a split, so results come
back by basis index: a dense vector (or a table over one register) that the
state's amplitudes and key words are scattered into on the library's stream.
"""
import ctypes
import math

import numpy as np
import torch

import sparqsim_gb300 as ps
from sparqsim_gb300 import _native, cks, cks_qram, qda, qram_encoding, workloads

QDA_STEPS = 2000  # schedule length of the QDA walks


# ------------------------------------------------------------------ read-out
_ext = None


def _stream():
    global _ext
    if _ext is None:
        p = ctypes.c_void_p()
        _native.call("sq_get_stream", ctypes.byref(p))
        _ext = torch.cuda.ExternalStream(p.value)
    return _ext


class _Device:
    """A device array of the engine as torch sees it (kept alive by `owner`)."""

    def __init__(self, ptr, n, typestr, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (n,), "typestr": typestr, "version": 3}


def _arrays(st):
    """(key words as int64 tensors, amplitudes as complex128), the state's own buffers."""
    n = st.size()
    keys, amp = st.device_arrays()
    return ([torch.as_tensor(_Device(p, n, "<i8", st), device="cuda") for p in keys],
            torch.as_tensor(_Device(amp, n, "<c16", st), device="cuda"))


def _dense(st, bits):
    """The state vector over the low `bits` bits of the first key word."""
    with torch.cuda.stream(_stream()):
        keys, amp = _arrays(st)
        out = torch.zeros(1 << bits, dtype=torch.complex128, device="cuda")
        k = keys[0]
        if len(keys) > 1 or bits < 63:
            k = k & ((1 << bits) - 1)
        out.index_copy_(0, k, amp)
        return torch.view_as_real(out)


def _table(st, size, index):
    """(key words by index, amplitudes by index), index = index(first key word)."""
    with torch.cuda.stream(_stream()):
        keys, amp = _arrays(st)
        i = index(keys[0])
        words = []
        for k in keys:
            w = torch.zeros(size, dtype=torch.int64, device="cuda")
            words.append(w.index_copy_(0, i, k))
        out = torch.zeros(size, dtype=torch.complex128, device="cuda")
        out.index_copy_(0, i, amp)
        return {"words": words, "amps": torch.view_as_real(out)}


def _pairs(v):
    v = np.ascontiguousarray(v, dtype=np.complex128)
    return v.view(np.float64).reshape(-1, 2)


def _fwht(x, bits):
    """Orthonormal Walsh-Hadamard transform over the last axis."""
    x = x.copy()
    n = 1 << bits
    for q in range(bits):
        y = x.reshape(x.shape[:-1] + (n >> (q + 1), 2, 1 << q))
        a, b = y[..., 0, :].copy(), y[..., 1, :].copy()
        y[..., 0, :], y[..., 1, :] = a + b, a - b
    return x / math.sqrt(n)


def _register_table(*regs):
    """The register table of a program: cleared, then (name, type, width) in order."""
    ps.System.clear()
    for name, typ, width in regs:
        ps.System.add_register(name, typ, width)
    ps.set_fwht_arithmetic("exact-sum")


# ------------------------------------------------------------------ gates
# A layered ansatz on one qubit register: RY on `rotated` bits of each layer
# (every second one controlled by another bit), a chain of controlled X and a
# controlled phase. From |0...0> at the sizes of a first program or a unit
# test, where each call's latency is the time; from a dense state at
# simulation sizes, where each rotation is a split and merge of every entry.
def _gate_angles(c, seed):
    rng = np.random.default_rng([seed, 1, c["bits"]])
    return rng, rng.uniform(0.1, math.pi - 0.1, (c["layers"], c["rotated"])), rng.uniform(0, 2 * math.pi, c["layers"])


def _gate_bits(c, layer):
    n = c["bits"]
    return [(layer + j * max(1, n // c["rotated"])) % n for j in range(c["rotated"])]


def _gate_start(c, rng):
    n = 1 << c["bits"]
    v = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    return v / np.linalg.norm(v)


def gates_prepare(c, seed):
    _register_table(("q", ps.UnsignedInteger, c["bits"]))
    rng, theta, phi = _gate_angles(c, seed)
    ops = []
    for l in range(c["layers"]):
        for j, b in enumerate(_gate_bits(c, l)):
            g = ps.RY_Bool("q", b, float(theta[l, j]))
            if j % 2:
                g.conditioned_by_bit("q", (b + 1) % c["bits"])
            ops.append(g)
        for b in range(0, c["bits"] - 1, 2):
            ops.append(ps.X_Bool("q", b + 1).conditioned_by_bit("q", b))
        ops.append(ps.Phase_Bool("q", 0, float(phi[l])).conditioned_by_bit("q", c["bits"] - 1))
    init = None
    if c["dense"]:
        n = 1 << c["bits"]
        init = ps.SparseState(capacity=n)
        k = rng.permutation(n).astype(np.uint64)
        init.upload(k.reshape(-1, 1), _gate_start(c, np.random.default_rng([seed, 2]))[k.astype(np.int64)])
    return {"f": "gates", "c": c, "ops": ops, "init": init, "st": ps.SparseState()}


def gates_run(s):
    st = s["st"]
    if s["init"] is not None:
        st = s["init"].copy()
    else:
        st.reset()
    for op in s["ops"]:
        op(st)
    return _dense(st, s["c"]["bits"])


def gates_work(c):
    n, E = 1 << c["bits"], 24.0
    per_layer = c["rotated"] * 2 * n * E + ((c["bits"] // 2) * 16 + 40) * n
    if c["dense"]:
        return {"bytes": c["layers"] * per_layer + n * (2 * E + 16), "flops": c["layers"] * c["rotated"] * 12 * n}
    return {"bytes": per_layer + n * 16, "flops": c["layers"] * c["rotated"] * 12 * n}


def gates_exact(c, seed):
    n = 1 << c["bits"]
    _, theta, phi = _gate_angles(c, seed)
    k = np.arange(n)
    v = np.zeros(n, dtype=np.complex128)
    v[0] = 1
    if c["dense"]:
        v = _gate_start(c, np.random.default_rng([seed, 2]))
    for l in range(c["layers"]):
        for j, b in enumerate(_gate_bits(c, l)):
            co, si = math.cos(theta[l, j] / 2), math.sin(theta[l, j] / 2)
            w = v.reshape(n >> (b + 1), 2, 1 << b)
            r = np.stack([co * w[:, 0] - si * w[:, 1], si * w[:, 0] + co * w[:, 1]], axis=1).reshape(-1)
            if j % 2:
                r = np.where((k >> ((b + 1) % c["bits"])) & 1, r, v)
            v = r
        for b in range(0, c["bits"] - 1, 2):
            v = v[np.where((k >> b) & 1, k ^ (1 << (b + 1)), k)]
        on = ((k >> (c["bits"] - 1)) & 1 & k).astype(bool)
        v = np.where(on, v * np.exp(1j * phi[l]), v)
    return _pairs(v)


# ------------------------------------------------------------------ state preparation through QRAM
# Amplitude encoding of a table: Hadamard on the address register, QRAM load
# of the angles, a rotation of the flag qubit by the loaded angle, and the
# load undone. The flag starts at 0, so the rotation is a fan-out.
def _rotation_table(c, seed):
    return np.random.default_rng([seed, 3]).integers(0, 1 << (c["word_bits"] - 2), 1 << c["address_bits"], dtype=np.uint64)


def qram_rotation_prepare(c, seed):
    _register_table(("i", ps.UnsignedInteger, c["address_bits"]), ("flag", ps.Boolean, 1),
                    ("x", ps.Rational, c["word_bits"]))
    table = ps.QRAMCircuit_qutrit(c["address_bits"], c["word_bits"], _rotation_table(c, seed))
    load = ps.QRAMLoad(table, "i", "x")
    ops = [ps.Hadamard_Int_Full("i"), load, ps.CondRot_Rational_Bool("x", "flag"), load]
    return {"f": "qram_rotation", "c": c, "ops": ops, "table": table, "st": ps.SparseState()}


def qram_rotation_run(s):
    st = s["st"]
    st.reset()
    for op in s["ops"]:
        op(st)
    return _dense(st, s["c"]["address_bits"] + 1)


def qram_rotation_work(c):
    n, K = 1 << c["address_bits"], (c["address_bits"] + 1 + c["word_bits"] + 63) // 64
    E = 8.0 * K + 16
    return {"bytes": n * E + n * (16 + 8) + 3 * n * E + 2 * n * (16 + 8) + 2 * n * 40, "flops": 10.0 * n}


def qram_rotation_exact(c, seed):
    x = _rotation_table(c, seed).astype(np.float64) / (1 << c["word_bits"]) * 2 * math.pi
    return _pairs(np.concatenate([np.cos(x), np.sin(x)]) / math.sqrt(1 << c["address_bits"]))


# ------------------------------------------------------------------ register circuit
# The register circuit at scale (a 20, b 32, c 32, t 32 bits; 2^(2h) entries
# at the peak) from the uniform superposition over a: each layer's arithmetic
# on 2^h entries, the Hadamard that fans them out to the peak and the next
# layer's that merges them, so that the result is the register table over a.
# Replayed as one CUDA graph, as the repository's benchmark runs it, or issued
# operator by operator.
def register_circuit_prepare(c, seed):
    circ = workloads.RegisterCircuit(h=c["h"], layers=c["layers"], seed=seed).build()
    ps.set_fwht_arithmetic("exact-sum")
    n = 1 << c["h"]
    regs = np.zeros((n, 4), dtype=np.uint64)
    regs[:, 0] = np.arange(n)
    amps = np.full(n, 2.0 ** (-c["h"] / 2), dtype=np.complex128)
    st = ps.SparseState(capacity=n)

    def start():
        st.upload(regs, amps)

    def apply():
        for mid in circ.mid:
            mid(st)
            circ.H(st)
            circ.H(st)

    s = {"f": "register_circuit", "c": c, "circ": circ, "st": st, "start": start, "apply": apply, "graph": None}
    if c["replay"]:
        s["graph"] = ps.Graph(st, apply, start)
    return s


def register_circuit_run(s):
    if s["graph"] is not None:
        s["graph"].replay()
    else:
        s["start"]()
        s["apply"]()
    mask = (1 << s["c"]["h"]) - 1
    return _table(s["st"], mask + 1, lambda k: k & mask)


def register_circuit_work(c):
    n, E = 1 << c["h"], 32.0
    return {"bytes": c["layers"] * 2 * (n * n + n) * E + c["layers"] * n * 68, "flops": c["layers"] * 2 * c["h"] * 2.0 * n * n}


def register_circuit_exact(c, seed):
    rng = np.random.default_rng(seed)
    table = rng.integers(0, 1 << 32, 1 << workloads.RegisterCircuit.TABLE_BITS, dtype=np.uint64)
    thetas = rng.uniform(0.0, 2 * math.pi, c["layers"])
    a = np.arange(1 << c["h"], dtype=np.uint64)
    b, cc = np.zeros_like(a), np.zeros_like(a)
    m32 = np.uint64(0xFFFFFFFF)
    amp = np.full(a.size, 2.0 ** (-c["h"] / 2), dtype=np.complex128)
    for th in thetas:
        b ^= table[a.astype(np.int64)]
        cc = (cc + ((a * b) & m32)) & m32
        amp = np.where(cc & np.uint64(1), amp * np.exp(1j * th), amp)
    return {"words": [(a | (b << np.uint64(20))).astype(np.int64), cc.astype(np.int64)], "amps": _pairs(amp)}


# ------------------------------------------------------------------ hidden-function circuit
# Period finding / collision search: Hadamard, a table lookup into b, Hadamard,
# with a fresh random table per layer, so that each value of b is shared by
# none, one or a few addresses and the groups of the second Hadamard are
# partly filled. Both butterfly arithmetics.
def _hidden_tables(c, seed):
    rng = np.random.default_rng([seed, 4])
    return (rng.integers(0, 1 << c["word_bits"], (c["layers"], 1 << c["bits"]), dtype=np.uint64),
            rng.uniform(0, 2 * math.pi, c["layers"]))


def hidden_prepare(c, seed):
    _register_table(("a", ps.UnsignedInteger, c["bits"]), ("b", ps.UnsignedInteger, c["word_bits"]))
    tables, theta = _hidden_tables(c, seed)
    H = ps.Hadamard_Int("a", c["bits"])
    ops, keep = [], []
    for t, th in zip(tables, theta):
        q = ps.QRAMCircuit_qutrit(c["bits"], c["word_bits"], t)
        keep.append(q)
        ops += [H, ps.QRAMLoad(q, "a", "b"), ps.Phase_Bool("b", 0, float(th)), H]
    return {"f": "hidden", "c": c, "ops": ops, "keep": keep, "st": ps.SparseState()}


def hidden_run(s):
    ps.set_fwht_arithmetic(s["c"]["arithmetic"])
    st = s["st"]
    st.reset()
    for op in s["ops"]:
        op(st)
    return _dense(st, s["c"]["bits"] + s["c"]["word_bits"])


def hidden_work(c):
    n, E = 1 << c["bits"], 24.0
    peak = n * min(n, 1 << c["word_bits"]) * 0.8
    return {"bytes": (2 * c["layers"] - 1) * peak * E + 16.0 * (n << c["word_bits"]), "flops": (2 * c["layers"] - 1) * peak * 2 * c["bits"]}


def hidden_exact(c, seed):
    if c["bits"] + c["word_bits"] > 24:
        return None
    tables, theta = _hidden_tables(c, seed)
    n = 1 << c["bits"]
    a, b = np.arange(n), np.zeros(n, dtype=np.int64)
    amp = np.full(n, 2.0 ** (-c["bits"] / 2), dtype=np.complex128)
    for t, th in zip(tables, theta):
        b ^= t.astype(np.int64)
        amp = np.where(b & 1, amp * np.exp(1j * th), amp)
    v = np.zeros((1 << c["word_bits"], n), dtype=np.complex128)
    v[b, a] = amp
    return _pairs(_fwht(v, c["bits"]).reshape(-1))


# ------------------------------------------------------------------ noisy trajectories
# Thousands of noisy instances in one state, per-instance Hadamard widths
# h_t in [h_min, h_max] and per-instance Pauli noise; the last split merged
# back, so that an instance's result is its registers over a.
def trajectories_prepare(c, seed):
    w = workloads.NoisyTrajectories(n_traj=c["instances"], layers=c["layers"], h_min=c["h_min"], h_max=c["h_max"],
                                    seed=seed).build_batched()
    ps.set_fwht_arithmetic("exact-sum")
    return {"f": "trajectories", "c": c, "w": w, "H": ps.Hadamard_Int_Batched("a", "w", c["h_max"]),
            "st": ps.SparseState()}


def trajectories_run(s):
    w, st = s["w"], s["st"]
    w.run_batched(st)
    s["H"](st)
    tb, tmask = w.t_bits, (1 << w.t_bits) - 1
    return _table(st, 1 << (tb + 8), lambda k: (k & tmask) | (((k >> (tb + 4)) & 255) << tb))


def trajectories_work(c):
    hs = range(c["h_min"], c["h_max"] + 1)
    # instances whose (b, c) collide interfere, which leaves about 0.85 of the entries
    peak = 0.85 * c["instances"] * sum(4.0 ** h for h in hs) / len(hs)
    return {"bytes": c["layers"] * 2 * peak * 24.0 + c["instances"] * 24.0, "flops": c["layers"] * 2 * peak * 2 * (c["h_max"] - 0.5)}


def trajectories_exact(c, seed):
    w = workloads.NoisyTrajectories(n_traj=c["instances"], layers=c["layers"], h_min=c["h_min"], h_max=c["h_max"], seed=seed)
    n, u = c["instances"], np.uint64
    m16 = u(0xFFFF)
    a = np.tile(np.arange(256, dtype=np.uint64), (n, 1))
    live = a < (u(1) << w.widths.reshape(-1, 1))
    b, cc = np.zeros_like(a), np.zeros_like(a)
    amp = np.where(live, 2.0 ** (-w.widths.astype(np.float64).reshape(-1, 1) / 2), 0).astype(np.complex128)
    for th, m in zip(w.thetas, w.masks):
        b ^= w.table[a.astype(np.int64)]
        cc ^= (a * b) & m16
        amp = np.where(cc & u(1), amp * np.exp(1j * th), amp)
        par = np.zeros(a.shape, dtype=np.int64)
        regs = [a, b, cc]
        for j in range(3):
            regs[j] = regs[j] ^ m[:, j:j + 1]
            x = regs[j] & m[:, j + 3:j + 4]
            for sh in (8, 4, 2, 1):
                x = x ^ (x >> u(sh))
            par ^= (x & u(1)).astype(np.int64)
        a, b, cc = regs
        amp = np.where(par == 1, -amp, amp)
    tb = w.t_bits
    t = np.arange(n, dtype=np.uint64).reshape(-1, 1)
    key = t | (w.widths.reshape(-1, 1) << u(tb)) | (a << u(tb + 4)) | (b << u(tb + 20)) | (cc << u(tb + 36))
    idx = ((key & u((1 << tb) - 1)) | (((key >> u(tb + 4)) & u(255)) << u(tb))).astype(np.int64)[live]
    words, out = np.zeros(1 << (tb + 8), dtype=np.uint64), np.zeros(1 << (tb + 8), dtype=np.complex128)
    words[idx], out[idx] = key[live], amp[live]
    return {"words": [words.view(np.int64)], "amps": _pairs(out)}


# ------------------------------------------------------------------ QDA walks
# One step of the discrete-adiabatic solver of a tridiagonal system in the
# middle of its schedule, with the prune and normalisation that the driver
# does after each step: tens of splits, nearly all conditioned, between short
# runs of elementwise operators.
def qda_prepare(c, seed):
    rng = np.random.default_rng([seed, 5])
    alpha, beta = float(rng.uniform(2.1, 2.6)), -1.0
    ps.System.clear()
    ps.set_fwht_arithmetic("exact-sum")
    st = ps.SparseState()
    run = qda.Runner(st)
    qda.declare_registers(run, c["bits"])
    run.op(ps.Hadamard_Int_Full("main_reg"))
    enc = (qda.BlockEncodingTridiagonal("main_reg", "anc_UA", alpha, beta), qda.StatePrepHadamard("main_reg"))
    s = {"f": "qda", "c": c, "enc": enc, "kappa": (alpha + 2) / (alpha - 2 * math.cos(math.pi / ((1 << c["bits"]) + 1)))}
    for i in range(c["warm"]):
        _qda_step(s, run, i)
    s["init"] = st
    return s


def _qda_step(s, run, i):
    qda.WalkS(*s["enc"], *qda.REGS, i / QDA_STEPS, s["kappa"], 1.3).apply(run)
    run.op(ps.ClearZero())
    run.op(ps.Normalize())


def qda_run(s):
    st = s["init"].copy()
    _qda_step(s, qda.Runner(st), s["c"]["warm"])
    return _dense(st, s["c"]["bits"] + 8)


def qda_work(c):
    # about 460 entry visits (in or out of a split, 24 bytes each) per row and
    # step once the walk's ancilla sectors are filled
    n = 1 << c["bits"]
    return {"bytes": 460.0 * n * 24, "flops": 460.0 * n * 8}


# The same solver through the QRAM encoding of a banded matrix and right-hand
# side: hundreds of engine calls per step on a few thousand entries.
def qda_qram_prepare(c, seed):
    ps.System.clear()
    ps.set_fwht_arithmetic("exact-sum")
    n = 1 << c["bits"]
    A = qram_encoding.banded_spd(n, min(4, n // 2), c["kappa"], seed=seed)
    b = np.random.default_rng([seed, 6]).standard_normal(n)
    solver = qram_encoding.QDAviaQRAM(A, b)
    st = ps.SparseState()
    run = qda.Runner(st)
    solver.start(run)
    for i in range(c["warm"]):
        solver.step(run, i, QDA_STEPS)
    return {"f": "qda_qram", "c": c, "solver": solver, "init": st}


def qda_qram_run(s):
    st = s["init"].copy()
    s["solver"].step(qda.Runner(st), s["c"]["warm"], QDA_STEPS)
    out, prob = ps.get_output(st, [], list(qram_encoding.REGS))
    return {"vector": _pairs(out), "probability": prob}


def qda_qram_work(c):
    # entries grow about as n^1.7; about 1500 operators a step visit them
    n = 1 << c["bits"]
    peak = 12.0 * n ** 1.7
    return {"bytes": 800.0 * c["bits"] / 4 * peak * 0.25 * 48, "flops": 900.0 * peak}


# ------------------------------------------------------------------ CKS walks
# One term of the LCU sum: two quantum-walk steps and the accumulation into
# the solution state (add_systems), then the solution read out by
# post-selection as the driver does at a log point.
def cks_prepare(c, seed):
    rng = np.random.default_rng([seed, 7])
    ps.System.clear()
    ps.set_fwht_arithmetic("exact-sum")
    mat, spec = cks.make_tridiagonal_matrix_spec(float(rng.uniform(2.1, 2.6)), -1.0, 1 << c["bits"], 32)
    obj = cks.LCU_Container_NoiseFree_Tridiagonal(mat, spec, c["kappa"], 0.01)
    st = obj.step_state
    ps.Hadamard_Int(obj.GetInputVecReg(), c["bits"])(st)
    cks.TridiagParityPhase(obj.GetInputVecReg())(st)
    ps.ClearZero()(st)
    obj.quantum_walk_obj.FirstStep(obj.run)
    obj.Step()
    obj.Step()
    return {"f": "cks", "c": c, "obj": obj}


def cks_run(s):
    obj, n = s["obj"], 1 << s["c"]["bits"]
    obj.Step()
    st, prob = obj.PartialTrace_Nondestructive()
    info = ps.System._info(ps.System.resolve(obj.GetInputVecReg()))
    with torch.cuda.stream(_stream()):
        keys, amp = _arrays(st)
        out = torch.zeros(n, dtype=torch.complex128, device="cuda")
        out.index_copy_(0, (keys[info[3]] >> info[4]) & (n - 1), amp)
        return {"solution": torch.view_as_real(out), "probability": prob}


def cks_work(c):
    # 20 entries per row; per term eight splits, their elementwise oracles and
    # one merge of two states, 6 key words (tridiagonal) per entry
    n = 1 << c["bits"]
    return {"bytes": 20.0 * n * (8 * 2 + 20 * 0.5 + 3) * 64, "flops": 20.0 * n * 100}


# The general walk, its banded matrix and column lists read from QRAM.
def cks_qram_prepare(c, seed):
    ps.System.clear()
    ps.set_fwht_arithmetic("exact-sum")
    A = cks_qram.banded_symmetric(1 << c["bits"], c["half_bandwidth"], 100.0, seed=seed)
    obj = cks_qram.LCU_Container_NoiseFree(cks_qram.SparseMatrix(A, 24), c["kappa"], 0.01, checks=False)
    st = obj.step_state
    ps.Hadamard_Int(obj.GetInputVecReg(), c["bits"])(st)
    ps.ClearZero()(st)
    obj.quantum_walk_obj.FirstStep(obj.run)
    obj.Step()
    obj.Step()
    return {"f": "cks_qram", "c": c, "obj": obj}


cks_qram_run = cks_run


def cks_qram_work(c):
    n = 1 << c["bits"]
    m = 11.0 * {1: 4, 2: 8}.get(c["half_bandwidth"], 16)  # entries per row, 11 per element slot
    return {"bytes": m * n * (8 * 2 + 56 * 0.5 + 3) * 48, "flops": m * n * 100}


# ------------------------------------------------------------------ register arithmetic
# Compute, phase, uncompute on a large state: one fused chain of arithmetic,
# comparison and QRAM operators, a conditional phase, and the chain undone.
# The keys end where they began; entry order is kept, so the state's own
# buffers are the result.
_M32 = np.uint64(0xFFFFFFFF)


def _arithmetic_start(c, seed):
    rng = np.random.default_rng([seed, 8])
    n = c["entries"]
    regs = np.empty((n, 5), dtype=np.uint64)
    regs[:, 0] = rng.integers(0, 1 << 20, n, dtype=np.uint64)
    regs[:, 1:4] = rng.integers(0, 1 << 32, (n, 3), dtype=np.uint64)
    regs[:, 4] = 0
    amps = rng.standard_normal(2 * n).view(np.complex128) / math.sqrt(2 * n)
    table = rng.integers(0, 1 << 32, 1 << 20, dtype=np.uint64)
    return regs, amps, table, rng.integers(1, 1 << 31, 4), float(rng.uniform(0, 2 * math.pi))


def arithmetic_prepare(c, seed):
    _register_table(("a", ps.UnsignedInteger, 20), ("b", ps.UnsignedInteger, 32), ("x", ps.UnsignedInteger, 32),
                    ("t", ps.UnsignedInteger, 32), ("flag", ps.Boolean, 1))
    regs, amps, table, const, theta = _arithmetic_start(c, seed)
    q = ps.QRAMCircuit_qutrit(20, 32, table)
    st = ps.SparseState(capacity=c["entries"])
    st.upload(regs, amps)
    chain = [ps.QRAMLoad(q, "a", "b"), ps.Add_UInt_UInt_InPlace("b", "x"), ps.Mul_UInt_UInt("a", "x", "t"),
             ps.Add_ConstUInt_InPlace("x", int(const[0])), ps.ShiftLeft_InPlace("t", 7),
             ps.Add_Mult_UInt_ConstUInt_InPlace("b", int(const[1]) | 1, "x"), ps.Assign("x", "t"),
             ps.Less_UInt_UInt("b", "t", "flag")][:c["chain"] - 1] + [ps.Less_UInt_UInt("x", "t", "flag")]
    if not c["fused"]:
        forward, back = chain, [(op, True) for op in reversed(chain)]
    else:
        f = ps.Fused(chain)
        forward, back = [f], [(f, True)]
    return {"f": "arithmetic", "c": c, "st": st, "table": q, "forward": forward, "back": back,
            "phase": ps.Phase_Bool("flag", 0, theta)}


def arithmetic_run(s):
    st = s["st"]
    for op in s["forward"]:
        op(st)
    s["phase"](st)
    for op, _ in s["back"]:
        op.dag(st)
    keys, amp = _arrays(st)
    return {"words": keys, "amps": torch.view_as_real(amp)}


def arithmetic_work(c):
    n = float(c["entries"])
    passes = 2 if c["fused"] else 2 * c["chain"]
    return {"bytes": passes * n * (32 if c["fused"] else 24) + n * 40 + (1 << 22), "flops": n * 6}


def arithmetic_exact(c, seed):
    regs, amps, table, const, theta = _arithmetic_start(c, seed)
    a, b, x, t = (regs[:, j].copy() for j in range(4))
    u = np.uint64

    def shift(v):
        return ((v << u(7)) | (v >> u(25))) & _M32
    flag = np.zeros(a.size, dtype=bool)
    for k in range(c["chain"] - 1):
        if k == 0:
            b ^= table[a.astype(np.int64)]
        elif k == 1:
            x = (x + b) & _M32
        elif k == 2:
            t ^= (a * x) & _M32
        elif k == 3:
            x = (x + u(const[0])) & _M32
        elif k == 4:
            t = shift(t)
        elif k == 5:
            x = (x + ((b * u(int(const[1]) | 1)) & _M32)) & _M32
        elif k == 6:
            t ^= x
        elif k == 7:
            flag ^= b < t
    flag ^= x < t
    words = [(regs[:, 0] | (regs[:, 1] << u(20))).view(np.int64), (regs[:, 2] | (regs[:, 3] << u(32))).view(np.int64)]
    # the 1-bit flag takes the first word's next free bit and is 0 again at the end
    return {"words": words, "amps": _pairs(np.where(flag, amps * np.exp(1j * theta), amps))}


# ------------------------------------------------------------------ one multi-bit split
# A single Hadamard or unitary on a few bits of a large state with wide keys
# (an address, the word loaded for it, a control flag), controlled by the
# flag, its groups partly filled: the step that state-preparation and
# block-encoding circuits repeat.
def _block_start(c, seed):
    rng = np.random.default_rng([seed, 9])
    S, g = 1 << c["bits"], c["groups"]
    there = rng.random((g, S)) < c["fill"]
    there[:, 0] = True
    idx, q = np.nonzero(there)
    p = rng.permutation(idx.size)
    idx, q = idx[p].astype(np.uint64), q[p].astype(np.uint64)
    word = rng.integers(0, 1 << 60, g, dtype=np.uint64)
    flag = rng.integers(0, 4, g, dtype=np.uint64) > 0 if c["controlled"] else np.ones(g, dtype=bool)
    v = rng.standard_normal(idx.size) + 1j * rng.standard_normal(idx.size)
    m, _ = np.linalg.qr(rng.standard_normal((S, S)) + 1j * rng.standard_normal((S, S)))
    gb = max(1, math.ceil(math.log2(g)))
    return idx, q, word, flag, v / np.linalg.norm(v), m, gb


def block_prepare(c, seed):
    idx, q, word, flag, v, m, gb = _block_start(c, seed)
    _register_table(("q", ps.UnsignedInteger, c["bits"]), ("i", ps.UnsignedInteger, gb), ("flag", ps.Boolean, 1),
                    ("x", ps.UnsignedInteger, 60))
    i = idx.astype(np.int64)
    init = ps.SparseState(capacity=idx.size)
    init.upload(np.stack([q, idx, flag[i].astype(np.uint64), word[i]], axis=1), v)
    op = ps.Hadamard_Int("q", c["bits"]) if c["op"] == "hadamard" else ps.Rot_GeneralUnitary("q", m)
    if c["controlled"]:
        op.conditioned_by_nonzeros("flag")
    return {"f": "block", "c": c, "init": init, "op": op, "bits": c["bits"] + gb + 1}


def block_run(s):
    st = s["init"].copy()
    s["op"](st)
    return _dense(st, s["bits"])


def block_work(c):
    n_out = float(c["groups"] << c["bits"])
    n_in = n_out * max(c["fill"], 1.0 / (1 << c["bits"]))
    return {"bytes": (3 * n_in + n_out) * 32.0, "flops": n_out * (2 * c["bits"] if c["op"] == "hadamard" else 8.0 * (1 << c["bits"]))}


def block_exact(c, seed):
    idx, q, _, flag, v, m, gb = _block_start(c, seed)
    S, g = 1 << c["bits"], c["groups"]
    x = np.zeros((g, S), dtype=np.complex128)
    x[idx.astype(np.int64), q.astype(np.int64)] = v
    y = _fwht(x, c["bits"]) if c["op"] == "hadamard" else x @ m.T
    y = np.where(flag[:, None], y, x)
    out = np.zeros((2, 1 << gb, S), dtype=np.complex128)
    out[flag.astype(np.int64), np.arange(g)] = y
    return _pairs(out.reshape(-1))


# ------------------------------------------------------------------ cases
FAMILIES = {
    "gates": (gates_prepare, gates_run, gates_work, gates_exact),
    "qram_rotation": (qram_rotation_prepare, qram_rotation_run, qram_rotation_work, qram_rotation_exact),
    "register_circuit": (register_circuit_prepare, register_circuit_run, register_circuit_work, register_circuit_exact),
    "hidden": (hidden_prepare, hidden_run, hidden_work, hidden_exact),
    "trajectories": (trajectories_prepare, trajectories_run, trajectories_work, trajectories_exact),
    "qda": (qda_prepare, qda_run, qda_work, None),
    "qda_qram": (qda_qram_prepare, qda_qram_run, qda_qram_work, None),
    "cks": (cks_prepare, cks_run, cks_work, None),
    "cks_qram": (cks_qram_prepare, cks_qram_run, cks_qram_work, None),
    "arithmetic": (arithmetic_prepare, arithmetic_run, arithmetic_work, arithmetic_exact),
    "block": (block_prepare, block_run, block_work, block_exact),
}


def listed():
    return [
        # a first program: an 8-qubit layered ansatz from |0>, call latency
        {"name": "gates_8q", "family": "gates", "bits": 8, "layers": 2, "rotated": 8, "dense": False},
        # gate-by-gate simulation of a dense 21-qubit register
        {"name": "gates_21q", "family": "gates", "bits": 21, "layers": 1, "rotated": 6, "dense": True},
        # amplitude encoding of a 2^20-word table
        {"name": "qram_rotation_2p20", "family": "qram_rotation", "address_bits": 20, "word_bits": 24},
        # the register circuit at scale, graph replay: the repository's benchmark
        {"name": "register_circuit", "family": "register_circuit", "h": 12, "layers": 10, "replay": True},
        # period finding over 2^10 addresses, partly filled groups
        {"name": "hidden_10", "family": "hidden", "bits": 10, "word_bits": 12, "layers": 3, "arithmetic": "exact-sum"},
        # 4096 noisy instances, the batched benchmark
        {"name": "trajectories_4096", "family": "trajectories", "instances": 4096, "layers": 6, "h_min": 4, "h_max": 8},
        # tridiagonal QDA at the size of the published runs
        {"name": "qda_2p16", "family": "qda", "bits": 16, "warm": 24},
        # QDA through QRAM at the size of a whole solve (2000 such steps)
        {"name": "qda_qram_2p5", "family": "qda_qram", "bits": 5, "kappa": 50.0, "warm": 3},
        # CKS terms, tridiagonal and through QRAM
        {"name": "cks_2p17", "family": "cks", "bits": 17, "kappa": 100.0},
        {"name": "cks_qram_2p14", "family": "cks_qram", "bits": 14, "half_bandwidth": 4, "kappa": 100.0},
        # compute, phase, uncompute over 2^23 entries
        {"name": "arithmetic_2p23", "family": "arithmetic", "entries": 1 << 23, "chain": 9, "fused": True},
        # a controlled 6-bit Hadamard, groups half filled, 1.2M entries
        {"name": "block_h6", "family": "block", "op": "hadamard", "bits": 6, "groups": 37000, "fill": 0.5, "controlled": True},
    ]


def _between(rng, lo, hi):
    """A whole number, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    f = rng.choice(sorted(FAMILIES))
    c = {"family": f}
    if f == "gates":
        dense = rng.random() < 0.5
        n = rng.randint(13, 21) if dense else rng.randint(3, 12)
        c.update(bits=n, layers=rng.randint(1, 2), rotated=rng.randint(1, min(n, 6)), dense=dense)
    elif f == "qram_rotation":
        c.update(address_bits=rng.randint(4, 20), word_bits=rng.randint(8, 40))
    elif f == "register_circuit":
        c.update(h=rng.randint(3, 12), layers=rng.randint(1, 9), replay=rng.random() < 0.5)
    elif f == "hidden":
        m = rng.randint(3, 11)
        c.update(bits=m, word_bits=max(2, min(m + rng.randint(-1, 3), 24 - m)), layers=rng.randint(1, 4),
                 arithmetic=rng.choice(["exact-sum", "reference"]))
    elif f == "trajectories":
        lo = rng.randint(2, 8)
        c.update(instances=_between(rng, 5, 4000), layers=rng.randint(1, 6), h_min=lo, h_max=rng.randint(lo, 8))
    elif f == "qda":
        c.update(bits=rng.randint(4, 15), warm=rng.randint(2, 30))
    elif f == "qda_qram":
        c.update(bits=rng.randint(2, 5), kappa=round(rng.uniform(5, 100), 2), warm=rng.randint(1, 4))
    elif f == "cks":
        c.update(bits=rng.randint(4, 17), kappa=round(rng.uniform(60, 200), 2))
    elif f == "cks_qram":
        c.update(bits=rng.choice([5, 6, 7, 8, 9, 10, 13, 14]), half_bandwidth=rng.randint(1, 4),
                 kappa=round(rng.uniform(60, 200), 2))
    elif f == "arithmetic":
        c.update(entries=_between(rng, 100, 1 << 23), chain=rng.randint(2, 9), fused=rng.random() < 0.7)
    else:
        op = rng.choice(["hadamard", "unitary"])
        n = rng.randint(1, 10 if op == "hadamard" else 5)
        c.update(op=op, bits=n, groups=max(1, _between(rng, 3, 2400000) >> n), fill=rng.choice([0.0, 0.1, 0.5, 1.0]),
                 controlled=rng.random() < 0.5)
    return c


def prepare(case, seed):
    return FAMILIES[case["family"]][0](case, int(seed))


def run(state):
    return FAMILIES[state["f"]][1](state)


def work(case):
    return FAMILIES[case["family"]][2](case)


def exact(case, seed):
    f = FAMILIES[case["family"]][3]
    return None if f is None else f(case, int(seed))
