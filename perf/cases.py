"""The engine's working range as timed cases: what programs ask of it through
its public entry points, from a few qubits to the largest circuits.

A case is one kind of program at one size:

  program   a short circuit on a small state, state vector read back
  energy    a variational ansatz and the expectation values of its Ising terms
  measure   mid-circuit measurement and reset with supplied uniforms
  noisy     one depolarising Pauli trajectory after another (each has its own
            gates), probabilities read back
  shots     a deep random layered circuit, then shots in measure_all order
  gates     every gate kind the instruction set has, general unitaries included
  layered   a large layered circuit, then inverse-CDF shots and Z strings
  qft       the Fourier transform of a periodic state, then shots
  batch     many variational circuits together: added, run and read anew
            ("fresh"), or one prepared batch run again ("replay")
  serve     noisy requests through the server's loop

Circuit structure (which gate on which qubits) belongs to the case; the seed
gives angles, uniforms and masks, so the passes of a case cost the same from
seed to seed. States of 20 or more qubits compile their pass kernels while
they are prepared, as a program that runs a circuit many times does
(`QOA_JIT_SYNC`). Every program starts with QINIT (complex64 handles, which
take no QINIT, with RESETALL), which puts the state into |0..0>. Values read
from complex64 states are kept in 32 bits.
"""
import math

import numpy as np
import torch

import qoa_b200 as qb
from qoa_b200 import circuits as C


def listed():
    return [
        # a textbook program (teleportation, Grover on a few qubits): all latency
        {"name": "program_n6", "kind": "program", "n": 6, "depth": 6, "prec": "f64"},
        # one energy evaluation of a variational loop on ten qubits
        {"name": "energy_n10", "kind": "energy", "n": 10, "depth": 4, "prec": "f64"},
        # syndrome-style program: layers, measurements, resets, more layers
        {"name": "measure_n13", "kind": "measure", "n": 13, "depth": 4, "prec": "f64"},
        # trajectory loop at the noise level of the serving workload
        {"name": "noisy_n16", "kind": "noisy", "n": 16, "depth": 8, "prec": "f64"},
        # the reference executor's own workload: 20 qubits, 40 layers, 1024 shots
        {"name": "shots_n20", "kind": "shots", "n": 20, "depth": 40, "prec": "f64"},
        # a program that uses the whole instruction set
        {"name": "gates_n22", "kind": "gates", "n": 22, "depth": 240, "prec": "f64"},
        # an energy evaluation on a state larger than the caches hold comfortably, single precision
        {"name": "energy_n23_f32", "kind": "energy", "n": 23, "depth": 8, "prec": "f32"},
        # the large random circuit, a state well beyond the caches
        {"name": "layered_n27", "kind": "layered", "n": 27, "depth": 20, "prec": "f64"},
        # the precision form's Fourier transform, the largest state here
        {"name": "qft_n29_f32", "kind": "qft", "n": 29, "depth": 6, "prec": "f32"},
        # a gradient's worth of small circuits, new angles every time
        {"name": "batch_small_fresh", "kind": "batch", "n": 10, "nmin": 4, "depth": 6, "count": 256, "fresh": True, "prec": "f64"},
        # the batching form's mix of sizes, replayed
        {"name": "batch_mixed_replay", "kind": "batch", "n": 20, "nmin": 8, "depth": 10, "count": 192, "fresh": False, "prec": "f64"},
        # a burst of small noisy requests
        {"name": "serve_n14", "kind": "serve", "n": 14, "nmin": 8, "depth": 16, "count": 8, "prec": "f64"},
    ]


def draw(rng):
    kind = rng.choice(["program", "energy", "energy", "measure", "noisy", "shots", "gates", "layered", "qft", "batch", "batch",
                       "serve"])
    prec = rng.choice(["f64", "f64", "f32"])
    if kind == "program":
        return {"kind": kind, "n": rng.randint(3, 10), "depth": rng.randint(2, 12), "prec": prec}
    if kind == "energy":
        return {"kind": kind, "n": rng.randint(7, 25), "depth": rng.randint(2, 10), "prec": prec}
    if kind == "measure":
        return {"kind": kind, "n": rng.randint(4, 19), "depth": rng.randint(2, 6), "prec": "f64"}
    if kind == "noisy":
        return {"kind": kind, "n": rng.randint(6, 18), "depth": rng.randint(4, 16), "prec": "f64"}
    if kind == "shots":
        return {"kind": kind, "n": rng.randint(12, 24), "depth": rng.randint(10, 40), "prec": "f64"}
    if kind == "gates":
        return {"kind": kind, "n": rng.randint(8, 24), "depth": rng.randint(60, 240), "prec": "f64"}
    if kind == "layered":
        return {"kind": kind, "n": rng.randint(24, 27), "depth": rng.randint(6, 20), "prec": "f64"}
    if kind == "qft":
        return {"kind": kind, "n": rng.randint(18, 29 if prec == "f32" else 28), "depth": rng.randint(3, 7), "prec": prec}
    if kind == "batch":
        if rng.random() < 0.5:
            return {"kind": kind, "n": rng.randint(8, 12), "nmin": rng.randint(3, 8), "depth": rng.randint(2, 8),
                    "count": rng.randint(32, 512), "fresh": True, "prec": prec}
        return {"kind": kind, "n": rng.randint(13, 20), "nmin": rng.randint(6, 10), "depth": rng.randint(3, 10),
                "count": rng.randint(32, 192), "fresh": False, "prec": prec}
    return {"kind": kind, "n": rng.randint(10, 14), "nmin": rng.randint(6, 10), "depth": rng.randint(8, 24),
            "count": rng.randint(2, 8), "prec": "f64"}


# ------------------------------------------------------------------ circuits
NOISE_P = 1e-3


def _layered(n, depth, structure, rng, first_h=True):
    """Layers of one-qubit gates and disjoint pairs: kinds from `structure`, angles from `rng`."""
    ops = [C.Op(C.H, [q]) for q in range(n)] if first_h else []
    for _ in range(depth):
        for q in range(n):
            g = C.ONE_QUBIT_GATES[structure.integers(len(C.ONE_QUBIT_GATES))]
            ops.append(C.Op(g, [q], rng.uniform(0, 2 * math.pi) if g in C.ANGLED else 0.0))
        perm = structure.permutation(n)
        for k in range(n // 2):
            g = C.TWO_QUBIT_GATES[structure.integers(len(C.TWO_QUBIT_GATES))]
            ops.append(C.Op(g, perm[2 * k:2 * k + 2], rng.uniform(0, 2 * math.pi) if g == C.CPHASE else 0.0))
    return ops


def _variational(n, layers, rng, width):
    ops = []
    for _ in range(layers):
        for q in range(n):
            ops.append(C.Op(C.RY, [q], rng.uniform(-width, width)))
            ops.append(C.Op(C.RZ, [q], rng.uniform(-width, width)))
        ops += [C.Op(C.CZ, [q, q + 1]) for q in range(n - 1)]
    return ops


def _all_kinds(n, count, structure, rng):
    kinds = [C.H, C.X, C.Y, C.Z, C.T, C.S, C.P, C.RX, C.RY, C.RZ, C.CNOT, C.CZ, C.CPHASE, C.SWAP, C.CSWAP, C.TOFFOLI, C.CY,
             C.U1, C.U2, C.EBELL, C.ECLUSTER]
    ops = []
    for _ in range(count):
        g = kinds[structure.integers(len(kinds))]
        qs = [int(q) for q in structure.permutation(n)[:3]]
        if g in (C.U1, C.U2):
            d = 2 if g == C.U1 else 4
            u, _ = np.linalg.qr(rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d)))
            ops.append(C.Op(g, qs[:1 if g == C.U1 else 2], 0.0, u.reshape(-1)))
            continue
        k = 2 if g in (C.CNOT, C.CZ, C.CPHASE, C.SWAP, C.CY, C.EBELL) else 3 if g in (C.CSWAP, C.TOFFOLI, C.ECLUSTER) else 1
        ops.append(C.Op(g, qs[:k], rng.uniform(0, 2 * math.pi) if g in C.ANGLED else 0.0))
    return ops


def _rngs(case, seed):
    shape = [case["n"], case["depth"], len(case["kind"]), ord(case["kind"][0])]
    return np.random.default_rng(shape), np.random.default_rng([seed, 1])


def _quirk(case):
    return case["kind"] in ("shots", "layered")  # the reference executor's CZ / CPHASE masks


def _inputs(case, seed):
    """Everything of a case that the seed gives: op lists, masks, uniforms."""
    structure, rng = _rngs(case, seed)
    n, depth, kind = case["n"], case["depth"], case["kind"]
    d = {}
    if kind in ("program", "noisy", "shots"):
        d["ops"] = _layered(n, depth, structure, rng)
    elif kind == "energy":
        d["ops"] = _variational(n, depth, rng, 0.6)
        d["masks"] = [1 << q for q in range(n)] + [3 << q for q in range(n - 1)]
    elif kind == "measure":
        d["ops"] = _layered(n, depth, structure, rng)
        d["more"] = _layered(n, depth, structure, rng, first_h=False)
        d["qubits"] = [int(q) for q in structure.permutation(n)[:3]]
        d["reset"] = int(structure.integers(n))
        d["u"] = [float(x) for x in rng.random(3)]
    elif kind == "gates":
        d["ops"] = [C.Op(C.H, [q]) for q in range(n)] + _all_kinds(n, depth, structure, rng)
        d["masks"] = [int(x) for x in rng.integers(1, 1 << n, 8)]
    elif kind == "layered":
        d["ops"] = _layered(n, depth, structure, rng)
        d["masks"] = [int(x) for x in rng.integers(1, 1 << n, 16)]
        d["u"] = rng.random(4096)
    elif kind == "qft":
        # a comb of period 2^depth, shifted: its transform has 2^depth peaks
        d["ops"] = ([C.Op(C.H, [q]) for q in range(depth, n)] + [C.Op(C.X, [q]) for q in range(depth) if rng.random() < 0.5]
                    + C.qft(n))
        d["u"] = rng.random(1024)
    elif kind in ("batch", "serve"):
        d["items"] = []
        for _ in range(case["count"]):
            m = int(structure.integers(case["nmin"], n + 1))
            layers = int(structure.integers(2, depth + 1))
            if kind == "batch":
                d["items"].append({"n": m, "ops": _variational(m, layers, rng, math.pi),
                                   "masks": [int(x) for x in rng.integers(0, 1 << m, 8)]})
            else:
                d["items"].append({"n": m, "ops": _layered(m, layers, structure, rng), "seed": int(rng.integers(1 << 62))})
    if kind == "shots":
        d["u"] = rng.random(1024 * n)
    return d


def _init(n, ops, prec):
    return C.ops_to_array([C.Op(C.QINIT, [n]) if prec == "f64" else C.Op(C.RESETALL)] + ops)


def prepare(case, seed):
    d = _inputs(case, seed)
    kind, n, prec = case["kind"], case["n"], case["prec"]
    s = {"case": case, "in": d}
    if kind == "batch":
        for it in d["items"]:
            it["arr"] = C.ops_to_array(it["ops"])
        if not case["fresh"]:
            b = s["batch"] = qb.Batch(prec)
            for it in d["items"]:
                b.add(it["n"], it["arr"], it["masks"])
            b.run()
            b.run()
            qb.jit_wait()
            b.run()
        return s
    if kind == "serve":
        for it in d["items"]:
            it["arr"] = C.ops_to_array(it["ops"])
        s["server"] = qb.Server(prec)
        return s
    st = s["state"] = qb.QuantumState(n, qb.NoiseConfig.Fixed(NOISE_P) if kind == "noisy" else None, seed=seed,
                                      precision=prec, compat_mask_quirk=_quirk(case))
    s["ops"] = _init(n, d["ops"], prec)
    if kind == "measure":
        s["more"] = C.ops_to_array(d["more"])
    if kind == "noisy":
        s["trajectory"] = 0
    elif n >= 20:
        st.set_jit(qb.QOA_JIT_SYNC)
        st.execute(s["ops"])
        st.sync()
    return s


def _kept(x, case):
    return x.astype(np.float32) if case["prec"] == "f32" else x


def run(s):
    case, d = s["case"], s["in"]
    kind = case["kind"]
    if kind == "batch":
        b = s["batch"] if "batch" in s else qb.Batch(case["prec"])
        if "batch" not in s:
            for it in d["items"]:
                b.add(it["n"], it["arr"], it["masks"])
        b.run()
        r = b.results()
        if "batch" not in s:
            b.close()
        return _kept(r, case)
    if kind == "serve":
        srv = s["server"]
        ids = [srv.submit(it["n"], it["arr"], NOISE_P, 64, 16, it["seed"]) for it in d["items"]]
        left = set(ids)
        while left:
            left -= {r["id"] for r in srv.poll()}
        return np.concatenate([srv.take_shots(i, 64 * 16) for i in ids]).astype(np.int64)
    st = s["state"]
    if kind == "noisy":  # the next trajectory
        st.set_trajectory(s["trajectory"])
        s["trajectory"] += 1
    st.execute(s["ops"])
    if kind == "program":
        return st.get_state_vector()
    if kind == "energy":
        return _kept(st.expect_z(d["masks"]), case)
    if kind == "measure":
        bits = [st.measure(q, u) for q, u in zip(d["qubits"], d["u"])]
        st.reset_qubit(d["reset"])
        st.execute(s["more"])
        return {"bits": np.array(bits), "state": st.get_state_vector()}
    if kind == "noisy":
        return st.get_probabilities()
    if kind == "shots":
        return st.sample(1024, d["u"], mode=0).astype(np.int64)
    if kind == "gates":
        return st.expect_z(d["masks"])
    if kind == "layered":
        return {"z": st.expect_z(d["masks"]), "shots": st.sample(4096, d["u"], mode=1).astype(np.int64)}
    return st.sample(1024, d["u"], mode=1).astype(np.int64)  # qft


# ------------------------------------------------------------ what a pass needs
_FLOPS = {C.H: 2, C.X: 0, C.Y: 1, C.Z: 0.5, C.T: 3, C.S: 1, C.P: 3, C.RX: 4, C.RY: 4, C.RZ: 6, C.CNOT: 0, C.CZ: 0.25,
          C.CPHASE: 1.5, C.SWAP: 0, C.CSWAP: 0, C.TOFFOLI: 0, C.CY: 0.5, C.U1: 14, C.U2: 30, C.EBELL: 2, C.ECLUSTER: 6.5}


def work(case):
    """Flops of the gates on every amplitude; bytes: a state is written once and read once by what looks at it (a state
    that fits on the chip is not counted), results and uniforms once."""
    d = _inputs(case, 0)
    esz = 8 if case["prec"] == "f32" else 16

    def state(n, ops):
        size = float(1 << n)
        return (2 * size * esz if size * esz > (64 << 20) else 0), size * sum(_FLOPS[o.opcode] for o in ops)

    kind, n = case["kind"], case["n"]
    if kind in ("batch", "serve"):
        rep = 1 if kind == "batch" else 64
        parts = [state(it["n"], it["ops"]) for it in d["items"]]
        out = len(parts) * (64 if kind == "batch" else 64 * 16 * 8)
        held = sum(esz << it["n"] for it in d["items"])
        return {"bytes": float(out + (2 * held if held > (64 << 20) else 0)), "flops": rep * sum(f for _, f in parts)}
    b, f = state(n, d["ops"] + d.get("more", []))
    size = float(1 << n)
    out = {"program": size * esz, "measure": size * esz, "noisy": size * 8, "energy": 8 * 2 * n, "gates": 64,
           "shots": 1024 * 8 * (n + 1), "layered": 4096 * 16 + 128, "qft": 1024 * 16}[kind]
    reads = {"energy": 2, "gates": 2, "layered": 2, "shots": 2, "qft": 2}.get(kind, 0)  # |a|^2 and its sums
    return {"bytes": b + out, "flops": f + reads * 2 * size}


# ------------------------------------------------------------------- 64 bits
_SQ = math.sqrt(0.5)


def _matrix(o):
    g, a = o.opcode, o.angle
    c, s = math.cos(a / 2), math.sin(a / 2)
    if g == C.H:
        return [[_SQ, _SQ], [_SQ, -_SQ]]
    if g in (C.X, C.CNOT, C.TOFFOLI):
        return [[0, 1], [1, 0]]
    if g in (C.Y, C.CY):
        return [[0, -1j], [1j, 0]]
    if g == C.RX:
        return [[c, -1j * s], [-1j * s, c]]
    if g == C.RY:
        return [[c, -s], [s, c]]
    return np.asarray(o.matrix).reshape(2, 2)


def _apply(v, n, o, quirk):
    """One op on a state held as an n-dimensional tensor (qubit q on axis n - 1 - q)."""
    g, qs = o.opcode, list(o.qubits)

    def at(fixed):
        return tuple(fixed.get(n - 1 - a, slice(None)) for a in range(n))

    def phase(mask_qubits, f):
        v[at({q: 1 for q in mask_qubits})] *= f

    if g == C.EBELL:
        _apply(v, n, C.Op(C.H, qs[:1]), quirk)
        _apply(v, n, C.Op(C.CNOT, qs), quirk)
    elif g == C.ECLUSTER:
        for q in qs:
            _apply(v, n, C.Op(C.H, [q]), quirk)
        for a, b in zip(qs, qs[1:]):
            _apply(v, n, C.Op(C.CZ, [a, b]), quirk)
    elif g in (C.Z, C.T, C.S, C.P):
        phase(qs, {C.Z: -1.0, C.T: complex(_SQ, _SQ), C.S: 1j}.get(g, complex(math.cos(o.angle), math.sin(o.angle))))
    elif g == C.RZ:
        v[at({qs[0]: 0})] *= complex(math.cos(o.angle / 2), -math.sin(o.angle / 2))
        v[at({qs[0]: 1})] *= complex(math.cos(o.angle / 2), math.sin(o.angle / 2))
    elif g in (C.CZ, C.CPHASE):
        if quirk:
            m = qs[0] | qs[1]
            qs = [q for q in range(n) if (m >> q) & 1]
            if m >> n:
                return
        phase(qs, -1.0 if g == C.CZ else complex(math.cos(o.angle), math.sin(o.angle)))
    elif g in (C.SWAP, C.CSWAP):
        ctl = {qs[0]: 1} if g == C.CSWAP else {}
        a, b = qs[-2:]
        i, j = at({**ctl, a: 1, b: 0}), at({**ctl, a: 0, b: 1})
        t = v[i].clone()
        v[i] = v[j]
        v[j] = t
    elif g == C.U2:
        m = np.asarray(o.matrix).reshape(4, 4)  # basis 2 * bit(higher qubit) + bit(lower)
        lo, hi = min(qs), max(qs)
        idx = [at({hi: k >> 1, lo: k & 1}) for k in range(4)]
        x = [v[i].clone() for i in idx]
        for r in range(4):
            v[idx[r]] = sum(complex(m[r, k]) * x[k] for k in range(4))
    else:
        ctl = {q: 1 for q in qs[:-1]}
        m = _matrix(o)
        i, j = at({**ctl, qs[-1]: 0}), at({**ctl, qs[-1]: 1})
        x, y = v[i].clone(), v[j].clone()
        v[i] = complex(m[0][0]) * x + complex(m[0][1]) * y
        v[j] = complex(m[1][0]) * x + complex(m[1][1]) * y


def _zero(n):
    v = torch.zeros(1 << n, dtype=torch.complex128, device="cuda" if torch.cuda.is_available() else "cpu")
    v[0] = 1
    return v


def _simulate(n, ops, quirk=False, after=None):
    v = _zero(n)
    t = v.view([2] * n)
    for k, o in enumerate(ops):
        _apply(t, n, o, quirk)
        for e in (after[k] if after else ()):
            _apply(t, n, e, quirk)
    return v


def _p(v):
    p = v.real.square() + v.imag.square()
    return p / p.sum()


def _z(v, masks):
    p, n, out = _p(v), v.numel().bit_length() - 1, []
    for m in masks:
        x = p
        for q in range(n - 1, -1, -1):
            h = x.view(2, -1)
            x = h[0] - h[1] if (m >> q) & 1 else h[0] + h[1]
        out.append(float(x[0]))
    return np.array(out)


def _uniform(seed, stream, event, slots):
    """Philox4x32-10 uniforms of one event, as the engine documents them (counter: event, slot, stream; key: seed)."""
    mask = np.uint64(0xFFFFFFFF)
    full = lambda x: np.full(len(slots), x, dtype=np.uint64)  # noqa: E731
    c = [full(event & 0xFFFFFFFF), full(event >> 32), np.asarray(slots, dtype=np.uint64), full(stream & 0xFFFFFFFF)]
    k0, k1 = seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF
    for _ in range(10):
        a, b = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(b >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), b & mask, (a >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), a & mask]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return (((c[0] << np.uint64(32)) | c[1]) >> np.uint64(11)).astype(np.float64) * 2.0 ** -53


def exact(case, seed):
    d, kind, n = _inputs(case, seed), case["kind"], case["n"]
    if kind == "serve" or kind == "shots" or kind == "qft":
        return None  # whole numbers only
    if kind == "batch":
        return np.concatenate([_z(_simulate(it["n"], it["ops"]), it["masks"]) for it in d["items"]])
    if kind == "noisy":
        paulis = []
        for e in range(len(d["ops"])):
            hit = np.nonzero(_uniform(seed, 0, e, [2 * q + 1 for q in range(n)]) < NOISE_P)[0]
            kinds = _uniform(seed, 0, e, [2 * int(q) + 2 for q in hit])
            paulis.append([C.Op((C.X, C.Y, C.Z)[min(int(u * 3), 2)], [int(q)]) for q, u in zip(hit, kinds)])
        return _p(_simulate(n, d["ops"], after=paulis)).cpu().numpy()
    v = _simulate(n, d["ops"], _quirk(case))
    if kind == "program":
        return (v / v.abs().square().sum().sqrt()).cpu().numpy()
    if kind == "measure":
        t = v.view([2] * n)
        for q, u in list(zip(d["qubits"], d["u"])) + [(d["reset"], None)]:
            h = v.view(-1, 2, 1 << q)
            p = _p(v).view(-1, 2, 1 << q)[:, 0].sum().item()
            bit = 0 if u is None or u < p else 1
            h[:, 1 - bit] = 0
            v /= v.abs().square().sum().sqrt()
        for o in d["more"]:
            _apply(t, n, o, False)
        return {"bits": None, "state": (v / v.abs().square().sum().sqrt()).cpu().numpy()}
    if kind == "layered":
        return {"z": _z(v, d["masks"]), "shots": None}
    return _z(v, d["masks"])
