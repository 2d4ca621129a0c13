"""Performance cases: the work that programs have this library do, through its public entry points.

One case is one pass of one of five kinds:

  steps      a batch of moduli kept on the device: values and exponents in, `steps` exponent bits
             on every slot, raw Montgomery limbs out (ModBatch's backend calls: load_all,
             set_exponents, run, read_all). The inner loop of a Fermat test.
  mul        one product of two slots that share a modulus, and the result read back.
  serve      one cycle of the serving loop on a segment: some slots get new moduli in place, every
             slot a value and an exponent, one item-list launch, all values read.
  mixed      batches of several lengths stepped together by one Plan (persistent launches).
  transform  products in the transform domain (the Transform trait): two forward transforms of
             limb vectors, a pointwise product, the inverse, and the raw field values read.

Every output is whole numbers and has to be equal, limb for limb.
"""
from __future__ import annotations

import math
import random

import numpy as np

LIMB = 32


def listed():
    return [
        # The smallest call: one product of two 1,024-bit values, where launches, copies and one
        # block's latency are all there is.
        {"name": "mul_1024b", "kind": "mul", "bits": 1024, "wrap": True},
        # 64 full 4,096-bit Fermat tests (the CPU-sized batch): fewer slots than SMs, so the time
        # of one step on one slot counts.
        {"name": "fermat_4096b_64", "kind": "steps", "bits": 4096, "slots": 64, "steps": 4096, "base": 3, "wrap": True},
        # Many small moduli (the size sweep's 8,192 bits): several slots on every SM.
        {"name": "steps_8192b_2368", "kind": "steps", "bits": 8192, "slots": 2368, "steps": 256, "base": 3, "wrap": True},
        # Base 2 tests at the sweep's 32,768 bits, a batch that does not fill whole waves of SMs.
        {"name": "steps_32768b_1000", "kind": "steps", "bits": 32768, "slots": 1000, "steps": 128, "base": 2, "wrap": True},
        # The benchmark's 100,000-bit moduli, two full waves of the GPU.
        {"name": "steps_100000b_592", "kind": "steps", "bits": 100000, "slots": 592, "steps": 250, "base": 3, "wrap": True},
        # The plain REDC (wraparound off, the reference Cpu backend's default) at an odd size.
        {"name": "plain_20011b_600", "kind": "steps", "bits": 20011, "slots": 600, "steps": 200, "base": 3, "wrap": False},
        # A serving segment of the stream's largest requests (200,000 bits), a few of them new.
        {"name": "serve_200000b_148", "kind": "serve", "bits": 200000, "slots": 148, "fresh": 8, "steps": 200, "base": 3},
        # Beyond one SM's shared memory: the sweep's 300,000 and 1,000,000 bits.
        {"name": "steps_300000b_148", "kind": "steps", "bits": 300000, "slots": 148, "steps": 100, "base": 3, "wrap": True},
        {"name": "steps_1000000b_37", "kind": "steps", "bits": 1000000, "slots": 37, "steps": 30, "base": 3, "wrap": True},
        # The longest tests: 2,000,000 bits, the vector in device memory.
        {"name": "steps_2000000b_24", "kind": "steps", "bits": 2000000, "slots": 24, "steps": 8, "base": 3, "wrap": True},
        # Sizes from 8,192 to 300,000 bits in one persistent launch.
        {"name": "mixed_8k_300k_400", "kind": "mixed", "lo": 8192, "hi": 300000, "slots": 400, "steps": 256},
        # The Transform trait at the benchmark's length.
        {"name": "transform_8192_64", "kind": "transform", "len": 8192, "k": 4001, "count": 64},
    ]


# Budgets of a drawn case, below the largest listed one: device time by a rough cost per slot-step
# (a step of one slot takes at least about a full SM's share of it), and host set-up of the moduli.
_DRAW_NS = 60e6
_DRAW_BITS = 4.0e7


def _length(bits, wrap=True):
    k = -(-(bits + 4) // LIMB)
    length = 8
    while length < 2 * k:
        length *= 2
    return (length // 2 if wrap else k), length


def _slot_ns(length):
    return 0.08 * length * (1 + min(1.0, length / 65536))


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "steps", "mul", "serve", "mixed", "transform"])
    base = rng.choice([1, 2, 3, 3, 4])
    if kind == "mul":
        return {"kind": "mul", "bits": _log(rng, 200, 2000000), "wrap": rng.random() < 0.8}
    if kind == "transform":
        length = 1 << rng.randint(3, 17)
        return {"kind": "transform", "len": length, "k": rng.randint(max(1, length // 4), length // 2),
                "count": max(1, min(_log(rng, 1, 256), (1 << 19) // length))}
    if kind == "mixed":
        lo = _log(rng, 512, 50000)
        hi = max(lo + 1, _log(rng, lo, 300000))
        slots = _log(rng, 3, 300)
        return {"kind": "mixed", "lo": lo, "hi": hi, "slots": slots, "steps": rng.randint(16, min(lo, 200))}
    if kind == "serve":
        bits = _log(rng, 10000, 200000)
        slots = _log(rng, 2, 300)
        return {"kind": "serve", "bits": bits, "slots": slots, "fresh": rng.randint(1, min(8, slots)),
                "steps": rng.randint(16, 150), "base": base}
    bits = _log(rng, 256, 2000000)
    wrap = rng.random() < 0.85
    _, length = _length(bits, wrap)
    slots = max(1, min(_log(rng, 1, 2400), int(_DRAW_BITS / bits)))
    step = max(slots, 296) * _slot_ns(length) * (1.5 if not wrap else 1.0) + 10000
    return {"kind": "steps", "bits": bits, "slots": slots, "steps": max(1, min(bits, 1000, int(_DRAW_NS / step))),
            "base": base, "wrap": wrap}


# ---- inputs ----

def _modulus(rng, bits):
    return rng.getrandbits(bits) | (1 << (bits - 1)) | 1


def _limbs(x, k):
    return np.frombuffer(x.to_bytes(4 * k, "little"), dtype="<u4").astype(np.uint32)


def _exponent(rng, steps):
    """`steps` random bits, the top one set, as the backend takes them (MSB first)."""
    e = rng.getrandbits(steps) | (1 << (steps - 1))
    nw = -(-steps // 32)
    return np.frombuffer((e << (32 * nw - steps)).to_bytes(4 * nw, "big"), dtype=">u4").astype(np.uint32), e


def _batch_inputs(rng, sizes, steps):
    """Per slot: an odd modulus, a Montgomery-form value below it, an exponent of `steps` bits."""
    mods = [_modulus(rng, b) for b in sizes]
    xs = [rng.randrange(n) for n in mods]
    exps = [_exponent(rng, steps) for _ in mods]
    return mods, xs, exps


def _inputs(case, seed):
    rng = random.Random(seed)
    if case["kind"] == "mul":
        n = _modulus(rng, case["bits"])
        return [n, n, n], [rng.randrange(n), rng.randrange(n), 0], None
    if case["kind"] == "serve":
        mods, xs, exps = _batch_inputs(rng, [case["bits"]] * case["slots"], case["steps"])
        return mods, xs, exps, [_modulus(rng, case["bits"]) for _ in range(case["fresh"])]
    if case["kind"] == "mixed":
        # The sizes and bases are the case's, so every seed has the same groups.
        sizes = random.Random(f"{case['lo']} {case['hi']} {case['slots']}")
        groups = {}
        for _ in range(case["slots"]):
            bits = _log(sizes, case["lo"], case["hi"])
            base = sizes.choice([2, 3, 4])
            groups.setdefault((_length(bits)[1], base), []).append(bits)
        return [(base, *_batch_inputs(rng, sizes, case["steps"])) for (_, base), sizes in sorted(groups.items())]
    if case["kind"] == "transform":
        gen = np.random.default_rng(seed)
        shape = (case["count"], case["k"])
        a = gen.integers(0, 1 << 32, shape, dtype=np.uint32)
        b = gen.integers(0, 1 << 32, shape, dtype=np.uint32)
        return a, b, gen.integers(1, 5, case["count"], dtype=np.uint32)
    return _batch_inputs(rng, [case["bits"]] * case["slots"], case["steps"])


_devices = {}


def _device(wrap):
    from montmul_b200 import B200
    if wrap not in _devices:
        _devices[wrap] = B200(wraparound=wrap)
    return _devices[wrap]


def _rows(xs, k):
    return np.stack([_limbs(x, k) for x in xs])


def _words(exps):
    return np.stack([w for w, _ in exps]), np.array([e.bit_length() for _, e in exps], np.uint32)


def prepare(case, seed):
    from montmul_b200 import ModBatch
    kind = case["kind"]
    ins = _inputs(case, seed)
    if kind == "transform":
        return {"case": case, "dev": _device(True), "a": ins[0], "b": ins[1], "scales": ins[2]}
    if kind == "mixed":
        from montmul_b200.backend import Plan
        groups = []
        for base, mods, xs, exps in ins:
            b = ModBatch(_device(True), mods, base)
            groups.append((b, _rows(xs, b.params.k), *_words(exps)))
        return {"case": case, "groups": groups, "plan": Plan([g[0] for g in groups], 128)}
    batch = ModBatch(_device(case.get("wrap", True)), ins[0], case.get("base", 3))
    state = {"case": case, "batch": batch, "x": _rows(ins[1], batch.params.k)}
    if kind == "mul":
        batch.backend.load_all(batch.state, state["x"])
        batch.backend.push(batch.state)
        return state
    state["words"], state["nbits"] = _words(ins[2])
    if kind == "serve":
        fresh = [batch.prepare(n) for n in ins[3]]
        state["n"] = np.stack([p[0] for p in fresh])
        state["nprime"] = np.stack([p[1] for p in fresh])
    return state


# ---- one pass ----

def _split(rows):
    """The first row apart from the others: `exact` gives that one (all would take too long)."""
    return {"first": rows[:1], "rest": rows[1:]}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "transform":
        dev, length, count = state["dev"], case["len"], case["count"]
        a = dev.load_forward(state["a"], case["k"], length, count)
        b = dev.load_forward(state["b"], case["k"], length, count)
        dev.pointwise(a, a, b, state["scales"], length, count)
        dev.inverse(a, length, count)
        f1, f2 = dev.download_raw(a)
        return {"m31": f1, "m61": f2.view(np.int64)}
    if kind == "mixed":
        for b, x, words, nbits in state["groups"]:
            b.backend.load_all(b.state, x)
            b.backend.set_exponents(b.state, words, nbits)
        state["plan"].run(case["steps"])
        return [_split(b.backend.read_all(b.state)) for b, _, _, _ in state["groups"]]
    batch = state["batch"]
    dev, st = batch.backend, batch.state
    if kind == "mul":
        dev.mul(st, 2, 0, 1)
        return dev.read(st, 2)
    if kind == "serve":
        slots, fresh = list(range(case["slots"])), list(range(case["fresh"]))
        dev.set_moduli(st, fresh, state["n"], state["nprime"])
        dev.write_slots(st, slots, state["x"], state["words"], state["nbits"])
        dev.run_items_async(st, slots, [case["steps"]] * len(slots))
        dev.sync(st)
        return _split(dev.read_slots(st, slots))
    dev.load_all(st, state["x"])
    dev.set_exponents(st, state["words"], state["nbits"])
    dev.run(st, case["steps"])
    return _split(dev.read_all(st))


# ---- work, tolerance, exact values ----

def _pairs(n):
    """Butterfly pairs of one squaring with its reduction: four length-n transforms, two of n / 2."""
    m = max(1, int(math.log2(n)))
    return 4 * (n // 2) * m + 2 * (n // 4) * max(1, m - 1)


# 32-bit multiply-adds of one butterfly pair (a GF(M61^2) and a GF(M31^2) product).
_PAIR_OPS = 32


def _step_work(sizes, steps, wrap):
    byts = ops = 0
    for bits in sizes:
        k, length = _length(bits, wrap)
        byts += 4 * (2 * k + 2 * k) + 4 * -(-steps // 32)      # N and N', x in and out, exponent
        ops += steps * _pairs(length // 2) * _PAIR_OPS
    return byts, ops


def work(case):
    kind = case["kind"]
    if kind == "transform":
        n, count = case["len"] // 2, case["count"]
        m = int(math.log2(n))
        return {"bytes": count * (8 * case["k"] + 24 * n + 4), "flops": count * 3 * (n // 2) * m * _PAIR_OPS}
    if kind == "mul":
        b, f = _step_work([case["bits"]], 1, case["wrap"])
        return {"bytes": b, "flops": f}
    if kind == "mixed":
        # The mean over the log-uniform sizes, by quadrature.
        pts = 33
        sizes = [round(case["lo"] * (case["hi"] / case["lo"]) ** ((i + 0.5) / pts)) for i in range(pts)]
        b, f = _step_work(sizes, case["steps"], True)
        return {"bytes": b * case["slots"] / pts, "flops": f * case["slots"] / pts}
    b, f = _step_work([case["bits"]], case["steps"], case.get("wrap", True))
    return {"bytes": b * case["slots"], "flops": f * case["slots"]}


def tolerance(case):
    return "exact"


def _redc(t, n, nprime, k):
    r = 32 * k
    mask = (1 << r) - 1
    return (t + ((t & mask) * nprime & mask) * n) >> r


def _nprime(n, k):
    """-n^-1 mod 2^(32 k) by Newton's iteration."""
    inv, bits = 1, 1
    while bits < 32 * k:
        bits = min(2 * bits, 32 * k)
        inv = inv * (2 - n * inv) & ((1 << bits) - 1)
    return (1 << 32 * k) - inv


def _chain(n, x, e, base, k):
    np_ = _nprime(n, k)
    for bit in bin(e)[2:]:
        x = _redc(x * x * (base if bit == "1" else 1), n, np_, k)
    return x


def _seconds(k, steps):
    """A rough bound of _chain's time: three products per step."""
    return steps * 3 * 1.4e-6 * (32 * k / 1000) ** 1.59


def _exact_rows(mods, xs, exps, base, k, steps, budget=16.0):
    if _seconds(k, steps) > budget:
        return {"first": None, "rest": None}
    row = _limbs(_chain(mods[0], xs[0], exps[0][1], base, k), k)
    return {"first": row[None], "rest": None if len(mods) > 1 else np.zeros((0, k), np.uint32)}


def _some(rows):
    """None when no value of the case is given."""
    return rows if any(r["first"] is not None for r in (rows if isinstance(rows, list) else [rows])) else None


def _batch_k(mods, wrap):
    ks = [_length(n.bit_length(), wrap) for n in mods]
    return max(k for k, _ in ks)


def exact(case, seed):
    kind = case["kind"]
    ins = _inputs(case, seed)
    if kind == "mul":
        n = ins[0][0]
        k = _batch_k(ins[0], case["wrap"])
        return _limbs(_redc(ins[1][0] * ins[1][1], n, _nprime(n, k), k), k)
    if kind == "transform":
        return _exact_transform(case, *ins)
    if kind == "mixed":
        budget = 16.0 / len(ins)
        return _some([_exact_rows(mods, xs, exps, base, _batch_k(mods, True), case["steps"], budget)
                      for base, mods, xs, exps in ins])
    mods, xs, exps = ins[0], ins[1], ins[2]
    if kind == "serve":
        mods = list(ins[3]) + mods[len(ins[3]):]
    return _some(_exact_rows(mods, xs, exps, case["base"], _batch_k(mods, case.get("wrap", True)), case["steps"]))


def _exact_transform(case, a, b, scales):
    """Coefficient q of scale * a * b mod each prime, q < L/2 in the real part of element q and the
    others in the imaginary parts, from one big-integer product with 16-byte coefficients."""
    length, k, n = case["len"], case["k"], case["len"] // 2
    p1, p2 = (1 << 31) - 1, (1 << 61) - 1
    m31 = np.zeros((case["count"], n, 2), np.uint32)
    m61 = np.zeros((case["count"], n, 2), np.int64)

    def spread(v):
        w = np.zeros((k, 4), dtype="<u4")
        w[:, 0] = v
        return int.from_bytes(w.tobytes(), "little")

    for v in range(case["count"]):
        prod = spread(a[v]) * spread(b[v]) * int(scales[v])
        raw = prod.to_bytes(16 * length, "little")
        co = [int.from_bytes(raw[16 * q:16 * q + 16], "little") for q in range(length)]
        m31[v] = np.array([c % p1 for c in co], np.uint32).reshape(2, n).T
        m61[v] = np.array([c % p2 for c in co], np.int64).reshape(2, n).T
    return {"m31": m31.reshape(-1, 2), "m61": m61.reshape(-1, 2)}
