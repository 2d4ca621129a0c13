"""The shapes run chooses by itself (no counterpart in the reference): wide blocks for batches that
leave SMs idle, slots taken in rotation where they do not fill whole waves, clusters of eight blocks
at L = 131072. Raw limbs equal those of the same batch stepped another way."""
import random

import numpy as np
import pytest

import common
from montmul_b200 import ModBatch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from montmul_b200 import B200
    return B200()


def batch(gpu, bits, slots, nbits, base=3, seed=1):
    """Odd moduli of `bits` bits (the last one 2^bits - 1), random values, exponents of nbits[i] bits."""
    rng = random.Random(f"{bits} {slots} {seed}")
    mods = [rng.getrandbits(bits) | (1 << (bits - 1)) | 1 for _ in range(slots - 1)] + [(1 << bits) - 1]
    b = ModBatch(gpu, mods, base)
    for i, n in enumerate(mods):
        b.load_raw(i, 2 * n - 1 if i == slots - 1 else rng.randrange(2 * n))
        b.set_exponent(i, rng.getrandbits(nbits[i]) | (1 << (nbits[i] - 1)) if nbits[i] else 0)
    return b


def raw(b):
    be, st = b.backend_and_state()
    return np.array(be.read_all(st))


# Transform lengths with wide shapes (L = 128 to 4096): the top of a bucket, an odd size, and
# more slots than the widest shape holds at once (which takes the next one).
@pytest.mark.parametrize("bits,slots", [(16 * (1 << e) - 4, s) for e in range(7, 13) for s in (1, 3)] +
                         [(1500, 2), (4097, 400), (9001, 300), (33_000, 160)])
def test_wide_shapes_same_raw_as_default_shape(gpu, bits, slots):
    nbits = [9 + i % 3 for i in range(slots)]
    a, b = batch(gpu, bits, slots, nbits), batch(gpu, bits, slots, nbits)
    be, st = b.backend_and_state()
    be.set_schedule(st, 0, 0, 0.0, be.get_schedule(st)["threads"])   # a named shape stays
    a.run(100)
    b.run(100)
    assert np.array_equal(raw(a), raw(b))


# L = 16384 holds one slot per SM, L = 32768 and 65536 a cluster per 2 and 4 SMs: a few slots
# more than fit, with exponents that end at different steps, in one run and step by step (which
# does not rotate).
@pytest.mark.parametrize("bits,slots,steps", [(200_000, 150, 24), (500_000, 77, 12), (1_000_000, 38, 12)])
def test_rotation_same_raw_as_single_steps(gpu, bits, slots, steps):
    nbits = [steps if i % 5 else 1 + i % steps for i in range(slots)]
    a, b = batch(gpu, bits, slots, nbits, base=2), batch(gpu, bits, slots, nbits, base=2)
    be, st = a.backend_and_state()
    before = be.launches(st)
    a.run(steps)
    assert be.launches(st) - before > 1 and all(a.remaining(i) == 0 for i in range(slots))
    for _ in range(steps):
        b.run(1)
    assert np.array_equal(raw(a), raw(b))


def test_clusters_of_eight_same_raw_as_global_mode(gpu):
    """L = 131072: run takes clusters of eight blocks, a plan's items run in global mode."""
    from montmul_b200.backend import Plan
    for bits in (1_048_574, 2_097_148):
        a, b = batch(gpu, bits, 2, [6, 4]), batch(gpu, bits, 2, [6, 4])
        a.run(6)
        plan = Plan([b], 6)
        plan.run(6)
        plan.close()
        assert a.params.len == 131072 and np.array_equal(raw(a), raw(b))


def test_queued_runs_in_rotation_do_not_wait_on_the_host(gpu):
    """run_async returns at once however many runs are queued behind each other, in rotation too."""
    import time
    slots, steps = 150, 60
    b = batch(gpu, 200_000, slots, [6 * steps] * slots, base=2)
    be, st = b.backend_and_state()
    be.run_async(st, steps)   # uploads the exponents
    be.sync(st)
    t = time.perf_counter()
    be.run_async(st, steps)
    be.sync(st)
    one = time.perf_counter() - t
    before = be.launches(st)
    t = time.perf_counter()
    for _ in range(4):
        be.run_async(st, steps)
    host = time.perf_counter() - t
    assert be.launches(st) - before > 4
    be.sync(st)
    assert host < 0.5 * one, (host, one)


def test_rotation_in_a_run_of_many_launches(gpu):
    """More than 64 launches' worth of steps: still in rotation (71 launches of 148 slots; one launch over
    all slots after another would be 70)."""
    slots, steps = 150, 140
    nbits = [steps - i % 3 for i in range(slots)]
    a, b = batch(gpu, 200_000, slots, nbits), batch(gpu, 200_000, slots, nbits)
    be, st = a.backend_and_state()
    be.set_schedule(st, 0, 2)
    before = be.launches(st)
    a.run(steps)
    assert gpu.sm_count() != 148 or be.launches(st) - before == 71
    for _ in range(steps):
        b.run(1)
    assert np.array_equal(raw(a), raw(b))
