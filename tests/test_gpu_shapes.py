"""The shapes run chooses by itself (no counterpart in the reference): wide blocks for batches that
leave SMs idle, slots taken in rotation where they do not fill whole waves, clusters of eight blocks
at L = 131072. Raw limbs equal those of the same batch stepped another way."""
import random

import numpy as np
import pytest

import common
from montmul_b200 import ModBatch, tune

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


def ran(b):
    """What the launches of the batch's last run took."""
    be, st = b.backend_and_state()
    return be.last_run(st)


def wide_threads(length):
    """Threads of the default shape and of the wide ones, widest first (mm_abi.h wide_threads_for)."""
    default = tune.threads_for(length.bit_length() - 2)
    return default, [f * default for f in (4, 2) if f * default <= 512]


# Transform lengths with wide shapes (L = 128 to 4096): the top of a bucket and odd sizes. test_each_wide_shape
# has the slot counts at which each shape runs.
@pytest.mark.parametrize("bits,slots", [(16 * (1 << e) - 4, s) for e in range(7, 13) for s in (1, 3)] +
                         [(1500, 2), (4097, 400), (9001, 300), (33_000, 160)])
def test_wide_shapes_same_raw_as_default_shape(gpu, bits, slots):
    nbits = [9 + i % 3 for i in range(slots)]
    a, b = batch(gpu, bits, slots, nbits), batch(gpu, bits, slots, nbits)
    be, st = b.backend_and_state()
    be.set_schedule(st, 0, 0, 0.0, be.get_schedule(st)["threads"])   # a named shape stays
    a.run(100)
    b.run(100)
    default, wide = wide_threads(a.params.len)
    assert ran(b)["threads"] == default
    if slots <= gpu.sm_count():
        assert ran(a)["threads"] == wide[0]
    assert np.array_equal(raw(a), raw(b))


@pytest.mark.parametrize("length", [1 << e for e in range(7, 13)])
def test_each_wide_shape(gpu, length):
    """The slot counts of each shape: the widest one up to a block of 512 threads (or blocks of that many
    together) per SM, the next one beyond, the default from five per SM on."""
    sms = gpu.sm_count()
    default, wide = wide_threads(length)
    seen = []
    for slots in (sms * (512 // wide[0]), sms * (512 // wide[0]) + 1, 5 * sms + 1):
        nbits = [9 + i % 3 for i in range(slots)]
        a, b = batch(gpu, 16 * length - 4, slots, nbits), batch(gpu, 16 * length - 4, slots, nbits)
        be, st = b.backend_and_state()
        be.set_schedule(st, 0, 0, 0.0, default)
        a.run(100)
        b.run(100)
        seen.append(ran(a)["threads"])
        assert ran(b)["threads"] == default and np.array_equal(raw(a), raw(b))
    assert seen == [wide[0], (wide + [default])[1], default]


class Pinned:
    """A device whose batches name the default block shape of their length."""

    def __init__(self, dev):
        self.dev = dev

    def __getattr__(self, name):
        return getattr(self.dev, name)

    def create(self, *a):
        st = self.dev.create(*a)
        self.dev.set_schedule(st, 0, 0, 0.0, self.dev.get_schedule(st)["threads"])
        return st


@pytest.mark.parametrize("wraparound", [True, False])
@pytest.mark.parametrize("length", [1 << e for e in range(7, 13)])
def test_default_shape_same_raw_as_oracle(oracle, length, wraparound):
    """The shape that full batches run, on few slots: at the top of the bucket and just above the one below."""
    from montmul_b200 import B200
    make = oracle.OracleBackend.wraparound if wraparound else oracle.OracleBackend.plain
    dev = Pinned(B200(wraparound=wraparound))
    common.same_raw(lambda: dev, make, 16 * length - 36, 2, 12)
    common.same_raw(lambda: dev, make, 8 * length + 1, 3, 12)


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
    assert ran(a)["slots"] < slots
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
        assert (ran(a)["mode"], ran(a)["blocks"]) == ("cluster", 8)


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


# (bits, wraparound, forced global, slots beyond what the device holds, steps): several blocks per SM, the
# plain REDC, the global-mode kernel; 25 clusters of eight (18 fit on 148 SMs).
@pytest.mark.parametrize("bits,wrap,forced,more,steps", [
    (8_000, True, False, 40, 40), (12_000, True, False, 10, 40), (20_011, False, False, 5, 40), (131_068, True, True, 1, 12),
    (2_097_148, True, False, None, 4)])
def test_rotation_in_every_mode(bits, wrap, forced, more, steps):
    from montmul_b200 import B200
    dev = B200(wraparound=wrap, force_global=forced)
    be, st = ModBatch(dev, [(1 << (bits - 1)) | 1], 2).backend_and_state()
    resident = be.blocks_per_sm(st) * dev.sm_count()
    slots = 25 if more is None else resident + more
    nbits = [steps if i % 9 else 1 + i % steps for i in range(slots)]
    a, b = batch(dev, bits, slots, nbits, base=2), batch(dev, bits, slots, nbits, base=2)
    a.run(steps)
    assert ran(a)["slots"] < 25 if more is None else ran(a)["slots"] == resident
    for _ in range(steps):
        b.run(1)
    assert np.array_equal(raw(a), raw(b))


def test_bare_steps_in_rotation_leave_x_alone(gpu):
    slots, steps = 150, 24
    b = batch(gpu, 200_000, slots, [steps] * slots)
    before = raw(b)
    be, st = b.backend_and_state()
    be.run_bare(st, steps)
    assert ran(b)["slots"] < slots and np.array_equal(raw(b), before) and b.remaining(0) == 0


def test_a_named_mode_holds_at_131072(gpu, oracle):
    """Clusters of eight are run's own choice: a schedule that names global mode, and force_global, keep it (and
    the global kernel its oracle comparison at this length); a tuned row in the batch's mode names none."""
    from montmul_b200 import B200
    forced = B200(force_global=True)

    class Named:
        def __getattr__(self, name):
            return getattr(gpu, name)

        def create(self, *a):
            st = gpu.create(*a)
            gpu.set_schedule(st, 1)
            return st

    class Checked:
        """Asserts after every run that it took global mode."""

        def __init__(self, dev):
            self.dev = dev

        def __getattr__(self, name):
            return getattr(self.dev, name)

        def run(self, st, bits):
            self.dev.run(st, bits)
            assert self.dev.last_run(st)["mode"] == "global"

    for dev in (Checked(forced), Checked(Named())):
        common.same_raw(lambda: dev, oracle.OracleBackend.wraparound, 16 * 131072 - 4, 2, 3)
    b = batch(gpu, 2_000_000, 1, [4])
    b.run(1)
    assert ran(b)["mode"] == "cluster"
    tune.apply(b, {gpu.device_name(): {"131072": {"global": 1, "launch_steps": 64, "step_ns": 2e4}}})
    b.run(1)
    assert ran(b)["mode"] == "cluster"
    be, st = b.backend_and_state()
    be.set_schedule(st, 1)
    b.run(1)
    assert ran(b)["mode"] == "global"


def test_wide_blocks_only_while_they_fit_beside_other_batches():
    """L = 512: 64 slots run in 128-thread blocks alone and beside 64 more of the length, in the default
    32-thread ones beside a batch of another length: with run while that one has steps under way, with run_async
    (which cannot see what is enqueued after it) while it exists. The limbs are the same."""
    from montmul_b200 import B200
    dev = B200()
    a, twin = batch(dev, 8_000, 64, [400] * 64), batch(dev, 8_000, 64, [400] * 64)
    be, st = a.backend_and_state()
    tst = twin.backend_and_state()[1]
    be.set_schedule(tst, 0, 0, 0.0, 32)
    twin.run(400)
    seen = []

    def step(run):
        run(st, 50)
        be.sync(st)
        seen.append(ran(a)["threads"])

    step(be.run)
    step(be.run_async)
    other = batch(dev, 100_000, 8, [4000] * 8)
    ost = other.backend_and_state()[1]
    step(be.run)
    step(be.run_async)
    be.run_async(ost, 4000)   # about 0.4 s
    step(be.run)
    assert be.busy(ost)
    be.sync(ost)
    step(be.run)
    del other, ost
    step(be.run_async)
    step(be.run)
    assert seen == [128, 128, 128, 32, 32, 128, 128, 128]
    assert np.array_equal(raw(a), raw(twin))


def test_batches_run_by_threads_keep_their_limbs():
    """Four threads, each with its own batches, which come and go while the others run."""
    import threading
    from montmul_b200 import B200
    dev = B200()
    want = [batch(dev, bits, 40, [300] * 40) for bits in (4_000, 8_000, 16_000, 33_000)]
    for b in want:
        b.run(300)
    got = [[] for _ in want]

    def work(i, bits):
        for _ in range(3):
            b = batch(dev, bits, 40, [300] * 40)
            b.run(300)
            got[i].append(raw(b))

    threads = [threading.Thread(target=work, args=(i, bits)) for i, bits in enumerate((4_000, 8_000, 16_000, 33_000))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for b, rows in zip(want, got):
        assert len(rows) == 3 and all(np.array_equal(raw(b), r) for r in rows)
