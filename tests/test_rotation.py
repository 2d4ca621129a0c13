"""How run splits its steps into launches (montmul_b200/csrc/mm_rotation.hpp, built for the host with
g++): every slot gets the steps it has left, no more than the device holds are stepped at once, and
no slot is in a launch twice, for any slot counts and exponents. CPU only."""
import heapq
import os
import random
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "montmul_b200", "csrc")
SOURCE = r'''
#include "mm_rotation.hpp"
#include <cstdio>
#include <cstring>
#include <vector>
// "split slots resident steps chunk pos... nbits...": one line per launch, "first bits bits_next: slot/steps ...".
// "pays slots resident steps most chunk step_us launch_us left...": 1 or 0.
// "chunk slots resident steps most step_us launch_us half_wave": the rotation's steps per launch.
int main() {
    char what[16];
    size_t slots, resident, steps, last;
    while (std::scanf("%15s %zu %zu %zu %zu", what, &slots, &resident, &steps, &last) == 5) {
        if (!std::strcmp(what, "chunk")) {
            double step_us, launch_us, half_wave;
            if (std::scanf("%lf %lf %lf", &step_us, &launch_us, &half_wave) != 3) return 1;
            std::printf("%zu\n", mm::rotation_chunk(slots, resident, steps, last, step_us, launch_us, half_wave));
            continue;
        }
        if (!std::strcmp(what, "clusters")) {   // "clusters active sms clusters 0"
            std::printf("%d\n", (int)mm::clusters_pay(slots, resident, (int)steps));
            continue;
        }
        if (!std::strcmp(what, "pays")) {
            size_t chunk;
            double step_us, launch_us;
            if (std::scanf("%zu %lf %lf", &chunk, &step_us, &launch_us) != 3) return 1;
            std::vector<uint32_t> left(slots);
            for (auto& v : left) if (std::scanf("%u", &v) != 1) return 1;
            std::printf("%d\n", (int)mm::rotation_pays(left, resident, steps, last, chunk, step_us, launch_us));
            continue;
        }
        std::vector<uint32_t> pos(slots), nbits(slots);
        for (auto& v : pos) if (std::scanf("%u", &v) != 1) return 1;
        for (auto& v : nbits) if (std::scanf("%u", &v) != 1) return 1;
        mm::Rotation rot(slots, resident, steps, last);
        mm::StepRange r;
        size_t count;
        while (rot.next(pos.data(), nbits.data(), &r, &count)) {
            std::printf("%u %u %u:", r.first, r.bits, r.bits_next);
            for (uint32_t i = 0; i < count; ++i) {
                uint32_t bits;
                const uint32_t s = mm::range_slot(r, i, bits);
                std::printf(" %u/%u", s, bits);
            }
            std::printf("\n");
            rot.advance(r, count, pos.data(), nbits.data());
        }
        std::printf("end");
        for (auto v : pos) std::printf(" %u", v);
        std::printf("\n");
    }
}
'''


@pytest.fixture(scope="module")
def ask(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not found")
    d = tmp_path_factory.mktemp("rotation")
    (d / "r.cpp").write_text(SOURCE)
    subprocess.run([gxx, "-std=c++17", "-I", CSRC, str(d / "r.cpp"), "-o", str(d / "r")], check=True)
    return lambda q: subprocess.run([str(d / "r")], input=q, check=True, capture_output=True, text=True).stdout.splitlines()


def cases(n=400):
    rng = random.Random(5)
    for i in range(n):
        slots = rng.randint(1, 40)
        steps = rng.randint(1, 50)
        nbits = [rng.choice([0, 1, steps, rng.randint(0, 60)]) if i % 3 else steps for _ in range(slots)]
        pos = [rng.randint(0, b) if i % 2 else 0 for b in nbits]
        yield slots, rng.choice([slots, rng.randint(1, slots)]), steps, rng.randint(1, steps), pos, nbits


def test_every_slot_gets_its_steps(ask):
    all_cases = list(cases())
    out = iter(ask("\n".join("split " + " ".join(map(str, [*c[:4], *c[4], *c[5]])) for c in all_cases)))
    for slots, resident, steps, chunk, pos, nbits in all_cases:
        at = list(pos)
        for line in out:
            if line.startswith("end"):
                break
            items = [tuple(map(int, w.split("/"))) for w in line.split(":")[1].split()]
            assert len({s for s, _ in items}) == len(items) <= slots and all(0 <= s < slots for s, _ in items)
            live = [s for s, _ in items if at[s] < nbits[s]]
            assert 0 < len(live) <= resident and all(b <= chunk for _, b in items)
            for s, b in items:
                at[s] = min(nbits[s], at[s] + b)
        want = [min(b, p + steps) for p, b in zip(pos, nbits)]
        assert at == want == [int(v) for v in line.split()[1:]]


def test_full_launches_while_enough_slots_have_steps_left(ask):
    """Equal exponents: every launch but the last holds `resident` slots."""
    for slots, resident, steps, chunk in ((37, 18, 30, 1), (150, 148, 24, 3), (7, 3, 10, 4)):
        lines = ask(f"split {slots} {resident} {steps} {chunk} " + " ".join(["0"] * slots + [str(steps)] * slots))[:-1]
        rounds = -(-steps // chunk)
        assert len(lines) == -(-slots * rounds // resident)
        assert all(len(line.split(":")[1].split()) == resident for line in lines[:-1])


# (slots, resident, steps per launch at most, us per step): 2,368 slots at L = 1,024, 500 at L = 8,192,
# 37 clusters of L = 65,536, 150 slots at L = 16,384.
@pytest.mark.parametrize("slots,resident,most,us", [(2368, 888, 64, 94.0), (500, 296, 64, 186.0), (37, 36, 512, 370.0), (150, 148, 512, 223.0)])
def test_rotation_does_not_depend_on_the_length_of_a_run(ask, slots, resident, most, us):
    for steps in (200, 65 * most, 100_000, 1_000_000):
        chunk = int(ask(f"chunk {slots} {resident} {steps} {most} {us} 20 1")[0])
        assert 0 < chunk <= min(most, steps)
        launches = -(-slots * -(-steps // chunk) // resident)
        assert launches * (chunk * us + 20) < 1.05 * slots / resident * steps * us + chunk * us


def whole_time(left, resident, most, us, launch_us):
    """One launch over all slots after another: blocks start in order as places come free."""
    t, left = 0.0, list(left)
    while any(left):
        ends = [0.0] * resident
        for r in left:
            if r:
                heapq.heapreplace(ends, ends[0] + min(r, most) * us)
        t += max(ends) + launch_us
        left = [r - min(r, most) for r in left]
    return t


def rotation_time(ask, left, resident, steps, chunk, us, launch_us):
    """Launch after launch, each as long as its longest slot."""
    t, left = 0.0, list(left)
    for line in ask(f"split {len(left)} {resident} {steps} {chunk} " + " ".join(["0"] * len(left) + list(map(str, left))))[:-1]:
        longest = 0
        for w in line.split(":")[1].split():
            s, b = map(int, w.split("/"))
            longest = max(longest, min(b, left[s]))
            left[s] -= min(b, left[s])
        t += longest * us + launch_us
    return t


def test_rotation_of_unequal_exponents_pays_where_it_is_taken(ask):
    """Random exponent lengths: where rotation_pays takes a rotation it is not slower than launches over
    all slots (by both models written out), and it does take some."""
    rng = random.Random(7)
    taken = slower = 0
    for _ in range(150):
        resident = rng.choice([18, 36, 148])
        slots = int(resident * rng.uniform(1.02, 4))
        steps, most, us = rng.choice([100, 300, 1000]), rng.choice([64, 512]), rng.choice([20, 100, 400])
        share, lo = rng.random(), rng.randint(0, steps)
        kind = rng.choice(["two", "even", "sorted"])
        left = [steps if rng.random() < share else (lo if kind != "even" else rng.randint(0, steps)) for _ in range(slots)]
        left[rng.randrange(slots)] = steps
        if kind == "sorted":
            left.sort()
        active = sum(v > 0 for v in left)
        chunk = int(ask(f"chunk {active} {resident} {steps} {most} {us} 20 1")[0])
        if not chunk:
            continue
        ratio = rotation_time(ask, left, resident, steps, chunk, us, 20) / whole_time(left, resident, most, us, 0)
        if ask(f"pays {slots} {resident} {steps} {most} {chunk} {us} 20 " + " ".join(map(str, left)))[0] == "1":
            taken += 1
            assert ratio < 1.02, (ratio, slots, resident, steps, most, us, left)
        else:
            slower += ratio > 1.05
    assert taken > 20 and slower > 5


def test_half_full_last_wave_at_8192(ask):
    """Two blocks per SM, one alone at 0.94 of their rate: waves of 0.1 and 0.8 of the places are taken in
    rotation, a last wave near half full is not."""
    chunk = lambda slots, half: int(ask(f"chunk {slots} 296 256 64 186 90 {half}")[0])
    for slots, rotates in ((301, True), (370, True), (444, False), (540, True), (800, True), (1006, False)):
        assert (chunk(slots, 0.53) > 0) == rotates, slots
    assert all(chunk(slots, 1) > 0 for slots in (301, 370, 444, 540, 800, 1006))


def test_clusters_need_room_for_one(ask):
    assert ask("clusters 24 148 18 0 clusters 148 148 18 0 clusters 149 148 18 0 clusters 24 148 0 0") == ["1", "1", "0", "0"]
