// How run splits its steps into launches (host code): one launch over all slots, or launches that take
// the slots in rotation. A rotation needs no list on the device: round r gives every slot the steps
// from r `chunk` on, the launches cut the sequence of rounds into runs of consecutive slots, and
// each run is a StepRange in the launch's arguments.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <functional>
#include <queue>
#include <vector>

#include "mm_common.h"

namespace mm {

// Whether `active` slots of a length that global mode also runs are stepped in clusters, of which the
// device holds `clusters` at once (none where its SMs are shared out in smaller groups).
inline bool clusters_pay(size_t active, size_t sms, int clusters) { return clusters > 0 && active <= sms; }

// The steps per launch with which `slots` slots of which `resident` fit the device at once finish
// `steps` steps soonest when launches take the slots in rotation, `resident` at a time; 0 where one
// launch over all slots is as good. That launch takes ceil(slots / resident) whole waves, the last
// one of which may leave most SMs idle (37 clusters of L = 65536 where 36 fit: two waves for the
// work of one); in rotation the idle places go to the next round's slots and only the last launch
// is partly empty. A launch costs launch_us beyond its steps (its start, and the wait for its slowest
// block), so a chunk is no shorter than pays for that: 13 us measured for clusters, 0 to 26 us in shared
// memory (L = 1,024, 905 slots on 888 places: 5 launches of 2 steps 631 us, 9 of 8 4,133, a step is 57; L =
// 8,192, 301 on 296: 17 of 4 11,550, 33 of 2 11,790, a step is 166), 30 to 48 us with one block per SM (L =
// 16,384: 395 slots x 64 in 11 launches 33.4 ms, in 43 34.3; 503 x 256 in 17 165.3, in 109 170.6). The chunks
// tried are those of 64 numbers of rounds, from the fewest that `most` steps per launch allow: past
// that the last launch's idle places no longer count.
// half_wave: a step of a launch that fills at most half the places, of a full one's. 1 where a step is as
// long however few blocks an SM holds; at L = 8192, two blocks per SM of which one alone keeps the
// pipes nearly as busy, 0.53 (97 us against 2 x 91). There a last wave that is half full idles little:
// in rotation 444 slots took 1.005 and 1,006 slots (3.4 waves) 1.008 to 1.04 times as long.
inline size_t rotation_chunk(size_t slots, size_t resident, size_t steps, size_t most, double step_us, double launch_us,
                             double half_wave) {
    if (slots <= resident || slots % resident == 0 || slots > 16 * resident) return 0;
    const size_t full = slots / resident, rest = slots % resident;
    double best = 0.97 * ((double)full + (2 * rest <= resident ? half_wave : 1.0)) * (double)steps * step_us;
    size_t chunk = 0;
    const size_t fewest = (steps + most - 1) / most;
    for (size_t r = fewest; r < fewest + 64 && r <= steps; ++r) {
        const size_t s = (steps + r - 1) / r, rounds = (steps + s - 1) / s;
        const size_t launches = (slots * rounds + resident - 1) / resident;
        const double us = (double)launches * ((double)s * step_us + launch_us);
        if (us < best) {
            best = us;
            chunk = s;
        }
    }
    return chunk;
}

// The steps until a launch ends whose blocks run steps[i] steps each and start in order, `resident` at
// once, the next where one ends.
inline double launch_steps_of(const std::vector<uint32_t>& steps, size_t resident) {
    std::priority_queue<uint64_t, std::vector<uint64_t>, std::greater<uint64_t>> ends;
    uint64_t last = 0;
    for (const uint32_t s : steps) {
        if (!s) continue;
        uint64_t start = 0;
        if (ends.size() == resident) {
            start = ends.top();
            ends.pop();
        }
        ends.push(start + s);
        last = std::max(last, start + s);
    }
    return (double)last;
}

// Whether a rotation of `chunk` steps beats launches over all slots when slot i has left[i] of `steps`
// steps to do. rotation_chunk takes every slot to have them all; where exponents end early, launches
// over all slots refill their places by themselves (148 places, 13 % of 539 slots with 100 steps and
// the others with 9: a rotation of 34 would take 1.5 times as long), while in a rotation a launch
// lasts as long as its longest slot. At most 64 of the launches are looked at, evenly spaced.
// A slot without steps left costs each round about 5 us of one place.
inline bool rotation_pays(const std::vector<uint32_t>& left, size_t resident, size_t steps, size_t most, size_t chunk,
                          double step_us, double launch_us) {
    const size_t launches = (steps + most - 1) / most, every = (launches + 63) / 64;
    std::vector<uint32_t> now(left.size());
    double whole = 0;
    for (size_t l = 0; l < launches; l += every) {
        for (size_t i = 0; i < left.size(); ++i)
            now[i] = (uint32_t)std::min(most, left[i] > l * most ? left[i] - l * most : 0);
        whole += (double)std::min(every, launches - l) * launch_steps_of(now, resident) * step_us;
    }
    std::vector<uint32_t> ends(left);
    std::sort(ends.begin(), ends.end());
    double turns = (double)chunk * step_us + launch_us;   // the last launch
    size_t done = 0;                                      // slots without steps left
    for (size_t r = 0; r * chunk < steps; ++r) {
        while (done < ends.size() && ends[done] <= r * chunk) ++done;
        const double live = (double)(ends.size() - done) / (double)resident;
        turns += std::max(1.0, live) * ((double)std::min(chunk, steps - r * chunk) * step_us + launch_us) +
                 5.0 * (double)done / (double)resident;
    }
    return turns < 0.97 * whole;
}

// The launches of one run: `steps` steps on each of `slots` slots (fewer where its exponent ends),
// `chunk` per launch, in launches of at most `resident` slots with steps left. Slots without steps
// left are passed over: as blocks that return at once, and not counted. A launch covers at most
// `slots` consecutive slots, so no slot is in a launch twice.
class Rotation {
  public:
    Rotation(size_t slots, size_t resident, size_t steps, size_t chunk)
        : slots_(slots), resident_(resident), steps_(steps), chunk_(chunk) {}

    // The next launch that has a slot with steps left; false after the last one. pos and nbits:
    // per slot, the steps done (advance keeps pos) and the exponent's length.
    bool next(const uint32_t* pos, const uint32_t* nbits, StepRange* r, size_t* count) {
        while (round_ * chunk_ < steps_) {
            size_t n = 0, live = 0, at = slot_, round = round_;
            if (resident_ >= slots_) {   // a whole round: any slot with steps left will do
                for (; n < slots_ && !live; ++n) live += pos[n] < nbits[n];
                n = slots_;
                ++round;
            }
            while (n < slots_ && live < resident_ && round * chunk_ < steps_) {
                live += pos[at] < nbits[at];
                ++n;
                if (++at == slots_) {
                    at = 0;
                    ++round;
                }
            }
            *r = StepRange{(uint32_t)slot_, (uint32_t)slots_, bits(round_), bits(round_ + 1)};
            *count = n;
            slot_ = at;
            round_ = round;
            if (live) return true;
        }
        return false;
    }

    // What the launch does to pos.
    static void advance(const StepRange& r, size_t count, uint32_t* pos, const uint32_t* nbits) {
        const auto step = [&](size_t from, size_t to, uint32_t bits) {
            for (size_t s = from; s < to; ++s) pos[s] += std::min(bits, nbits[s] - pos[s]);
        };
        const size_t end = r.first + count;
        step(r.first, std::min<size_t>(end, r.slots), r.bits);
        if (end > r.slots) step(0, end - r.slots, r.bits_next);
    }

  private:
    uint32_t bits(size_t round) const {
        const size_t done = round * chunk_;
        return (uint32_t)(done < steps_ ? std::min(chunk_, steps_ - done) : 0);
    }

    size_t slots_, resident_, steps_, chunk_;
    size_t slot_ = 0, round_ = 0;   // where the next launch begins
};

}  // namespace mm
