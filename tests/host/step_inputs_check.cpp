// Random sequences of what a plan's owner and a run's host loop do with its inputs, against a model that keeps every value apart: the
// plan's, and the run's until a step accepts it. Argument: the seed. Prints what went wrong, or "ok".
#include "step_inputs.hpp"

#include <cstdio>
#include <cstdlib>
#include <random>

constexpr int kSlots = 8;

int main(int argc, char** argv) {
    std::mt19937 draw(argc > 1 ? std::atoi(argv[1]) : 0);
    const std::vector<uint64_t> sizes = {4, 8, 64, 16, 4096};
    const size_t n = sizes.size();
    msx::StepInputs inputs;
    uint64_t total = 0;
    std::vector<uint64_t> offsets;
    for (uint64_t bytes : sizes) {
        offsets.push_back(total);
        inputs.add(total, bytes);
        total += bytes;
    }
    std::vector<std::vector<char>> memory(kSlots, std::vector<char>(total, 0x55));
    char* slots[kSlots];
    for (int s = 0; s < kSlots; ++s) slots[s] = memory[s].data();
    inputs.use_slots(slots);

    std::vector<std::vector<char>> plan(n), run(n);  // run: empty where the run has set nothing
    std::vector<char> staged(n, 0);                  // the run's value lies in `inputs`
    for (size_t i = 0; i < n; ++i) plan[i].assign(sizes[i], 0);
    uint64_t steps = 0, finished = 0, taken = 0;
    bool changed = true;
    std::vector<std::vector<char>> in_flight(kSlots);  // what a step that has not run reads
    auto bad = [&](const char* what) {
        std::printf("step %llu: %s\n", static_cast<unsigned long long>(steps), what);
        std::exit(0);
    };
    auto value = [&](size_t i) {
        std::vector<char> v(sizes[i]);
        for (char& c : v) c = static_cast<char>(draw());
        return v;
    };
    auto try_open = [&] {
        if (steps < kSlots || steps - kSlots < finished) inputs.open(static_cast<int>(steps % kSlots));
    };
    auto check = [&] {
        for (int s = 0; s < kSlots; ++s)
            if (!in_flight[s].empty() && in_flight[s] != memory[s]) bad("a slot that a step still reads was written");
        for (size_t i = 0; i < n; ++i)
            if (staged[i] && std::memcmp(inputs.run_value(i), run[i].data(), sizes[i]) != 0) bad("the run's value is lost");
    };
    for (int turn = 0; turn < 4000; ++turn) {
        const size_t i = draw() % n;
        switch (draw() % 7) {
            case 0: {  // the plan's owner sets an input
                plan[i] = value(i);
                changed = true;
                try_open();
                inputs.set(i, plan[i].data());
                break;
            }
            case 1: case 2: {  // the run sets one
                run[i] = value(i);
                try_open();
                staged[i] = inputs.stage(i, run[i].data());
                break;
            }
            case 3: {  // a step of the run takes its batch, or the first few inputs of it before one is refused
                const size_t upto = draw() % 4 ? n : draw() % n;
                for (size_t j = 0; j < upto; ++j) {
                    if (run[j].empty()) continue;
                    changed = changed || plan[j] != run[j] || !staged[j];
                    plan[j] = run[j];
                    try_open();
                    if (staged[j]) inputs.accept(j);
                    else inputs.set(j, run[j].data());
                }
                break;
            }
            case 4: case 5: {  // a step is submitted
                while (steps >= kSlots && steps - kSlots >= finished) in_flight[finished++ % kSlots].clear();
                const bool take = inputs.changed();
                if (changed && !take) bad("what was set does not reach the step");
                if (take) inputs.open(static_cast<int>(steps % kSlots));
                inputs.submitted();
                if (inputs.changed() || inputs.open()) bad("a submitted step leaves its inputs open");
                if (take) {
                    ++taken;
                    const std::vector<char>& slot = memory[steps % kSlots];
                    for (size_t j = 0; j < n; ++j)
                        if (std::memcmp(slot.data() + offsets[j], plan[j].data(), sizes[j]) != 0) bad("the step reads something else than the plan's value");
                    in_flight[steps % kSlots] = slot;
                }
                changed = false;
                ++steps;
                break;
            }
            default: {  // some steps have run; a profiled one reads the plan's values too
                while (finished < steps && draw() % 4) in_flight[finished++ % kSlots].clear();
                if (finished == steps && draw() % 4 == 0) {
                    try_open();
                    const int from = inputs.complete();
                    for (size_t j = 0; j < n; ++j)
                        if (std::memcmp(slots[from] + offsets[j], plan[j].data(), sizes[j]) != 0) bad("a profiled step reads something else than the plan's value");
                }
            }
        }
        check();
    }
    std::printf(steps > 500 && taken > 200 ? "ok\n" : "too few steps\n");
    return 0;
}
