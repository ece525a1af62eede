// Where a plan's inputs wait for the step that reads them.
//
// A step reads its inputs from the slot of its turn. What is set for the next step is written into that slot once
// (through a host image of the plan's and from there into the slot a megabyte of inputs took 80 us more a step); an
// input that is not set again follows from the slot before when the step is submitted. The slot of the next step can
// still be read by the step that used it last: nothing is written there, and nothing waits, before that one has run.
// What is set meanwhile is kept beside it.
//
// Two callers set inputs. `set` gives the plan a value: the next step has it, whoever submits that step. `stage` is for a run's
// host loop, whose batch is the run's own until one of the run's steps accepts it: it writes into the same place, but
// a step that is submitted without `accept` has the plan's value, and the run's waits aside.
#pragma once

#include <cstdint>
#include <cstring>
#include <utility>
#include <vector>

namespace msx {

class StepInputs {
public:
    // Bytes [offset, offset + bytes) of every slot are one input. The slots outlive this object.
    void add(uint64_t offset, uint64_t bytes) {
        inputs_.emplace_back();
        inputs_.back().offset = offset;
        inputs_.back().bytes = bytes;
    }
    void use_slots(char* const* slots) { slots_ = slots; }
    bool ready() const { return slots_ != nullptr; }
    bool open() const { return opened_ >= 0; }
    // Whether the next step takes its inputs over: a value was set since the last one did, or none ever was (zeros).
    bool changed() const { return changed_ || current_ < 0; }

    // No step in flight reads `slot`, and the next one will.
    void open(int slot) {
        if (open()) return;
        opened_ = slot;
        for (Input& in : inputs_) {
            in.here = slot == current_;
            if (!in.is_held) continue;
            std::memcpy(place(in), in.held.data(), in.bytes);
            in.here = true;
            in.is_held = false;
        }
    }

    // The plan's value of input i.
    void set(size_t i, const void* host) {
        Input& in = inputs_[i];
        if (in.pending || in.from_run) {
            const char* const now = run_value(i);
            in.aside.assign(now, now + in.bytes);
            in.is_aside = true;
        }
        write(in, host);
        in.pending = in.from_run = false;
    }

    // The run's value of input i, where its place in the open slot holds nothing that the plan still needs; else false,
    // and the run keeps the value itself.
    bool stage(size_t i, const void* host) {
        Input& in = inputs_[i];
        in.from_run = in.is_aside = false;
        if (!open() || (in.here && !in.pending)) return false;
        std::memcpy(place(in), host, in.bytes);
        in.here = in.pending = true;
        return true;
    }

    // Where the run's value of a staged input lies until something is set again.
    const char* run_value(size_t i) const {
        const Input& in = inputs_[i];
        return in.is_aside ? in.aside.data() : in.pending ? place(in) : plan_value(in);
    }

    // The run's value becomes the plan's.
    void accept(size_t i) {
        Input& in = inputs_[i];
        if (in.is_aside) {
            write(in, in.aside.data());
            in.is_aside = false;
        } else if (in.pending) {
            changed_ = true;
        }
        in.pending = false;
        in.from_run = true;
    }

    // What no step of the run has accepted leaves the open slot.
    void put_aside() {
        if (!open()) return;
        for (Input& in : inputs_) {
            if (!in.pending) continue;
            in.aside.assign(place(in), place(in) + in.bytes);
            in.is_aside = true;
            in.here = in.pending = false;
        }
    }

    // The open slot holds every input's plan value afterwards; returns it.
    int complete() {
        put_aside();
        for (Input& in : inputs_) {
            if (in.here) continue;
            if (current_ >= 0) std::memcpy(place(in), slots_[current_] + in.offset, in.bytes);
            else std::memset(place(in), 0, in.bytes);
            in.here = true;
        }
        return opened_;
    }

    // The step that reads the open slot is submitted; where nothing changed it reads what the one before left.
    void submitted() {
        put_aside();
        if (changed() && open()) {
            complete();
            current_ = opened_;
            changed_ = false;
        }
        opened_ = -1;
    }

private:
    struct Input {
        uint64_t offset = 0, bytes = 0;
        bool here = false;      // the open slot holds it: the plan's value or,
        bool pending = false;   // where no step has accepted it yet, the run's
        bool from_run = false;  // the plan's value is the run's last one
        bool is_held = false, is_aside = false;
        std::vector<char> held;   // the plan's value, set while no slot was open
        std::vector<char> aside;  // the run's value, where the plan has another
    };

    char* place(const Input& in) const { return slots_[opened_] + in.offset; }

    const char* plan_value(const Input& in) const {
        if (in.is_held) return in.held.data();
        if (open() && in.here) return place(in);
        return current_ >= 0 ? slots_[current_] + in.offset : nullptr;
    }

    void write(Input& in, const void* host) {
        if (open()) {
            std::memcpy(place(in), host, in.bytes);
            in.here = true;
        } else {
            const char* const from = static_cast<const char*>(host);
            in.held.assign(from, from + in.bytes);
            in.is_held = true;
        }
        changed_ = true;
    }

    std::vector<Input> inputs_;
    char* const* slots_ = nullptr;
    int opened_ = -1;   // the slot of the next step, once it may be written
    int current_ = -1;  // the slot of the last step that took its inputs over
    bool changed_ = false;
};

}  // namespace msx
