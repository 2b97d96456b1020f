// The page-locked buffer of a context, lent to one call at a time (host code only; plain C++).
//
// A call that finds the buffer lent, as one from a second thread may, gets none and delivers its results through
// memory of its own: no call's totals or records are ever read by another.
#pragma once
#include <atomic>
#include <stdint.h>

struct StageBuffer {
    uint64_t *words = nullptr;       // from the first loan on
    std::atomic<bool> lent{false};
};

class StageLoan {
public:
    StageLoan() = default;
    // `alloc` makes the buffer at the first loan; null when it cannot be had.
    template <class Alloc>
    StageLoan(StageBuffer &buffer, Alloc alloc) {
        if (buffer.lent.exchange(true, std::memory_order_acquire)) return;
        if (!buffer.words) buffer.words = alloc();
        if (buffer.words) of = &buffer;
        else buffer.lent.store(false, std::memory_order_release);
    }
    StageLoan(StageLoan &&other) noexcept : of(other.of) { other.of = nullptr; }
    StageLoan &operator=(StageLoan &&other) noexcept {
        if (this != &other) {
            give_back();
            of = other.of;
            other.of = nullptr;
        }
        return *this;
    }
    StageLoan(const StageLoan &) = delete;
    StageLoan &operator=(const StageLoan &) = delete;
    ~StageLoan() { give_back(); }
    // The buffer, or null; valid until the loan ends.
    uint64_t *get() const { return of ? of->words : nullptr; }

private:
    void give_back() {
        if (of) of->lent.store(false, std::memory_order_release);
        of = nullptr;
    }
    StageBuffer *of = nullptr;
};
