// pinned_pool.hpp — a few pinned host buffers of one size that calls borrow for the arrays they copy to the device.
//
// Pinning and unpinning are slow driver calls that other streams can wait for, so no call does either once the buffers stand: a call that asks for more than a
// buffer holds, that finds all of them in use or whose pinning is refused gets none and copies from pageable memory, as it would without the pool.
#pragma once
#include <cstddef>
#include <cstdint>
#include <mutex>

namespace oa {

class PinnedPool {
public:
    static constexpr size_t BUF_BYTES = 1 << 20;
    static constexpr int BUFFERS = 8;
    explicit PinnedPool(uint8_t* (*pin)(size_t)) : pin_(pin) {}      // pin: page-locked memory, nullptr where there is none
    PinnedPool(const PinnedPool&) = delete;
    uint8_t* take(size_t bytes) {
        if (bytes > BUF_BYTES) return nullptr;
        std::lock_guard<std::mutex> lk(mu_);
        if (n_free_ > 0) return free_[--n_free_];
        if (made_ == BUFFERS) return nullptr;
        uint8_t* p = pin_(BUF_BYTES);
        made_ += p != nullptr;
        return p;
    }
    void give(uint8_t* p) { std::lock_guard<std::mutex> lk(mu_); free_[n_free_++] = p; }

private:
    uint8_t* (*pin_)(size_t);
    std::mutex mu_;
    uint8_t* free_[BUFFERS];
    int n_free_ = 0, made_ = 0;
};

// Memory of one call: a buffer of the pool, or pageable
class CallMemory {
public:
    CallMemory(PinnedPool& pool, size_t bytes) : pool_(pool), p_(pool.take(bytes)), pinned_(p_ != nullptr) { if (!pinned_) p_ = new uint8_t[bytes ? bytes : 1]; }
    CallMemory(const CallMemory&) = delete;
    ~CallMemory() { if (pinned_) pool_.give(p_); else delete[] p_; }
    uint8_t* get() const { return p_; }
    bool pinned() const { return pinned_; }

private:
    PinnedPool& pool_;
    uint8_t* p_;
    bool pinned_;
};

}  // namespace oa
