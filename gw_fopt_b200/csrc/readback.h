// Device -> host copies of a call's results (host code; no CUDA header, the runtime is a parameter).
#pragma once

#include <cstddef>
#include <cstring>
#include <mutex>
#include <vector>

namespace bgw {

// Staging blocks that outlive a handle: each call takes one and gives it back, at most kIdle wait for the next call
// and the others are freed.  Any number of threads; the lock is not held while a block is made or freed.
class BlockPool {
public:
    static constexpr size_t kIdle = 4;
    template <class Make>
    void* take(Make&& make) {
        {
            std::lock_guard<std::mutex> lock(mutex_);
            if (n_idle_ > 0) return idle_[--n_idle_];
        }
        return make();
    }
    template <class Free>
    void give(void* block, Free&& free_block) {
        {
            std::lock_guard<std::mutex> lock(mutex_);
            if (n_idle_ < kIdle) {
                idle_[n_idle_++] = block;
                return;
            }
        }
        free_block(block);
    }

private:
    std::mutex mutex_;
    void* idle_[kIdle] = {};
    size_t n_idle_ = 0;
};

// Small results are queued into a staging block of pinned memory and handed over after the one synchronisation (a copy
// to pageable memory waits for the device by itself); larger ones are copied directly.  With a status (error counters
// of the call, queued first) nothing reaches a result's place before the status was looked at: a call that fails
// leaves the caller's arrays alone.
//
// Rt: void copy(void* dst, const void* src, size_t bytes), which queues a device -> host copy, and void wait(), which
// waits for everything queued; both throw on failure.  void* take() makes the staging block (kBytes), void give(block)
// gets it back when no copy into it is in flight any more.
template <class Rt>
class Readback {
public:
    static constexpr size_t kBytes = 1 << 18;  // of the staging block

    explicit Readback(Rt rt) : rt_(rt), block_(static_cast<char*>(rt_.take())) {}
    ~Readback() {
        if (used_ > 0) {  // not waited for: an error on the way
            try {
                rt_.wait();
            } catch (...) {
                return;  // the copies' end is not known: the block is not used again
            }
        }
        rt_.give(block_);
    }
    Readback(const Readback&) = delete;
    Readback& operator=(const Readback&) = delete;

    // At most once, before any result.
    void status(void* dst, const void* src, size_t bytes) {
        stage(dst, src, bytes);
        has_status_ = true;
    }
    void add(void* dst, const void* src, size_t bytes) {
        if (used_ + bytes <= kBytes)
            stage(dst, src, bytes);
        else if (has_status_)
            large_.push_back({dst, src, bytes});
        else
            rt_.copy(dst, src, bytes);
    }
    // Waits; `check` looks at the status and throws when the results are invalid.
    template <class Check>
    void wait(Check&& check) {
        rt_.wait();
        used_ = 0;
        size_t q = 0;
        if (has_status_) {
            deliver(staged_[q++]);
            check();
        }
        for (; q < staged_.size(); ++q) deliver(staged_[q]);
        for (const Part& p : large_) rt_.copy(p.dst, p.src, p.bytes);
        if (!large_.empty()) rt_.wait();
        staged_.clear();
        large_.clear();
        has_status_ = false;
    }
    void wait() {
        wait([] {});
    }

private:
    struct Part {
        void* dst;
        const void* src;  // in the staging block or, of a large part, on the device
        size_t bytes;
    };
    void stage(void* dst, const void* src, size_t bytes) {
        char* at = block_ + used_;
        used_ = (used_ + bytes + 15) & ~(size_t)15;
        rt_.copy(at, src, bytes);
        staged_.push_back({dst, at, bytes});
    }
    static void deliver(const Part& p) { std::memcpy(p.dst, p.src, p.bytes); }

    Rt rt_;
    char* block_;
    size_t used_ = 0;
    bool has_status_ = false;
    std::vector<Part> staged_, large_;
};

}  // namespace bgw
