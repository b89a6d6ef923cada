// Barrier waits that ran out inside a kernel. Such a kernel stores a code to its context's word in mapped host memory, skips what it can no longer compute
// and returns; whoever next waits for the context's work on the host finds the code here and reports an error instead of results. Plain C++: a test on
// the host uses the same class.
#pragma once
#include <atomic>
#include <cstdint>
#include <mutex>

namespace uzu {

class WaitErrors {
public:
    unsigned int* word = nullptr;          // host address, 0: no wait ran out since it was last looked at
    unsigned int* device_word = nullptr;   // the same word for kernels

    // a command buffer starts encoding: its number
    uint64_t start() {
        std::lock_guard<std::mutex> lock(mutex_);
        return ++started_;
    }
    // The buffer's work is done: 0, or the code. It does not say which buffer's kernel gave up, so every buffer that had started by then reports it.
    unsigned int finished(uint64_t number) {
        std::lock_guard<std::mutex> lock(mutex_);
        collect();
        return number <= suspect_ ? code_ : 0u;
    }
    // 0, or the code if one was found since `seen` (of an engine: its passes run in no command buffer, or in one of its own)
    unsigned int since(uint64_t& seen) {
        std::lock_guard<std::mutex> lock(mutex_);
        collect();
        if (seen == found_) return 0;
        seen = found_;
        return code_;
    }
    uint64_t found() {
        std::lock_guard<std::mutex> lock(mutex_);
        return found_;
    }

private:
    void collect() {
        const unsigned int c = word ? __atomic_exchange_n(word, 0u, __ATOMIC_ACQ_REL) : 0u;
        if (!c) return;
        code_ = c;
        suspect_ = started_;
        ++found_;
    }
    std::mutex mutex_;
    uint64_t started_ = 0, suspect_ = 0, found_ = 0;
    unsigned int code_ = 0;
};

}  // namespace uzu
