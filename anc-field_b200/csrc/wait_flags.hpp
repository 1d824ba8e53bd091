// Error words that kernels raise when a wait runs out, one for each call in
// flight: a call takes one, cleared, before its launch and gives it back after
// its kernel has ended. (With one word for all calls on a device, clearing it for
// one call erased what another call's kernel had just raised.)
#pragma once

#include <cstddef>
#include <mutex>
#include <vector>

namespace afd {

class WaitFlags {
public:
    // `make` returns a new word that lives as long as the process (or throws)
    explicit WaitFlags(int* (*make)()) : make_(make) {}

    class Lease {
    public:
        explicit Lease(WaitFlags& from) : from_(from), word_(from.take()) { *word_ = 0; }
        ~Lease() { from_.give(word_); }
        Lease(const Lease&) = delete;
        Lease& operator=(const Lease&) = delete;
        int* word() const { return word_; }
        bool raised() const { return *static_cast<volatile int*>(word_) != 0; }

    private:
        WaitFlags& from_;
        int* word_;
    };

private:
    int* take() {
        std::lock_guard<std::mutex> lock(mu_);
        if (free_.empty()) {
            free_.reserve(made_ + 1);  // so that giving one back cannot fail
            int* w = make_();
            ++made_;
            return w;
        }
        int* w = free_.back();
        free_.pop_back();
        return w;
    }
    void give(int* w) {
        std::lock_guard<std::mutex> lock(mu_);
        free_.push_back(w);
    }
    std::mutex mu_;
    std::vector<int*> free_;
    size_t made_ = 0;
    int* (*make_)();
};

}  // namespace afd
