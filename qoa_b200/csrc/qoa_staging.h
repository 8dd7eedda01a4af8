// qoa_staging.h — buffers handed out for the length of a call and kept for the
// next one, shared by all threads.
#pragma once
#include <cstddef>
#include <mutex>

namespace qoa {

// A::get() makes a buffer (null: none to be had), A::put() frees one. A buffer
// is made only when no kept one is free, so there are as many as calls were in
// flight at once; up to Most of them stay between calls.
template <typename A, size_t Most>
class KeptBuffers {
public:
    void* take() {
        {
            std::lock_guard<std::mutex> lk(mu_);
            if (n_) return kept_[--n_];
        }
        return A::get();
    }
    void give(void* p) {
        {
            std::lock_guard<std::mutex> lk(mu_);
            if (n_ < Most) {
                kept_[n_++] = p;
                return;
            }
        }
        A::put(p);
    }
    // Frees all free buffers but the first `keep`.
    void trim(size_t keep) {
        while (true) {
            void* p;
            {
                std::lock_guard<std::mutex> lk(mu_);
                if (n_ <= keep) return;
                p = kept_[--n_];
            }
            A::put(p);
        }
    }

private:
    std::mutex mu_;
    void* kept_[Most];  // the first n_ are free buffers
    size_t n_ = 0;
};

}  // namespace qoa
