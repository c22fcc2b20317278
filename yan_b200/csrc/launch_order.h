#pragma once
// Which kernels let their successors in the stream start before they have waited for what is in front of them.
// Plain host code, so that the rules can be walked without a GPU.

#include <atomic>
#include <mutex>

namespace yan {

// Whether the quantizer as a call of its own lets its successor start before it has waited for what is in front of it.
// Under the promise that the call in front of a GEMM does not write its weights, the GEMM loads them before its own wait; that call
// is this quantizer, so whatever lies in front of the quantizer has to be complete when the GEMM starts.  Without the promise every
// GEMM waits before it reads anything.
// It pays for the small batches alone, in a graph of (quantizer, GEMM), us before / after the wait: M=16 N=7168 K=2048 5.7 / 6.4,
// M=64 N=7168 K=2048 6.9 / 7.6, but M=128 N=2048 K=7168 10.85 / 10.87, M=256 N=1024 K=1024 5.41 / 5.43, M=1111 N=5136 K=3072
// 24.2 / 24.2.  Larger quantizers behind one another crowd the SMs with CTAs that wait: 1111 x 3072 3.9 / 2.8, 2048 x 1024 3.5 / 2.2.
inline bool cast_releases_early(unsigned m, bool constant_weights) { return m <= 64 && !constant_weights; }

// Where a GEMM is launched, and under which state of the promise.
struct LaunchPlace {
    unsigned era = 0;  // odd: weights are promised to be constant (see ConstantWeights)
    int device = 0;
    const void* stream = nullptr;
    unsigned long long capture = 0;  // id of the graph capture that records the launch, 0 outside of one
    bool known = true;               // false: the three above do not tell two streams apart

    bool operator==(const LaunchPlace& o) const {
        return era == o.era && device == o.device && stream == o.stream && capture == o.capture;
    }
};

// The promise, which may be switched between any two calls: a quantizer launched while it was off lets its successor start before the
// kernel in front of the quantizer has completed.  So the first GEMM of a stream after the promise was made waits before it loads
// weights, and later ones, behind it, need not.  A call reads the state once, as an era that every switch ends; what was settled
// in one era says nothing about the next.  The places settled last are kept, one that is not among them counts as new.
class ConstantWeights {
public:
    void set(bool promised) {
        std::lock_guard<std::mutex> lock(mutex_);
        if (promised != (era_.load() % 2 != 0)) era_.fetch_add(1);
    }
    unsigned era() const { return era_.load(); }
    static bool promised(unsigned era) { return era % 2 != 0; }

    // Whether a GEMM at `place` may load weights before it waits.
    bool holds(const LaunchPlace& place) {
        if (!promised(place.era) || !place.known) return false;
        std::lock_guard<std::mutex> lock(mutex_);
        return find(place);
    }
    // A GEMM has been launched there.
    void settle(const LaunchPlace& place) {
        if (!promised(place.era) || !place.known) return;
        std::lock_guard<std::mutex> lock(mutex_);
        if (!find(place)) settled_[next_++ % kPlaces] = place;
    }

private:
    static constexpr unsigned kPlaces = 64;
    bool find(const LaunchPlace& place) const {
        for (const LaunchPlace& p : settled_)
            if (p == place) return true;
        return false;
    }
    std::atomic<unsigned> era_{0};
    std::mutex mutex_;
    LaunchPlace settled_[kPlaces];
    unsigned next_ = 0;
};

}  // namespace yan
