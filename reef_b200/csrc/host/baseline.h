// What a real-time request takes without best-effort work beside it: the time that the padding throttle's target is
// measured against.
#pragma once
#include <algorithm>
#include <cstdint>
#include <vector>

namespace reef {
namespace server {

// A replay can have more than one speed (ResNet-152 on one executor: 832 us by itself; 806 us, at times 832, as an unpadded
// window between padded ones), so neither the least sample nor a mean says what to compare with.  Two kinds of samples, a
// median each: requests served while there was no best-effort work (`alone`, the latency that a client knows), and probe
// windows among padded ones.  The larger counts: a client that was ever served alone is promised its latency alone plus
// the target (by the least of the last four samples of either kind, ResNet-152 beside four clients ran 3 % above its
// latency alone instead of 6.5, with the best-effort share that goes with it); one that never was has the probes only.
class ReplayBaseline {
public:
    void add_alone(double ns) {
        if (alone_.seen++ >= kCold) alone_.add(ns);   // the first requests of a model find nothing in the caches
    }
    void add_probe(double ns) { probes_.add(ns); }
    double ns() const {
        const double probe = probes_.median(4);
        return alone_.n < kAlone ? probe : std::max(probe, alone_.median(kAlone));
    }

private:
    static const uint32_t kCold = 3, kAlone = 8;
    struct Ring {
        double v[8] = {0};
        uint32_t n = 0, seen = 0;
        void add(double ns) { v[n++ % 8] = ns; }
        // of the last `count` samples, or of as many as there are (the lower of the middle two: a disturbance only lengthens)
        double median(uint32_t count) const {
            std::vector<double> s;
            const uint32_t have = std::min(n, count);
            for (uint32_t i = 0; i < have; i++) s.push_back(v[(n - 1 - i) % 8]);
            std::sort(s.begin(), s.end());
            return have == 0 ? 0.0 : s[(have - 1) / 2];
        }
    } alone_, probes_;
};

}  // namespace server
}  // namespace reef
