// Answers of the device that do not change while the process runs, by key.  A question that failed (a negative answer)
// counts as 0 for this caller and is asked again the next time.
#pragma once
#include <mutex>
#include <unordered_map>

namespace rt {

class AskedOnce {
    std::mutex mu_;
    std::unordered_map<int, int> known_;

  public:
    template <typename Ask> int get(int key, Ask ask) {
        std::lock_guard<std::mutex> lk(mu_);
        auto it = known_.find(key);
        if (it != known_.end()) return it->second;
        const int answer = ask();
        if (answer < 0) return 0;
        known_.emplace(key, answer);
        return answer;
    }
};

} // namespace rt
