// Captured rounds by their key, bounded: when the table is full the round that has waited longest for its next use goes, not the
// whole table, so that the rounds of a service that moves between a few shapes stay captured.
#pragma once
#include <cstddef>
#include <map>
#include <vector>

namespace lcu {

template <class Value, class Drop>
class RoundTable {
public:
    RoundTable(size_t most, Drop drop) : most_(most), drop_(drop) {}
    ~RoundTable() { clear(); }
    RoundTable(const RoundTable &) = delete;
    RoundTable &operator=(const RoundTable &) = delete;

    Value *find(const std::vector<int> &key) {
        const auto it = rounds_.find(key);
        if (it == rounds_.end()) return nullptr;
        it->second.used = ++clock_;
        return &it->second.value;
    }
    Value *insert(const std::vector<int> &key, const Value &value) {  // (the key is not in the table)
        if (rounds_.size() >= most_) {
            auto oldest = rounds_.begin();
            for (auto it = rounds_.begin(); it != rounds_.end(); ++it)
                if (it->second.used < oldest->second.used) oldest = it;
            drop_(oldest->second.value);
            rounds_.erase(oldest);
        }
        return &rounds_.emplace(key, Entry{value, ++clock_}).first->second.value;
    }
    void clear() {
        for (auto &r : rounds_) drop_(r.second.value);
        rounds_.clear();
    }
    size_t size() const { return rounds_.size(); }

private:
    struct Entry {
        Value value;
        unsigned long long used;
    };
    std::map<std::vector<int>, Entry> rounds_;
    size_t most_;
    Drop drop_;
    unsigned long long clock_ = 0;
};

}  // namespace lcu
