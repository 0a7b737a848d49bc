// A bounded map from a few whole numbers to a value that is costly to make.  Host code only.
#pragma once
#include <array>
#include <cstddef>
#include <cstdint>
#include <vector>

namespace lb200 {

// kSets (a power of two) sets of kWays entries; a key belongs to one set, and a set that is full gives up its oldest entry.
// A look-up compares kWays keys at most, however many are kept.  Not for several threads at once: `thread_local`.
template <typename Value, int kWords, int kSets, int kWays>
class KeyedCache {
public:
    typedef std::array<int64_t, kWords> Key;
    const Value* find(const Key& key) const {
        if (entries_.empty()) return nullptr;
        const Entry* set = &entries_[set_of(key) * kWays];
        for (int i = 0; i < kWays; ++i)
            if (set[i].used && set[i].key == key) return &set[i].value;
        return nullptr;
    }
    void put(const Key& key, const Value& value) {
        if (entries_.empty()) { entries_.resize((size_t)kSets * kWays); next_.resize(kSets); }
        const size_t s = set_of(key);
        Entry& e = entries_[s * kWays + next_[s]];
        next_[s] = (unsigned char)((next_[s] + 1) % kWays);
        e.used = true; e.key = key; e.value = value;
    }

private:
    static_assert((kSets & (kSets - 1)) == 0 && kWays <= 255, "sets are a power of two");
    struct Entry { bool used = false; Key key; Value value; };
    static size_t set_of(const Key& key) {
        uint64_t h = 0;
        for (int64_t w : key) {                            // every word, then every bit of it, moves the set (splitmix64's mixing steps)
            h = (h ^ (uint64_t)w) + 0x9e3779b97f4a7c15ull;
            h = (h ^ (h >> 30)) * 0xbf58476d1ce4e5b9ull;
            h = (h ^ (h >> 27)) * 0x94d049bb133111ebull;
            h ^= h >> 31;
        }
        return (size_t)(h & (uint64_t)(kSets - 1));
    }
    std::vector<Entry> entries_;                           // made at the first `put`
    std::vector<unsigned char> next_;
};

}  // namespace lb200
