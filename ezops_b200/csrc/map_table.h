// A bounded table of computed values: sets of sixteen entries, the least recently used entry of a full set replaced.
#pragma once
#include <cstddef>
#include <cstdint>

namespace ezb {

inline uint64_t hash_mix(uint64_t h, uint64_t v) {  // one round of a multiply-xorshift hash
    h = (h ^ v) * 0x9E3779B97F4A7C15ull;
    return h ^ (h >> 29);
}

// Key: operator== and hash().  Not synchronised: the caller holds a lock.
template <class Key, class Value, size_t Sets>
class MapTable {
public:
    static constexpr size_t kWays = 16;

    // The value stored for `key`, or null.  Valid until the next put().
    const Value* find(const Key& key) {
        Entry* set = set_of(key);
        for (size_t i = 0; i < kWays; ++i)
            if (set[i].used && set[i].key == key) {
                set[i].used = ++clock_;
                return &set[i].value;
            }
        return nullptr;
    }

    void put(const Key& key, const Value& value) {
        Entry* set = set_of(key);
        Entry* oldest = set;
        for (size_t i = 1; i < kWays; ++i)
            if (set[i].used < oldest->used) oldest = &set[i];
        oldest->key = key, oldest->value = value, oldest->used = ++clock_;
    }

private:
    struct Entry {
        Value value;
        Key key;
        uint64_t used;  // 0: empty
    };
    Entry* set_of(const Key& key) { return entries_ + (size_t)(key.hash() % Sets) * kWays; }

    Entry entries_[Sets * kWays] = {};
    uint64_t clock_ = 0;
};

}  // namespace ezb
