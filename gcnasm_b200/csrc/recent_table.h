// The results of the last kEntries different questions, found by hash; the oldest makes room.  Any loop over up to kEntries keys finds
// all of them from its second pass on, wherever their bytes lie: a key's place does not depend on its hash, only the way to it does.
// Host code without CUDA, safe with several threads.  Keys are compared byte by byte, so their padding has to be cleared.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cstring>
#include <mutex>

namespace b200 {

template <class Key, class Value, int kEntries>
class RecentTable {
  public:
    bool find(const Key& key, Value* value) {
        const uint32_t h = hash(key);
        std::lock_guard<std::mutex> lk(mu_);
        const int i = look_up(key, h);
        if (i < 0) return false;
        *value = slots_[i].value;
        return true;
    }
    void add(const Key& key, const Value& value) {
        const uint32_t h = hash(key);
        std::lock_guard<std::mutex> lk(mu_);
        if (look_up(key, h) >= 0) return;                 // another thread has asked the same meanwhile
        Slot& s = slots_[oldest_];
        if (s.used) {
            int* link = &heads_[s.hash % kChains];        // out of its chain
            while (*link - 1 != oldest_) link = &slots_[*link - 1].next;
            *link = s.next;
        }
        s.key = key;
        s.value = value;
        s.hash = h;
        s.used = true;
        s.next = heads_[h % kChains];
        heads_[h % kChains] = oldest_ + 1;
        oldest_ = (oldest_ + 1) % kEntries;
    }

  private:
    static constexpr int kChains = 2 * kEntries;
    struct Slot {
        Key key;
        Value value;
        uint32_t hash;
        int next;            // index + 1 of the next slot of the chain, 0: none
        bool used;
    };
    static uint32_t hash(const Key& key) {
        static_assert(sizeof(Key) % 16 == 0, "hashed word by word, two chains of products beside each other");
        uint64_t words[sizeof(Key) / 8], h = 0, g = 0;
        std::memcpy(words, &key, sizeof(key));
        for (size_t i = 0; i < sizeof(Key) / 8; i += 2) {
            h = (h ^ words[i]) * 0x9E3779B97F4A7C15ull;
            g = (g ^ words[i + 1]) * 0xD1342543DE82EF95ull;
        }
        h ^= g;
        return static_cast<uint32_t>((h ^ h >> 32) * 0x9E3779B97F4A7C15ull >> 32);
    }
    int look_up(const Key& key, uint32_t h) const {
        for (int i = heads_[h % kChains]; i != 0; i = slots_[i - 1].next)
            if (slots_[i - 1].hash == h && std::memcmp(&slots_[i - 1].key, &key, sizeof(key)) == 0) return i - 1;
        return -1;
    }
    Slot slots_[kEntries] = {};
    int heads_[kChains] = {};
    int oldest_ = 0;
    std::mutex mu_;
};

}  // namespace b200
