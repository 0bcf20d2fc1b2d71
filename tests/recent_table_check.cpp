// Scenarios for csrc/recent_table.h on the CPU: keys like those of tensor maps, values that follow from the key.
#include "recent_table.h"

#include <atomic>
#include <cstdio>
#include <string>
#include <thread>
#include <vector>

using namespace b200;

#define CHECK(cond)                                                     \
    do {                                                                \
        if (!(cond)) {                                                  \
            std::printf("line %d: %s\n", __LINE__, #cond);              \
            return 1;                                                   \
        }                                                               \
    } while (0)

struct Key {
    uint64_t base, dims[5], strides[4];
    uint32_t box[5], rank, swizzle, type;
};
struct Value {
    uint64_t word[16];
};
constexpr int kEntries = 512;
using Table = RecentTable<Key, Value, kEntries>;

// weight-sized blocks one behind the other
static Key key(uint64_t i, uint64_t step = 7168 * 2048) {
    Key k;
    std::memset(&k, 0, sizeof(k));
    k.base = 0x7f0000000000ull + i * step;
    k.dims[0] = k.strides[0] = 2048;
    k.dims[1] = 7168;
    k.dims[2] = 1;
    k.box[0] = k.box[1] = 128;
    k.rank = 3;
    return k;
}
static Value value(const Key& k) {
    Value v;
    for (int i = 0; i < 16; ++i) v.word[i] = k.base * 31 + k.dims[1] + i;
    return v;
}
// what the launcher does: 0 found, 1 made and kept, -1 found with another key's value
static int ask(Table& t, const Key& k) {
    const Value want = value(k);
    Value got;
    if (!t.find(k, &got)) {
        t.add(k, want);
        return 1;
    }
    return std::memcmp(&got, &want, sizeof(got)) == 0 ? 0 : -1;
}

// a loop over as many keys as are kept makes each of them once, whatever the distance of their addresses
static int loop_is_kept() {
    for (uint64_t step : {16ull, 128ull, 4096ull, 7168ull * 2048, 18432ull * 7168, 1ull << 33})
        for (int count : {1, 2, 40, 48, 60, 64, 128, 300, kEntries}) {
            static Table t;
            const uint64_t from = 1000000 * (step % 1009) + 1000 * count;          // keys of their own in the one table
            for (int pass = 0; pass < 3; ++pass)
                for (int i = 0; i < count; ++i) CHECK(ask(t, key(from + i, step)) == (pass == 0));
        }
    return 0;
}
// more keys than are kept: the oldest go, and what is found is right
static int oldest_go() {
    static Table t;
    for (int pass = 0; pass < 3; ++pass)
        for (int i = 0; i < 3 * kEntries + 7; ++i) CHECK(ask(t, key(i)) == 1);
    for (int i = 3 * kEntries + 6; i >= 2 * kEntries + 7; --i) CHECK(ask(t, key(i)) == 0);
    CHECK(ask(t, key(2 * kEntries + 6)) == 1);                                       // makes room: the oldest one goes for it
    CHECK(ask(t, key(2 * kEntries + 7)) == 1);
    CHECK(ask(t, key(3 * kEntries + 6)) == 0);
    // keys that differ in one field each
    Key k = key(0), one = k;
    one.box[1] = 16;
    CHECK(ask(t, k) == 1 && ask(t, one) == 1 && ask(t, k) == 0 && ask(t, one) == 0);
    return 0;
}
static int threads() {
    static Table t;
    std::atomic<int> wrong{0};
    std::vector<std::thread> all;
    for (int n = 0; n < 8; ++n)
        all.emplace_back([&, n] {
            for (int i = 0; i < 200000; ++i) wrong += ask(t, key((i * (n + 1) + n) % (n < 4 ? 40 : 700))) < 0;
        });
    for (auto& x : all) x.join();
    CHECK(wrong == 0);
    return 0;
}

int main(int argc, char** argv) {
    const std::string s = argc > 1 ? argv[1] : "";
    const int rc = s == "loop_is_kept" ? loop_is_kept() : s == "oldest_go" ? oldest_go() : s == "threads" ? threads() : 2;
    if (rc == 0) std::printf("ok\n");
    return rc;
}
