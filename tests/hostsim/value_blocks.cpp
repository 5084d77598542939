// The store of page-locked value blocks (value_blocks.h) with ordinary memory
// in place of page-locked, for the test suite.
#include "../../gpjson_b200/csrc/value_blocks.h"

namespace {

int64_t locks = 0, locked_bytes = 0;
constexpr size_t kHead = 64;

struct Pages {
    static void* lock(size_t size) {
        auto* p = static_cast<uint8_t*>(std::malloc(size + kHead));
        std::memcpy(p, &size, sizeof size);
        ++locks;
        locked_bytes += static_cast<int64_t>(size);
        return p + kHead;
    }
    static void unlock(void* p) {
        size_t size = 0;
        std::memcpy(&size, static_cast<uint8_t*>(p) - kHead, sizeof size);
        locked_bytes -= static_cast<int64_t>(size);
        std::free(static_cast<uint8_t*>(p) - kHead);
    }
};

gpj::ValueBlocks<Pages> store;

}  // namespace

extern "C" {

void vb_context(int created) { created ? store.context_created() : store.context_destroyed(); }
uint8_t* vb_take(uint64_t size, uint64_t* cap, int* pinned) {
    size_t c = 0;
    bool p = false;
    uint8_t* b = store.take(size, &c, &p);
    *cap = c;
    *pinned = p;
    return b;
}
void vb_give(uint8_t* p, uint64_t cap, int pinned) { store.give(p, cap, pinned != 0); }
int64_t vb_locks() { return locks; }
int64_t vb_locked_bytes() { return locked_bytes; }

}  // extern "C"
