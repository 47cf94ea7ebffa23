// KeptBuffers: the calls of a stream of large updates with small read-outs
// between them allocate once; the large call's buffers go when it stays away;
// buffers left out by a failed call come back; a failed allocation keeps nothing.
#include <cstdio>
#include <cstdlib>
#include <set>

#include "kept_buffers.h"

#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main() {
    std::set<void*> live;
    size_t made = 0, held = 0;
    bool full = false;
    size_t limit = ~(size_t)0 >> 1;
    char* next = (char*)4096;
    static size_t size_of[4096];
    auto alloc = [&](size_t n) -> void* {
        if (full || held + n > limit) return nullptr;
        size_of[made] = n;
        void* p = next + 16 * made++;
        live.insert(p);
        held += n;
        return p;
    };
    auto release = [&](void* p) {
        held -= size_of[((char*)p - (char*)4096) / 16];
        live.erase(p);
    };
    const size_t MB = 1u << 20;
    cgb::KeptBuffers b;
    auto update = [&] {  // 12 arrays, 480 MiB in all
        b.give_back(release);
        std::set<void*> mine;
        for (int i = 1; i <= 12; ++i) mine.insert(b.take((10 + 5 * i) * MB, alloc, release));
        if (mine.size() != 12 || mine.count(nullptr)) std::abort();
        b.give_back(release);
    };
    auto readout = [&] {
        b.give_back(release);
        if (!b.take(3 * MB, alloc, release)) std::abort();
        b.give_back(release);
    };
    for (int pass = 0; pass < 50; ++pass) {
        update();
        for (int d = 0; d < 12; ++d) readout();
        if (pass == 0) continue;
        static size_t first;
        if (pass == 1) first = made;
        CHECK(made == first);  // nothing allocated after the first passes
    }
    CHECK(held <= 3 * 520 * MB);
    for (int i = 0; i < 3 * (int)cgb::KeptBuffers::kWindow; ++i) readout();
    CHECK(held <= cgb::KeptBuffers::kFloor);
    update();
    for (int i = 1; i <= 5; ++i) b.take(30 * MB, alloc, release);  // a call that fails here
    const size_t before = made;
    b.give_back(release);
    update();
    CHECK(made <= before + 12);
    limit = held + 100 * MB;
    CHECK(b.take(400 * MB, alloc, release) != nullptr);  // the free buffers make room
    b.give_back(release);
    full = true;
    CHECK(b.take(1000 * MB, alloc, release) == nullptr);
    full = false;
    b.release_all(release);
    CHECK(live.empty() && held == 0);
    std::puts("ok");
}
