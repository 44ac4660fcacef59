// DevArena (device/arena.hpp) over counted host calls: what is freed when,
// and what a dry arena counts.  Prints "arena ok".
#include <cstdio>
#include <random>

#include "arena.hpp"

#define REQUIRE(x)                                          \
    do {                                                    \
        if (!(x)) {                                         \
            std::printf("line %d: %s\n", __LINE__, #x);     \
            return 1;                                       \
        }                                                   \
    } while (0)

int main() {
    const size_t MiB = size_t(1) << 20;
    // a buffer with memory of its own is freed by release, whatever its size; one in a chunk stays
    for (size_t n : {2 * MiB, 8 * MiB - 512, 8 * MiB, 8 * MiB + 512, 100 * MiB}) {
        htf::DevArena a;
        void *small = nullptr, *big = nullptr;
        REQUIRE(a.get(&small, 1000) == cudaSuccess && a.get(&big, n) == cudaSuccess);
        REQUIRE(fake.bytes == 8 * MiB + n && a.bytes() == fake.bytes);
        a.release(big);
        REQUIRE(fake.bytes == 8 * MiB && a.bytes() == fake.bytes);
        a.release(small);
        REQUIRE(fake.bytes == 8 * MiB);
        void *next = nullptr;
        REQUIRE(a.get(&next, 1000) == cudaSuccess && next == static_cast<char *>(small) + 1024);
    }
    REQUIRE(fake.bytes == 0 && fake.live.empty());
    // a dry arena counts what a real one takes, and allocates nothing
    std::mt19937_64 rng(1);
    for (int rep = 0; rep < 20; ++rep) {
        htf::DevArena a, dry(true);
        const int before = fake.mallocs;
        for (int i = 0; i < 100; ++i) {
            const size_t n = size_t(1) << (rng() % 25);
            const size_t bytes = n + rng() % n;
            void *p = nullptr;
            REQUIRE(dry.get(&p, bytes) == cudaSuccess && p == nullptr);
            REQUIRE(fake.mallocs == before);
        }
        rng.seed(1);
        for (int r = 0; r < rep; ++r)
            for (int i = 0; i < 200; ++i) rng();
        for (int i = 0; i < 100; ++i) {
            const size_t n = size_t(1) << (rng() % 25);
            const size_t bytes = n + rng() % n;
            void *p = nullptr;
            REQUIRE(a.get(&p, bytes) == cudaSuccess);
        }
        REQUIRE(a.bytes() == dry.bytes() && a.bytes() == fake.bytes);
    }
    REQUIRE(fake.bytes == 0);
    // no room for a chunk: the buffer alone, and an error only when that does not fit either
    {
        htf::DevArena a, b;
        fake.limit = 4 * MiB;
        void *p = nullptr;
        REQUIRE(a.get(&p, 1 * MiB) == cudaSuccess && fake.bytes == 1 * MiB && fake.errors_cleared == 1);
        REQUIRE(a.get(&p, 5 * MiB) == cudaErrorMemoryAllocation && fake.bytes == 1 * MiB);
        a.swap(b);
        REQUIRE(a.bytes() == 0 && b.bytes() == 1 * MiB);
        a.clear();
        REQUIRE(fake.bytes == 1 * MiB);
    }
    REQUIRE(fake.bytes == 0 && fake.mallocs == fake.frees);
    std::printf("arena ok\n");
    return 0;
}
