// A staged download where threads cannot be started, and where copies fail. Arguments: how many threads
// may be started, which copy is the first to fail (-1: none), and whether memory can be registered. Prints the result of the download and
// whether all bytes arrived.
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>

#include <cstdio>

#include "host_copy.hpp"

namespace {
std::atomic<int> may_start{0};
}

// In front of the C library's: the thread class of the standard library calls it.
extern "C" int pthread_create(pthread_t* thread, const pthread_attr_t* attributes, void* (*body)(void*), void* argument) {
    if (may_start-- <= 0) return EAGAIN;
    using Create = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
    return reinterpret_cast<Create>(dlsym(RTLD_NEXT, "pthread_create"))(thread, attributes, body, argument);
}

int main(int argc, char** argv) {
    if (argc != 4) return 2;
    may_start = std::atoi(argv[1]);
    if (std::atoi(argv[2]) >= 0) fake::fail_after = std::atoi(argv[2]);
    fake::may_register = std::atoi(argv[3]) != 0;
    msx::HostCopier copier;
    // The first copy into pages that nothing has touched, which makes the lanes; then pieces of all sizes,
    // into fresh pages and into the same ones again.
    for (uint64_t bytes : {(40ull << 20) + 12345, 1ull << 18, (1ull << 18) - 1, (1ull << 20) + 3, (2ull << 20) - 1, 2ull << 20, (5ull << 20) + 77, (18ull << 20) - 1, 18ull << 20}) {
        std::vector<char> from(bytes);
        for (uint64_t i = 0; i < bytes; ++i) from[i] = static_cast<char>(i * 2654435761u >> 13);
        char* const to = static_cast<char*>(mmap(nullptr, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
        for (int again = 0; again < 2; ++again) {
            const int rc = copier.to_host(0, to, from.data(), bytes, nullptr);
            const bool whole = std::memcmp(to, from.data(), bytes) == 0;
            if (rc != 0 || !whole) {
                std::printf("%d %s\n", rc, whole ? "whole" : "not whole");
                return 0;
            }
            std::memset(to, 0, bytes);
        }
        munmap(to, bytes);
    }
    std::printf("0 whole\n");
    return 0;
}
