// A staged download where threads cannot be started, and where copies fail. Arguments: how many threads
// may be started, and which copy is the first to fail (-1: none). Prints the result of the download and
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
    if (argc != 3) return 2;
    may_start = std::atoi(argv[1]);
    if (std::atoi(argv[2]) >= 0) fake::fail_after = std::atoi(argv[2]);
    const uint64_t bytes = (40ull << 20) + 12345;
    std::vector<char> from(bytes), to(bytes, 0);
    for (uint64_t i = 0; i < bytes; ++i) from[i] = static_cast<char>(i * 2654435761u >> 13);
    msx::HostCopier copier;
    const int rc = copier.to_host(0, to.data(), from.data(), bytes, nullptr);
    std::printf("%d %s\n", rc, to == from ? "whole" : "not whole");
    return 0;
}
