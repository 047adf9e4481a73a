// What a context keeps of freed blocks: it goes back when an allocation of another context is
// refused, and when it is trimmed; blocks in use stay.
#include <cstdio>

#include "internal.h"
#include "runtime.h"

#define CHECK(x)                                         \
    do {                                                 \
        if (!(x)) {                                      \
            std::printf("%s does not hold\n", #x);       \
            return 1;                                    \
        }                                                \
    } while (0)

static size_t bytes() {
    size_t n = 0;
    for (const auto& b : fake::live) n += b.second;
    return n;
}

int main() {
    constexpr size_t MB = 1 << 20;
    mi_context *a = nullptr, *b = nullptr;
    CHECK(mi_context_create(0, &a) == MI_OK && mi_context_create(0, &b) == MI_OK);
    const size_t empty = bytes();
    void *used = nullptr, *kept = nullptr, *host = nullptr, *other = nullptr;
    CHECK(mi::dev_alloc_bytes(a, &used, 8 * MB) == cudaSuccess && mi::dev_alloc_bytes(a, &kept, 8 * MB) == cudaSuccess);
    CHECK(mi::pinned_alloc(a, &host, nullptr, MB) == cudaSuccess);
    mi::dev_free(a, kept);
    mi::pinned_free(a, host, MB);
    CHECK(bytes() == empty + 17 * MB);
    // another context's allocation is refused once: what the first one keeps goes, and it fits
    fake::allocations = 0;
    fake::fail_at = 0;
    CHECK(mi::dev_alloc_bytes(b, &other, 4 * MB) == cudaSuccess && other);
    fake::fail_at = -1;
    CHECK(bytes() == empty + 12 * MB);
    CHECK(!fake::live.count(kept) && fake::live.count(used) && fake::live.count(other));
    // refused again: the call fails, and the words the contexts wait with are refused, too
    fake::allocations = 0;
    fake::fail_at = 0;
    fake::fail_on = 1;
    void* none = nullptr;
    CHECK(mi::dev_alloc_bytes(b, &none, 4 * MB) == cudaErrorMemoryAllocation && !none);
    fake::fail_at = -1;
    // trimmed
    mi::dev_free(b, other);
    CHECK(bytes() >= empty + 12 * MB - 1);
    CHECK(mi_context_trim(b) == MI_OK);
    CHECK(bytes() <= empty + 8 * MB);
    mi::dev_free(a, used);
    CHECK(mi_context_destroy(a) == MI_OK && mi_context_destroy(b) == MI_OK);
    CHECK(bytes() == 0);
    std::printf("kept memory went back\n");
    return 0;
}
