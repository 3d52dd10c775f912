// The ring of pinned chunks is for large reads into memory that has no pages yet, once
// such reads have come to more than it costs to make; all bytes arrive on every route.
#include "fake_cudart.h"
#include "mpm_readback.h"

#include <cstdio>
#include <vector>

#include <sys/mman.h>

using namespace mpm;

static int bad = 0;
static std::vector<char> src;

// Reads `bytes` into fresh or written memory; `ring`: whether the chunks of the ring are expected.
static void read(const char* what, size_t bytes, bool fresh, bool ring, size_t pinned) {
    char* dst = static_cast<char*>(mmap(nullptr, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
    if (!fresh) std::memset(dst, 1, bytes);
    const FakeCounts before = fake;
    const cudaError_t e = ReadbackRing::get().read(nullptr, src.data(), dst, bytes);
    const bool same = std::memcmp(src.data(), dst, bytes) == 0;
    const int copies = fake.copies - before.copies;
    if (e != cudaSuccess || !same || (copies > 1) != ring || fake.pinned != pinned) {
        std::printf("%s: error %d, %s, %d copies, %zu bytes pinned for %zu\n", what, (int)e, same ? "same" : "other bytes", copies,
                    fake.pinned, pinned);
        ++bad;
    }
    munmap(dst, bytes);
}

int main() {
    constexpr size_t MB = 1 << 20, kRing = ReadbackRing::kChunk * ReadbackRing::kChunks;
    src.resize(64 * MB);
    for (size_t i = 0; i < src.size(); ++i) src[i] = (char)(i * 2654435761u >> 13);
    {
        ReadbackUser user;
        read("written, 12 MB", 12 * MB, false, false, 0);
        read("written, 64 MB", 64 * MB, false, false, 0);
        read("fresh, 12 MB, first", 12 * MB, true, false, 0);
        read("fresh, 12 MB, second", 12 * MB + 8, true, false, 0);
        read("fresh, below 8 MB", 8 * MB - 4, true, false, 0);
        read("fresh, 12 MB, third", 12 * MB, true, false, 0);
        read("fresh, 12 MB, fourth", 12 * MB, true, true, kRing);
        read("fresh, 8 MB", 8 * MB, true, true, kRing);
        read("fresh, ragged", 9 * MB + 12, true, true, kRing);
        read("written again", 12 * MB, false, false, kRing);
    }
    fake = FakeCounts{};
    {
        ReadbackUser user;  // a new start
        read("fresh, 12 MB, after the last user", 12 * MB, true, false, 0);
    }
    {
        ReadbackUser user;
        read("fresh, 46 MB, first", 46 * MB, true, true, kRing);
    }
    if (fake.unpins != 1) {
        std::printf("%d buffers given back\n", fake.unpins);
        ++bad;
    }
    return bad;
}
