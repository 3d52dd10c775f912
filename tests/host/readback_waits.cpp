// Reads that take the driver's copy wait once, for the copy behind the kernels.
#include "fake_cudart.h"
#include "mpm_readback.h"

#include <cstdio>
#include <vector>

using namespace mpm;

static int bad = 0;

static void read(const char* what, size_t bytes, bool pinned, int waits) {
    std::vector<char> src(bytes), dst(bytes, 1);
    for (size_t i = 0; i < bytes; ++i) src[i] = (char)(i * 2654435761u >> 13);
    fake_pinned[0] = pinned ? dst.data() : nullptr;
    fake_pinned[1] = pinned ? dst.data() + bytes : nullptr;
    fake = FakeCounts{};
    const cudaError_t e = ReadbackRing::get().read(nullptr, src.data(), dst.data(), bytes);
    if (e != cudaSuccess || src != dst || fake.syncs != waits) {
        std::printf("%s: error %d, %s, %d waits for %d\n", what, (int)e, src == dst ? "same" : "other bytes", fake.syncs, waits);
        ++bad;
    }
}

int main() {
    ReadbackUser user;
    read("small", 1000, false, 1);
    read("a small field's limit", 256 << 10, false, 1);
    read("a picture", 2160000, false, 1);
    read("a large field's limit", (8 << 20) - 4, false, 1);
    read("a large field into pinned memory", 12 << 20, true, 1);
    return bad;
}
