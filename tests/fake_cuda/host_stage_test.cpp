/* host_stage.h against the fake runtime beside it; exits 0 when every check holds. */
#include <cstdio>
#include <vector>

#include "host_stage.h"

using namespace apus;
using Bytes = std::vector<char>;

static FakeStream sa, sb;
static int bad = 0;
static void check(bool ok, const char *what, size_t n) {
    if (!ok) {
        printf("wrong: %s (%zu)\n", what, n);
        bad = 1;
    }
}
static Bytes pattern(size_t n, unsigned seed) {
    Bytes b(n);
    for (size_t i = 0; i < n; i++) b[i] = (char)((i * 2654435761u + seed * 97u) >> 13);
    return b;
}

int main() {
    HostStage hs;
    const size_t slot = HostStage::SLOT_BYTES;
    unsigned seed = 1;
    /* every number of pieces, their edges; pageable and page-locked memory */
    for (size_t n : {size_t(1), slot / 16, slot / 16 + 1, slot / 2 - 1, slot / 2, slot, slot + 1,
                     4 * slot, 4 * slot + 7, 9 * slot - 3})
        for (int locked = 0; locked < 2; locked++) {
            Bytes src = pattern(n, seed++), dev(n), dst(n);
            const Bytes want = src;
            const int before = fake_direct_copies;
            fake_locked_lo = locked ? src.data() : nullptr;
            fake_locked_hi = locked ? src.data() + n : nullptr;
            check(hs.upload(dev.data(), src.data(), n, &sa) == cudaSuccess, "upload", n);
            if (!locked || n <= slot / 16) memset(src.data(), 0, n);   /* may be reused */
            fake_locked_lo = locked ? dst.data() : nullptr;
            fake_locked_hi = locked ? dst.data() + n : nullptr;
            check(hs.download(dst.data(), dev.data(), n, &sa) == cudaSuccess, "download", n);
            if (locked) cudaStreamSynchronize(&sa);
            check(dst == want, "round trip", n);
            check(fake_direct_copies - before == (locked && n > slot / 16 ? 2 : 0),
                  "page-locked memory goes to the DMA engine as it is", n);
        }
    fake_locked_lo = fake_locked_hi = nullptr;
    /* a download that fails after n copies leaves slots with copies under way on its
     * stream; whatever they do next, the following call on another stream is right */
    for (int n = 1; n <= 8; n++) {
        Bytes old = pattern(6 * slot, seed++), now = pattern(3 * slot + 5, seed++),
              dst(6 * slot), dst2(3 * slot + 5);
        fake_fail_copy_in = n;
        const bool failed = hs.download(dst.data(), old.data(), old.size(), &sa) != cudaSuccess;
        fake_fail_copy_in = -1;
        check(failed == (n < 6), "failure is reported", n);
        fake_after_sync = [] { sa.run(sa.put); };
        check(hs.download(dst2.data(), now.data(), now.size(), &sb) == cudaSuccess, "next", n);
        fake_after_sync = nullptr;
        check(dst2 == now, "download after an abandoned one", n);
    }
    hs.release();
    return bad;
}
