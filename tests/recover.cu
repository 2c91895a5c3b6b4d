// Host-side check of the C entries' error handling (csrc/capi_stage.cuh,
// P3G_TRY): an entry that fails for any reason leaves no word of a hash kernel
// that gave up for the next call. Needs no device: the entry fails because its
// context's device does not exist.
#include <cstdio>

#include "../p3-miden_b200/csrc/capi_stage.cuh"

static int entry(p3g_ctx *x) {
    P3G_TRY(x, {})
}

int main() {
    p3g_ctx x{};
    uint32_t word = 1;
    x.c.device = 1 << 20;
    x.c.hash_err = &word;
    const int status = entry(&x);
    if (status == p3g::OK || word != 0) return std::printf("status %d, word %u\n", status, word), 1;
    std::printf("ok\n");
    return 0;
}
