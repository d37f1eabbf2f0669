// Host build of the one-copy read-back's plan (rt_stage.h) over memory that can be made
// to fail, for the CPU check.  Test-only.
#include "rt_stage.h"

namespace {
struct Fake {
    char* base;
    int fail;  // 1: no device memory, 2: no pinned memory
    size_t asked = 0;
    char* device(size_t bytes) { return fail == 1 ? nullptr : (asked = bytes, base); }
    bool pinned(size_t bytes) { return fail != 2 && bytes == asked; }
};
}  // namespace

// Fields of the mask (bit f) and pixels over n rays: the staged bytes; at[0..17] the
// fields' places in the buffer and at[18] the pixels' (-1: not set).
extern "C" long host_stage(unsigned mask, int pixels, long n, int fail, long* at) {
    static char anything, buffer;
    rt_ray_out rays{}, dev{};
    void** hp = reinterpret_cast<void**>(&rays);
    for (int f = 0; f < relsim::kRayFields; ++f)
        if (mask >> f & 1u) hp[f] = &anything;
    Fake mem{&buffer, fail};
    rt_pixel_out* dpix = nullptr;
    const size_t bytes = relsim::stage_outputs(mem, &rays, pixels != 0, static_cast<size_t>(n), dev, dpix);
    void* const* dp = reinterpret_cast<void* const*>(&dev);
    for (int f = 0; f < relsim::kRayFields; ++f) at[f] = dp[f] ? static_cast<char*>(dp[f]) - &buffer : -1;
    at[relsim::kRayFields] = dpix ? reinterpret_cast<char*>(dpix) - &buffer : -1;
    return static_cast<long>(bytes);
}
