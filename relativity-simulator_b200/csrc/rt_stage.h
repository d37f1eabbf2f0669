// rt_stage.h -- the one-copy read-back of a small host dispatch: which dispatches take
// it and how their outputs lie in one device buffer.  Host code, without CUDA calls.
#pragma once

#include <cstddef>
#include <cstdint>

#include "rt_internal.h"

namespace relsim {

// Rays of a launch from which a host dispatch is traced and copied back in bands.
constexpr uint64_t kBandedMinRays = uint64_t{1} << 20;

// Outputs of a small host dispatch side by side in one device buffer, read back in one
// copy to pinned memory: a copy per field into the caller's pageable arrays waits for the
// device and stages each time.  Measured, the call less its kernel, a copy per field /
// one copy: six fields of a 64x64 tile 110 / 49 us, of 192^2 rays 213 / 172; all fields
// and pixels of 64^2 rays 310 / 92, of 192^2 (4.7 MB) 675 / 535.  From 6 MB on both take
// as long (first touches of the caller's arrays).  A dispatch of kBandedMinRays and more
// copies band by band and is never staged.
constexpr size_t kStagedBytes = size_t{4} << 20;

// Points dev's fields (those set in rays) and dpix (with pixels) into a device buffer of
// `mem` and returns the bytes to read back; 0, with nothing set, where the dispatch copies
// field by field: nothing asked for, too large, banded, or no memory for either buffer
// (that route needs no pinned memory).  Memory: char* device(size_t) and
// bool pinned(size_t), null or false without memory.
template <class Memory>
size_t stage_outputs(Memory& mem, const rt_ray_out* rays, bool pixels, size_t n, rt_ray_out& dev, rt_pixel_out*& dpix) {
    constexpr size_t kAlign = 256;
    if (n >= kBandedMinRays) return 0;
    const auto round_up = [](size_t b) { return (b + kAlign - 1) / kAlign * kAlign; };
    void* const* hp = reinterpret_cast<void* const*>(rays);
    const size_t first_field = pixels ? round_up(n * sizeof(rt_pixel_out)) : 0;
    size_t total = first_field;
    for (int f = 0; rays && f < kRayFields; ++f)
        if (hp[f]) total += round_up(n * kRayFieldBytes[f]);
    if (total == 0 || total > kStagedBytes) return 0;
    char* base = mem.device(total);
    if (!base || !mem.pinned(total)) return 0;
    if (pixels) dpix = reinterpret_cast<rt_pixel_out*>(base);
    void** dp = reinterpret_cast<void**>(&dev);
    size_t at = first_field;
    for (int f = 0; rays && f < kRayFields; ++f) {
        if (!hp[f]) continue;
        dp[f] = base + at;
        at += round_up(n * kRayFieldBytes[f]);
    }
    return total;
}

}  // namespace relsim
