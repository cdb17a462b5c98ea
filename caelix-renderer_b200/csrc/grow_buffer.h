// Device memory that is kept between calls and grown on demand.
#pragma once
#include <cstdint>

#include "../../include/caelix_b200.h"

namespace cx {

// Never shrunk; freed by release().
struct GrowBuffer
{
    void* ptr = nullptr;
    uint64_t bytes = 0;
    CaelixResult reserve(uint64_t want, const char* what);
    // reserve, growing by an extra eighth when it has to grow (buffers sized by a scene).
    CaelixResult reserve_grow(uint64_t want, const char* what) { return want <= bytes ? CAELIX_OK : reserve(want + want / 8, what); }
    // Growth that may fail: false, without a word in the log, and a buffer of `keep` bytes or more stays as it was.
    bool try_reserve(uint64_t want, uint64_t keep);
    void release();
};

// The memory of a wavefront call's path state, in one of two sizes: `merged`, for waves of several sample
// indices, or where that does not fit `single`, for one sample index a wave. A merged size that did not
// fit is not asked for again, nor a larger one, until forget(): a renderer that lives with the single size
// makes no allocation per frame.
struct WaveMemory
{
    GrowBuffer buffer;
    uint64_t refused = ~0ull;  // the smallest merged size that did not fit
    // *fits: whether the buffer holds `merged` bytes; else it holds single() (at most `merged`).
    template <typename Size>
    CaelixResult reserve(uint64_t merged, Size single, const char* what, bool* fits)
    {
        *fits = merged <= buffer.bytes;
        if (*fits) return CAELIX_OK;
        const uint64_t least = single();
        *fits = merged < refused && buffer.try_reserve(merged, least);
        if (*fits) return CAELIX_OK;
        if (merged > least && merged < refused) refused = merged;
        return buffer.reserve(least, what);
    }
    void forget() { refused = ~0ull; }
};

}  // namespace cx
