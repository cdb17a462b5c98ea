// Device functions of the brick tables: the hash functions of the canonical hash table (the scene
// build) and the lookups in the cell table (the build and the trace kernels).
//
// The key slot layout and the fingerprint are the reference's hash module
// (lib/src/rhi/hash_table_layout.h:24-34: 16-byte slots key_lo, key_hi, payload, pad;
// shaders/common/caelix_hash_table.hlsl:102-128: splitmix64 rounds over the key words, key_lo >= 1,
// key_hi != 0). The table is built canonically (scene.cu): the home slot of a key is
// floor(key_lo * capacity / 2^32) (capacity = 2 x keys: load factor 0.5), keys are placed in the
// order (home, brick index) at the first free slot at or after the home, and no probe wraps (a
// tail follows the table). A lookup probes from the home until the key or an empty slot, at most
// max_probe + 1 slots.
#pragma once
#include <cstdint>

namespace cx {

__host__ __device__ __forceinline__ uint64_t splitmix64(uint64_t x)
{
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

__host__ __device__ __forceinline__ void hash_fingerprint(int32_t x, int32_t y, int32_t z, uint32_t& lo, uint32_t& hi)
{
    uint64_t h = splitmix64(0ull ^ (((uint64_t)(uint32_t)y << 32) | (uint32_t)x));
    h = splitmix64(h ^ (uint64_t)(uint32_t)z);
    const uint32_t l = (uint32_t)h;
    const uint32_t u = (uint32_t)(h >> 32);
    lo = l > 1u ? l : 1u;
    hi = u != 0u ? u : 1u;
}

__host__ __device__ __forceinline__ uint32_t hash_home(uint32_t key_lo, uint32_t capacity)
{
    return (uint32_t)(((uint64_t)key_lo * capacity) >> 32);
}

// The brick of linear brick index `lin` in the cell table: the records are in
// increasing linear brick index, so a brick's record is the first of its 32-cell word plus the
// bricks before it in the word. One 8-byte load and a population count in the place of a bitmap
// word, the fingerprint's four 64-bit multiplications and a dependent probe of the hash table; the
// table is a sixteenth of a dense index grid (1 MB against 16 MB for 256 x 256 x 64 cells).
// The lookup is in two steps so that a walk over empty cells does not count bits (population counts run
// at an eighth of the rate of the rest).
__device__ __forceinline__ bool cell_occupied(const uint2* __restrict__ cells, uint32_t lin, uint2& word)
{
    word = __ldg(cells + (lin >> 5));
    return (word.x >> (lin & 31u)) & 1u;
}
// The record of an occupied cell, from its word.
__device__ __forceinline__ uint32_t cell_record(const uint2 word, uint32_t lin)
{
    return word.y + (uint32_t)__popc(word.x & ((1u << (lin & 31u)) - 1u));
}

// The cell table with its grid, for lookups by brick key.
struct CellGrid
{
    const uint2* cells;
    int32_t origin[3];
    uint32_t grid[3];
};
// The record of brick (x, y, z), or 0xFFFFFFFF.
__device__ __forceinline__ uint32_t brick_record(const CellGrid& g, int32_t x, int32_t y, int32_t z)
{
    const uint32_t cx = (uint32_t)(x - g.origin[0]), cy = (uint32_t)(y - g.origin[1]), cz = (uint32_t)(z - g.origin[2]);
    if (cx >= g.grid[0] || cy >= g.grid[1] || cz >= g.grid[2]) return 0xFFFFFFFFu;
    const uint32_t lin = cx + g.grid[0] * (cy + g.grid[1] * cz);  // (the grid has at most 2^32 cells)
    uint2 word;
    return cell_occupied(g.cells, lin, word) ? cell_record(word, lin) : 0xFFFFFFFFu;
}

}  // namespace cx
