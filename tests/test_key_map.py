"""The host's key map (csrc/key_map.h) against std::unordered_map: insertions, overwrites and removals of
keys that collide, around the array's end and across its growth."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "caelix-renderer_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <random>
#include <unordered_map>
#include "key_map.h"

int main(int, char** argv)
{
    const uint64_t range = strtoull(argv[1], nullptr, 10), stride = strtoull(argv[2], nullptr, 10);
    std::mt19937_64 rng(7);
    KeyMap map;
    std::unordered_map<uint64_t, uint32_t> want;
    const int steps = 60000;
    for (int step = 0; step < steps; ++step) {
        const uint64_t key = rng() % range * stride;
        const uint32_t value = (uint32_t)rng(), what = (uint32_t)(rng() % 8);
        map.prefetch(key);
        if (what < (step < steps / 2 ? 4u : 2u)) {
            bool added = false;
            const uint32_t got = map.insert(key, value, &added);
            const auto it = want.emplace(key, value);
            if (added != it.second || got != it.first->second) return 1;
        } else if (what == 4) {
            map.set(key, value);
            want[key] = value;
        } else if (what > 4) {
            map.erase(key);
            want.erase(key);
        }
        const uint64_t probe = rng() % range * stride;
        const uint32_t* at = map.find(probe);
        const auto it = want.find(probe);
        if ((at != nullptr) != (it != want.end()) || (at && *at != it->second) || map.size() != want.size()) return 2;
    }
    size_t seen = 0;
    bool same = true;
    map.each([&](uint64_t key, uint32_t value) {
        ++seen;
        const auto it = want.find(key);
        same = same && it != want.end() && it->second == value;
    });
    return same && seen == want.size() ? 0 : 3;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    at = tmp_path_factory.mktemp("key_map")
    (at / "main.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", CSRC, str(at / "main.cpp"), "-o", str(at / "main")], check=True)
    return str(at / "main")


# 20 keys stay in the first array; 33 and 1,000 cross its growth; strides of 2^21 and 2^42 are
# neighbouring bricks along the second and third axis of a packed key.
@pytest.mark.parametrize("keys", [1, 20, 33, 1000, 200_000])
@pytest.mark.parametrize("stride", [1, 1 << 21, 1 << 42])
def test_against_unordered_map(program, keys, stride):
    assert subprocess.run([program, str(keys), str(stride)]).returncode == 0
