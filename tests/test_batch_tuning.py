"""Which tuning a batch runs with and when its captured graph still serves it (csrc/batch_tuning.h), on the host."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "caelix-renderer_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "batch_tuning.h"

#define CHECK(c) if (!(c)) { printf("line %d: %s\n", __LINE__, #c); return 1; }

int main()
{
    CaelixBatchTuning given{};
    given.min_blocks = 6;
    given.block_width = 16;
    BatchTuning b{given};
    // Untuned: the wavefront kernels in 8 x 4 blocks.
    CaelixBatchTuning wave = b.run();
    CHECK(wave.kernel == CAELIX_BATCH_WAVEFRONT && wave.block_width == 8);
    b.captured();
    CHECK(b.serves());
    // Setting what the graph was captured with keeps it; another tuning does not.
    b.set(wave);
    CHECK(b.serves());
    b.set(given);
    CHECK(!b.serves());

    // Untuned without room for the path state: the persistent kernel, without asking at every capture.
    BatchTuning low{given};
    CHECK(low.give_way() && same_tuning(low.run(), given) && !low.give_way());
    low.captured();
    CHECK(low.serves());
    // The graph is the persistent one: the wavefront tuning, now set by hand, is captured anew.
    low.set(wave);
    CHECK(!low.serves() && same_tuning(low.run(), wave));
    CHECK(!low.give_way());  // a tuning that was set is run or fails
    low.captured();
    CHECK(low.serves());
    low.set(given);
    CHECK(!low.serves());
    return 0;
}
"""


def test_captured_tuning(tmp_path):
    (tmp_path / "main.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-Wextra", "-Wno-missing-field-initializers", "-I", CSRC,
                    str(tmp_path / "main.cpp"), "-o", str(tmp_path / "main")], check=True)
    out = subprocess.run([str(tmp_path / "main")], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
