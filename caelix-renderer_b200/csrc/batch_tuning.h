// Which tuning a batch runs with, and whether a captured graph still serves it.
#pragma once
#include <cstring>

#include "../../include/caelix_b200.h"

inline bool same_tuning(const CaelixBatchTuning& a, const CaelixBatchTuning& b)
{
    return std::memcmp(&a, &b, sizeof(a)) == 0;
}

struct BatchTuning
{
    CaelixBatchTuning own;       // set, autotuned, or the default
    bool tuned = false;          // set or autotuned
    bool no_wave = false;        // untuned: the wavefront kernels' path state did not fit
    CaelixBatchTuning graph{};   // what the captured graph was captured with

    void set(const CaelixBatchTuning& t)
    {
        own = t;
        tuned = true;
        no_wave = false;
    }
    // The tuning a run uses: the batch's, or while none was set or autotuned the wavefront kernels over
    // 8 x 4 pixel blocks, or where their path state does not fit the persistent kernel, which keeps it in
    // registers. The wavefront kernels are the faster organisation at every size measured (one B200, persistent
    // against wavefront kernels): one view of 32 x 32 0.160 / 0.133 ms, 4 views of 64 and 128 squared
    // 0.430 / 0.357, 12 views of 256 and 512 squared with 2 spp 17.0 / 5.84, 8 views of scenes of up to
    // 200 k bricks 12.5 / 4.57 (1 spp to 2 spp, 2 to 4 bounces).
    CaelixBatchTuning run() const
    {
        CaelixBatchTuning t = own;
        if (!tuned && !no_wave) {
            t.kernel = CAELIX_BATCH_WAVEFRONT;
            t.block_width = 8;
        }
        return t;
    }
    // After a capture of run() that ran out of memory: whether another tuning is left to try.
    bool give_way()
    {
        if (tuned || no_wave) return false;
        no_wave = true;
        return true;
    }
    void captured() { graph = run(); }
    bool serves() const { return same_tuning(graph, run()); }
};
