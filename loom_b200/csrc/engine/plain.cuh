// Plain drop-in engine: one CUDA thread per Loom thread, in input order.
//
// The generated K::run_burst<> lowers the kernel's basic blocks to a goto CFG
// inside one function, so divergence and reconvergence are the hardware's
// (Blackwell independent thread scheduling).  This replaces Loom's test-only
// CUDA backend (src/vm/cuda.hpp:1329-1579), which launched one kernel per
// basic block and sorted every register column by PC on each round.
#pragma once

#include "common.cuh"

namespace loom_b200
{
/// Loom threads per CUDA thread of a large launch of a program without loops:
/// their inputs are loaded together, and what a CUDA thread spends before and
/// after its work (indices, input forms, launch) is spent once.
constexpr unsigned kStraightPer = 4;

/// Launch: grid = ceil(n / (kPer * blockDim.x)); a CTA runs kPer * blockDim.x
/// consecutive Loom threads, CUDA thread t of it those at t, t + blockDim.x,
/// ... (Loom threads [first, first + n); inputs and outputs are indexed by
/// the Loom thread id).  Inputs are read once, outputs written
/// once, registers live in CUDA registers; counters[0..1] receive
/// thread/warp VM-instruction totals when kProf is set (lane efficiency =
/// counters[0] / (32 * counters[1])).  kFlat: the launch's table is flat
/// (only kernels that read table records have that instantiation).  With
/// lanes < 32 (CTAs of one warp) a warp runs that many Loom threads.
template <typename K, bool kProf, bool kFlat, unsigned kPer>
__global__ void
plain_kernel(const Columns                  cols,
             const unsigned long long       first,
             const unsigned long long       n,
             const unsigned long long       max_steps,
             unsigned* __restrict__         status,
             unsigned long long* __restrict__ counters,
             const unsigned                 lanes)
{
    __shared__ unsigned long long s_blk[2 * (kProf ? K::kNumBlocks : 1)];
    Ctx ctx{0ull, 0ull, status, &cols, kProf ? s_blk : nullptr};
    if constexpr(kProf) block_counters_clear(s_blk, K::kNumBlocks);
    // lanes < 32 (small launches of large kernels, CTAs of one warp): only the first lanes of
    // a warp hold threads
    const unsigned long long i0 =
        K::kSpread && lanes < 32u
            ? static_cast<unsigned long long>(blockIdx.x) * lanes + (threadIdx.x < lanes ? threadIdx.x : n)
            : static_cast<unsigned long long>(blockIdx.x) * blockDim.x * kPer + threadIdx.x;
    // the block budget is the step guard: a thread that has not halted
    // when it runs out is stopped and flagged
    const unsigned budget = max_steps < 0xffffffffull
                                ? static_cast<unsigned>(max_steps)
                                : 0xffffffffu;
    if(kPer > 1 && i0 + (kPer - 1ull) * blockDim.x < n)
    {
        typename K::In in[kPer];
#pragma unroll
        for(unsigned j = 0; j < kPer; ++j) K::load_in(in[j], cols, first + i0 + static_cast<unsigned long long>(j) * blockDim.x);
#pragma unroll
        for(unsigned j = 0; j < kPer; ++j)
        {
            typename K::Regs R;
            K::start(R, in[j]);
            if(K::template run_burst<kProf, kFlat, true>(0, R, ctx, budget) != kHalt) ctx.flag(kStatusStepLimit);
            K::store_outputs(R, cols, first + i0 + static_cast<unsigned long long>(j) * blockDim.x);
        }
    }
    else
        for(unsigned j = 0; j < kPer; ++j)
        {
            const unsigned long long i = i0 + static_cast<unsigned long long>(j) * blockDim.x;
            if(i >= n) break;
            typename K::Regs R;
            K::load_inputs(R, cols, first + i);
            if(K::template run_burst<kProf, kFlat, true>(0, R, ctx, budget) != kHalt)
                ctx.flag(kStatusStepLimit);
            K::store_outputs(R, cols, first + i);
        }
    if constexpr(kProf)
    {
        flush_counters(counters, ctx.thread_instr, ctx.warp_instr, 0ull);
        block_counters_flush(s_blk, K::kNumBlocks, counters + 8);
    }
}

} // namespace loom_b200
