// Generated by loom_b200.codegen from loom_b200/ir/fac_u32.lir.
// Kernel IR digest 65a54b87b1c17409; regenerate instead of editing.
#include "../engine/plain.cuh"
#include "../engine/regroup.cuh"
#include "../runtime_iface.h"

namespace loom_b200 { namespace k_fac_u32 {

__constant__ unsigned kInstrTab[3] = {3, 2, 4};
__constant__ unsigned kLiveTab[3] = {4, 4, 8};
__constant__ int kQueueBlock[3] = {0, 1, 2};
__constant__ unsigned kQuorumTab[3] = {7, 0, 5};
__constant__ unsigned kRankTab[3] = {0, 1, 2};

struct K
{
    static constexpr int kNumBlocks = 3;
    static constexpr int kNumQueues = 3;
    static constexpr int kRegroupMaxRegs = 64;
    static constexpr bool kSplitCallSites = true;
    static constexpr bool kAnyOrder = true; // schedule 2: lanes need no order
    static constexpr bool kSpread = false; // a large program with loops
    static constexpr bool kTableRows = false;
    struct Regs
    {
        unsigned int r1; // a: u32
        unsigned int r2; // cmp: u32
        unsigned int r3; // c: u32
    };

    struct In
    {
        unsigned int v0; // a
    };

    // Reads the input columns of thread `tid` (a NULL column is iota).
    __device__ __forceinline__ static void
    load_in(In& in, const Columns& c, const unsigned long long tid)
    {
        in.v0 = load_input<unsigned int>(c, 0, tid);
        (void)in; (void)c; (void)tid;
    }

    // Loom's set_inputs: input variables written, every other register zero.
    // Only registers live at START (those its queue carries) are written:
    // the others are written before they are read on every path.
    __device__ __forceinline__ static void
    start(Regs& R, const In& in)
    {
        R.r1 = static_cast<unsigned int>(in.v0);
        (void)in;
    }

    __device__ __forceinline__ static void
    load_inputs(Regs& R, const Columns& c, const unsigned long long tid)
    {
        In in;
        load_in(in, c, tid);
        start(R, in);
    }

    __device__ __forceinline__ static void
    store_outputs(const Regs& R, const Columns& c, const unsigned long long tid)
    {
        static_cast<unsigned int*>(c.p[1])[col_index(c, tid)] = R.r1; // a
    }

    __device__ __forceinline__ static unsigned instr(const int b) { return kInstrTab[b]; }
    __device__ __forceinline__ static unsigned live_bytes(const int q) { return kLiveTab[q]; }
    __device__ __forceinline__ static int block_of(const int q) { return kQueueBlock[q]; }
    __device__ __forceinline__ static unsigned quorum(const int b) { return kQuorumTab[b]; }
    __device__ __forceinline__ static unsigned rank(const int b) { return kRankTab[b]; }
    static constexpr int kNumLong = 0;
    // j-th long block (most instructions first)
    __device__ __forceinline__ static int long_block(const int j)
    {
        (void)j;
        return -1;
    }

    static constexpr int kMaxQueuesPerBlock = 1;
    // j-th queue holding threads that stand at block b (-1: none).
    __device__ __forceinline__ static int
    queue_list(const int b, const int j)
    {
        return j == 0 ? b : -1;
    }

    // Queue a thread standing at block pc waits in: the block's own queue,
    // or for a dispatch block the queue of the context its register selects.
    __device__ __forceinline__ static int
    queue_of(const int pc, const Regs& R)
    {
        (void)R;
        return pc;
    }

    // Runs the lane's own path from block `entry` for at most `budget`
    // loop iterations (visits of a loop header); returns the block it
    // stopped at, or kHalt.  With `stop_heavy`, a block whose quorum is
    // above zero is entered only as the first block of the burst, when
    // the warp's vote chose it.  A block that loops on itself takes up
    // to `spin` iterations (not 0) for one of the budget (a loop the
    // warp's lanes run together needs no step of its own per iteration).
    // kFlat: the launch's table is flat (Columns::table_flat).  kAllHeaders:
    // every loop header spends budget (the plain engine's step guard);
    // otherwise a minimal set of them that every cycle passes.
    template <bool kProf, bool kFlat, bool kAllHeaders>
    __device__ __forceinline__ static int
    run_burst(const int entry, Regs& R, Ctx& ctx, const unsigned budget, const bool stop_heavy = false,
              unsigned spin = 0u)
    {
        return run_steps<kProf, kFlat, kAllHeaders>(entry, R, ctx, budget, stop_heavy, spin);
    }
    // ... which takes the iterations it ran off `spin` (programs of several
    // loops; one loop's last iterations stay uncounted, as only HALT follows).
    template <bool kProf, bool kFlat, bool kAllHeaders>
    __device__ __forceinline__ static int
    run_steps(const int entry, Regs& R, Ctx& ctx, unsigned budget, const bool stop_heavy, unsigned& spin)
    {
        (void)ctx;
        (void)stop_heavy;
        (void)spin;
        unsigned left = 0u; // iterations of a self-loop left
        unsigned sure = 0u; // of them, those that surely go on
        (void)sure;
        bool fresh = true; // no block run yet in this burst
        (void)fresh;
        switch(entry)
        {
        case 0: goto L_B0;
        case 1: goto L_B1;
        case 2: goto L_B2;
        default: return kHalt;
        }
    L_B0: // START
        if(stop_heavy && !fresh) return 0;
    L_B0_again:
        fresh = false;
        if constexpr(kProf) count_block(ctx, 0, 3u);
        R.r2 = static_cast<unsigned int>(static_cast<bool>(static_cast<unsigned int>(R.r1) <= static_cast<unsigned int>(((unsigned int)0x1ull))));
        R.r1 = static_cast<unsigned int>(((R.r2) ? (((unsigned int)0x1ull)) : (R.r1)));
        if(R.r2) goto L_HALT; else goto L_B1;
    L_B1: // cinit
        fresh = false;
        if constexpr(kProf) count_block(ctx, 1, 2u);
        R.r3 = static_cast<unsigned int>(static_cast<unsigned int>(static_cast<unsigned int>(R.r1) - static_cast<unsigned int>(((unsigned int)0x1ull))));
        goto L_B2;
    L_B2: // loop
        if(stop_heavy && !fresh) return 2;
    L_B2_again:
        if(budget == 0u) return 2;
        left = spin ? spin : budget;
        while(left >= 8u)
        {
            fresh = false;
            if constexpr(kProf) count_block(ctx, 2, 4u);
            R.r1 = static_cast<unsigned int>(static_cast<unsigned int>(static_cast<unsigned int>(R.r1) * static_cast<unsigned int>(R.r3)));
            R.r3 = static_cast<unsigned int>(static_cast<unsigned int>(static_cast<unsigned int>(R.r3) - static_cast<unsigned int>(((unsigned int)0x1ull))));
            R.r2 = static_cast<unsigned int>(static_cast<bool>(static_cast<unsigned int>(R.r3) == static_cast<unsigned int>(((unsigned int)0x0ull))));
            if(!!(R.r2)) goto L_HALT;
            fresh = false;
            if constexpr(kProf) count_block(ctx, 2, 4u);
            R.r1 = static_cast<unsigned int>(static_cast<unsigned int>(static_cast<unsigned int>(R.r1) * static_cast<unsigned int>(R.r3)));
            R.r3 = static_cast<unsigned int>(static_cast<unsigned int>(static_cast<unsigned int>(R.r3) - static_cast<unsigned int>(((unsigned int)0x1ull))));
            R.r2 = static_cast<unsigned int>(static_cast<bool>(static_cast<unsigned int>(R.r3) == static_cast<unsigned int>(((unsigned int)0x0ull))));
            if(!!(R.r2)) goto L_HALT;
            fresh = false;
            if constexpr(kProf) count_block(ctx, 2, 4u);
            R.r1 = static_cast<unsigned int>(static_cast<unsigned int>(static_cast<unsigned int>(R.r1) * static_cast<unsigned int>(R.r3)));
            R.r3 = static_cast<unsigned int>(static_cast<unsigned int>(static_cast<unsigned int>(R.r3) - static_cast<unsigned int>(((unsigned int)0x1ull))));
            R.r2 = static_cast<unsigned int>(static_cast<bool>(static_cast<unsigned int>(R.r3) == static_cast<unsigned int>(((unsigned int)0x0ull))));
            if(!!(R.r2)) goto L_HALT;
            fresh = false;
            if constexpr(kProf) count_block(ctx, 2, 4u);
            R.r1 = static_cast<unsigned int>(static_cast<unsigned int>(static_cast<unsigned int>(R.r1) * static_cast<unsigned int>(R.r3)));
            R.r3 = static_cast<unsigned int>(static_cast<unsigned int>(static_cast<unsigned int>(R.r3) - static_cast<unsigned int>(((unsigned int)0x1ull))));
            R.r2 = static_cast<unsigned int>(static_cast<bool>(static_cast<unsigned int>(R.r3) == static_cast<unsigned int>(((unsigned int)0x0ull))));
            if(!!(R.r2)) goto L_HALT;
            fresh = false;
            if constexpr(kProf) count_block(ctx, 2, 4u);
            R.r1 = static_cast<unsigned int>(static_cast<unsigned int>(static_cast<unsigned int>(R.r1) * static_cast<unsigned int>(R.r3)));
            R.r3 = static_cast<unsigned int>(static_cast<unsigned int>(static_cast<unsigned int>(R.r3) - static_cast<unsigned int>(((unsigned int)0x1ull))));
            R.r2 = static_cast<unsigned int>(static_cast<bool>(static_cast<unsigned int>(R.r3) == static_cast<unsigned int>(((unsigned int)0x0ull))));
            if(!!(R.r2)) goto L_HALT;
            fresh = false;
            if constexpr(kProf) count_block(ctx, 2, 4u);
            R.r1 = static_cast<unsigned int>(static_cast<unsigned int>(static_cast<unsigned int>(R.r1) * static_cast<unsigned int>(R.r3)));
            R.r3 = static_cast<unsigned int>(static_cast<unsigned int>(static_cast<unsigned int>(R.r3) - static_cast<unsigned int>(((unsigned int)0x1ull))));
            R.r2 = static_cast<unsigned int>(static_cast<bool>(static_cast<unsigned int>(R.r3) == static_cast<unsigned int>(((unsigned int)0x0ull))));
            if(!!(R.r2)) goto L_HALT;
            fresh = false;
            if constexpr(kProf) count_block(ctx, 2, 4u);
            R.r1 = static_cast<unsigned int>(static_cast<unsigned int>(static_cast<unsigned int>(R.r1) * static_cast<unsigned int>(R.r3)));
            R.r3 = static_cast<unsigned int>(static_cast<unsigned int>(static_cast<unsigned int>(R.r3) - static_cast<unsigned int>(((unsigned int)0x1ull))));
            R.r2 = static_cast<unsigned int>(static_cast<bool>(static_cast<unsigned int>(R.r3) == static_cast<unsigned int>(((unsigned int)0x0ull))));
            if(!!(R.r2)) goto L_HALT;
            fresh = false;
            if constexpr(kProf) count_block(ctx, 2, 4u);
            R.r1 = static_cast<unsigned int>(static_cast<unsigned int>(static_cast<unsigned int>(R.r1) * static_cast<unsigned int>(R.r3)));
            R.r3 = static_cast<unsigned int>(static_cast<unsigned int>(static_cast<unsigned int>(R.r3) - static_cast<unsigned int>(((unsigned int)0x1ull))));
            R.r2 = static_cast<unsigned int>(static_cast<bool>(static_cast<unsigned int>(R.r3) == static_cast<unsigned int>(((unsigned int)0x0ull))));
            if(!!(R.r2)) goto L_HALT;
            left -= 8u;
        }
        while(left)
        {
            fresh = false;
            if constexpr(kProf) count_block(ctx, 2, 4u);
            R.r1 = static_cast<unsigned int>(static_cast<unsigned int>(static_cast<unsigned int>(R.r1) * static_cast<unsigned int>(R.r3)));
            R.r3 = static_cast<unsigned int>(static_cast<unsigned int>(static_cast<unsigned int>(R.r3) - static_cast<unsigned int>(((unsigned int)0x1ull))));
            R.r2 = static_cast<unsigned int>(static_cast<bool>(static_cast<unsigned int>(R.r3) == static_cast<unsigned int>(((unsigned int)0x0ull))));
            --left;
            if(!!(R.r2)) goto L_HALT;
        }
        if(spin) { spin = 0u; --budget; } else budget = 0u;
        goto L_B2_again;
    L_HALT:
        return kHalt;
    }

    static constexpr unsigned long long kRowBytes = 32ull;
    __device__ __forceinline__ static void
    save(const int q, const Regs& R, char* st, const unsigned cap, const unsigned par,
         const unsigned idx, const unsigned tid)
    {
        char* base = st + static_cast<unsigned long long>(par) * kRowBytes * cap;
        switch(q)
        {
        case 0: // START
        {
            {
                uint2 v0;
                v0.x = bitcast<unsigned>(R.r1);
                v0.y = tid;
                reinterpret_cast<uint2*>(base + 0ull * cap)[idx] = v0;
            }
            return;
        }
        case 1: // cinit
        {
            {
                uint2 v0;
                v0.x = bitcast<unsigned>(R.r1);
                v0.y = tid;
                reinterpret_cast<uint2*>(base + 8ull * cap)[idx] = v0;
            }
            return;
        }
        case 2: // loop
        {
            {
                uint4 v0;
                v0.x = bitcast<unsigned>(R.r1);
                v0.y = bitcast<unsigned>(R.r3);
                v0.z = tid;
                reinterpret_cast<uint4*>(base + 16ull * cap)[idx] = v0;
            }
            return;
        }
        default: return;
        }
    }

    __device__ __forceinline__ static unsigned
    restore(const int q, Regs& R, const char* st, const unsigned cap, const unsigned par,
            const unsigned idx)
    {
        const char* base = st + static_cast<unsigned long long>(par) * kRowBytes * cap;
        switch(q)
        {
        case 0: // START
        {
            const uint2 v0 = reinterpret_cast<const uint2*>(base + 0ull * cap)[idx];
            R.r1 = bitcast<unsigned int>(v0.x);
            return v0.y;
        }
        case 1: // cinit
        {
            const uint2 v0 = reinterpret_cast<const uint2*>(base + 8ull * cap)[idx];
            R.r1 = bitcast<unsigned int>(v0.x);
            return v0.y;
        }
        case 2: // loop
        {
            const uint4 v0 = reinterpret_cast<const uint4*>(base + 16ull * cap)[idx];
            R.r1 = bitcast<unsigned int>(v0.x);
            R.r3 = bitcast<unsigned int>(v0.y);
            return v0.z;
        }
        default: return 0xffffffffu;
        }
    }

    // bytes of one queue entry's slots, the largest over the queues
    static constexpr unsigned kMaxStageRow = 16u;
    // Lane 0 of a warp: copies the full tile [toff, toff + 32) of queue q
    // (state half `base`) into `stage` (32 x kMaxStageRow bytes of shared
    // memory) with one bulk copy per slot column, completing on the
    // mbarrier at `mbar`; false (nothing issued) when an address is not on
    // a 16-byte boundary.
    __device__ __forceinline__ static bool
    bulk_issue(const int q, unsigned char* stage, const char* base, const unsigned cap, const unsigned toff,
               unsigned long long* mbar)
    {
        unsigned bytes = 0;
        switch(q)
        {
        case 0: bytes = 256u; break;
        case 1: bytes = 256u; break;
        case 2: bytes = 512u; break;
        default: return false;
        }
        if((reinterpret_cast<unsigned long long>(base) | reinterpret_cast<unsigned long long>(stage)) & 15ull) return false;
        bulk_expect(mbar, bytes);
        switch(q)
        {
        case 0:
            bulk_copy(stage + 0u, base + 0ull * cap + static_cast<unsigned long long>(toff) * 8u, 256u, mbar);
            break;
        case 1:
            bulk_copy(stage + 0u, base + 8ull * cap + static_cast<unsigned long long>(toff) * 8u, 256u, mbar);
            break;
        case 2:
            bulk_copy(stage + 0u, base + 16ull * cap + static_cast<unsigned long long>(toff) * 16u, 512u, mbar);
            break;
        default: break;
        }
        return true;
    }

    // A lane's entry of a tile staged by bulk_issue; returns its thread id.
    __device__ __forceinline__ static unsigned
    restore_stage(const int q, Regs& R, const unsigned char* stage, const unsigned lane)
    {
        switch(q)
        {
        case 0:
        {
            const uint2 v0 = reinterpret_cast<const uint2*>(stage + 0u)[lane];
            R.r1 = bitcast<unsigned int>(v0.x);
            return v0.y;
        }
        case 1:
        {
            const uint2 v0 = reinterpret_cast<const uint2*>(stage + 0u)[lane];
            R.r1 = bitcast<unsigned int>(v0.x);
            return v0.y;
        }
        case 2:
        {
            const uint4 v0 = reinterpret_cast<const uint4*>(stage + 0u)[lane];
            R.r1 = bitcast<unsigned int>(v0.x);
            R.r3 = bitcast<unsigned int>(v0.y);
            return v0.z;
        }
        default: return 0xffffffffu;
        }
    }
};

const int kInTypes[] = {LOOM_B200_U32};
const int kOutTypes[] = {LOOM_B200_U32};
const char* const kInNames[] = {"a"};
const char* const kOutNames[] = {"a"};
const uint32_t kInstrs[] = {3, 2, 4};
const uint32_t kLive[] = {4, 4, 8};

const loom_b200_kernel_info kInfo = {
    "fac_u32", "65a54b87b1c17409", 1u, 1u, kInTypes, kOutTypes, kInNames, kOutNames,
    3u, 4u, 16u, 2u, kInstrs, kLive};

const uint32_t kQRegs0[] = {1u};
const int kQTypes0[] = {LOOM_B200_U32};
const char* const kQNames0[] = {"a"};
const unsigned long long kQOffs0[] = {0ull};
const unsigned kQSubs0[] = {0u};
const unsigned kQWidths0[] = {8u};
const uint32_t kQRegs1[] = {1u};
const int kQTypes1[] = {LOOM_B200_U32};
const char* const kQNames1[] = {"a"};
const unsigned long long kQOffs1[] = {8ull};
const unsigned kQSubs1[] = {0u};
const unsigned kQWidths1[] = {8u};
const uint32_t kQRegs2[] = {1u, 3u};
const int kQTypes2[] = {LOOM_B200_U32, LOOM_B200_U32};
const char* const kQNames2[] = {"a", "c"};
const unsigned long long kQOffs2[] = {16ull, 16ull};
const unsigned kQSubs2[] = {0u, 4u};
const unsigned kQWidths2[] = {16u, 16u};
const loom_b200_queue_layout kQueues[] = {
    {0u, -1, 1u, kQRegs0, kQTypes0, kQNames0},
    {1u, -1, 1u, kQRegs1, kQTypes1, kQNames1},
    {2u, -1, 2u, kQRegs2, kQTypes2, kQNames2},
};
const QueueSegment kSegments[] = {
    {kQOffs0, kQSubs0, kQWidths0, 0ull, 4u, 8u},
    {kQOffs1, kQSubs1, kQWidths1, 8ull, 4u, 8u},
    {kQOffs2, kQSubs2, kQWidths2, 16ull, 8u, 16u},
};

const void* plain_fn(bool profile, bool flat, unsigned per)
{
    if(profile) return reinterpret_cast<const void*>(&plain_kernel<K, true, false, 1>);
    (void)per;
    (void)flat;
    return reinterpret_cast<const void*>(&plain_kernel<K, false, false, 1>);
}

cudaError_t launch_plain(const PlainLaunch& a)
{
    const bool               flat = a.cols.table_flat != 0u;
    const unsigned long long cta  = a.lanes < 32u ? a.lanes : static_cast<unsigned long long>(a.block) * a.per;
    const unsigned long long grid = (a.n + cta - 1) / cta;
    if(grid == 0) return cudaSuccess;
    const void* fn     = plain_fn(a.profile, flat, a.per);
    void*       args[] = {const_cast<Columns*>(&a.cols), const_cast<unsigned long long*>(&a.first),
                          const_cast<unsigned long long*>(&a.n), const_cast<unsigned long long*>(&a.max_steps),
                          const_cast<unsigned**>(&a.status), const_cast<unsigned long long**>(&a.counters),
                          const_cast<unsigned*>(&a.lanes)};
    return cudaLaunchKernel(fn, dim3(static_cast<unsigned>(grid)), dim3(a.block), args, 0, a.stream);
}

// registers of a thread of the plain kernel, and the threads a CTA of it can have
cudaError_t plain_attrs(bool profile, bool flat, unsigned per, int* regs, int* max_threads)
{
    cudaFuncAttributes  at{};
    const cudaError_t e = cudaFuncGetAttributes(&at, plain_fn(profile, flat, per));
    *regs        = at.numRegs;
    *max_threads = at.maxThreadsPerBlock;
    return e;
}

const unsigned kRegCaps[] = {64u, 40u, 48u};

/// The megakernel at register cap `regs` (0: the default), in its form
/// for launches of `form`; profiled launches
/// and launches with the staged restore (`bulk`) use the default cap and
/// the parking form, and so do launches of a kernel with table records on
/// a table that is not flat (the staged-restore instantiation reads
/// every word by its own index).  NULL: no such cap compiled.
const void* regroup_fn(unsigned regs, bool profile, bool bulk, RegroupForm form, bool flat)
{
    if(profile) return reinterpret_cast<const void*>(&regroup_kernel<K, true, K::kRegroupMaxRegs, true>);
    if(bulk) return reinterpret_cast<const void*>(&regroup_kernel<K, false, K::kRegroupMaxRegs, true>);
    if(K::kTableRows && !flat)
    {
        bool known = regs == 0u;
        for(const unsigned c: kRegCaps) known |= c == regs;
        return known ? reinterpret_cast<const void*>(&regroup_kernel<K, false, K::kRegroupMaxRegs, true>) : nullptr;
    }
    const bool park = form != RegroupForm::kNeverPark;
    switch(regs)
    {
    case 0u:
    case 64u: return park ? reinterpret_cast<const void*>(&regroup_kernel<K, false, 64, false, true>)
                          : reinterpret_cast<const void*>(&regroup_kernel<K, false, 64, false, false>);
    case 40u: return park ? reinterpret_cast<const void*>(&regroup_kernel<K, false, 40, false, true>)
                          : reinterpret_cast<const void*>(&regroup_kernel<K, false, 40, false, false>);
    case 48u: return park ? reinterpret_cast<const void*>(&regroup_kernel<K, false, 48, false, true>)
                          : reinterpret_cast<const void*>(&regroup_kernel<K, false, 48, false, false>);
    default: return nullptr;
    }
}

cudaError_t launch_regroup(const RegroupLaunch& a)
{
    void* args[] = {const_cast<RegroupParams*>(&a.params)};
    const void* fn = regroup_fn(a.regs, a.profile, a.params.bulk_restore != 0u, a.form, a.params.cols.table_flat != 0u);
    if(!fn) return cudaErrorInvalidValue;
    if(a.dyn_smem)
    {
        const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   static_cast<int>(a.dyn_smem));
        if(e != cudaSuccess) return e;
    }
    if(a.ordinary && a.params.slice_rounds == 1u)
        return cudaLaunchKernel(fn, dim3(a.grid), dim3(a.block), args, a.dyn_smem, a.stream);
    return cudaLaunchCooperativeKernel(fn, dim3(a.grid), dim3(a.block), args, a.dyn_smem, a.stream);
}

cudaError_t regroup_occupancy(int block, bool profile, unsigned regs, unsigned dyn_smem, RegroupForm form, bool flat,
                              int* ctas)
{
    const void* fn = regroup_fn(regs, profile, dyn_smem != 0u, form, flat);
    if(!fn) return cudaErrorInvalidValue;
    if(dyn_smem)
    {
        const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   static_cast<int>(dyn_smem));
        if(e != cudaSuccess) return e;
    }
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas, fn, block, dyn_smem);
}

} } // namespace loom_b200::k_fac_u32

extern const loom_b200::KernelEntry loom_b200_entry_fac_u32;
const loom_b200::KernelEntry loom_b200_entry_fac_u32 = {
    &loom_b200::k_fac_u32::kInfo, loom_b200::k_fac_u32::K::kRowBytes, 3,
    &loom_b200::k_fac_u32::launch_plain, &loom_b200::k_fac_u32::launch_regroup,
    &loom_b200::k_fac_u32::regroup_occupancy,
    &loom_b200::k_fac_u32::plain_attrs,
    loom_b200::k_fac_u32::kQueues, loom_b200::k_fac_u32::kSegments,
    loom_b200::k_fac_u32::kRegCaps, 3u, loom_b200::k_fac_u32::K::kMaxStageRow, loom_b200::k_fac_u32::K::kSpread, 1u};
