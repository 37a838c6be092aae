// pfk_classes.cu -- launchers of quartet classes PFK_CLASS_BEGIN ..
// PFK_CLASS_END - 1 (the build compiles this file once per class range so the
// 55 class instantiations build in parallel).
#include "pfk_internal.h"
#include "pfk_kernels.cuh"
#include "pfk_os.cuh"

#if !defined(PFK_CLASS_BEGIN) || !defined(PFK_CLASS_END)
#error "PFK_CLASS_BEGIN and PFK_CLASS_END must be defined (0 <= begin < end <= 55)"
#endif

namespace pfk {
namespace {

// The split kernels' SPLIT build exists for the s..d classes, whose basis sets
// have contracted shells in molecules small enough to need it.
template <int LA>
constexpr bool kSplitTeams = LA <= 2;

// One-lane quartets that go along in the SPLIT launch, at most (in lanes).
// Build times in us with 0, 2^13, 2^15, 2^17, 2^19: water / 6-31G** 165, 88, 88, 88,
// 88; (H2O)5 407, 406, 367, 371, 379; ethane / cc-pVDZ 277, 176, 176, 176, 176;
// C8H18 / 6-31G* 1407, 1392, 1396, 1393, 1423.
constexpr long long kJoinLanes = 1 << 15;

// The segments of a that give a quartet several lanes in one launch of the
// SPLIT build, the runs of the others (all n quartets when a has no segments)
// in launches of the one-lane build.
// per: lanes (or teams) per block, of 128 / per threads each.
template <typename SplitLaunch, typename PlainLaunch>
void launch_segments(const uint2 *q, long long n, const JKArgs &a, int per, SplitLaunch &&split, PlainLaunch &&plain)
{
    if (a.seg.n == 0) {
        plain(q, n, (unsigned)((n + per - 1) / per));
        return;
    }
    // few one-lane quartets go along in the SPLIT launch: a launch less
    long long single = 0;
    for (int s = 0; s < a.seg.n; ++s)
        if (a.seg.glog[s] == 0) single += a.seg.count[s];
    const bool all = single < n && single * (128 / per) <= kJoinLanes;
    JKArgs b = a;
    b.seg.n = 0;
    unsigned blocks = 0;
    for (int s = 0; s < a.seg.n; ++s) {
        if (a.seg.glog[s] == 0 && !all) continue;
        const int k = b.seg.n++;
        b.seg.glog[k] = a.seg.glog[s];
        b.seg.first[k] = a.seg.first[s];
        b.seg.count[k] = a.seg.count[s];
        b.seg.block0[k] = blocks;
        blocks += (unsigned)(((a.seg.count[s] << a.seg.glog[s]) + per - 1) / per);
    }
    if (blocks) split(b, blocks);
    if (all) return;
    for (int s = 0; s < a.seg.n; ++s) {
        if (a.seg.glog[s] != 0) continue;
        const long long first = a.seg.first[s];
        long long cnt = a.seg.count[s];
        while (s + 1 < a.seg.n && a.seg.glog[s + 1] == 0) cnt += a.seg.count[++s];
        plain(q + first * a.qstride, cnt, (unsigned)((cnt + per - 1) / per));
    }
}

// The build that the tensor and block modes take (one-lane form).
struct OutBuild {
    void (*kernel)(const uint2 *, long long, JKArgs);
    int threads;
    size_t smem;
    int per;         // quartets per block
    int few_waves;   // up to so many waves this build, if it is the one for short lists
};
// the plain Obara-Saika build: left alone the compiler takes 94 registers at
// L = 1 and 190 at L = 3 to have more of the Boys polynomials in flight, at 5
// and 2 blocks per SM.  In FP32 L = 3 needs 123 registers: 4 blocks.
template <int L, typename R>
constexpr int kOSBlocks = L == 0 ? 8 : L == 1 ? 6 : L == 2 ? 5 : L == 3 ? (sizeof(R) == 4 ? 4 : 3) : 1;

template <int LA, int LB, int LC, int LD>
OutBuild out_build(int flags)
{
    using S = ClassShape<LA, LB, LC, LD>;
    using SS = SplitShape<LA, LB, LC, LD>;
    const bool fp32 = flags & kLaunchFP32, few = flags & kLaunchShort;
    constexpr int L = LA + LB + LC + LD;
    if constexpr (L <= kOSMaxL) {
        if (flags & kLaunchOS)
            return {fp32 ? &eri_os_kernel<LA, LB, LC, LD, 1, float, kOSBlocks<L, float>, false, true>
                         : &eri_os_kernel<LA, LB, LC, LD, 1, double, kOSBlocks<L, double>, false, true>,
                    128, 0, 128, 1};
    }
    if constexpr (S::N <= kRegMaxComponents) {
        if (fp32)
            return {few ? &eri_reg_kernel<LA, LB, LC, LD, 1, float, true, RegShape<LA, LB, LC, LD, float>::MINB_SHORT>
                        : &eri_reg_kernel<LA, LB, LC, LD, 1, float, true>,
                    128, 0, 128, 1};
        return {&eri_reg_kernel<LA, LB, LC, LD, 1, double, true>, 128, 0, 128, 1};
    } else if constexpr (SS::OK) {
        using SF = SplitShape<LA, LB, LC, LD, float>;
        if (fp32)
            return {few ? &eri_split_kernel<LA, LB, LC, LD, 1, float, false, true, SF::MINB_SHORT>
                        : &eri_split_kernel<LA, LB, LC, LD, 1, float, false, true>,
                    128, SF::SMEM, SF::TEAMS, SF::FEW_WAVES};
        return {few ? &eri_split_kernel<LA, LB, LC, LD, 1, double, false, true, SS::MINB_SHORT>
                    : &eri_split_kernel<LA, LB, LC, LD, 1, double, false, true>,
                128, SS::SMEM, SS::TEAMS, SS::FEW_WAVES};
    } else {
        using TS = TeamShape<LA, LB, LC, LD>;
        using TF = TeamShape<LA, LB, LC, LD, float>;
        if (fp32) return {&eri_team_kernel<LA, LB, LC, LD, 1, float>, TF::BLOCK, TF::SMEM, TF::TEAMS, 1};
        return {&eri_team_kernel<LA, LB, LC, LD, 1>, TS::BLOCK, TS::SMEM, TS::TEAMS, 1};
    }
}

template <int LA, int LB, int LC, int LD>
BlockWaves block_waves(int flags)
{
    const OutBuild few = out_build<LA, LB, LC, LD>(flags | kLaunchShort), many = out_build<LA, LB, LC, LD>(flags);
    int dev = 0, sms = 0, blocks[2] = {};
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks[0], few.kernel, few.threads, few.smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks[1], many.kernel, many.threads, many.smem) != cudaSuccess) {
        cudaGetLastError();
        return {};
    }
    const long long wave = (long long)blocks[0] * sms * few.per;
    return {wave, wave * few.few_waves, (long long)blocks[1] * sms * many.per};
}

template <int LA, int LB, int LC, int LD>
void launch_class(const uint2 *q, long long n, const JKArgs &args, int nk, int flags, cudaStream_t st)
{
    using S = ClassShape<LA, LB, LC, LD>;
    using SS = SplitShape<LA, LB, LC, LD>;
    using TS = TeamShape<LA, LB, LC, LD>;
    const int fp32 = flags & kLaunchFP32;
    const bool out = args.blk_out || args.eri_out;   // tensor and block modes: out_build, one density
    JKArgs a = args;
    if (out && fp32) a.seg.n = 0;                    // their FP32 builds have no SPLIT form
    if constexpr (LA + LB + LC + LD <= kOSMaxL) {
        if (flags & kLaunchOS) {
            if (n <= 0) return;
            const bool dense = flags & kLaunchDense;
            // the denser build: blocks per SM its register cap must allow.  Up
            // to L = 2 the kernels need at most 104 registers, so 4 blocks would
            // change nothing; there 8 (L <= 1: 64 registers) and 6 (L = 2: 80)
            // trade a few spilled values for occupancy.  The autotuner keeps
            // whichever build is faster on the molecule's lists.
            constexpr int L = LA + LB + LC + LD;
            constexpr int MB = L <= 1 ? 8 : L == 2 ? 6 : 4;
            constexpr int PB = kOSBlocks<L, double>, PF = kOSBlocks<L, float>;
            launch_segments(
                q, n, a, 128,
                [&](const JKArgs &b, unsigned grid) {
                    if (out) eri_os_kernel<LA, LB, LC, LD, 1, double, 1, true, true><<<grid, 128, 0, st>>>(q, n, b);
                    else if (nk == 2) eri_os_kernel<LA, LB, LC, LD, 2, double, 1, true><<<grid, 128, 0, st>>>(q, n, b);
                    else if (fp32) eri_os_kernel<LA, LB, LC, LD, 1, float, 1, true><<<grid, 128, 0, st>>>(q, n, b);
                    else eri_os_kernel<LA, LB, LC, LD, 1, double, 1, true><<<grid, 128, 0, st>>>(q, n, b);
                },
                [&](const uint2 *r, long long m, unsigned grid) {
                    if (out) out_build<LA, LB, LC, LD>(flags).kernel<<<grid, 128, 0, st>>>(r, m, a);
                    else if (nk == 2) eri_os_kernel<LA, LB, LC, LD, 2, double, PB><<<grid, 128, 0, st>>>(r, m, a);
                    else if (fp32 && dense) eri_os_kernel<LA, LB, LC, LD, 1, float, MB><<<grid, 128, 0, st>>>(r, m, a);
                    else if (fp32) eri_os_kernel<LA, LB, LC, LD, 1, float, PF><<<grid, 128, 0, st>>>(r, m, a);
                    else if (dense) eri_os_kernel<LA, LB, LC, LD, 1, double, MB><<<grid, 128, 0, st>>>(r, m, a);
                    else eri_os_kernel<LA, LB, LC, LD, 1, double, PB><<<grid, 128, 0, st>>>(r, m, a);
                });
            return;
        }
    }
    if constexpr (S::N <= kRegMaxComponents) {
        if (n <= 0) return;
        const long long grid = (n + 127) / 128;
        if (out) out_build<LA, LB, LC, LD>(flags).kernel<<<(unsigned)grid, 128, 0, st>>>(q, n, a);
        else if (nk == 2) eri_reg_kernel<LA, LB, LC, LD, 2><<<(unsigned)grid, 128, 0, st>>>(q, n, a);
        else if (fp32) eri_reg_kernel<LA, LB, LC, LD, 1, float><<<(unsigned)grid, 128, 0, st>>>(q, n, a);
        else eri_reg_kernel<LA, LB, LC, LD, 1><<<(unsigned)grid, 128, 0, st>>>(q, n, a);
    } else if constexpr (SS::OK) {
        using SF = SplitShape<LA, LB, LC, LD, float>;
        if (n < 0) {  // configure the current device (shared-memory opt-in)
            cudaFuncSetAttribute(eri_split_kernel<LA, LB, LC, LD, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SS::SMEM);
            cudaFuncSetAttribute(eri_split_kernel<LA, LB, LC, LD, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SS::SMEM);
            cudaFuncSetAttribute(eri_split_kernel<LA, LB, LC, LD, 1, float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)SF::SMEM);
            for (int f : {0, kLaunchShort, (int)kLaunchFP32, kLaunchFP32 | kLaunchShort}) {
                const OutBuild o = out_build<LA, LB, LC, LD>(f);
                cudaFuncSetAttribute(o.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)o.smem);
            }
            if constexpr (kSplitTeams<LA>) {
                cudaFuncSetAttribute(eri_split_kernel<LA, LB, LC, LD, 1, double, true, true>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SS::SMEM_SPLIT);
                cudaFuncSetAttribute(eri_split_kernel<LA, LB, LC, LD, 1, double, true>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SS::SMEM_SPLIT);
                cudaFuncSetAttribute(eri_split_kernel<LA, LB, LC, LD, 2, double, true>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SS::SMEM_SPLIT);
                cudaFuncSetAttribute(eri_split_kernel<LA, LB, LC, LD, 1, float, true>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SF::SMEM_SPLIT);
            }
            return;
        }
        if (n == 0) return;
        const auto plain = [&](const uint2 *r, long long m, unsigned grid) {
            if (out) {
                const OutBuild o = out_build<LA, LB, LC, LD>(flags);
                o.kernel<<<grid, 128, o.smem, st>>>(r, m, a);
            } else if (nk == 2) eri_split_kernel<LA, LB, LC, LD, 2><<<grid, 128, SS::SMEM, st>>>(r, m, a);
            else if (fp32) eri_split_kernel<LA, LB, LC, LD, 1, float><<<grid, 128, SF::SMEM, st>>>(r, m, a);
            else eri_split_kernel<LA, LB, LC, LD, 1><<<grid, 128, SS::SMEM, st>>>(r, m, a);
        };
        if constexpr (kSplitTeams<LA>)
            launch_segments(
                q, n, a, SS::TEAMS,
                [&](const JKArgs &b, unsigned grid) {
                    if (out)
                        eri_split_kernel<LA, LB, LC, LD, 1, double, true, true><<<grid, 128, SS::SMEM_SPLIT, st>>>(q, n, b);
                    else if (nk == 2) eri_split_kernel<LA, LB, LC, LD, 2, double, true><<<grid, 128, SS::SMEM_SPLIT, st>>>(q, n, b);
                    else if (fp32) eri_split_kernel<LA, LB, LC, LD, 1, float, true><<<grid, 128, SF::SMEM_SPLIT, st>>>(q, n, b);
                    else eri_split_kernel<LA, LB, LC, LD, 1, double, true><<<grid, 128, SS::SMEM_SPLIT, st>>>(q, n, b);
                },
                plain);
        else
            plain(q, n, (unsigned)((n + SS::TEAMS - 1) / SS::TEAMS));
    } else {
        using TF = TeamShape<LA, LB, LC, LD, float>;
        if (n < 0) {
            cudaFuncSetAttribute(eri_team_kernel<LA, LB, LC, LD, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TS::SMEM);
            cudaFuncSetAttribute(eri_team_kernel<LA, LB, LC, LD, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TS::SMEM);
            cudaFuncSetAttribute(eri_team_kernel<LA, LB, LC, LD, 1, float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)TF::SMEM);
            return;
        }
        if (n == 0) return;
        const long long grid = (n + TS::TEAMS - 1) / TS::TEAMS;
        if (nk == 2) eri_team_kernel<LA, LB, LC, LD, 2><<<(unsigned)grid, TS::BLOCK, TS::SMEM, st>>>(q, n, a);
        else if (fp32) eri_team_kernel<LA, LB, LC, LD, 1, float><<<(unsigned)grid, TF::BLOCK, TF::SMEM, st>>>(q, n, a);
        else eri_team_kernel<LA, LB, LC, LD, 1><<<(unsigned)grid, TS::BLOCK, TS::SMEM, st>>>(q, n, a);
    }
}

// class index -> (bra pair class, ket pair class)
constexpr int cls_bra(int c)
{
    int x = 0;
    while ((x + 1) * (x + 2) / 2 <= c) ++x;
    return x;
}
constexpr int cls_ket(int c) { return c - cls_bra(c) * (cls_bra(c) + 1) / 2; }

template <int C>
void reg_range()
{
    constexpr int X = cls_bra(C), Y = cls_ket(C);
    using SS = SplitShape<pc_la(X), pc_lb(X), pc_la(Y), pc_lb(Y)>;
    constexpr bool split = pc_la(X) + pc_lb(X) + pc_la(Y) + pc_lb(Y) > kOSMaxL && SS::S::N > kRegMaxComponents && SS::OK;
    static_assert(!split || class_team(C) == SS::TEAM, "list_segments counts in teams of the split kernel's size");
    static_assert(split || SS::S::N > kRegMaxComponents || class_team(C) == 1, "register and OS kernels: one lane");
    g_class_launchers[C] = &launch_class<pc_la(X), pc_lb(X), pc_la(Y), pc_lb(Y)>;
    g_class_waves[C] = &block_waves<pc_la(X), pc_lb(X), pc_la(Y), pc_lb(Y)>;
    if constexpr (C + 1 < PFK_CLASS_END) reg_range<C + 1>();
}

// Runs at library load: puts this unit's launchers into the shared table.
struct Registrar {
    Registrar() { reg_range<PFK_CLASS_BEGIN>(); }
};
const Registrar registrar;

}  // namespace
}  // namespace pfk
