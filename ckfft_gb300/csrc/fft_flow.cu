// fft_flow.cu -- both passes of a batch of complex 2^17 .. 2^20 transforms in
// one launch, the intermediate kept in L2.
//
// A multi-pass transform (fft_passes.cuh) sends every value through HBM once
// per pass.  Here the two passes run as one stream of work items: item order is
//     A(0) .. A(D-1), then A(s) and B(s - D) for s = D .. P-1, then the last B
// where A(f) are the column tiles of transform f and B(f) its row tiles.  B(f)
// runs about a thousand items after A(f), so the intermediates of the
// transforms in between (20-50 MB) stay in the 129 MB L2 until B(f) has read
// them (DRAM reads equal the input's bytes; at twice the distance 70 % more),
// and HBM moves each value once in and once out.
//
// One persistent CTA per SM:
//  * a scheduler thread claims items in order from a global ticket and queues
//    them;
//  * two loader threads, one per pass, wait for the item's buffer and (B) for
//    its transform's counter and start the item's loads into one of NB shared
//    buffers: a TMA tile for columns, one bulk copy for rows;
//  * G compute groups: group g takes buffers g, g + G, ..: values from the
//    landing buffer to registers, stages and exchanges in the same buffer
//    (fft_pair.cuh: two columns or rows a thread, packed arithmetic), buffer
//    handed back after the last exchange read, results stored from registers;
//  * a counter warp counts finished column tiles, so that no group waits for
//    its stores to reach L2.
//
// What bounds it: the SM - L2 fabric.  Both passes together move every value
// four times through it; an L2-resident copy reaches 8.2-9.3 TB/s, and this
// kernel with all butterflies and exchanges taken out ran 2^17 at 8.4, 2^20
// at 7.2 TB/s.  Measured on GB300 (GB/s of algorithmic bytes, two launches
// through HBM -> here): 2^17 x 255 2910 -> 3570, 2^18 x 128 2580 -> 3130, 2^19 x
// 64 2350 -> 3060, 2^20 x 32 2360 -> 2970; forward and inverse alternating on
// three streams, us a pair: 2^17 x 255 337 -> 293, 2^20 x 32 427 -> 362.
// Not used, measured: 2^15 / 2^16 (the cluster kernel of fft_l2pass.cu is bound
// the same way and as fast), the real forward and the first two of three
// passes (5-12 % faster alone, 6-20 % slower with other streams' kernels, whose
// small CTAs keep the whole SM a CTA needs here from falling free), the real
// inverse (its mirrored columns start at odd bins, which TMA cannot load).
//
// Progress: an item waits only for items with lower tickets; a CTA's items of
// one pass are loaded in ticket order and groups never wait for other CTAs,
// so the lowest unfinished item can always run, whatever else holds the GPU.
// Waits are bounded and report through the error word.
#include <cuda.h>

#include <atomic>
#include <cstdint>

#include "fft_pair_passes.cuh"
#include "kernels.h"
#include "tma.cuh"

namespace ckg {

constexpr int kFlowComputeThreads = 512;
constexpr int kFlowThreads = kFlowComputeThreads + 32 * 4;   // scheduler, counter, two loaders

// Columns of 2^LA, rows of 2^LB: groups of 256 threads and 64 KiB tiles (32
// columns or rows of 2^8, 16 of 2^9, 8 of 2^10).  Groups of 128 and 32 KiB tiles measured the same
// at 2^17 and 2^18 and 5-10 % slower above.
template <int LA, int LB>
struct FlowCfg {
    static constexpr int GT = 256;
    static constexpr int G = kFlowComputeThreads / GT;
    using PA = PairCfg<LA, GT>;
    using PB = PairCfg<LB, GT>;
    static_assert(PA::THREADS == GT && PB::THREADS == GT, "one tile a group");
    static constexpr int mx(int a, int b) { return a > b ? a : b; }
    static constexpr int BUF = mx(mx(PA::COL_SLOTS, PB::COL_SLOTS), PB::ROW_SLOTS);   // 16-byte slots
    static constexpr int TW = mx(PA::TW_SLOTS, PB::TW_SLOTS);                          // per group, twice
    // twiddles (8 bytes each): the stages' and W_N
    static constexpr int kStageA = StageTable<LA, false>::kEntries;
    static constexpr int kStageB = LA == LB ? 0 : StageTable<LB, false>::kEntries;
    static constexpr int kBig = BigTable<LA + LB, false>::kEntries;
    static constexpr int kTab = (kStageA + kStageB + kBig) * 8;
    static constexpr int kCtl = 768;
    static constexpr int kRest = kCtl + kTab + 2 * G * TW * 16;
    static constexpr int NB = (227 * 1024 - kRest) / (BUF * 16) < 8 ? (227 * 1024 - kRest) / (BUF * 16) : 8;
    static constexpr size_t SMEM = (size_t)kRest + 16 * (size_t)(NB * BUF);
    static_assert(NB > G, "at least one buffer loads while the groups compute");
    // Items claimed at once, and the distance of B(f) behind A(f) in items per
    // SM: far enough that B(f) finds A(f) finished, near enough that the
    // intermediates stay in L2 (13 costs 0-3 %, 20 5 %).
    static constexpr int kChunk = 1;
    static constexpr int kLag = 8;
};

struct FlowArgs {
    float2* out;
    float2* scratch;           // the intermediates (128-byte aligned)
    long long out_dist;
    const float2* tw;
    int count;                 // transforms
    int lag;                   // D
    int* ctl;                  // [0] ticket, [1 + f] finished column tiles of transform f
    unsigned* err;
    int tries;                 // bound of every wait (kWaitTries)
};

// Zeroes the ticket and the counters.
__global__ void k_flow_reset(int* ctl, int n)
{
    pdl_start();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) ctl[i] = 0;
}

// Item i -> pass, transform and tile (TA = RATIO * TB tiles a transform; within
// a step, RATIO A items to one B item).
template <int TB, int RATIO>
__device__ __forceinline__ void flow_item(int i, int count, int lag, bool* b, int* f, int* tile)
{
    constexpr int TA = TB * RATIO;
    const int head = lag * TA, mid = (count - lag) * (TA + TB);
    if (i < head) {
        *b = false;
        *f = i / TA;
        *tile = i % TA;
    } else if (i < head + mid) {
        const int j = i - head, s = j / (TA + TB), r = j % (TA + TB), q = r / (RATIO + 1), m = r % (RATIO + 1);
        *b = m == RATIO;
        *f = *b ? s : s + lag;
        *tile = *b ? q : q * RATIO + m;
    } else {
        const int j = i - head - mid;
        *b = true;
        *f = count - lag + j / TB;
        *tile = j % TB;
    }
}

__device__ __forceinline__ int ld_acquire(const int* p)
{
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void red_release(int* p)
{
    asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(p) : "memory");
}
__device__ __forceinline__ int ld_acquire_cta(const int* p)
{
    int v;
    asm volatile("ld.acquire.cta.shared.s32 %0, [%1];" : "=r"(v) : "r"(smem_addr(p)) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_cta(int* p, int v)
{
    asm volatile("st.release.cta.shared.s32 [%0], %1;" ::"r"(smem_addr(p)), "r"(v) : "memory");
}
// The tile of C columns from column c0 by ROWS rows of plane z of a tensor
// map (two floats a value), in boxes of at most 256 rows.  Read once: first to
// leave L2, so that it does not push the intermediates out (2^17 x 255 160 ->
// 151 us).
template <int C, int ROWS>
__device__ __forceinline__ void tile_load(uint32_t dst, const CUtensorMap* map, int c0, int z, uint32_t bar)
{
    unsigned long long once;
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(once));
    constexpr int BOX = ROWS < 256 ? ROWS : 256;
#pragma unroll
    for (int r = 0; r < ROWS; r += BOX)
        asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint "
                     "[%0], [%1, {%2, %3, %4}], [%5], %6;"
                     ::"r"(dst + (uint32_t)(r * C * 8)), "l"(map), "r"(2 * c0), "r"(r), "r"(z), "r"(bar), "l"(once)
                     : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// A bounded wait of one thread for a condition, briefly spinning, then asleep
// between tries; false (error word set) when it runs out.
template <class F>
__device__ __forceinline__ bool flow_wait(F&& ready, const FlowArgs& a)
{
#pragma unroll 1
    for (int tries = 0; !ready(); ++tries) {
        if (tries == a.tries) {
            if (a.err) *(volatile unsigned*)a.err = kErrWaitTimeout;
            return false;
        }
        __nanosleep(tries > 1000 ? 500 : 20);
    }
    return true;
}

template <int LA, int LB, bool INV>
__global__ void __launch_bounds__(kFlowThreads, 1) k_flow(const FlowArgs a, const __grid_constant__ CUtensorMap map)
{
    using C = FlowCfg<LA, LB>;
    using PA = typename C::PA;
    using PB = typename C::PB;
    constexpr int NB = C::NB, G = C::G, GT = C::GT;
    constexpr int N1 = 1 << LA, N2 = 1 << LB;
    constexpr int TA = N2 / PA::C, TB = N1 / PB::C;                    // tiles of a transform
    constexpr int RATIO = TA >= TB ? TA / TB : 1;
    static_assert(TA == RATIO * TB, "A items per B item");

    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(smem_raw);      // full[NB], empty[NB], done[G]
    struct Meta { int item, seq; };
    volatile Meta* meta = reinterpret_cast<volatile Meta*>(smem_raw + 256);           // [NB] what a buffer holds
    int* q_head = reinterpret_cast<int*>(smem_raw + 400);                              // items queued
    int* q_tail = reinterpret_cast<int*>(smem_raw + 404);                              // [2] items a loader is through with
    volatile int* sig_f = reinterpret_cast<volatile int*>(smem_raw + 448);            // [G] transform of a finished item
    volatile int* sig_done = reinterpret_cast<volatile int*>(smem_raw + 480);         // [G] finished items counted
    volatile int* queue = reinterpret_cast<volatile int*>(smem_raw + 512);            // [NB]
    float2* tab = reinterpret_cast<float2*>(smem_raw + C::kCtl);
    cpair* tws = reinterpret_cast<cpair*>(smem_raw + C::kCtl + C::kTab);
    cpair* bufs = tws + 2 * G * C::TW;
    auto full = [&](int b) { return smem_addr(&bars[b]); };
    auto empty = [&](int b) { return smem_addr(&bars[NB + b]); };
    auto done = [&](int g) { return smem_addr(&bars[2 * NB + g]); };

    if (threadIdx.x == 0) {
        for (int b = 0; b < NB; ++b) {
            mbar_init(full(b), 1);
            mbar_init(empty(b), GT);
            meta[b].seq = -1;
        }
        for (int g = 0; g < G; ++g) {
            mbar_init(done(g), GT);
            sig_done[g] = 0;
        }
        *q_head = 0;
        q_tail[0] = q_tail[1] = 0;
        fence_mbar_init();
    }
    // The twiddle table never changes: copied before the wait for the kernels
    // ahead in the stream.  The next kernel is not let in early: its CTAs,
    // waiting on the SMs that fall free, cost the end of this one more than
    // their early start gains (alternating with the real inverse's passes 263
    // against 226 us a pair).
    const StageTable<LA, INV> tabA{tab};
    const StageTable<LB, INV> tabB{LA == LB ? tab : tab + C::kStageA};
    const BigTable<LA + LB, INV> bigA{tab + C::kStageA + C::kStageB};
    StageTable<LA, INV>::fill(tab, a.tw, threadIdx.x, kFlowThreads);
    if constexpr (LA != LB) StageTable<LB, INV>::fill(tab + C::kStageA, a.tw, threadIdx.x, kFlowThreads);
    BigTable<LA + LB, INV>::fill(tab + C::kStageA + C::kStageB, a.tw, threadIdx.x, kFlowThreads);
    pdl_wait();
    __syncthreads();

    const int warp = threadIdx.x / 32;
    constexpr long long n = (long long)N1 * N2;
    const int total = a.count * (TA + TB);

    constexpr int W0 = kFlowComputeThreads / 32;
    if (warp == W0) {
        // ---------------------------------------------------- scheduler
        // Claims tickets in chunks (the next chunk's atomic in flight behind
        // this one) and queues the items for the loaders in ticket order, up
        // to NB ahead, then one end mark for every group.
        if (threadIdx.x % 32 != 0) return;
        int next = atomicAdd(a.ctl, C::kChunk), head = 0;
        auto put = [&](int item) {
            if (!flow_wait([&] { return min(ld_acquire_cta(&q_tail[0]), ld_acquire_cta(&q_tail[1])) > head - NB; }, a))
                return false;
            queue[head % NB] = item;
            st_release_cta(q_head, ++head);
            return true;
        };
#pragma unroll 1
        for (bool more = true; more;) {
            const int base = next;
            next = atomicAdd(a.ctl, C::kChunk);
#pragma unroll 1
            for (int i = 0; i < C::kChunk && more; ++i) {
                if (base + i >= total) more = false;
                else if (!put(base + i)) return;
            }
        }
#pragma unroll 1
        for (int g = 0; g < G; ++g)
            if (!put(-1)) return;
        return;
    }
    if (warp == W0 + 1) {
        // ------------------------------------------------------- counters
        // Lane g counts group g's finished column tiles.  The release
        // that makes a tile's stores visible before its count waits for them
        // to reach L2; here that costs the groups nothing.
        // All lanes stay to the end and leave together: when every group is
        // through, or after a.tries rounds in which no lane counted anything.
        const int lane = threadIdx.x % 32;
        int k = 0, quiet = 0;
        bool fin = lane >= G;
#pragma unroll 1
        while (!__all_sync(0xffffffffu, fin)) {
            bool counted = false;
            if (!fin && mbar_try_wait(done(lane), (uint32_t)k & 1u)) {
                const int p = sig_f[lane];
                if (p < 0) fin = true;
                else red_release(a.ctl + 1 + p);
                sig_done[lane] = ++k;
                counted = true;
            }
            if (__any_sync(0xffffffffu, counted)) {
                quiet = 0;
            } else if (++quiet > a.tries) {
                if (lane == 0 && a.err) *(volatile unsigned*)a.err = kErrWaitTimeout;
                return;
            }
        }
        return;
    }
    if (warp > W0 + 1) {
        // ------------------------------------------------------ loaders
        // Both walk the queue; the first loads column tiles, the other row
        // tiles, and passes on the end marks.
        if (threadIdx.x % 32 != 0) return;
        const bool for_second = warp != W0 + 2;
#pragma unroll 1
        for (int seq = 0, ends = 0; ends < G; ++seq) {
            const int b = seq % NB;
            if (!flow_wait([&] { return ld_acquire_cta(q_head) > seq; }, a)) return;
            const int it = queue[seq % NB];
            bool second = true;
            int f = 0, tile = 0;
            if (it >= 0) flow_item<TB, RATIO>(it, a.count, a.lag, &second, &f, &tile);
            if (second != for_second) {
                if (it < 0) {                            // the first loader stops at the first end mark
                    st_release_cta(&q_tail[0], 0x7ffffff0);
                    return;
                }
                st_release_cta(&q_tail[for_second], seq + 1);
                continue;
            }
            // rows: the transform's columns are all done (asked before the
            // wait for the buffer, which covers the latency)
            int have = second && it >= 0 ? ld_acquire(a.ctl + 1 + f) : TA;
            // the group that used the buffer before has read it for the last time
            if (seq >= NB && !mbar_wait(empty(b), (uint32_t)(seq / NB - 1) & 1u, a.err, a.tries)) return;
            if (have < TA && !flow_wait([&] { return ld_acquire(a.ctl + 1 + f) >= TA; }, a)) return;
            meta[b].item = it;
            st_release_cta(const_cast<int*>(&meta[b].seq), seq);
            // Only now, and a queue of NB: the other loader is then less than
            // NB items ahead, so it never waits for a use of a buffer whose
            // load this one has still to start.
            st_release_cta(&q_tail[for_second], seq + 1);
            if (it < 0) {
                mbar_arrive(full(b));
                ++ends;
                continue;
            }
            const uint32_t dst = smem_addr(bufs + b * C::BUF);
            if (!second) {
                // columns of the input, [n1][column]
                fence_proxy_async_shared();
                mbar_arrive_expect_tx(full(b), PA::C * (8u << LA));
                tile_load<PA::C, N1>(dst, &map, tile * PA::C, f, full(b));
            } else {
                // the groups' accesses to the landing buffer, and the other
                // CTAs' stores the counter stands for, come before these
                // copies (1200 cycles: the reason for a loader of its own)
                asm volatile("fence.proxy.async;" ::: "memory");
                mbar_arrive_expect_tx(full(b), PB::C * (8u << LB));
                bulk_load(dst, a.scratch + f * n + ((long long)(tile * PB::C) << LB), PB::C * (8u << LB), full(b));
            }
        }
        return;
    }

    // ------------------------------------------------------------ groups
    const int g = threadIdx.x / GT, tid = threadIdx.x % GT;
    int k = 0;                                          // items given to the counter warp so far
    // first barrier of an item: false when a wait of any of its warps ran out
    auto sync_and = [&](bool ok) {
        int all;
        asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %3, 0;\n\tbar.red.and.pred q, %1, %2, p;\n\tselp.s32 %0, 1, 0, q;\n\t}"
                     : "=r"(all) : "r"(1 + g), "n"(GT), "r"((int)ok) : "memory");
        return all != 0;
    };
    auto sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + g), "n"(GT) : "memory"); };
    bool ok = true;                                     // none of this thread's waits has run out
    // The load of use `seq` of its buffer has been started (an earlier use may
    // still be loading for another group: the phase bit alone cannot tell), and
    // its data is here.
    auto landed = [&](int seq) {
        const int b = seq % NB;
        return flow_wait([&] { return ld_acquire_cta(const_cast<int*>(&meta[b].seq)) == seq; }, a) &&
               mbar_wait(full(b), (uint32_t)(seq / NB) & 1u, a.err, a.tries);
    };
    // After a wait has run out the group leaves as a whole, at its next
    // meeting; one thread stays until the loads in flight to the group's buffers
    // have landed (bounded again).
    auto leave = [&](int seq) {
        if (tid == 0)
            while (landed(seq) && meta[seq % NB].item >= 0) seq += G;
    };
#pragma unroll 1
    for (int seq = g;; seq += G) {
        const int b = seq % NB;
        // (the warp's answer: its threads take the same way to the barriers)
        ok = __all_sync(0xffffffffu, ok && landed(seq));
        const int it = meta[b].item;
        // a column tile's stores are made: to the counter warp (-1: no more),
        // once it is through with the tile before
        auto finish = [&](int f) {
            if (!flow_wait([&] { return sig_done[g] >= k; }, a)) {
                ok = false;
                return;
            }
            if (tid == 0) sig_f[g] = f;
            mbar_arrive(done(g));
            ++k;
        };
        if (it < 0 || !ok) {
            if (sync_and(ok)) finish(-1);
            else leave(seq);
            return;
        }
        cpair* twsm = tws + (2 * g + (k & 1)) * C::TW;
        bool second;
        int f, tile;
        flow_item<TB, RATIO>(it, a.count, a.lag, &second, &f, &tile);
        cpair* buf = bufs + b * C::BUF;
        auto freed = [&]() { mbar_arrive(empty(b)); };
        cpair v[16];
        if (!second) {
            const int cp = tid % PA::CP, t = tid / PA::CP;
            const int n2 = tile * PA::C + 2 * cp;
            const float2 went = cols_twiddle_entry<LA, PA>(LB, tid, bigA, [&](int c) { return tile * PA::C + c; });
            const cpair wt = cols_twiddle_t<LA>(LB, n2, n2 + 1, t, bigA);
            const float4* land = reinterpret_cast<const float4*>(buf) + cp;
#pragma unroll
            for (int m = 0; m < 16; ++m) v[m] = make_pair2(land[(t + m * PA::T) * PA::CP]);
            if (!sync_and(true)) return leave(seq);
            typename PA::ColView view{buf + cp};
            stockham<LA, 4, INV, false>(v, t, tabA, view, sync, [&] { cols_twiddle_put<PA>(twsm, tid, went); }, freed);
            cols_twiddle_store<PA>(v, a.scratch + f * n, LB, n2, cp, t, twsm, wt);
            finish(f);
        } else {
            constexpr int T = PB::T;
            const int rp = tid / T, t = tid % T;
            {
                const float2* r0 = reinterpret_cast<const float2*>(buf) + 2 * rp * N2 + t;
#pragma unroll
                for (int m = 0; m < 16; ++m) v[m] = make_pair2(r0[m * T], r0[N2 + m * T]);
            }
            if (!sync_and(true)) return leave(seq);
            // the bulk copy has read the rows: drop the intermediate's L2 lines
            const char* lines = (const char*)(a.scratch + f * n + ((long long)(tile * PB::C) << LB));
#pragma unroll
            for (int l = tid; l < PB::C * (N2 / 16); l += GT)
                asm volatile("discard.global.L2 [%0], 128;" ::"l"(lines + 128 * l) : "memory");
            PairView<1, true> view{buf + rp * PB::RS};
            using S = Sched<LB, 4>;
            constexpr int NST = S::nstages;
            static_for<0, NST - 1>([&](auto sc) {
                constexpr int st = decltype(sc)::value;
                stage_compute<LB, 4, S::lrs(st), S::lns(st), INV>(v, t, tabB);
                stage_write<LB, 4, S::lrs(st), S::lns(st)>(v, t, view);
                if constexpr (st + 2 < NST) {
                    if constexpr (T <= 32) __syncwarp();
                    else sync();
                    stage_read<LB, 4>(v, t, view);
                    if constexpr (T <= 32) __syncwarp();
                    else sync();
                }
            });
            sync();
            // the last stage with the rows over the lanes: C consecutive bins k1 a store
            const int rq = tid % PB::CP, tq = tid / PB::CP;
            stage_read<LB, 4>(v, tq, PairView<1, true>{buf + rq * PB::RS});
            freed();
            constexpr int LRS = S::lrs(NST - 1), LNS = S::lns(NST - 1), U = 16 >> LRS, NS = 1 << LNS;
            stage_compute<LB, 4, LRS, LNS, INV>(v, tq, tabB);
            float2* y = a.out + f * a.out_dist;
            float2* dst = y + tile * PB::C + 2 * rq + ((long long)tq << LA);
            const bool al = ((uintptr_t)y & 15) == 0;
#pragma unroll
            for (int u = 0; u < U; ++u) {
#pragma unroll
                for (int j = 0; j < (1 << LRS); ++j) {
                    float2* d = dst + ((u * T + j * NS) << LA);
                    const cpair x = v[u + j * U];
                    if (al) {
                        __stcs(reinterpret_cast<float4*>(d), interleave(x));
                    } else {
                        __stcs(d, lane0(x));
                        __stcs(d + 1, lane1(x));
                    }
                }
            }
        }
    }
}

// ---------------------------------------------------------------- launch

static int sm_count()
{
    static int n[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1;
    if (!n[dev]) {
        int v = 0;
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v < 1) v = 1;
        n[dev] = v;
    }
    return n[dev];
}

// cuTensorMapEncodeTiled, taken from the driver through the runtime (the
// library links the runtime only).
using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                              const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeFn encode_fn()
{
    static const EncodeFn fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            return (EncodeFn) nullptr;
        }
        return (EncodeFn)f;
    }();
    return fn;
}

// [planes][rows][cols] complex values, rows `cols` and planes `plane` apart,
// in boxes of c columns by up to 256 rows.  TMA wants 16-byte aligned
// addresses and distances: false when the array has others, or planes that
// overlap (one input transformed many times, overlapping frames).
static bool encode_map(CUtensorMap* m, const void* base, long long cols, long long rows, long long planes, long long plane,
                       int c)
{
    if (((uintptr_t)base & 15) || (plane & 1) || plane < cols * rows || planes < 1) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)(2 * cols), (cuuint64_t)rows, (cuuint64_t)planes};
    const cuuint64_t strides[2] = {(cuuint64_t)(8 * cols), (cuuint64_t)(8 * plane)};
    const cuuint32_t box[3] = {(cuuint32_t)(2 * c), (cuuint32_t)(rows < 256 ? rows : 256), 1};
    const cuuint32_t one[3] = {1, 1, 1};
    const EncodeFn fn = encode_fn();
    return fn && fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), dims, strides, box, one,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Below this the passes as launches of their own are faster: the CTAs' start,
// the wait for the last A items and the last items' tail cost about 10 us, and
// other streams' kernels fill the gaps of small-CTA launches.  Measured, us
// (apart -> here): 2^17 x 32 24.4 -> 28.8, x 64 49.1 -> 45.7; 2^18 x 16 29.3 ->
// 30.8, x 32 57.7 -> 50.0; 2^20 x 4 32.4 -> 33.6, x 8 60.1 -> 51.6; pairs of
// forward and inverse on three streams: 2^17 x 64 86.1 -> 93.7, 2^20 x 8 108.1 ->
// 106.9, 2^18 x 64 195 -> 172.
constexpr long long kFlowMinPoints = 3ll << 22;

static std::atomic<long long> g_flow_launches{0};
extern "C" long long ckg_flow_launches() { return g_flow_launches.load(std::memory_order_relaxed); }

template <int LA, int LB>
static bool launch_flow_L(bool inverse, FlowArgs a, const void* in, long long in_dist, cudaStream_t s, cudaError_t* e)
{
    using C = FlowCfg<LA, LB>;
    CUtensorMap map;
    if (!encode_map(&map, in, 1 << LB, 1 << LA, a.count, in_dist, C::PA::C)) return false;
    const int tiles = (1 << LB) / C::PA::C + (1 << LA) / C::PB::C, sms = sm_count();
    const long long lag = ((long long)sms * C::kLag + tiles - 1) / tiles + 1;
    a.lag = (int)(lag < a.count ? lag : a.count);
    *e = launch_pdl(k_flow_reset, dim3(1), dim3(256), 0, s, a.ctl, a.count + 1);
    const dim3 grid((unsigned)sms), block(kFlowThreads);           // kFlowMinPoints: items for every SM
    if (*e == cudaSuccess)
        *e = inverse ? launch_pdl(k_flow<LA, LB, true>, grid, block, C::SMEM, s, a, map)
                     : launch_pdl(k_flow<LA, LB, false>, grid, block, C::SMEM, s, a, map);
    if (*e == cudaSuccess) {
        count_launch(2);
        g_flow_launches.fetch_add(1, std::memory_order_relaxed);
    }
    return true;
}

// Bytes of counters a launch needs behind its intermediates.
size_t flow_scratch_extra(int log2n, long long count)
{
    return log2n < 17 || log2n > 20 ? 0 : (sizeof(int) * (size_t)(count + 1) + 255) & ~(size_t)255;
}

bool launch_flow(bool inverse, int log2n, const void* in, void* out, long long count, long long in_dist,
                 long long out_dist, const float2* tw, void* scratch, size_t scratch_bytes, cudaStream_t s, cudaError_t* e)
{
    if (count < 1 || (count << log2n) < kFlowMinPoints || ((uintptr_t)scratch & 127)) return false;
    const size_t mid = (sizeof(float2) << log2n) * (size_t)count;
    if (scratch_bytes < mid + flow_scratch_extra(log2n, count)) return false;
    if (plain_loads_only() || !spans_disjoint(in, in_dist, out, out_dist, count, 1ll << log2n)) return false;
    FlowArgs a = {};
    a.out = (float2*)out;
    a.scratch = (float2*)scratch;
    a.out_dist = out_dist;
    a.tw = tw;
    a.count = (int)count;
    a.ctl = (int*)((char*)scratch + mid);
    a.err = device_error_word();
    a.tries = kWaitTries;
    switch (log2n) {
    case 17: return launch_flow_L<8, 9>(inverse, a, in, in_dist, s, e);
    case 18: return launch_flow_L<9, 9>(inverse, a, in, in_dist, s, e);
    case 19: return launch_flow_L<9, 10>(inverse, a, in, in_dist, s, e);
    case 20: return launch_flow_L<10, 10>(inverse, a, in, in_dist, s, e);
    default: return false;
    }
}

// For the self-test: one CTA starts at the first row tile of one transform none
// of whose column tiles is ever counted.  Its waits run out after `tries`
// rounds; no tile is loaded or stored.  `mem`: flow_selftest_bytes(), 128-byte
// aligned, any contents (it stands for the twiddle table too).
constexpr size_t kSelftestCtl = sizeof(float2) << 18;
size_t flow_selftest_bytes() { return kSelftestCtl + 256; }
cudaError_t launch_flow_selftest(void* mem, int tries, cudaStream_t s)
{
    using C = FlowCfg<8, 9>;
    FlowArgs a = {};
    a.out = a.scratch = (float2*)mem;
    a.tw = (const float2*)mem;
    a.count = a.lag = 1;
    a.ctl = (int*)((char*)mem + kSelftestCtl);
    a.err = device_error_word();
    a.tries = tries;
    CUtensorMap map;
    if (!encode_map(&map, mem, 1 << 9, 1 << 8, 1, 1 << 17, C::PA::C)) return cudaErrorNotSupported;
    const int ctl[2] = {(1 << 9) / C::PA::C, 0};                       // ticket: behind the column tiles
    const cudaError_t e = cudaMemcpyAsync(a.ctl, ctl, sizeof ctl, cudaMemcpyHostToDevice, s);
    return e == cudaSuccess ? launch_pdl(k_flow<8, 9, false>, dim3(1), dim3(kFlowThreads), C::SMEM, s, a, map) : e;
}

template <int LA, int LB>
static cudaError_t attr_flow()
{
    const int smem = (int)FlowCfg<LA, LB>::SMEM;
    const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(k_flow<LA, LB, false>, a, smem);
    return e == cudaSuccess ? cudaFuncSetAttribute(k_flow<LA, LB, true>, a, smem) : e;
}

cudaError_t prepare_flow()
{
    cudaError_t e = attr_flow<8, 9>();
    if (e == cudaSuccess) e = attr_flow<9, 9>();
    if (e == cudaSuccess) e = attr_flow<9, 10>();
    if (e == cudaSuccess) e = attr_flow<10, 10>();
    return e;
}

}  // namespace ckg
