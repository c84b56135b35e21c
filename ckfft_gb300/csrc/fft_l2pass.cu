// fft_l2pass.cu -- complex 2^15 and 2^16 in two passes whose intermediate
// never reaches HBM.
//
// The multi-pass transform of fft_large.cu (columns, then rows: the packed
// passes of fft_pair_passes.cuh) runs here inside one thread-block cluster of
// K CTAs per transform: the cluster's CTAs share the column tiles, meet at a
// cluster barrier (release / acquire at cluster scope), share the row tiles,
// and each row tile's CTA drops the intermediate's L2 lines once it has read
// them.  The intermediate of the transforms in flight (resident clusters x 8n
// bytes, 20 to 40 MB) stays in the 129 MB L2, so HBM sees the input read once
// and the output written once -- the traffic of a single pass.  What bounds it
// at large batches is the path between the SMs and L2, which each value takes
// four times: 8.2-9.3 TB/s for a plain copy inside L2, 8.4 here (complex 2^16
// x 1023, 4.2 TB/s algorithmic).  Real transforms of 2^16 / 2^17 points (these
// half lengths) split in the row tiles and merge in the column tiles.
// One value a thread (256 threads, 64 registers) before, a forward and an
// inverse in us: real 2^17 x 512 417 -> 338, x 8 24 -> 22; real 2^16 x 1000 389
// -> 313, x 158 75 -> 61; complex 2^16 x 1023 551 -> 543, x 16 38 -> 24; complex
// 2^15 x 4000 1060 -> 1032, x 16 21 -> 14.
#include <cooperative_groups.h>

#include "fft_pair_passes.cuh"
#include "jobs.h"
#include "kernels.h"

namespace cg = cooperative_groups;

namespace ckg {

__device__ __forceinline__ void cluster_barrier()
{
    // global stores before the barrier are seen by the peers' loads after it:
    // the arrive releases and the wait acquires at cluster scope (no separate
    // fence: one cost a membar stall of about 1 per issued instruction)
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// CTAs per transform (K) and threads per CTA.  Eight CTAs of 128 threads, four
// such CTAs an SM, two columns or rows a thread; four CTAs of twice the tiles
// at 2^15 from kLongBatch transforms on, where fewer CTAs at each barrier
// count for more than shorter transforms do (real 2^16, 8 / 4 CTAs on three
// streams: x 158 50 / 48, x 400 124 / 118, x 1000 310 / 293; on one stream x 158
// 61 / 70, x 400 137 / 138, x 1000 322 / 313).  Measured, a forward and an inverse
// in us, 8 x 128 / 4 x 128 / 8 x 256 / 4 x 256 threads: real 2^17 x 512 338 /
// 389 / 383 / 368, x 8 23 / 39 / 19 / 33; complex 2^16 x 1023 543 / 576 / 688 /
// 641, x 16 24 / 33 / 22 / 28; real 2^16 x 158 61 / 69 / - / 71, x 1000 321 / 312 /
// - / 372; complex 2^15 x 16 14 / 19 / - / 16, x 2000 517 / 515 / - / 652.
constexpr int kL2Threads = 128;
constexpr long long kLongBatch = 384;

// Complex tiles are 16 columns or rows wide, the real ones up to 16 pairs (a
// mirrored pair's halves are separate 8-byte accesses).
template <int LA, int LB, int KIND, int K_>
struct L2Cfg {
    static constexpr int K = K_;
    using PA = PairCfg<LA, kL2Threads, (KIND < 2 ? 8 : 16)>;
    using PB = PairCfg<LB, kL2Threads, (KIND < 2 ? 8 : 16)>;
    static constexpr int SGA = kL2Threads / PA::THREADS;     // column tiles at once
    static constexpr int TILES_A = (1 << LB) / PA::C;        // column tiles of one transform
    static constexpr int TILES_B = (1 << LA) / PB::C;        // row tiles
    static constexpr int ITER_A = TILES_A / (K * SGA);
    static constexpr int ITER_B = TILES_B / K;
    static constexpr size_t SMEM_A = PA::SMEM * SGA;
    static constexpr size_t SMEM = SMEM_A > PB::SMEM ? SMEM_A : PB::SMEM;
    static_assert(PA::THREADS * SGA == kL2Threads && PB::THREADS == kL2Threads, "whole CTAs per phase");
    static_assert(ITER_A >= 1 && ITER_A * K * SGA == TILES_A, "column tiles split evenly");
    static_assert(ITER_B >= 1 && ITER_B * K == TILES_B, "row tiles split evenly");
};

// One transform per cluster: blockIdx.x / K.  scratch holds 2^(LA+LB) values
// per transform of the launch (128-byte aligned rows).
// KIND 0 / 1: complex forward / inverse of n = 2^(LA+LB) points.
// KIND 2: real forward of 2n reals (read as n packed complex values) to
// n + 1 bins, the split fused into the row tiles (pair_rows_split).
// KIND 3: real inverse of n + 1 bins to 2n reals, the merge fused into the
// column tiles (pair_cols_merge).
// fr != nullptr: transform f reads fr[f].in and writes fr[f].out (a grouped
// launch of a job run) instead of in + f in_dist, out + f out_dist.
template <int LA, int LB, int KIND, int K>
__global__ void __cluster_dims__(K, 1, 1) __launch_bounds__(kL2Threads, 4)
k_l2(const float2* __restrict__ in, float2* __restrict__ out, float2* __restrict__ scratch, long long in_dist,
     long long out_dist, const float2* __restrict__ tw, const FrameDesc* __restrict__ fr)
{
    using C = L2Cfg<LA, LB, KIND, K>;
    using PA = typename C::PA;
    using PB = typename C::PB;
    constexpr bool INV = KIND == 1 || KIND == 3;
    constexpr long long n = 1ll << (LA + LB);
    const int rank = (int)cg::this_cluster().block_rank();
    const long long f = blockIdx.x / K;
    extern __shared__ __align__(128) cpair smem[];
    // (the table is read ahead of the wait: it arrives by a copy ahead of all the
    // grouped launches, and no kernel writes it)
    const float2* x = fr ? fr[f].in : in + f * in_dist;
    float2* y = fr ? fr[f].out : out + f * out_dist;
    float2* s = scratch + f * n;
    // columns: the input -> s
    const int sga = threadIdx.x / PA::THREADS, ta = threadIdx.x % PA::THREADS;
#pragma unroll 1
    for (int i = 0; i < C::ITER_A; ++i) {
        const int tile = (i * K + rank) * C::SGA + sga;
        cpair* tsm = smem + sga * PA::TILE_SLOTS;
        if constexpr (KIND == 3) pair_cols_merge<LA, PA>(x, s, LB, tile, ta, tsm, tw, [] { pdl_wait_then_launch(); });
        else pair_cols<LA, INV, KIND == 2, PA>(x, s, LB, tile, ta, tsm, tw, [] { pdl_wait_then_launch(); });
        __syncthreads();                             // the tile's shared memory is reused
    }
    // every column tile of the transform is in L2 before any row tile reads it:
    // the peers' stores are released by the arrive and acquired by the wait, so
    // that the row pass's cached loads cannot find older lines
    cluster_barrier();
    // the row pass reloads its twiddles: keeping those it shares with the
    // column pass live across the barrier spills registers
    const float2* twb = tw;
    asm volatile("" : "+l"(twb));
#pragma unroll 1
    for (int i = 0; i < C::ITER_B; ++i) {
        const int tile = i * K + rank;
        if constexpr (KIND == 2) pair_rows_split<LB, PB>(s, y, LA, tile, threadIdx.x, smem, twb, LA, [] {});
        else pair_rows<LB, INV, PB>(s, y, LA, tile, threadIdx.x, smem, twb, LB, [] {});
        __syncthreads();
    }
}

template <int LA, int LB, int KIND>
static cudaError_t launch_l2_L(const float2* in, float2* out, float2* scratch, long long count, long long in_dist,
                               long long out_dist, const float2* tw, cudaStream_t s, const FrameDesc* fr = nullptr)
{
    if constexpr (LA + LB == 15) {
        if (count >= kLongBatch)
            return launch_pdl(k_l2<LA, LB, KIND, 4>, dim3((unsigned)(count * 4)), dim3(kL2Threads),
                              L2Cfg<LA, LB, KIND, 4>::SMEM, s, in, out, scratch, in_dist, out_dist, tw, fr);
    }
    return launch_pdl(k_l2<LA, LB, KIND, 8>, dim3((unsigned)(count * 8)), dim3(kL2Threads), L2Cfg<LA, LB, KIND, 8>::SMEM,
                      s, in, out, scratch, in_dist, out_dist, tw, fr);
}

bool l2pass_supported(int log2n) { return log2n >= 15 && log2n <= 16; }

// kind: 0 / 1 complex forward / inverse, 2 / 3 real forward / inverse of
// 2^(log2n+1) reals (log2n: the complex half length); dists in complex units.
cudaError_t launch_l2pass(int kind, int log2n, const void* in, void* out, long long count, long long in_dist,
                          long long out_dist, const float2* tw, void* scratch, size_t scratch_bytes, cudaStream_t s)
{
    if (!l2pass_supported(log2n) || kind < 0 || kind > 3) return cudaErrorInvalidValue;
    if (count <= 0) return cudaSuccess;
    const long long n = 1ll << log2n;
    const long long group = (long long)(scratch_bytes / (sizeof(float2) * (size_t)n));
    if (group < 1 || ((uintptr_t)scratch & 127)) return cudaErrorInvalidValue;
    const float2* src = (const float2*)in;
    float2* dst = (float2*)out;
    float2* tmp = (float2*)scratch;
    for (long long off = 0; off < count; off += group) {
        const long long cnt = count - off < group ? count - off : group;
        const float2* a = src + off * in_dist;
        float2* b = dst + off * out_dist;
        cudaError_t e;
#define CKG_L2_KIND(LA, LB)                                                                        \
    switch (kind) {                                                                                \
    case 0: e = launch_l2_L<LA, LB, 0>(a, b, tmp, cnt, in_dist, out_dist, tw, s); break;           \
    case 1: e = launch_l2_L<LA, LB, 1>(a, b, tmp, cnt, in_dist, out_dist, tw, s); break;           \
    case 2: e = launch_l2_L<LA, LB, 2>(a, b, tmp, cnt, in_dist, out_dist, tw, s); break;           \
    default: e = launch_l2_L<LA, LB, 3>(a, b, tmp, cnt, in_dist, out_dist, tw, s); break;          \
    }
        if (log2n == 15) { CKG_L2_KIND(7, 8) }
        else { CKG_L2_KIND(8, 8) }
#undef CKG_L2_KIND
        if (e != cudaSuccess) return e;
        count_launch();
    }
    return cudaSuccess;
}

// The same over a table of transforms (a grouped launch of a job run).
cudaError_t launch_l2pass_table(int kind, int log2n, const FrameDesc* fr, long long count, const float2* tw,
                                void* scratch, size_t scratch_bytes, cudaStream_t s)
{
    if (!l2pass_supported(log2n) || kind < 0 || kind > 3) return cudaErrorInvalidValue;
    if (count <= 0) return cudaSuccess;
    const long long n = 1ll << log2n;
    const long long group = (long long)(scratch_bytes / (sizeof(float2) * (size_t)n));
    if (group < 1 || ((uintptr_t)scratch & 127)) return cudaErrorInvalidValue;
    float2* tmp = (float2*)scratch;
    for (long long off = 0; off < count; off += group) {
        const long long cnt = count - off < group ? count - off : group;
        const FrameDesc* g = fr + off;
        cudaError_t e;
#define CKG_L2_KIND(LA, LB)                                                                              \
    switch (kind) {                                                                                      \
    case 0: e = launch_l2_L<LA, LB, 0>(nullptr, nullptr, tmp, cnt, 0, 0, tw, s, g); break;               \
    case 1: e = launch_l2_L<LA, LB, 1>(nullptr, nullptr, tmp, cnt, 0, 0, tw, s, g); break;               \
    case 2: e = launch_l2_L<LA, LB, 2>(nullptr, nullptr, tmp, cnt, 0, 0, tw, s, g); break;               \
    default: e = launch_l2_L<LA, LB, 3>(nullptr, nullptr, tmp, cnt, 0, 0, tw, s, g); break;              \
    }
        if (log2n == 15) { CKG_L2_KIND(7, 8) }
        else { CKG_L2_KIND(8, 8) }
#undef CKG_L2_KIND
        if (e != cudaSuccess) return e;
        count_launch();
    }
    return cudaSuccess;
}

template <int LA, int LB, int K>
static cudaError_t attr_l2()
{
    const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(k_l2<LA, LB, 0, K>, a, (int)L2Cfg<LA, LB, 0, K>::SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_l2<LA, LB, 1, K>, a, (int)L2Cfg<LA, LB, 1, K>::SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_l2<LA, LB, 2, K>, a, (int)L2Cfg<LA, LB, 2, K>::SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_l2<LA, LB, 3, K>, a, (int)L2Cfg<LA, LB, 3, K>::SMEM);
    return e;
}

cudaError_t prepare_l2pass()
{
    cudaError_t e = attr_l2<7, 8, 4>();
    if (e == cudaSuccess) e = attr_l2<7, 8, 8>();
    if (e == cudaSuccess) e = attr_l2<8, 8, 8>();
    return e;
}

}  // namespace ckg
