// fft_large.cu -- multi-pass transforms above the single-CTA size limit.
//
// Replaces the reference's recursion (src/ckfft/fft_default.cpp:168-266) for
// sizes whose data cannot stay on chip.  N = N1 * N2, x[n] viewed as N1 rows
// of N2 columns (n = N2*n1 + n2):
//
//   pass 1 (columns): for each column n2, Y[k1] = DFT_N1 over n1 of x[N2*n1 + n2],
//                     times W_N^(n2*k1), stored at scratch[N2*k1 + n2];
//   pass 2 (rows):    for each row k1, DFT_N2 over n2, X[k1 + N1*k2] stored
//                     transposed through shared memory.
//
// Both passes read and write HBM once, with C adjacent columns (pass 1) or
// rows (pass 2) per CTA so every warp access covers C*8 contiguous bytes
// (large batches of complex 2^17 .. 2^20: fft_flow.cu).
// Real sizes run the half-length complex transform with the split (forward)
// fused into its last pass and the merge (inverse) into its first, the
// algebra of src/ckfft/fft_real_default.cpp.
#include <cstdint>

#include "fft_pair_passes.cuh"
#include "jobs.h"
#include "kernels.h"

namespace ckg {

// ------------------------------------------------------------ pass kernels

// Tiles of 16 columns or rows (128-byte row accesses), 8 at sub-length 2^10,
// two columns or rows a thread (fft_pair_passes.cuh), at most 256 threads and
// 128 registers a thread.
template <int LS>
using BPass = PairCfg<LS, 256, 8>;
template <int LS>
constexpr int kPassBlocks = 65536 / (BPass<LS>::THREADS * 128);

template <int LA, bool INV, bool MIRROR>
__global__ void __launch_bounds__(BPass<LA>::THREADS, kPassBlocks<LA>)
k_cols(const float2* __restrict__ in, float2* __restrict__ out, int log2n2, long long in_dist, long long out_dist,
       const float2* __restrict__ tw)
{
    using P = BPass<LA>;
    extern __shared__ __align__(128) cpair smem[];
    const int log2tiles = log2n2 - ilog2(P::C);
    const long long f = blockIdx.x >> log2tiles;
    pair_cols<LA, INV, MIRROR, P>(in + f * in_dist, out + f * out_dist, log2n2, blockIdx.x & ((1 << log2tiles) - 1), threadIdx.x,
                          smem, tw, [] { pdl_wait_then_launch(); });
}

template <int LB, bool INV>
__global__ void __launch_bounds__(BPass<LB>::THREADS, kPassBlocks<LB>)
k_rows(const float2* __restrict__ in, float2* __restrict__ out, int log2n1, long long in_dist, long long out_dist,
       const float2* __restrict__ tw)
{
    using P = BPass<LB>;
    extern __shared__ __align__(128) cpair smem[];
    const int log2tiles = log2n1 - ilog2(P::C);
    const long long f = blockIdx.x >> log2tiles;
    pair_rows<LB, INV, P>(in + f * in_dist, out + f * out_dist, log2n1, blockIdx.x & ((1 << log2tiles) - 1), threadIdx.x,
                          smem, tw, LB, [] { pdl_wait_then_launch(); });
}

// Passes 1 and 2 of the three-pass transform, one step of a chain of launches.
// A panel -- gc neighbouring n3 of one transform, every n1 and n2 -- is closed
// under both passes.  Step s runs pass 1 on panel s and pass 2 (in place) on
// panel s - 1, tile by tile alternating, so the panels between the passes
// (16-32 MB) are read back from L2: HBM sees both passes as one.  The pass-1
// tiles depend on nothing in the chain, so they do not wait for the step before
// (only step 0 waits, for the work ahead of the call); the pass-2 tiles do.  A
// step lets the next one in once its own tiles have passed their waits, so a
// step's start means that the step before the previous one is complete, and
// the next step's pass-1 tiles fill this step's tail.
// A pass-1 tile that does not wait still sees what was written ahead of the call:
// every CTA of step 0 was through its wait, which completes those kernels, before
// step 1 could start, and so on; and a kernel starts with no lines in L1, so its
// loads find nothing older than its start.
template <int L1, int L2>
struct Cols12 {
    static constexpr int THREADS = 8 * (1 << ((L1 > L2 ? L1 : L2) - 4));
    using P1 = PairCfg<L1, THREADS>;
    using P2 = PairCfg<L2, THREADS>;
    static_assert(P1::THREADS == THREADS && P2::THREADS == THREADS, "one tile a CTA");
    static constexpr size_t SMEM = P1::SMEM > P2::SMEM ? P1::SMEM : P2::SMEM;
};
template <int L1, int L2, bool INV, bool MIRROR>
__global__ void __launch_bounds__((Cols12<L1, L2>::THREADS), (65536 / (Cols12<L1, L2>::THREADS * 128)))
k_cols12(const float2* __restrict__ in, float2* __restrict__ mid, int l3, int lgc, int s, int panels, long long in_dist,
         const float2* __restrict__ tw)
{
    using P1 = typename Cols12<L1, L2>::P1;
    using P2 = typename Cols12<L1, L2>::P2;
    extern __shared__ __align__(128) cpair smem[];
    const bool both = s > 0 && s < panels;
    const int i = both ? blockIdx.x >> 1 : blockIdx.x;
    const bool second = both ? blockIdx.x & 1 : s > 0;
    const int panel = second ? s - 1 : s, lper = l3 - lgc;              // panels of one transform: 2^lper
    const long long f = panel >> lper;
    const int n3 = (panel & ((1 << lper) - 1)) << lgc;
    if (!second) {
        const int lt = lgc - ilog2(P1::C), n2 = i >> lt, c0 = n3 + ((i & ((1 << lt) - 1)) << ilog2(P1::C));
        pair_cols<L1, INV, false, P1>(in + f * in_dist, mid + (f << (L1 + L2 + l3)), L2 + l3, ((n2 << l3) + c0) >> ilog2(P1::C),
                               threadIdx.x, smem, tw, [s] {
                                   if (s == 0) pdl_wait();
                                   pdl_launch_dependents();
                               });
    } else {
        const int lt = lgc - ilog2(P2::C), k1 = i >> lt, c0 = n3 + ((i & ((1 << lt) - 1)) << ilog2(P2::C));
        float2* row = mid + (f << (L1 + L2 + l3)) + ((long long)k1 << (L2 + l3));
        pair_cols<L2, INV, MIRROR, P2>(row, row, l3, c0 >> ilog2(P2::C), threadIdx.x, smem, tw,
                                       [] { pdl_wait_then_launch(); }, k1 == 0);
    }
}

// Third pass of the three-pass transform (N = N1 N2 N3, sub-lengths 2^l1,
// 2^l2, 2^LB): block (f, k2, tile) runs DFT_N3 along the C rows k1 of the
// tile, row (k1, k2) of transform f at in[f N + k1 N2 N3 + k2 N3 ..], and
// stores X[k1 + N1 k2 + N1 N2 k3] -- C consecutive outputs per k3.
template <int LB, bool INV>
__global__ void __launch_bounds__(BPass<LB>::THREADS, kPassBlocks<LB>)
k_rows3(const float2* __restrict__ in, float2* __restrict__ out, int l1, int l2, long long out_dist,
        const float2* __restrict__ tw)
{
    using P = BPass<LB>;
    extern __shared__ __align__(128) cpair smem[];
    const int log2tiles = l1 - ilog2(P::C);
    const long long b = blockIdx.x;
    const int tile = (int)(b & ((1 << log2tiles) - 1));
    const long long k2 = (b >> log2tiles) & ((1ll << l2) - 1);
    const long long f = b >> (log2tiles + l2);
    const long long n = 1ll << (l1 + l2 + LB);
    pair_rows<LB, INV, P>(in + f * n + (k2 << LB), out + f * out_dist + (k2 << l1), l1 + l2, tile, threadIdx.x, smem, tw,
                          l2 + LB, [] { pdl_wait_then_launch(); });
}

// The split and merge passes: a pair is a row (column) and its mirror, and the
// split or merge happens inside the pair's registers.  With one value a thread
// (512 threads, 64 registers) the mirror had to be found through shared
// memory, and shared memory was the bound (77-79 % of its rate, HBM at 40 %):
// five accesses a value for the merge and six for the split, two and four now.
// 8-byte stores (loads) of up to 16 neighbours either way; 256 threads against
// 512 (real 2^20 x 32, a forward and an inverse: 232 against 255 us), 16 pairs
// against 8 (2^22 x 8: 255 against 271).  Before and after, us: 2^18 x 127 228
// -> 203, 2^20 x 32 287 -> 234, 2^22 x 8 307 -> 256, 2^24 x 2 316 -> 259, 2^22
// alone 50 -> 39.
template <int LS>
using SPass = PairCfg<LS, 256, 16>;
template <int LS>
constexpr int kSplitBlocks = 65536 / (SPass<LS>::THREADS * 128);

// Row pass of a real forward transform with the split fused: block
// (f, tile) writes the M+1 output bins of its row pairs (pair_rows_split).
template <int LB>
__global__ void __launch_bounds__(SPass<LB>::THREADS, kSplitBlocks<LB>)
k_rows_split(const float2* __restrict__ in, float2* __restrict__ out, int log2n1, int log2k1, long long in_dist,
             long long out_dist, const float2* __restrict__ tw)
{
    using P = SPass<LB>;
    extern __shared__ __align__(128) cpair smem[];
    const int log2tiles = log2n1 - ilog2(P::C);
    const long long f = blockIdx.x >> log2tiles;
    pair_rows_split<LB, P>(in + f * in_dist, out + f * out_dist, log2n1, blockIdx.x & ((1 << log2tiles) - 1), threadIdx.x,
                           smem, tw, log2k1, [] { pdl_wait_then_launch(); });
}

// Column pass of a real inverse transform with the merge fused: block
// (f, tile) reads the M+1 bins of its column pairs (pair_cols_merge).
template <int LA>
__global__ void __launch_bounds__(SPass<LA>::THREADS, kSplitBlocks<LA>)
k_cols_merge(const float2* __restrict__ in, float2* __restrict__ out, int log2n2, long long in_dist,
             long long out_dist, const float2* __restrict__ tw)
{
    using P = SPass<LA>;
    extern __shared__ __align__(128) cpair smem[];
    const int log2tiles = log2n2 - ilog2(P::C);
    const long long f = blockIdx.x >> log2tiles;
    pair_cols_merge<LA, P>(in + f * in_dist, out + f * out_dist, log2n2, blockIdx.x & ((1 << log2tiles) - 1), threadIdx.x,
                           smem, tw, [] { pdl_wait_then_launch(); });
}

// Both passes of a large batch of real transforms, one step of a chain of
// launches as in k_cols12: a panel is `per` whole transforms (16 MB of
// intermediates); step s runs the column pass on panel s, then the row pass on
// panel s - 1, so the intermediates are read back from L2 and HBM sees the input
// and the output once (the column tiles read the caller's input without a wait of
// their own on the grounds given there).  The column tiles come first: they need no wait, fill
// the tail of the step before, and by the time the row tiles' turn comes that
// step is complete (alternating tiles hold half the SMs in their waits: real
// 2^18 x 127, a forward and an inverse, 226 us on one stream against 199).  Panels
// of 32 MB measured 202 us on one stream and 192 on three, of 16 MB 199 and 175,
// two launches over everything 206 and 192.  2^20 x 32: 237 / 219 us on one / three
// streams in two launches, 220 / 197 here; 2^21 x 50 784 / 749 and 724 / 688.
template <int LA, int LB>
struct RealChain {
    static constexpr int THREADS = 256;
    using PA = PairCfg<LA, THREADS, 16>;
    using PB = PairCfg<LB, THREADS, 16>;
    static_assert(PA::THREADS == THREADS && PB::THREADS == THREADS, "one tile a CTA");
    static constexpr int LOG2TILES = LA + LB - ilog2(32 * THREADS);      // tiles of one transform and pass
    static constexpr size_t SMEM = PA::SMEM > PB::SMEM ? PA::SMEM : PB::SMEM;
};
template <int LA, int LB, bool INV>
__global__ void __launch_bounds__(256, 2)
k_real_chain(const float2* __restrict__ in, float2* __restrict__ out, float2* __restrict__ mid, int per, int s, int cols,
             long long in_dist, long long out_dist, const float2* __restrict__ tw)
{
    using C = RealChain<LA, LB>;
    extern __shared__ __align__(128) cpair smem[];
    const bool second = (int)blockIdx.x >= cols;
    const int i = second ? blockIdx.x - cols : blockIdx.x;
    const int tile = i & ((1 << C::LOG2TILES) - 1);
    const long long f = (long long)(second ? s - 1 : s) * per + (i >> C::LOG2TILES);
    float2* m = mid + (f << (LA + LB));
    if (!second) {
        auto wait = [s] {
            if (s == 0) pdl_wait();
            pdl_launch_dependents();
        };
        if constexpr (INV) pair_cols_merge<LA, typename C::PA>(in + f * in_dist, m, LB, tile, threadIdx.x, smem, tw, wait);
        else pair_cols<LA, false, true, typename C::PA>(in + f * in_dist, m, LB, tile, threadIdx.x, smem, tw, wait);
    } else {
        auto wait = [] { pdl_wait_then_launch(); };
        if constexpr (INV) pair_rows<LB, true, typename C::PB>(m, out + f * out_dist, LA, tile, threadIdx.x, smem, tw, LB, wait);
        else pair_rows_split<LB, typename C::PB>(m, out + f * out_dist, LA, tile, threadIdx.x, smem, tw, LA, wait);
    }
}

// ---------------------------------------------------------------- launch

// Bytes of a panel of the chained passes, and the values from which a batch of
// real transforms is chained.
constexpr int kPanelLog2 = 24;
constexpr long long kChainMinPoints = 1ll << 22;

template <int LA, int LB, bool INV>
static cudaError_t launch_real_chain_L(const float2* in, float2* out, float2* mid, long long count, long long in_dist,
                                       long long out_dist, const float2* tw, cudaStream_t s)
{
    using C = RealChain<LA, LB>;
    constexpr long long per = 1ll << (kPanelLog2 - 3 - LA - LB);
    const int panels = (int)((count + per - 1) / per);
    auto tiles = [&](int p) { return p < 0 || p >= panels ? 0 : (int)((count - p * per < per ? count - p * per : per) << C::LOG2TILES); };
    for (int st = 0; st <= panels; ++st) {
        const int a = tiles(st), b = tiles(st - 1);
        const cudaError_t e = launch_pdl(k_real_chain<LA, LB, INV>, dim3((unsigned)(a + b)), dim3(C::THREADS), C::SMEM, s, in,
                                         out, mid, (int)per, st, a, in_dist, out_dist, tw);
        if (e != cudaSuccess) return e;
        count_launch();
    }
    return cudaSuccess;
}

// Half lengths 2^lm; in_dist / out_dist in float2.  *done: the batch ran here:
// from 32 MB of intermediates on, two panels (2^18 x 32: 59 against 60 us; less of
// it stays in L2 between two launches anyway), and where input and output do not
// overlap (two launches read all inputs before the first output).
template <bool INV>
static cudaError_t launch_real_chain(int lm, const float2* in, float2* out, float2* mid, long long count, long long in_dist,
                                     long long out_dist, const float2* tw, cudaStream_t s, bool* done)
{
    *done = (count << lm) >= kChainMinPoints && spans_disjoint(in, in_dist, out, out_dist, count, (1ll << lm) + 1);
    if (!*done) return cudaSuccess;
    switch (lm) {
    case 17: return launch_real_chain_L<8, 9, INV>(in, out, mid, count, in_dist, out_dist, tw, s);
    case 18: return launch_real_chain_L<9, 9, INV>(in, out, mid, count, in_dist, out_dist, tw, s);
    case 19: return launch_real_chain_L<9, 10, INV>(in, out, mid, count, in_dist, out_dist, tw, s);
    case 20: return launch_real_chain_L<10, 10, INV>(in, out, mid, count, in_dist, out_dist, tw, s);
    default: *done = false; return cudaSuccess;
    }
}

template <int LA, bool INV, bool MIRROR>
static cudaError_t launch_cols_L(const float2* in, float2* out, long long count, int log2n2,
                                 long long in_dist, long long out_dist, const float2* tw, cudaStream_t s)
{
    using P = BPass<LA>;
    const long long blocks = count * ((1ll << log2n2) / P::C);
    return launch_pdl(k_cols<LA, INV, MIRROR>, dim3((unsigned)blocks), dim3(P::THREADS), P::SMEM, s, in, out, log2n2, in_dist,
                      out_dist, tw);
}

template <int LB, bool INV>
static cudaError_t launch_rows_L(const float2* in, float2* out, long long count, int log2n1,
                                 long long in_dist, long long out_dist, const float2* tw, cudaStream_t s)
{
    using P = BPass<LB>;
    const long long blocks = count * ((1ll << log2n1) / P::C);
    return launch_pdl(k_rows<LB, INV>, dim3((unsigned)blocks), dim3(P::THREADS), P::SMEM, s, in, out, log2n1, in_dist,
                      out_dist, tw);
}

// MIRROR: of a real forward transform (pair_rows_split reads the result).
template <bool INV, bool MIRROR = false>
static cudaError_t launch_cols(int la, const float2* in, float2* out, long long count, int log2n2,
                               long long in_dist, long long out_dist, const float2* tw, cudaStream_t s)
{
    switch (la) {
    case 7: return launch_cols_L<7, INV, MIRROR>(in, out, count, log2n2, in_dist, out_dist, tw, s);
    case 8: return launch_cols_L<8, INV, MIRROR>(in, out, count, log2n2, in_dist, out_dist, tw, s);
    case 9: return launch_cols_L<9, INV, MIRROR>(in, out, count, log2n2, in_dist, out_dist, tw, s);
    case 10: return launch_cols_L<10, INV, MIRROR>(in, out, count, log2n2, in_dist, out_dist, tw, s);
    default: return cudaErrorInvalidValue;
    }
}

template <bool INV>
static cudaError_t launch_rows(int lb, const float2* in, float2* out, long long count, int log2n1,
                               long long in_dist, long long out_dist, const float2* tw, cudaStream_t s)
{
    switch (lb) {
    case 7: return launch_rows_L<7, INV>(in, out, count, log2n1, in_dist, out_dist, tw, s);
    case 8: return launch_rows_L<8, INV>(in, out, count, log2n1, in_dist, out_dist, tw, s);
    case 9: return launch_rows_L<9, INV>(in, out, count, log2n1, in_dist, out_dist, tw, s);
    case 10: return launch_rows_L<10, INV>(in, out, count, log2n1, in_dist, out_dist, tw, s);
    default: return cudaErrorInvalidValue;
    }
}

template <int LB, bool INV>
static cudaError_t launch_rows3_L(const float2* in, float2* out, long long count, int l1, int l2, long long out_dist,
                                  const float2* tw, cudaStream_t s)
{
    using P = BPass<LB>;
    const long long blocks = count * ((1ll << l1) / P::C) << l2;
    return launch_pdl(k_rows3<LB, INV>, dim3((unsigned)blocks), dim3(P::THREADS), P::SMEM, s, in, out, l1, l2, out_dist,
                      tw);
}

template <bool INV>
static cudaError_t launch_rows3(int l3, const float2* in, float2* out, long long count, int l1, int l2,
                                long long out_dist, const float2* tw, cudaStream_t s)
{
    switch (l3) {
    case 7: return launch_rows3_L<7, INV>(in, out, count, l1, l2, out_dist, tw, s);
    case 8: return launch_rows3_L<8, INV>(in, out, count, l1, l2, out_dist, tw, s);
    case 9: return launch_rows3_L<9, INV>(in, out, count, l1, l2, out_dist, tw, s);
    case 10: return launch_rows3_L<10, INV>(in, out, count, l1, l2, out_dist, tw, s);
    default: return cudaErrorInvalidValue;
    }
}

template <int L1, int L2, bool INV, bool MIRROR>
static cudaError_t launch_cols12_L(const float2* in, float2* mid, int l3, long long count, long long in_dist,
                                   const float2* tw, cudaStream_t s)
{
    using C = Cols12<L1, L2>;
    int lgc = kPanelLog2 - 3 - L1 - L2;
    if (lgc < 5) lgc = 5;
    if (lgc > l3) lgc = l3;
    const int panels = (int)(count << (l3 - lgc));
    const unsigned tiles = 1u << (L1 + L2 + lgc - ilog2(C::THREADS * 32));
    for (int st = 0; st <= panels; ++st) {
        const unsigned blocks = st > 0 && st < panels ? 2 * tiles : tiles;
        const cudaError_t e = launch_pdl(k_cols12<L1, L2, INV, MIRROR>, dim3(blocks), dim3(C::THREADS), C::SMEM, s, in, mid, l3, lgc,
                                         st, panels, in_dist, tw);
        if (e != cudaSuccess) return e;
        count_launch();
    }
    return cudaSuccess;
}

// Three sub-lengths of at most 2^10 (each >= 2^7), as equal as possible.
static constexpr bool plan3(int log2n, int* l1, int* l2, int* l3)
{
    if (log2n < 21 || log2n > 30) return false;
    *l3 = (log2n + 2) / 3;
    *l2 = (log2n - *l3 + 1) / 2;
    *l1 = log2n - *l3 - *l2;
    return *l1 >= 7 && *l3 <= 10 && *l2 <= 10;
}

// The (l1, l2) that plan3 makes of 2^21 .. 2^28, and for real forward transforms of
// 2^29 packed pairs (n = 2^30; complex sizes end at 2^28).  A panel there is 128 MB
// and no longer stays in L2: the chain is then two passes like any other.
#define CKG_COLS12_PAIRS(X) X(7, 7) X(7, 8) X(8, 8) X(8, 9) X(9, 9)
constexpr int kMaxLog2Half = 29;

static constexpr bool cols12_covers_plan3()
{
    for (int log2n = 21; log2n <= kMaxLog2Half; ++log2n) {
        int l1 = 0, l2 = 0, l3 = 0;
        if (!plan3(log2n, &l1, &l2, &l3)) return false;
        bool found = log2n == kMaxLog2Half && l1 == 9 && l2 == 10;
#define CKG_CASE(L1, L2) found = found || (l1 == L1 && l2 == L2);
        CKG_COLS12_PAIRS(CKG_CASE)
#undef CKG_CASE
        if (!found) return false;
    }
    return true;
}
static_assert(cols12_covers_plan3(), "every three-pass size has its kernels");

template <bool INV, bool MIRROR>
static cudaError_t launch_cols12(int l1, int l2, int l3, const float2* in, float2* mid, long long count, long long in_dist,
                                 const float2* tw, cudaStream_t s)
{
    switch (l1 * 16 + l2) {
#define CKG_CASE(L1, L2) \
    case L1 * 16 + L2: return launch_cols12_L<L1, L2, INV, MIRROR>(in, mid, l3, count, in_dist, tw, s);
        CKG_COLS12_PAIRS(CKG_CASE)
#undef CKG_CASE
    case 9 * 16 + 10:
        if constexpr (MIRROR) return launch_cols12_L<9, 10, INV, MIRROR>(in, mid, l3, count, in_dist, tw, s);
        return cudaErrorInvalidValue;
    default: return cudaErrorInvalidValue;
    }
}

// Sizes from 2^kThreePassMinLog2 on run as three passes whose tiles are all
// 16 columns / rows wide (128-byte accesses); two passes there would need
// sub-lengths above 2^10, whose tiles are 4 or 8 wide.
constexpr int kThreePassMinLog2 = 21;

static cudaError_t launch_rows_split(int lb, const float2* in, float2* out, long long count, int log2n1, int log2k1,
                                     long long in_dist, long long out_dist, const float2* tw, cudaStream_t s);
static cudaError_t launch_cols_merge(int la, const float2* in, float2* out, long long count, int log2n2,
                                     long long in_dist, long long out_dist, const float2* tw, cudaStream_t s);

// kind C2C_FWD / C2C_INV: complex transforms of 2^log2n points.  R2C: real
// forward of 2^(log2n+1) reals read as 2^log2n packed pairs, the split fused
// into the third pass (2^log2n + 1 bins out).  C2R: real inverse from
// 2^log2n + 1 bins, the merge fused into the first pass.  Distances in float2.
static cudaError_t launch_three_pass(Kind kind, int log2n, const float2* in, float2* out, long long count,
                                     long long in_dist, long long out_dist, const float2* tw, float2* tmp,
                                     long long group, cudaStream_t s)
{
    int l1, l2, l3;
    if (!plan3(log2n, &l1, &l2, &l3)) return cudaErrorInvalidValue;
    const bool inverse = kind == C2C_INV || kind == C2R;
    const long long n = 1ll << log2n, M = 1ll << (l2 + l3);
    for (long long off = 0; off < count; off += group) {
        const long long cnt = count - off < group ? count - off : group;
        const float2* src = in + off * in_dist;
        float2* dst = out + off * out_dist;
        cudaError_t e;
        if (kind != C2R) {
            e = inverse       ? launch_cols12<true, false>(l1, l2, l3, src, tmp, cnt, in_dist, tw, s)
                : kind == R2C ? launch_cols12<false, true>(l1, l2, l3, src, tmp, cnt, in_dist, tw, s)
                              : launch_cols12<false, false>(l1, l2, l3, src, tmp, cnt, in_dist, tw, s);
        } else {
            // pass 1: columns of length N1 over the M = N2 N3 columns -> tmp,
            // with the merge (its tiles mirror across panels); pass 2: in every
            // row k1, columns of length N2 over the N3 columns, in place
            e = launch_cols_merge(l1, src, tmp, cnt, l2 + l3, in_dist, n, tw, s);
            if (e == cudaSuccess) e = launch_cols<true>(l2, tmp, tmp, cnt << l1, l3, M, M, tw, s);
            count_launch(2);
        }
        // pass 3: rows of length N3, C consecutive k1 per tile -> out (real
        // forward: row pairs k, N1 N2 - k with the split)
        if (e == cudaSuccess)
            e = kind == R2C ? launch_rows_split(l3, tmp, dst, cnt, l1 + l2, l1, n, out_dist, tw, s)
                : inverse   ? launch_rows3<true>(l3, tmp, dst, cnt, l1, l2, out_dist, tw, s)
                            : launch_rows3<false>(l3, tmp, dst, cnt, l1, l2, out_dist, tw, s);
        if (e != cudaSuccess) return e;
        count_launch();
    }
    return cudaSuccess;
}

LargePlan large_plan(int log2n)
{
    LargePlan p;
    p.log2n = log2n;
    p.log2n1 = log2n / 2;
    p.log2n2 = log2n - p.log2n1;
    return p;
}

static bool large_supported(int log2n)
{
    const LargePlan p = large_plan(log2n);
    return log2n > kSmallMaxLog2Complex && p.log2n1 >= 7 && p.log2n2 <= 14;
}

size_t large_scratch_bytes(Kind kind, int log2n)
{
    // complex: one N-point intermediate; real: one (N/2)-point intermediate
    const int lc = (kind == R2C || kind == C2R) ? log2n - 1 : log2n;
    return sizeof(float2) << lc;
}

cudaError_t launch_large_c2c(bool inverse, int log2n, const void* in, void* out, long long count,
                             long long in_dist, long long out_dist, const float2* tw,
                             void* scratch, size_t scratch_bytes, cudaStream_t s)
{
    // the row passes drop the intermediate's 128-byte L2 lines
    if (!large_supported(log2n) || ((uintptr_t)scratch & 127)) return cudaErrorInvalidValue;
    if (count <= 0) return cudaSuccess;
    // 2^15, 2^16: both passes inside one persistent CTA per transform
    // (fft_mid.cu), or inside one cluster per transform (fft_l2pass.cu); the
    // intermediate kept in L2 either way
    if (mid_supported(log2n) && mid_enabled(log2n) && ((uintptr_t)in & 15) == 0 &&
        (in_dist & 1) == 0 && scratch_bytes >= mid_scratch_bytes(log2n, count))
        return launch_mid(inverse ? 1 : 0, log2n, in, out, count, in_dist, out_dist, tw, scratch, scratch_bytes, s);
    if (l2pass_supported(log2n))
        return launch_l2pass(inverse ? 1 : 0, log2n, in, out, count, in_dist, out_dist, tw, scratch, scratch_bytes, s);
    const LargePlan p = large_plan(log2n);
    const long long n = 1ll << log2n;
    const long long group = (long long)(scratch_bytes / (sizeof(float2) * (size_t)n));
    if (group < 1) return cudaErrorInvalidValue;
    const float2* src = (const float2*)in;
    float2* dst = (float2*)out;
    float2* tmp = (float2*)scratch;
    if (log2n >= kThreePassMinLog2)
        return launch_three_pass(inverse ? C2C_INV : C2C_FWD, log2n, src, dst, count, in_dist, out_dist, tw, tmp,
                                 group, s);
    for (long long off = 0; off < count; off += group) {
        const long long cnt = count - off < group ? count - off : group;
        cudaError_t e = cudaSuccess;
        if (launch_flow(inverse, log2n, src + off * in_dist, dst + off * out_dist, cnt, in_dist, out_dist, tw, tmp,
                        scratch_bytes, s, &e)) {
            if (e != cudaSuccess) return e;
            continue;
        }
        e = inverse
            ? launch_cols<true>(p.log2n1, src + off * in_dist, tmp, cnt, p.log2n2, in_dist, n, tw, s)
            : launch_cols<false>(p.log2n1, src + off * in_dist, tmp, cnt, p.log2n2, in_dist, n, tw, s);
        if (e != cudaSuccess) return e;
        e = inverse
            ? launch_rows<true>(p.log2n2, tmp, dst + off * out_dist, cnt, p.log2n1, n, out_dist, tw, s)
            : launch_rows<false>(p.log2n2, tmp, dst + off * out_dist, cnt, p.log2n1, n, out_dist, tw, s);
        if (e != cudaSuccess) return e;
        count_launch(2);
    }
    return cudaSuccess;
}

template <int LB>
static cudaError_t launch_rows_split_L(const float2* in, float2* out, long long count, int log2n1, int log2k1,
                                       long long in_dist, long long out_dist, const float2* tw, cudaStream_t s)
{
    using P = SPass<LB>;
    const long long blocks = count * ((1ll << log2n1) / P::C);
    return launch_pdl(k_rows_split<LB>, dim3((unsigned)blocks), dim3(P::THREADS), P::SMEM, s, in, out, log2n1,
                      log2k1, in_dist, out_dist, tw);
}

// Row pass with the real split fused, row sub-length 2^lb (7 .. 10).
static cudaError_t launch_rows_split(int lb, const float2* in, float2* out, long long count, int log2n1, int log2k1,
                                     long long in_dist, long long out_dist, const float2* tw, cudaStream_t s)
{
    switch (lb) {
    case 7: return launch_rows_split_L<7>(in, out, count, log2n1, log2k1, in_dist, out_dist, tw, s);
    case 8: return launch_rows_split_L<8>(in, out, count, log2n1, log2k1, in_dist, out_dist, tw, s);
    case 9: return launch_rows_split_L<9>(in, out, count, log2n1, log2k1, in_dist, out_dist, tw, s);
    case 10: return launch_rows_split_L<10>(in, out, count, log2n1, log2k1, in_dist, out_dist, tw, s);
    default: return cudaErrorInvalidValue;
    }
}

// Two-pass real forward with the split fused into the row pass, for half
// lengths whose row sub-length is 2^8 .. 2^10 below the three-pass sizes.
static bool rows_split_supported(int lm)
{
    const LargePlan p = large_plan(lm);
    return lm > kSmallMaxLog2Complex && lm < kThreePassMinLog2 && p.log2n1 >= 7 && p.log2n2 >= 8 && p.log2n2 <= 10;
}

static cudaError_t launch_r2c_rows_split(int lm, const float2* in, float2* out, long long count, long long in_dist,
                                         long long out_dist, const float2* tw, float2* tmp, size_t scratch_bytes,
                                         cudaStream_t s)
{
    const LargePlan p = large_plan(lm);
    const long long M = 1ll << lm;
    const long long group = (long long)(scratch_bytes / (sizeof(float2) * (size_t)M));
    if (group < 1) return cudaErrorInvalidValue;
    for (long long off = 0; off < count; off += group) {
        const long long cnt = count - off < group ? count - off : group;
        bool done;
        cudaError_t e = launch_real_chain<false>(lm, in + off * in_dist, out + off * out_dist, tmp, cnt, in_dist, out_dist,
                                                 tw, s, &done);
        if (e != cudaSuccess) return e;
        if (done) continue;
        e = launch_cols<false, true>(p.log2n1, in + off * in_dist, tmp, cnt, p.log2n2, in_dist, M, tw, s);
        if (e == cudaSuccess)
            e = launch_rows_split(p.log2n2, tmp, out + off * out_dist, cnt, p.log2n1, p.log2n1, M, out_dist, tw, s);
        if (e != cudaSuccess) return e;
        count_launch(2);
    }
    return cudaSuccess;
}

cudaError_t launch_large_r2c(int log2n, const void* in, void* out, long long count,
                             long long in_dist, long long out_dist, const float2* tw,
                             void* scratch, size_t scratch_bytes, cudaStream_t s)
{
    // in: n floats per frame (n/2 packed complex), out: n/2+1 complex per frame
    // (half lengths 2^15 / 2^16: the cluster kernel with the split fused into
    // its row tiles, 3355 / 3303 GB/s batched at n = 2^16 / 2^17; two launches
    // through HBM, one value a thread, 2507 / 2609)
    const int lm = log2n - 1;
    const long long M = 1ll << lm;
    if ((uintptr_t)scratch & 127) return cudaErrorInvalidValue;
    if (count <= 0) return cudaSuccess;
    if (l2pass_supported(lm))
        return launch_l2pass(2, lm, in, out, count, in_dist / 2, out_dist, tw, scratch, scratch_bytes, s);
    if (rows_split_supported(lm))
        return launch_r2c_rows_split(lm, (const float2*)in, (float2*)out, count, in_dist / 2, out_dist, tw,
                                     (float2*)scratch, scratch_bytes, s);
    int l1, l2, l3;
    if (lm >= kThreePassMinLog2 && plan3(lm, &l1, &l2, &l3)) {
        const long long group = (long long)(scratch_bytes / (sizeof(float2) * (size_t)M));
        if (group < 1) return cudaErrorInvalidValue;
        return launch_three_pass(R2C, lm, (const float2*)in, (float2*)out, count, in_dist / 2, out_dist, tw,
                                 (float2*)scratch, group, s);
    }
    return cudaErrorInvalidValue;
}

template <int LA>
static cudaError_t launch_cols_merge_L(const float2* in, float2* out, long long count, int log2n2,
                                       long long in_dist, long long out_dist, const float2* tw, cudaStream_t s)
{
    using P = SPass<LA>;
    const long long blocks = count * ((1ll << log2n2) / P::C);
    return launch_pdl(k_cols_merge<LA>, dim3((unsigned)blocks), dim3(P::THREADS), P::SMEM, s, in, out, log2n2,
                      in_dist, out_dist, tw);
}

// Column pass with the real merge fused, column sub-length 2^la (7 .. 10).
static cudaError_t launch_cols_merge(int la, const float2* in, float2* out, long long count, int log2n2,
                                     long long in_dist, long long out_dist, const float2* tw, cudaStream_t s)
{
    switch (la) {
    case 7: return launch_cols_merge_L<7>(in, out, count, log2n2, in_dist, out_dist, tw, s);
    case 8: return launch_cols_merge_L<8>(in, out, count, log2n2, in_dist, out_dist, tw, s);
    case 9: return launch_cols_merge_L<9>(in, out, count, log2n2, in_dist, out_dist, tw, s);
    case 10: return launch_cols_merge_L<10>(in, out, count, log2n2, in_dist, out_dist, tw, s);
    default: return cudaErrorInvalidValue;
    }
}

// Two-pass real inverse with the merge fused into the column pass, for half
// lengths whose column sub-length is 2^7 .. 2^10 below the three-pass sizes.
static bool cols_merge_supported(int lm)
{
    const LargePlan p = large_plan(lm);
    return lm > kSmallMaxLog2Complex && lm < kThreePassMinLog2 && p.log2n1 >= 7 && p.log2n1 <= 10 &&
           p.log2n2 <= 14;
}

static cudaError_t launch_c2r_cols_merge(int lm, const float2* in, float2* out, long long count, long long in_dist,
                                         long long out_dist, const float2* tw, float2* tmp, size_t scratch_bytes,
                                         cudaStream_t s)
{
    const LargePlan p = large_plan(lm);
    const long long M = 1ll << lm;
    const long long group = (long long)(scratch_bytes / (sizeof(float2) * (size_t)M));
    if (group < 1) return cudaErrorInvalidValue;
    for (long long off = 0; off < count; off += group) {
        const long long cnt = count - off < group ? count - off : group;
        bool done;
        cudaError_t e = launch_real_chain<true>(lm, in + off * in_dist, out + off * out_dist, tmp, cnt, in_dist, out_dist,
                                                tw, s, &done);
        if (e != cudaSuccess) return e;
        if (done) continue;
        e = launch_cols_merge(p.log2n1, in + off * in_dist, tmp, cnt, p.log2n2, in_dist, M, tw, s);
        if (e != cudaSuccess) return e;
        e = launch_rows<true>(p.log2n2, tmp, out + off * out_dist, cnt, p.log2n1, M, out_dist, tw, s);
        if (e != cudaSuccess) return e;
        count_launch(2);
    }
    return cudaSuccess;
}

cudaError_t launch_large_c2r(int log2n, const void* in, void* out, long long count,
                             long long in_dist, long long out_dist, const float2* tw,
                             void* scratch, size_t scratch_bytes, cudaStream_t s)
{
    // in: n/2+1 complex per frame, out: n floats per frame (n/2 packed complex)
    // (half lengths 2^15 / 2^16: the cluster kernel with the merge fused into
    // its column tiles, 3347 / 3018 GB/s batched at n = 2^16 / 2^17; two launches
    // through HBM, one value a thread, 2714 / 2554)
    const int lm = log2n - 1;
    const long long M = 1ll << lm;
    if ((uintptr_t)scratch & 127) return cudaErrorInvalidValue;
    if (count <= 0) return cudaSuccess;
    if (l2pass_supported(lm))
        return launch_l2pass(3, lm, in, out, count, in_dist, out_dist / 2, tw, scratch, scratch_bytes, s);
    if (cols_merge_supported(lm))
        return launch_c2r_cols_merge(lm, (const float2*)in, (float2*)out, count, in_dist, out_dist / 2, tw,
                                     (float2*)scratch, scratch_bytes, s);
    int l1, l2, l3;
    if (lm >= kThreePassMinLog2 && plan3(lm, &l1, &l2, &l3)) {
        const long long group = (long long)(scratch_bytes / (sizeof(float2) * (size_t)M));
        if (group < 1) return cudaErrorInvalidValue;
        return launch_three_pass(C2R, lm, (const float2*)in, (float2*)out, count, in_dist, out_dist / 2, tw,
                                 (float2*)scratch, group, s);
    }
    return cudaErrorInvalidValue;
}

template <int L1, int L2>
static cudaError_t attr_cols12()
{
    const int smem = (int)Cols12<L1, L2>::SMEM;
    const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(k_cols12<L1, L2, false, false>, a, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_cols12<L1, L2, false, true>, a, smem);
    return e == cudaSuccess ? cudaFuncSetAttribute(k_cols12<L1, L2, true, false>, a, smem) : e;
}

template <int LA, int LB>
static cudaError_t attr_real_chain()
{
    const int smem = (int)RealChain<LA, LB>::SMEM;
    const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(k_real_chain<LA, LB, false>, a, smem);
    return e == cudaSuccess ? cudaFuncSetAttribute(k_real_chain<LA, LB, true>, a, smem) : e;
}

template <int L>
static cudaError_t attr_pass()
{
    const int smem = (int)BPass<L>::SMEM;
    const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(k_rows3<L, false>, a, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_rows3<L, true>, a, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_rows_split<L>, a, (int)SPass<L>::SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_cols_merge<L>, a, (int)SPass<L>::SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_cols<L, false, false>, a, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_cols<L, false, true>, a, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_cols<L, true, false>, a, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_rows<L, false>, a, smem);
    return e == cudaSuccess ? cudaFuncSetAttribute(k_rows<L, true>, a, smem) : e;
}

cudaError_t prepare_large()
{
    cudaError_t e = attr_pass<7>();
    if (e == cudaSuccess) e = attr_pass<8>();
    if (e == cudaSuccess) e = attr_pass<9>();
    if (e == cudaSuccess) e = attr_pass<10>();
    if (e == cudaSuccess) e = attr_real_chain<8, 9>();
    if (e == cudaSuccess) e = attr_real_chain<9, 9>();
    if (e == cudaSuccess) e = attr_real_chain<9, 10>();
    if (e == cudaSuccess) e = attr_real_chain<10, 10>();
#define CKG_CASE(L1, L2) \
    if (e == cudaSuccess) e = attr_cols12<L1, L2>();
    CKG_COLS12_PAIRS(CKG_CASE)
#undef CKG_CASE
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_cols12<9, 10, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)Cols12<9, 10>::SMEM);
    return e;
}

}  // namespace ckg
