// fft_pair_passes.cuh -- the passes of the multi-pass transform
// (fft_passes.cuh) with two neighbouring columns or rows per thread in packed
// FP32 arithmetic (fft_pair.cuh).  Same stages, twiddles and rounding as the
// one-value passes, so the results are the same bits; a third fewer
// instructions per value (both passes of 2^16: 85 -> 54), and every twiddle
// load ahead of the data.  With them a pass over more data than L2 runs at the
// HBM copy rate (2^24 in three passes: 135 -> 120 us, 6.7 TB/s), and the two
// passes of one 2^20 transform, bound by latency, take 10.1 us instead of 17.1.
//
// A tile is CP pairs (C = 2 CP columns or rows).  Loads and stores of
// neighbouring columns are one 16-byte access where the array allows it, two
// 8-byte ones where it does not (a base or a distance that is an odd number
// of values; the same for a whole launch or transform, so the branch is
// uniform).
#pragma once
#include "fft_pair.cuh"
#include "fft_passes.cuh"

namespace ckg {

// Sub-transforms of 2^LS points (7 <= LS <= 10), 16 values per thread and
// column, in tiles of at most CPMAX pairs and MAXT threads.
template <int LS, int MAXT, int CPMAX = 16>
struct PairCfg {
    static_assert(LS >= 7 && LS <= 10, "sub-lengths of 2^7 .. 2^10");
    static constexpr int LOG2R = 4, R = 16;
    static constexpr int T = (1 << LS) / R;
    static constexpr int CP = MAXT / T < CPMAX ? MAXT / T : CPMAX;
    static constexpr int C = 2 * CP;
    static constexpr int THREADS = CP * T;
    static_assert(CP >= 2 && CP <= 16, "2 to 16 pairs a tile");
    // column tiles: CP pairs side by side
    using ColView = PairView<CP, (CP < 8)>;
    static constexpr int COL_SLOTS = CP * (CP < 8 ? padded_len(1 << LS) : (1 << LS));
    // row tiles: one padded image per row pair, RS slots apart.  The lanes of
    // the row passes' last step hold neighbouring row pairs: an image
    // distance of 8 / (pairs side by side) mod 8 keeps eight lanes in
    // distinct 16-byte banks.
    static constexpr int rowdist(int want)
    {
        int d = padded_len(1 << LS);
        while (d % 8 != want % 8) ++d;
        return d;
    }
    static constexpr int RS = rowdist(CP < 8 ? 8 / CP : 1);     // CP pairs side by side
    static constexpr int ROW_SLOTS = CP * RS;
    // column twiddles W^(n2 T 2^e), e = 0..3, one entry per pair, behind the tile
    static constexpr int TW_SLOTS = 4 * CP;
    static constexpr int TILE_SLOTS = COL_SLOTS + TW_SLOTS > ROW_SLOTS ? COL_SLOTS + TW_SLOTS : ROW_SLOTS;
    static constexpr size_t SMEM = sizeof(cpair) * (size_t)TILE_SLOTS;
};

// W_N^p from the two short levels of big_twiddle, copied to shared memory:
// lo[2^s], then hi[2^(ln - s)], s = ceil(ln / 2); the same product, conjugated
// factors for the inverse.
template <int LN, bool INV>
struct BigTable {
    static constexpr int S = (LN + 1) / 2;
    static constexpr int kEntries = (1 << S) + (1 << (LN - S));
    const float2* s;
    __device__ __forceinline__ float2 operator()(int p) const { return cmul(s[(1 << S) + (p >> S)], s[p & ((1 << S) - 1)]); }
    __device__ static void fill(float2* d, const float2* __restrict__ tw, int tid, int threads)
    {
        for (int k = tid; k < (1 << S); k += threads) d[k] = tw_load<INV>(tw + (1 << LN), k);
        for (int k = tid; k < (1 << (LN - S)); k += threads) d[(1 << S) + k] = tw_load<INV>(tw + (1 << (LN - S)), k);
    }
};
// The same from global memory, for transforms whose levels are too long.
template <bool INV>
struct BigGlobal {
    const float2* __restrict__ tw;
    int ln;
    __device__ __forceinline__ float2 operator()(int p) const { return big_twiddle<INV>(tw, ln, p); }
};

// The column passes' twiddles W_N^(n2 k1), k1 = t + m T, m = 4q + r:
//   W^(n2 t) * W^(4 n2 T q) * W^(n2 T r).
// The factors that do not depend on t, W^(n2 T 2^e), e = 0..3, are made once
// per tile: threads tid < 4 C look one up each (cols_twiddle_entry, early, so
// that the lookup's latency is hidden) and put it in shared memory before a
// barrier (cols_twiddle_put).  10 table lookups a thread and column before, 2
// now: these lookups were most of the difference between the column pass's
// 64 instructions per value and the row pass's 42.
// Big: W_N^p for 0 <= p < N (BigTable, or a lookup in global memory).
template <int LA, class P, class Big, class Col>
__device__ __forceinline__ float2 cols_twiddle_entry(int log2n2, int tid, const Big& big, Col&& col)
{
    static_assert(P::THREADS >= 4 * P::C, "one entry a thread");
    if (tid >= 4 * P::C) return make_float2(0.f, 0.f);
    const int c = tid % P::C, e = tid / P::C, ln = LA + log2n2;
    return big((int)((((unsigned)col(c) * (unsigned)P::T) << e) & ((1u << ln) - 1u)));
}
template <class P>
__device__ __forceinline__ void cols_twiddle_put(cpair* twsm, int tid, float2 w)
{
    if (tid < 4 * P::C) {
        const int c = tid % P::C, e = tid / P::C;
        float* d = reinterpret_cast<float*>(twsm + e * P::CP + c / 2) + (c & 1);
        d[0] = w.x;
        d[2] = w.y;
    }
}
// W_N^(n2 t) of the thread's two columns.
template <int LA, class Big>
__device__ __forceinline__ cpair cols_twiddle_t(int log2n2, int n2a, int n2b, int t, const Big& big)
{
    const int ln = LA + log2n2, mask = (1 << ln) - 1;
    return make_pair2(big((n2a * t) & mask), big((n2b * t) & mask));
}

// Last step of a column pass: v[m] = Y[k1], k1 = t + m T, of columns n2 and
// n2 + 1, times W_N^(n2 k1) (a = W_N^(n2 t)), stored at out[N2 k1 + n2].
template <class P>
__device__ __forceinline__ void cols_twiddle_store(cpair (&v)[P::R], float2* __restrict__ out, int log2n2, int n2,
                                                   int cp, int t, const cpair* twsm, cpair a)
{
    const cpair b1 = twsm[cp], b2 = twsm[P::CP + cp];
    const cpair b3 = cmul(b1, b2);
    const cpair lad0 = twsm[2 * P::CP + cp], lad1 = twsm[3 * P::CP + cp];
    float2* dst = out + n2 + ((long long)t << log2n2);
    const long long step = (long long)P::T << log2n2;
    auto store = [&](int m, cpair x) { *reinterpret_cast<float4*>(dst + m * step) = interleave(x); };
    static_for<0, 4>([&](auto qc) {
        constexpr int q = decltype(qc)::value;
        cpair aq = a;
        if constexpr (q & 1) aq = cmul(aq, lad0);
        if constexpr (q & 2) aq = cmul(aq, lad1);
        store(4 * q + 0, cmul(v[4 * q + 0], aq));
        store(4 * q + 1, cmul(v[4 * q + 1], cmul(aq, b1)));
        store(4 * q + 2, cmul(v[4 * q + 2], cmul(aq, b2)));
        store(4 * q + 3, cmul(v[4 * q + 3], cmul(aq, b3)));
    });
}

// ------------------------------------------------------------ whole passes
// One tile a CTA.  Each pass loads every twiddle it needs, then calls wait()
// (for the kernels ahead in the stream: the twiddle table is never written),
// then loads its data.

// Column pass (pass_cols); al: 16-byte aligned input rows.  `out` (scratch)
// always is.
template <int LA, bool INV, class P, class Wait>
__device__ __forceinline__ void pair_cols(const float2* __restrict__ in, float2* __restrict__ out, int log2n2, int tile,
                                          int tid, cpair* smem, const float2* __restrict__ tw, Wait&& wait)
{
    const int cp = tid % P::CP, t = tid / P::CP;
    const int n2 = tile * P::C + 2 * cp;
    const StageRegs<LA, INV> regs(tw, t, t);
    const BigGlobal<INV> big{tw, LA + log2n2};
    const float2 went = cols_twiddle_entry<LA, P>(log2n2, tid, big, [&](int c) { return tile * P::C + c; });
    const cpair wt = cols_twiddle_t<LA>(log2n2, n2, n2 + 1, t, big);
    wait();
    const float2* src = in + n2 + ((long long)t << log2n2);
    const long long step = (long long)P::T << log2n2;
    cpair v[16];
    if (((uintptr_t)in & 15) == 0) {
#pragma unroll
        for (int m = 0; m < 16; ++m) v[m] = make_pair2(__ldcs(reinterpret_cast<const float4*>(src + m * step)));
    } else {
#pragma unroll
        for (int m = 0; m < 16; ++m) v[m] = make_pair2(__ldcs(src + m * step), __ldcs(src + m * step + 1));
    }
    cpair* twsm = smem + P::COL_SLOTS;
    typename P::ColView view{smem + cp};
    stockham<LA, 4, INV, false>(v, t, regs, view, [] { __syncthreads(); }, [&] { cols_twiddle_put<P>(twsm, tid, went); },
                                [] {});
    cols_twiddle_store<P>(v, out, log2n2, n2, cp, t, twsm, wt);
}

// Row pass with the output transpose folded into the last stage exchange
// (pass_rows_xt): thread (pair, t) = (tid / T, tid mod T) for all stages but
// the last, (tid mod CP, tid / CP) for the last.  The input is a dead
// intermediate (128-byte aligned): its L2 lines are dropped once read.
template <int LB, bool INV, class P, class Wait>
__device__ __forceinline__ void pair_rows(const float2* __restrict__ in, float2* __restrict__ out, int log2n1, int tile,
                                          int tid, cpair* smem, const float2* __restrict__ tw, int log2_row_stride,
                                          Wait&& wait)
{
    using S = Sched<LB, 4>;
    constexpr int N2 = 1 << LB, T = P::T, NST = S::nstages;
    const int row0 = tile * P::C;
    const int rp = tid / T, t = tid % T, rq = tid % P::CP, tq = tid / P::CP;
    const StageRegs<LB, INV> regs(tw, NST > 2 ? t : tq, tq);
    wait();
    cpair v[16];
    {
        const float2* src = in + ((long long)(row0 + 2 * rp) << log2_row_stride) + t;
        const float2* src1 = src + (1ll << log2_row_stride);
#pragma unroll
        for (int m = 0; m < 16; ++m) v[m] = make_pair2(__ldcs(src + m * T), __ldcs(src1 + m * T));
        PairView<1, true> view{smem + rp * P::RS};
        static_for<0, NST - 1>([&](auto sc) {
            constexpr int st = decltype(sc)::value;
            stage_compute<LB, 4, S::lrs(st), S::lns(st), INV>(v, t, regs);
            stage_write<LB, 4, S::lrs(st), S::lns(st)>(v, t, view);
            if constexpr (st + 2 < NST) {
                xsync<(T <= 32)>();
                stage_read<LB, 4>(v, t, view);
                xsync<(T <= 32)>();
            }
        });
    }
    __syncthreads();
    // every thread of the tile has consumed its inputs
    constexpr int LINES = N2 / 16;
#pragma unroll
    for (int l = tid; l < P::C * LINES; l += P::THREADS) {
        const char* row = (const char*)(in + ((long long)(row0 + l / LINES) << log2_row_stride));
        asm volatile("discard.global.L2 [%0], 128;" ::"l"(row + 128 * (l % LINES)) : "memory");
    }
    stage_read<LB, 4>(v, tq, PairView<1, true>{smem + rq * P::RS});
    constexpr int LRS = S::lrs(NST - 1), LNS = S::lns(NST - 1), U = 16 >> LRS, NS = 1 << LNS;
    stage_compute<LB, 4, LRS, LNS, INV>(v, tq, regs);
    // v[u + j U] = X[tq + u T + j NS] of rows row0 + 2 rq and the next one
    float2* dst = out + row0 + 2 * rq + ((long long)tq << log2n1);
    if (((uintptr_t)out & 15) == 0) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
            for (int j = 0; j < (1 << LRS); ++j)
                __stcs(reinterpret_cast<float4*>(dst + ((long long)(u * T + j * NS) << log2n1)), interleave(v[u + j * U]));
        }
    } else {
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
            for (int j = 0; j < (1 << LRS); ++j) {
                // shifted by one row: the second half of an aligned pair
                // comes from the next lane
                float2* d = dst + ((long long)(u * T + j * NS) << log2n1);
                const float2 a = lane0(v[u + j * U]), b = lane1(v[u + j * U]);
                const float nx = __shfl_down_sync(0xffffffffu, a.x, 1), ny = __shfl_down_sync(0xffffffffu, a.y, 1);
                if (rq == 0) __stcs(d, a);
                if (rq < P::CP - 1) __stcs(reinterpret_cast<float4*>(d + 1), make_float4(b.x, b.y, nx, ny));
                else __stcs(d + 1, b);
            }
        }
    }
}

}  // namespace ckg
