// fft_pair_passes.cuh -- the passes of the multi-pass transform
// (fft_passes.cuh) with two neighbouring columns or rows per thread in packed
// FP32 arithmetic (fft_pair.cuh).  The complex passes have the stages, twiddles
// and rounding of the one-value passes, so the same bits (the split and merge
// passes round their own twiddles, rot32_exact, and mirrored rows and columns in
// another order: real transforms of a job run, on the one-value passes, differ in the
// last bits, both within the same error); a third fewer
// instructions per value (both passes of 2^16: 85 -> 54), and every twiddle
// load ahead of the data.  With them a pass over more data than L2 runs at the
// HBM copy rate (2^24 in three passes: 135 -> 120 us, 6.7 TB/s), and the two
// passes of one 2^20 transform, bound by latency, take 10.6 us instead of 17.1.
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

// The column pass of a real forward transform: rows k1 > N1/2 are stored as
//   conj(Y[k1]) * W_N^(n2 (N1 - k1)),
// the conjugate of what the complex pass stores times W_N2^n2, so that the row
// pass, DFT over n2, gives conj(Z[M - k]) at the very k2 where the row
// N1 - k1 gives Z[k] (see pair_rows_split).  N1 - k1 = (T - t) + (15 - m) T:
// the same products, from a2 = W_N^(n2 (T - t)).  Row N1/2 (m = 8 of t = 0)
// is its own mirror and stays plain (plain_half: every column of this tile
// belongs to that row).
template <class P>
__device__ __forceinline__ void cols_twiddle_store_mirror(cpair (&v)[P::R], float2* __restrict__ out, int log2n2, int n2,
                                                          int cp, int t, const cpair* twsm, cpair a, cpair a2,
                                                          bool plain_half)
{
    const cpair b1 = twsm[cp], b2 = twsm[P::CP + cp];
    const cpair b3 = cmul(b1, b2);
    const cpair lad0 = twsm[2 * P::CP + cp];
    float2* dst = out + n2 + ((long long)t << log2n2);
    const long long step = (long long)P::T << log2n2;
    auto store = [&](int m, cpair x) { *reinterpret_cast<float4*>(dst + m * step) = interleave(x); };
    static_for<0, 2>([&](auto qc) {
        constexpr int q = decltype(qc)::value;
        const cpair aq = q ? cmul(a, lad0) : a;
        store(4 * q + 0, cmul(v[4 * q + 0], aq));
        store(4 * q + 1, cmul(v[4 * q + 1], cmul(aq, b1)));
        store(4 * q + 2, cmul(v[4 * q + 2], cmul(aq, b2)));
        store(4 * q + 3, cmul(v[4 * q + 3], cmul(aq, b3)));
    });
    static_for<0, 2>([&](auto qc) {
        constexpr int q = decltype(qc)::value;
        const cpair aq = q ? cmul(a2, lad0) : a2;
        store(15 - 4 * q, cmul(conj2(v[15 - 4 * q]), aq));
        store(14 - 4 * q, cmul(conj2(v[14 - 4 * q]), cmul(aq, b1)));
        store(13 - 4 * q, cmul(conj2(v[13 - 4 * q]), cmul(aq, b2)));
        cpair x = v[12 - 4 * q];
        if (!(q == 1 && plain_half && t == 0)) x = conj2(x);
        store(12 - 4 * q, cmul(x, cmul(aq, b3)));
    });
}

// ------------------------------------------------------------ whole passes
// One tile a CTA.  Each pass loads every twiddle it needs, then calls wait()
// (for the kernels ahead in the stream: the twiddle table is never written),
// then loads its data.

// Column pass (pass_cols).  `out` (scratch) is 16-byte aligned.  MIRROR: of a
// real forward transform (cols_twiddle_store_mirror).
template <int LA, bool INV, bool MIRROR, class P, class Wait>
__device__ __forceinline__ void pair_cols(const float2* __restrict__ in, float2* __restrict__ out, int log2n2, int tile,
                                          int tid, cpair* smem, const float2* __restrict__ tw, Wait&& wait,
                                          bool plain_half = true)
{
    const int cp = tid % P::CP, t = tid / P::CP;
    const int n2 = tile * P::C + 2 * cp;
    const StageRegs<LA, INV> regs(tw, t, t);
    const BigGlobal<INV> big{tw, LA + log2n2};
    const float2 went = cols_twiddle_entry<LA, P>(log2n2, tid, big, [&](int c) { return tile * P::C + c; });
    const cpair wt = cols_twiddle_t<LA>(log2n2, n2, n2 + 1, t, big);
    cpair wt2;
    if constexpr (MIRROR) wt2 = cols_twiddle_t<LA>(log2n2, n2, n2 + 1, P::T - t, big);
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
    if constexpr (MIRROR) cols_twiddle_store_mirror<P>(v, out, log2n2, n2, cp, t, twsm, wt, wt2, plain_half);
    else cols_twiddle_store<P>(v, out, log2n2, n2, cp, t, twsm, wt);
}

// w * W_32^M, the constant in two parts: only w's own rounding and the last
// one stay.  A once rounded constant is 1-2 % faster and costs 1-2 % in accuracy,
// a bias of the scale included (real 2^17 forward 1.83e-7 against 1.79e-7 with
// the table's products that these twiddles replace).
template <int M>
__device__ __forceinline__ float2 rot32_exact(float2 w)
{
    static_assert(M >= 0 && M < 16, "the forward half circle");
    if constexpr (M % 8 == 0) {
        return rot<32, M, false>(w);
    } else {
        constexpr float c = (float)cos32(M), cl = (float)(cos32(M) - (double)c);
        constexpr float s = (float)sin32(M), sl = (float)(sin32(M) - (double)s);
        return make_float2(fmaf(w.x, c, fmaf(w.y, s, fmaf(w.x, cl, w.y * sl))),
                           fmaf(w.y, c, fmaf(-w.x, s, fmaf(w.y, cl, -w.x * sl))));
    }
}

// Column pass of a real inverse transform with the merge fused (the M + 1
// bins X of 2 M reals -> M = N1 N2 complex values y, k = N2 n1 + n2):
//   y[k] = s + c,  conj(y[M - k]) = s - c,
//   s = X[k] + conj X[M - k],  c = i conj(W_2M^k) (X[k] - conj X[M - k]).
// A thread's pair is column n2 and, as its second lane, the mirror column
// N2 - n2 conjugated and read from its end: S[n1] = conj(y[M - k]).  The
// column DFT D of S relates to the mirror column's by
//   (mirror's DFT)[k1] W_N^((N2 - n2) k1) = conj(D[k1] W_N^(n2 k1)),
// so both lanes take the same rows, stage twiddles and column twiddles, the
// merge is done in the registers that the loads filled (one s and c for two
// values, nothing staged in shared memory), and the second lane is conjugated
// on its way out.  Column 0 mirrors itself, and so does column N2/2: these two
// are the lanes of tile 0's first pair, each with its own partner loads.
// W_2M^k = W_2M^(N2 t + n2) * W_32^m for n1 = t + m T.
template <int LA, class P, class Wait>
__device__ __forceinline__ void pair_cols_merge(const float2* __restrict__ in, float2* __restrict__ out, int log2n2,
                                                int tile, int tid, cpair* smem, const float2* __restrict__ tw, Wait&& wait)
{
    const int cp = tid % P::CP, t = tid / P::CP;
    const int n2len = 1 << log2n2;
    const bool edge = tile == 0 && cp == 0;
    const int ca = tile * P::CP + cp, cb = edge ? n2len / 2 : n2len - ca;       // the lanes' columns
    const long long M = 1ll << (LA + log2n2);
    const StageRegs<LA, true> regs(tw, t, t);
    const BigGlobal<true> big{tw, LA + log2n2};
    const float2 went = cols_twiddle_entry<LA, P>(log2n2, tid, big, [&](int c) {
        return tile == 0 && c == 1 ? n2len / 2 : tile * P::CP + c / 2;
    });
    const cpair wt = cols_twiddle_t<LA>(log2n2, ca, edge ? cb : ca, t, big);
    const float2 wm = __ldg(tw + 2 * M + ((long long)t << log2n2) + ca);
    wait();
    const float2* up = in + ca + ((long long)t << log2n2);
    const float2* down = in + M - ca - ((long long)t << log2n2);
    const long long step = (long long)P::T << log2n2;
    cpair v[16];
    if (!edge) {
#pragma unroll
        for (int m = 0; m < 16; ++m) v[m] = make_pair2(__ldcs(up + m * step), __ldcs(down - m * step));
        static_for<0, 16>([&](auto mc) {
            constexpr int m = decltype(mc)::value;
            const float2 w = rot32_exact<m>(wm), a = lane0(v[m]), b = lane1(v[m]);
            const float sx = a.x + b.x, sy = a.y - b.y, dx = a.x - b.x, dy = a.y + b.y;
            const float cx = fmaf(w.y, dx, -w.x * dy), cy = fmaf(w.x, dx, w.y * dy);
            v[m] = make_pair2(make_float2(sx + cx, sy + cy), make_float2(sx - cx, sy - cy));
        });
    } else {
        const int h = n2len / 2;
        const float2 wh = __ldg(tw + 2 * M + ((long long)t << log2n2) + h);
        static_for<0, 16>([&](auto mc) {
            constexpr int m = decltype(mc)::value;
            v[m] = make_pair2(real_merge(__ldcs(up + m * step), __ldcs(down - m * step), rot32_exact<m>(wm)),
                              real_merge(__ldcs(up + m * step + h), __ldcs(down - m * step - h), rot32_exact<m>(wh)));
        });
    }
    cpair* twsm = smem + P::COL_SLOTS;
    typename P::ColView view{smem + cp};
    stockham<LA, 4, true, false>(v, t, regs, view, [] { __syncthreads(); }, [&] { cols_twiddle_put<P>(twsm, tid, went); },
                                 [] {});
    // as in cols_twiddle_store
    const cpair b1 = twsm[cp], b2 = twsm[P::CP + cp];
    const cpair b3 = cmul(b1, b2);
    const cpair lad0 = twsm[2 * P::CP + cp], lad1 = twsm[3 * P::CP + cp];
    float2* dst = out + ((long long)t << log2n2);
    const float sign = edge ? 1.f : -1.f;
    auto store = [&](int m, cpair x) {
        const float2 b = lane1(x);
        dst[ca + m * step] = lane0(x);
        dst[cb + m * step] = make_float2(b.x, sign * b.y);
    };
    static_for<0, 4>([&](auto qc) {
        constexpr int q = decltype(qc)::value;
        cpair aq = wt;
        if constexpr (q & 1) aq = cmul(aq, lad0);
        if constexpr (q & 2) aq = cmul(aq, lad1);
        store(4 * q + 0, cmul(v[4 * q + 0], aq));
        store(4 * q + 1, cmul(v[4 * q + 1], cmul(aq, b1)));
        store(4 * q + 2, cmul(v[4 * q + 2], cmul(aq, b2)));
        store(4 * q + 3, cmul(v[4 * q + 3], cmul(aq, b3)));
    });
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

// Row pass of a real forward transform with the split fused (x2 scaling of the
// reference): a pair is row k1 and its mirror N1 - k1, stored by the column
// pass so that its DFT is conj(Z[M - k]) (cols_twiddle_store_mirror), k = k1 +
// N1 k2.  Both lanes run the same stages with the same twiddles, and
//   s = Z[k] + conj Z[M - k],  c = i W_2M^k (Z[k] - conj Z[M - k]),
//   X[k] = s - c,  X[M - k] = conj(s + c)
// needs only the two lanes of one register pair: no exchange, one s and c for
// two bins.  W_2M^k = W_2M^(k1 + N1 tq) * W_32^m for k2 = tq + m T.  Rows 0 and
// N1/2 mirror themselves: they are the lanes of tile 0's first pair, stored
// plain, and find their partners through shared memory.
// log2k1: row k1' + N1' k2' at in[k1' N2' N3 + k2' N3], log2k1 = log2 N1' (the
// third pass of the three-pass transform); log2k1 = log2n1: rows back to back.
template <int LB, class P, class Wait>
__device__ __forceinline__ void pair_rows_split(const float2* __restrict__ in, float2* __restrict__ out, int log2n1,
                                                int tile, int tid, cpair* smem, const float2* __restrict__ tw, int log2k1,
                                                Wait&& wait)
{
    using S = Sched<LB, 4>;
    constexpr int N2 = 1 << LB, T = P::T, NST = S::nstages;
    const int n1 = 1 << log2n1;
    const long long M = (long long)n1 << LB;
    const int rp = tid / T, t = tid % T, rq = tid % P::CP, tq = tid / P::CP;
    auto mirror = [&](int k1) { return k1 ? n1 - k1 : n1 / 2; };
    auto row = [&](int k1) {
        return in + ((long long)(k1 & ((1 << log2k1) - 1)) << (log2n1 - log2k1 + LB)) + ((long long)(k1 >> log2k1) << LB);
    };
    const StageRegs<LB, false> regs(tw, NST > 2 ? t : tq, tq);
    const int k1 = tile * P::CP + rq;
    const float2 ws = __ldg(tw + 2 * M + k1 + ((long long)tq << log2n1));
    wait();
    cpair v[16];
    {
        const float2* src = row(tile * P::CP + rp) + t;
        const float2* src1 = row(mirror(tile * P::CP + rp)) + t;
#pragma unroll
        for (int m = 0; m < 16; ++m) v[m] = make_pair2(__ldcs(src + m * T), __ldcs(src1 + m * T));
        PairView<1, true> view{smem + rp * P::RS};
        static_for<0, NST - 1>([&](auto sc) {
            constexpr int st = decltype(sc)::value;
            stage_compute<LB, 4, S::lrs(st), S::lns(st), false>(v, t, regs);
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
        const int r = tile * P::CP + l / (2 * LINES);
        const char* line = (const char*)row(l / LINES & 1 ? mirror(r) : r);
        asm volatile("discard.global.L2 [%0], 128;" ::"l"(line + 128 * (l % LINES)) : "memory");
    }
    const PairView<1, true> image{smem + rq * P::RS};
    stage_read<LB, 4>(v, tq, image);
    constexpr int LRS = S::lrs(NST - 1), LNS = S::lns(NST - 1);
    stage_compute<LB, 4, LRS, LNS, false>(v, tq, regs);
    // v[m] = rows k1 and N1 - k1 at k2 = tq + m T
    if (tile == 0) {
        __syncthreads();
        if (rq == 0) {
#pragma unroll
            for (int m = 0; m < 16; ++m) image.st(tq + m * T, v[m]);
        }
        __syncthreads();
    }
    const long long step = (long long)T << log2n1;
    float2* up = out + k1 + ((long long)tq << log2n1);
    if (tile == 0 && rq == 0) {
        const float2 wrow = __ldg(tw + 2 * M + n1 / 2);
#pragma unroll 4
        for (int m = 0; m < 16; ++m) {
            const int k2 = tq + m * T;
            const cpair z = image.ld(k2);
            const float2 w = __ldg(tw + 2 * N2 + k2);                       // W_2M^(N1 k2)
            const float2 a = lane0(z), b = lane1(z);
            __stcs(up + m * step, real_split(a, lane0(image.ld((N2 - k2) & (N2 - 1))), w));
            if (k2 == 0) out[M] = real_split(a, a, make_float2(-w.x, w.y));
            __stcs(up + m * step + n1 / 2, real_split(b, lane1(image.ld(N2 - 1 - k2)), cmul(w, wrow)));
        }
        return;
    }
    float2* down = out + M - k1 - ((long long)tq << log2n1);
    static_for<0, 16>([&](auto mc) {
        constexpr int m = decltype(mc)::value;
        const float2 w = rot32_exact<m>(ws), a = lane0(v[m]), b = lane1(v[m]);
        const float sx = a.x + b.x, sy = a.y + b.y, dx = a.x - b.x, dy = a.y - b.y;
        const float cx = fmaf(-w.y, dx, -w.x * dy), cy = fmaf(w.x, dx, -w.y * dy);
        __stcs(up + m * step, make_float2(sx - cx, sy - cy));
        __stcs(down - m * step, make_float2(sx + cx, -(sy + cy)));
    });
}

}  // namespace ckg
