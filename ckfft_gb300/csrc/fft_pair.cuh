// fft_pair.cuh -- two transforms per thread in packed FP32 arithmetic.
//
// sm_100+ has FP32 instructions on register pairs (add / sub / mul / fma
// .rn.f32x2).  They do not raise the FP32 rate -- 128 lanes a cycle and SM
// either way, measured 32 T element operations a second for scalar and packed
// FMA alike -- but a packed instruction takes one issue slot for two results.
// The multi-pass kernels issue 42 to 85 instructions per value, half of them
// FP32, and ran at 50-67 % of the issue rate with HBM half idle; so here a
// thread carries TWO neighbouring columns (or rows) of a tile, real parts of
// both in one register pair and imaginary parts in another.  Every butterfly
// is then packed without any shuffling, both columns share their stage
// twiddles (loads and power products once instead of twice), and shared
// memory and HBM are accessed 16 bytes at a time.
//
// Each lane rounds exactly as the one-value code of fft_core.cuh: same
// operations, same order, so both forms of a transform give the same bits.
#pragma once
#include "fft_core.cuh"

namespace ckg {

using f32x2 = unsigned long long;

__device__ __forceinline__ f32x2 pack2(float lo, float hi)
{
    f32x2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ float2 unpack2(f32x2 v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 dup2(float a) { return pack2(a, a); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b)
{
    f32x2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b)
{
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 neg2(f32x2 a) { return a ^ 0x8000000080000000ull; }

// Two complex values: real parts in x, imaginary parts in y (lane 0 low).
struct __align__(16) cpair {
    f32x2 x, y;
};

__device__ __forceinline__ cpair make_pair2(float2 a, float2 b) { return {pack2(a.x, b.x), pack2(a.y, b.y)}; }
__device__ __forceinline__ cpair make_pair2(float4 ab) { return {pack2(ab.x, ab.z), pack2(ab.y, ab.w)}; }
__device__ __forceinline__ float2 lane0(cpair v) { return make_float2(unpack2(v.x).x, unpack2(v.y).x); }
__device__ __forceinline__ float2 lane1(cpair v) { return make_float2(unpack2(v.x).y, unpack2(v.y).y); }
// (re 0, im 0, re 1, im 1): the two values as neighbours in memory
__device__ __forceinline__ float4 interleave(cpair v)
{
    const float2 a = unpack2(v.x), b = unpack2(v.y);
    return make_float4(a.x, b.x, a.y, b.y);
}

__device__ __forceinline__ cpair cadd(cpair a, cpair b) { return {add2(a.x, b.x), add2(a.y, b.y)}; }
__device__ __forceinline__ cpair csub(cpair a, cpair b) { return {sub2(a.x, b.x), sub2(a.y, b.y)}; }
__device__ __forceinline__ cpair cadd_i(cpair a, cpair b) { return {sub2(a.x, b.y), add2(a.y, b.x)}; }
__device__ __forceinline__ cpair csub_i(cpair a, cpair b) { return {add2(a.x, b.y), sub2(a.y, b.x)}; }
__device__ __forceinline__ cpair conj2(cpair a) { return {a.x, neg2(a.y)}; }
// lane-wise product, and the product with one value for both lanes
__device__ __forceinline__ cpair cmul(cpair a, cpair w)
{
    return {fma2(a.x, w.x, neg2(mul2(a.y, w.y))), fma2(a.x, w.y, mul2(a.y, w.x))};
}
__device__ __forceinline__ cpair cmul(cpair a, float2 w)
{
    const f32x2 wx = dup2(w.x), wy = dup2(w.y);
    return {fma2(a.x, wx, mul2(a.y, dup2(-w.y))), fma2(a.x, wy, mul2(a.y, wx))};
}

// rot<R, K, INV> of fft_core.cuh on both lanes.
template <int R, int K, bool INV>
__device__ __forceinline__ cpair rot(cpair a)
{
    constexpr int m = ((K * (32 / R)) % 32 + 32) % 32;
    if constexpr (m == 0) {
        return a;
    } else if constexpr (m == 16) {
        return {neg2(a.x), neg2(a.y)};
    } else if constexpr (m == 8) {
        if constexpr (INV) return {neg2(a.y), a.x};
        else return {a.y, neg2(a.x)};
    } else if constexpr (m == 24) {
        if constexpr (INV) return {a.y, neg2(a.x)};
        else return {neg2(a.y), a.x};
    } else if constexpr (m % 8 == 4) {
        constexpr float c = (float)cos32(m);
        constexpr float s = INV ? (float)sin32(m) : -(float)sin32(m);
        constexpr bool same = (s > 0.f) == (c > 0.f);
        const f32x2 c2 = dup2(c);
        if constexpr (same) return {mul2(c2, sub2(a.x, a.y)), mul2(c2, add2(a.x, a.y))};
        else return {mul2(c2, add2(a.x, a.y)), mul2(c2, sub2(a.y, a.x))};
    } else {
        constexpr float c = (float)cos32(m);
        constexpr float s = INV ? (float)sin32(m) : -(float)sin32(m);
        const f32x2 c2 = dup2(c);
        return {fma2(a.x, c2, mul2(a.y, dup2(-s))), fma2(a.x, dup2(s), mul2(a.y, c2))};
    }
}

// ------------------------------------------------------------ shared memory
// Position pos of the transform pair a view belongs to, at
// base[(PAD ? pos + pos / 16 : pos) * MUL]: a tile of MUL pairs side by side
// (MUL >= 8: eight neighbouring lanes cover 128 bytes, no padding needed), or
// one pair's own padded image (MUL = 1).  Stage positions are one base slot
// plus compile-time offsets.
template <int MUL, bool PAD>
struct PairView {
    cpair* base;
    __device__ __forceinline__ static constexpr int slot(int pos) { return (PAD ? pos + (pos >> 4) : pos) * MUL; }
    // slot(pos + d) - slot(pos) for pos a multiple of 16 or d a multiple of 16
    __device__ __forceinline__ static constexpr int step(int d) { return (PAD ? d + (d >> 4) : d) * MUL; }
    __device__ __forceinline__ void st(int pos, cpair v) const { base[slot(pos)] = v; }
    __device__ __forceinline__ cpair ld(int pos) const { return base[slot(pos)]; }
};

// Where a stage's table twiddles come from: element k of level 2^q (W_{2^q}^k,
// conjugated for the inverse), for the thread's butterfly u.  StageTable: a copy of the levels a transform
// of 2^LS points (16 values a thread) uses, in shared memory, so that no
// stage waits for L2.
template <int LS, bool INV>
struct StageTable {
    static constexpr int kLast = LS == 9 ? 256 : LS == 10 ? 512 : 0;     // third stage: span 256
    static constexpr int kEntries = 64 + kLast;
    const float2* s;
    template <int LEVEL>
    __device__ __forceinline__ static int at(int k)
    {
        if constexpr (LEVEL <= 256) return (ilog2(LEVEL) - 5) * 16 + k;    // 32 .. 256, k < 16
        else if constexpr (LEVEL == 1024) return 64 + k;                   // k < 256
        else return 64 + (LS == 10 ? 256 : 0) + k;                         // 512
    }
    template <int LEVEL, int U>
    __device__ __forceinline__ float2 get(int k) const { return s[at<LEVEL>(k)]; }
    // fills the copy from the table of all levels, by threads tid of `threads`
    __device__ static void fill(float2* d, const float2* __restrict__ tw, int tid, int threads)
    {
        auto level = [&](auto lc, int n) {
            constexpr int LEVEL = decltype(lc)::value;
            for (int k = tid; k < n; k += threads) d[at<LEVEL>(k)] = tw_load<INV>(tw + LEVEL, k);
        };
        level(std::integral_constant<int, 32>{}, 16);
        level(std::integral_constant<int, 64>{}, 16);
        level(std::integral_constant<int, 128>{}, 16);
        level(std::integral_constant<int, 256>{}, 16);
        if constexpr (LS >= 9) level(std::integral_constant<int, 512>{}, 256);
        if constexpr (LS == 10) level(std::integral_constant<int, 1024>{}, 256);
    }
};

// The same twiddles of one thread in registers, for a kernel that runs each
// stage once a thread: all of them are loaded before the thread's data (and
// before the wait for the previous kernel), so no stage waits for them.
// Second stage (span 16, radix RS2) at thread position t2, third (span 256)
// at t3 (the row passes' last stage runs on other positions).
template <int LS, bool INV>
struct StageRegs {
    using S = Sched<LS, 4>;
    static constexpr int T = (1 << LS) / 16;
    static constexpr int L2 = S::lrs(1), U2 = 16 >> L2;
    static constexpr int L3 = S::nstages > 2 ? S::lrs(2) : 0, U3 = L3 ? 16 >> L3 : 0;
    float2 a[U2 * L2];
    float2 b[U3 ? U3 * L3 : 1];
    __device__ __forceinline__ StageRegs(const float2* __restrict__ tw, int t2, int t3)
    {
#pragma unroll
        for (int u = 0; u < U2; ++u) {
#pragma unroll
            for (int i = 0; i < L2; ++i)
                a[u * L2 + i] = tw_load<INV>(tw + (16 << L2 >> i), (t2 + u * T) & 15);
        }
#pragma unroll
        for (int u = 0; u < U3; ++u) {
#pragma unroll
            for (int i = 0; i < L3; ++i)
                b[u * L3 + i] = tw_load<INV>(tw + (256 << L3 >> i), (t3 + u * T) & 255);
        }
    }
    template <int LEVEL, int U>
    __device__ __forceinline__ float2 get(int) const
    {
        if constexpr (LEVEL <= (16 << L2)) return a[U * L2 + ilog2((16 << L2) / LEVEL)];
        else return b[U * L3 + ilog2((256 << L3) / LEVEL)];
    }
};

// stage_compute of fft_core.cuh on two transforms that share their twiddles.
template <int LOG2N, int LOG2R, int LRS, int LNS, bool INV, class Table>
__device__ __forceinline__ void stage_compute(cpair (&v)[1 << LOG2R], int t, const Table& tab)
{
    constexpr int R = 1 << LOG2R, RS = 1 << LRS, NS = 1 << LNS;
    constexpr int T = (1 << LOG2N) / R;
    constexpr int U = R / RS;
    static_for<0, U>([&](auto uc) {
        constexpr int u = decltype(uc)::value;
        cpair x[RS];
#pragma unroll
        for (int j = 0; j < RS; ++j) x[j] = v[u + j * U];
        if constexpr (NS > 1) {
            const int k = (t + u * T) & (NS - 1);
            float2 w[RS];
            static_for<0, LRS>([&](auto ic) {
                constexpr int p = 1 << decltype(ic)::value;
                w[p] = tab.template get<NS * RS / p, u>(k);
            });
#pragma unroll
            for (int j = 3; j < RS; ++j) {
                if ((j & (j - 1)) == 0) continue;
                const int hb = 1 << (31 - __clz(j));
                w[j] = cmul(w[hb], w[j - hb]);
            }
#pragma unroll
            for (int j = 1; j < RS; ++j) x[j] = cmul(x[j], w[j]);
        }
        dft<RS, INV>(x);
#pragma unroll
        for (int j = 0; j < RS; ++j) v[u + j * U] = x[j];
    });
}

template <int LOG2N, int LOG2R, int LRS, int LNS, class View>
__device__ __forceinline__ void stage_write(const cpair (&v)[1 << LOG2R], int t, const View& view)
{
    constexpr int R = 1 << LOG2R, RS = 1 << LRS, NS = 1 << LNS;
    constexpr int T = (1 << LOG2N) / R;
    constexpr int U = R / RS;
    static_assert((NS == 1 && RS == 16) || NS % 16 == 0, "stage offsets are compile-time constants");
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int b = t + u * T;
        cpair* p = view.base + View::slot(((b >> LNS) << (LNS + LRS)) + (b & (NS - 1)));
#pragma unroll
        for (int j = 0; j < RS; ++j) p[View::step(j * NS)] = v[u + j * U];
    }
}

template <int LOG2N, int LOG2R, class View>
__device__ __forceinline__ void stage_read(cpair (&v)[1 << LOG2R], int t, const View& view)
{
    constexpr int R = 1 << LOG2R;
    constexpr int T = (1 << LOG2N) / R;
    if constexpr (T % 16 == 0) {
        const cpair* q = view.base + View::slot(t);
#pragma unroll
        for (int m = 0; m < R; ++m) v[m] = q[View::step(m * T)];
    } else {
#pragma unroll
        for (int m = 0; m < R; ++m) v[m] = view.ld(t + m * T);
    }
}

// All stages of two length-2^LOG2N transforms held as v[m] = x[t + mT]; on
// return v[m] = X[t + mT].  sync(): barrier of the threads that share the
// view (WARP: they are in one warp).  pre() runs before the first one;
// read_done() follows a thread's last read of the view.
template <int LOG2N, int LOG2R, bool INV, bool WARP, class Table, class View, class Sync, class Pre, class Done>
__device__ __forceinline__ void stockham(cpair (&v)[1 << LOG2R], int t, const Table& tab, const View& view,
                                         Sync&& sync, Pre&& pre, Done&& read_done)
{
    using S = Sched<LOG2N, LOG2R>;
    static_for<0, S::nstages>([&](auto sc) {
        constexpr int s = decltype(sc)::value;
        constexpr int lrs = S::lrs(s), lns = S::lns(s);
        stage_compute<LOG2N, LOG2R, lrs, lns, INV>(v, t, tab);
        if constexpr (s + 1 < S::nstages) {
            stage_write<LOG2N, LOG2R, lrs, lns>(v, t, view);
            if constexpr (s == 0) pre();
            if constexpr (WARP) __syncwarp();
            else sync();
            stage_read<LOG2N, LOG2R>(v, t, view);
            if constexpr (s + 2 < S::nstages) {
                if constexpr (WARP) __syncwarp();
                else sync();
            } else {
                read_done();
            }
        }
    });
}

}  // namespace ckg
