// fft_columns.cu -- transforms down the columns of a matrix: element p of
// transform f at in[p * in_stride + f], result bin k at out[k * out_stride + f]
// (distance 1 on both sides: matrix columns, interleaved channels).
//
// A thread carries two neighbouring columns in packed FP32 arithmetic
// (fft_pair.cuh): 16-byte loads and stores of whole row segments straight
// between HBM and registers, stage exchanges in a tile of C columns side by
// side, twiddles loaded once for both columns and before the data.  The row
// kernels of fft_inter.cu, which serve one-sided layouts and the other sizes,
// stage every value in shared memory on the way in and out and run one column
// a thread.  Real transforms read two neighbouring reals as one register pair
// (no shuffling at all) and write both bins of a split pair for two columns.
//
// Same stages and rounding as the batched kernels, so the same bits: the sizes
// with 16 values a thread there (complex 2^8 .. 2^12, real 2^9 .. 2^13).
//
// What bounds it: the row segments -- 16 columns a row at 2^9 run at 0.83 of the
// HBM copy rate, 8 at 2^10 at 0.69, 4 at 2^12 at 0.48, all of them transforms a
// stride apart.  Measured on GB300 (GB/s, kernels of fft_inter.cu -> here):
// complex 2^8 x 65536 4620 -> 6140, 2^9 x 30000 3600 -> 5640, 2^10 x 65536 3160
// -> 4650, 2^11 x 16384 2900 -> 3810, 2^12 x 16384 2250 -> 3250; real forward 2^11
// x 20000 1330 -> 3610, inverse 1440 -> 3650.
#include "fft_pair_passes.cuh"
#include "fft_small.cuh"

namespace ckg {

template <int L>
struct ColsCfg {
    static_assert(default_log2r(L) == 4, "the batched kernels' stages");
    static constexpr int T = (1 << L) / 16;
    // pairs a tile: rows of 128 bytes up to 2^9, of 64 at 2^10 (two CTAs an SM:
    // 1024 x 65536 231 us, 265 with 128 bytes and one CTA), 2^11 (one CTA an SM;
    // 32 bytes and two CTAs tie for complex data, real n = 2^12 x 16384 inverse
    // 251 against 177 us), of 32 at 2^12
    static constexpr int CP = L <= 9 ? 8 : L <= 11 ? 4 : 2;
    static constexpr int C = 2 * CP, THREADS = T * CP;
    using View = PairView<CP, (CP < 8)>;
    static constexpr size_t SMEM = sizeof(cpair) * (size_t)CP * (CP < 8 ? padded_len(1 << L) : (1 << L));
    static constexpr int MINB = 65536 / (THREADS * 128);
};

// Two neighbouring values of a row whose start is not aligned for a pair (an odd
// number of columns, a base off by one), or with the second (or both) past the
// last column.  Cached loads: the second finds the first one's sector; not the
// read-only path, since the kernel ahead may still write the data when this one
// starts (pdl_wait).
// (Aligned pairs shifted by one value through the neighbouring lane moved fewer
// bytes but serialised the loads: complex 2^9 x 30001 65 -> 146 us.)
__device__ __forceinline__ cpair cols_ld(const float2* p, int live)
{
    const float2 a = live > 0 ? __ldca(p) : make_float2(0.f, 0.f);
    const float2 b = live > 1 ? __ldca(p + 1) : make_float2(0.f, 0.f);
    return make_pair2(a, b);
}
__device__ __forceinline__ void cols_st(float2* p, cpair v, int live)
{
    if (live > 0) __stcs(p, lane0(v));
    if (live > 1) __stcs(p + 1, lane1(v));
}
// The same for neighbouring reals.
__device__ __forceinline__ f32x2 cols_ld(const float* p, int live)
{
    return pack2(live > 0 ? __ldca(p) : 0.f, live > 1 ? __ldca(p + 1) : 0.f);
}
__device__ __forceinline__ void cols_st(float* p, f32x2 v, int live)
{
    const float2 a = unpack2(v);
    if (live > 0) __stcs(p, a.x);
    if (live > 1) __stcs(p + 1, a.y);
}
__device__ __forceinline__ f32x2 cols_ld8(const float* p)
{
    const float2 a = __ldcs(reinterpret_cast<const float2*>(p));
    return pack2(a.x, a.y);
}

// The thread's columns: pair cp of the CTA's tile, first column f0 + 2 cp.
template <class C>
struct ColsPos {
    int cp, t, live;                    // live: how many of the two columns exist
    long long f;
    bool whole;                         // every column of the tile exists
    __device__ __forceinline__ explicit ColsPos(long long count)
    {
        cp = threadIdx.x % C::CP;
        t = threadIdx.x / C::CP;
        const long long f0 = (long long)blockIdx.x * C::C;
        f = f0 + 2 * cp;
        whole = f0 + C::C <= count;
        const long long left = count - f;
        live = left >= 2 ? 2 : left > 0 ? (int)left : 0;
    }
};

template <int L, bool INV>
__global__ void __launch_bounds__(ColsCfg<L>::THREADS, ColsCfg<L>::MINB)
k_c2c_columns(const float2* __restrict__ in, float2* __restrict__ out, long long count, long long is, long long os,
              const float2* __restrict__ tw)
{
    using C = ColsCfg<L>;
    extern __shared__ __align__(128) cpair tile[];
    const ColsPos<C> q(count);
    const StageRegs<L, INV> regs(tw, q.t, q.t);
    pdl_wait_then_launch();
    const float2* src = in + q.f + q.t * is;
    const long long step = C::T * is;
    cpair v[16];
    if (q.whole && (((uintptr_t)in | (is << 3)) & 15) == 0) {
#pragma unroll
        for (int m = 0; m < 16; ++m) v[m] = make_pair2(__ldcs(reinterpret_cast<const float4*>(src + m * step)));
    } else {
#pragma unroll
        for (int m = 0; m < 16; ++m) v[m] = cols_ld(src + m * step, q.live);
    }
    stockham<L, 4, INV, false>(v, q.t, regs, typename C::View{tile + q.cp}, [] { __syncthreads(); }, [] {}, [] {});
    float2* dst = out + q.f + q.t * os;
    const long long ostep = C::T * os;
    if (q.whole && (((uintptr_t)out | (os << 3)) & 15) == 0) {
#pragma unroll
        for (int m = 0; m < 16; ++m) __stcs(reinterpret_cast<float4*>(dst + m * ostep), interleave(v[m]));
    } else {
#pragma unroll
        for (int m = 0; m < 16; ++m) cols_st(dst + m * ostep, v[m], q.live);
    }
}

// Real forward of 2M reals a column to M + 1 bins a column (split_store of
// fft_small.cuh for two columns).
template <int LM>
__global__ void __launch_bounds__(ColsCfg<LM>::THREADS, ColsCfg<LM>::MINB)
k_r2c_columns(const float* __restrict__ in, float2* __restrict__ out, long long count, long long is, long long os,
              const float2* __restrict__ tw)
{
    using C = ColsCfg<LM>;
    constexpr int M = 1 << LM;
    extern __shared__ __align__(128) cpair tile[];
    const ColsPos<C> q(count);
    const StageRegs<LM, false> regs(tw, q.t, q.t);
    const float2 w0 = __ldg(tw + 2 * M + q.t);
    pdl_wait_then_launch();
    const float* src = in + q.f + 2 * q.t * is;
    const long long step = 2 * C::T * is;
    cpair v[16];
    if (q.whole && (((uintptr_t)in | (is << 2)) & 7) == 0) {
#pragma unroll
        for (int m = 0; m < 16; ++m) v[m] = {cols_ld8(src + m * step), cols_ld8(src + m * step + is)};
    } else if (q.whole && ((uintptr_t)in & 7) == 0) {               // odd stride: the even rows are aligned
#pragma unroll
        for (int m = 0; m < 16; ++m) v[m] = {cols_ld8(src + m * step), cols_ld(src + m * step + is, 2)};
    } else {
#pragma unroll
        for (int m = 0; m < 16; ++m) v[m] = {cols_ld(src + m * step, q.live), cols_ld(src + m * step + is, q.live)};
    }
    const typename C::View view{tile + q.cp};
    stockham<LM, 4, false, false>(v, q.t, regs, view, [] { __syncthreads(); }, [] {}, [] { __syncthreads(); });
#pragma unroll
    for (int m = 0; m < 16; ++m) view.st(q.t + m * C::T, v[m]);
    __syncthreads();
    const bool fast = q.whole && (((uintptr_t)out | (os << 3)) & 15) == 0;
    float2* dst = out + q.f;
    auto put = [&](int k, cpair x) {
        if (fast) __stcs(reinterpret_cast<float4*>(dst + k * os), interleave(x));
        else cols_st(dst + k * os, x, q.live);
    };
    static_for<0, 8>([&](auto mc) {
        constexpr int m = decltype(mc)::value;
        const int k = q.t + m * C::T;
        const cpair z0 = view.ld(k), z1 = view.ld((M - k) & (M - 1));
        const float2 w = rot<32, m, false>(w0);                     // W_2M^k
        const f32x2 sx = add2(z0.x, z1.x), sy = sub2(z0.y, z1.y);
        const f32x2 dx = sub2(z0.x, z1.x), dy = add2(z0.y, z1.y);
        const f32x2 wx = dup2(w.x), wy = dup2(w.y);
        const f32x2 px = fma2(wx, dx, mul2(dup2(-w.y), dy)), py = fma2(wx, dy, mul2(wy, dx));
        put(k, {add2(sx, py), sub2(sy, px)});
        put(M - k, {sub2(sx, py), neg2(add2(sy, px))});
    });
    if (q.t == 0) {
        const cpair z = view.ld(M / 2);                             // X[M/2] = 2 conj Z[M/2]
        put(M / 2, {add2(z.x, z.x), neg2(add2(z.y, z.y))});
    }
}

// Real inverse of M + 1 bins a column to 2M reals a column: the tile's bins are
// staged in its shared memory and every thread merges its own with their
// partners M - k (real_merge of fft_core.cuh for two columns).  Reading both
// operands from memory, as the one-column kernels do, fetched every row
// segment twice: n = 2^11 x 20000 212 against 150 us.
template <int LM>
__global__ void __launch_bounds__(ColsCfg<LM>::THREADS, ColsCfg<LM>::MINB)
k_c2r_columns(const float2* __restrict__ in, float* __restrict__ out, long long count, long long is, long long os,
              const float2* __restrict__ tw)
{
    using C = ColsCfg<LM>;
    constexpr int M = 1 << LM;
    extern __shared__ __align__(128) cpair tile[];
    const ColsPos<C> q(count);
    const StageRegs<LM, true> regs(tw, q.t, q.t);
    const float2 w0 = __ldg(tw + 2 * M + q.t);
    pdl_wait_then_launch();
    const float2* src = in + q.f;
    cpair v[16], last = {0, 0};                                     // last: X[M], the partner of X[0]
    if (q.whole && (((uintptr_t)in | (is << 3)) & 15) == 0) {
#pragma unroll
        for (int m = 0; m < 16; ++m)
            v[m] = make_pair2(__ldcs(reinterpret_cast<const float4*>(src + (q.t + m * C::T) * is)));
    } else {
#pragma unroll
        for (int m = 0; m < 16; ++m) v[m] = cols_ld(src + (q.t + m * C::T) * is, q.live);
    }
    if (q.t == 0) last = cols_ld(src + M * is, q.live);
    const typename C::View view{tile + q.cp};
#pragma unroll
    for (int m = 0; m < 16; ++m) view.st(q.t + m * C::T, v[m]);
    __syncthreads();
    static_for<0, 16>([&](auto mc) {
        constexpr int m = decltype(mc)::value;
        const int k = q.t + m * C::T;
        const cpair z0 = v[m];
        cpair z1 = view.ld((M - k) & (M - 1));
        if (m == 0 && q.t == 0) z1 = last;
        const float2 w = rot<32, m, false>(w0);                     // W_2M^k
        const f32x2 sx = add2(z0.x, z1.x), sy = sub2(z0.y, z1.y);
        const f32x2 dx = sub2(z0.x, z1.x), dy = add2(z0.y, z1.y);
        const f32x2 wx = dup2(w.x), wy = dup2(w.y);
        v[m] = {add2(sx, fma2(wy, dx, neg2(mul2(wx, dy)))), add2(sy, fma2(wx, dx, mul2(wy, dy)))};
    });
    __syncthreads();
    stockham<LM, 4, true, false>(v, q.t, regs, view, [] { __syncthreads(); }, [] {}, [] {});
    float* dst = out + q.f + 2 * q.t * os;
    const long long step = 2 * C::T * os;
    if (q.whole && (((uintptr_t)out | (os << 2)) & 7) == 0) {
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            __stcs(reinterpret_cast<float2*>(dst + m * step), unpack2(v[m].x));
            __stcs(reinterpret_cast<float2*>(dst + m * step + os), unpack2(v[m].y));
        }
    } else if (q.whole && ((uintptr_t)out & 7) == 0) {              // odd stride: the even rows are aligned
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            __stcs(reinterpret_cast<float2*>(dst + m * step), unpack2(v[m].x));
            cols_st(dst + m * step + os, v[m].y, 2);
        }
    } else {
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            cols_st(dst + m * step, v[m].x, q.live);
            cols_st(dst + m * step + os, v[m].y, q.live);
        }
    }
}

// ---------------------------------------------------------------- launch

template <int L>
static cudaError_t launch_columns_L(Kind kind, const void* in, void* out, long long count, long long is, long long os,
                                    const float2* tw, cudaStream_t s)
{
    using C = ColsCfg<L>;
    const dim3 grid((unsigned)((count + C::C - 1) / C::C)), block(C::THREADS);
    const float2* ci = (const float2*)in;
    float2* co = (float2*)out;
    switch (kind) {
    case C2C_FWD: return launch_pdl(k_c2c_columns<L, false>, grid, block, C::SMEM, s, ci, co, count, is, os, tw);
    case C2C_INV: return launch_pdl(k_c2c_columns<L, true>, grid, block, C::SMEM, s, ci, co, count, is, os, tw);
    case R2C: return launch_pdl(k_r2c_columns<L>, grid, block, C::SMEM, s, (const float*)in, co, count, is, os, tw);
    case C2R: return launch_pdl(k_c2r_columns<L>, grid, block, C::SMEM, s, ci, (float*)out, count, is, os, tw);
    }
    return cudaErrorInvalidValue;
}

// log2n: of the transform (real: of n reals).  Rows that do not start aligned
// (an odd stride, a base off by a value) cost two accesses a pair: still ahead
// of the staged rows of fft_inter.cu from 2^9 (complex 2^9 x 30001 74 -> 71 us,
// 2^10 x 65535 369 -> 305; real inverse 2^10 x 30001 99 -> 94), behind them at 2^8
// (complex x 65533 60 -> 63 us, real inverse 2^9 x 40001 53 -> 68).
bool columns_apply(Kind kind, int log2n, const void* in, const void* out, long long in_stride, long long out_stride)
{
    const int l = kind == R2C || kind == C2R ? log2n - 1 : log2n;
    const uintptr_t a = (uintptr_t)in | (uintptr_t)(in_stride << (kind == R2C ? 2 : 3));
    const uintptr_t b = (uintptr_t)out | (uintptr_t)(out_stride << (kind == C2R ? 2 : 3));
    const bool aligned = (a & (kind == R2C ? 7 : 15)) == 0 && (b & (kind == C2R ? 7 : 15)) == 0;
    return l >= (aligned ? 8 : 9) && l <= 12;
}

cudaError_t launch_columns(Kind kind, int log2n, const void* in, void* out, long long count, long long in_stride,
                           long long out_stride, const float2* tw, cudaStream_t s)
{
    if (count <= 0) return cudaSuccess;
    cudaError_t e = cudaErrorInvalidValue;
    switch (kind == R2C || kind == C2R ? log2n - 1 : log2n) {
    case 8: e = launch_columns_L<8>(kind, in, out, count, in_stride, out_stride, tw, s); break;
    case 9: e = launch_columns_L<9>(kind, in, out, count, in_stride, out_stride, tw, s); break;
    case 10: e = launch_columns_L<10>(kind, in, out, count, in_stride, out_stride, tw, s); break;
    case 11: e = launch_columns_L<11>(kind, in, out, count, in_stride, out_stride, tw, s); break;
    case 12: e = launch_columns_L<12>(kind, in, out, count, in_stride, out_stride, tw, s); break;
    default: break;
    }
    if (e == cudaSuccess) count_launch();
    return e;
}

template <int L>
static cudaError_t attr_columns()
{
    const int smem = (int)ColsCfg<L>::SMEM;
    const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(k_c2c_columns<L, false>, a, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_c2c_columns<L, true>, a, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_r2c_columns<L>, a, smem);
    return e == cudaSuccess ? cudaFuncSetAttribute(k_c2r_columns<L>, a, smem) : e;
}

cudaError_t prepare_columns()
{
    cudaError_t e = attr_columns<9>();
    if (e == cudaSuccess) e = attr_columns<10>();
    if (e == cudaSuccess) e = attr_columns<11>();
    return e == cudaSuccess ? attr_columns<12>() : e;
}

}  // namespace ckg
