// gpufft-b200: contiguous passes of the drop-in transforms on tiles of 2^LT points
// (TileOf, gf_tile.cuh) with the caller's tables.
//
// The pass runs the last LT forward (first LT inverse) stages of every 2^LT-point
// tile. Tables come from the caller, so nothing links a table's odd entries to its
// even ones or the inverse table to the forward one: every twiddle of the tile is
// staged in shared memory, thread-major for the innermost round (straight from the
// table, a warp's loads of that round touch 340 sectors per 16 points in FP64, as
// many shared-memory cycles as the data's whole way through the pass). The tile's
// index T selects its twiddles, so the CTAs are persistent, each with a run of
// (T, row) pairs in T-major order: the twiddles are staged once for many rows.
// While a tile is transformed the next one's loads are in flight; for products, whose
// two operands of two tiles do not fit the registers, the next tile's rows are asked
// for in L2 (FFNT product FP64, N = 2^16, batch 256: 360 -> 354 us).
//
// FP64 forward tiles leave through the TMA unit: after its last round a thread holds
// 16 consecutive points, writes them to its own 256 bytes of the padded buffer and
// starts one bulk copy of them, instead of a last transpose and 16 coalesced stores.
//
// One complex row per tile and m = LT: the load may be the fold with the twist, a
// real row or a zero-padded one, the store the unfold, a real row or a scaled one
// (the variants of pass_body).
#pragma once

#include "gf_tile.cuh"

namespace gfb
{

template <int LT> struct TilePass : TileOf<LT>
{
    using B = TileOf<LT>;
    static constexpr int R = B::R, HT = B::HT, W1 = B::W1, W2 = B::W2, HI0 = B::HI0;
    static constexpr int S0 = HT + 1;
    static constexpr int N0 = HI0 == 4 ? 15 : 14; // twiddles per thread of the innermost round
    static constexpr int S2 = 17;
    static constexpr int TWN = N0 * S0 + 16 * S2 + 16;
    template <typename C> static __device__ __forceinline__ C* outer(C* tw) { return tw + N0 * S0 + 16 * S2; }
    template <typename C> static __device__ __forceinline__ C* middle(C* tw, int i) { return tw + N0 * S0 + i * S2; }
    // position nt + h of thread i's twiddle h of the stage with nt twiddles
    template <typename C> static __device__ __forceinline__ C* inner(C* tw, int i) { return tw + (N0 - 16) * S0 + i; }

    // All twiddles of tile T: stage u of the tile uses table[neg 2^(s0+u) + (T << u)
    // + nt i + h], h < nt, at position nt + h of index i.
    template <typename C>
    static __device__ __forceinline__ void stage(C* tw, const C* __restrict__ tab, long long T, int s0, int neg, int t)
    {
        auto base = [&](int u) { return tab + (T << u) + (neg ? 1LL << (s0 + u) : 0LL); };
#pragma unroll
        for (int k = 0; k < N0; k++)
        {
            // linear entry p of the stage with nt = 2^lg twiddles per thread
            const int q = k + (16 - N0); // 1 + 2 + 4 + 8 arrays of HT entries
            const int lg = q >= 8 ? 3 : q >= 4 ? 2 : q >= 2 ? 1 : 0;
            const int p = (q - (1 << lg)) * HT + t;
            inner(tw, p >> lg)[((1 << lg) + (p & ((1 << lg) - 1))) * S0] = __ldg(base(LT - 4 + lg) + p);
        }
#pragma unroll
        for (int k = 0; k < 256 / HT; k++)
        {
            const int p = k * HT + t, i = p >> 4, pos = p & 15;
            if (pos)
            {
                const int lg = 31 - __clz(pos);
                middle(tw, i)[pos] = __ldg(base(4 + lg) + (i << lg) + (pos - (1 << lg)));
            }
        }
        if (t > 0 && t < 16)
        {
            const int lg = 31 - __clz(t);
            outer(tw)[t] = __ldg(base(lg) + (t - (1 << lg)));
        }
    }

    template <typename T, bool FWD, int HI>
    static __device__ __forceinline__ void round(cx<T> (&x)[R], const cx<T>* tw, int st)
    {
#pragma unroll
        for (int k = 0; k < HI; k++)
        {
            const int pb = FWD ? HI - 1 - k : k;
            const int nt = 1 << (3 - pb);
            cx<T> w[8];
#pragma unroll
            for (int h = 0; h < 8; h++)
                if (h < nt) w[h] = tw[(nt + h) * st];
#pragma unroll
            for (int r = 0; r < R; r++)
            {
                if (r & (1 << pb)) continue;
                if (FWD)
                    ct_bfly<T>(x[r], x[r | (1 << pb)], w[r >> (pb + 1)]);
                else
                    gs_bfly<T>(x[r], x[r | (1 << pb)], w[r >> (pb + 1)]);
            }
        }
    }
    template <typename T> static __device__ __forceinline__ void forward(cx<T> (&x)[R], cx<T>* sm, cx<T>* tw, int t)
    {
        round<T, true, 4>(x, outer(tw), 1);
        B::template put<W1>(x, sm, t);
        __syncthreads();
        B::template get<W2>(x, sm, t);
        round<T, true, 4>(x, middle(tw, t >> W2), 1);
        B::template put<W2>(x, sm, t);
        __syncthreads();
        B::template get<0>(x, sm, t);
        round<T, true, HI0>(x, inner(tw, t), S0);
        B::template put<0>(x, sm, t); // the positions this thread read
    }
    template <typename T> static __device__ __forceinline__ void inverse(cx<T> (&x)[R], cx<T>* sm, cx<T>* tw, int t)
    {
        // coalesced loads in window W1, moved to window 0
        B::template put<W1>(x, sm, t);
        __syncthreads();
        B::template get<0>(x, sm, t);
        round<T, false, HI0>(x, inner(tw, t), S0);
        B::template put<0>(x, sm, t);
        __syncthreads();
        B::template get<W2>(x, sm, t);
        round<T, false, 4>(x, middle(tw, t >> W2), 1);
        B::template put<W2>(x, sm, t);
        __syncthreads();
        B::template get<W1>(x, sm, t);
        round<T, false, 4>(x, outer(tw), 1);
    }
};

// CTAs per SM. Shared memory per CTA: 68 / 136 KB in FP64 (LT = 11 / 12), 34 / 69 KB
// in FP32. (Two tiles to a CTA, sharing the twiddles with a warp group each, made 16
// warps per SM of the 12 at LT = 11 in FP64, but left no registers for the next
// tile's loads: no faster on long runs, 25 % slower on one-pass rows.)
template <typename T, int LT> constexpr int tile_pass_blocks()
{
    if (sizeof(T) == 8) return LT == 11 ? 3 : 1;
    return LT == 11 ? 5 : 3;
}

// Row b's tile g (2^LT points, a whole row where m = LT) in window W1.
template <typename T, int LT, int IK>
__device__ __forceinline__ void tile_load(const PassArgs<T>& a, cx<T> (&x)[16], long long g, long long b, int t)
{
    constexpr int R = 16, HT = TilePass<LT>::HT;
    const long long M = 1LL << a.geo.m;
    if constexpr (IK == IN_FOLD)
    {
        const T* p = reinterpret_cast<const T*>(a.in) + b * 2 * M + t;
#pragma unroll
        for (int r = 0; r < R; r++) x[r] = mk<T>(ld_stream(p + r * HT), ld_stream(p + M + r * HT));
    }
    else if constexpr (IK == IN_REAL)
    {
        // a zero-padded row is one tile: its upper half is the registers' upper half
        const T* p = reinterpret_cast<const T*>(a.in) + b * M + t;
#pragma unroll
        for (int r = 0; r < R / 2; r++) x[r] = mk<T>(p[r * HT], T(0));
#pragma unroll
        for (int r = R / 2; r < R; r++) x[r] = mk<T>(T(0), T(0));
        if (!a.zero_pad)
        {
#pragma unroll
            for (int r = R / 2; r < R; r++) x[r].x = p[r * HT];
        }
    }
    else
    {
        const cx<T>* p = reinterpret_cast<const cx<T>*>(a.in) + b * M + (g << LT) + t;
#pragma unroll
        for (int r = 0; r < R; r++) x[r] = p[r * HT];
        if constexpr (IK == IN_PROD)
        {
#pragma unroll
            for (int r = 0; r < R; r++) x[r] = cmul<T>(x[r], p[a.prod_off + r * HT]);
        }
    }
}

template <typename T, bool FWD, int LT, int IK, int OK>
__global__ void __launch_bounds__(TilePass<LT>::HT, tile_pass_blocks<T, LT>())
    tile_pass_kernel(const PassArgs<T> a)
{
    pdl_begin(); // before any global-memory access (programmatic launch)
    using tl = TilePass<LT>;
    constexpr int R = tl::R, HT = tl::HT;
    constexpr bool AHEAD = IK != IN_PROD;
    constexpr bool BULK = FWD && sizeof(T) == 8;        // rows of 16 points on 16-byte boundaries
    extern __shared__ __align__(16) unsigned char smraw[];
    cx<T>* sm = reinterpret_cast<cx<T>*>(smraw);
    cx<T>* tw = sm + tl::SLOT;
    const int t = threadIdx.x;
    const int m = a.geo.m, s0 = m - LT;
    const long long M = 1LL << m;
    const long long units = a.batch << s0; // (T, row), T-major
    const long long u0 = (long long)blockIdx.x * units / gridDim.x, u1 = (long long)(blockIdx.x + 1) * units / gridDim.x;
    long long g = u0 / a.batch, row = u0 - g * a.batch, staged = -1;
    cx<T> nx[AHEAD ? 16 : 1];
    if constexpr (AHEAD)
    {
        if (u0 < u1) tile_load<T, LT, IK>(a, nx, g, row, t);
    }
    for (long long u = u0; u < u1; u++)
    {
        if (g != staged)
        {
            __syncthreads(); // the old twiddles are used
            tl::stage(tw, a.table, g, s0, a.geo.neg, t);
            staged = g; // visible after the barrier below
        }
        const long long gc = g, b = row;
        if (++row == a.batch)
        {
            row = 0;
            g++;
        }
        cx<T> x[16];
        if constexpr (AHEAD)
        {
#pragma unroll
            for (int r = 0; r < R; r++) x[r] = nx[r];
            if (u + 1 < u1) tile_load<T, LT, IK>(a, nx, g, row, t);
        }
        else
        {
            if (t == 0 && u + 1 < u1)
            {
                const cx<T>* p = reinterpret_cast<const cx<T>*>(a.in) + row * M + (g << LT);
                prefetch_l2(p, tl::P * sizeof(cx<T>));
                prefetch_l2(p + a.prod_off, tl::P * sizeof(cx<T>));
            }
            tile_load<T, LT, IK>(a, x, gc, b, t);
        }
        if constexpr (IK == IN_FOLD)
        {
#pragma unroll
            for (int r = 0; r < R; r++) x[r] = cmul<T>(x[r], ldg<T>(a.twist + t + r * HT));
        }
        // the buffer is free: this thread's bulk copy out of it, then everyone's (and
        // their reads of the last transpose), is done
        if constexpr (BULK) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        __syncthreads();
        if (FWD)
            tl::template forward<T>(x, sm, tw, t);
        else
            tl::template inverse<T>(x, sm, tw, t);
        if constexpr (BULK)
        {
            cx<T>* dst = reinterpret_cast<cx<T>*>(a.out) + b * M + (gc << LT) + 16 * t;
            const unsigned src = static_cast<unsigned>(__cvta_generic_to_shared(sm + tl::ppos(16 * t)));
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], 256;" ::"l"(dst), "r"(src) : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            continue;
        }
        if constexpr (FWD)
        {
            // back to window W1, where the stores are coalesced
            __syncthreads();
            tl::template get<tl::W1>(x, sm, t);
        }
        if constexpr (OK == OUT_UNFOLD)
        {
            T* p = reinterpret_cast<T*>(a.out) + b * 2 * M + t;
#pragma unroll
            for (int r = 0; r < R; r++)
            {
                const cx<T> v = cmul<T>(cmul<T>(x[r], a.scale), ldg<T>(a.twist + t + r * HT));
                st_stream(p + r * HT, v.x);
                st_stream(p + M + r * HT, v.y);
            }
        }
        else if constexpr (OK == OUT_REAL)
        {
            T* p = reinterpret_cast<T*>(a.out) + b * M + t;
#pragma unroll
            for (int r = 0; r < R; r++) p[r * HT] = (a.do_scale ? cmul<T>(x[r], a.scale) : x[r]).x;
        }
        else
        {
            cx<T>* p = reinterpret_cast<cx<T>*>(a.out) + b * M + (gc << LT) + t;
#pragma unroll
            for (int r = 0; r < R; r++) p[r * HT] = a.do_scale ? cmul<T>(x[r], a.scale) : x[r];
        }
    }
    if constexpr (BULK) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); // the copies read this CTA's memory
}

} // namespace gfb
