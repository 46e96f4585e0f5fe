// gpufft-b200: whole products of 2^m-point transforms, m = 4 .. 12, in one kernel on
// tiles (TileOf, gf_tile.cuh): 2^(11-m) products to a CTA of 128 threads, one product
// of 4096 points to a CTA of 256.
//
// One operand is transformed and parked in registers, then each other operand is
// transformed, multiplied and transformed back; an operand's loads are in flight
// while the one before it is transformed, the next tile's first operand's while the
// result is. The CTAs are persistent: every tile starts its transforms at group 0, so
// the twiddles are staged once per CTA. The engine's form (256 threads, 16 points of
// both operands per thread) had one CTA per SM in FP64 and two in FP32, whose load,
// transform and store phases did not overlap, and read the innermost twiddles from
// the table at a stride of 128 bytes. Values have its bits.
//
// Measured (B200, the engine's form -> this one): negacyclic N = 2^11, batch 4000:
// FP64 156 -> 64 us (47 % of the HBM rate on operands and result), FP32 78 -> 37;
// N = 2^13, batch 500, FP64 94 -> 49; cyclic 2^10, batch 4000, FP64 99 -> 57; adjoint
// N = 2^12, batch 1000: 231 -> 109 with the forward product.
#pragma once

#include "gf_tile.cuh"

namespace gfb
{

enum SingleKind
{
    SINGLE_NEG = 0, // a, b rows of 2M reals (fold, twist); c rows of 2M reals (scale, untwist, unfold)
    SINGLE_LIN = 1, // a, b rows of M reals (zero-padded operands, twist); c as above
    SINGLE_CYC = 2, // a, b, c rows of M complex (scale)
    SINGLE_VJP = 3  // parked g rows of 2M reals, operands b and a rows of M reals; results rows of M reals
};

template <typename T> struct SingleArgs
{
    const void* park;  // b; g for the adjoint
    const void* op[2]; // a; b and a for the adjoint
    void* out[2];      // c; grad_a and grad_b
    const cx<T>* roots;
    const cx<T>* twist;
    const cx<T>* untwist;
    T scale;
    long long batch;
};

// CTAs per SM: two operands of 16 points, and the next tile's loads on their way, take
// 240 registers in FP64 and 128 in FP32 (three and five CTAs spill 300 and 180 bytes
// a thread).
template <typename T, int m> constexpr int single_blocks()
{
    if (m == 12) return sizeof(T) == 8 ? 1 : 2;
    return sizeof(T) == 8 ? 2 : 4;
}

template <typename T, int m, int KIND>
__global__ void __launch_bounds__(m == 12 ? 256 : 128, single_blocks<T, m>()) single_kernel(const SingleArgs<T> a)
{
    pdl_begin(); // before any global-memory access (programmatic launch)
    using tl = TileOf<m == 12 ? 12 : 11>;
    constexpr int R = tl::R, HT = tl::HT;
    constexpr int M = 1 << m;
    constexpr int NOPS = KIND == SINGLE_VJP ? 2 : 1;
    extern __shared__ __align__(16) unsigned char smraw[];
    cx<T>* sm = reinterpret_cast<cx<T>*>(smraw);
    cx<T>* tw = sm + tl::SLOT;
    const int t = threadIdx.x;
    const long long points = a.batch << m; // of the batch
    const long long tiles = (points + tl::P - 1) / tl::P;
    const long long u0 = (long long)blockIdx.x * tiles / gridDim.x, u1 = (long long)(blockIdx.x + 1) * tiles / gridDim.x;
    // point e = t + r HT of tile u: row (u P + e) / M, position e mod M
    auto pos = [&](int r) { return (t + r * HT) & (M - 1); };
    // rows of 2M reals: the row's start is at twice its first point
    auto fold_at = [&](long long u, int r) { return 2 * (u * tl::P + t + r * HT) - pos(r); };
    auto load = [&](cx<T> (&x)[16], const void* src, long long u, auto fold) {
        const bool whole = (u + 1) * tl::P <= points;
#pragma unroll
        for (int r = 0; r < R; r++)
        {
            const long long e = u * tl::P + t + r * HT;
            const bool ok = whole || e < points;
            if constexpr (KIND == SINGLE_CYC)
            {
                x[r] = ok ? ld_stream(static_cast<const cx<T>*>(src) + e) : mk<T>(T(0), T(0));
            }
            else if constexpr (decltype(fold)::value)
            {
                const T* p = static_cast<const T*>(src) + fold_at(u, r);
                x[r] = mk<T>(ok ? ld_stream(p) : T(0), ok ? ld_stream(p + M) : T(0));
            }
            else
            {
                x[r] = mk<T>(ok ? ld_stream(static_cast<const T*>(src) + e) : T(0), T(0));
            }
        }
    };
    auto twist = [&](cx<T> (&x)[16]) {
        if constexpr (KIND != SINGLE_CYC)
        {
#pragma unroll
            for (int r = 0; r < R; r++) x[r] = cmul<T>(x[r], ldg<T>(a.twist + pos(r)));
        }
    };
    constexpr std::bool_constant<KIND == SINGLE_NEG || KIND == SINGLE_VJP> park_fold{};
    constexpr std::bool_constant<KIND == SINGLE_NEG> op_fold{};
    cx<T> pk[16], x[16];
    if (u0 < u1) load(pk, a.park, u0, park_fold);
    tl::template stage_twiddles<(m < 11)>(tw, a.roots, 0, t, M / 2);
    __syncthreads();
    for (long long u = u0; u < u1; u++)
    {
        load(x, a.op[0], u, op_fold);
        twist(pk);
        tl::template forward<T, m>(pk, sm, tw, t); // first writes the positions this thread read last
        __syncthreads();                           // the last transpose is read
#pragma unroll
        for (int l = 0; l < NOPS; l++)
        {
            if (l > 0) load(x, a.op[l], u, op_fold);
            twist(x);
            tl::template forward<T, m>(x, sm, tw, t);
#pragma unroll
            for (int r = 0; r < R; r++) x[r] = KIND == SINGLE_VJP ? cmulc<T>(pk[r], x[r]) : cmul<T>(x[r], pk[r]);
            if (l == NOPS - 1 && u + 1 < u1) load(pk, a.park, u + 1, park_fold);
            tl::template inverse<T, m>(x, sm, tw, t);
            const cx<T> sc = mk<T>(a.scale, T(0));
            const bool whole = (u + 1) * tl::P <= points;
#pragma unroll
            for (int r = 0; r < R; r++)
            {
                const long long e = u * tl::P + t + r * HT;
                cx<T> v = cmul<T>(x[r], sc);
                if constexpr (KIND != SINGLE_CYC) v = cmul<T>(v, ldg<T>(a.untwist + pos(r)));
                if (!whole && e >= points) continue;
                if constexpr (KIND == SINGLE_CYC)
                {
                    st_stream(static_cast<cx<T>*>(a.out[l]) + e, v);
                }
                else if constexpr (KIND == SINGLE_VJP)
                {
                    st_stream(static_cast<T*>(a.out[l]) + e, v.x);
                }
                else
                {
                    T* p = static_cast<T*>(a.out[l]) + fold_at(u, r);
                    st_stream(p, v.x);
                    st_stream(p + M, v.y);
                }
            }
        }
    }
}

// Products of 2^m points, m = 4 .. 12. The operands' tables are the native block.
template <typename T> int launch_single(int kind, int m, const SingleArgs<T>& a, cudaStream_t s);

} // namespace gfb
