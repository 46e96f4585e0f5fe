// gpufft-b200: the exact (split) product on FP64 transforms, with one operand cut
// into limbs and the other whole.
//
// c = a b mod (X^N + 1) for integers |a_i|, |b_i| < 2^B. An FP64 transform pair
// leaves an error of about 7 rms(a) rms(b) sqrt(N log2 N) 2^-53 per coefficient
// (the model of gf_split.cu): at B = 23 and N = 2^16 that is 18, far above 0.5, but
// with a alone cut into K = 2 limbs of 12 bits it is 0.005. Rows whose coefficients
// add up need more: a limb's product of N 2^11 2^23 or three times that is beyond
// what a double holds to 0.5, and three limbs of 8 bits keep it below 2^48
// (exact_plan). So a is cut into the fewest limbs that hold every row of the call
// (one up to 16 bits, three at 24 bits and N = 2^16) and b stays whole: K + 1 forward
// and K inverse FP64 transforms, where equal FP32 limbs of both operands take 4k - 1
// (19 for 24 bits). B200 runs FP64 at half the FP32 rate, so 7 against 19 is three
// quarters of the arithmetic, and the spectra in memory fall from 19 x 8 to 4 x 16
// bytes per point.
//
// Non-negative inputs are centred, a = a' + C u, b = b' + C u (C = 2^B, u the
// all-ones polynomial):
//     a b = sum_l 2^(w l) A_l (b' + C u) + C u b' + C^2 u u.
// The tile kernel forms A_l (B' + C U), adds 2^(B - w(K-1)) U B' to the last limb's
// product (U = transform of u), and C^2 u u is added exactly in int64.
//
// Kernels, rings N = 2^14 .. 2^17 (transforms of 2^m points, m = N's log2 - 1):
//   exact_fwd_col   digits, fold, twist and the first m - 11 stages of every limb
//                   of a and of b (a column of 2^(m-11) points on one lane, on two
//                   from 16 points on);
//   exact_tile      the eleven stages on 2048-point tiles of b (parked in
//                   registers) and of each limb, the product, the inverse stages
//                   (gf_tile.cuh);
//   exact_inv_col   last inverse stages, rounding, the error report and the int64
//                   sum of the limbs' products.
// Rings N = 2^5 .. 2^13 run in one kernel, exact_single, a CTA holding whole
// products.
//
// Measured (B200) against the limb chain: N = 2^16, batch 256, 24 bits, three limbs:
// 516 us (columns 126 + 110, tiles 296, tables 7) against 1076; 16 bits, one limb: 230
// against 867; N = 2^13, batch 333, 16 bits: 39 against 378; N = 2^12, batch 2000, 16
// bits: 77 against 809; one product of N = 2^12, 24 bits: 19 against 21.5.
#pragma once

#include "gf_split.cuh"
#include "gf_tile.cuh"

namespace gfb
{

constexpr int EXACT_MAX_LIMBS = 4;

struct ExactArgs
{
    const int32_t* a;
    const int32_t* b;
    int64_t* c;
    cx<double>* spec; // [K+1][W][M]: a's limbs, then b
    const cx<double>* roots;
    const cx<double>* twist;
    const cx<double>* uspec; // U; each 4096-point tile permuted e -> (e >> 4) + 256 (e & 15) when M > 4096
    unsigned* max_err;       // float bits of the largest pre-rounding error (may be null)
    long long cen;           // centring offset C (0: none)
    long long voff;          // digits of a: V = x + voff
    double ushift;           // 2^(B - w(K-1)): weight of U B' in the last limb's product
    double scale;
    int w;       // limb width
    long long W; // products of this launch
};

// The pointer again, hidden from the compiler: table entries used by several
// limbs are loaded for each (they are in L1) instead of being kept in registers.
__device__ __forceinline__ const cx<double>* fresh(const cx<double>* p)
{
    asm volatile("" : "+l"(p));
    return p;
}

// 1.5 2^52 and its encoding: v + MAGIC is v rounded to the nearest even integer
// for |v| < 2^51, and the integer is the sum's encoding minus MAGIC's.
constexpr double RND64 = 6755399441055744.0;
constexpr long long RND64_BITS = 0x4338000000000000LL;

// The double value of a 32-bit integer, through the mantissa of 2^52 (one
// addition instead of a conversion instruction).
__device__ __forceinline__ double int_f64(int d)
{
    return __hiloint2double(0x43300000, d ^ (int)0x80000000) - 4503601774854144.0; // 2^52 + 2^31
}

// Digit l of K of a's coefficient (balanced; the last takes what is left); K = 1
// (and b) the centred value itself.
template <int K> __device__ __forceinline__ int exact_digit(int x, long long voff, int l, int w)
{
    if (K == 1) return (int)((long long)x + voff);
    const long long V = (long long)x + voff;
    if (l == K - 1) return (int)(V >> (w * l));
    return (int)(((unsigned)(V >> (w * l))) & ((1u << w) - 1)) - (1 << (w - 1));
}

// Largest distance to the nearest integer and largest magnitude, kept as the high
// words of the doubles (ordered like the values, 20 bits of mantissa).
struct ExactErr
{
    int e = 0, big = 0;
    __device__ __forceinline__ void add(double d, double v)
    {
        e = max(e, __double2hiint(fabs(d)));
        big = max(big, __double2hiint(fabs(v)));
    }
    // exact_plan keeps in-range rows at or below 2^48; from 2^49 on (coefficients out
    // of range) the error nears 0.5 and the distance no longer certifies anything
    __device__ __forceinline__ float value() const
    {
        if (big >= 0x43000000) return 1.0f;
        return e == 0 ? 0.f : fminf((float)__hiloint2double(e, -1), 0.5f); // rounded up; a distance is at most 0.5
    }
};

// C^2 u u: coefficient j is C^2 (2j + 2 - N)
__device__ __forceinline__ long long exact_uu(long long cen, long long j, long long N)
{
    return (long long)((unsigned long long)cen * (unsigned long long)cen * (unsigned long long)(2 * j + 2 - N));
}

// ---------------------------------------------------------------------------
// column kernels: m = L + 11, columns of 2^L points 2048 apart
// ---------------------------------------------------------------------------
// One lane per column up to 8 points, two (the rows of one parity each) from 16.
template <int L> constexpr bool exact_pair() { return L >= 4; }
template <int L> constexpr int exact_rows() { return exact_pair<L>() ? 1 << (L - 1) : 1 << L; }

// The column's stages on its rows (lane half hb of a pair): the butterflies,
// twiddles and order of col_pass_kernel. Inverse twiddles are conjugate roots.
template <bool FWD, int L>
__device__ __forceinline__ void exact_stages(cx<double> (&x)[exact_rows<L>()], const cx<double>* __restrict__ roots, int hb)
{
    constexpr bool PAIR = exact_pair<L>();
    constexpr int H = exact_rows<L>();
#pragma unroll
    for (int k = 0; k < L; k++)
    {
        const int u = FWD ? k : L - 1 - k;
        if (PAIR && u == L - 1)
        {
#pragma unroll
            for (int q = 0; q < H; q++)
            {
                cx<double> wt = ldg<double>(roots + q);
                if (FWD)
                {
                    const cx<double> mine = hb ? cmul<double>(x[q], wt) : x[q];
                    const cx<double> other = shfl_half<double>(mine);
                    x[q] = hb ? csub<double>(other, mine) : cadd<double>(mine, other);
                }
                else
                {
                    wt.y = -wt.y;
                    const cx<double> other = shfl_half<double>(x[q]);
                    x[q] = hb ? cmul<double>(csub<double>(other, x[q]), wt) : cadd<double>(x[q], other);
                }
            }
            continue;
        }
        const int lg = (PAIR ? L - 2 : L - 1) - u; // log2 of the pair's distance in rows of this lane
#pragma unroll
        for (int q = 0; q < H; q++)
        {
            if (q & (1 << lg)) continue;
            cx<double> wt = ldg<double>(roots + (q >> (lg + 1)));
            if (FWD)
            {
                ct_bfly<double>(x[q], x[q + (1 << lg)], wt);
            }
            else
            {
                wt.y = -wt.y;
                gs_bfly<double>(x[q], x[q + (1 << lg)], wt);
            }
        }
    }
}

constexpr int EXACT_COL_THREADS = 128;

template <int L, int K>
__global__ void __launch_bounds__(EXACT_COL_THREADS, L <= 3 ? 6 : 4) exact_fwd_col(const ExactArgs a)
{
    pdl_begin(); // before any global-memory access (programmatic launch)
    constexpr bool PAIR = exact_pair<L>();
    constexpr int H = exact_rows<L>(), LS = PAIR ? 2 : 1;
    constexpr long long C = 2048, M = C << L;
    const long long idx = (long long)blockIdx.x * EXACT_COL_THREADS + threadIdx.x;
    const int hb = PAIR ? (int)((idx >> 4) & 1) : 0;
    const long long col = PAIR ? ((idx >> 5) << 4) + (idx & 15) : idx; // over (operand, product, column)
    const long long c = (col & (C - 1)) + hb * C;
    const long long bb = col >> 11; // the grid covers whole columns: C is a multiple of the block
    const bool isb = bb >= a.W;
    const long long p = isb ? bb - a.W : bb;
    const int32_t* src = (isb ? a.b : a.a) + p * 2 * M + c;
    int v0[H], v1[H];
#pragma unroll
    for (int q = 0; q < H; q++)
    {
        v0[q] = __ldg(src + q * LS * C);
        v1[q] = __ldg(src + q * LS * C + M);
    }
    auto transform = [&](auto digit, cx<double>* dst) {
        cx<double> x[H];
        const cx<double>* tw = fresh(a.twist) + c;
#pragma unroll
        for (int q = 0; q < H; q++)
            x[q] = cmul<double>(mk<double>(int_f64(digit(v0[q])), int_f64(digit(v1[q]))), ldg<double>(tw + q * LS * C));
        exact_stages<true, L>(x, fresh(a.roots), hb);
#pragma unroll
        for (int q = 0; q < H; q++) dst[q * LS * C] = x[q];
    };
    cx<double>* dst = a.spec + p * M + c;
    if (isb)
    {
        transform([&](int x) { return (int)((long long)x - a.cen); }, dst + K * a.W * M);
        return;
    }
#pragma unroll 1
    for (int l = 0; l < K; l++)
    {
        long long voff = a.voff;
        asm volatile("" : "+l"(voff)); // x + voff is formed per limb, not kept in registers
        transform([&](int x) { return exact_digit<K>(x, voff, l, a.w); }, dst + l * a.W * M);
    }
}

template <int L, int K>
__global__ void __launch_bounds__(EXACT_COL_THREADS, L == 5 ? 2 : K > 1 ? 4 : 5) exact_inv_col(const ExactArgs a)
{
    pdl_begin(); // before any global-memory access (programmatic launch)
    constexpr bool PAIR = exact_pair<L>();
    constexpr int H = exact_rows<L>(), LS = PAIR ? 2 : 1;
    constexpr long long C = 2048, M = C << L;
    const long long idx = (long long)blockIdx.x * EXACT_COL_THREADS + threadIdx.x;
    const int hb = PAIR ? (int)((idx >> 4) & 1) : 0;
    const long long col = PAIR ? ((idx >> 5) << 4) + (idx & 15) : idx;
    const long long c = (col & (C - 1)) + hb * C;
    const long long p = col >> 11;
    const cx<double>* src = a.spec + p * M + c;
    long long lo[H], hi[H];
#pragma unroll
    for (int q = 0; q < H; q++)
    {
        const long long j = c + q * LS * C;
        lo[q] = exact_uu(a.cen, j, 2 * M);
        hi[q] = exact_uu(a.cen, j + M, 2 * M);
    }
    ExactErr err;
    // the next limb's loads are in flight while this one is transformed
    cx<double> nx[H];
#pragma unroll
    for (int q = 0; q < H; q++) nx[q] = __ldcs(src + q * LS * C);
#pragma unroll 1
    for (int l = 0; l < K; l++)
    {
        cx<double> x[H];
#pragma unroll
        for (int q = 0; q < H; q++) x[q] = nx[q];
        if (l + 1 < K)
        {
#pragma unroll
            for (int q = 0; q < H; q++) nx[q] = __ldcs(src + (l + 1) * a.W * M + q * LS * C);
        }
        exact_stages<false, L>(x, fresh(a.roots), hb);
        const cx<double>* tw = fresh(a.twist) + c;
        const int sh = a.w * l;
#pragma unroll
        for (int q = 0; q < H; q++)
        {
            const cx<double> t = ldg<double>(tw + q * LS * C);
            // untwist = conj(twist); the scale is a power of two
            const cx<double> v = cmul<double>(x[q], mk<double>(t.x * a.scale, -t.y * a.scale));
            const double r0 = __dadd_rn(v.x, RND64), r1 = __dadd_rn(v.y, RND64);
            err.add(__dsub_rn(v.x, __dsub_rn(r0, RND64)), v.x);
            err.add(__dsub_rn(v.y, __dsub_rn(r1, RND64)), v.y);
            const long long i0 = __double_as_longlong(r0) - RND64_BITS, i1 = __double_as_longlong(r1) - RND64_BITS;
            lo[q] = (long long)((unsigned long long)lo[q] + ((unsigned long long)i0 << sh));
            hi[q] = (long long)((unsigned long long)hi[q] + ((unsigned long long)i1 << sh));
        }
    }
    long long* dst = reinterpret_cast<long long*>(a.c + p * 2 * M + c);
#pragma unroll
    for (int q = 0; q < H; q++)
    {
        __stcs(dst + q * LS * C, lo[q]);
        __stcs(dst + q * LS * C + M, hi[q]);
    }
    report_err(a.max_err, err.value());
}

// The product of a limb's spectrum value x with b's (pk); `last`: the limb that U B'
// joins.
__device__ __forceinline__ cx<double> exact_product(cx<double> x, cx<double> pk, const ExactArgs& a, double ui, bool last)
{
    // U = 1 + i ui
    const double C = (double)a.cen;
    cx<double> v = cmul<double>(x, mk<double>(pk.x + C, rfma(C, ui, pk.y)));
    if (last)
    {
        v.x = rfma(a.ushift, rfma(-ui, pk.y, pk.x), v.x);
        v.y = rfma(a.ushift, rfma(ui, pk.x, pk.y), v.y);
    }
    return v;
}

template <int K> __global__ void __launch_bounds__(tile::HT, tile_min_blocks<double>()) exact_tile(const ExactArgs a, int m)
{
    pdl_begin(); // before any global-memory access (programmatic launch)
    constexpr int R = tile::R;
    extern __shared__ __align__(16) unsigned char smraw[];
    cx<double>* sm = reinterpret_cast<cx<double>*>(smraw);
    cx<double>* tw = sm + tile::SLOT;
    const int t = threadIdx.x;
    const long long M = 1LL << m;
    const long long base = ((long long)blockIdx.x << 11) + t; // flat over the products
    const long long g = (long long)blockIdx.x & ((1LL << (m - 11)) - 1);
    const long long WM = a.W * M;
    if (t == 0) // the other limbs wait in L2 (N = 2^16, batch 256, two limbs: 437 -> 431 us)
    {
#pragma unroll
        for (int l = 1; l < K; l++) prefetch_l2(a.spec + l * WM + base, tile::P * sizeof(cx<double>));
    }
    cx<double> pk[R], x[R];
#pragma unroll
    for (int r = 0; r < R; r++) pk[r] = a.spec[K * WM + base + (r << 7)];
    tile::stage_twiddles<false>(tw, a.roots, g, t, 0);
#pragma unroll
    for (int r = 0; r < R; r++) x[r] = a.spec[base + (r << 7)];
    __syncthreads();
    tile::forward<double>(pk, sm, tw, t);
    __syncthreads(); // the parked operand's last transpose is read
    // U of the thread's points j = 2048 g + 16 t + r: coalesced in the permuted order
    // (m > 12 here)
    const cx<double>* up = a.uspec + ((g >> 1) << EBITS) + ((g & 1) << 7) + t;
    // a loop: unrolled, three limbs spilled and waited for instructions (0.74 of the
    // stalls per issue; N = 2^16, 24 bits, batch 256: 324 -> 296 us, two limbs 212 -> 199)
#pragma unroll 1
    for (int l = 0; l < K; l++)
    {
        if (l > 0)
        {
#pragma unroll
            for (int r = 0; r < R; r++) x[r] = a.spec[l * WM + base + (r << 7)];
        }
        tile::forward<double>(x, sm, tw, t); // first writes the positions this thread read last
        if (a.cen == 0)
        {
#pragma unroll
            for (int r = 0; r < R; r++) x[r] = cmul<double>(x[r], pk[r]);
        }
        else
        {
#pragma unroll
            for (int r = 0; r < R; r++) x[r] = exact_product(x[r], pk[r], a, __ldg(&up[r * 256].y), l == K - 1);
        }
        tile::inverse<double>(x, sm, tw, t);
#pragma unroll
        for (int r = 0; r < R; r++) a.spec[l * WM + base + (r << 7)] = x[r];
    }
}

// ---------------------------------------------------------------------------
// whole products of 2^m-point transforms, m = 4 .. 12: 2^(11-m) to a CTA of 128
// threads, one of 4096 points to a CTA of 256
// ---------------------------------------------------------------------------
// Two CTAs per SM (one at 4096 points) where a thread holds 16 twist factors of its
// own; three below, where they repeat (BLOCKS, exact_single_blocks).
template <int m, int K, int BLOCKS>
__global__ void __launch_bounds__(m == 12 ? 256 : 128, BLOCKS) exact_single(const ExactArgs a)
{
    pdl_begin(); // before any global-memory access (programmatic launch)
    using tl = TileOf<m == 12 ? 12 : 11>;
    constexpr int R = tl::R, HT = tl::HT;
    constexpr int M = 1 << m;
    extern __shared__ __align__(16) unsigned char smraw[];
    cx<double>* sm = reinterpret_cast<cx<double>*>(smraw);
    cx<double>* tw = sm + tl::SLOT;
    const int t = threadIdx.x;
    const long long p0 = (long long)blockIdx.x << (m == 12 ? 0 : 11 - m); // first product of this CTA
    const long long left = (a.W - p0) << m;                 // points of the batch from there on
    // register r: point e = t + r HT, product p0 + (e >> m), position e mod M; a
    // row has 2M coefficients, so the coefficient is at 2e - (e mod M), and + M
    auto at = [&](int r) {
        const int e = t + r * HT;
        return 2 * e - (e & (M - 1));
    };
    auto load = [&](cx<double> (&x)[16], const int32_t* src, auto digit) {
        const cx<double>* tws = fresh(a.twist);
        constexpr int Q = m >= 10 ? 4 : 8; // points at a time: as many loads in flight as registers allow
#pragma unroll
        for (int h = 0; h < R; h += Q)
        {
            int v0[Q], v1[Q];
#pragma unroll
            for (int q = 0; q < Q; q++)
            {
                const bool ok = t + (h + q) * HT < left;
                v0[q] = ok ? __ldg(src + p0 * 2 * M + at(h + q)) : 0;
                v1[q] = ok ? __ldg(src + p0 * 2 * M + at(h + q) + M) : 0;
            }
#pragma unroll
            for (int q = 0; q < Q; q++)
                x[h + q] = cmul<double>(mk<double>(int_f64(digit(v0[q])), int_f64(digit(v1[q]))),
                                        ldg<double>(tws + ((t + (h + q) * HT) & (M - 1))));
        }
    };
    cx<double> pk[R];
    load(pk, a.b, [&](int v) { return (int)((long long)v - a.cen); });
    tl::template stage_twiddles<(m < 11)>(tw, a.roots, 0, t, M / 2);
    __syncthreads();
    tl::template forward<double, m>(pk, sm, tw, t);
    __syncthreads(); // the parked operand's last transpose is read
    ExactErr err;
    long long* dst = reinterpret_cast<long long*>(a.c) + p0 * 2 * M;
#pragma unroll
    for (int l = 0; l < K; l++)
    {
        cx<double> x[R];
        load(x, a.a, [&](int v) { return exact_digit<K>(v, a.voff, l, a.w); });
        tl::template forward<double, m>(x, sm, tw, t); // first writes the positions this thread read last
        if (a.cen == 0)
        {
#pragma unroll
            for (int r = 0; r < R; r++) x[r] = cmul<double>(x[r], pk[r]);
        }
        else
        {
#pragma unroll
            for (int r = 0; r < R; r++)
                x[r] = exact_product(x[r], pk[r], a, __ldg(&a.uspec[(16 * t + r) & (M - 1)].y), l == K - 1);
        }
        tl::template inverse<double, m>(x, sm, tw, t);
        const int sh = a.w * l;
        const cx<double>* tws = fresh(a.twist);
#pragma unroll
        for (int r = 0; r < R; r++)
        {
            const int j = (t + r * HT) & (M - 1);
            const cx<double> u = ldg<double>(tws + j);
            const cx<double> v = cmul<double>(x[r], mk<double>(u.x * a.scale, -u.y * a.scale));
            const double r0 = __dadd_rn(v.x, RND64), r1 = __dadd_rn(v.y, RND64);
            if (t + r * HT >= left) continue;
            err.add(__dsub_rn(v.x, __dsub_rn(r0, RND64)), v.x);
            err.add(__dsub_rn(v.y, __dsub_rn(r1, RND64)), v.y);
            unsigned long long i0 = (unsigned long long)(__double_as_longlong(r0) - RND64_BITS) << sh;
            unsigned long long i1 = (unsigned long long)(__double_as_longlong(r1) - RND64_BITS) << sh;
            if (l == 0)
            {
                i0 += (unsigned long long)exact_uu(a.cen, j, 2 * M);
                i1 += (unsigned long long)exact_uu(a.cen, j + M, 2 * M);
            }
            else
            {
                // the sum so far is this thread's own store
                i0 += (unsigned long long)dst[at(r)];
                i1 += (unsigned long long)dst[at(r) + M];
            }
            dst[at(r)] = (long long)i0;
            dst[at(r) + M] = (long long)i1;
        }
    }
    report_err(a.max_err, err.value());
}

// CTAs per SM that exact_single is compiled for. 1024 points: at three, several limbs
// spill (two limbs 290 bytes a thread, three 520), so a launch that two per SM hold
// takes two (N = 2^11, 24 bits, 2 / 40 / 400 products: 19 / 19 / 31 us against 27 / 28 /
// 34), and one that three hold takes three (800: 41 against 51). Beyond, two limbs
// take three (4000: 160 against 173) and more limbs two (28 bits, 1200 / 4000: 103 / 261
// against 108 / 281).
template <int m> constexpr int exact_single_blocks(bool two)
{
    return m == 12 ? 1 : m == 11 || (m == 10 && two) ? 2 : 3;
}

} // namespace gfb
