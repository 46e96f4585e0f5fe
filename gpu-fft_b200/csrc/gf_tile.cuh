// gpufft-b200: the products' middle on 2048-point tiles, one 128-thread CTA per
// tile, one operand's spectrum parked in registers.
//
// A product whose transforms have M = 2^m > 4096 points runs its first m - 11
// forward and last m - 11 inverse stages in the column passes (gf_pass.cuh) and
// the eleven stages in between here: for a tile T (2048 consecutive points, the
// stage-(m-11) group T of the transform) the CTA
//   1. transforms the tile of the parked operand: 16 points per thread, eleven
//      stages as three radix-16 register rounds on the e-bits [7,11), [3,7) and
//      [0,3), with a padded shared-memory transpose between them;
//   2. for each other operand: transforms its tile the same way, multiplies by
//      the parked spectrum in registers, runs the eleven inverse stages and
//      stores the result tile.
// Modes: TILE_MUL  x := x p          (products: b parked, a the other operand);
//        TILE_VJP  x := p conj(x)    (adjoint: g parked, the operands b and a).
//
// Why this shape. The pass is a chain of load, butterfly, transpose and store
// phases; on one large CTA per SM (4096 points, 512 threads x 8 points of both
// operands) those phases do not overlap, and the FP64 pipe ran at 39 %, the
// load/store pipe at 52 %. CTAs of four warps drift apart, so one CTA's memory
// phase runs under another's arithmetic. Sixteen points per thread need two
// transposes per transform where eight need three, and parking one operand (64
// registers in FP64) leaves room for one more, so three CTAs fit an SM in FP64
// (168 registers) and five in FP32.
//
// Twiddles come from the native tables only (gpufft_ffnt_make_tables_*): an odd
// entry is exactly i times its even neighbour and the inverse roots are exact
// conjugates, so the tile's even entries of the forward table serve every stage
// of both directions. They are staged once per CTA in shared memory, thread-major
// for the innermost round: read from the table there, a warp's loads would stride
// 128 bytes and cost as many shared-memory cycles as five of the six data passes.
//
// Butterflies, twiddle indices and stage order are the engine's (stage u of the
// tile on e-bit q = 10 - u pairs e with e + 2^q and uses table[(T << u) +
// (e >> (q + 1))]), so every value has the bits of the engine's passes.
#pragma once

#include "gf_pass.cuh"

namespace gfb
{
namespace tile
{
constexpr int LT = 11;            // log2 points per tile
constexpr int P = 1 << LT;        // 2048 points
constexpr int HT = 128;           // threads
constexpr int R = P / HT;         // 16 points per thread
constexpr int SLOT = P + P / 16;  // padded transpose buffer
constexpr int S0 = HT + 1;        // stride of the staged innermost twiddles
constexpr int S3 = 9;             // stride of the staged middle twiddles
constexpr int TWN = 7 * S0 + 16 * S3 + 8;

// e of register 0 of thread t when the registers are the e-bits [W, W+4)
template <int W> __device__ __forceinline__ int ebase(int t)
{
    return (t & ((1 << W) - 1)) | ((t >> W) << (W + 4));
}
__device__ __forceinline__ constexpr int ppos(int e) { return e + (e >> 4); }
// ppos(ebase + (r << W)) - ppos(ebase): the window bits of ebase are clear
template <int W> __device__ __forceinline__ constexpr int poff(int r) { return (r << W) + ((r << W) >> 4); }

template <int W, typename C> __device__ __forceinline__ void put(const C (&x)[R], C* sm, int t)
{
    const int b = ppos(ebase<W>(t));
#pragma unroll
    for (int r = 0; r < R; r++) sm[b + poff<W>(r)] = x[r];
}
template <int W, typename C> __device__ __forceinline__ void get(C (&x)[R], const C* sm, int t)
{
    const int b = ppos(ebase<W>(t));
#pragma unroll
    for (int r = 0; r < R; r++) x[r] = sm[b + poff<W>(r)];
}

// The tile's even twiddles. A stage with nt = 2^k >= 2 twiddles per thread uses
// table[(T << u) + nt i + h], h < nt, for an i of the thread; the even h of the
// stages of a round sit at positions nt/2 + h/2 (0 for the stage with one
// twiddle, whose entry may be odd):
//   window 7 (u = 0..3)  i = 0:       tw7[pos],             pos 0..7
//   window 3 (u = 4..7)  i = t >> 3:  tw3[(t >> 3) S3 + pos], pos 0..7
//   window 0 (u = 8..10) i = t:       tw0[(pos - 1) S0 + t],  pos 1..7
template <typename C> __device__ __forceinline__ void stage_twiddles(C* tw, const C* __restrict__ tab, long long T, int t)
{
    C* tw0 = tw;
    C* tw3 = tw + 7 * S0;
    C* tw7 = tw3 + 16 * S3;
    // window 0: linear even entry p of stage u is table[(T << u) + 2p]
#pragma unroll
    for (int k = 0; k < 7; k++)
    {
        const int p = (k == 0 ? 0 : k < 3 ? (k - 1) * HT : (k - 3) * HT) + t; // of stage 8, 9 or 10
        const int lg = k == 0 ? 0 : k < 3 ? 1 : 2;                           // log2 evens per thread
        const int i = p >> lg, pos = (1 << lg) + (p & ((1 << lg) - 1));
        tw0[(pos - 1) * S0 + i] = __ldg(tab + (T << (8 + lg)) + 2 * p);
    }
    // window 3: 16 i x 8 positions
    {
        const int i = t >> 3, pos = t & 7;
        const int lg = pos == 0 ? 0 : 32 - __clz(pos); // log2 twiddles per thread of the stage
        const int h = pos == 0 ? 0 : 2 * (pos - (1 << (lg - 1)));
        tw3[i * S3 + pos] = __ldg(tab + (T << (4 + lg)) + (i << lg) + h);
    }
    if (t < 8)
    {
        const int lg = t == 0 ? 0 : 32 - __clz(t);
        const int h = t == 0 ? 0 : 2 * (t - (1 << (lg - 1)));
        tw7[t] = __ldg(tab + (T << lg) + h);
    }
}

// One round on the register bits [LO, HI): the stage on bit pb has 2^(3-pb)
// twiddles per thread. `tw` points to the thread's entry of position 0, `st` is
// the distance between positions.
template <typename T, bool FWD, int LO, int HI>
__device__ __forceinline__ void round(cx<T> (&x)[R], const cx<T>* tw, int st)
{
#pragma unroll
    for (int k = 0; k < HI - LO; k++)
    {
        const int pb = FWD ? HI - 1 - k : LO + k;
        const int nt = 1 << (3 - pb); // twiddles of this stage per thread
        cx<T> e[4];
#pragma unroll
        for (int i = 0; i < (nt > 1 ? nt / 2 : 1); i++)
        {
            e[i] = tw[((nt >> 1) + i) * st];
            if (!FWD) e[i].y = -e[i].y; // inverse root
        }
#pragma unroll
        for (int r = 0; r < R; r++)
        {
            if (r & (1 << pb)) continue;
            const int h = r >> (pb + 1);
            const cx<T> ev = e[h >> 1];
            const cx<T> w = !(h & 1) ? ev : (FWD ? mk<T>(-ev.y, ev.x) : mk<T>(ev.y, -ev.x));
            if (FWD)
                ct_bfly<T>(x[r], x[r | (1 << pb)], w);
            else
                gs_bfly<T>(x[r], x[r | (1 << pb)], w);
        }
    }
}

// Eleven forward stages: x in window 7, out in window 0. The caller has made
// sure that no thread still reads the buffer.
template <typename T> __device__ __forceinline__ void forward(cx<T> (&x)[R], cx<T>* sm, const cx<T>* tw, int t)
{
    round<T, true, 0, 4>(x, tw + 7 * S0 + 16 * S3, 1);
    put<7>(x, sm, t);
    __syncthreads();
    get<3>(x, sm, t);
    round<T, true, 0, 4>(x, tw + 7 * S0 + (t >> 3) * S3, 1);
    put<3>(x, sm, t); // the positions this thread read
    __syncthreads();
    get<0>(x, sm, t);
    round<T, true, 0, 3>(x, tw - S0 + t, S0);
}

// Eleven inverse stages: x in window 0 (its positions of the buffer are this
// thread's), out in window 7.
template <typename T> __device__ __forceinline__ void inverse(cx<T> (&x)[R], cx<T>* sm, const cx<T>* tw, int t)
{
    round<T, false, 0, 3>(x, tw - S0 + t, S0);
    put<0>(x, sm, t);
    __syncthreads();
    get<3>(x, sm, t);
    round<T, false, 0, 4>(x, tw + 7 * S0 + (t >> 3) * S3, 1);
    put<3>(x, sm, t);
    __syncthreads();
    get<7>(x, sm, t);
    round<T, false, 0, 4>(x, tw + 7 * S0 + 16 * S3, 1);
}
} // namespace tile

enum TileMode
{
    TILE_MUL = 0,
    TILE_VJP = 1
};

// Operand l of product p has its spectrum at in[l] + p M and its result goes to
// out[l] + p M; the parked operand is at park + p M.
template <typename T> struct TileArgs
{
    const cx<T>* park;
    const cx<T>* in[2];
    cx<T>* out[2];
    const cx<T>* roots; // native forward table
    int m;              // log2 transform length
};

template <typename T> constexpr int tile_min_blocks() { return sizeof(T) == 8 ? 3 : 5; }

template <typename T, int MODE>
__global__ void __launch_bounds__(tile::HT, tile_min_blocks<T>()) tile_product_kernel(const TileArgs<T> a)
{
    pdl_begin(); // before any global-memory access (programmatic launch)
    using namespace tile;
    constexpr int NOPS = MODE == TILE_VJP ? 2 : 1;
    extern __shared__ __align__(16) unsigned char smraw[];
    cx<T>* sm = reinterpret_cast<cx<T>*>(smraw);
    cx<T>* tw = sm + SLOT;
    const int t = threadIdx.x;
    const long long base = ((long long)blockIdx.x << LT) + t; // flat over the products
    const long long g = (long long)blockIdx.x & ((1LL << (a.m - LT)) - 1);
    // both operands' loads are in flight before the first stage
    cx<T> pk[R], x[R];
#pragma unroll
    for (int r = 0; r < R; r++) pk[r] = a.park[base + (r << 7)];
    stage_twiddles(tw, a.roots, g, t);
#pragma unroll
    for (int r = 0; r < R; r++) x[r] = a.in[0][base + (r << 7)];
    __syncthreads();
    forward<T>(pk, sm, tw, t);
    __syncthreads(); // the parked operand's last transpose is read
#pragma unroll
    for (int l = 0; l < NOPS; l++)
    {
        if (l > 0)
        {
#pragma unroll
            for (int r = 0; r < R; r++) x[r] = a.in[l][base + (r << 7)];
        }
        forward<T>(x, sm, tw, t); // first writes the positions this thread read last
#pragma unroll
        for (int r = 0; r < R; r++) x[r] = MODE == TILE_VJP ? cmulc<T>(pk[r], x[r]) : cmul<T>(x[r], pk[r]);
        inverse<T>(x, sm, tw, t);
#pragma unroll
        for (int r = 0; r < R; r++) a.out[l][base + (r << 7)] = x[r];
    }
}

// tiles = products << (m - 11)
template <typename T, int MODE> int launch_tile_product(const TileArgs<T>& a, long long tiles, cudaStream_t s);

} // namespace gfb
