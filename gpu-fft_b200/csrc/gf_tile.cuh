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

// Asks for `bytes` (a multiple of 16) from p in L2, for a later read of this CTA that
// its registers do not hold yet. One thread calls it. Rows that do not start on 16
// bytes (FP32 buffers on 8) go without. (For the adjoint's second operand it gave
// nothing: 307 against 305 us for 512 rows of N = 2^14.)
__device__ __forceinline__ void prefetch_l2(const void* p, unsigned bytes)
{
    if (reinterpret_cast<uintptr_t>(p) & 15) return;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "r"(bytes) : "memory");
}

// One tile of 2^LT points on 2^LT / 16 threads: LT = 11 as above; LT = 12 (256
// threads, rounds on the e-bits [8,12), [4,8), [0,4)) for whole transforms of 4096
// points (gf_single.cuh).
template <int LT> struct TileOf
{
    static constexpr int P = 1 << LT;           // points
    static constexpr int R = 16;                // points per thread
    static constexpr int HT = P / R;            // threads
    static constexpr int SLOT = P + P / 16;     // padded transpose buffer
    static constexpr int W1 = LT - 4, W2 = LT - 8, HI0 = LT - 8; // windows of the rounds, bits of the last
    static_assert(LT == 11 || LT == 12, "three rounds");
    static constexpr int N0 = HI0 == 4 ? 8 : 7; // even twiddles per thread of the innermost round
    static constexpr int S0 = HT + 1;           // stride of the staged innermost twiddles
    static constexpr int S2 = 9;                // stride of the staged middle twiddles
    static constexpr int TWN = N0 * S0 + 16 * S2 + 8;

    // e of register 0 of thread t when the registers are the e-bits [W, W+4)
    template <int W> static __device__ __forceinline__ int ebase(int t)
    {
        return (t & ((1 << W) - 1)) | ((t >> W) << (W + 4));
    }
    static __device__ __forceinline__ constexpr int ppos(int e) { return e + (e >> 4); }
    // ppos(ebase + (r << W)) - ppos(ebase): the window bits of ebase are clear
    template <int W> static __device__ __forceinline__ constexpr int poff(int r) { return (r << W) + ((r << W) >> 4); }

    template <int W, typename C> static __device__ __forceinline__ void put(const C (&x)[R], C* sm, int t)
    {
        const int b = ppos(ebase<W>(t));
#pragma unroll
        for (int r = 0; r < R; r++) sm[b + poff<W>(r)] = x[r];
    }
    template <int W, typename C> static __device__ __forceinline__ void get(C (&x)[R], const C* sm, int t)
    {
        const int b = ppos(ebase<W>(t));
#pragma unroll
        for (int r = 0; r < R; r++) x[r] = sm[b + poff<W>(r)];
    }

    // The tile's even twiddles. A stage with nt = 2^k twiddles per thread uses
    // table[(T << u) + nt i + h], h < nt, for an i of the thread; the even h of the
    // stages of a round sit at positions nt/2 + h/2 (0 for the stage with one
    // twiddle, whose entry may be odd):
    //   outer round   (u = 0..3)  i = 0:
    //   middle round  (u = 4..7)  i = t >> W2
    //   inner round   (u = 8..)   i = t (LT = 11 has no stage with one twiddle here)
    template <typename C> static __device__ __forceinline__ C* outer(C* tw) { return tw + N0 * S0 + 16 * S2; }
    template <typename C> static __device__ __forceinline__ C* middle(C* tw, int i) { return tw + N0 * S0 + i * S2; }
    template <typename C> static __device__ __forceinline__ C* inner(C* tw, int i) { return tw + (N0 - 8) * S0 + i; }

    // SHORT: whole transforms shorter than the tile have a shorter table (`entries`)
    // and use no others
    template <bool SHORT, typename C>
    static __device__ __forceinline__ void stage_twiddles(C* tw, const C* __restrict__ tab, long long T, int t, long long entries)
    {
        // inner round: linear even entry p of a stage is table[(T << u) + 2p]
        if constexpr (HI0 == 4) inner(tw, t)[0] = __ldg(tab + (T << 8) + t);
#pragma unroll
        for (int k = 0; k < 7; k++)
        {
            const int p = (k == 0 ? 0 : k < 3 ? (k - 1) * HT : (k - 3) * HT) + t; // of one of the last three stages
            const int lg = k == 0 ? 0 : k < 3 ? 1 : 2;                           // log2 evens per thread
            const long long e = (T << (LT - 3 + lg)) + 2 * p;
            if (!SHORT || e < entries) inner(tw, p >> lg)[((1 << lg) + (p & ((1 << lg) - 1))) * S0] = __ldg(tab + e);
        }
        // middle round: 16 i x 8 positions
        if (HT == 128 || t < 128)
        {
            const int i = t >> 3, pos = t & 7;
            const int lg = pos == 0 ? 0 : 32 - __clz(pos); // log2 twiddles per thread of the stage
            const int h = pos == 0 ? 0 : 2 * (pos - (1 << (lg - 1)));
            const long long e = (T << (4 + lg)) + (i << lg) + h;
            if (!SHORT || e < entries) middle(tw, i)[pos] = __ldg(tab + e);
        }
        if (t < 8)
        {
            const int lg = t == 0 ? 0 : 32 - __clz(t);
            const int h = t == 0 ? 0 : 2 * (t - (1 << (lg - 1)));
            const long long e = (T << lg) + h;
            if (!SHORT || e < entries) outer(tw)[t] = __ldg(tab + e);
        }
    }

    // One round on the register bits [LO, HI): the stage on bit pb has 2^(3-pb)
    // twiddles per thread. `tw` points to the thread's entry of position 0, `st` is
    // the distance between positions.
    template <typename T, bool FWD, int LO, int HI>
    static __device__ __forceinline__ void round(cx<T> (&x)[R], const cx<T>* tw, int st)
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

    // The round of window W on its HI lowest bits, for 2^m-point transforms side by
    // side in the tile (m = LT: one transform, or one tile of a longer one): only
    // the stages on e-bits below m, with the group index taken inside the transform.
    // With m < W + 4 the registers' upper bits number sub-networks and the twiddles
    // are table[0 .. 8).
    template <typename T, bool FWD, int W, int HI, int m>
    static __device__ __forceinline__ void round_m(cx<T> (&x)[R], cx<T>* tw, int t)
    {
        if constexpr (m >= W + 4)
        {
            constexpr int mask = (1 << (m - 4 - W)) - 1;
            if constexpr (W == W1) round<T, FWD, 0, HI>(x, outer(tw), 1);
            else if constexpr (W == W2) round<T, FWD, 0, HI>(x, middle(tw, (t >> W2) & mask), 1);
            else round<T, FWD, 0, HI>(x, inner(tw, t & mask), S0);
        }
        else if constexpr (m > W)
        {
            constexpr int NB = m - W;
#pragma unroll
            for (int k = 0; k < NB; k++)
            {
                const int pb = FWD ? NB - 1 - k : k;
                const int nt = 1 << (NB - 1 - pb); // twiddles of the stage: table[0 .. nt)
#pragma unroll
                for (int r = 0; r < R; r++)
                {
                    if (r & (1 << pb)) continue;
                    const int h = (r >> (pb + 1)) & (nt - 1);
                    cx<T> ev = outer(tw)[4 + (h >> 1)];
                    if (!FWD) ev.y = -ev.y;
                    const cx<T> w = !(h & 1) ? ev : (FWD ? mk<T>(-ev.y, ev.x) : mk<T>(ev.y, -ev.x));
                    if (FWD)
                        ct_bfly<T>(x[r], x[r | (1 << pb)], w);
                    else
                        gs_bfly<T>(x[r], x[r | (1 << pb)], w);
                }
            }
        }
    }

    // Forward stages: x in window W1, out in window 0. The caller has made sure that
    // no thread still reads the buffer.
    template <typename T, int m = LT>
    static __device__ __forceinline__ void forward(cx<T> (&x)[R], cx<T>* sm, cx<T>* tw, int t)
    {
        round_m<T, true, W1, 4, m>(x, tw, t);
        put<W1>(x, sm, t);
        __syncthreads();
        get<W2>(x, sm, t);
        round_m<T, true, W2, 4, m>(x, tw, t);
        put<W2>(x, sm, t); // the positions this thread read
        __syncthreads();
        get<0>(x, sm, t);
        round_m<T, true, 0, HI0, m>(x, tw, t);
    }

    // Inverse stages: x in window 0 (its positions of the buffer are this thread's),
    // out in window W1.
    template <typename T, int m = LT>
    static __device__ __forceinline__ void inverse(cx<T> (&x)[R], cx<T>* sm, cx<T>* tw, int t)
    {
        round_m<T, false, 0, HI0, m>(x, tw, t);
        put<0>(x, sm, t);
        __syncthreads();
        get<W2>(x, sm, t);
        round_m<T, false, W2, 4, m>(x, tw, t);
        put<W2>(x, sm, t);
        __syncthreads();
        get<W1>(x, sm, t);
        round_m<T, false, W1, 4, m>(x, tw, t);
    }
};
constexpr int TILE_LT = 11;
// most stages left for the pass before the tiles (a column pass up to COL_MAX_L, a
// strided pass of 4096-point tiles above)
constexpr int TILE_MAX_L = 9;
using tile = TileOf<TILE_LT>;

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
    constexpr int NOPS = MODE == TILE_VJP ? 2 : 1, R = tile::R;
    extern __shared__ __align__(16) unsigned char smraw[];
    cx<T>* sm = reinterpret_cast<cx<T>*>(smraw);
    cx<T>* tw = sm + tile::SLOT;
    const int t = threadIdx.x;
    const long long base = ((long long)blockIdx.x << 11) + t; // flat over the products
    const long long g = (long long)blockIdx.x & ((1LL << (a.m - 11)) - 1);
    // both operands' loads are in flight before the first stage
    cx<T> pk[R], x[R];
#pragma unroll
    for (int r = 0; r < R; r++) pk[r] = a.park[base + (r << 7)];
    tile::stage_twiddles<false>(tw, a.roots, g, t, 0);
#pragma unroll
    for (int r = 0; r < R; r++) x[r] = a.in[0][base + (r << 7)];
    __syncthreads();
    tile::forward<T>(pk, sm, tw, t);
    __syncthreads(); // the parked operand's last transpose is read
#pragma unroll
    for (int l = 0; l < NOPS; l++)
    {
        if (l > 0)
        {
#pragma unroll
            for (int r = 0; r < R; r++) x[r] = a.in[l][base + (r << 7)];
        }
        tile::forward<T>(x, sm, tw, t); // first writes the positions this thread read last
#pragma unroll
        for (int r = 0; r < R; r++) x[r] = MODE == TILE_VJP ? cmulc<T>(pk[r], x[r]) : cmul<T>(x[r], pk[r]);
        tile::inverse<T>(x, sm, tw, t);
#pragma unroll
        for (int r = 0; r < R; r++) a.out[l][base + (r << 7)] = x[r];
    }
}

// tiles = products << (m - 11)
template <typename T, int MODE> int launch_tile_product(const TileArgs<T>& a, long long tiles, cudaStream_t s);

} // namespace gfb
