// gpufft-b200: plans, launches and C ABI of the exact product on FP64 transforms
// (gf_split_tile.cuh), in a translation unit of its own.
#include "gf_split_tile.cuh"
#include "gf_fused.cuh"

namespace gfb
{
// Twiddles of a call whose caller holds FP32 ones, in its workspace:
// [roots M/2 | twist M | U M], the values of the native FP64 block.
__global__ void exact_tables_kernel(cx<double>* tab, int m)
{
    pdl_begin(); // before any global-memory access (programmatic launch)
    // one value per thread: a call of few products waits for this kernel
    const long long M = 1LL << m, H = M >> 1;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    double s, c;
    if (i < H)
    {
        native_root(i, m, c, s);
        tab[i] = mk<double>(c, s);
    }
    else if (i < H + M)
    {
        sincospi((double)(i - H) / (double)(2 * M), &s, &c);
        tab[i] = mk<double>(c, s);
    }
    else if (i < H + 2 * M)
    {
        const long long j = i - H - M;
        const unsigned k = __brev((unsigned)j) >> (32 - m);
        sincospi((4.0 * (double)k + 1.0) / (4.0 * (double)M), &s, &c);
        const long long pu = (m > EBITS) ? ((j & ~4095LL) | ((j & 4095) >> 4) | ((j & 15) << 8)) : j;
        tab[H + M + pu] = mk<double>(1.0, c / s);
    }
}

// The fewest limbs K of a (width w) that hold both kinds of data, for operands of
// magnitude at most 2^B (after centring):
//   - uniform: the error model of the equal-limb plans (7.1 rms rms sqrt(N)
//     sqrt(log2(N/2)) 2^-53 per pair, pairs of a group in quadrature; measured at
//     most 1.2 of it) predicts at most 0.06;
//   - coherent (constant, half-range or zero rows, zero-padded ones), whose
//     coefficients add up: limb l's product reaches N 2^t 2^B (t: the limb's bits),
//     with b' + C u of up to 2^(B+1) for centred calls, whose last limb also carries
//     2^t U B'. The error such rows leave is at most 2^-50 of that bound (measured
//     over rings 2^5 .. 2^17 and 8 to 30 bits, on constant, half-range, zero-padded,
//     ramped and alternating rows: 0.3 .. 1.0 of 2^-50), so the bound may not pass
//     2^48 (largest error seen 0.19; 24 bits at N = 2^16 take three limbs).
// The bound does not depend on what the caller's own plan would hold.
static bool exact_plan(int n_power, int B, bool centred, int* w_out, int* k_out)
{
    const double rb = std::ldexp(1.0, B) / std::sqrt(3.0), cen = centred ? std::ldexp(1.0, B) : 0.0;
    const double model = 7.1 * std::sqrt(std::ldexp(1.0, n_power)) * std::sqrt((double)(n_power - 1)) * std::ldexp(1.0, -53);
    for (int K = 1; K <= EXACT_MAX_LIMBS; K++)
    {
        double best = 0;
        int bw = 0;
        for (int w = 1; w <= (K > 1 ? 20 : 1); w++)
        {
            const int top = B - w * (K - 1);
            if (top < 0) continue;
            double worst = 0, mag = 0;
            for (int l = 0; l < K; l++)
            {
                const bool last = l == K - 1;
                const double da = std::ldexp(1.0, last ? top : w - 1), ra = da / std::sqrt(3.0);
                double e2 = ra * ra * (rb * rb + cen * cen);
                double g = da * (std::ldexp(1.0, B) + cen);
                if (last && centred)
                {
                    e2 += rb * rb * std::ldexp(1.0, 2 * top);
                    g += std::ldexp(1.0, top + B);
                }
                worst = std::max(worst, std::sqrt(e2));
                mag = std::max(mag, std::ldexp(g, n_power));
            }
            if (model * worst > 0.06 || mag > std::ldexp(1.0, 48)) continue;
            if (bw == 0 || worst < best)
            {
                best = worst;
                bw = w;
            }
        }
        if (bw == 0) continue;
        *w_out = bw;
        *k_out = K;
        return true;
    }
    return false;
}

template <int L, int K> static int launch_exact_cols(const ExactArgs& a, bool fwd, cudaStream_t s)
{
    constexpr int LS = exact_pair<L>() ? 2 : 1;
    const double M = (double)(2048LL << L);
    if (fwd)
    {
        const unsigned blocks = (unsigned)(2 * a.W * 2048 * LS / EXACT_COL_THREADS);
        GF_TRACE(tr, (double)a.W * M * (2 * 2 * 4 + (K + 1) * sizeof(cx<double>)), s, "exact_fwd_col<L%d,k%d>", L, K);
        return launch_k(exact_fwd_col<L, K>, blocks, EXACT_COL_THREADS, 0, s, a);
    }
    const unsigned blocks = (unsigned)(a.W * 2048 * LS / EXACT_COL_THREADS);
    GF_TRACE(tr, (double)a.W * M * (K * sizeof(cx<double>) + 2 * 8), s, "exact_inv_col<L%d,k%d>", L, K);
    return launch_k(exact_inv_col<L, K>, blocks, EXACT_COL_THREADS, 0, s, a);
}

constexpr size_t EXACT_SMEM = (size_t)(tile::SLOT + tile::TWN) * sizeof(cx<double>);

template <int K> static int launch_exact_tile(const ExactArgs& a, int m, cudaStream_t s)
{
    static int done[64] = {0};
    const int st = ensure_smem(exact_tile<K>, EXACT_SMEM, done);
    if (st) return st;
    const long long tiles = a.W << (m - 11);
    GF_TRACE(tr, (double)(a.W << m) * (2 * K + 1) * sizeof(cx<double>), s, "split_tile<f64,k%d>", K);
    return launch_k(exact_tile<K>, dim3((unsigned)tiles), dim3(tile::HT), EXACT_SMEM, s, a, m);
}

template <int m, int K, int BLOCKS> static int launch_exact_single_b(const ExactArgs& a, long long ctas, cudaStream_t s)
{
    using tl = TileOf<m == 12 ? 12 : 11>;
    static int done[64] = {0};
    const size_t smem = (size_t)(tl::SLOT + tl::TWN) * sizeof(cx<double>);
    const int st = ensure_smem(exact_single<m, K, BLOCKS>, smem, done);
    if (st) return st;
    GF_TRACE(tr, (double)(a.W << m) * (2 * 2 * 4 + 2 * 8), s, "exact_single<L%d,k%d>", m, K);
    return launch_k(exact_single<m, K, BLOCKS>, dim3((unsigned)ctas), dim3(tl::HT), smem, s, a);
}

template <int m, int K> static int launch_exact_single(const ExactArgs& a, cudaStream_t s)
{
    using tl = TileOf<m == 12 ? 12 : 11>;
    const long long ctas = ((a.W << m) + tl::P - 1) / tl::P;
    const bool two = K > 1 && (ctas <= 2LL * sm_count() || (K > 2 && ctas > 3LL * sm_count()));
    return two ? launch_exact_single_b<m, K, exact_single_blocks<m>(true)>(a, ctas, s)
               : launch_exact_single_b<m, K, exact_single_blocks<m>(false)>(a, ctas, s);
}

int split_exact(const int32_t* a, const int32_t* b, int64_t* c, int m, int batch, int input_bits, bool non_negative,
                const cx<double>* tables, void* ws, size_t ws_bytes, unsigned* max_err, cudaStream_t s)
{
    const long long M = 1LL << m;
    if (m < 4 || m > 16 || (reinterpret_cast<uintptr_t>(ws) & 15)) return -1;
    const int B = non_negative ? input_bits - 1 : input_bits;
    int w = 0, K = 0;
    if (!exact_plan(m + 1, B, non_negative, &w, &K)) return -1;
    const bool single = m <= 12;
    // one CTA runs its product's transforms in turn: up to 16 products of 4096-point
    // ones take the chain, which spreads them (16 products, two limbs 28.1 us against
    // 33.3, three 28.0 against 54). The chain stays ahead up to 30 products with two
    // limbs and 72 with three, but it does not hold every row (exact_plan): from 17 on
    // calls keep the form that does.
    if (m == 12 && K > 1 && batch <= 16) return -1;
    // the result is written while operands are still read
    const size_t in = (size_t)batch * 2 * M * sizeof(int32_t);
    auto apart = [&](const int32_t* x) {
        const char *px = reinterpret_cast<const char*>(x), *pc = reinterpret_cast<const char*>(c);
        return px + in <= pc || pc + 2 * in <= px;
    };
    if (!apart(a) || !apart(b)) return -1;
    ExactArgs A{};
    const size_t tab = tables ? 0 : (size_t)(M / 2 + 2 * M) * sizeof(cx<double>);
    const size_t per = single ? 0 : (size_t)(K + 1) * M * sizeof(cx<double>);
    if (ws_bytes < tab + per) return -1;
    long long W = single ? batch : (long long)((ws_bytes - tab) / per);
    if (W > batch) W = batch;
    // a wave with fewer tiles than SMs takes the limb chain (N = 2^16; at the line, ten
    // products, the two forms: one limb 26.5 against 46.5 us, two 42.0 / 46.5, three
    // 53.3 / 54.8; below it, four products: 21.7 / 33.6, 37.5 / 33.9, 48.0 / 37.5). One
    // limb would win there too; four lose up to six products of N = 2^17 (73 / 69 us).
    if (!single && (W << (m - 11)) < (long long)sm_count()) return -1;
    if (tables)
    {
        A.roots = tables;
        A.twist = tables + M;
        A.uspec = tables + 3 * M;
    }
    else
    {
        auto* t = static_cast<cx<double>*>(ws);
        GF_TRACE(tr, (double)tab, s, "exact_tables");
        const long long n = M / 2 + (non_negative ? 2 : 1) * M; // U serves centred inputs only
        const int st = launch_k(exact_tables_kernel, dim3((unsigned)((n + 127) / 128)), dim3(128), 0, s, t, m);
        if (st) return st;
        A.roots = t;
        A.twist = t + M / 2;
        A.uspec = t + M / 2 + M;
    }
    A.spec = reinterpret_cast<cx<double>*>(static_cast<char*>(ws) + tab);
    A.max_err = max_err;
    A.cen = non_negative ? 1LL << (input_bits - 1) : 0;
    A.voff = -A.cen;
    for (int l = 0; l + 1 < K; l++) A.voff += 1LL << (w * l + w - 1);
    A.ushift = (double)A.cen / std::ldexp(1.0, w * (K - 1));
    A.scale = 1.0 / (double)M;
    A.w = w;
    for (long long p0 = 0; p0 < batch; p0 += W)
    {
        A.a = a + p0 * 2 * M;
        A.b = b + p0 * 2 * M;
        A.c = c + p0 * 2 * M;
        A.W = (batch - p0) < W ? (batch - p0) : W;
        int st;
        if (single)
        {
            st = dispatch_int<4, 12>(m, [&]<int MM>() {
                return dispatch_int<1, EXACT_MAX_LIMBS>(K, [&]<int KK>() { return launch_exact_single<MM, KK>(A, s); });
            });
            if (st) return st;
            continue;
        }
        auto cols = [&](bool fwd) {
            return dispatch_int<2, 5>(m - 11, [&]<int L>() {
                return dispatch_int<1, EXACT_MAX_LIMBS>(K, [&]<int KK>() { return launch_exact_cols<L, KK>(A, fwd, s); });
            });
        };
        st = cols(true);
        if (st) return st;
        st = dispatch_int<1, EXACT_MAX_LIMBS>(K, [&]<int KK>() { return launch_exact_tile<KK>(A, m, s); });
        if (st) return st;
        st = cols(false);
        if (st) return st;
    }
    return GPUFFT_SUCCESS;
}
} // namespace gfb

// The kernels of the exact product have no waits of their own any more; the entry
// point stays for callers that check it.
extern "C" int gpufft_split_wait_timeouts(unsigned* count, int clear)
{
    (void)clear;
    if (!count) return GPUFFT_ERROR_INVALID_VALUE;
    *count = 0;
    return GPUFFT_SUCCESS;
}
