// gpufft-b200: launchers of the 2048-point tile product kernel (gf_tile.cuh).
#include "gf_tile.cuh"

namespace gfb
{
template <typename T, int MODE> int launch_tile_product(const TileArgs<T>& a, long long tiles, cudaStream_t s)
{
    if (tiles <= 0) return GPUFFT_SUCCESS;
    if (tiles > 0x7fffffffLL) return GPUFFT_ERROR_INVALID_VALUE;
    static int done[64] = {0};
    const size_t smem = (size_t)(tile::SLOT + tile::TWN) * sizeof(cx<T>);
    const int st = ensure_smem(tile_product_kernel<T, MODE>, smem, done);
    if (st) return st;
    // the parked operand and every other one in, every result out
    const int nops = MODE == TILE_VJP ? 2 : 1;
    GF_TRACE(tr, (double)tiles * tile::P * (1 + 2 * nops) * sizeof(cx<T>), s, "tile_product<%s,%s>",
             sizeof(T) == 4 ? "f32" : "f64", MODE == TILE_VJP ? "vjp" : "mul");
    return launch_k(tile_product_kernel<T, MODE>, dim3((unsigned)tiles), dim3(tile::HT), smem, s, a);
}

template int launch_tile_product<double, TILE_MUL>(const TileArgs<double>&, long long, cudaStream_t);
template int launch_tile_product<float, TILE_MUL>(const TileArgs<float>&, long long, cudaStream_t);
template int launch_tile_product<float, TILE_VJP>(const TileArgs<float>&, long long, cudaStream_t);
} // namespace gfb
