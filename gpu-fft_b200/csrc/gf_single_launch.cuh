// gpufft-b200: launcher of the one-kernel products (gf_single.cuh), compiled once per
// data type.
#pragma once

#include "gf_single.cuh"

namespace gfb
{
template <typename T, int m, int KIND> static int launch_single_k(const SingleArgs<T>& a, cudaStream_t s)
{
    using tl = TileOf<m == 12 ? 12 : 11>;
    static int done[64] = {0};
    const size_t smem = (size_t)(tl::SLOT + tl::TWN) * sizeof(cx<T>);
    const int st = ensure_smem(single_kernel<T, m, KIND>, smem, done);
    if (st) return st;
    const long long tiles = ((a.batch << m) + tl::P - 1) / tl::P;
    const long long slots = (long long)sm_count() * single_blocks<T, m>();
    static const char* const names[] = {"neg", "lin", "cyc", "vjp"};
    static const double per_point[] = {6, 4, 6, 6}; // reals in and out per point
    GF_TRACE(tr, (double)(a.batch << m) * per_point[KIND] * sizeof(T), s, "single<%s,%s,L%d>",
             sizeof(T) == 4 ? "f32" : "f64", names[KIND], m);
    return launch_k(single_kernel<T, m, KIND>, dim3((unsigned)(tiles < slots ? tiles : slots)), dim3(tl::HT), smem, s, a);
}
} // namespace gfb
