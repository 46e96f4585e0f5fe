// gpufft-b200: launcher of the tile passes (gf_tile_pass.cuh), compiled once per
// data type.
#pragma once

#include "gf_tile_pass.cuh"

namespace gfb
{
template <typename T, bool FWD, int LT, int IK, int OK> static int launch_tile_pass_k(const PassArgs<T>& a, cudaStream_t s)
{
    using tl = TilePass<LT>;
    const size_t smem = (size_t)(tl::SLOT + tl::TWN) * sizeof(cx<T>);
    static int done[64] = {0};
    const int st = ensure_smem(tile_pass_kernel<T, FWD, LT, IK, OK>, smem, done);
    if (st) return st;
    const long long units = a.batch << (a.geo.m - LT);
    const long long slots = (long long)sm_count() * tile_pass_blocks<T, LT>();
    GF_TRACE(tr, pass_alg_bytes(a), s, "tile_pass<%s,%s,L%d,in%d,out%d>", sizeof(T) == 4 ? "f32" : "f64",
             kind_name(FWD), LT, IK, OK);
    return launch_k(tile_pass_kernel<T, FWD, LT, IK, OK>, dim3((unsigned)(units < slots ? units : slots)), dim3(tl::HT),
                    smem, s, a);
}

template <typename T, int LT> static int launch_tile_pass_lt(const PassArgs<T>& a, bool fwd, cudaStream_t s)
{
    const bool whole = a.geo.m == LT;
    if (a.perm || (a.zero_pad && a.in_kind != IN_REAL)) return -1;
    if (fwd)
    {
        if (a.out_kind != OUT_CPX) return -1;
        if (a.do_scale) return -1;
        if (a.in_kind == IN_CPX) return launch_tile_pass_k<T, true, LT, IN_CPX, OUT_CPX>(a, s);
        if (!whole) return -1;
        if (a.in_kind == IN_FOLD) return launch_tile_pass_k<T, true, LT, IN_FOLD, OUT_CPX>(a, s);
        if (a.in_kind == IN_REAL) return launch_tile_pass_k<T, true, LT, IN_REAL, OUT_CPX>(a, s);
        return -1;
    }
    if (a.in_kind != IN_CPX && a.in_kind != IN_PROD) return -1;
    const bool prod = a.in_kind == IN_PROD;
    if (a.out_kind == OUT_CPX)
        return prod ? launch_tile_pass_k<T, false, LT, IN_PROD, OUT_CPX>(a, s)
                    : launch_tile_pass_k<T, false, LT, IN_CPX, OUT_CPX>(a, s);
    if (!whole) return -1;
    if (a.out_kind == OUT_UNFOLD)
        return prod ? launch_tile_pass_k<T, false, LT, IN_PROD, OUT_UNFOLD>(a, s)
                    : launch_tile_pass_k<T, false, LT, IN_CPX, OUT_UNFOLD>(a, s);
    if (a.out_kind == OUT_REAL)
        return prod ? launch_tile_pass_k<T, false, LT, IN_PROD, OUT_REAL>(a, s)
                    : launch_tile_pass_k<T, false, LT, IN_CPX, OUT_REAL>(a, s);
    return -1;
}

template <typename T> static int launch_tile_pass_t(const PassArgs<T>& a, bool fwd, int LT, cudaStream_t s)
{
    if (LT == 11) return launch_tile_pass_lt<T, 11>(a, fwd, s);
    if (LT == 12) return launch_tile_pass_lt<T, 12>(a, fwd, s);
    return -1;
}
} // namespace gfb
