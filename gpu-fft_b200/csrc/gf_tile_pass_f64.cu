// gpufft-b200: the FP64 tile passes (gf_tile_pass.cuh).
#include "gf_tile_pass_launch.cuh"

namespace gfb
{
template <> int launch_tile_pass<double>(const PassArgs<double>& a, bool fwd, int LT, cudaStream_t s)
{
    return launch_tile_pass_t<double>(a, fwd, LT, s);
}
} // namespace gfb
