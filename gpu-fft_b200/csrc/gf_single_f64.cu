// gpufft-b200: the FP64 one-kernel products (gf_single.cuh).
#include "gf_single_launch.cuh"

namespace gfb
{
template <> int launch_single<double>(int kind, int m, const SingleArgs<double>& a, cudaStream_t s)
{
    return dispatch_int<4, 12>(m, [&]<int MM>() {
        switch (kind)
        {
        case SINGLE_NEG: return launch_single_k<double, MM, SINGLE_NEG>(a, s);
        case SINGLE_LIN: return launch_single_k<double, MM, SINGLE_LIN>(a, s);
        case SINGLE_CYC: return launch_single_k<double, MM, SINGLE_CYC>(a, s);
        default: return (int)GPUFFT_ERROR_INVALID_VALUE;
        }
    });
}
} // namespace gfb
