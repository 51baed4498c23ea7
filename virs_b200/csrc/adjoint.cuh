// What the reverse-mode kernels share (kernels_adjoint.cu, kernels_fused.cu).
#pragma once
#include "step_common.cuh"

namespace virs {
namespace {

using namespace step;

// the transposed correction of one slot: the value F left in the adjoint
// field, the cascade output's adjoint and what dbar and RR' take beyond it
struct AdjCorr {
    double fr, ybar, db, cq;
};
// kg: K * gain
__device__ __forceinline__ AdjCorr adj_correct(const BndWeight *wtab, int form, double kg, double mix_y, double mix_d,
                                               float f, uint32_t meta)
{
    const BndWeight e = wtab[meta >> 16];
    AdjCorr c;
    if (form == VIRS_BOUNDARY_REFERENCE) {
        const double kgw = kg * e.kgw; // the weight itself
        c.fr = f;
        c.ybar = -kgw * mix_y * f;
        c.db = -kgw * mix_d * f;
        c.cq = 0.0;
    } else {
        c.fr = quotient((double)f, e.den, e.rden);
        c.ybar = -e.kgw * mix_y * c.fr;
        c.db = 0.0;
        c.cq = e.ac * c.fr;
    }
    return c;
}
// The sums of v[0..N) over a warp (N a power of two): each exchange halves
// the values a lane holds, so N values cost N - 1 + log2(32 / N) shuffles
// instead of 5 N.  Returns the sum of value *idx, the same on every lane of
// a group of 32 / N.
template <int N> __device__ __forceinline__ double warp_sums(double (&v)[N], int *idx)
{
    const int lane = (int)(threadIdx.x & 31u);
    int k = 0;
    int n = N;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (n > 1) {
            n /= 2;
            const bool up = (lane & o) != 0;
#pragma unroll
            for (int j = 0; j < N / 2; ++j)
                if (j < n) {
                    const double give = up ? v[j] : v[j + n], keep = up ? v[j + n] : v[j];
                    v[j] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                }
            k += up ? n : 0;
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        }
    }
    *idx = k;
    return v[0];
}

} // namespace
} // namespace virs
