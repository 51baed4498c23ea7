// What the reverse-mode kernels share (kernels_adjoint.cu, kernels_fused.cu).
#pragma once
#include "step_common.cuh"

namespace virs {
namespace {

using namespace step;

// The reverse pass keeps subnormals outside its stencil (state adjoints and
// boundary terms of a loss gradient near the end of FP32's range), also where
// a kernel is compiled with -ftz=true for the forward step: a gradient with a
// loss gradient of 1e-34 was off by 2e-3 of its largest value with them
// flushed, and is by 2e-4 (the stencil's flushes) with them kept.  The forward
// states and the coefficients hold none and are converted plainly (through
// these too, a gradient over 256 steps of 128x128x96 took 4.24 instead of
// 4.15 ms; 4.13 with everything flushed).
namespace keep {
__device__ __forceinline__ double wide(float v)
{
    double d;
    asm("cvt.f64.f32 %0, %1;" : "=d"(d) : "f"(v));
    return d;
}
__device__ __forceinline__ float narrow(double v)
{
    float f;
    asm("cvt.rn.f32.f64 %0, %1;" : "=f"(f) : "d"(v));
    return f;
}
__device__ __forceinline__ float add(float a, float b)
{
    float r;
    asm("add.rn.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float sub(float a, float b)
{
    float r;
    asm("sub.rn.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float mul(float a, float b)
{
    float r;
    asm("mul.rn.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float fma(float a, float b, float c)
{
    float r;
    asm("fma.rn.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
} // namespace keep

// the transposed correction of one slot: the value F left in the adjoint
// field, the cascade output's adjoint and what dbar and RR' take beyond it
struct AdjCorr {
    double fr, ybar, db, cq;
};
// kg: K * gain
__device__ __forceinline__ AdjCorr adj_correct(const BndWeight *wtab, int form, double kg, double mix_y, double mix_d,
                                               float t, uint32_t meta)
{
    const double f = keep::wide(t);
    const BndWeight e = wtab[meta >> 16];
    AdjCorr c;
    if (form == VIRS_BOUNDARY_REFERENCE) {
        const double kgw = kg * e.kgw; // the weight itself
        c.fr = f;
        c.ybar = -kgw * mix_y * f;
        c.db = -kgw * mix_d * f;
        c.cq = 0.0;
    } else {
        c.fr = quotient(f, e.den, e.rden);
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
