// IR post-processing on the GPU: the receiver traces recorded at the
// simulation rate 1/dt become output-rate signals.
//
// The reference does this on the host after the step loop
// (simulator.cpp:1029-1080): a library resampler (kfr) to 48 kHz, then
// division by the peak magnitude.  Here, per receiver channel:
//   k_ir_sos       the anti-alias cascade of second-order sections in FP64,
//                  transposed direct form II (the recursion of
//                  src/util/downsampling_filter_iir.cpp:210-240), as a
//                  systolic warp: lane s owns section s and its two states,
//                  and at tick t it filters sample t - 2 s, its input being
//                  lane s-1's output of two ticks before (a shuffle); the
//                  last lane's output is the filtered sample.  A chain of
//                  four dependent FP64 operations per sample bounds it (y to
//                  the first state to the next y), so the shuffle's latency
//                  is kept off it: with one tick per lane it was on it
//   k_ir_resample  linear interpolation at k / rate (simulator.cpp:1046-1057),
//                  then, if asked, division by the channel's peak
// Every product and sum is written with _rn intrinsics in the CPU
// recursion's order (no contraction), so the result is bit for bit the
// oracle's.
#include "internal.hpp"

namespace virs {
namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int CHUNK = 1024; // input samples staged per round of ticks

// One tick of a lane: the recursion's operations in its order.
struct Sos {
    double b0, b1, b2, a1, a2, z1, z2;
    __device__ __forceinline__ double tick(double v)
    {
        const double yo = __dadd_rn(__dmul_rn(b0, v), z1);
        z1 = __dadd_rn(__dsub_rn(__dmul_rn(b1, v), __dmul_rn(a1, yo)), z2);
        z2 = __dsub_rn(__dmul_rn(b2, v), __dmul_rn(a2, yo));
        return yo;
    }
};

// 4000 samples of 8 channels through 6 sections: 449 us with one tick per
// lane and per-tick range tests, 150 us in this form.
__global__ void __launch_bounds__(32) k_ir_sos(const float *__restrict in, uint64_t in_stride, uint64_t len,
                                               const double *__restrict sos, int ns, float *__restrict out,
                                               uint64_t out_stride)
{
    __shared__ float xin[CHUNK];
    const int lane = threadIdx.x;
    const float *x = in + blockIdx.x * in_stride;
    Sos f{0, 0, 0, 0, 0, 0, 0};
    if (lane < ns) {
        const double *s = sos + 6 * lane;
        f.b0 = s[0]; f.b1 = s[1]; f.b2 = s[2]; f.a1 = s[4]; f.a2 = s[5];
    }
    const uint64_t skew = 2u * (uint64_t)(ns - 1), ticks = len + skew;
    const bool last = lane == ns - 1;
    float *y = out + blockIdx.x * out_stride; // the last lane's next output
    double in1 = 0.0, in2 = 0.0;              // lane s-1's outputs of the last tick and of the one before
    for (uint64_t c0 = 0; c0 < ticks; c0 += CHUNK) {
        __syncwarp();
        for (int i = lane; i < CHUNK; i += 32) {
            const uint64_t t = c0 + (uint64_t)i;
            xin[i] = t < len ? x[t] : 0.f;
        }
        __syncwarp();
        const int m = ticks - c0 < (uint64_t)CHUNK ? (int)(ticks - c0) : CHUNK;
        int i = 0;
        // until every lane has begun (at most 62 ticks: inside the first
        // chunk): a lane waits for its first sample.  Afterwards a lane that
        // runs past the last sample computes values that nobody reads.
        if (c0 == 0)
            for (; i < m && i < (int)skew; ++i) {
                const double v = lane == 0 ? (double)xin[i] : in2;
                double yo = 0.0;
                if (i >= 2 * lane) yo = f.tick(v);
                in2 = in1;
                in1 = __shfl_up_sync(FULL, yo, 1);
            }
#pragma unroll 4
        for (; i < m; ++i) {
            const double v = lane == 0 ? (double)xin[i] : in2;
            const double yo = f.tick(v);
            in2 = in1;
            in1 = __shfl_up_sync(FULL, yo, 1);
            if (last) *y = __double2float_rn(yo);
            ++y;
        }
    }
}

constexpr int RB = 256;

// one block per channel (the peak); 1024 threads: 13 us with 256 at 5049 samples
constexpr int LB = 1024;

__global__ void __launch_bounds__(LB) k_ir_resample(const float *__restrict in, uint64_t in_stride, uint64_t len,
                                                    double sim_rate, float rate, float *__restrict out,
                                                    uint64_t out_len, int normalize)
{
    __shared__ float red[LB / 32];
    const float *f = in + blockIdx.x * in_stride;
    float *o = out + blockIdx.x * out_len;
    float peak = 0.f;
    for (uint64_t k = threadIdx.x; k < out_len; k += LB) {
        const float t = __fdiv_rn((float)k, rate);
        const float index = __double2float_rn(__dmul_rn((double)t, sim_rate));
        uint64_t lo = (uint64_t)floorf(index);
        if (lo >= len) lo = len - 1;
        const uint64_t hi = lo + 1 < len ? lo + 1 : lo;
        const float frac = __fsub_rn(index, (float)lo);
        const float v = __fadd_rn(__fmul_rn(f[lo], __fsub_rn(1.f, frac)), __fmul_rn(f[hi], frac));
        o[k] = v;
        peak = fmaxf(peak, fabsf(v));
    }
    if (!normalize) return;
    for (int s = 16; s > 0; s >>= 1) peak = fmaxf(peak, __shfl_xor_sync(FULL, peak, s));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x / 32] = peak;
    __syncthreads();
    peak = 0.f;
    for (int w = 0; w < LB / 32; ++w) peak = fmaxf(peak, red[w]);
    if (!(peak > 0.f)) return; // a silent channel stays zero
    for (uint64_t k = threadIdx.x; k < out_len; k += LB) o[k] = __fdiv_rn(o[k], peak);
}

// Band-limited resampling with a Kaiser-windowed sinc: output sample k is
// at input position t = k * fs_in / rate; y_k = sum over the input samples
// n with |t - n| < half of x[n] * 2 fc sinc(2 fc (t - n)) * w(t - n), with
// fc = cutoff * min(fs_in, rate) / 2 / fs_in (cycles per input sample),
// sinc(u) = sin(pi u) / (pi u) and the Kaiser window
// w(tau) = I0(beta sqrt(1 - (tau / half)^2)) / I0(beta).  FP64 throughout.
//
// The weights are the work (channels share them): a warp takes one output
// sample of up to CH channels (G = 32), its lanes every G-th tap.  The window is the
// power series of I0 in 1 - (tau / half)^2 itself, sum_k c_k v^k with
// c_k = (beta / 2)^(2k) / (k!)^2 / I0(beta) (all terms positive: no
// cancellation), from the kernel's parameters; the sine of
// a lane's next tap follows from the last by the rotation by G taps, except
// near tau = 0, where its relative error would matter.  8 channels, 4000 to
// 5049 samples, 490 taps: 1463 us with the series, a sine and a division per
// tap and channel, one output per thread; 46 us in this form (two chains of
// half the length, odd and even powers, were no faster: the FP64 rate bounds
// it, not the chain).  Short windows leave most of 32 lanes idle, and the sums
// over the lanes become the work: there four lanes take a sample, a warp
// eight (8 channels, 6300 samples, 2 to 32 taps: 213 to 250 us a call with a
// thread per output and channel, 257 with a warp, 176 with four lanes; 1000
// channels, 2 taps: 2.9, 3.9 and 2.2 ms).
constexpr int CH = 8;            // channels per warp
constexpr int SINC_TERMS = 128;  // of the series (beta <= 50 needs 80)
struct SincArgs {
    double step_ratio, fc2, inv_half, rot_s, rot_c; // sine and cosine of pi * fc2 * G
    int half, terms;
    double c[SINC_TERMS];
};

// G: the lanes of an output sample
template <int G>
__global__ void __launch_bounds__(RB) k_ir_sinc(const float *__restrict in, uint64_t in_stride, uint64_t len,
                                                const __grid_constant__ SincArgs a, float *__restrict out,
                                                uint64_t out_len, uint32_t channels, uint32_t *__restrict peak)
{
    // the series' coefficients, two per load (indexed reads of the parameters
    // are served one at a time: 49 us)
    __shared__ double2 cf[SINC_TERMS / 2];
    for (int j = threadIdx.x; j < SINC_TERMS / 2; j += RB)
        cf[j] = make_double2(2 * j < a.terms ? a.c[2 * j] : 0.0, 2 * j + 1 < a.terms ? a.c[2 * j + 1] : 0.0);
    __syncthreads();
    const int lane = threadIdx.x & (G - 1), pairs = (a.terms + 1) / 2;
    const uint64_t kg = (uint64_t)blockIdx.x * (RB / G) + threadIdx.x / G;
    if (G == 32 && kg >= out_len) return;                // the whole warp
    const uint64_t k = kg < out_len ? kg : out_len - 1;  // idle groups repeat the last sample, unstored
    const uint32_t c0 = blockIdx.y * CH, nc = min(channels - c0, (uint32_t)CH);
    const float *f = in + (uint64_t)c0 * in_stride;
    const double t = (double)k * a.step_ratio;
    const double n0 = fmax(0.0, ceil(t - (double)a.half)), n1 = fmin((double)len - 1.0, floor(t + (double)a.half));
    double acc[CH];
#pragma unroll
    for (int c = 0; c < CH; ++c) acc[c] = 0.0;
    double sn, cs;
    sincospi(a.fc2 * (t - (n0 + (double)lane)), &sn, &cs);
    for (double n = n0 + (double)lane; n <= n1; n += (double)G) {
        const double tau = t - n, u = tau * a.inv_half, x = a.fc2 * tau;
        const double s = fabs(x) < 0.5 ? sinpi(x) : sn;
        // sin(x - d) and cos(x - d) for the next tap
        const double s2 = sn * a.rot_c - cs * a.rot_s;
        cs = cs * a.rot_c + sn * a.rot_s;
        sn = s2;
        if (!(fabs(tau) < (double)a.half)) continue; // not |u| < 1: 49 * (1 / 49) rounds below 1
        const double v = 1.0 - u * u;
        double w = 0.0;
#pragma unroll 4
        for (int j = pairs - 1; j >= 0; --j) {
            const double2 c = cf[j];
            w = fma(fma(w, v, c.y), v, c.x);
        }
        w *= tau == 0.0 ? a.fc2 : s / (M_PI * tau);
        const float *fn = f + (uint64_t)n;
#pragma unroll
        for (int c = 0; c < CH; ++c)
            if (c < (int)nc) acc[c] += (double)fn[(uint64_t)c * in_stride] * w;
    }
#pragma unroll
    for (int c = 0; c < CH; ++c) {
        if (c >= (int)nc) break;
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) acc[c] += __shfl_xor_sync(FULL, acc[c], o);
        if (lane == 0 && kg < out_len) {
            const float v = (float)acc[c];
            out[(uint64_t)(c0 + c) * out_len + k] = v;
            if (peak) atomicMax(peak + c0 + c, __float_as_uint(fabsf(v))); // non-negative floats order as integers
        }
    }
}

__global__ void k_ir_normalize(float *__restrict out, uint64_t out_len, const uint32_t *__restrict peak)
{
    const uint64_t k = (uint64_t)blockIdx.x * RB + threadIdx.x;
    const float p = __uint_as_float(peak[blockIdx.y]);
    if (k < out_len && p > 0.f) out[blockIdx.y * out_len + k] = __fdiv_rn(out[blockIdx.y * out_len + k], p);
}

} // namespace

cudaError_t launch_ir_sinc(const float *in, uint64_t in_stride, uint64_t len, double fs_in, double rate, int half,
                           double beta, double cutoff, float *out, uint64_t out_len, uint32_t *peak, uint32_t channels,
                           cudaStream_t s)
{
    if (!channels || !out_len || !len) return cudaSuccess;
    SincArgs a;
    a.step_ratio = fs_in / rate;
    a.fc2 = cutoff * fmin(fs_in, rate) / fs_in; // 2 fc
    a.half = half;
    a.inv_half = 1.0 / (double)half;
    // Four lanes per output sample for short windows, as long as those fill
    // the device (one channel of 380 samples, 32 taps: 41 us with 32 lanes, 44
    // with four; of 6300 samples, 64 taps: 70 and 70, 128 taps 77 and 81).
    const uint64_t warps = out_len * ((channels + CH - 1) / CH);
    const int G = half <= 32 && warps >= 4096 ? 4 : 32;
    const double turn = fmod((double)G * a.fc2, 2.0);
    a.rot_s = sin(M_PI * turn);
    a.rot_c = cos(M_PI * turn);
    // I0(beta) and the window's coefficients, as many as change the sum
    const double q = 0.25 * beta * beta;
    double term = 1.0, i0b = 1.0;
    a.c[0] = 1.0;
    a.terms = 1;
    for (int k = 1; k < SINC_TERMS; ++k) {
        term = term * q / ((double)k * (double)k);
        if (term < 1e-18 * i0b) break;
        i0b += term;
        a.c[k] = term;
        a.terms = k + 1;
    }
    for (int k = 0; k < a.terms; ++k) a.c[k] /= i0b;
    const unsigned per = (unsigned)(RB / G); // output samples per block
    const dim3 g((unsigned)((out_len + per - 1) / per), (channels + CH - 1) / CH);
    if (peak) {
        cudaError_t e = cudaMemsetAsync(peak, 0, channels * sizeof(uint32_t), s);
        if (e != cudaSuccess) return e;
    }
    (G == 4 ? k_ir_sinc<4> : k_ir_sinc<32>)<<<g, RB, 0, s>>>(in, in_stride, len, a, out, out_len, channels, peak);
    if (peak)
        k_ir_normalize<<<dim3((unsigned)((out_len + RB - 1) / RB), channels), RB, 0, s>>>(out, out_len, peak);
    return cudaGetLastError();
}

cudaError_t launch_ir_sos(const float *in, uint64_t in_stride, uint64_t len, const double *sos, int ns, float *out,
                          uint64_t out_stride, uint32_t channels, cudaStream_t s)
{
    if (!channels || !len || ns < 1) return cudaSuccess;
    k_ir_sos<<<channels, 32, 0, s>>>(in, in_stride, len, sos, ns, out, out_stride);
    return cudaGetLastError();
}

cudaError_t launch_ir_resample(const float *in, uint64_t in_stride, uint64_t len, double sim_rate, float rate,
                               float *out, uint64_t out_len, int normalize, uint32_t channels, cudaStream_t s)
{
    if (!channels || !out_len || !len) return cudaSuccess;
    k_ir_resample<<<channels, LB, 0, s>>>(in, in_stride, len, sim_rate, rate, out, out_len, normalize);
    return cudaGetLastError();
}

} // namespace virs
