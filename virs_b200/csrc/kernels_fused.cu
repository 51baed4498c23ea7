// One launch per step for grids whose fields stay near the L2: the stencil,
// the boundary pass and the sources and receivers together.
//
// On such grids a step of three launches (stencil, boundary pass, post) is
// bound by latency: each kernel runs for a few microseconds, most of them
// ramp-up, dependent loads and the gap to the next launch.  The three parts
// do not need that order:
//   * the boundary pass reads p^n, and p^{n-1} and the states of its own
//     voxel, so it can run beside the stencil as long as the stencil stores
//     nothing at boundary voxels (a vector that holds some is stored voxel
//     by voxel);
//   * a hard-source voxel takes its value in the stencil;
//   * a soft source adds to, and a receiver reads, one voxel of p^{n+1}: the
//     block that wrote it does that after its own barrier (the probe list
//     says which block that is), so no grid-wide order is needed;
//   * the step counter alternates between two words (step n reads word
//     parity, writes the other), so no block has to be the last.
// Blocks [0, gb) take 256 * PL boundary slots each, the others 256 vectors of
// four voxels of PL consecutive planes.  The planes are walked as one row of
// px * ny voxels: the y neighbours are px further on, no tile hangs over the
// grid's edge, and what the row ends mix up are border voxels, whose result
// is not kept.  Every load of a thread is independent of the others and
// issued before any arithmetic: the latency is paid once.  Two planes and two
// slots per thread (PL = 2) share the block's fixed costs and a plane of
// loads; one (PL = 1) where that would leave SMs idle (fused_geo).
//
// Consecutive steps overlap at their ends (programmatic dependent launch):
// a block loads what no step writes (codes, boundary positions, its probe
// flag), then waits for the previous step's grid.
//
// 160x120x100 voxels with a sponge of 8 (0.64 M boundary slots): 17.4 us a
// step in three launches, 10.4 with one plane and slot per thread, 8.8 now;
// 300x200x130 with a sponge of 1: 28.6, 24.4 and 19.0.  Where the lines to the
// staged kernels lie: fused_on and batch_fused in capi.cpp.
#include <algorithm>
#include <type_traits>

#include "adjoint.cuh"
#include "pdl.cuh"
#include "step_voxel.cuh"

namespace virs {
namespace {

using namespace step;

constexpr int FB = 256;

// Four voxels of a row in one load: 16 bytes in FP32, 8 in 16-bit storage
// (eight per thread would need 77 registers, too few warps for this kernel).
constexpr int V = 4;
template <typename T> struct Vec {
    using Raw = std::conditional_t<sizeof(T) == 4, uint4, uint2>;
    Raw v;
    __device__ void load(const T *p) { v = *reinterpret_cast<const Raw *>(p); }
    __device__ void get(float (&r)[V]) const
    {
        const T *h = reinterpret_cast<const T *>(&v);
#pragma unroll
        for (int k = 0; k < V; ++k) r[k] = Io<T>::get(h[k]);
    }
};

// rounded and stored; SR: stochastically (pos is a multiple of four)
template <typename T, bool SR>
__device__ __forceinline__ void put4(T *p, const float (&r)[V], uint64_t pos, uint64_t base, uint32_t key)
{
    typename Vec<T>::Raw raw;
    if constexpr (SR) {
        uint32_t v[2];
        sr_pack<T>(r, pos, base, key, v);
        raw = make_uint2(v[0], v[1]);
    } else {
        T *h = reinterpret_cast<T *>(&raw);
#pragma unroll
        for (int k = 0; k < V; ++k) h[k] = Io<T>::put(r[k]);
    }
    *reinterpret_cast<typename Vec<T>::Raw *>(p) = raw;
}

// the block with number blk: a boundary block or one of the stencil's
struct Site {
    uint32_t bx, z;
};
__device__ __forceinline__ Site stencil_site(uint32_t blk, const FusedGeo &g)
{
    const uint32_t s = blk - g.gb, bz = g.magic ? __umulhi(s, g.magic) : s / g.gx;
    return {s - bz * g.gx, 1u + bz * g.pl};
}

// the probe list towards the L1 of a block that will go through it
__device__ __forceinline__ void prefetch_probes(const Probe *probe, uint32_t n)
{
    if (threadIdx.x < n) asm volatile("prefetch.global.L1 [%0];" ::"l"(probe + threadIdx.x));
}

// Sources and receivers at the voxels this block wrote, as post_body
// (kernels_step.cu) does for all of them; only blocks with a probe come here.
template <typename T> __device__ __forceinline__ void post_owned(const PostArgs &po, uint32_t blk, uint32_t sn)
{
    using IO = Io<T>;
    __syncthreads(); // every store of this block is visible to it
    T *Q = static_cast<T *>(po.q);
    const uint32_t k1 = po.sr ? sr_step_key(sn, 1u) : 0u;
    for (uint32_t k = threadIdx.x; k < po.nsrc; k += FB) {
        const Probe p = po.probe[k];
        if (p.blk != blk) continue;
        const float v = sn < po.siglen ? po.sig[(uint64_t)k * po.siglen + sn] : 0.f;
        Q[p.pos] = put_rounded<T>(__fadd_rn(IO::get(Q[p.pos]), v), po.sr, p.pos, po.sr_base, k1);
    }
    __syncthreads();
    if (sn >= po.cap) return;
    for (uint32_t k = threadIdx.x; k < po.nrcv; k += FB) {
        const Probe p = po.probe[po.nsrc + k];
        if (p.blk != blk) continue;
        const float v = __fmul_rn(IO::get(Q[p.pos]), po.inv_scale);
        po.ir[(uint64_t)k * po.cap + sn] = v;
        if (k == 0 && po.host0) *po.host0 = v;
    }
}

// out of line for PL = 2, whose registers it would take
template <typename T> __device__ __noinline__ void post_owned_call(const PostArgs &po, uint32_t blk)
{
    post_owned<T>(po, blk, *po.ctr);
}

// the loads of the PL vectors at plane offset o of planes z .. z + PL - 1 (the
// last block of an odd number of planes repeats its first plane, unstored)
template <typename T, int PL> struct StencilVecs {
    uint32_t i[PL];        // positions
    Codes<V> code[PL];
    Vec<T> c[PL + 2], yp[PL], ym[PL], q[PL]; // c: planes z - 1 .. z + PL
    float left[PL], right[PL];

    __device__ __forceinline__ void site(const StepArgs &a, uint32_t z, uint32_t o, uint32_t plane)
    {
#pragma unroll
        for (int k = 0; k < PL; ++k) {
            i[k] = (z + k < a.nz - 1u ? z + k : z) * plane + o;
            code[k].load(a.code + i[k]);
        }
    }
    __device__ __forceinline__ void values(const StepArgs &a, uint32_t plane)
    {
        using IO = Io<T>;
        const T *P = static_cast<const T *>(a.p);
        const T *Q = static_cast<const T *>(a.q);
        c[0].load(P + (i[0] - plane));
        c[1].load(P + i[0]);
#pragma unroll
        for (int k = 0; k < PL; ++k) {
            const T *p = P + i[k];
            c[k + 2].load(p + plane); // the plane after an unstored one: as the one after the first
            ym[k].load(p - a.px);
            yp[k].load(p + a.px);
            q[k].load(Q + i[k]);
            left[k] = IO::ld1(p - 1);
            right[k] = IO::ld1(p + V);
        }
    }
};

template <typename T, int PL, bool SR, bool EACH = false>
__device__ __forceinline__ void stencil_update(const StepArgs &a, const StencilVecs<T, PL> &s, bool act, uint32_t z)
{
    using IO = Io<T>;
    T *Q = static_cast<T *>(a.q);
    const float2 c2dt2 = make_float2(a.c2dt2, a.c2dt2), inv_h2 = make_float2(a.inv_h2, a.inv_h2);
    const uint32_t srk = SR ? sr_step_key(*a.ctr, 0u) : 0u;
#pragma unroll
    for (int k = 0; k < PL; ++k) {
        if (k > 0 && z + k >= a.nz - 1u) break;
        const Codes<V> &code = s.code[k];
        const uint32_t i = s.i[k];
        const float left = s.left[k], right = s.right[k];
        float fc[V], fzp[V], fzm[V], fyp[V], fym[V], fq[V], r[V];
        s.c[k].get(fzm);
        s.c[k + 1].get(fc);
        s.c[k + 2].get(fzp);
        s.ym[k].get(fym);
        s.yp[k].get(fyp);
        s.q[k].get(fq);
        air_update(fc, left, right, fyp, fym, fzp, fzm, fq, c2dt2, inv_h2, r);
        if (!act) continue;
        if (!code.any()) {
            put4<T, SR>(Q + i, r, i, a.sr_base, srk);
            continue;
        }
        // Border voxels keep their value and boundary voxels belong to the
        // blocks of their slots, so the others, air and walls (0), are stored
        // one by one.  The row ends put such vectors in every warp of a
        // room, so the rare codes are sought in all four bytes at once (bit 7
        // of each byte): per step 300x200x130 FP32 21.5 -> 19.0 us,
        // 160x120x100 with a sponge of 8 9.43 -> 8.78, 24 rooms of 1.1 M
        // voxels in BF16 108 -> 99.  Not in FP32 batches (EACH), whose
        // registers are full: it spilled 20 bytes there (8 rooms of 4 M voxels
        // 141 -> 147 us).
        const uint32_t w = code.w, top = w & (w << 1); // top: bits 7 and 6 of the byte are set
        const uint32_t air = ~(((w & 0x7f7f7f7fu) + 0x7f7f7f7fu) | w);
        const uint32_t rare = ((top & ~(w << 6)) | (~w & ~air)) & 0x80808080u; // hard sources, mirror voxels
        if (!EACH && rare == 0u) {
#pragma unroll
            for (int j = 0; j < V; ++j) {
                const uint32_t cj = code.get(j);
                const float v = cj == 0u ? r[j] : 0.f;
                if (cj == 0u || cj == CODE_WALL)
                    Q[i + j] = SR ? Sr<T>::put(v, sr_bits((uint64_t)i + j, a.sr_base, srk)) : IO::put(v);
            }
            continue;
        }
        // only air next to a wall outside a boundary layer takes the mirror rule
        if (code.mirror()) {
#pragma unroll
            for (int j = 0; j < V; ++j)
                if (code.get(j) != 0u && code.get(j) < CODE_BND)
                    r[j] = leapfrog((uint8_t)code.get(j), fc[j], j == V - 1 ? right : fc[j + 1],
                                    j == 0 ? left : fc[j - 1], fyp[j], fym[j], fzp[j], fzm[j], fq[j], a.c2dt2, a.inv_h2);
        }
#pragma unroll
        for (int j = 0; j < V; ++j) {
            const uint32_t cj = code.get(j);
            if (cj == CODE_NONE || (cj & 0xC0u) == CODE_BND) continue;
            float v = r[j];
            if (cj == CODE_WALL) v = 0.f;
            else if (cj == CODE_HARD) {
                const uint32_t sn = *a.ctr;
                v = sn < a.nhard ? a.hard[sn] : 0.f;
            }
            Q[i + j] = SR ? Sr<T>::put(v, sr_bits((uint64_t)i + j, a.sr_base, srk)) : IO::put(v);
        }
    }
}

template <typename T, int PL, int MAXS, int MODE, bool SR, bool EACH = false>
__device__ __forceinline__ void fused_block(const StepArgs &a, const PostArgs &po, uint32_t blk, const FusedGeo &g)
{
    const uint32_t tid = threadIdx.x;
    const bool probes = __ldg(g.has_probe + blk) != 0;
    uint32_t sn = 0;
    if (blk < g.gb) {
        BVox<T, MAXS> v[PL];
        bool act[PL];
#pragma unroll
        for (int k = 0; k < PL; ++k) {
            const uint64_t s = ((uint64_t)blk * PL + k) * FB + tid;
            act[k] = s < a.nb;
            if (act[k]) bvox_site<T, MAXS>(a, s, v[k]);
        }
        if (PL == 1 && probes) prefetch_probes(po.probe, po.nsrc + po.nrcv);
        pdl_wait();
        if (PL == 1 && probes) sn = *po.ctr;
#pragma unroll
        for (int k = 0; k < PL; ++k)
            if (act[k]) bvox_values<T, MAXS>(a, ((uint64_t)blk * PL + k) * FB + tid, v[k]);
#pragma unroll
        for (int k = 0; k < PL; ++k)
            if (act[k]) bvox_update<T, MODE, MAXS>(a, ((uint64_t)blk * PL + k) * FB + tid, v[k]);
    } else {
        const Site st = stencil_site(blk, g);
        const uint32_t plane = a.px * a.ny, o = (st.bx * FB + tid) * V;
        const bool act = o < plane;
        StencilVecs<T, PL> s;
        s.site(a, st.z, act ? o : plane - V, plane); // the last block of a plane repeats its last vector, unstored
        if (PL == 1 && probes) prefetch_probes(po.probe, po.nsrc + po.nrcv);
        pdl_wait();
        if (PL == 1 && probes) sn = *po.ctr;
        s.values(a, plane);
        stencil_update<T, PL, SR, EACH>(a, s, act, st.z);
    }
    if (blk == 0 && tid == 0) *po.ctr_out = *po.ctr + 1u;
    if (probes) {
        if constexpr (PL == 1) post_owned<T>(po, blk, sn);
        else post_owned_call<T>(po, blk);
    }
}

// blocks per SM the register allocation must allow
template <int PL> constexpr int fused_min_blocks() { return PL == 1 ? 5 : 4; }

template <typename T, int PL, int MAXS, int MODE, bool SR>
__global__ void __launch_bounds__(FB, fused_min_blocks<PL>()) k_fused(const __grid_constant__ StepArgs a,
                                                                      const __grid_constant__ PostArgs po,
                                                                      const __grid_constant__ FusedGeo g)
{
    pdl_trigger();
    fused_block<T, PL, MAXS, MODE, SR>(a, po, blockIdx.x, g);
}

// One step of the adjoint fields after the transposed correction
// (k_adj_boundary, kernels_adjoint.cu; cascades of more than four sections): the stencil T' = A F - RR (F in a.p, RR and then T'
// in a.q), at a boundary slot T' = (the mirrored leapfrog on F with the
// slot's own RR) + dbar, and on what a block wrote the sources' gradients
// and the receivers' loss gradients of the next reverse step n (n < 0: none).
// RR at boundary voxels lives in an array per slot (rr), not in the field, so
// that no slot's RR is overwritten while its neighbours read F from the same
// buffer.
template <int PL>
__global__ void __launch_bounds__(FB, fused_min_blocks<PL>()) k_adj_step(const __grid_constant__ StepArgs a,
                                                                         const __grid_constant__ AdjPost po,
                                                                         const __grid_constant__ FusedGeo g)
{
    pdl_trigger();
    const uint32_t tid = threadIdx.x, blk = blockIdx.x;
    const bool probes = po.n >= 0 && __ldg(g.has_probe + blk) != 0;
    if (blk < g.gb) {
        BVox<float, 0> v[PL];
        bool act[PL];
#pragma unroll
        for (int k = 0; k < PL; ++k) {
            const uint64_t s = ((uint64_t)blk * PL + k) * FB + tid;
            act[k] = s < a.nb;
            if (act[k]) bvox_site<float, 0>(a, s, v[k]);
        }
        pdl_wait();
#pragma unroll
        for (int k = 0; k < PL; ++k)
            if (act[k]) bvox_values<float, 0>(a, 0, v[k]);
#pragma unroll
        for (int k = 0; k < PL; ++k) {
            const uint64_t s = ((uint64_t)blk * PL + k) * FB + tid;
            if (!act[k]) continue;
            const BVox<float, 0> &x = v[k];
            const float r = leapfrog((uint8_t)x.meta, x.ce, x.nb[0], x.nb[1], x.nb[2], x.nb[3], x.nb[4], x.nb[5],
                                     po.rr[s], a.c2dt2, a.inv_h2);
            static_cast<float *>(a.q)[x.i] = keep::add(r, po.dbar[s]);
        }
    } else {
        const Site st = stencil_site(blk, g);
        const uint32_t plane = a.px * a.ny, o = (st.bx * FB + tid) * V;
        const bool act = o < plane;
        StencilVecs<float, PL> s;
        s.site(a, st.z, act ? o : plane - V, plane);
        pdl_wait();
        s.values(a, plane);
        stencil_update<float, PL, false>(a, s, act, st.z);
    }
    if (!probes) return;
    __syncthreads();
    float *T = static_cast<float *>(a.q);
    for (uint32_t k = tid; k < po.nrcv; k += FB) {
        const Probe p = po.probe[po.nsrc + k];
        // a receiver on a voxel that no step updates reads a constant
        if (p.blk == blk && a.code[p.pos] < CODE_HARD)
            atomicAdd(T + p.pos, po.dl[(uint64_t)k * po.stride + (uint64_t)po.n]);
    }
    __syncthreads();
    for (uint32_t k = tid; k < po.nsrc; k += FB) {
        const Probe p = po.probe[k];
        if (p.blk == blk) po.gsig[(uint64_t)k * po.stride + (uint64_t)po.n] = T[p.pos];
    }
}

// One reverse step in one launch, for cascades of S = 1..4 sections: as
// k_adj_step, with a slot's transposed correction and cascade run by the
// thread that then updates its voxel.  That needs no value of another slot of
// this step, because what the neighbours read at a boundary voxel, F, depends
// on T there alone: the thread that makes T' leaves F' = the transposed
// correction of T' in the field and T' itself in an array per slot (traw).
// Records and states, which the recomputation wrote, are read before the wait
// for the kernel before; the launch that opens a segment does not overlap
// with what came before it.  The gradient terms of a warp's slots are summed
// in FP64 one material at a time, nearly always one or two per warp.  A
// gradient over 256 steps of 128x128x96 (79 K slots of two sections), the
// recomputation beside it: 5.60 ms with the cascade in a launch of its own
// before the stencil's, 4.78 now; over 128 steps of 300x200x160 (three
// sections) 12.78 and 12.38.
//
// adj_sections: sections [q0, q0 + N) of a slot, transposed, and their sums.
template <int N, int NH, int NK, int S>
__device__ __forceinline__ void adj_sections(const StepArgs &a, const AdjSlots &x, uint64_t b, bool act, uint32_t m, int q0,
                                             const float (&h)[NH], const float (&kc)[NK], const float (&xin)[S],
                                             const float4 (&aq)[S], double &yb, double *gsm)
{
    constexpr int NV = 5 * N, NP = NV <= 8 ? 8 : 16;
    double gv[NP];
#pragma unroll
    for (int j = NV; j < NP; ++j) gv[j] = 0.0;
#pragma unroll
    for (int n = N - 1; n >= 0; --n) {
        const int q = q0 + n;
        const double yt = yb + keep::wide(aq[q].z);
        gv[5 * n] = yt * keep::wide(xin[q]);
        gv[5 * n + 1] = yt * (double)h[2 * q];
        gv[5 * n + 2] = yt * (double)h[2 * q + 1];
        gv[5 * n + 3] = -yt * (double)h[2 * q + 2];
        gv[5 * n + 4] = -yt * (double)h[2 * q + 3];
        const double xbar = (double)kc[5 * q] * yt + keep::wide(aq[q].x);
        const double x1 = (double)kc[5 * q + 1] * yt + keep::wide(aq[q].y);
        const double x2 = (double)kc[5 * q + 2] * yt;
        const double y1 = -(double)kc[5 * q + 3] * yt + keep::wide(aq[q].w);
        const double y2 = -(double)kc[5 * q + 4] * yt;
        if (act)
            x.ast[(uint64_t)q * a.nb + b] =
                make_float4(keep::narrow(x1), keep::narrow(x2), keep::narrow(y1), keep::narrow(y2));
        yb = xbar;
    }
    unsigned left = __ballot_sync(0xffffffffu, act);
    while (left) {
        const uint32_t mm = __shfl_sync(0xffffffffu, m, __ffs(left) - 1);
        const bool mine = act && m == mm;
        left &= ~__ballot_sync(0xffffffffu, mine);
        double v[NP];
#pragma unroll
        for (int j = 0; j < NP; ++j) v[j] = mine ? gv[j] : 0.0;
        int idx;
        const double sum = warp_sums<NP>(v, &idx);
        if (idx < NV && (threadIdx.x & (32 / NP - 1)) == 0) atomicAdd(gsm + (mm * S + q0) * 5 + idx, sum);
    }
}

template <int S>
__device__ __forceinline__ void adj_slot(const StepArgs &a, const AdjSlots &x, uint64_t b, bool first, double *gsm)
{
    constexpr int NG = (2 * (S + 1) + 3) / 4, NC = (5 * S + 3) / 4;
    const bool act = b < a.nb;
    const uint64_t bl = act ? b : a.nb - 1; // idle lanes of the last block repeat its last slot, unstored
    const uint32_t pos = __ldg(a.bpos + bl), meta = __ldg(a.bmeta + bl), m = (meta >> 8) & 0xffu;
    const float4 rec = x.rec[bl];
    float h[4 * NG], kc[4 * NC];
#pragma unroll
    for (int g = 0; g < NG; ++g) {
        const float4 v = reinterpret_cast<const float4 *>(x.fst)[(uint64_t)g * a.nb + bl];
        h[4 * g] = v.x;
        h[4 * g + 1] = v.y;
        h[4 * g + 2] = v.z;
        h[4 * g + 3] = v.w;
    }
#pragma unroll
    for (int g = 0; g < NC; ++g) {
        const float4 v = __ldg(reinterpret_cast<const float4 *>(a.coefp) + m * NC + g);
        kc[4 * g] = v.x;
        kc[4 * g + 1] = v.y;
        kc[4 * g + 2] = v.z;
        kc[4 * g + 3] = v.w;
    }
    // forward inputs of every section at this step
    float xin[S];
    float in = keep::sub(rec.y, rec.z);
#pragma unroll
    for (int q = 0; q < S; ++q) {
        xin[q] = in;
        float yv = keep::fma(kc[5 * q], in, keep::mul(kc[5 * q + 1], h[2 * q]));
        yv = keep::fma(kc[5 * q + 2], h[2 * q + 1], yv);
        yv = keep::fma(-kc[5 * q + 3], h[2 * q + 2], yv);
        in = keep::fma(-kc[5 * q + 4], h[2 * q + 3], yv);
    }
    if (first) {
        pdl_wait();
        __syncthreads(); // gsm is zero
    }
    const float *P = static_cast<const float *>(a.p);
    const uint32_t sy = a.px, sz = a.px * a.ny;
    const float t = x.traw[bl], rr = x.rr[bl];
    float4 aq[S];
#pragma unroll
    for (int q = 0; q < S; ++q) aq[q] = x.ast[(uint64_t)q * a.nb + bl];
    const float n0 = P[pos + 1], n1 = P[pos - 1], n2 = P[pos + sy], n3 = P[pos - sy], n4 = P[pos + sz], n5 = P[pos - sz];
    const double kg = a.K * a.gain;
    const AdjCorr c = adj_correct(a.wtab, a.form, kg, a.mix_y, a.mix_d, t, meta);
    const float fr = keep::narrow(c.fr);
    const float r = leapfrog((uint8_t)meta, fr, n0, n1, n2, n3, n4, n5, rr, a.c2dt2, a.inv_h2);
    double yb = c.ybar;
#pragma unroll
    for (int q0 = (S - 1) / 2 * 2; q0 >= 0; q0 -= 2) { // two sections at a time: more terms at once cost registers
        if (q0 + 1 < S) adj_sections<2, 4 * NG, 4 * NC, S>(a, x, b, act, m, q0, h, kc, xin, aq, yb, gsm);
        else adj_sections<1, 4 * NG, 4 * NC, S>(a, x, b, act, m, q0, h, kc, xin, aq, yb, gsm);
    }
    if (act) {
        const float db = keep::narrow(c.db + yb), tn = keep::add(r, db);
        x.rr[b] = keep::sub(keep::add(fr, db), keep::narrow(c.cq));
        x.traw[b] = tn;
        static_cast<float *>(a.q)[pos] = keep::narrow(adj_correct(a.wtab, a.form, kg, a.mix_y, a.mix_d, tn, meta).fr);
    }
}

// the slot at a position a slot block owns
__device__ __forceinline__ uint64_t slot_of(const StepArgs &a, uint32_t pos, uint64_t lo, uint64_t hi)
{
    while (hi - lo > 1) {
        const uint64_t mid = (lo + hi) / 2;
        if (a.bpos[mid] <= pos) lo = mid;
        else hi = mid;
    }
    return lo;
}

// sources and receivers at the voxels this block wrote; `slots`: it owns slots
// [s0, s1), whose T' is in traw and whose F' is in the field
__device__ __noinline__ void adj_owned(const StepArgs &a, const AdjPost &po, const AdjSlots &x, uint32_t blk, bool slots,
                                       uint64_t s0, uint64_t s1)
{
    __syncthreads();
    float *T = static_cast<float *>(a.q);
    for (uint32_t k = threadIdx.x; k < po.nrcv; k += FB) {
        const Probe p = po.probe[po.nsrc + k];
        // a receiver on a voxel that no step updates reads a constant
        if (p.blk == blk && a.code[p.pos] < CODE_HARD)
            atomicAdd(slots ? x.traw + slot_of(a, p.pos, s0, s1) : T + p.pos,
                      po.dl[(uint64_t)k * po.stride + (uint64_t)po.n]);
    }
    __syncthreads();
    if (slots)
        for (uint32_t k = threadIdx.x; k < po.nrcv; k += FB) {
            const Probe p = po.probe[po.nsrc + k];
            // a receiver on a border plane, which comes to the first block
            // too, has no slot (sources are interior)
            if (p.blk != blk || a.code[p.pos] >= CODE_HARD) continue;
            const uint64_t b = slot_of(a, p.pos, s0, s1);
            T[p.pos] = keep::narrow(adj_correct(a.wtab, a.form, a.K * a.gain, a.mix_y, a.mix_d, x.traw[b], a.bmeta[b]).fr);
        }
    for (uint32_t k = threadIdx.x; k < po.nsrc; k += FB) {
        const Probe p = po.probe[k];
        if (p.blk == blk)
            po.gsig[(uint64_t)k * po.stride + (uint64_t)po.n] = slots ? x.traw[slot_of(a, p.pos, s0, s1)] : T[p.pos];
    }
}

// blocks per SM the register allocation must allow.  Grids of one plane per
// thread do not fill more.  Else four where that spills at most 24 bytes (three
// sections, 128 steps of 300x200x160: 13.06 ms with three blocks, 12.38 with
// four); with four sections it would spill 112 (170x120x110, 0.5 M slots: 9.21
// against 9.03 with three).
template <int PL, int S> constexpr int adj_min_blocks() { return PL == 2 && S <= 3 ? 4 : 3; }

template <int PL, int S>
__global__ void __launch_bounds__(FB, adj_min_blocks<PL, S>()) k_adj_one(const __grid_constant__ StepArgs a,
                                                                     const __grid_constant__ AdjPost po,
                                                                     const __grid_constant__ AdjSlots x,
                                                                     const __grid_constant__ FusedGeo g)
{
    extern __shared__ double gsm[]; // a slot block's sums of the coefficient gradients
    pdl_trigger();
    const uint32_t tid = threadIdx.x, blk = blockIdx.x;
    const bool probes = po.n >= 0 && __ldg(g.has_probe + blk) != 0;
    const uint64_t s0 = (uint64_t)blk * PL * FB;
    if (blk < g.gb) {
        for (uint32_t k = tid; k < x.ncoef; k += FB) gsm[k] = 0.0;
#pragma unroll 1
        for (int k = 0; k < PL; ++k) adj_slot<S>(a, x, s0 + k * FB + tid, k == 0, gsm);
        __syncthreads();
        for (uint32_t k = tid; k < x.ncoef; k += FB)
            if (gsm[k] != 0.0) atomicAdd(x.grad + k, gsm[k]);
    } else {
        const Site st = stencil_site(blk, g);
        const uint32_t plane = a.px * a.ny, o = (st.bx * FB + tid) * V;
        const bool act = o < plane;
        StencilVecs<float, PL> s;
        s.site(a, st.z, act ? o : plane - V, plane);
        pdl_wait();
        s.values(a, plane);
        stencil_update<float, PL, false>(a, s, act, st.z);
    }
    if (probes) adj_owned(a, po, x, blk, blk < g.gb, s0, s0 + PL * FB < a.nb ? s0 + PL * FB : a.nb);
}

// before the first reverse step: T of the slots' voxels into traw, F in its place
__global__ void k_adj_open(const StepArgs a, const AdjSlots x, float *T)
{
    const uint64_t b = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= a.nb) return;
    const uint32_t pos = a.bpos[b];
    const float t = T[pos];
    x.traw[b] = t;
    T[pos] = keep::narrow(adj_correct(a.wtab, a.form, a.K * a.gain, a.mix_y, a.mix_d, t, a.bmeta[b]).fr);
}

// Many simulations in one launch.  The members' arguments are kernel
// parameters (constant memory): a block finds its member by a binary search
// of the first blocks there, and no load from global memory stands before its
// own.  (Through a table of {member, block} and arguments copied from global
// to shared memory, two dependent loads and a barrier per block, 24 rooms of
// 1.1 M voxels took 124 us a step in FP32 and 111 in BF16; 111 and 109 this way.)
template <typename T, int MAXS, bool SR>
__global__ void __launch_bounds__(FB, fused_min_blocks<2>()) k_fused_batch(const __grid_constant__ FusedBatch b)
{
    pdl_trigger();
    uint32_t lo = 0, hi = b.n - 1u;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1u) / 2u;
        if (b.first[mid] <= blockIdx.x) lo = mid;
        else hi = mid - 1u;
    }
    const FusedMember &m = b.m[lo];
    fused_block<T, 2, MAXS, BND_UPDATE, SR, sizeof(T) == 4>(m.step, m.post, blockIdx.x - b.first[lo], m.geo);
}

// The block of each probe's voxel: its slot's (a binary search in the
// ascending boundary positions), else its plane's; a probe on a border plane,
// which no block covers and no step writes, goes to the first block.
__global__ void k_probe_blocks(Probe *probe, uint32_t n, const uint32_t *__restrict bpos, uint64_t nb, uint32_t plane,
                               uint32_t nz, const FusedGeo g, uint8_t *has_probe)
{
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint32_t pos = probe[k].pos, z = pos / plane;
    uint64_t lo = 0, hi = nb;
    while (lo < hi) {
        const uint64_t mid = (lo + hi) / 2;
        if (bpos[mid] < pos) lo = mid + 1;
        else hi = mid;
    }
    uint32_t blk = 0;
    if (lo < nb && bpos[lo] == pos) blk = (uint32_t)(lo / (FB * g.pl));
    else if (z >= 1 && z < nz - 1) blk = g.gb + (z - 1) / g.pl * g.gx + (pos - z * plane) / (FB * V);
    probe[k].blk = blk;
    has_probe[blk] = 1;
}

template <typename... P, typename... A>
cudaError_t launch_pdl(void (*kern)(P...), unsigned grid, cudaStream_t s, const A &...args)
{
    return launch_overlapped(kern, grid, FB, 0, s, args...);
}

template <typename T, int PL, int MODE, bool SR>
cudaError_t fused_by_sections(const StepArgs &a, const PostArgs &po, const FusedGeo &g, cudaStream_t s)
{
    switch (a.nsec) {
    case 1: return launch_pdl(k_fused<T, PL, 1, MODE, SR>, g.blocks, s, a, po, g);
    case 2: return launch_pdl(k_fused<T, PL, 2, MODE, SR>, g.blocks, s, a, po, g);
    case 3: return launch_pdl(k_fused<T, PL, 3, MODE, SR>, g.blocks, s, a, po, g);
    case 4: return launch_pdl(k_fused<T, PL, 4, MODE, SR>, g.blocks, s, a, po, g);
    default: return launch_pdl(k_fused<T, PL, 0, MODE, SR>, g.blocks, s, a, po, g);
    }
}

template <typename T, int MODE, bool SR>
cudaError_t fused_by_planes(const StepArgs &a, const PostArgs &po, const FusedGeo &g, cudaStream_t s)
{
    return g.pl == 1 ? fused_by_sections<T, 1, MODE, SR>(a, po, g, s) : fused_by_sections<T, 2, MODE, SR>(a, po, g, s);
}

template <typename T> cudaError_t fused_16(const StepArgs &a, const PostArgs &po, const FusedGeo &g, cudaStream_t s)
{
    if (a.sr) return fused_by_planes<T, BND_UPDATE, true>(a, po, g, s);
    return fused_by_planes<T, BND_UPDATE, false>(a, po, g, s);
}

template <typename T, bool SR> cudaError_t fused_batch_t(int sections, const FusedBatch &b, cudaStream_t s)
{
    switch (sections) {
    case 1: return launch_pdl(k_fused_batch<T, 1, SR>, b.blocks, s, b);
    case 2: return launch_pdl(k_fused_batch<T, 2, SR>, b.blocks, s, b);
    case 3: return launch_pdl(k_fused_batch<T, 3, SR>, b.blocks, s, b);
    case 4: return launch_pdl(k_fused_batch<T, 4, SR>, b.blocks, s, b);
    case -4: return launch_pdl(k_fused_batch<T, -4, SR>, b.blocks, s, b);
    default: return launch_pdl(k_fused_batch<T, 0, SR>, b.blocks, s, b);
    }
}

} // namespace

FusedGeo fused_geo(uint32_t px, uint32_t ny, uint32_t nz, uint64_t nb, int sms, int pl)
{
    FusedGeo g{};
    const uint64_t plane = (uint64_t)px * ny;
    g.gx = (uint32_t)((plane + FB * V - 1) / (FB * V));
    const uint64_t one = (uint64_t)g.gx * (nz - 2) + (nb + FB - 1) / FB;
    g.pl = pl ? (uint32_t)pl : one <= 5ull * (uint64_t)sms ? 1u : 2u;
    g.gb = (uint32_t)((nb + FB * g.pl - 1) / (FB * g.pl));
    const uint64_t st = (uint64_t)g.gx * ((nz - 2 + g.pl - 1) / g.pl);
    g.blocks = (uint32_t)(g.gb + st);
    // s / gx as a multiplication: exact for s * gx below 2^32
    g.magic = g.gx > 1 && st * g.gx < (1ull << 32) ? (uint32_t)(((1ull << 32) + g.gx - 1) / g.gx) : 0u;
    return g;
}

cudaError_t launch_fused(int storage, int mode, const StepArgs &a, const PostArgs &po, const FusedGeo &g, cudaStream_t s)
{
    switch (storage) {
    case VIRS_STORAGE_F16: return fused_16<__half>(a, po, g, s);
    case VIRS_STORAGE_BF16: return fused_16<__nv_bfloat16>(a, po, g, s);
    default:
        return mode == BND_KEEP ? fused_by_planes<float, BND_KEEP, false>(a, po, g, s)
                                : fused_by_planes<float, BND_UPDATE, false>(a, po, g, s);
    }
}

cudaError_t launch_adj_step(const StepArgs &a, const AdjPost &po, const FusedGeo &g, cudaStream_t s)
{
    return g.pl == 1 ? launch_pdl(k_adj_step<1>, g.blocks, s, a, po, g) : launch_pdl(k_adj_step<2>, g.blocks, s, a, po, g);
}

cudaError_t launch_adj_open(const StepArgs &a, const AdjSlots &x, float *T, cudaStream_t s)
{
    if (a.nb) k_adj_open<<<(unsigned)((a.nb + 255) / 256), 256, 0, s>>>(a, x, T);
    return cudaGetLastError();
}

cudaError_t launch_adj_one(const StepArgs &a, const AdjPost &po, const AdjSlots &x, const FusedGeo &g, bool overlap,
                           cudaStream_t s)
{
    const size_t sm = (size_t)x.ncoef * sizeof(double);
    const auto run = [&](auto *k1, auto *k2) {
        const auto kern = g.pl == 1 ? k1 : k2;
        if (overlap) return launch_overlapped(kern, g.blocks, FB, sm, s, a, po, x, g);
        kern<<<g.blocks, FB, sm, s>>>(a, po, x, g);
        return cudaGetLastError();
    };
    switch (a.nsec) {
    case 1: return run(k_adj_one<1, 1>, k_adj_one<2, 1>);
    case 2: return run(k_adj_one<1, 2>, k_adj_one<2, 2>);
    case 3: return run(k_adj_one<1, 3>, k_adj_one<2, 3>);
    default: return run(k_adj_one<1, 4>, k_adj_one<2, 4>);
    }
}

cudaError_t launch_fused_batch(int storage, int sections, const FusedBatch &b, cudaStream_t s, bool sr)
{
    switch (storage) {
    case VIRS_STORAGE_F16: return sr ? fused_batch_t<__half, true>(sections, b, s) : fused_batch_t<__half, false>(sections, b, s);
    case VIRS_STORAGE_BF16:
        return sr ? fused_batch_t<__nv_bfloat16, true>(sections, b, s) : fused_batch_t<__nv_bfloat16, false>(sections, b, s);
    default: return fused_batch_t<float, false>(sections, b, s);
    }
}

cudaError_t launch_probe_blocks(Probe *probe, uint32_t n, const uint32_t *bpos, uint64_t nb, uint32_t plane,
                                uint32_t nz, const FusedGeo &g, uint8_t *has_probe, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    k_probe_blocks<<<(n + 127) / 128, 128, 0, s>>>(probe, n, bpos, nb, plane, nz, g, has_probe);
    return cudaGetLastError();
}

} // namespace virs
