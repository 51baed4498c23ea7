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
// Blocks [0, gb) take 256 boundary slots each, the others 256 vectors of four
// voxels of one plane.  The planes are walked as one row of
// px * ny voxels: the y neighbours are px further on, no tile hangs over the
// grid's edge, and what the row ends mix up are border voxels, whose result
// is not kept.  Every load of a thread is independent of the others and
// issued before any arithmetic: the latency is paid once.  One vector and
// one plane per thread: two or four planes need 64 and 116 registers and
// measured 5 to 60 % slower on rooms with a thick sponge layer (the boundary
// slots share the kernel's occupancy).
//
// A 160x120x100 room with a sponge of 8 (0.64 M boundary slots): 17.4 us a
// step in three launches, 10.6 us in this one; 48x40x36: 9.2 and 3.4 us.
// From about eight million voxels on the fields come from HBM and the
// kernels that stage planes ahead of their use win (fused_on in capi.cpp).
//
// Consecutive steps overlap at their ends (programmatic dependent launch):
// a block loads what no step writes (codes, boundary positions, probes),
// then waits for the previous step's grid.
#include <type_traits>

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
    __device__ void zero() { v = Raw{}; }
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

// which probes this block owns: those at boundary slots [lo, hi) (slots) or
// those at offsets [lo, hi) of plane z
struct Owned {
    bool slots;
    uint32_t lo, hi, z;
    __device__ bool has(const Probe &p) const
    {
        return slots ? p.slot >= lo && p.slot < hi
                     : p.slot == PROBE_NO_SLOT && p.z == z && p.off >= lo && p.off < hi;
    }
};

__device__ __forceinline__ bool owns_any(const PostArgs &po, const Owned &o)
{
    bool mine = false;
    const uint32_t n = po.nsrc + po.nrcv;
    for (uint32_t k = threadIdx.x; k < n; k += FB) mine |= o.has(po.probe[k]);
    return mine;
}

// sources and receivers at the voxels this block wrote, as post_body
// (kernels_step.cu) does for all of them
template <typename T> __device__ __forceinline__ void post_owned(const PostArgs &po, const Owned &o, bool mine)
{
    using IO = Io<T>;
    if (!__syncthreads_or(mine)) return; // also: every store of this block is visible to it
    T *Q = static_cast<T *>(po.q);
    const uint32_t sn = *po.ctr;
    const uint32_t k1 = po.sr ? sr_step_key(sn, 1u) : 0u;
    for (uint32_t k = threadIdx.x; k < po.nsrc; k += FB) {
        const Probe p = po.probe[k];
        if (!o.has(p)) continue;
        const float v = sn < po.siglen ? po.sig[(uint64_t)k * po.siglen + sn] : 0.f;
        Q[p.pos] = put_rounded<T>(__fadd_rn(IO::get(Q[p.pos]), v), po.sr, p.pos, po.sr_base, k1);
    }
    __syncthreads();
    if (sn >= po.cap) return;
    for (uint32_t k = threadIdx.x; k < po.nrcv; k += FB) {
        const Probe p = po.probe[po.nsrc + k];
        if (o.has(p)) po.ir[(uint64_t)k * po.cap + sn] = __fmul_rn(IO::get(Q[p.pos]), po.inv_scale);
    }
}

// the four voxels at position i of a plane's row, after the wait; `act`
// false: nothing stored
template <typename T, bool SR>
__device__ __forceinline__ void step_vec(const StepArgs &a, const Codes<V> &code, uint32_t i, uint32_t plane, bool act)
{
    using IO = Io<T>;
    const T *P = static_cast<const T *>(a.p);
    T *Q = static_cast<T *>(a.q);
    Vec<T> c, zp, zm, yp, ym, q;
    c.load(P + i);
    zm.load(P + (i - plane));
    zp.load(P + (i + plane));
    ym.load(P + (i - a.px));
    yp.load(P + (i + a.px));
    q.load(Q + i);
    const float left = IO::ld1(P + (i - 1u)), right = IO::ld1(P + (i + V));
    const float2 c2dt2 = make_float2(a.c2dt2, a.c2dt2), inv_h2 = make_float2(a.inv_h2, a.inv_h2);
    float fc[V], fzp[V], fzm[V], fyp[V], fym[V], fq[V], r[V];
    c.get(fc);
    zm.get(fzm);
    zp.get(fzp);
    ym.get(fym);
    yp.get(fyp);
    q.get(fq);
    air_update(fc, left, right, fyp, fym, fzp, fzm, fq, c2dt2, inv_h2, r);
    if (act) {
        const uint32_t srk = SR ? sr_step_key(*a.ctr, 0u) : 0u;
        if (!code.any()) {
            put4<T, SR>(Q + i, r, i, a.sr_base, srk);
        } else {
            // voxel by voxel: border voxels keep their value, boundary
            // voxels belong to the blocks of their slots; only air next to a
            // wall outside a boundary layer takes the mirror rule
            if (code.mirror()) {
#pragma unroll
                for (int j = 0; j < V; ++j)
                    if (code.get(j) != 0u && code.get(j) < CODE_BND)
                        r[j] = leapfrog((uint8_t)code.get(j), fc[j], j == V - 1 ? right : fc[j + 1],
                                        j == 0 ? left : fc[j - 1], fyp[j], fym[j], fzp[j], fzm[j], fq[j], a.c2dt2,
                                        a.inv_h2);
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
}

template <typename T, int MAXS, int MODE, bool SR>
__device__ __forceinline__ void fused_block(const StepArgs &a, const PostArgs &po, uint32_t blk, uint32_t gb, uint32_t gx)
{
    const uint32_t tid = threadIdx.x;
    if (blk < gb) {
        const uint64_t s0 = (uint64_t)blk * FB + tid;
        const Owned own{true, blk * FB, blk * FB + FB, 0u};
        const bool mine = owns_any(po, own), act = s0 < a.nb;
        BVox<T, MAXS> v;
        if (act) bvox_site<T, MAXS>(a, s0, v);
        pdl_wait();
        if (act) {
            bvox_values<T, MAXS>(a, s0, v);
            bvox_update<T, MODE, MAXS>(a, s0, v);
        }
        if (blk == 0 && tid == 0) *po.ctr_out = *po.ctr + 1u;
        post_owned<T>(po, own, mine);
        return;
    }
    const uint32_t s = blk - gb, bz = s / gx, bx = s - bz * gx;
    const uint32_t plane = a.px * a.ny, z = (uint32_t)a.zb + bz, first = bx * FB * V;
    const bool act = first + tid * V < plane;
    const Owned own{false, first, first + FB * V, z};
    const bool mine = owns_any(po, own);
    // the last block of a plane repeats the plane's last vector, unstored
    const uint32_t i = z * plane + (act ? first + tid * V : plane - V);
    Codes<V> code;
    code.load(a.code + i);
    pdl_wait();
    if (blk == 0 && tid == 0) *po.ctr_out = *po.ctr + 1u;
    step_vec<T, SR>(a, code, i, plane, act);
    post_owned<T>(po, own, mine);
}

template <typename T, int MAXS, int MODE, bool SR>
__global__ void __launch_bounds__(FB) k_fused(const __grid_constant__ StepArgs a, const __grid_constant__ PostArgs po,
                                              uint32_t gb, uint32_t gx)
{
    pdl_trigger();
    fused_block<T, MAXS, MODE, SR>(a, po, blockIdx.x, gb, gx);
}

// One step of the adjoint fields after the transposed correction
// (kernels_adjoint.cu): the stencil T' = A F - RR (F in a.p, RR and then T'
// in a.q), at a boundary slot T' = (the mirrored leapfrog on F with the
// slot's own RR) + dbar, and on what a block wrote the sources' gradients
// and the receivers' loss gradients of the next reverse step n (n < 0: none).
// RR at boundary voxels lives in an array per slot (rr), not in the field, so
// that no slot's RR is overwritten while its neighbours read F from the same
// buffer.
__global__ void __launch_bounds__(FB) k_adj_step(const __grid_constant__ StepArgs a, const __grid_constant__ AdjPost po,
                                                 uint32_t gb, uint32_t gx)
{
    pdl_trigger();
    const uint32_t tid = threadIdx.x, blk = blockIdx.x;
    Owned own;
    bool mine = false;
    const uint32_t np = po.n < 0 ? 0u : po.nsrc + po.nrcv;
    if (blk < gb) {
        const uint64_t s0 = (uint64_t)blk * FB + tid;
        own = Owned{true, blk * FB, blk * FB + FB, 0u};
        for (uint32_t k = tid; k < np; k += FB) mine |= own.has(po.probe[k]);
        const bool act = s0 < a.nb;
        BVox<float, 0> v;
        if (act) bvox_site<float, 0>(a, s0, v);
        pdl_wait();
        if (act) {
            bvox_values<float, 0>(a, s0, v);
            const float r = leapfrog((uint8_t)v.meta, v.ce, v.nb[0], v.nb[1], v.nb[2], v.nb[3], v.nb[4], v.nb[5],
                                     po.rr[s0], a.c2dt2, a.inv_h2);
            static_cast<float *>(a.q)[v.i] = __fadd_rn(r, po.dbar[s0]);
        }
    } else {
        const uint32_t s = blk - gb, bz = s / gx, bx = s - bz * gx;
        const uint32_t plane = a.px * a.ny, z = (uint32_t)a.zb + bz, first = bx * FB * V;
        const bool act = first + tid * V < plane;
        own = Owned{false, first, first + FB * V, z};
        for (uint32_t k = tid; k < np; k += FB) mine |= own.has(po.probe[k]);
        const uint32_t i = z * plane + (act ? first + tid * V : plane - V);
        Codes<V> code;
        code.load(a.code + i);
        pdl_wait();
        step_vec<float, false>(a, code, i, plane, act);
    }
    if (!__syncthreads_or(mine)) return;
    float *T = static_cast<float *>(a.q);
    for (uint32_t k = tid; k < po.nrcv; k += FB) {
        const Probe p = po.probe[po.nsrc + k];
        // a receiver on a voxel that no step updates reads a constant
        if (own.has(p) && a.code[p.pos] < CODE_HARD) atomicAdd(T + p.pos, po.dl[(uint64_t)k * po.stride + (uint64_t)po.n]);
    }
    __syncthreads();
    for (uint32_t k = tid; k < po.nsrc; k += FB) {
        const Probe p = po.probe[k];
        if (own.has(p)) po.gsig[(uint64_t)k * po.stride + (uint64_t)po.n] = T[p.pos];
    }
}

// Many simulations: a table gives each block its member and its number in
// it; the block copies that member's arguments into shared memory once.
// Both are constant over the steps and read before the wait.
template <typename T, int MAXS, bool SR>
__global__ void __launch_bounds__(FB) k_fused_batch(const BatchMember *__restrict mem, const uint2 *__restrict table,
                                                    int parity)
{
    __shared__ StepArgs a;
    __shared__ PostArgs po;
    pdl_trigger();
    const uint2 e = __ldg(table + blockIdx.x);
    {
        const uint32_t *sa = reinterpret_cast<const uint32_t *>(&mem[e.x].step[parity]);
        const uint32_t *sp = reinterpret_cast<const uint32_t *>(&mem[e.x].post[parity]);
        constexpr uint32_t na = sizeof(StepArgs) / 4, np = sizeof(PostArgs) / 4;
        static_assert(na + np <= FB, "one word per thread");
        const uint32_t t = threadIdx.x;
        if (t < na) reinterpret_cast<uint32_t *>(&a)[t] = __ldg(sa + t);
        else if (t < na + np) reinterpret_cast<uint32_t *>(&po)[t - na] = __ldg(sp + (t - na));
    }
    __syncthreads();
    const uint32_t gb = (uint32_t)((a.nb + FB - 1) / FB), gx = (a.px * a.ny + FB * V - 1) / (FB * V);
    fused_block<T, MAXS, BND_UPDATE, SR>(a, po, e.y, gb, gx);
}

// the slot of each probe's voxel in the boundary list (ascending positions)
__global__ void k_probe_slots(Probe *probe, uint32_t n, const uint32_t *__restrict bpos, uint64_t nb)
{
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint32_t pos = probe[k].pos;
    uint64_t lo = 0, hi = nb;
    while (lo < hi) {
        const uint64_t mid = (lo + hi) / 2;
        if (bpos[mid] < pos) lo = mid + 1;
        else hi = mid;
    }
    probe[k].slot = lo < nb && bpos[lo] == pos ? (uint32_t)lo : PROBE_NO_SLOT;
}

template <typename... P, typename... A>
cudaError_t launch_pdl(void (*kern)(P...), unsigned grid, cudaStream_t s, const A &...args)
{
    return launch_overlapped(kern, grid, FB, 0, s, args...);
}

template <typename T, int MODE, bool SR>
cudaError_t fused_by_sections(const StepArgs &a, const PostArgs &po, cudaStream_t s)
{
    const uint32_t gb = (uint32_t)((a.nb + FB - 1) / FB);
    const uint32_t gx = (a.px * a.ny + FB * V - 1) / (FB * V);
    const unsigned grid = gb + gx * (a.nz - 2);
    if (a.nsec <= 1) return launch_pdl(k_fused<T, 1, MODE, SR>, grid, s, a, po, gb, gx);
    if (a.nsec == 2) return launch_pdl(k_fused<T, 2, MODE, SR>, grid, s, a, po, gb, gx);
    if (a.nsec == 3) return launch_pdl(k_fused<T, 3, MODE, SR>, grid, s, a, po, gb, gx);
    if (a.nsec == 4) return launch_pdl(k_fused<T, 4, MODE, SR>, grid, s, a, po, gb, gx);
    return launch_pdl(k_fused<T, 0, MODE, SR>, grid, s, a, po, gb, gx);
}

template <typename T> cudaError_t fused_16(const StepArgs &a, const PostArgs &po, cudaStream_t s)
{
    if (a.sr) return fused_by_sections<T, BND_UPDATE, true>(a, po, s);
    return fused_by_sections<T, BND_UPDATE, false>(a, po, s);
}

} // namespace

cudaError_t launch_fused(int storage, int mode, const StepArgs &a, const PostArgs &po, cudaStream_t s)
{
    switch (storage) {
    case VIRS_STORAGE_F16: return fused_16<__half>(a, po, s);
    case VIRS_STORAGE_BF16: return fused_16<__nv_bfloat16>(a, po, s);
    default:
        return mode == BND_KEEP ? fused_by_sections<float, BND_KEEP, false>(a, po, s)
                                : fused_by_sections<float, BND_UPDATE, false>(a, po, s);
    }
}

cudaError_t launch_adj_step(const StepArgs &a, const AdjPost &po, cudaStream_t s)
{
    const uint32_t gb = (uint32_t)((a.nb + FB - 1) / FB);
    const uint32_t gx = (a.px * a.ny + FB * V - 1) / (FB * V);
    return launch_pdl(k_adj_step, gb + gx * (a.nz - 2), s, a, po, gb, gx);
}

namespace {
template <typename T, bool SR>
cudaError_t fused_batch_t(int sections, const BatchMember *mem, const uint2 *table, uint32_t nblocks, int parity,
                          cudaStream_t s)
{
    switch (sections) {
    case 1: return launch_pdl(k_fused_batch<T, 1, SR>, nblocks, s, mem, table, parity);
    case 2: return launch_pdl(k_fused_batch<T, 2, SR>, nblocks, s, mem, table, parity);
    case 3: return launch_pdl(k_fused_batch<T, 3, SR>, nblocks, s, mem, table, parity);
    case 4: return launch_pdl(k_fused_batch<T, 4, SR>, nblocks, s, mem, table, parity);
    case -4: return launch_pdl(k_fused_batch<T, -4, SR>, nblocks, s, mem, table, parity);
    default: return launch_pdl(k_fused_batch<T, 0, SR>, nblocks, s, mem, table, parity);
    }
}
} // namespace

uint64_t fused_blocks(uint32_t px, uint32_t ny, uint32_t nz, uint64_t nb)
{
    return (nb + FB - 1) / FB + ((uint64_t)px * ny + FB * V - 1) / (FB * V) * (nz - 2);
}

cudaError_t launch_fused_batch(int storage, int sections, const BatchMember *mem, const uint2 *table, uint32_t nblocks,
                               int parity, cudaStream_t s, bool sr)
{
    switch (storage) {
    case VIRS_STORAGE_F16:
        return sr ? fused_batch_t<__half, true>(sections, mem, table, nblocks, parity, s)
                  : fused_batch_t<__half, false>(sections, mem, table, nblocks, parity, s);
    case VIRS_STORAGE_BF16:
        return sr ? fused_batch_t<__nv_bfloat16, true>(sections, mem, table, nblocks, parity, s)
                  : fused_batch_t<__nv_bfloat16, false>(sections, mem, table, nblocks, parity, s);
    default: return fused_batch_t<float, false>(sections, mem, table, nblocks, parity, s);
    }
}

cudaError_t launch_probe_slots(Probe *probe, uint32_t n, const uint32_t *bpos, uint64_t nb, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    k_probe_slots<<<(n + 127) / 128, 128, 0, s>>>(probe, n, bpos, nb);
    return cudaGetLastError();
}

} // namespace virs
