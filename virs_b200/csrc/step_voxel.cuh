// The update of one thread's voxels, shared by the step kernels: a vector of
// voxels of a row by cell code (tile_update), and one boundary voxel of the
// compacted list (BVox).
#pragma once

#include "step_common.cuh"

namespace virs {
namespace step {
namespace {

// the V cell codes of a thread (4 or 8 bytes)
template <int V> struct Codes;
// bytes with bit 7 clear and some other bit set: bit 7 of each byte of
// ((w & 0x7f..) + 0x7f..) & ~w
__device__ __forceinline__ uint32_t mirror_bytes(uint32_t w)
{
    return ((w & 0x7f7f7f7fu) + 0x7f7f7f7fu) & ~w & 0x80808080u;
}
template <> struct Codes<4> {
    uint32_t w;
    __device__ void load(const unsigned char *p) { w = *reinterpret_cast<const uint32_t *>(p); }
    __device__ void clear() { w = 0u; }
    __device__ bool any() const { return w != 0u; }
    __device__ uint32_t get(int k) const { return (w >> (8 * k)) & 0xffu; }
    __device__ uint32_t mirror() const { return mirror_bytes(w); }
    __device__ bool is_mirror(uint32_t m, int k) const { return (m >> (8 * k + 7)) & 1u; }
};
template <> struct Codes<8> {
    uint2 w;
    __device__ void load(const unsigned char *p) { w = *reinterpret_cast<const uint2 *>(p); }
    __device__ void clear() { w = make_uint2(0u, 0u); }
    __device__ bool any() const { return (w.x | w.y) != 0u; }
    __device__ uint32_t get(int k) const { return ((k < 4 ? w.x : w.y) >> (8 * (k & 3))) & 0xffu; }
    // the mirror bytes of the two words folded into one: bit 7 of byte k
    // (k < 4) from w.x, bit 6 of byte k - 4 from w.y
    __device__ uint32_t mirror() const { return mirror_bytes(w.x) | (mirror_bytes(w.y) >> 1); }
    __device__ bool is_mirror(uint32_t m, int k) const { return (m >> (8 * (k & 3) + (k < 4 ? 7 : 6))) & 1u; }
};

// every voxel as air without wall neighbours, two at a time
template <int V>
__device__ __forceinline__ void air_update(const float (&cc)[V], float left, float right, const float (&yp)[V],
                                           const float (&ym)[V], const float (&zp)[V], const float (&zm)[V],
                                           const float (&qv)[V], float2 c2dt2, float2 inv_h2, float (&r)[V])
{
#pragma unroll
    for (int k = 0; k < V; k += 2) {
        const float2 x2 = make_float2(__fadd_rn(cc[k + 1], k > 0 ? cc[k - 1] : left),
                                      __fadd_rn(k + 2 < V ? cc[k + 2] : right, cc[k]));
        const float2 o = leapfrog_air2(make_float2(cc[k], cc[k + 1]), x2, make_float2(yp[k], yp[k + 1]),
                                       make_float2(ym[k], ym[k + 1]), make_float2(zp[k], zp[k + 1]),
                                       make_float2(zm[k], zm[k + 1]), make_float2(qv[k], qv[k + 1]), c2dt2, inv_h2);
        r[k] = o.x;
        r[k + 1] = o.y;
    }
}

// The update of one thread's V voxels of a plane: cc holds the centres,
// left / right the x neighbours beyond the vector, ym / yp / zm / zp the y
// and z neighbours, qv p^{n-1}.
template <typename T>
__device__ __forceinline__ void tile_update(const Codes<Io<T>::VEC> &code, const float (&cc)[Io<T>::VEC], float left,
                                        float right, const float (&yp)[Io<T>::VEC], const float (&ym)[Io<T>::VEC],
                                        const float (&zp)[Io<T>::VEC], const float (&zm)[Io<T>::VEC],
                                        const float (&qv)[Io<T>::VEC], float2 c2dt2, float2 inv_h2, float c2dt2s,
                                        float inv_h2s, float (&r)[Io<T>::VEC])
{
    constexpr int V = Io<T>::VEC;
    // every voxel as air without wall neighbours, the common case ...
    air_update(cc, left, right, yp, ym, zp, zm, qv, c2dt2, inv_h2, r);
    // ... then the voxels with another code.  Walls take 0; border,
    // hard-source and boundary voxels keep p^{n-1} (the post kernel
    // writes the hard-source value, the boundary pass updates boundary
    // voxels from the untouched p^n buffer): a test and a select per
    // voxel, no divergence.  Only air next to a wall outside the
    // boundary layer (a grid without a sponge layer) needs the update
    // with the mirror rule; such codes have bit 7 clear and other bits
    // set, found for four bytes at once.
    if (__any_sync(FULL, code.any())) {
#pragma unroll
        for (int k = 0; k < V; ++k) {
            const uint32_t c = code.get(k);
            if (c & CODE_BND) r[k] = c == CODE_WALL ? 0.f : qv[k];
        }
        const uint32_t mirror = code.mirror();
        if (__any_sync(FULL, mirror != 0u)) {
#pragma unroll
            for (int k = 0; k < V; ++k)
                if (code.is_mirror(mirror, k))
                    r[k] = leapfrog((uint8_t)code.get(k), cc[k], k == V - 1 ? right : cc[k + 1],
                                    k == 0 ? left : cc[k - 1], yp[k], ym[k], zp[k], zm[k], qv[k], c2dt2s, inv_h2s);
        }
    }
}

// The loads of one boundary voxel (first part) and its update (second).
template <typename T, int MAXS> struct BVox {
    uint32_t i, meta; // device position; code, material and weight entry (StepArgs::bmeta)
    uint8_t nm;
    float ce, qv, nb[6];
    BState<MAXS> st;
};

// what no step writes: where the voxel is and its code
template <typename T, int MAXS>
__device__ __forceinline__ void bvox_site(const StepArgs &a, uint64_t slot, BVox<T, MAXS> &v)
{
    v.i = __ldg(a.bpos + slot);
    v.meta = __ldg(a.bmeta + slot);
    v.nm = a.rigid ? __ldg(a.bnrm + slot) : 0;
}

// the pressures around it and its filter states (MAXS == 0: not the states)
template <typename T, int MAXS>
__device__ __forceinline__ void bvox_values(const StepArgs &a, uint64_t slot, BVox<T, MAXS> &v)
{
    using IO = Io<T>;
    const uint32_t i = v.i, sy = a.px, sz = a.px * a.ny;
    const T *P = static_cast<const T *>(a.p);
    const T *Q = static_cast<const T *>(a.q);
    v.ce = IO::get(P[i]);
    v.qv = IO::get(Q[i]);
    v.nb[0] = IO::get(P[i + 1]);
    v.nb[1] = IO::get(P[i - 1]);
    v.nb[2] = IO::get(P[i + sy]);
    v.nb[3] = IO::get(P[i - sy]);
    v.nb[4] = IO::get(P[i + sz]);
    v.nb[5] = IO::get(P[i - sz]);
    if constexpr (MAXS != 0) bload<MAXS>(a, slot, v.st);
}

template <typename T, int MAXS>
__device__ __forceinline__ void bvox_load(const StepArgs &a, uint64_t slot, BVox<T, MAXS> &v)
{
    bvox_site<T, MAXS>(a, slot, v);
    bvox_values<T, MAXS>(a, slot, v);
}

template <typename T, int MODE, int MAXS>
__device__ __forceinline__ void bvox_update(const StepArgs &a, uint64_t slot, const BVox<T, MAXS> &v)
{
    float r;
    if (a.rigid) {
        // fdtd_kernel_rigid_walls (simulator_gpu.cu:152-180): the air
        // neighbours only (normals mask), p+ = (2 - l2 n) p - p- + the sum
        // of (l2 * s) * p_nb over +x, -x, +y, -y, +z, -z with s = 1 for air;
        // with the reference build's contractions
        const float b1 = __fmaf_rn(-a.l2, (float)__popc(v.nm), 2.f);
        r = __fmaf_rn(b1, v.ce, -v.qv);
#pragma unroll
        for (int k = 0; k < 6; ++k) r = __fmaf_rn(__fmul_rn(a.l2, (v.nm & (1u << k)) ? 1.f : 0.f), v.nb[k], r);
    } else {
        r = leapfrog((uint8_t)v.meta, v.ce, v.nb[0], v.nb[1], v.nb[2], v.nb[3], v.nb[4], v.nb[5], v.qv, a.c2dt2, a.inv_h2);
    }
    if (MODE != BND_UPDATE) a.side[slot] = make_float4(r, v.ce, v.qv, 0.f);
    if constexpr (MAXS != 0) r = bcompute<MAXS>(a, r, v.ce, v.qv, slot, v.meta, v.st);
    else r = boundary_loop(a, r, v.ce, v.qv, slot, v.meta);
    static_cast<T *>(a.q)[v.i] =
        put_rounded<T>(r, a.sr, v.i, a.sr_base, a.sr ? sr_step_key(*a.ctr, 0u) : 0u);
}

} // namespace
} // namespace step
} // namespace virs
