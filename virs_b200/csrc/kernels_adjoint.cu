// Reverse-mode (adjoint) kernels: gradients of a receiver loss with respect
// to the boundary filter coefficients and the source signals.
//
// One forward step maps (p, q, S) -> (p+, p, S+), linear in the fields and
// the filter states.  With T the adjoint of p^{n+1} and RR the negated
// adjoint carried by p^n through its role as q of the next step, one
// reverse step n is
//   k_adj_boundary   at boundary voxels the correction and the biquad cascade
//                    run transposed: F = T (reference form) or T/(1+a)
//                    (centered form), the cascade's state adjoints and the
//                    coefficient gradients (FP64), dbar = d(loss)/d(p - q),
//                    and the voxel's next RR' = F + dbar - cq, kept per slot
//   k_adj_step       T' = A F - RR into RR's buffer, at boundary voxels
//                    T'_b = A F_b - RR_b + dbar_b (kernels_fused.cu): the
//                    forward stencil, since A (2 + lambda^2 * Laplacian with
//                    mirrored walls and zero fixed voxels) is symmetric on
//                    the updated voxels; hard-source voxels take 0.  Then, for
//                    the next reverse step, T'[rcv] += dL/dIR and
//                    dL/dsig = T'[src]
// and the buffers swap.  k_adj_inject does the latter before the first step.
// The forward values the cascade needs (p - q and the states before step n)
// come from a recomputation of the segment from the last checkpoint.
//
// Cascades of up to four sections take both in one launch (k_adj_one,
// kernels_fused.cu).  128x128x96 voxels, 79 K slots of two sections: a reverse
// step was five launches of 28.7 us and their gaps, then two of 12, now one.
#include "adjoint.cuh"
#include "pdl.cuh"

namespace virs {
namespace {

using namespace step;

__global__ void k_adj_inject(float *T, const uint8_t *__restrict code, const uint64_t *__restrict rcv, uint32_t nrcv,
                             const float *__restrict dl, uint64_t dl_stride, uint64_t n, const uint64_t *__restrict src,
                             uint32_t nsrc, float *__restrict gsig, uint64_t gs_stride)
{
    for (uint32_t r = threadIdx.x; r < nrcv; r += blockDim.x) {
        // receivers read the new field; a receiver on a voxel that is not
        // updated (wall, hard source, border) reads a constant
        const uint64_t i = rcv[r];
        if (code[i] < CODE_HARD) atomicAdd(T + i, dl[(uint64_t)r * dl_stride + n]);
    }
    __syncthreads();
    for (uint32_t s = threadIdx.x; s < nsrc; s += blockDim.x) gsig[(uint64_t)s * gs_stride + n] = T[src[s]];
}

struct AdjArgs {
    float *T;                  // adjoint field (p role)
    const uint32_t *bpos, *bmeta; // as StepArgs
    const BndWeight *wtab;
    const float *coef;         // [M][S][5]
    const float4 *rec;         // forward records of this step {free, p, q, 0}
    const float *fst;          // forward states before this step (the cascade's layout, state_index)
    float4 *ast;               // state adjoints, one vector per section [S][nb]
    float *dbar, *rr;          // per slot: dbar, and the voxel's next RR
    double *grad;              // [M][S][5]
    uint64_t nb;
    uint32_t nsec, ncoef;
    int form;
    double kg, mix_y, mix_d;   // K * gain
};

// the slot's results: F into the field, dbar, and RR' = F + dbar - cq
__device__ __forceinline__ void adj_store(const AdjArgs &a, uint64_t b, uint32_t pos, const AdjCorr &c, double yb)
{
    const float fr = (float)c.fr, db = (float)(c.db + yb), cq = (float)c.cq;
    a.T[pos] = fr;
    a.dbar[b] = db;
    a.rr[b] = __fsub_rn(__fadd_rn(fr, db), cq);
}

constexpr int AB = 128;

// The sum of v over the lanes of a full warp that share this lane's key
// (peers = __match_any_sync of the key), complete at the group's lowest
// lane: a tree over each group's ranks, every lane taking part in every
// shuffle.  Lanes of a mixed warp (boundary slots of two or more
// materials) then make one shared-memory add per group instead of one
// each.
__device__ __forceinline__ double peer_sum(unsigned peers, double v)
{
    const unsigned lane = threadIdx.x & 31u;
    unsigned rank = __popc(peers & ((1u << lane) - 1u));
    peers &= 0xfffffffeu << lane; // the peers above this lane
    while (__any_sync(0xffffffffu, peers != 0u)) {
        const int next = __ffs(peers);
        const double u = __shfl_sync(0xffffffffu, v, next > 0 ? next - 1 : 0);
        if (next > 0) v += u;
        peers &= __ballot_sync(0xffffffffu, (rank & 1u) == 0u);
        rank >>= 1;
    }
    return v;
}

__global__ void __launch_bounds__(AB) k_adj_boundary(const AdjArgs a)
{
    pdl_trigger();
    extern __shared__ double gsm[]; // block partial sums of the coefficient gradients
    for (uint32_t k = threadIdx.x; k < a.ncoef; k += AB) gsm[k] = 0.0;
    __syncthreads();
    pdl_wait();
    const uint64_t b = (uint64_t)blockIdx.x * AB + threadIdx.x;
    if (b < a.nb) {
        const uint32_t pos = a.bpos[b], meta = a.bmeta[b];
        const AdjCorr c = adj_correct(a.wtab, a.form, a.kg, a.mix_y, a.mix_d, a.T[pos], meta);
        // forward inputs of every section at this step
        const uint32_t S = a.nsec, m = (meta >> 8) & 0xffu;
        const float *kc = a.coef + (uint64_t)m * S * 5;
        const float4 rec = a.rec[b];
        float xin[16];
        float in = __fsub_rn(rec.y, rec.z);
        for (uint32_t q = 0; q < S; ++q) {
            const float *kq = kc + 5 * q;
            const float s0 = a.fst[state_index(2 * q + 0, b, a.nb)], s1 = a.fst[state_index(2 * q + 1, b, a.nb)];
            const float s2 = a.fst[state_index(2 * q + 2, b, a.nb)], s3 = a.fst[state_index(2 * q + 3, b, a.nb)];
            xin[q] = in;
            float yv = __fmaf_rn(kq[0], in, __fmul_rn(kq[1], s0));
            yv = __fmaf_rn(kq[2], s1, yv);
            yv = __fmaf_rn(-kq[3], s2, yv);
            in = __fmaf_rn(-kq[4], s3, yv);
        }
        // every lane of this warp holds a slot of one material (the loops
        // over the sections are uniform: S is the same for every slot)
        // full warps sum over the lanes of each material first
        const bool full = __activemask() == 0xffffffffu;
        const unsigned peers = full ? __match_any_sync(0xffffffffu, m) : 0u;
        const bool lead = full && (int)(threadIdx.x & 31u) == __ffs(peers) - 1;
        double yb = c.ybar;
        for (int q = (int)S - 1; q >= 0; --q) {
            const float *kq = kc + 5 * q;
            const float4 aq = a.ast[(uint64_t)q * a.nb + b];
            const double yt = yb + (double)aq.z;
            const double s0 = a.fst[state_index(2 * q, b, a.nb)], s1 = a.fst[state_index(2 * q + 1, b, a.nb)],
                         s2 = a.fst[state_index(2 * q + 2, b, a.nb)], s3 = a.fst[state_index(2 * q + 3, b, a.nb)];
            double *g = gsm + (uint64_t)(m * S + q) * 5;
            const double gv[5] = {yt * (double)xin[q], yt * s0, yt * s1, -yt * s2, -yt * s3};
            if (full) {
#pragma unroll
                for (int j = 0; j < 5; ++j) {
                    const double v = peer_sum(peers, gv[j]);
                    if (lead) atomicAdd(g + j, v);
                }
            } else {
#pragma unroll
                for (int j = 0; j < 5; ++j) atomicAdd(g + j, gv[j]);
            }
            const double xbar = (double)kq[0] * yt + (double)aq.x;
            const double x1 = (double)kq[1] * yt + (double)aq.y;
            const double x2 = (double)kq[2] * yt;
            const double y1 = -(double)kq[3] * yt + (double)aq.w;
            const double y2 = -(double)kq[4] * yt;
            a.ast[(uint64_t)q * a.nb + b] = make_float4((float)x1, (float)x2, (float)y1, (float)y2);
            yb = xbar;
        }
        adj_store(a, b, pos, c, yb);
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < a.ncoef; k += AB)
        if (gsm[k] != 0.0) atomicAdd(a.grad + k, gsm[k]);
}

} // namespace

cudaError_t launch_adj_inject(float *T, const uint8_t *code, const uint64_t *rcv, uint32_t nrcv, const float *dl,
                              uint64_t dl_stride, uint64_t n, const uint64_t *src, uint32_t nsrc, float *gsig,
                              uint64_t gs_stride, cudaStream_t s)
{
    k_adj_inject<<<1, 256, 0, s>>>(T, code, rcv, nrcv, dl, dl_stride, n, src, nsrc, gsig, gs_stride);
    return cudaGetLastError();
}

cudaError_t launch_adj_boundary(const StepArgs &f, float *T, const float4 *rec, const float *fst, float4 *ast,
                                float *dbar, float *rr, double *grad, uint32_t nmat, cudaStream_t s)
{
    if (f.nb == 0) return cudaSuccess;
    const AdjArgs a{T, f.bpos, f.bmeta, f.wtab, f.coef, rec, fst, ast, dbar, rr, grad, f.nb, f.nsec,
                    nmat * f.nsec * 5, f.form, f.K * f.gain, f.mix_y, f.mix_d};
    return launch_overlapped(k_adj_boundary, (unsigned)((f.nb + AB - 1) / AB), AB, (size_t)a.ncoef * sizeof(double), s, a);
}

namespace {
__global__ void k_set_u32(uint32_t *p, uint32_t v) { *p = v; }
} // namespace

// one device word set in stream order (no host staging buffer)
cudaError_t launch_set_u32(uint32_t *p, uint32_t v, cudaStream_t s)
{
    k_set_u32<<<1, 1, 0, s>>>(p, v);
    return cudaGetLastError();
}

} // namespace virs
