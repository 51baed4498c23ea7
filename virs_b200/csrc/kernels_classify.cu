// Voxel classification on the GPU: the sponge-layer distance build, the
// normals bitmask, the cell codes of the step kernel and the compacted,
// ascending boundary-voxel list.
//
// Reference semantics (src/simulator/sponge_kernel.cu:8-62, generalised to
// width W): an interior air voxel (flag 0) becomes a boundary voxel (flag 2)
// when some wall voxel (flag 1) lies in the cube [-W, W]^3 around it with
// squared distance d2 < W*W + 1.  The reference scans the whole cube per
// voxel, (2W+1)^3 flag reads.  Here the minimum is taken one axis at a time,
// which is exact because the squared distance separates, min over the cube of
// dx^2+dy^2+dz^2 equals min_dz(dz^2 + min_dy(dy^2 + min_dx dx^2)).  Among
// equal distances the first voxel in the reference's scan order (dz, then dy,
// then dx ascending) wins: each axis is scanned upwards and only a smaller
// distance replaces the best, and along x the lower of two equally near walls
// is taken.  The winner's offsets locate the nearest wall voxel, whose
// material becomes the boundary voxel's material.  W <= 31.
//
//   k_wall_bits   one bit per voxel: flag 1
//   k_sponge_xy   the nearest wall along x from 64 bits around the voxel (two
//                 funnel shifts, two bit scans), once per row of a tile, then
//                 the scan along y in shared memory
//   k_sponge_z    the scan along z and the classification
// A tile whose window holds no wall is marked empty and skipped by the next
// pass: most of a large room, where the passes then read the flags and
// write them once.  1024x768x512 voxels, W = 1: the three passes over 32-bit
// keys, a thread per voxel, took 6.9 ms, these 1.3 (the copy of the flags
// included); codes and list, a block per 128 voxels, 3.4 ms, 1.0 with 16
// voxels per thread and empty segments skipped; the hard-source search, two
// sweeps of the codes, 1.3 ms, none now without such voxels.
#include <algorithm>

#include "internal.hpp"

namespace virs {
namespace {

// bytes of w equal to v: 0xff each
__device__ __forceinline__ uint32_t eq4(uint32_t w, uint32_t v) { return __vcmpeq4(w, v * 0x01010101u); }

// bytes of w that equal v, as bits 0-3
__device__ __forceinline__ uint32_t nibble(uint32_t w, uint32_t v)
{
    const uint32_t e = eq4(w, v) & 0x08040201u;
    return (e | e >> 8 | e >> 16 | e >> 24) & 0xfu;
}

// sixteen voxels per thread (one load), two threads per word; n: voxels, a
// multiple of 32
__global__ void __launch_bounds__(256) k_wall_bits(const uint4 *__restrict flags, uint32_t *__restrict bits, uint64_t n)
{
    const uint64_t t = (uint64_t)blockIdx.x * 256 + threadIdx.x;
    const uint4 f = t < n / 16 ? __ldg(flags + t) : make_uint4(0u, 0u, 0u, 0u);
    const uint32_t v = nibble(f.x, 1u) | nibble(f.y, 1u) << 4 | nibble(f.z, 1u) << 8 | nibble(f.w, 1u) << 12;
    const uint32_t o = __shfl_down_sync(0xffffffffu, v, 1);
    if (!(t & 1u) && t < n / 16) bits[t / 2] = v | o << 16;
}

// Tiles of 128 x XY_ROWS voxels of a plane: for every voxel the nearest wall
// within W in the plane, as (dy + 32) << 6 | (dx + 32) in near2 (NEAR_NONE:
// none); live: whether the tile has any.
constexpr int XY_ROWS = 32;
constexpr uint16_t NEAR_NONE = 0xffffu;
constexpr int8_t DX_NONE = 127;

__global__ void __launch_bounds__(256) k_sponge_xy(const uint32_t *__restrict bits, uint16_t *__restrict near2,
                                                   uint8_t *__restrict live, int ny, int px, int W)
{
    __shared__ int8_t dxt[XY_ROWS + 62][SEG];
    __shared__ uint32_t win[XY_ROWS + 62][6];          // the window's words: one beyond the tile on each side
    __shared__ uint32_t any[(XY_ROWS + 62 + 31) / 32]; // rows of the window with a wall near
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int words = px / 32, x0 = blockIdx.x * SEG, y0 = blockIdx.y * XY_ROWS, z = blockIdx.z;
    const int rows = XY_ROWS + 2 * W;
    if (tid < (int)(sizeof(any) / 4)) any[tid] = 0u;
    uint32_t seen = 0;
    for (int t = tid; t < rows * 6; t += 256) {
        const int r = t / 6, c = t - 6 * r, k = x0 / 32 - 1 + c, y = y0 - W + r;
        const bool in = y >= 0 && y < ny && k >= 0 && k < words;
        const uint32_t v = in ? __ldg(bits + ((size_t)z * ny + y) * words + k) : 0u;
        win[r][c] = v;
        seen |= v;
    }
    if (!__syncthreads_or(seen != 0u)) { // no wall in the window: most tiles of a large room
        if (tid == 0) live[((size_t)z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = 0;
        return;
    }
    // four x-words per row; a warp takes one word of a row at a time
    for (int t = wid; t < rows * 4; t += 8) {
        const int r = t >> 2;
        const uint32_t *b = &win[r][t & 3];
        const uint32_t wl = b[0], wc = b[1], wr = b[2];
        int dx = DX_NONE;
        if (wl | wc | wr) { // uniform over the warp
            const int dl = __clz(__funnelshift_l(wl, wc, 31 - lane));             // at or left of x
            const int dr = __clz(__brev(__funnelshift_r(wc, wr, lane)));          // at or right of x
            if (min(dl, dr) <= W) dx = dl <= dr ? -dl : dr;
            if (__any_sync(0xffffffffu, dx != DX_NONE) && lane == 0) atomicOr(&any[r >> 5], 1u << (r & 31));
        }
        dxt[r][(t & 3) * 32 + lane] = (int8_t)dx;
    }
    __syncthreads();
    bool some = false;
    for (int k = 0; k < (int)(sizeof(any) / 4); ++k) some |= any[k] != 0u;
    bool found = false;
    if (some) {
        const int lim = W * W, c = tid & (SEG - 1), x = x0 + c;
        for (int r = tid / SEG; r < XY_ROWS; r += 256 / SEG) {
            const int y = y0 + r;
            if (y >= ny || x >= px) continue;
            int best = lim + 1;
            uint16_t key = NEAR_NONE;
            for (int j = 0; j <= 2 * W; ++j) {
                const int q = r + j; // window row of dy = j - W
                if (!((any[q >> 5] >> (q & 31)) & 1u)) continue;
                const int dx = dxt[q][c], dy = j - W;
                const int d2 = dx * dx + dy * dy; // DX_NONE: beyond any limit
                if (d2 < best) {
                    best = d2;
                    key = (uint16_t)((dy + 32) << 6 | (dx + 32));
                }
            }
            found |= key != NEAR_NONE;
            near2[((size_t)z * ny + y) * px + x] = key;
        }
    }
    const int f = __syncthreads_or(found);
    if (tid == 0) live[((size_t)z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = f ? 1 : 0;
}

// The scan along z over the live tiles' planes, then the classification, one
// tile of k_sponge_xy per block: a tile without a live one in its window
// leaves at once.  flags_out holds a copy of flags_in; its boundary voxels are
// set here, as are bmat_full and bd2_full.
__global__ void __launch_bounds__(256) k_sponge_z(const ClassifyArgs a)
{
    const int tid = threadIdx.x, W = a.W;
    const int nx = a.nx, ny = a.ny, nz = a.nz, px = a.px;
    const int x = blockIdx.x * SEG + (tid & 31) * 4, z = blockIdx.z;
    if (z == 0 || z == nz - 1) return;
    // bit j: the tile of plane z - W + j is live
    uint64_t mask = 0;
    {
        const size_t tiles = (size_t)gridDim.x * gridDim.y;
        const uint8_t *l = a.live + (size_t)blockIdx.y * gridDim.x + blockIdx.x;
        for (int j = tid & 31; j <= 2 * W; j += 32) {
            const int k = z - W + j;
            if (k >= 0 && k < nz && l[(size_t)k * tiles]) mask |= 1ull << j;
        }
        const uint32_t lo = __reduce_or_sync(0xffffffffu, (uint32_t)mask), hi = __reduce_or_sync(0xffffffffu, (uint32_t)(mask >> 32));
        mask = (uint64_t)hi << 32 | lo;
    }
    if (!mask || x >= px) return;
    const size_t plane = (size_t)px * ny;
    const int lim = W * W;
    for (int y = blockIdx.y * XY_ROWS + (tid >> 5); y < min((int)(blockIdx.y + 1) * XY_ROWS, ny - 1); y += 8) {
        if (y == 0) continue;
        const size_t i = ((size_t)z * ny + y) * px + x;
        uint32_t f = __ldg(reinterpret_cast<const uint32_t *>(a.flags_in + i));
        int best[4] = {lim + 1, lim + 1, lim + 1, lim + 1};
        uint32_t key[4] = {0, 0, 0, 0};
        for (uint64_t m = mask; m; m &= m - 1) {
            const int j = __ffsll((long long)m) - 1, dz = j - W;
            const uint2 v = __ldg(reinterpret_cast<const uint2 *>(a.near2 + i + (ptrdiff_t)dz * (ptrdiff_t)plane));
            if ((v.x & v.y) == 0xffffffffu) continue;
            const uint32_t n[4] = {v.x & 0xffffu, v.x >> 16, v.y & 0xffffu, v.y >> 16};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int dx = (int)(n[c] & 63u) - 32, dy = (int)((n[c] >> 6) & 63u) - 32;
                const int d2 = dx * dx + dy * dy + dz * dz;
                if (n[c] != NEAR_NONE && d2 < best[c]) {
                    best[c] = d2;
                    key[c] = (uint32_t)(dz + 32) << 12 | n[c];
                }
            }
        }
        uint32_t set = 0;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (best[c] > lim || ((f >> (8 * c)) & 0xffu) != 0u || x + c == 0 || x + c >= nx - 1) continue;
            const int dx = (int)(key[c] & 63u) - 32, dy = (int)((key[c] >> 6) & 63u) - 32, dz = (int)(key[c] >> 12) - 32;
            set |= 2u << (8 * c);
            a.bmat_full[i + c] =
                a.wall_mat[i + c + (ptrdiff_t)dz * (ptrdiff_t)plane + (ptrdiff_t)dy * (ptrdiff_t)px + dx];
            a.bd2_full[i + c] = (uint16_t)best[c];
        }
        if (set) *reinterpret_cast<uint32_t *>(a.flags_out + i) = f | set;
    }
}

// the code and normals of four voxels (f), given their neighbours' flags
// +x -x +y -y +z -z and the bytes of interior columns
__device__ __forceinline__ uint2 codes4(uint32_t f, const uint32_t (&n)[6], uint32_t in)
{
    uint32_t nrm = 0, wall = 0;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        nrm |= eq4(n[k], 0u) & (0x01010101u << k);  // simulator.cpp:480-531
        wall |= eq4(n[k], 1u) & (0x01010101u << k); // W_XP .. W_ZM
    }
    const uint32_t bnd = eq4(f, 2u), is1 = eq4(f, 1u), is3 = eq4(f, 3u);
    const uint32_t code = (wall & ~(is1 | is3)) | (bnd & 0x80808080u) | (is1 & 0xfefefefeu) | (is3 & 0xfdfdfdfdu);
    return make_uint2((code & in) | ~in, nrm & in);
}

// Cell codes, normals, per-segment boundary counts and whether a segment
// holds any non-zero code, and the number of hard-source voxels: sixteen
// voxels per lane, a warp for the four segments of 512 voxels of a row (spr
// is a multiple of four), bytes compared four at a time.
__global__ void __launch_bounds__(256) k_codes(const CodesArgs a, uint64_t nwarp)
{
    const uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const uint32_t lane = threadIdx.x & 31u;
    if (w >= nwarp) return; // the whole warp
    const uint32_t per = a.spr / 4;
    const uint64_t row = w / per;
    const uint32_t x = ((uint32_t)(w % per) * 32 + lane) * 16;
    const uint32_t y = (uint32_t)(row % a.ny), z = (uint32_t)(row / a.ny);
    const bool act = x < a.px, inner = y > 0 && z > 0 && y < a.ny - 1 && z < a.nz - 1;
    const size_t i = row * a.px + x, sy = a.px, sz = (size_t)a.px * a.ny;
    const auto at = [&](size_t k) { return __ldg(reinterpret_cast<const uint4 *>(a.flags + k)); };
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    const bool on = act && inner;
    const uint4 f = on ? at(i) : zero, yp = on ? at(i + sy) : zero, ym = on ? at(i - sy) : zero;
    const uint4 zp = on ? at(i + sz) : zero, zm = on ? at(i - sz) : zero;
    uint32_t fl = __shfl_up_sync(0xffffffffu, f.w, 1) >> 24, fr = __shfl_down_sync(0xffffffffu, f.x, 1) & 0xffu;
    uint32_t cnt = 0, hard = 0, any = 0;
    if (act) {
        uint4 code = make_uint4(~0u, ~0u, ~0u, ~0u), nrm = zero; // CODE_NONE
        if (inner) {
            if (lane == 0) fl = x > 0 ? a.flags[i - 1] : 0u;
            if (lane == 31) fr = x + 16 < a.px ? a.flags[i + 16] : 0u;
            const uint32_t F[6] = {fl << 24, f.x, f.y, f.z, f.w, fr};
            const uint32_t YP[4] = {yp.x, yp.y, yp.z, yp.w}, YM[4] = {ym.x, ym.y, ym.z, ym.w};
            const uint32_t ZP[4] = {zp.x, zp.y, zp.z, zp.w}, ZM[4] = {zm.x, zm.y, zm.z, zm.w};
            uint32_t C[4], N[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t xq = x + 4 * q;
                uint32_t in = ~0u; // bytes of interior columns
                if (xq == 0) in &= ~0xffu;
                if (xq + 4 >= a.nx) {
                    // voxels from nx - 1 on are outside
                    const uint32_t keep = xq < a.nx - 1 ? a.nx - 1 - xq : 0u; // 0..3
                    in &= keep ? ~0u >> (32 - 8 * keep) : 0u;
                }
                const uint32_t c = F[q + 1];
                const uint32_t n[6] = {c >> 8 | F[q + 2] << 24, c << 8 | F[q] >> 24, YP[q], YM[q], ZP[q], ZM[q]};
                const uint2 cn = codes4(c, n, in);
                C[q] = cn.x;
                N[q] = cn.y;
                cnt += __popc(eq4(c, 2u) & in & 0x01010101u);
                hard += __popc(eq4(c, 3u) & in & 0x01010101u);
            }
            code = make_uint4(C[0], C[1], C[2], C[3]);
            nrm = make_uint4(N[0], N[1], N[2], N[3]);
        }
        *reinterpret_cast<uint4 *>(a.code + i) = code;
        *reinterpret_cast<uint4 *>(a.normals + i) = nrm;
        any = code.x | code.y | code.z | code.w;
    }
    hard = __reduce_add_sync(0xffffffffu, hard);
    if (lane == 0 && hard) atomicAdd(a.nhard, hard);
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) { // the eight lanes of a segment
        cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        any |= __shfl_xor_sync(0xffffffffu, any, o);
    }
    if ((lane & 7u) == 0) {
        const uint64_t seg = row * a.spr + x / SEG;
        a.segcnt[seg] = cnt;
        a.segnz[seg] = any ? 1 : 0;
    }
}

// boundary voxels of a segment get consecutive slots after bseg[segment]: a
// warp looks at 32 segments and takes those that have any in turn
__global__ void __launch_bounds__(256) k_compact(const CompactArgs a, uint64_t nseg, uint32_t total)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t s0 = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32 * 32;
    uint32_t mine = 0, next = 0;
    if (s0 + lane < nseg) {
        mine = a.bseg[s0 + lane];
        next = s0 + lane + 1 < nseg ? a.bseg[s0 + lane + 1] : total;
    }
    for (uint32_t todo = __ballot_sync(0xffffffffu, mine != next); todo; todo &= todo - 1) {
        const int l = __ffs(todo) - 1;
        const uint64_t seg = s0 + (uint64_t)l, row = seg / a.spr;
        const uint32_t first = __shfl_sync(0xffffffffu, mine, l);
        const uint32_t x = (uint32_t)(seg % a.spr) * SEG + lane * 4;
        const size_t i = row * a.px + x;
        const uint32_t code = x < a.px ? __ldg(reinterpret_cast<const uint32_t *>(a.code + i)) : 0xffffffffu;
        const uint32_t bnd = code & ~(code << 1) & 0x80808080u; // boundary codes: bits 7-6 are 10
        const uint32_t n = __popc(bnd);
        uint32_t inc = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= (uint32_t)o) inc += t;
        }
        uint64_t slot = (uint64_t)first + inc - n;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (!((bnd >> (8 * c + 7)) & 1u)) continue;
            const uint32_t m = a.bmat_full[i + c], d2 = a.bd2_full[i + c];
            a.bidx[slot] = (uint32_t)(row * a.nx + x + c);
            a.bpos[slot] = (uint32_t)(i + c);
            a.bmeta[slot] = ((code >> (8 * c)) & 0xffu) | m << 8 | d2 << 16;
            a.bnrm[slot] = a.normals[i + c];
            a.bmat[slot] = (uint8_t)m;
            a.bw[slot] = a.wtab[d2];
            ++slot;
        }
    }
}

// ---- exclusive scan (three phases) -------------------------------------------

constexpr int SCAN_B = 1024;

__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t *total)
{
    __shared__ uint32_t ws[SCAN_B / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) ws[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        uint32_t w = lane < SCAN_B / 32 ? ws[lane] : 0;
        uint32_t wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += t;
        }
        if (lane < SCAN_B / 32) ws[lane] = wi - w;
        if (lane == SCAN_B / 32 - 1) *total = wi;
    }
    __syncthreads();
    return inc - v + ws[wid];
}

__global__ void k_scan_blocks(uint32_t *data, size_t n, uint32_t *bsum)
{
    __shared__ uint32_t tot;
    const size_t i = (size_t)blockIdx.x * SCAN_B + threadIdx.x;
    const uint32_t v = i < n ? data[i] : 0;
    const uint32_t e = block_excl_scan(v, &tot);
    if (i < n) data[i] = e;
    if (threadIdx.x == 0) bsum[blockIdx.x] = tot;
}

__global__ void k_scan_add(uint32_t *data, size_t n, const uint32_t *boff)
{
    const size_t i = (size_t)blockIdx.x * SCAN_B + threadIdx.x;
    if (i < n) data[i] += boff[blockIdx.x];
}

__global__ void k_scan_total(const uint32_t *data, const uint32_t *orig_last, size_t n, uint32_t *total)
{
    *total = data[n - 1] + *orig_last;
}

__global__ void k_copy1(const uint32_t *src, uint32_t *dst) { *dst = *src; }

} // namespace

size_t sponge_live_tiles(uint32_t px, uint32_t ny, uint32_t nz)
{
    return (size_t)((px + SEG - 1) / SEG) * ((ny + XY_ROWS - 1) / XY_ROWS) * nz;
}

namespace {
// blocks of eight warps, one warp each
unsigned warp_blocks(uint64_t warps) { return (unsigned)((warps + 7) / 8); }
} // namespace

cudaError_t launch_sponge(const ClassifyArgs &a, cudaStream_t s)
{
    const uint64_t n = (uint64_t)a.px * a.ny * a.nz;
    cudaError_t e = cudaMemcpyAsync(a.flags_out, a.flags_in, n, cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) return e;
    k_wall_bits<<<(unsigned)((n / 16 + 255) / 256), 256, 0, s>>>(reinterpret_cast<const uint4 *>(a.flags_in), a.bits, n);
    const dim3 tiles((a.px + SEG - 1) / SEG, (a.ny + XY_ROWS - 1) / XY_ROWS, a.nz);
    k_sponge_xy<<<tiles, 256, 0, s>>>(a.bits, a.near2, a.live, (int)a.ny, (int)a.px, a.W);
    k_sponge_z<<<tiles, 256, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_codes(const CodesArgs &a, cudaStream_t s)
{
    const uint64_t nwarp = (uint64_t)(a.spr / 4) * a.ny * a.nz;
    k_codes<<<warp_blocks(nwarp), 256, 0, s>>>(a, nwarp);
    return cudaGetLastError();
}

size_t scan_tmp_words(size_t n)
{
    size_t words = 1;
    do {
        n = (n + SCAN_B - 1) / SCAN_B;
        words += n;
    } while (n > 1);
    return words;
}

namespace {
// exclusive scan of data[0..n) in place; tmp holds the per-block sums of
// every level
cudaError_t scan_levels(uint32_t *data, size_t n, uint32_t *tmp, cudaStream_t s)
{
    const size_t nb = (n + SCAN_B - 1) / SCAN_B;
    uint32_t *bsum = tmp;
    k_scan_blocks<<<(unsigned)nb, SCAN_B, 0, s>>>(data, n, bsum);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || nb == 1) return e;
    e = scan_levels(bsum, nb, tmp + nb, s);
    if (e != cudaSuccess) return e;
    k_scan_add<<<(unsigned)nb, SCAN_B, 0, s>>>(data, n, bsum);
    return cudaGetLastError();
}
} // namespace

// data[0..n) <- exclusive prefix sums; *total <- their sum.
cudaError_t launch_scan(uint32_t *data, size_t n, uint32_t *tmp, uint32_t *total, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    k_copy1<<<1, 1, 0, s>>>(data + n - 1, tmp); // the last input, for the total
    cudaError_t e = scan_levels(data, n, tmp + 1, s);
    if (e != cudaSuccess) return e;
    k_scan_total<<<1, 1, 0, s>>>(data, tmp, n, total);
    return cudaGetLastError();
}

namespace {
// device positions of the hard-source voxels (code CODE_HARD), at most cap.
// The order is arbitrary: every step
// writes the same value to all of them.
__global__ void k_hard_list(const uint8_t *__restrict code, uint64_t n, uint32_t *count, uint32_t *out, uint32_t cap)
{
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        if (code[i] == CODE_HARD) {
            const uint32_t k = atomicAdd(count, 1u);
            if (k < cap) out[k] = (uint32_t)i;
        }
}
} // namespace

cudaError_t launch_hard_list(const uint8_t *code, uint64_t n, uint32_t *count, uint32_t *out, uint32_t cap,
                             cudaStream_t s)
{
    k_hard_list<<<1184, 256, 0, s>>>(code, n, count, out, cap);
    return cudaGetLastError();
}

cudaError_t launch_compact(const CompactArgs &a, uint32_t total, cudaStream_t s)
{
    const uint64_t nseg = (uint64_t)a.spr * a.ny * a.nz;
    k_compact<<<warp_blocks((nseg + 31) / 32), 256, 0, s>>>(a, nseg, total);
    return cudaGetLastError();
}


// ---- planes of a stencil tile whose codes are all zero ---------------------------
//
// For a rows x zc tiling, bit j of a tile's mask is set when the codes of
// the plane staged in stage j (plane z0 - 1 + j, j < 64, one of the tile's
// own planes) are all zero over the tile's 128 x rows voxels: the stencil
// then skips their copy and treats every voxel as plain air.  From the
// per-segment flags of k_codes (a tile row is one segment).
namespace {
__global__ void __launch_bounds__(64) k_tile_zero_mask(const uint8_t *__restrict segnz, uint32_t ny, uint32_t nz,
                                                       uint32_t spr, uint32_t rows, uint32_t zc, uint32_t gx,
                                                       uint32_t gy, uint32_t zb, uint32_t ze,
                                                       uint64_t *__restrict mask)
{
    __shared__ unsigned w[2];
    const uint32_t t = blockIdx.x, j = threadIdx.x;
    const uint32_t bx = t % gx, by = (t / gx) % gy, bz = t / (gx * gy);
    const uint32_t z0 = zb + bz * zc, z1 = min(z0 + zc, ze);
    const uint32_t k = z0 - 1 + j;
    bool zero = false;
    if (k >= z0 && k < z1) {
        zero = true;
        const uint32_t y1 = min(by * rows + rows, ny);
        for (uint32_t y = by * rows; y < y1 && zero; ++y) zero = segnz[((size_t)k * ny + y) * spr + bx] == 0;
    }
    const unsigned b = __ballot_sync(0xffffffffu, zero);
    if ((j & 31) == 0) w[j >> 5] = b;
    __syncthreads();
    if (j == 0) mask[t] = (uint64_t)w[0] | ((uint64_t)w[1] << 32);
}
} // namespace

cudaError_t launch_tile_zero_masks(const uint8_t *segnz, uint32_t ny, uint32_t nz, uint32_t spr, uint32_t rows,
                                   uint32_t zc, uint32_t gx, uint32_t gy, uint32_t gz, uint32_t zb, uint32_t ze,
                                   uint64_t *mask, cudaStream_t s)
{
    const uint64_t ntiles = (uint64_t)gx * gy * gz;
    if (ntiles == 0) return cudaSuccess;
    k_tile_zero_mask<<<(unsigned)ntiles, 64, 0, s>>>(segnz, ny, nz, spr, rows, zc, gx, gy, zb, ze, mask);
    return cudaGetLastError();
}

// The same masks for the tiles of the two-step kernel: a tile covers x in
// [bx*ix - v, bx*ix - v + 128) and rows [by*iy - 1, by*iy - 1 + rows) (the
// parts outside the grid read as code 0), and stage j holds plane
// zs - 2 + j with zs = 1 + bz*zc; the stages with codes are the planes
// zs-1 .. z1.  A bit is set when every 128-voxel segment the tile's codes
// touch on that plane holds only zeros.
namespace {
__global__ void __launch_bounds__(64) k_pair_zero_mask(const uint8_t *__restrict segnz, uint32_t px, uint32_t ny,
                                                       uint32_t nz, uint32_t spr, uint32_t rows, uint32_t zc,
                                                       uint32_t ix, uint32_t v, uint32_t gx, uint32_t gy,
                                                       uint64_t *__restrict mask)
{
    __shared__ unsigned w[2];
    const uint32_t t = blockIdx.x, j = threadIdx.x;
    const uint32_t bx = t % gx, by = (t / gx) % gy, bz = t / (gx * gy);
    const int zs = 1 + (int)(bz * zc), z1 = min(zs + (int)zc, (int)nz - 1);
    const int k = zs - 2 + (int)j;
    bool zero = false;
    if (k >= zs - 1 && k <= z1 && k >= 0 && k < (int)nz) {
        zero = true;
        const int xs = (int)(bx * ix) - (int)v, ys = (int)(by * (rows - 2)) - 1;
        const int xa = max(xs, 0), xb = min(xs + 128, (int)px);
        const int ya = max(ys, 0), yb = min(ys + (int)rows, (int)ny);
        for (int y = ya; y < yb && zero; ++y)
            for (int sx = xa / 128; sx <= (xb - 1) / 128 && zero; ++sx)
                zero = segnz[((size_t)k * ny + y) * spr + sx] == 0;
    }
    const unsigned b = __ballot_sync(0xffffffffu, zero);
    if ((j & 31) == 0) w[j >> 5] = b;
    __syncthreads();
    if (j == 0) mask[t] = (uint64_t)w[0] | ((uint64_t)w[1] << 32);
}
} // namespace

cudaError_t launch_pair_zero_masks(const uint8_t *segnz, uint32_t px, uint32_t ny, uint32_t nz, uint32_t spr,
                                   uint32_t rows, uint32_t zc, uint32_t ix, uint32_t v, uint32_t gx, uint32_t gy,
                                   uint32_t gz, uint64_t *mask, cudaStream_t s)
{
    const uint64_t ntiles = (uint64_t)gx * gy * gz;
    if (ntiles == 0) return cudaSuccess;
    k_pair_zero_mask<<<(unsigned)ntiles, 64, 0, s>>>(segnz, px, ny, nz, spr, rows, zc, ix, v, gx, gy, mask);
    return cudaGetLastError();
}

// ---- voxels whose second step of a two-step pass is provisional --------------
//
// The two-step stencil computes p^{n+2} from p^{n+1} before the post kernel
// has changed p^{n+1} at the sources.  The p^{n+2} of every voxel the stencil
// updates (air or mirror code: bit 7 clear) that is a source or its face
// neighbour must be recomputed afterwards.  k_pair_mark marks them,
// k_mark_count counts the marks of each 1024-voxel segment, and after an
// exclusive scan of the counts k_mark_list writes their positions in
// ascending order.
namespace {
constexpr int MARK_B = 1024;

__device__ __forceinline__ void mark_around(const uint8_t *__restrict code, uint8_t *mark, uint64_t v, uint32_t px,
                                            uint32_t ny, uint32_t nz)
{
    const uint64_t plane = (uint64_t)px * ny;
    const uint32_t x = (uint32_t)(v % px), y = (uint32_t)((v / px) % ny), z = (uint32_t)(v / plane);
    if (z >= nz) return;
    const uint64_t nbv[7] = {v, v + 1, v - 1, v + px, v - px, v + plane, v - plane};
    const bool in[7] = {true, x + 1 < px, x > 0, y + 1 < ny, y > 0, z + 1 < nz, z > 0};
#pragma unroll
    for (int k = 0; k < 7; ++k)
        if (in[k] && (code[nbv[k]] & CODE_BND) == 0) mark[nbv[k]] = 1;
}

__global__ void k_pair_mark(const uint8_t *__restrict code, uint32_t px, uint32_t ny, uint32_t nz,
                            const uint32_t *__restrict hpos, uint32_t nh, const uint64_t *__restrict src,
                            uint32_t nsrc, uint8_t *mark)
{
    const uint64_t n = (uint64_t)nh + nsrc;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t v = i < nh ? (uint64_t)hpos[i] : src[i - nh];
        mark_around(code, mark, v, px, ny, nz);
    }
}

__global__ void __launch_bounds__(MARK_B) k_mark_count(const uint8_t *__restrict mark, uint64_t n, uint32_t *cnt)
{
    const uint64_t i = (uint64_t)blockIdx.x * MARK_B + threadIdx.x;
    const int c = __syncthreads_count(i < n && mark[i] != 0);
    if (threadIdx.x == 0) cnt[blockIdx.x] = (uint32_t)c;
}

__global__ void __launch_bounds__(MARK_B) k_mark_list(const uint8_t *__restrict mark, uint64_t n,
                                                      const uint32_t *__restrict off, uint32_t *list)
{
    __shared__ uint32_t tot;
    const uint64_t i = (uint64_t)blockIdx.x * MARK_B + threadIdx.x;
    const uint32_t f = i < n && mark[i] != 0 ? 1u : 0u;
    const uint32_t e = block_excl_scan(f, &tot);
    if (f) list[off[blockIdx.x] + e] = (uint32_t)i;
}
} // namespace

size_t mark_segments(uint64_t nvox) { return (size_t)((nvox + MARK_B - 1) / MARK_B); }

cudaError_t launch_pair_marks(const uint8_t *code, uint32_t px, uint32_t ny, uint32_t nz, const uint32_t *hpos,
                              uint32_t nh, const uint64_t *src, uint32_t nsrc,
                              uint8_t *mark, uint32_t *cnt, cudaStream_t s)
{
    const uint64_t nvox = (uint64_t)px * ny * nz;
    if (nh + nsrc) {
        const uint64_t n = (uint64_t)nh + nsrc;
        const unsigned g = (unsigned)std::min<uint64_t>((n + 255) / 256, 148ull * 16);
        k_pair_mark<<<g, 256, 0, s>>>(code, px, ny, nz, hpos, nh, src, nsrc, mark);
    }
    k_mark_count<<<(unsigned)mark_segments(nvox), MARK_B, 0, s>>>(mark, nvox, cnt);
    return cudaGetLastError();
}

cudaError_t launch_mark_list(const uint8_t *mark, uint64_t nvox, const uint32_t *off, uint32_t *list, cudaStream_t s)
{
    k_mark_list<<<(unsigned)mark_segments(nvox), MARK_B, 0, s>>>(mark, nvox, off, list);
    return cudaGetLastError();
}

} // namespace virs
