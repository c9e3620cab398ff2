// Whole-configuration sums: the spatial order of the atoms in tiles of 32 with bounding boxes, the
// real-space energy and forces over the tile pairs within the cutoff, the structure factors and the
// k-space forces factored along the rows of the k grid.
//
// Real space.  A configuration has N^2/2 pairs but only N (4/3 pi rc^3 rho)/2 inside the cutoff
// (1.5 % of them at 49,752 atoms).  The atoms are put in the order of a cell grid's Morton index
// (a stable counting sort, so the order and every sum are the same from run to run), 32 consecutive
// ones form a tile, and a tile only meets the tiles whose boxes come within the cutoff.
//
// k space.  exp(i k r) = X^kx Y^ky Z^kz, so a sum over atoms for all kz of a row (kx, ky) is a small
// matrix product: with A = X^kx Y^ky of an atom, the four sums A.re cos, A.im sin, A.re sin, A.im
// cos over the atoms give both signs of kz: 2 FP64 FMAs per atom and signed k vector instead of the
// 16 operations of the full product, and the kz-factors are read once for a warp of rows.
#pragma once

#include "yamc_chain.cuh"

namespace yamc {

// ------------------------------------------------------------------------------------------
// spatial order
// ------------------------------------------------------------------------------------------
constexpr int kTile = 32;          // points per tile: one warp's lanes
// Points per block of the counting sort: at least kSortChunk, and as many as make kSortBlocks blocks,
// up to kSortMaxChunk, whose cells beside those of the grid fill the 48 KB that a block has without
// asking (from there on there are more blocks).
constexpr int kSortChunk = 256, kSortMaxChunk = 8192;
constexpr int kSortBlocks = 64;
constexpr int kSortMaxCells = 4096;
constexpr int kSortThreads = 256;

// cells per axis: a power of two <= 16, about four points per cell or more
__host__ __device__ inline int sort_cells(int n) {
    int nc = 1;
    while (nc < 16 && 4 * (2 * nc) * (2 * nc) * (2 * nc) <= n) nc *= 2;
    return nc;
}

// coordinates p[stride i] of points (box units), as the counting sort and the tiles read them
struct Points {
    const double *x, *y, *z;
    int stride, n;
};

__device__ __forceinline__ int point_cell(const Points &P, int i, int nc) {
    return (int)(spread3(cell_axis(P.x[(size_t)P.stride * i], nc)) | (spread3(cell_axis(P.y[(size_t)P.stride * i], nc)) << 1) |
                 (spread3(cell_axis(P.z[(size_t)P.stride * i], nc)) << 2));
}

// counts per cell of the block's chunk of points, added to the totals per cell
static __global__ void __launch_bounds__(kSortThreads) k_sort_count(Points P, int nc, int chunk, int *hist, int *total) {
    __shared__ int h[kSortMaxCells];
    const int ncell = nc * nc * nc;
    for (int c = threadIdx.x; c < ncell; c += kSortThreads) h[c] = 0;
    __syncthreads();
    const int i1 = min(P.n, (int)(blockIdx.x + 1) * chunk);
    for (int i = blockIdx.x * chunk + threadIdx.x; i < i1; i += kSortThreads) atomicAdd(&h[point_cell(P, i, nc)], 1);
    __syncthreads();
    for (int c = threadIdx.x; c < ncell; c += kSortThreads) {
        hist[(size_t)blockIdx.x * ncell + c] = h[c];
        if (h[c]) atomicAdd(&total[c], h[c]);
    }
}

// the counts of (block, cell) replaced by the first position of that block's points of the cell:
// every block of the grid takes 256 cells, after the points of the cells before them
static __global__ void __launch_bounds__(256) k_sort_scan(const int *total, int *hist, int nb, int ncell) {
    __shared__ int wsum[8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, c0 = blockIdx.x * 256;
    int before = 0;  // points in the cells before c0, this thread's share
    for (int c = tid; c < c0; c += 256) before += total[c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    const int own = c0 + tid < ncell ? total[c0 + tid] : 0;
    int x = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    // (wsum: the points before c0 counted by the warp, then with the warp's own cells)
    __shared__ int bsum[8];
    if (lane == 31) { wsum[warp] = x; bsum[warp] = before; }
    __syncthreads();
    int at = x - own;
    for (int w = 0; w < 8; ++w) at += bsum[w] + (w < warp ? wsum[w] : 0);
    if (c0 + tid >= ncell) return;
    // (eight loads at a time before their stores: one after the other they are nb round trips)
    int *h = hist + c0 + tid;
    for (int b = 0; b < nb; b += 8) {
        int t[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) t[k] = b + k < nb ? h[(size_t)(b + k) * ncell] : 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (b + k < nb) h[(size_t)(b + k) * ncell] = at;
            at += t[k];
        }
    }
}

// order[p] = the point at position p: the chunk's points to their cells' positions, points of one
// cell in index order (one warp places, 32 points at a time)
static __global__ void __launch_bounds__(kSortThreads) k_sort_place(Points P, int nc, int chunk, const int *hist, int *total, int *order) {
    extern __shared__ int at[];  // [ncell], then [chunk] cells of the chunk's points
    const int ncell = nc * nc * nc;
    int *key = at + ncell;
    const int i0 = blockIdx.x * chunk, m = min(chunk, P.n - i0);
    for (int c = threadIdx.x; c < ncell; c += kSortThreads) {
        at[c] = hist[(size_t)blockIdx.x * ncell + c];
        if (blockIdx.x == 0) total[c] = 0;  // for the next sort
    }
    for (int i = threadIdx.x; i < m; i += kSortThreads) key[i] = point_cell(P, i0 + i, nc);
    __syncthreads();
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    for (int b = 0; b < m; b += 32) {
        const int k = b + lane < m ? key[b + lane] : -1;
        const unsigned peers = __match_any_sync(0xffffffffu, k);
        const int before = __popc(peers & ((1u << lane) - 1u));
        const int pos = k >= 0 ? at[k] + before : 0;
        __syncwarp();
        if (k >= 0) {
            order[pos] = i0 + b + lane;
            if (before == __popc(peers) - 1) at[k] = pos + 1;
        }
        __syncwarp();
    }
}

// per tile of the order a bounding box (centre, half extents; box units, periodic), as the chain
// kernel's blocks have them; a box with a coordinate that is not finite has no bounds
static __global__ void __launch_bounds__(256) k_tile_boxes(Points P, const int *order, int ntile, float4 *box) {
    const int t = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (t >= ntile) return;
    const int p = t * kTile + lane, i = order[min(p, P.n - 1)];
    const double v[3] = {P.x[(size_t)P.stride * i], P.y[(size_t)P.stride * i], P.z[(size_t)P.stride * i]};
    double r[3], lo[3], hi[3];
    bool fine = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        r[d] = __shfl_sync(0xffffffffu, v[d], 0);
        lo[d] = hi[d] = wrap_half(v[d] - r[d]);
        fine = fine && isfinite(lo[d]);
    }
    fine = __all_sync(0xffffffffu, fine);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            lo[d] = fmin(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
            hi[d] = fmax(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
        }
    }
    if (lane != 0) return;
    const float inf = __int_as_float(0x7f800000);
    box[2 * t] = fine ? make_float4((float)wrap_half(r[0] + 0.5 * (lo[0] + hi[0])), (float)wrap_half(r[1] + 0.5 * (lo[1] + hi[1])),
                                    (float)wrap_half(r[2] + 0.5 * (lo[2] + hi[2])), 0.f)
                      : make_float4(0.f, 0.f, 0.f, 0.f);
    box[2 * t + 1] = fine ? make_float4(__double2float_ru(0.5 * (hi[0] - lo[0]) + kBoxPad), __double2float_ru(0.5 * (hi[1] - lo[1]) + kBoxPad),
                                        __double2float_ru(0.5 * (hi[2] - lo[2]) + kBoxPad), 0.f)
                          : make_float4(inf, inf, inf, 0.f);
}

// false only if no two points of the two boxes are within sqrt(r2) under any periodic image
__device__ __forceinline__ bool boxes_near(float4 ca, float4 ha, float4 cb, float4 hb, double r2) {
    const double ex = fmax(fabs(wrap_half((double)ca.x - (double)cb.x)) - ((double)ha.x + (double)hb.x), 0.0);
    const double ey = fmax(fabs(wrap_half((double)ca.y - (double)cb.y)) - ((double)ha.y + (double)hb.y), 0.0);
    const double ez = fmax(fabs(wrap_half((double)ca.z - (double)cb.z)) - ((double)ha.z + (double)hb.z), 0.0);
    return ex * ex + ey * ey + ez * ez < r2;
}

// The near tiles of tile ti among [base, base + kNearSpan), in increasing order, into list (shared);
// returns their number (check: the index check word, or null).  All threads of a block of NW warps; HALF: each unordered pair of tiles
// belongs to one of the two (by the parity of their sum, so the tiles' shares are even), the tile
// itself included.
constexpr int kNearSpan = 1024;
template <bool HALF, int NW>
__device__ __forceinline__ int near_tiles(const float4 *box, int ntile, int ti, int base, double r2, unsigned *words, int *list,
                                          int *count, int *check) {
    const float4 c = box[2 * ti], h = box[2 * ti + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < kNearSpan / (32 * NW); ++k) {
        const int w = k * NW + warp, t = base + w * 32 + lane;
        bool near = t < ntile;
        if (HALF && near) near = t == ti || (((t + ti) & 1) ? t > ti : t < ti);
        if (near) near = boxes_near(c, h, box[2 * t], box[2 * t + 1], r2);
        const unsigned b = __ballot_sync(0xffffffffu, near);
        if (lane == 0) words[w] = b;
    }
    __syncthreads();
    if (warp == 0) {
        unsigned b = words[lane];
        const int n = __popc(b);
        int x = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        for (int at = x - n; b; b &= b - 1, ++at) list[YAMC_IXC(at, kNearSpan, check)] = base + lane * 32 + __ffs(b) - 1;
        if (lane == 31) *count = x;
    }
    __syncthreads();
    return *count;
}

// ------------------------------------------------------------------------------------------
// real space
// ------------------------------------------------------------------------------------------
constexpr int kFullParts = 8;  // ew, lj6, lj12, ew_intra, lj6_intra, lj12_intra, overlap, spare
constexpr int kRealWarps = 4;  // (8 take the same time: 0.41 ms of energy at 49,752 atoms)

// one atom of a tile as the pair loops read it
struct TileAtom { double x, y, z, q, dhs; int mol, type; };

__device__ __forceinline__ TileAtom tile_atom(const DevSys &D, int i, double4 v) {
    TileAtom a;
    const int2 m = D.meta[i];
    a.x = v.x; a.y = v.y; a.z = v.z; a.q = v.w; a.dhs = D.dhs[i]; a.mol = m.x; a.type = m.y;
    return a;
}

// Candidate pairs of a lane's point with the 32 points of a tile: FP32 coordinates in the unit box,
// nearest image, against a limit wider than the FP32 rounding (coordinates to 3e-8, so squared
// distances below 1 to under 1e-6); the exact FP64 test follows.  A point whose coordinates are not
// finite is a candidate.  The FP32 test takes 17 full-rate operations where the FP64 one takes 35 at
// half the rate.
__device__ __forceinline__ float3 tile_point(double x, double y, double z) {
    return make_float3((float)wrap_half(x), (float)wrap_half(y), (float)wrap_half(z));
}
__device__ __forceinline__ float candidate_limit(double r2) { return (float)(r2 * (1.0 + 1e-4) + 2e-6); }
// Only the tile's points within the reach of the lanes' own tile's box are tested: near_point, once
// per point, leaves 1.6 to 2 times fewer of them than the boxes of the tile's groups of 8.
__device__ __forceinline__ bool near_point(float3 p, float4 c, float4 h, float limit) {
    constexpr float magic = 12582912.0f;  // 1.5 2^23: adding and subtracting it rounds to an integer
    float dx = p.x - c.x, dy = p.y - c.y, dz = p.z - c.z;
    dx -= (dx + magic) - magic; dy -= (dy + magic) - magic; dz -= (dz + magic) - magic;
    dx = fmaxf(fabsf(dx) - h.x, 0.f); dy = fmaxf(fabsf(dy) - h.y, 0.f); dz = fmaxf(fabsf(dz) - h.z, 0.f);
    return !(dx * dx + dy * dy + dz * dz >= limit);
}
// (b: the n near points, in groups of 4; what lies beyond them in the 32 places is masked)
__device__ __forceinline__ unsigned candidates(float3 a, const float3 *b, int n, float limit) {
    constexpr float magic = 12582912.0f;
    unsigned mask = 0;
    for (int g = 0; g < n; g += 4) {
        unsigned m = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float3 p = b[g + j];
            float dx = a.x - p.x, dy = a.y - p.y, dz = a.z - p.z;
            dx -= (dx + magic) - magic; dy -= (dy + magic) - magic; dz -= (dz + magic) - magic;
            if (!(dx * dx + dy * dy + dz * dz >= limit)) m |= 1u << j;
        }
        mask |= m << g;
    }
    return n < 32 ? mask & ((1u << n) - 1u) : mask;
}

// The lanes' candidates one after the other in the warp's queue (lane << 5 | j, in lane order):
// returns their number; *at: where the lane's own begin.
__device__ __forceinline__ int queue_pairs(unsigned mask, unsigned short *queue, int *at, int *check) {
    const int lane = threadIdx.x & 31, n = __popc(mask);
    int x = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    *at = x - n;
    for (int k = x - n; mask; mask &= mask - 1, ++k) queue[YAMC_IXC(k, kTile * kTile, check)] = (unsigned short)(lane << 5 | (__ffs(mask) - 1));
    return __shfl_sync(0xffffffffu, x, 31);
}

// EwaldSumRealSpace_calc on the full sum (EwaldSumRealSpace.f90:233-500): the energy totals of every
// pair once.  One block per tile (blockIdx.y: a share of its near tiles when the tiles alone do not
// fill the GPU), the near tiles dealt to the warps; per pair of tiles each lane finds its atom's
// candidates among the 32 others, and the warp evaluates all lanes' candidates 32 at a time, so the
// pair term runs on full warps.  Intra-molecular pairs use -erf_Luc and count in the intra totals
// too; LJ-LJ pairs of different molecules closer than their mean hard-core diameter set the overlap
// flag.  reach2: squared reach of the cutoff and the hard cores.  One partial per block, reduced in
// block order by k_sum_parts.
// Issue bound (63 % of the slots).  49,752 atoms: 3.23 ms over all pairs of 256-atom tiles, 0.76 ms over
// the near tiles with FP64 tests in the same loop, 0.39 ms with FP32 candidates from the groups of 8
// whose boxes are near (half the instructions tested them, 16 % were pairs), 0.35 ms from the near points.
static __global__ void __launch_bounds__(32 * kRealWarps) k_real_energy(DevSys D, const int *order, const float4 *box, int ntile,
                                                                        double reach2, double *part) {
    __shared__ TileAtom ai[kTile], aj[kRealWarps][kTile];
    __shared__ float3 fj[kRealWarps][kTile];
    __shared__ unsigned short queue[kRealWarps][kTile * kTile];
    __shared__ unsigned words[32];
    __shared__ int list[kNearSpan], count;
    __shared__ double red[kRealWarps][kFullParts], s6[kMaxDevTypes * kMaxDevTypes], fe[kMaxDevTypes * kMaxDevTypes];
    for (int k = threadIdx.x; k < D.nt * D.nt; k += blockDim.x) { s6[k] = D.lj_sig6[k]; fe[k] = D.lj_feps[k]; }
    const int ti = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ni = min(kTile, D.N - ti * kTile);
    if (warp == 0 && lane < ni) {
        const int i = (int)YAMC_IX(order[YAMC_IX(ti * kTile + lane, D.N)], D.N);
        ai[lane] = tile_atom(D, i, D.atom[i]);
    }
    __syncthreads();
    const float limit = candidate_limit(reach2);
    const float4 boxc = box[2 * ti], boxh = box[2 * ti + 1];
    const float3 own = tile_point(ai[min(lane, ni - 1)].x, ai[min(lane, ni - 1)].y, ai[min(lane, ni - 1)].z);
    double acc[6] = {0, 0, 0, 0, 0, 0};
    bool ovl = false;
    const int nt = D.nt;
    for (int base = 0; base < ntile; base += kNearSpan) {
        const int near = near_tiles<true, kRealWarps>(box, ntile, ti, base, reach2, words, list, &count, D.check);
        for (int m = blockIdx.y * kRealWarps + warp; m < near; m += gridDim.y * kRealWarps) {
            const int tj = list[YAMC_IX(m, kNearSpan)], ij = (int)YAMC_IX(order[YAMC_IX(min(tj * kTile + lane, D.N - 1), D.N)], D.N);
            const double4 v = D.atom[ij];
            const float3 f = tile_point(v.x, v.y, v.z);
            const bool in_reach = tj * kTile + lane < D.N && near_point(f, boxc, boxh, limit);
            const unsigned take = __ballot_sync(0xffffffffu, in_reach);
            __syncwarp();
            if (in_reach) {  // (the tile's own points are all in reach: each in its lane's place)
                const int k = __popc(take & ((1u << lane) - 1u));
                aj[warp][k] = tile_atom(D, ij, v);
                fj[warp][k] = f;
            }
            __syncwarp();
            unsigned mask = candidates(own, fj[warp], __popc(take), limit);
            if (tj == ti) mask &= lane < 31 ? ~((2u << lane) - 1u) : 0u;  // (each pair of the tile itself once)
            if (lane >= ni) mask = 0;
            int at;
            const int total = queue_pairs(mask, queue[warp], &at, D.check);
            __syncwarp();
            for (int q = lane; q < total; q += 32) {
                const int pair = queue[warp][YAMC_IX(q, kTile * kTile)];
                const TileAtom &a = ai[pair >> 5], &b = aj[warp][pair & 31];
                const double dx = min_image(a.x - b.x), dy = min_image(a.y - b.y), dz = min_image(a.z - b.z);
                const double r2 = dx * dx + dy * dy + dz * dz;
                const bool lj = a.type > 0 && b.type > 0, same = a.mol == b.mol;
                if (lj && !same) {
                    const double d12 = (a.dhs + b.dhs) / 2;
                    if (r2 < d12 * d12) ovl = true;
                }
                if (r2 >= D.rmax2) continue;
                const int off = lj ? (a.type - 1) * nt + (b.type - 1) : 0;
                const PairTerm<double> t = pair_term<double, false>(r2, D.xclb * a.q * b.q, lj, lj ? s6[off] : 0.0,
                                                                     lj ? fe[off] : 0.0, D.alpha, D.taosp, same);
                acc[0] += t.ew; acc[1] += t.lj6; acc[2] += t.lj12;
                if (same) { acc[3] += t.ew; acc[4] += t.lj6; acc[5] += t.lj12; }
            }
        }
        __syncthreads();
    }
    const double s = warp_sums(acc);
    const bool any = __any_sync(0xffffffffu, ovl);
    if (!(lane & 1) && lane < 12) red[warp][lane >> 1] = s;
    if (lane == 31) { red[warp][6] = any ? 1.0 : 0.0; red[warp][7] = 0.0; }
    __syncthreads();
    if (threadIdx.x < kFullParts) {
        double x = 0;
        for (int w = 0; w < kRealWarps; ++w) x += red[w][threadIdx.x];
        part[(size_t)threadIdx.x * gridDim.x * gridDim.y + (size_t)blockIdx.y * gridDim.x + ti] = x;
    }
}

// The adjoint's real space (F_i += FR (r_i - r_j), intra-molecular pairs with the -erf_Luc energy):
// every tile over all its near tiles as in k_real_energy; the forces of a batch of candidates go to
// shared memory, where each lane adds those of its own atom (they follow one another in the queue),
// the warps' sums are added in order.  gf[(blockIdx.y 3 + component) N + atom].
// 49,752 atoms: 11.5 ms over all tiles, 0.93 ms; 12,440 atoms: 0.59 ms with every lane evaluating its
// own pairs from a bit mask, 0.30 ms so, 0.28 ms with candidates from the near points only.
constexpr int kForceBatch = 128;  // candidates evaluated between two gathers
static __global__ void __launch_bounds__(32 * kRealWarps) k_real_forces(DevSys D, const int *order, const float4 *box, int ntile,
                                                                        double reach2, double *gf) {
    extern __shared__ double batch[];  // [kRealWarps][3][kForceBatch]
    __shared__ TileAtom ai[kTile], aj[kRealWarps][kTile];
    __shared__ float3 fj[kRealWarps][kTile];
    __shared__ unsigned short queue[kRealWarps][kTile * kTile];
    __shared__ unsigned words[32];
    __shared__ int list[kNearSpan], count;
    __shared__ double s6[kMaxDevTypes * kMaxDevTypes], fe[kMaxDevTypes * kMaxDevTypes];
    for (int k = threadIdx.x; k < D.nt * D.nt; k += blockDim.x) { s6[k] = D.lj_sig6[k]; fe[k] = D.lj_feps[k]; }
    const int ti = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ni = min(kTile, D.N - ti * kTile);
    if (warp == 0 && lane < ni) {
        const int i = (int)YAMC_IX(order[YAMC_IX(ti * kTile + lane, D.N)], D.N);
        ai[lane] = tile_atom(D, i, D.atom[i]);
    }
    __syncthreads();
    const float limit = candidate_limit(reach2);
    const float4 boxc = box[2 * ti], boxh = box[2 * ti + 1];
    const float3 own = tile_point(ai[min(lane, ni - 1)].x, ai[min(lane, ni - 1)].y, ai[min(lane, ni - 1)].z);
    double *bx = batch + (size_t)warp * 3 * kForceBatch, *by = bx + kForceBatch, *bz = by + kForceBatch;
    double gx = 0, gy = 0, gz = 0;
    const int nt = D.nt;
    for (int base = 0; base < ntile; base += kNearSpan) {
        const int near = near_tiles<false, kRealWarps>(box, ntile, ti, base, reach2, words, list, &count, D.check);
        for (int m = blockIdx.y * kRealWarps + warp; m < near; m += gridDim.y * kRealWarps) {
            const int tj = list[YAMC_IX(m, kNearSpan)], ij = (int)YAMC_IX(order[YAMC_IX(min(tj * kTile + lane, D.N - 1), D.N)], D.N);
            const double4 v = D.atom[ij];
            const float3 f = tile_point(v.x, v.y, v.z);
            const bool in_reach = tj * kTile + lane < D.N && near_point(f, boxc, boxh, limit);
            const unsigned take = __ballot_sync(0xffffffffu, in_reach);
            __syncwarp();
            if (in_reach) {  // (the tile's own points are all in reach: each in its lane's place)
                const int k = __popc(take & ((1u << lane) - 1u));
                aj[warp][k] = tile_atom(D, ij, v);
                fj[warp][k] = f;
            }
            __syncwarp();
            unsigned mask = candidates(own, fj[warp], __popc(take), limit);
            if (tj == ti) mask &= ~(1u << lane);
            if (lane >= ni) mask = 0;
            int at;
            const int mine = __popc(mask), total = queue_pairs(mask, queue[warp], &at, D.check);
            __syncwarp();
            for (int q0 = 0; q0 < total; q0 += kForceBatch) {
                const int q1 = min(total, q0 + kForceBatch);
                for (int q = q0 + lane; q < q1; q += 32) {
                    const int pair = queue[warp][YAMC_IX(q, kTile * kTile)];
                    const TileAtom &a = ai[pair >> 5], &b = aj[warp][pair & 31];
                    const double dx = min_image(a.x - b.x), dy = min_image(a.y - b.y), dz = min_image(a.z - b.z);
                    const double r2 = dx * dx + dy * dy + dz * dz;
                    double FR = 0.0;
                    const bool in = !(r2 >= D.rmax2);
                    if (in) {
                        const bool lj = a.type > 0 && b.type > 0;
                        const int off = lj ? (a.type - 1) * nt + (b.type - 1) : 0;
                        FR = pair_force_adjoint<double>(r2, D.xclb * a.q * b.q, lj, lj ? s6[off] : 0.0,
                                                        lj ? fe[off] : 0.0, D.alpha, a.mol == b.mol);
                    }
                    bx[q - q0] = in ? dx * FR : 0.0; by[q - q0] = in ? dy * FR : 0.0; bz[q - q0] = in ? dz * FR : 0.0;
                }
                __syncwarp();
                for (int q = max(at, q0), e = min(at + mine, q1); q < e; ++q) { gx += bx[q - q0]; gy += by[q - q0]; gz += bz[q - q0]; }
                __syncwarp();
            }
        }
        __syncthreads();
    }
    bx[lane] = gx; by[lane] = gy; bz[lane] = gz;
    __syncthreads();
    if (warp < 3 && lane < ni) {
        double x = 0;
        for (int w = 0; w < kRealWarps; ++w) x += batch[((size_t)w * 3 + warp) * kForceBatch + lane];
        gf[((size_t)blockIdx.y * 3 + warp) * D.N + YAMC_IX(order[YAMC_IX(ti * kTile + lane, D.N)], D.N)] = x;
    }
}

// ------------------------------------------------------------------------------------------
// k space along the rows of the k grid
// ------------------------------------------------------------------------------------------
// The atoms of each structure: list 0 the charged atoms (weight q), list t the atoms of LJ type t
// (weight 1), each padded to a multiple of 32 with -1, one after the other in `alist`; lbeg[l] is
// where list l begins.
constexpr int kMaxLists = 1 + 4;
struct AtomLists { const int *alist; int lbeg[kMaxLists + 1]; };

// One thread's part of the structure factors: the rows (kx, +-ky) and kRowZ consecutive kz >= 0 from
// z0; emap[kRowZ item + j] = the entries of (+ky, +kz), (+ky, -kz), (-ky, +kz), (-ky, -kz), -1 where
// there is none.
constexpr int kRowZ = 4;
constexpr int kRhoChunk = 32;        // atoms whose phase tables a block holds at a time
constexpr int kRhoMaxThreads = 512;  // items of a block: its tables serve up to 512 rows

// RhoSquared_addAtoms (RhoSquared.f90:188-243) per structure (blockIdx.y: one slice of one list).
// The eight sums over the slice's atoms of w (cos, sin)(kx x) (cos, sin)(ky y) (cos, sin)(kz z) give
// the four signs of (ky, kz): 8 FMAs per 4 signed entries, the product of the first two factors once
// per row.  The items of a warp share z0 (sorted by it).  part[slice S + e]; k_rho_reduce adds a
// list's slices.  FP64 pipe bound while it sums (38 operations per atom and 16 signed entries, against
// 16 per entry of the full product), with the tables' phases and three barriers per 32 atoms between
// (pipe 53 % active over the kernel); both signs of ky in one thread, since a 16-byte shared load fills
// 512 bytes of registers, four cycles of an SM, broadcast or not (7 loads per 36 operations, 11 with
// one sign and 8 kz).  49,752 atoms x 29,784 entries: 5.7 ms with the full product per entry, 0.74 ms
// with one sign of ky per thread, 0.72 ms so.
static __global__ void __launch_bounds__(kRhoMaxThreads) k_rho_rows(DevSys D, AtomLists L, const int4 *slices, const int4 *items,
                                                                    const int4 *emap, int nitem, double2 *part) {
    extern __shared__ double2 rtab[];  // [3][KM][kRhoChunk + 1], then kRowZ rows of zeros
    __shared__ double4 atom[kRhoChunk];  // the chunk's atoms: x, y, z, weight (0 past the list's end)
    const int KM = D.kmax + 1, P = kRhoChunk + 1;
    const int it = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = it < nitem;
    const int4 im = items[min(it, nitem - 1)];  // kx, ky, z0, number of kz
    const int4 sl = slices[blockIdx.y];         // list, first position, end
    const double2 *tx = rtab + im.x * P, *ty = rtab + (KM + im.y) * P, *tz = rtab + (2 * KM + im.z) * P;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int nbase = min(8, KM) + (KM - 1) / 8;  // multiples 0..7, 8, 16, ... of an axis
    // sums of the products cc, ss, sc, cs of the x and y factors with cos and sin of kz z
    double2 cc[kRowZ], ss[kRowZ], sc[kRowZ], cs[kRowZ];
#pragma unroll
    for (int j = 0; j < kRowZ; ++j) cc[j] = ss[j] = sc[j] = cs[j] = make_double2(0.0, 0.0);
    // (the next chunk's atoms are on their way while this one is summed)
    auto fetch = [&](int p) {
        const int i = p < sl.z ? L.alist[YAMC_IX(p, L.lbeg[kMaxLists])] : -1;
        double4 v = make_double4(0.0, 0.0, 0.0, 0.0);
        if (i >= 0) { v = D.atom[YAMC_IX(i, D.N)]; if (sl.x > 0) v.w = 1.0; }
        return v;
    };
    for (int k = threadIdx.x; k < kRowZ * P; k += blockDim.x) rtab[3 * KM * P + k] = make_double2(0.0, 0.0);
    double4 next = make_double4(0.0, 0.0, 0.0, 0.0);
    if (warp == 0) next = fetch(sl.y + lane);
    for (int a0 = sl.y; a0 < sl.z; a0 += kRhoChunk) {
        if (warp == 0) {
            atom[lane] = next;
            next = fetch(a0 + kRhoChunk + lane);
        }
        __syncthreads();
        const double4 p = atom[lane];
        // the axis tables: multiples 0..7 and 8, 16, ... from sincospi, the others as the product of
        // two of those (one rounding more than sincospi of the multiple; a quarter of the work)
        for (int r = warp; r < 3 * nbase; r += nw) {
            const int d = r >= 2 * nbase ? 2 : (r >= nbase ? 1 : 0), b = r - d * nbase, m = b < 8 ? b : 8 * (b - 7);
            const double u = d == 0 ? p.x : (d == 1 ? p.y : p.z);
            double s, c;
            sincospi(2.0 * (double)m * u, &s, &c);
            if (m == 0) { s = 0.0; c = 1.0; }
            rtab[(d * KM + m) * P + lane] = make_double2(c, s);
        }
        __syncthreads();
        for (int r = warp; r < 3 * (KM - nbase); r += nw) {
            const int d = r >= 2 * (KM - nbase) ? 2 : (r >= KM - nbase ? 1 : 0), b = r - d * (KM - nbase);
            const int hi = 8 * (1 + b / 7), lo = 1 + b % 7;
            const double2 A = rtab[(d * KM + hi) * P + lane];
            const double2 B = rtab[(d * KM + lo) * P + lane];
            rtab[(d * KM + hi + lo) * P + lane] = make_double2(A.x * B.x - A.y * B.y, A.y * B.x + A.x * B.y);
        }
        __syncthreads();
        const int na = min(kRhoChunk, sl.z - a0);
#pragma unroll 2
        for (int a = 0; a < na; ++a) {
            const double2 X = tx[a], Y = ty[a];
            const double w = atom[a].w, cy = w * Y.x, sy = w * Y.y;
            const double pcc = X.x * cy, pss = X.y * sy, psc = X.y * cy, pcs = X.x * sy;
#pragma unroll
            for (int j = 0; j < kRowZ; ++j) {
                const double2 Z = tz[j * P + a];  // (past the row's last kz: sums that are not stored)
                cc[j].x += pcc * Z.x; cc[j].y += pcc * Z.y; ss[j].x += pss * Z.x; ss[j].y += pss * Z.y;
                sc[j].x += psc * Z.x; sc[j].y += psc * Z.y; cs[j].x += pcs * Z.x; cs[j].y += pcs * Z.y;
            }
        }
        __syncthreads();
    }
    if (valid) {
        double2 *out = part + (size_t)blockIdx.y * D.S;
#pragma unroll
        for (int j = 0; j < kRowZ; ++j) {
            if (j >= im.w) continue;
            const int4 e = emap[(size_t)it * kRowZ + j];
#pragma unroll
            for (int y = 0; y < 2; ++y) {  // A = X^kx Y^(+-ky): sums of A.re cos, A.im sin, A.re sin, A.im cos
                const double rc = y ? cc[j].x + ss[j].x : cc[j].x - ss[j].x, is = y ? sc[j].y - cs[j].y : sc[j].y + cs[j].y;
                const double rs = y ? cc[j].y + ss[j].y : cc[j].y - ss[j].y, ic = y ? sc[j].x - cs[j].x : sc[j].x + cs[j].x;
                const int ep = y ? e.z : e.x, em = y ? e.w : e.y;
                if (ep >= 0) out[YAMC_IX(ep, D.S)] = make_double2(rc - is, rs + ic);
                if (em >= 0) out[YAMC_IX(em, D.S)] = make_double2(rc + is, ic - rs);
            }
        }
    }
}

// rho[l S + e] = sum over the slices of list l; sbeg: the lists' first slices (a list without atoms
// has none: its row is 0).  32 entries per block; its 8 warps each add every eighth slice in order,
// then their sums are added in order.
static __global__ void __launch_bounds__(256) k_rho_reduce(const double2 *part, const int *sbeg, int S, double2 *rho) {
    __shared__ double2 red[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, e = blockIdx.x * 32 + lane, l = blockIdx.y;
    double c = 0, s = 0;
    const int s1 = sbeg[l + 1];
    if (e < S)
#pragma unroll 8
        for (int k = sbeg[l] + warp; k < s1; k += 8) {
            const double2 v = part[(size_t)k * S + e];
            c = c + v.x; s = s + v.y;
        }
    red[warp][lane] = make_double2(c, s);
    __syncthreads();
    if (warp == 0 && e < S) {
        for (int w = 1; w < 8; ++w) { c += red[w][lane].x; s += red[w][lane].y; }
        rho[(size_t)l * S + e] = make_double2(c, s);
    }
}

// The fields that the k-space forces sum: for list l and each (kx, ky >= 0, kz >= 0) the rows +ky
// and -ky of (a, b, c, d) = (Gr+ + Gr-, Gr+ - Gr-, Gi+ + Gi-, Gi+ - Gi-) over the signs of kz, with
// G = beta rho (Coulomb) or the sum over types t' of beta_LJ(t, t') rho_t'.  fmap: the entries of
// (+ky, +kz), (+ky, -kz), (-ky, +kz), (-ky, -kz), -1 where there is none.
template <int NT>
static __global__ void __launch_bounds__(256) k_row_fields(DevSys D, const int4 *fmap, int nf, double4 *field) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x, l = blockIdx.y;
    if (f >= nf) return;
    const int4 m = fmap[f];
    int e[4] = {m.x, m.y, m.z, m.w};
    double2 g[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        g[k] = make_double2(0.0, 0.0);
        if (e[k] < 0) continue;
        e[k] = (int)YAMC_IX(e[k], D.S);
        if (l == 0) {
            const double2 r = D.rho[e[k]];
            const double b = D.ebeta[e[k]];
            g[k] = make_double2(b * r.x, b * r.y);
        } else {
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                const double2 r = D.rho[(size_t)(1 + t) * D.S + e[k]];
                const double b = D.ebetalj[(size_t)pair_idx<NT>(l - 1, t) * D.S + e[k]];
                g[k].x += b * r.x; g[k].y += b * r.y;
            }
        }
    }
#pragma unroll
    for (int y = 0; y < 2; ++y)
        field[((size_t)l * nf + f) * 2 + y] = make_double4(g[2 * y].x + g[2 * y + 1].x, g[2 * y].x - g[2 * y + 1].x,
                                                           g[2 * y].y + g[2 * y + 1].y, g[2 * y].y - g[2 * y + 1].y);
}

// k-space forces (ForceKSpace_coulomb / _LJ, ForceKSpace.f90:59-302): for an atom the weight of a
// signed k vector is w = G.re sin - G.im cos of its phase; with A = X^kx Y^ky the sums over kz of a
// row give w = A.im R1 + A.re R2 (and the kz-weighted sums the z component), 4 FMAs per signed k
// vector, the phase of a single k vector never formed.  A block holds 32 A atoms of one list (their
// axis tables in shared memory), its warps take the row pairs (kx, +-ky) in turn, a lane A atoms;
// blockIdx.y splits the row pairs when the atoms alone do not fill the GPU.  rows: (kx, ky, first
// field, number of kz).  kf[(y 3 + component) npos + position].
// With one atom per lane the loads bind: 4 uniform 16-byte loads and one of the lane's table per 18 FP64
// operations, 20 cycles of an SM against 9.  Two atoms share the uniform loads (24 against 18); the wait for
// the fields' loads leads then (2.9 of 9 cycles per instruction; load pipe 65 %, FP64 pipe 57 %).
// 49,752 atoms x 29,784 entries: 6.6 ms with the phase formed per atom and entry, 1.56 ms with one
// atom per lane, 1.23 ms with two.
constexpr int kForceRowWarps = 8;
template <int A>
static __global__ void __launch_bounds__(32 * kForceRowWarps) k_forces_rows(DevSys D, AtomLists L, const int4 *rows, int nrow,
                                                                            const double4 *field, int nf, int npos, double *kf) {
    constexpr int W = 32 * A;
    extern __shared__ double2 ftab[];  // [3][KM][W]
    __shared__ double red[kForceRowWarps][3][W];
    const int KM = D.kmax + 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int l = 0, b = blockIdx.x;
    for (int n; b >= (n = (L.lbeg[l + 1] - L.lbeg[l] + W - 1) / W); ++l) b -= n;
    const int p0 = L.lbeg[l] + W * b, pe = L.lbeg[l + 1];
    const double4 *F = field + (size_t)l * nf * 2;
    for (int idx = threadIdx.x; idx < W * 3 * KM; idx += blockDim.x) {
        const int r = idx / W, d = r / KM, m = r % KM, p = p0 + idx % W, i = p < pe ? L.alist[YAMC_IX(p, L.lbeg[kMaxLists])] : -1;
        double s = 0.0, c = 0.0;
        if (i >= 0) {
            const double4 v = D.atom[YAMC_IX(i, D.N)];
            const double u = d == 0 ? v.x : (d == 1 ? v.y : v.z);
            sincospi(2.0 * (double)m * u, &s, &c);
            if (m == 0) { s = 0.0; c = 1.0; }
        }
        ftab[idx] = make_double2(c, s);
    }
    __syncthreads();
    double gx[A] = {}, gy[A] = {}, gz[A] = {};
    for (int r = blockIdx.y * kForceRowWarps + warp; r < nrow; r += gridDim.y * kForceRowWarps) {
        const int4 row = rows[r];
        const double2 *tz = ftab + 2 * KM * W + lane;
        const double4 *f = F + 2 * (size_t)YAMC_IX(row.z, nf - row.w + 1);
        double r1[A][2] = {}, r2[A][2] = {}, z1[A][2] = {}, z2[A][2] = {};
#pragma unroll (4 / A)
        for (int k = 0; k < row.w; ++k) {
            double2 Z[A];
            double kc[A], ks[A];
#pragma unroll
            for (int a = 0; a < A; ++a) {
                Z[a] = tz[k * W + 32 * a];
                kc[a] = (double)k * Z[a].x; ks[a] = (double)k * Z[a].y;
            }
#pragma unroll
            for (int y = 0; y < 2; ++y) {
                const double2 ab = __ldg(reinterpret_cast<const double2 *>(f + 2 * k + y));
                const double2 cd = __ldg(reinterpret_cast<const double2 *>(f + 2 * k + y) + 1);
#pragma unroll
                for (int a = 0; a < A; ++a) {
                    r1[a][y] += ab.x * Z[a].x; r1[a][y] += cd.y * Z[a].y;
                    r2[a][y] += ab.y * Z[a].y; r2[a][y] -= cd.x * Z[a].x;
                    z1[a][y] += ab.y * kc[a]; z1[a][y] += cd.x * ks[a];
                    z2[a][y] += ab.x * ks[a]; z2[a][y] -= cd.y * kc[a];
                }
            }
        }
#pragma unroll
        for (int a = 0; a < A; ++a) {
            const double2 X = ftab[row.x * W + 32 * a + lane], Y = ftab[(KM + row.y) * W + 32 * a + lane];
#pragma unroll
            for (int y = 0; y < 2; ++y) {
                const double sy = y ? -Y.y : Y.y;
                const double ar = X.x * Y.x - X.y * sy, ai = X.y * Y.x + X.x * sy;
                const double w = ai * r1[a][y] + ar * r2[a][y];
                gx[a] += (double)row.x * w;
                gy[a] += (double)(y ? -row.y : row.y) * w;
                gz[a] += ai * z1[a][y] + ar * z2[a][y];
            }
        }
    }
#pragma unroll
    for (int a = 0; a < A; ++a) {
        red[warp][0][32 * a + lane] = gx[a]; red[warp][1][32 * a + lane] = gy[a]; red[warp][2][32 * a + lane] = gz[a];
    }
    __syncthreads();
    if (warp < 3) {
#pragma unroll
        for (int a = 0; a < A; ++a) {
            double x = 0;
            for (int w = 0; w < kForceRowWarps; ++w) x += red[w][warp][32 * a + lane];
            if (p0 + 32 * a < pe) kf[((size_t)blockIdx.y * 3 + warp) * npos + p0 + 32 * a + lane] = x;
        }
    }
}

// The forces of every atom: the real-space parts (nreal of them) in order, plus 4 pi (q kf of the
// atom's place in list 0 + kf of its place in its type's list), the parts of the row split in order;
// place: the two positions, -1 where the atom is not in a list.  f[component N + atom].
static __global__ void k_forces_add(DevSys D, const int2 *place, const double *gf, int nreal, const double *kf, int npos, int nsplit,
                                    double *f) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= D.N) return;
    const int2 p = place[i];
    const double q = D.atom[i].w;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        double g = 0, a = 0, b = 0;
        for (int s = 0; s < nreal; ++s) g += gf[((size_t)s * 3 + c) * D.N + i];
        for (int s = 0; s < nsplit; ++s) {
            const double *v = kf + ((size_t)s * 3 + c) * npos;
            if (p.x >= 0) a += v[YAMC_IX(p.x, npos)];
            if (p.y >= 0) b += v[YAMC_IX(p.y, npos)];
        }
        f[(size_t)c * D.N + i] = g + kFourPi * (q * a + b);
    }
}

// ------------------------------------------------------------------------------------------
// radial distribution functions: the pairs of near tiles (count_distances, mcrdf2.f90:110-333)
// ------------------------------------------------------------------------------------------
// Every ordered pair of centres of the tile and its near tiles, counted as k_rdf_count counts it
// (the same explicitly rounded distance, so the same bins), for frames without periodic images
// (rmax < L / 2).  16,984 centres, rmax 12 of 79.3 A: 2.1 ms over all pairs, 0.10 ms; the barriers around
// each tile's near list bind (4.9 of 13 cycles per instruction; load pipe 50 %).
static __global__ void __launch_bounds__(256) k_rdf_tiles(const double *cx, const double *cy, const double *cz, const int *type,
                                                          const int *order, const float4 *box, int ntile, double reach2, int M,
                                                          int ntypes, int nbin, double L, double dr, double rmax2,
                                                          unsigned long long *hist) {
    extern __shared__ unsigned int hs[];
    __shared__ unsigned words[32];
    __shared__ int list[kNearSpan], count;
    __shared__ double4 ci[kTile], cj[8][kTile];  // x, y, z, type
    __shared__ float3 fj[8][kTile];
    __shared__ unsigned short queue[8][kTile * kTile];
    const int npair = ntypes * ntypes, nh = npair * nbin + npair;
    for (int k = threadIdx.x; k < nh; k += blockDim.x) hs[k] = 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float limit = candidate_limit(reach2);
    auto centre = [&](int p) {
        const int i = order[min(p, M - 1)];
        return make_double4(cx[i], cy[i], cz[i], (double)(type[i] - 1));
    };
    for (int ti = blockIdx.x; ti < ntile; ti += gridDim.x) {
        __syncthreads();
        if (warp == 0) ci[lane] = centre(ti * kTile + lane);
        __syncthreads();
        const int ni = min(kTile, M - ti * kTile);
        const float4 boxc = box[2 * ti], boxh = box[2 * ti + 1];
        const float3 own = tile_point(ci[lane].x, ci[lane].y, ci[lane].z);
        for (int base = 0; base < ntile; base += kNearSpan) {
            const int near = near_tiles<false, 8>(box, ntile, ti, base, reach2, words, list, &count, nullptr);
            for (int m = blockIdx.y * 8 + warp; m < near; m += gridDim.y * 8) {
                const int tj = list[m];
                const double4 p = centre(tj * kTile + lane);
                const float3 f = tile_point(p.x, p.y, p.z);
                const bool in_reach = tj * kTile + lane < M && near_point(f, boxc, boxh, limit);
                const unsigned take = __ballot_sync(0xffffffffu, in_reach);
                __syncwarp();
                if (in_reach) {
                    const int k = __popc(take & ((1u << lane) - 1u));
                    cj[warp][k] = p;
                    fj[warp][k] = f;
                }
                __syncwarp();
                unsigned mask = candidates(own, fj[warp], __popc(take), limit);
                if (tj == ti) mask &= ~(1u << lane);
                if (lane >= ni) mask = 0;
                int at;
                const int total = queue_pairs(mask, queue[warp], &at, nullptr);
                __syncwarp();
                for (int q = lane; q < total; q += 32) {
                    const double4 a = ci[queue[warp][q] >> 5], b = cj[warp][queue[warp][q] & 31];
                    double x2 = b.x, y2 = b.y, z2 = b.z;
                    if (__dsub_rn(a.x, x2) > 0.5) x2 = __dadd_rn(x2, 1.0);
                    if (__dsub_rn(a.x, x2) < -0.5) x2 = __dsub_rn(x2, 1.0);
                    if (__dsub_rn(a.y, y2) > 0.5) y2 = __dadd_rn(y2, 1.0);
                    if (__dsub_rn(a.y, y2) < -0.5) y2 = __dsub_rn(y2, 1.0);
                    if (__dsub_rn(a.z, z2) > 0.5) z2 = __dadd_rn(z2, 1.0);
                    if (__dsub_rn(a.z, z2) < -0.5) z2 = __dsub_rn(z2, 1.0);
                    const double dx = __dmul_rn(__dsub_rn(a.x, x2), L), dy = __dmul_rn(__dsub_rn(a.y, y2), L),
                                 dz = __dmul_rn(__dsub_rn(a.z, z2), L);
                    const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
                    if (!(r2 <= __dsub_rn(rmax2, 1e-10))) continue;  // (a NaN, whose bin would be no index, too)
                    const int t1 = (int)a.w, t2 = (int)b.w, off = t1 < t2 ? t1 * ntypes + t2 : t2 * ntypes + t1;
                    const int bin = (int)__ddiv_rn(__dsqrt_rn(r2), dr);
                    atomicAdd(&hs[npair * nbin + off], 1u);
                    if (bin < nbin) atomicAdd(&hs[off * nbin + bin], 1u);
                }
            }
            __syncthreads();
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < nh; k += blockDim.x)
        if (hs[k]) atomicAdd(&hist[k], (unsigned long long)hs[k]);
}

}  // namespace yamc
