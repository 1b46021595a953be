// kernels_sort.cu -- labelling and the counting sort of particles by cell.
//
// Replaces labelGrid (FluidSolver3D.cu:340-397: ClearNonSolidFunctor,
// MarkBodyCellsFunctor, MarkFluidCellsFunctor).  The cell key is the
// reference's floorf(p/dx) with its clamp, so labels are bit-identical; the
// FLUID mark falls out of the per-cell particle counts that the sort needs
// anyway.  The sort is a counting sort: one atomic per particle for its rank
// in its cell, a three-pass exclusive scan of the counts into cell offsets,
// and a scatter of the particle records into cell order.
#include "kernels.hpp"
#include "scan.cuh"

namespace fp {

namespace {
constexpr int SCAN_BLOCK = 1024;
constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_TILE = SCAN_BLOCK * SCAN_ITEMS;

// Particles arrive nearly in cell order (sorted last step, moved less than a
// cell), so a warp's lanes share a few cells: one atomic per distinct cell of
// the warp (lanes grouped by __match_any_sync), each lane's rank the group's
// base plus its place among the group's lanes.  The order of a cell's
// particles is arbitrary either way.  Every lane of every warp reaches the
// match (the block size is a multiple of 32; lanes past np carry key -1).
//
// Bound by the latency of the positions and of the atomics, so a thread takes
// BIN_ITEMS particles and issues their loads, then their atomics, together:
// 16.6 us at 128^3 (3.8 M particles), 43 at 160^3 (11 M), 71 for 17.5 M (64 at
// memory speed), against 24, 68 and 106 with one particle a thread.
constexpr int BIN_THREADS = 256, BIN_ITEMS = 4;
template <bool P2>
__global__ void __launch_bounds__(BIN_THREADS) k_bin(const float4* __restrict__ pos, int64_t np, Dims g,
                                                     int* __restrict__ counts, int* __restrict__ key,
                                                     int* __restrict__ rank) {
    const int64_t q0 = int64_t(blockIdx.x) * (BIN_THREADS * BIN_ITEMS) + threadIdx.x;
    const int lane = threadIdx.x & 31;
    float4 p[BIN_ITEMS];
    int c[BIN_ITEMS], at[BIN_ITEMS];
    unsigned grp[BIN_ITEMS];
#pragma unroll
    for (int m = 0; m < BIN_ITEMS; ++m) {
        const int64_t q = q0 + m * BIN_THREADS;
        if (q < np) p[m] = pos[q];
    }
#pragma unroll
    for (int m = 0; m < BIN_ITEMS; ++m) {
        const bool ok = q0 + m * BIN_THREADS < np;
        c[m] = ok ? cell_key<P2>(p[m].x, p[m].y, p[m].z, g) : -1;
        grp[m] = __match_any_sync(0xffffffffu, c[m]);
        at[m] = 0;
        if (ok && lane == __ffs(grp[m]) - 1) at[m] = atomicAdd(&counts[c[m]], __popc(grp[m]));
    }
#pragma unroll
    for (int m = 0; m < BIN_ITEMS; ++m) {
        const int64_t q = q0 + m * BIN_THREADS;
        const int first = __shfl_sync(0xffffffffu, at[m], __ffs(grp[m]) - 1);
        if (q < np) {
            key[q] = c[m];
            rank[q] = first + __popc(grp[m] & ((1u << lane) - 1u));
        }
    }
}

__device__ __forceinline__ uint8_t label_of(uint8_t base, uint8_t body, int count) {
    if (base == SOLID) return SOLID;        // ClearNonSolidFunctor keeps SOLID
    if (body) return BODY;                  // MarkBodyCellsFunctor
    return count > 0 ? FLUID : AIR;         // MarkFluidCellsFunctor
}

// The four counts from e0 on (a multiple of four; 0 beyond the grid), as one
// vector where they lie inside.
static_assert(SCAN_ITEMS == 4, "vectors of four");
__device__ __forceinline__ int4 load_counts(const int* __restrict__ counts, int64_t e0, int64_t nc) {
    if (e0 + 3 < nc) return *reinterpret_cast<const int4*>(counts + e0);
    int4 v = make_int4(0, 0, 0, 0);
    if (e0 < nc) v.x = counts[e0];
    if (e0 + 1 < nc) v.y = counts[e0 + 1];
    if (e0 + 2 < nc) v.z = counts[e0 + 2];
    return v;
}

// Pass 1: labels and the per-tile sums of the counts.  Both passes are bound by
// memory: with vectors of four cells 10 and 7.5 us at 160^3, 17.5 and 13 for 256
// x 128 x 256, against 12 and 13, 20 and 25 cell by cell.
__global__ void __launch_bounds__(SCAN_BLOCK) k_label_tiles(const uint8_t* __restrict__ base,
                                                            const uint8_t* __restrict__ body,
                                                            const int* __restrict__ counts,
                                                            uint8_t* __restrict__ labels, int64_t nc,
                                                            int* __restrict__ tile_sums) {
    const int64_t e0 = int64_t(blockIdx.x) * SCAN_TILE + int64_t(threadIdx.x) * SCAN_ITEMS;
    const int4 v = load_counts(counts, e0, nc);
    if (e0 + 3 < nc) {
        const uchar4 s = *reinterpret_cast<const uchar4*>(base + e0);
        const uchar4 b = body ? *reinterpret_cast<const uchar4*>(body + e0) : make_uchar4(0, 0, 0, 0);
        *reinterpret_cast<uchar4*>(labels + e0) =
            make_uchar4(label_of(s.x, b.x, v.x), label_of(s.y, b.y, v.y), label_of(s.z, b.z, v.z), label_of(s.w, b.w, v.w));
    } else {
        const int c[3] = {v.x, v.y, v.z};
#pragma unroll
        for (int t = 0; t < 3; ++t)
            if (e0 + t < nc) labels[e0 + t] = label_of(base[e0 + t], body ? body[e0 + t] : 0, c[t]);
    }
    int total;
    block_exclusive_scan<SCAN_BLOCK>(v.x + v.y + v.z + v.w, total);
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

// Pass 3: exclusive scan inside each tile plus the tile offset; the counts that
// are not 0 become 0 again, ready for the next sort.
__global__ void __launch_bounds__(SCAN_BLOCK) k_start_tiles(int* __restrict__ counts, int64_t nc,
                                                            const int* __restrict__ tile_offsets,
                                                            int* __restrict__ start) {
    const int64_t e0 = int64_t(blockIdx.x) * SCAN_TILE + int64_t(threadIdx.x) * SCAN_ITEMS;
    const int4 v = load_counts(counts, e0, nc);
    int total;
    int4 o;
    o.x = block_exclusive_scan<SCAN_BLOCK>(v.x + v.y + v.z + v.w, total) + tile_offsets[blockIdx.x];
    o.y = o.x + v.x;
    o.z = o.y + v.y;
    o.w = o.z + v.z;
    if (e0 + 3 < nc) {
        *reinterpret_cast<int4*>(start + e0) = o;
        if (v.x | v.y | v.z | v.w) *reinterpret_cast<int4*>(counts + e0) = make_int4(0, 0, 0, 0);
    } else {
        const int c[3] = {o.x, o.y, o.z};
#pragma unroll
        for (int t = 0; t < 3; ++t)
            if (e0 + t < nc) {
                start[e0 + t] = c[t];
                counts[e0 + t] = 0;
            }
    }
}

__global__ void k_scatter(const float4* __restrict__ pos, const float4* __restrict__ vel,
                          const int* __restrict__ key, const int* __restrict__ rank,
                          const int* __restrict__ start, int64_t np, float4* __restrict__ pos2,
                          float4* __restrict__ vel2) {
    int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (q >= np) return;
    int slot = start[key[q]] + rank[q];
    pos2[slot] = pos[q];
    vel2[slot] = vel[q];
}

// 16 consecutive ints per thread and pass, as four vectors (data is 16-byte
// aligned): one pass of a block covers 16,384.
__device__ __forceinline__ void scan_block(int* data, int n, int* total) {
    constexpr int ITEMS = 16;
    int carry = 0;
    for (int base = 0; base < n; base += 1024 * ITEMS) {
        const int e0 = base + int(threadIdx.x) * ITEMS;
        int v[ITEMS];
#pragma unroll
        for (int t = 0; t < ITEMS; t += 4) {
            if (e0 + t + 3 < n) {
                const int4 q = *reinterpret_cast<const int4*>(data + e0 + t);
                v[t] = q.x; v[t + 1] = q.y; v[t + 2] = q.z; v[t + 3] = q.w;
            } else {
                for (int u = 0; u < 4; ++u) v[t + u] = e0 + t + u < n ? data[e0 + t + u] : 0;
            }
        }
        int s = 0;
#pragma unroll
        for (int t = 0; t < ITEMS; ++t) s += v[t];
        int tot;
        int pre = carry + block_exclusive_scan<1024>(s, tot);
#pragma unroll
        for (int t = 0; t < ITEMS; ++t) {
            const int x = v[t];
            v[t] = pre;
            pre += x;
        }
#pragma unroll
        for (int t = 0; t < ITEMS; t += 4) {
            if (e0 + t + 3 < n) *reinterpret_cast<int4*>(data + e0 + t) = make_int4(v[t], v[t + 1], v[t + 2], v[t + 3]);
            else
                for (int u = 0; u < 4; ++u)
                    if (e0 + t + u < n) data[e0 + t + u] = v[t + u];
        }
        carry += tot;
    }
    if (threadIdx.x == 0 && total) *total = carry;
}
}  // namespace

__global__ void __launch_bounds__(1024) k_scan_single_block(int* data, int n, int* total, unsigned long long* at) {
    note_clock(at);
    scan_block(data, n, total);
}
__global__ void __launch_bounds__(1024) k_scan_rows(int* data, int n, int stride, int* total0, int* total1) {
    scan_block(data + blockIdx.x * stride, n, blockIdx.x ? total1 : total0);
}

// The tile sums of data, and the scan of each tile from its offset.
__global__ void __launch_bounds__(SCAN_BLOCK) k_scan_tile_sums(const int* __restrict__ data, int n,
                                                               int* __restrict__ tile_sums, unsigned long long* at) {
    note_clock(at);
    const int e0 = (blockIdx.x * SCAN_BLOCK + threadIdx.x) * SCAN_ITEMS;
    int s = 0;
#pragma unroll
    for (int t = 0; t < SCAN_ITEMS; ++t) s += e0 + t < n ? data[e0 + t] : 0;
    int total;
    block_exclusive_scan<SCAN_BLOCK>(s, total);
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}
__global__ void __launch_bounds__(SCAN_BLOCK) k_scan_tiles(int* __restrict__ data, int n,
                                                           const int* __restrict__ tile_offsets) {
    const int e0 = (blockIdx.x * SCAN_BLOCK + threadIdx.x) * SCAN_ITEMS;
    int v[SCAN_ITEMS];
    int s = 0;
#pragma unroll
    for (int t = 0; t < SCAN_ITEMS; ++t) {
        v[t] = e0 + t < n ? data[e0 + t] : 0;
        s += v[t];
    }
    int total;
    int pre = block_exclusive_scan<SCAN_BLOCK>(s, total) + tile_offsets[blockIdx.x];
#pragma unroll
    for (int t = 0; t < SCAN_ITEMS; ++t) {
        if (e0 + t < n) data[e0 + t] = pre;
        pre += v[t];
    }
}

int scan_tiles(int64_t n) { return int((n + SCAN_TILE - 1) / SCAN_TILE); }

int launch_scan(int* data, int n, int* total, int* tile_sums, cudaStream_t st, unsigned long long* at) {
    // One pass of a single block, or the whole chip's three launches.
    if (n <= 1024 * 16) {
        k_scan_single_block<<<1, 1024, 0, st>>>(data, n, total, at);
        return 1;
    }
    const int tiles = scan_tiles(n);
    k_scan_tile_sums<<<tiles, SCAN_BLOCK, 0, st>>>(data, n, tile_sums, at);
    k_scan_single_block<<<1, 1024, 0, st>>>(tile_sums, tiles, total);
    k_scan_tiles<<<tiles, SCAN_BLOCK, 0, st>>>(data, n, tile_sums);
    return 3;
}

void launch_bin(const float4* pos, int64_t np, Dims g, int* counts, int* key, int* rank, cudaStream_t st) {
    if (np == 0) return;
    constexpr int per = BIN_THREADS * BIN_ITEMS;
    const unsigned nb = unsigned((np + per - 1) / per);
    if (g.idx != 0.0f) k_bin<true><<<nb, BIN_THREADS, 0, st>>>(pos, np, g, counts, key, rank);
    else k_bin<false><<<nb, BIN_THREADS, 0, st>>>(pos, np, g, counts, key, rank);
}

void launch_label_scan(const uint8_t* base, const uint8_t* body_mark, int* counts, uint8_t* labels, int* start,
                       int* tile_sums, Dims g, cudaStream_t st) {
    int64_t nc = g.nc();
    int ntiles = int((nc + SCAN_TILE - 1) / SCAN_TILE);
    k_label_tiles<<<ntiles, SCAN_BLOCK, 0, st>>>(base, body_mark, counts, labels, nc, tile_sums);
    k_scan_single_block<<<1, 1024, 0, st>>>(tile_sums, ntiles, start + nc);  // start[nc] = np
    k_start_tiles<<<ntiles, SCAN_BLOCK, 0, st>>>(counts, nc, tile_sums, start);
}

void launch_scatter(const float4* pos, const float4* vel, const int* key, const int* rank, const int* start, int64_t np,
                    float4* pos2, float4* vel2, cudaStream_t st) {
    if (np == 0) return;
    k_scatter<<<unsigned((np + 255) / 256), 256, 0, st>>>(pos, vel, key, rank, start, np, pos2, vel2);
}

}  // namespace fp
