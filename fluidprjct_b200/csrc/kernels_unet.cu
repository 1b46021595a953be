// kernels_unet.cu -- kernels of the learned pressure preconditioner (a 3D
// U-Net; the layer table is in unet.hpp).
//
// The convolutions run on tcgen05 (kernels_unet_tma.cu).  This file holds the
// rest: the weight gradients, input and output, pooling, the element-wise parts
// of the backward pass, the loss and Adam.
#include <algorithm>
#include <cstdio>

#include "device_memo.hpp"
#include "unet.hpp"

namespace fp {
namespace unet {
namespace {

constexpr int THREADS = 256;

// ---------------------------------------------------------------- weight gradients
// k_corr3: dw[t][co][ci] = sum_v g[v][co] x[v + off(t)][ci] on the BF16 mma.sync
// path (m16n8k16, FP32 accumulation; M = COUT, N = CIN, K = voxels), over bricks
// of 8 x 8 x 4 voxels whose operands, x's with a zero-padded halo, are staged
// with cp.async.  A CTA keeps the sums of its TPC taps over its bricks in
// registers and writes one partial; the partials are added in a fixed order.
//
// Bound by latency: the 18 warps of an SM wait for ldmatrix (its shared-memory
// pipe is 56 to 60 % busy), for the MMA before on the same sums and for the
// block; the tensor pipe is 40 to 43 % busy.  A warp's unit is a tap, 16 input
// and 16 COG output channels: one x4 load of x serves 2 COG MMAs, and g's are
// loaded once per 16 voxels for all the warp's units, where a warp that took
// 16 x 8 tiles one by one loaded both for each (x4 and x2 per MMA).  Two buffers,
// where two CTAs of them fit an SM, let a brick's loads run during the one
// before.  1.31 ms per 128^3 training step, against 3.07.
//
// Each sum keeps its order, brick by brick and 16 voxels at a time, one MMA after
// the other: FP32 accumulation of the tensor cores is not exact, and a training
// step's weights (Adam divides by the gradient's size) show another order's
// rounding where a gradient nearly cancels.  tcgen05 sums over stacked planes took
// 0.76 ms for the same layers, but moved single weights by 1e-3 of the weights'
// size after one step.
constexpr int BX = 8, BY = 8, BZ = 4, BRICK = BX * BY * BZ;
constexpr int HX = BX + 2, HY = BY + 2, HZ = BZ + 2, HALO = HX * HY * HZ;  // 600

__device__ __forceinline__ unsigned smem_addr(const void* p) {
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void cp_async16(unsigned dst, const void* src, bool pred) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(pred ? 16 : 0));
}
__device__ __forceinline__ void ldsm_x4_t(unsigned (&r)[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
__device__ __forceinline__ void mma16816(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

struct CorrArgs {
    const bf16 *x, *g;
    float* part;  // [gridDim.x][27][COUT][CIN] partial sums
    Lvl lv;
};

// A CTA's TPC taps and 16 NCI input channels go to NW warps of U units each, unit
// u = warp + NW i: output channels group u % NCG, then input channels, then taps
// (NW is a multiple of NCG: a warp has one group).
template <int CIN, int COUT, int TPC, int NCI, int NW, int COG, int NBUF>
__global__ void __launch_bounds__(32 * NW) k_corr3(CorrArgs a) {
    constexpr int NT = 32 * NW, RS = 16 * NCI + 8, GS = COUT + 8;  // (rows padded by 16 bytes: ldmatrix without conflicts)
    constexpr int NCG = COUT / 16 / COG, UNITS = TPC * NCI * NCG, U = UNITS / NW, CIGS = CIN / 16 / NCI;
    static_assert(27 % TPC == 0 && COUT % (16 * COG) == 0 && CIN % (16 * NCI) == 0, "tiling");
    static_assert(UNITS % NW == 0 && NW % NCG == 0, "units");
    constexpr int XB = HALO * RS * 2, BUF = XB + BRICK * GS * 2;  // bytes
    extern __shared__ __align__(16) unsigned char smem[];
    const unsigned base = smem_addr(smem);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tap0 = int(blockIdx.y) / CIGS * TPC, ci0 = int(blockIdx.y) % CIGS * (16 * NCI), cg = warp % NCG;
    const Lvl lv = a.lv;
    const int nbx = (lv.W + BX - 1) / BX, nby = (lv.H + BY - 1) / BY, nbz = (lv.D + BZ - 1) / BZ;
    const int nbricks = nbx * nby * nbz;

    auto load = [&](int brick, unsigned buf) {
        const int x0 = brick % nbx * BX, y0 = brick / nbx % nby * BY, z0 = brick / (nbx * nby) * BZ;
        const int64_t n = lv.n();
        for (int hv = tid; hv < HALO; hv += NT) {
            const int gx = x0 - 1 + hv % HX, gy = y0 - 1 + hv / HX % HY, gz = z0 - 1 + hv / (HX * HY);
            const bool in = gx >= 0 && gx < lv.W && gy >= 0 && gy < lv.H && gz >= 0 && gz < lv.D;
            const bf16* src = in ? a.x + blk8(n, (int64_t(gz) * lv.H + gy) * lv.W + gx, ci0 / 8) : a.x;
            const int64_t step = in ? 8 * n : 0;
#pragma unroll
            for (int ch = 0; ch < 2 * NCI; ++ch) cp_async16(buf + unsigned((hv * RS + ch * 8) * 2), src + ch * step, in);
        }
        for (int v = tid; v < BRICK; v += NT) {
            const int gx = x0 + (v & 7), gy = y0 + ((v >> 3) & 7), gz = z0 + (v >> 6);
            const bool in = gx < lv.W && gy < lv.H && gz < lv.D;
            const bf16* src = in ? a.g + blk8(n, (int64_t(gz) * lv.H + gy) * lv.W + gx, 0) : a.g;
            const int64_t step = in ? 8 * n : 0;
#pragma unroll
            for (int ch = 0; ch < COUT / 8; ++ch)
                cp_async16(buf + unsigned(XB + (v * GS + ch * 8) * 2), src + ch * step, in);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    // g^T (16 channels x 16 voxels): voxel row, channel offset; x (16 voxels x 16 channels): the same the other way
    const int akr = (lane & 7) + 8 * (lane >> 4), amoff = 8 * ((lane >> 3) & 1);
    const int bkr = (lane & 7) + 8 * ((lane >> 3) & 1), bmoff = 8 * (lane >> 4);
    int boff[U];
#pragma unroll
    for (int i = 0; i < U; ++i) {
        const int u = (warp + NW * i) / NCG, cip = u % NCI, tap = tap0 + u / NCI;
        const int toff = ((tap / 9 - 1) * HY + ((tap / 3) % 3 - 1)) * HX + (tap % 3 - 1);
        boff[i] = (toff * RS + cip * 16) * 2;
    }
    float acc[U][COG][2][4];
#pragma unroll
    for (int i = 0; i < U * COG * 8; ++i) (&acc[0][0][0][0])[i] = 0.0f;

    int it = 0;
    if (int(blockIdx.x) < nbricks) load(blockIdx.x, base);
    for (int brick = blockIdx.x; brick < nbricks; brick += gridDim.x, ++it) {
        const unsigned buf = base + unsigned(NBUF == 2 ? (it & 1) * BUF : 0);
        if (NBUF == 2 && brick + int(gridDim.x) < nbricks) {
            load(brick + gridDim.x, base + unsigned(((it + 1) & 1) * BUF));
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        }
        __syncthreads();
#pragma unroll 1
        for (int ks = 0; ks < 16; ++ks) {
            const int z = ks >> 2, yy = (ks & 3) * 2;
            const int av = (z * BY + yy + (akr >> 3)) * BX + (akr & 7);
            const int bh = ((z + 1) * HY + (yy + (bkr >> 3) + 1)) * HX + ((bkr & 7) + 1);
            unsigned ar[COG][4];
#pragma unroll
            for (int c = 0; c < COG; ++c)
                ldsm_x4_t(ar[c], buf + unsigned(XB + (av * GS + (cg * COG + c) * 16 + amoff) * 2));
            const unsigned bx = buf + unsigned((bh * RS + bmoff) * 2);
#pragma unroll
            for (int i = 0; i < U; ++i) {
                unsigned br[4];
                ldsm_x4_t(br, bx + unsigned(boff[i]));
#pragma unroll
                for (int c = 0; c < COG; ++c) {
                    mma16816(acc[i][c][0], ar[c], br[0], br[1]);
                    mma16816(acc[i][c][1], ar[c], br[2], br[3]);
                }
            }
        }
        __syncthreads();
        if (NBUF == 1 && brick + int(gridDim.x) < nbricks) load(brick + gridDim.x, base);
    }
    const int gr = lane >> 2, tq = lane & 3;
    float* part = a.part + int64_t(blockIdx.x) * 27 * COUT * CIN;
#pragma unroll
    for (int i = 0; i < U; ++i) {
        const int u = (warp + NW * i) / NCG, cip = u % NCI, tap = tap0 + u / NCI;
#pragma unroll
        for (int c = 0; c < COG; ++c)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int co = (cg * COG + c) * 16 + gr, ci = ci0 + cip * 16 + h * 8 + 2 * tq;
                float* p0 = part + (int64_t(tap) * COUT + co) * CIN + ci;
                p0[0] = acc[i][c][h][0];
                p0[1] = acc[i][c][h][1];
                p0[8 * CIN] = acc[i][c][h][2];
                p0[8 * CIN + 1] = acc[i][c][h][3];
            }
    }
}

__global__ void k_reduce_partials(const float* __restrict__ part, int nblk, int64_t n, float* __restrict__ out) {
    for (int64_t j = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; j < n; j += int64_t(gridDim.x) * blockDim.x) {
        float s = 0.0f;
        for (int b = 0; b < nblk; ++b) s += part[int64_t(b) * n + j];
        out[j] = s;
    }
}

// ---------------------------------------------------------------- small kernels
constexpr int RED_BLOCKS = 256;

template <int N>
__device__ __forceinline__ void block_sum_d(double (&v)[N], double* sh) {
    // fixed-order tree over a 256-thread block; result in thread 0's v
#pragma unroll
    for (int k = 0; k < N; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < N; ++k) sh[warp * N + k] = v[k];
    __syncthreads();
    if (threadIdx.x == 0)
#pragma unroll
        for (int k = 0; k < N; ++k) {
            double s = 0.0;
            for (int w = 0; w < THREADS / 32; ++w) s += sh[w * N + k];
            v[k] = s;
        }
    __syncthreads();
}

// Coordinates of voxel t of a level.  A level has fewer than 2^32 voxels (its
// activations take over 100 bytes each), and 64-bit divisions would take most of
// the time of these kernels.
__device__ __forceinline__ void voxel(int64_t t, const Lvl& l, int& i, int& j, int& k) {
    const unsigned u = unsigned(t), r = u / unsigned(l.W);
    i = int(u - r * unsigned(l.W));
    k = int(r / unsigned(l.H));
    j = int(r - unsigned(k) * unsigned(l.H));
}
// The same of item t of C / 8 channel blocks, voxels fastest.
__device__ __forceinline__ void block_voxel(int64_t t, const Lvl& l, int64_t& v, int& ch) {
    ch = 0;
    const int64_t n = l.n();
    while (t >= n) { t -= n; ++ch; }  // at most 12 blocks
    v = t;
}
// Sum of n <= THREADS values in their order, by a block of THREADS threads; in
// thread 0.  Loaded together: one thread that loaded as it added took 12 us for
// two sums of 256, this 4.5.
__device__ __forceinline__ double ordered_sum(const double* __restrict__ a, int n) {
    __shared__ double sh[THREADS];
    __syncthreads();
    if (int(threadIdx.x) < n) sh[threadIdx.x] = a[threadIdx.x];
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int b = 0; b < n; ++b) s += sh[b];
    return s;
}

__device__ __forceinline__ uint8_t label_net(const uint8_t* __restrict__ lab, const Lvl& real, int i, int j, int k) {
    if (i >= real.W || j >= real.H || k >= real.D) return 0;  // padding counts as SOLID
    return lab[(int64_t(k) * real.H + j) * real.W + i];
}

// A thread's terms are added in their order, but loaded in batches: one after the
// other, each waited for a memory round trip (10 us at 128^3, k_loss_part 36;
// in batches 6 and 25).
constexpr int RED_BATCH = 8;
__global__ void __launch_bounds__(THREADS) k_rhs_scale_part(const uint8_t* __restrict__ lab,
                                                             const float* __restrict__ rhs, Lvl real,
                                                             double* __restrict__ red) {
    __shared__ double sh[2 * THREADS / 32];
    double v[2] = {0.0, 0.0};
    const int64_t n = real.n(), st = int64_t(gridDim.x) * blockDim.x;
    for (int64_t t0 = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; t0 < n; t0 += RED_BATCH * st) {
        uint8_t l[RED_BATCH];
        float r[RED_BATCH];
#pragma unroll
        for (int m = 0; m < RED_BATCH; ++m) {
            const int64_t t = t0 + m * st;
            l[m] = t < n ? lab[t] : 0;
            r[m] = t < n ? rhs[t] : 0.0f;
        }
#pragma unroll
        for (int m = 0; m < RED_BATCH; ++m)
            if (l[m] == 1) {
                v[0] += double(r[m]) * double(r[m]);
                v[1] += 1.0;
            }
    }
    block_sum_d<2>(v, sh);
    if (threadIdx.x == 0) {
        red[blockIdx.x] = v[0];
        red[RED_BLOCKS + blockIdx.x] = v[1];
    }
}
__global__ void __launch_bounds__(THREADS) k_rhs_scale_final(const double* __restrict__ red, float* __restrict__ scal) {
    const double ss = ordered_sum(red, RED_BLOCKS), n = ordered_sum(red + RED_BLOCKS, RED_BLOCKS);
    if (threadIdx.x != 0) return;
    const double s = (n > 0.0 && ss > 0.0) ? sqrt(ss / n) : 1.0;
    scal[0] = float(s);
    scal[1] = float(1.0 / s);
}

__global__ void k_input(const uint8_t* __restrict__ lab, const float* __restrict__ rhs, Lvl real, Lvl net,
                        const float* __restrict__ scal, bf16* __restrict__ x0) {
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= net.n()) return;
    int i, j, k;
    voxel(t, net, i, j, k);
    const uint8_t l = label_net(lab, real, i, j, k);
    const float c0 = l == 1 ? __fmul_rn(rhs[(int64_t(k) * real.H + j) * real.W + i], scal[1]) : 0.0f;
    __align__(16) bf16 v[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) v[c] = __float2bfloat16_rn(0.0f);
    v[0] = __float2bfloat16_rn(c0);
    v[1] = __float2bfloat16_rn(l == 1 ? 1.0f : 0.0f);
    v[2] = __float2bfloat16_rn(l == 2 ? 1.0f : 0.0f);
    v[3] = __float2bfloat16_rn((l == 0 || l == 3) ? 1.0f : 0.0f);
    *reinterpret_cast<uint4*>(x0 + blk8(net.n(), t, 0)) = reinterpret_cast<const uint4*>(v)[0];
    *reinterpret_cast<uint4*>(x0 + blk8(net.n(), t, 1)) = reinterpret_cast<const uint4*>(v)[1];
}

__device__ __forceinline__ void load8(const bf16* p, float* f) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float2 x = __bfloat1622float2(h[q]);
        f[2 * q] = x.x;
        f[2 * q + 1] = x.y;
    }
}
__device__ __forceinline__ void store8(bf16* p, const float* f) {
    uint4 u;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
    for (int q = 0; q < 4; ++q) h[q] = __floats2bfloat162_rn(f[2 * q], f[2 * q + 1]);
    *reinterpret_cast<uint4*>(p) = u;
}

// One thread per (coarse voxel, 8 channels), voxels fastest.  Fine dims are even.
__global__ void k_pool(const bf16* __restrict__ e, Lvl fine, int C, bf16* __restrict__ q) {
    const int CH = C / 8;
    const Lvl cl{fine.W / 2, fine.H / 2, fine.D / 2};
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= cl.n() * CH) return;
    int64_t V;
    int ch, I, J, K;
    block_voxel(t, cl, V, ch);
    voxel(V, cl, I, J, K);
    float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int dz = 0; dz < 2; ++dz)
        for (int dy = 0; dy < 2; ++dy)
            for (int dx = 0; dx < 2; ++dx) {
                float f[8];
                load8(e + blk8(fine.n(), (int64_t(2 * K + dz) * fine.H + 2 * J + dy) * fine.W + 2 * I + dx, ch), f);
#pragma unroll
                for (int c = 0; c < 8; ++c) s[c] += f[c];
            }
#pragma unroll
    for (int c = 0; c < 8; ++c) s[c] *= 0.125f;
    store8(q + blk8(cl.n(), V, ch), s);
}

// g[V][c] = (sum over the 8 children of raw[child][c]) * (act[V][c] > 0), c < C.
__global__ void k_sum_children_mask(const bf16* __restrict__ raw, Lvl fine, int ctot, int C,
                                    const bf16* __restrict__ act, bf16* __restrict__ gout) {
    const int CH = C / 8;
    const Lvl cl{fine.W / 2, fine.H / 2, fine.D / 2};
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= cl.n() * CH) return;
    int64_t V;
    int ch, I, J, K;
    block_voxel(t, cl, V, ch);
    voxel(V, cl, I, J, K);
    float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int dz = 0; dz < 2; ++dz)
        for (int dy = 0; dy < 2; ++dy)
            for (int dx = 0; dx < 2; ++dx) {
                float f[8];
                load8(raw + blk8(fine.n(), (int64_t(2 * K + dz) * fine.H + 2 * J + dy) * fine.W + 2 * I + dx, ch), f);
#pragma unroll
                for (int c = 0; c < 8; ++c) s[c] += f[c];
            }
    float m[8];
    load8(act + blk8(cl.n(), V, ch), m);
#pragma unroll
    for (int c = 0; c < 8; ++c) s[c] = m[c] > 0.0f ? s[c] : 0.0f;
    store8(gout + blk8(cl.n(), V, ch), s);
}

// g[v][c] = (raw[v][ca + c] + gq[v>>1][c] / 8) * (act[v][c] > 0), c < C.
__global__ void k_skip_combine(const bf16* __restrict__ raw, Lvl fine, int ctot, int ca, int C,
                               const bf16* __restrict__ gq, const bf16* __restrict__ act, bf16* __restrict__ gout) {
    const int CH = C / 8;
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= fine.n() * CH) return;
    int64_t v;
    int ch, i, j, k;
    block_voxel(t, fine, v, ch);
    voxel(v, fine, i, j, k);
    const Lvl cl{fine.W / 2, fine.H / 2, fine.D / 2};
    float r[8], q[8], m[8];
    load8(raw + blk8(fine.n(), v, ca / 8 + ch), r);
    load8(gq + blk8(cl.n(), (int64_t(k >> 1) * cl.H + (j >> 1)) * cl.W + (i >> 1), ch), q);
    load8(act + blk8(fine.n(), v, ch), m);
#pragma unroll
    for (int c = 0; c < 8; ++c) r[c] = m[c] > 0.0f ? r[c] + 0.125f * q[c] : 0.0f;
    store8(gout + blk8(fine.n(), v, ch), r);
}

__global__ void __launch_bounds__(THREADS) k_loss_part(const uint8_t* __restrict__ lab, const float* __restrict__ p,
                                                        Lvl real, Lvl net, const float* __restrict__ out,
                                                        const float* __restrict__ scal, double* __restrict__ red) {
    __shared__ double sh[2 * THREADS / 32];
    double v[2] = {0.0, 0.0};
    const float inv_s = scal[1];
    const int64_t n = real.n(), st = int64_t(gridDim.x) * blockDim.x;
    for (int64_t t0 = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; t0 < n; t0 += RED_BATCH * st) {
        uint8_t l[RED_BATCH];
        float pv[RED_BATCH], ov[RED_BATCH];
#pragma unroll
        for (int m = 0; m < RED_BATCH; ++m) {
            const int64_t t = t0 + m * st;
            l[m] = 0;
            if (t >= n) continue;
            int i, j, k;
            voxel(t, real, i, j, k);
            l[m] = lab[t];
            pv[m] = p[t];
            ov[m] = out[(int64_t(k) * net.H + j) * net.W + i];
        }
#pragma unroll
        for (int m = 0; m < RED_BATCH; ++m) {
            if (l[m] != 1) continue;
            const float tv = __fmul_rn(pv[m], inv_s);
            const double e = double(ov[m]) - double(tv);
            v[0] += e * e;
            v[1] += double(tv) * double(tv);
        }
    }
    block_sum_d<2>(v, sh);
    if (threadIdx.x == 0) {
        red[blockIdx.x] = v[0];
        red[RED_BLOCKS + blockIdx.x] = v[1];
    }
}
__global__ void __launch_bounds__(THREADS) k_loss_final(double* __restrict__ red, float* __restrict__ scal) {
    const double ee = ordered_sum(red, RED_BLOCKS);
    double tt = ordered_sum(red + RED_BLOCKS, RED_BLOCKS);
    if (threadIdx.x != 0) return;
    if (!(tt > 0.0)) tt = 1.0;
    red[2 * RED_BLOCKS] = ee / tt;  // loss
    scal[2] = float(2.0 / tt);
}

// As in k_rhs_scale_part, HEAD_BATCH voxels' loads together (70 us at 128^3 one
// by one, 49 by two; 22 at memory speed, the rest is the FP64 sums).
constexpr int HEAD_BATCH = 2;
__global__ void __launch_bounds__(THREADS) k_head_bwd(const uint8_t* __restrict__ lab, const float* __restrict__ p,
                                                       Lvl real, Lvl net, const float* __restrict__ out,
                                                       const bf16* __restrict__ d0, const float* __restrict__ hw,
                                                       const float* __restrict__ scal, bf16* __restrict__ g9,
                                                       float* __restrict__ hpart) {
    __shared__ double sh[16 * THREADS / 32];
    double hp[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) hp[c] = 0.0;
    const float inv_s = scal[1], k2 = scal[2];
    const int64_t n = net.n(), st = int64_t(gridDim.x) * blockDim.x;
    for (int64_t t0 = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; t0 < n; t0 += HEAD_BATCH * st) {
        uint4 lo[HEAD_BATCH], hi[HEAD_BATCH];
        float go[HEAD_BATCH];
#pragma unroll
        for (int m = 0; m < HEAD_BATCH; ++m) {
            const int64_t t = t0 + m * st;
            go[m] = 0.0f;
            if (t >= n) continue;
            int i, j, k;
            voxel(t, net, i, j, k);
            lo[m] = *reinterpret_cast<const uint4*>(d0 + blk8(n, t, 0));
            hi[m] = *reinterpret_cast<const uint4*>(d0 + blk8(n, t, 1));
            if (i >= real.W || j >= real.H || k >= real.D) continue;
            const int64_t r = (int64_t(k) * real.H + j) * real.W + i;
            const float pv = p[r], ov = out[t];
            if (lab[r] == 1) go[m] = (ov - __fmul_rn(pv, inv_s)) * k2;
        }
#pragma unroll
        for (int m = 0; m < HEAD_BATCH; ++m) {
            const int64_t t = t0 + m * st;
            if (t >= n) break;
            float f[16], o[16];
            load8(reinterpret_cast<const bf16*>(&lo[m]), f);
            load8(reinterpret_cast<const bf16*>(&hi[m]), f + 8);
#pragma unroll
            for (int c = 0; c < 16; ++c) {
                o[c] = f[c] > 0.0f ? go[m] * hw[c] : 0.0f;
                hp[c] += double(go[m]) * double(f[c]);
            }
            store8(g9 + blk8(n, t, 0), o);
            store8(g9 + blk8(n, t, 1), o + 8);
        }
    }
    block_sum_d<16>(hp, sh);
    if (threadIdx.x == 0)
#pragma unroll
        for (int c = 0; c < 16; ++c) hpart[blockIdx.x * 16 + c] = float(hp[c]);
}

__global__ void k_output_dense(const uint8_t* __restrict__ lab, Lvl real, Lvl net, const float* __restrict__ out,
                               const float* __restrict__ scal, float* __restrict__ x) {
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= real.n()) return;
    int i, j, k;
    voxel(t, real, i, j, k);
    x[t] = lab[t] == 1 ? out[(int64_t(k) * net.H + j) * net.W + i] * scal[0] : 0.0f;
}

__global__ void k_output_compact(const int* __restrict__ nf_p, const int* __restrict__ fidx, Lvl real, Lvl net,
                                 const float* __restrict__ out, const float* __restrict__ scal,
                                 float* __restrict__ x0) {
    const int nf = *nf_p;
    const float s = scal[0];
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < nf; n += gridDim.x * blockDim.x) {
        const int c = fidx[n];
        const int i = c % (real.W + 2) - 1, j = (c / (real.W + 2)) % (real.H + 2) - 1,
                  k = c / ((real.W + 2) * (real.H + 2)) - 1;
        x0[n] = out[(int64_t(k) * net.H + j) * net.W + i] * s;
    }
}

__global__ void k_rhs_dense(const int* __restrict__ nf_p, const int* __restrict__ fidx, Lvl real,
                            const float* __restrict__ b, float* __restrict__ dense) {
    const int nf = *nf_p;
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < nf; n += gridDim.x * blockDim.x) {
        const int c = fidx[n];
        const int i = c % (real.W + 2) - 1, j = (c / (real.W + 2)) % (real.H + 2) - 1,
                  k = c / ((real.W + 2) * (real.H + 2)) - 1;
        dense[(int64_t(k) * real.H + j) * real.W + i] = b[n];
    }
}

// Global gradient norm (fixed-order, FP64) and the clipping factor
// min(1, clip / norm) in scal[3]; the norm itself goes to red[2 * RED_BLOCKS + 1].
__global__ void __launch_bounds__(THREADS) k_gnorm_part(const float* __restrict__ g, int64_t n,
                                                         double* __restrict__ red) {
    __shared__ double sh[THREADS / 32];
    double v[1] = {0.0};
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
        v[0] += double(g[i]) * double(g[i]);
    block_sum_d<1>(v, sh);
    if (threadIdx.x == 0) red[blockIdx.x] = v[0];
}
__global__ void __launch_bounds__(THREADS) k_gnorm_final(double* __restrict__ red, float clip,
                                                         float* __restrict__ scal) {
    const double ss = ordered_sum(red, RED_BLOCKS);
    if (threadIdx.x != 0) return;
    const double nrm = sqrt(ss);
    red[2 * RED_BLOCKS + 1] = nrm;
    scal[3] = (nrm > double(clip) && isfinite(nrm)) ? float(double(clip) / nrm) : (isfinite(nrm) ? 1.0f : 0.0f);
}

__global__ void k_adam(float* __restrict__ w, float* __restrict__ m, float* __restrict__ v,
                       const float* __restrict__ g, const float* __restrict__ scal, int64_t n, float lr, float b1,
                       float b2, float eps, float bc1, float bc2) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i] * scal[3];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    w[i] -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
}

// BF16 copies of the 3x3x3 weights: wf in the forward layout [t][co][ci] and
// wt, the backward-data layout [26 - t][ci][co].
struct LayerTable {
    int64_t off[kLayers + 1];
    int cin[kLayers], cout[kLayers];
};
__global__ void k_weights_bf16(const float* __restrict__ w, bf16* __restrict__ wf, bf16* __restrict__ wt,
                               LayerTable lt) {
    const int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (idx >= lt.off[kLayers]) return;
    int l = 0;
    while (l + 1 < kLayers && idx >= lt.off[l + 1]) ++l;
    const int64_t r = idx - lt.off[l];
    const int cin = lt.cin[l], cout = lt.cout[l];
    const int ci = int(r % cin), co = int((r / cin) % cout), t = int(r / (int64_t(cin) * cout));
    const bf16 b = __float2bfloat16_rn(w[idx]);
    wf[idx] = b;
    wt[lt.off[l] + (int64_t(26 - t) * cin + ci) * cout + co] = b;
}

// ---------------------------------------------------------------- dispatch
int sm_count() {
    static DeviceMemo memo;
    const int n = memo.get([](int dev) {
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        return std::max(sms, 0);
    });
    return n > 0 ? n : 148;
}

int nbricks_of(const Lvl& lv) {
    return ((lv.W + BX - 1) / BX) * ((lv.H + BY - 1) / BY) * ((lv.D + BZ - 1) / BZ);
}

template <int CIN, int COUT, int TPC, int NCI, int NW, int COG>
int run_corr(const CorrArgs& a, int nblk, cudaStream_t st) {
    constexpr size_t one = size_t(HALO * (16 * NCI + 8) + BRICK * (COUT + 8)) * sizeof(bf16);
    constexpr int NBUF = 4 * (one + 1024) <= 228 * 1024 ? 2 : 1;  // two CTAs per SM of two buffers
    constexpr size_t smem = NBUF * one;
    static DeviceMemo memo;
    auto kern = k_corr3<CIN, COUT, TPC, NCI, NW, COG, NBUF>;
    memo.get([&](int) {
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        return 1;
    });
    kern<<<dim3(nblk, 27 / TPC * (CIN / 16 / NCI)), 32 * NW, smem, st>>>(a);
    return int(cudaPeekAtLastError());
}

// The number of brick shares of a layer, and so the order of its sums, goes by
// these; how a share's taps and channels are spread over CTAs (corr_layer) does
// not change a sum.
constexpr int kTpc[kLayers] = {27, 27, 9, 9, 3, 3, 3, 9, 9, 27};

}  // namespace

int corr_blocks(int layer, const Lvl& lv) {
    const int groups = 27 / kTpc[layer];
    return std::max(1, std::min(nbricks_of(lv), 2 * sm_count() / groups));
}

int corr_layer(int layer, const bf16* x, const bf16* g, const Lvl& lv, float* part, int nblk, cudaStream_t st) {
    const CorrArgs a{x, g, part, lv};
    // A CTA of few input channels and all taps stages little for much work and has
    // room for two buffers, but there are fewer of them.  us at 128^3 (64^3 for
    // layers 2, 3, 6 and 7, 32^3 for 4 and 5), all channels and few taps against
    // this: 48 -> 16 622 and 401, 96 -> 32 466 and 245 (255 with 27 taps of 16
    // channels), 64 -> 64 55 and 38; for 32 -> 32 83 and 87, so not there.
    switch (layer) {
        case 0: case 1: case 9: return run_corr<16, 16, 27, 1, 9, 1>(a, nblk, st);
        case 2: return run_corr<16, 32, 9, 1, 9, 2>(a, nblk, st);
        case 3: case 7: return run_corr<32, 32, 9, 2, 9, 2>(a, nblk, st);
        case 4: return run_corr<32, 64, 3, 2, 12, 2>(a, nblk, st);
        case 5: return run_corr<64, 64, 27, 1, 18, 2>(a, nblk, st);
        case 6: return run_corr<96, 32, 9, 2, 9, 2>(a, nblk, st);
        case 8: return run_corr<48, 16, 27, 1, 9, 1>(a, nblk, st);
    }
    return int(cudaErrorInvalidValue);
}

void reduce_partials(const float* part, int nblk, int64_t n, float* out, cudaStream_t st) {
    const int blocks = int(std::min<int64_t>((n + 255) / 256, 4 * sm_count()));
    k_reduce_partials<<<blocks, 256, 0, st>>>(part, nblk, n, out);
}

void launch_rhs_scale(const uint8_t* labels, const float* rhs, Lvl real, double* red, float* scal, cudaStream_t st) {
    k_rhs_scale_part<<<RED_BLOCKS, THREADS, 0, st>>>(labels, rhs, real, red);
    k_rhs_scale_final<<<1, THREADS, 0, st>>>(red, scal);
}

void launch_input(const uint8_t* labels, const float* rhs, Lvl real, Lvl net, const float* scal, bf16* x0,
                  cudaStream_t st) {
    k_input<<<unsigned((net.n() + 255) / 256), 256, 0, st>>>(labels, rhs, real, net, scal, x0);
}

void launch_pool(const bf16* e, Lvl fine, int C, bf16* q, cudaStream_t st) {
    const int64_t n = fine.n() / 8 * (C / 8);
    k_pool<<<unsigned((n + 255) / 256), 256, 0, st>>>(e, fine, C, q);
}

void launch_sum_children_mask(const bf16* raw, Lvl fine, int ctot, int C, const bf16* act, bf16* g, cudaStream_t st) {
    const int64_t n = fine.n() / 8 * (C / 8);
    k_sum_children_mask<<<unsigned((n + 255) / 256), 256, 0, st>>>(raw, fine, ctot, C, act, g);
}

void launch_skip_combine(const bf16* raw, Lvl fine, int ctot, int ca, int C, const bf16* gq, const bf16* act,
                         bf16* g, cudaStream_t st) {
    const int64_t n = fine.n() * (C / 8);
    k_skip_combine<<<unsigned((n + 255) / 256), 256, 0, st>>>(raw, fine, ctot, ca, C, gq, act, g);
}

void launch_loss(const uint8_t* labels, const float* p, Lvl real, Lvl net, const float* out, double* red, float* scal,
                 cudaStream_t st) {
    k_loss_part<<<RED_BLOCKS, THREADS, 0, st>>>(labels, p, real, net, out, scal, red);
    k_loss_final<<<1, THREADS, 0, st>>>(red, scal);
}

int head_blocks(Lvl net) { return int(std::min<int64_t>((net.n() + THREADS - 1) / THREADS, 2 * sm_count())); }

void launch_head_backward(const uint8_t* labels, const float* p, Lvl real, Lvl net, const float* out, const bf16* d0,
                          const float* head_w, const float* scal, bf16* g9, float* head_part, int nblk,
                          cudaStream_t st) {
    k_head_bwd<<<nblk, THREADS, 0, st>>>(labels, p, real, net, out, d0, head_w, scal, g9, head_part);
}

void launch_output_dense(const uint8_t* labels, Lvl real, Lvl net, const float* out, const float* scal, float* x,
                         cudaStream_t st) {
    k_output_dense<<<unsigned((real.n() + 255) / 256), 256, 0, st>>>(labels, real, net, out, scal, x);
}

void launch_output_compact(const int* nf, const int* fidx, Lvl real, Lvl net, const float* out, const float* scal,
                           float* x0, cudaStream_t st) {
    k_output_compact<<<4 * sm_count(), 256, 0, st>>>(nf, fidx, real, net, out, scal, x0);
}

void launch_rhs_dense(const int* nf, const int* fidx, Lvl real, const float* b, float* dense, cudaStream_t st) {
    cudaMemsetAsync(dense, 0, sizeof(float) * size_t(real.n()), st);
    k_rhs_dense<<<4 * sm_count(), 256, 0, st>>>(nf, fidx, real, b, dense);
}

void launch_adam(float* w, float* m, float* v, const float* g, int64_t n, float lr, float b1, float b2, float eps,
                 float bc1, float bc2, float clip, double* red, float* scal, cudaStream_t st) {
    k_gnorm_part<<<RED_BLOCKS, THREADS, 0, st>>>(g, n, red);
    k_gnorm_final<<<1, THREADS, 0, st>>>(red, clip, scal);
    k_adam<<<unsigned((n + 255) / 256), 256, 0, st>>>(w, m, v, g, scal, n, lr, b1, b2, eps, bc1, bc2);
}

void launch_weights_bf16(const float* w32, bf16* wf, bf16* wt, cudaStream_t st) {
    LayerTable lt;
    for (int l = 0; l <= kLayers; ++l) lt.off[l] = layer_offset(l);
    for (int l = 0; l < kLayers; ++l) {
        lt.cin[l] = kSpec[l].ca + kSpec[l].cb;
        lt.cout[l] = kSpec[l].cout;
    }
    const int64_t n = lt.off[kLayers];
    k_weights_bf16<<<unsigned((n + 255) / 256), 256, 0, st>>>(w32, wf, wt, lt);
}

}  // namespace unet
}  // namespace fp
