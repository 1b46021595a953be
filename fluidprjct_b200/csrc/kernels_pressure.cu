// kernels_pressure.cu -- pressure set-up (compaction, RHS), projection, and the
// stand-alone CSR solve.
//
// Replaces pressureSolve (FluidSolver3D.cu:1815-2062) and applyPressure
// (:2072-2464).  The reference assembles an upper-triangle CSR of the unit
// 7-point Laplacian over FLUID cells (MatrixBuilder3D/MatrixFiller3D,
// :1598-1777) and hands it to cuDSS every step.  Here the operator is never
// stored: A*d at a FLUID cell is diag*d - sum of d over FLUID neighbours, with
// diag = number of in-domain FLUID or AIR neighbours (SOLID, BODY and
// out-of-domain neighbours are Neumann walls; AIR is Dirichlet p = 0).
//
// Layout: FLUID cells are compacted once per solve (fidx: padded dense index of
// the n-th FLUID cell, in i-fastest order, the reference's fluidNumbers order)
// with their diagonal and right-hand side; the solvers (kernels_pcg.cu,
// kernels_mg.cu) keep the vectors that a stencil reads on padded grids with a
// one-cell zero halo, so that it needs no bounds tests.
#include <algorithm>
#include <cmath>
#include <cstdio>

#include "../../include/fluidprjct.h"
#include "device_memo.hpp"
#include "kernels.hpp"
#include "pcg_common.cuh"
#include "scan.cuh"

namespace fp {

namespace {

constexpr int SCAN_BLOCK = 1024;

__device__ __forceinline__ bool solidish(uint8_t l) { return l == SOLID || l == BODY; }

// The compaction works on quads, four aligned cells of a row (fewer at the end
// of a row whose width is no multiple of four), one per thread, in row order:
// the FLUID cells come out in i-fastest order, and so do the quads that hold
// any.  A tile is one block's quads; its counts of both are packed in one int.
__device__ __forceinline__ int quads_of_row(const Dims& g) { return (g.W + 3) >> 2; }

// The labels of a quad's m cells (SOLID beyond them), at a row's address that is
// a multiple of four if the width W is one.
__device__ __forceinline__ uchar4 quad_labels(const uint8_t* __restrict__ l, int m, int W) {
    if ((W & 3) == 0) return *reinterpret_cast<const uchar4*>(l);
    return make_uchar4(l[0], m > 1 ? l[1] : SOLID, m > 2 ? l[2] : SOLID, m > 3 ? l[3] : SOLID);
}
__device__ __forceinline__ void quad_floats(const float* __restrict__ a, int m, int W, float (&v)[4]) {
    if ((W & 3) == 0) {
        const float4 q = *reinterpret_cast<const float4*>(a);
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else {
#pragma unroll
        for (int t = 0; t < 4; ++t) v[t] = t < m ? a[t] : 0.0f;
    }
}

// Pass 1: the tiles' counts; zero p off the fluid (the solve writes every FLUID
// cell; until then they keep the previous pressure, which a warm-started MG
// solve reads as its guess); ready the solvers' barrier, status and list
// lengths.  Bound by memory; with a quad's labels and zeros as vectors, where the
// width is a multiple of four, 5.6 us at 128^3, 8.9 at 160^3 and 16 for 256 x 128
// x 256, against 7.7, 12.2 and 22.
__global__ void __launch_bounds__(SCAN_BLOCK) k_fluid_tiles(const uint8_t* __restrict__ labels, Dims g,
                                                            float* __restrict__ p, int* __restrict__ tile_sums,
                                                            int stride, GridBar* bar, PcgOut* out, unsigned limit,
                                                            int* __restrict__ nq) {
    note_clock(&out->t_setup);
    const int nqr = quads_of_row(g), q = blockIdx.x * SCAN_BLOCK + threadIdx.x;
    int s = 0;
    if (q < nqr * g.H * g.D) {
        const int row = q / nqr, Q = q - row * nqr;
        const int64_t e0 = int64_t(row) * g.W + 4 * Q;
        const uchar4 l = quad_labels(labels + e0, g.W - 4 * Q, g.W);
        const bool f[4] = {l.x == FLUID, l.y == FLUID, l.z == FLUID, l.w == FLUID};
        s = f[0] + f[1] + f[2] + f[3];
        if (s == 0 && (g.W & 3) == 0) {
            *reinterpret_cast<float4*>(p + e0) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        } else {
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (!f[t] && 4 * Q + t < g.W) p[e0 + t] = 0.0f;
        }
        s |= int(s > 0) << 16;
    }
    int total;
    block_exclusive_scan<SCAN_BLOCK>(s, total);
    if (threadIdx.x == 0) {
        tile_sums[blockIdx.x] = total & 0xFFFF;
        tile_sums[stride + blockIdx.x] = total >> 16;
        if (blockIdx.x == 0) {
            bar->count = 0;
            bar->limit = limit;
            bar->gave_up = &out->t_end;
            out->status = DEV_OK;
            if (nq)
                for (int l = 0; l < MG_MAX_LEVELS; ++l) nq[l] = 0;
        }
    }
}

// RHSCalculator3D::operator() (FluidSolver3D.cu:1371-1456) at FLUID cell
// (i,j,k) from its faces' velocities and its neighbours' labels (-x, +x, -y,
// +y, -z, +z).
__device__ __forceinline__ float rhs_at(float u0, float u1, float v0, float v1, float w0, float w1,
                                        const uint8_t (&nl)[6], float dx, int i, int j, int k, float scale,
                                        const BodyKin& body) {
    float div = u1 - u0 + v1 - v0 + w1 - w0;
    float rhs = -scale * div;
    uint8_t l;
    l = nl[0];
    if (solidish(l)) {
        float s = l == BODY ? body_vel_at(body, make_float3(float(i) * dx, (float(j) + 0.5f) * dx, (float(k) + 0.5f) * dx)).x : 0.0f;
        rhs -= scale * (u0 - s);
    }
    l = nl[1];
    if (solidish(l)) {
        float s = l == BODY ? body_vel_at(body, make_float3(float(i + 1) * dx, (float(j) + 0.5f) * dx, (float(k) + 0.5f) * dx)).x : 0.0f;
        rhs += scale * (u1 - s);
    }
    l = nl[2];
    if (solidish(l)) {
        float s = l == BODY ? body_vel_at(body, make_float3((float(i) + 0.5f) * dx, float(j) * dx, (float(k) + 0.5f) * dx)).y : 0.0f;
        rhs -= scale * (v0 - s);
    }
    l = nl[3];
    if (solidish(l)) {
        float s = l == BODY ? body_vel_at(body, make_float3((float(i) + 0.5f) * dx, float(j + 1) * dx, (float(k) + 0.5f) * dx)).y : 0.0f;
        rhs += scale * (v1 - s);
    }
    l = nl[4];
    if (solidish(l)) {
        float s = l == BODY ? body_vel_at(body, make_float3((float(i) + 0.5f) * dx, (float(j) + 0.5f) * dx, float(k) * dx)).z : 0.0f;
        rhs -= scale * (w0 - s);
    }
    l = nl[5];
    if (solidish(l)) {
        float s = l == BODY ? body_vel_at(body, make_float3((float(i) + 0.5f) * dx, (float(j) + 0.5f) * dx, float(k + 1) * dx)).z : 0.0f;
        rhs += scale * (w1 - s);
    }
    return rhs;
}

// Level 0's quad list for the multigrid solver (null pointers: not wanted).
struct QuadOut {
    int4* q;
    float4* rhs;
    int sy0, sz0, sy1, sz1;  // padded strides of levels 0 and 1 (sy1 = 0: there is no level 1)
};

// Pass 3: the compact system (fidx, diag, b) of every FLUID cell, and the quad
// list.  A thread loads all labels and velocities of its quad before it uses
// any: cell by cell, each cell's loads waited for the one before (27 us at
// 128^3, 34 at 160^3, 51 for 256 x 128 x 256, where the writes bound it, against
// 18, 30 and 51, and 18, 29 and 48 with vector loads).
__global__ void __launch_bounds__(SCAN_BLOCK) k_fluid_build(const uint8_t* __restrict__ labels,
                                                            const float* __restrict__ u, const float* __restrict__ v,
                                                            const float* __restrict__ w, Dims g, float scale,
                                                            BodyKin body, const float* __restrict__ rhs_dense,
                                                            const int* __restrict__ tile_off, int stride,
                                                            int* __restrict__ fidx, uint8_t* __restrict__ diag,
                                                            float* __restrict__ b, QuadOut qo) {
    const int W = g.W, H = g.H, D = g.D;
    const int nqr = quads_of_row(g), q = blockIdx.x * SCAN_BLOCK + threadIdx.x;
    const int row = q / nqr, Q = q - row * nqr, k = row / H, j = row - k * H, i0 = 4 * Q;
    const bool in = q < nqr * H * D;
    const int64_t e0 = int64_t(row) * W + i0, wh = int64_t(W) * H;
    // labels i0 - 1 .. i0 + 4 of the row; cells beyond the grid are SOLID
    const uchar4 none = make_uchar4(SOLID, SOLID, SOLID, SOLID), lq = in ? quad_labels(labels + e0, W - i0, W) : none;
    const uint8_t lx[6] = {in && i0 > 0 ? labels[e0 - 1] : SOLID, lq.x, lq.y, lq.z, lq.w,
                           in && i0 + 4 < W ? labels[e0 + 4] : SOLID};
    int s = 0;
#pragma unroll
    for (int t = 0; t < 4; ++t) s += lx[t + 1] == FLUID;
    s |= int(s > 0) << 16;
    int total;
    const int pre = block_exclusive_scan<SCAN_BLOCK>(s, total);
    if ((s & 0xFFFF) == 0) return;
    int n = (pre & 0xFFFF) + tile_off[blockIdx.x];
    const int nq = (pre >> 16) + tile_off[stride + blockIdx.x];

    float uf[5], vf[2][4], wf[2][4], rd[4];
    const int64_t ui = int64_t(i0) + int64_t(row) * (W + 1);
    const int64_t vi = int64_t(i0) + int64_t(j) * W + int64_t(k) * W * (H + 1);
    const int m = W - i0;
    const uchar4 y0 = j > 0 ? quad_labels(labels + e0 - W, m, W) : none,
                 y1 = j + 1 < H ? quad_labels(labels + e0 + W, m, W) : none,
                 z0 = k > 0 ? quad_labels(labels + e0 - wh, m, W) : none,
                 z1 = k + 1 < D ? quad_labels(labels + e0 + wh, m, W) : none;
    const uint8_t ly[2][4] = {{y0.x, y0.y, y0.z, y0.w}, {y1.x, y1.y, y1.z, y1.w}};
    const uint8_t lz[2][4] = {{z0.x, z0.y, z0.z, z0.w}, {z1.x, z1.y, z1.z, z1.w}};
    if (rhs_dense) {
        quad_floats(rhs_dense + e0, m, W, rd);
    } else {
        quad_floats(v + vi, m, W, vf[0]);
        quad_floats(v + vi + W, m, W, vf[1]);
        quad_floats(w + e0, m, W, wf[0]);
        quad_floats(w + e0 + wh, m, W, wf[1]);
    }
    if (!rhs_dense)
#pragma unroll
        for (int t = 0; t < 5; ++t) uf[t] = i0 + t <= W ? u[ui + t] : 0.0f;

    const int pidx = (i0 + 1) + (j + 1) * (W + 2) + (k + 1) * (W + 2) * (H + 2);
    uint32_t codes = 0;
    float rq[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        if (lx[t + 1] != FLUID) continue;
        const uint8_t nl[6] = {lx[t], lx[t + 2], ly[0][t], ly[1][t], lz[0][t], lz[1][t]};
        int d = 0;
#pragma unroll
        for (int o = 0; o < 6; ++o) d += (nl[o] == FLUID || nl[o] == AIR);
        const float r = rhs_dense ? rd[t]
                                  : rhs_at(uf[t], uf[t + 1], vf[0][t], vf[1][t], wf[0][t], wf[1][t], nl, g.dx, i0 + t,
                                           j, k, scale, body);
        fidx[n] = pidx + t;
        diag[n] = uint8_t(d);
        b[n] = r;
        rq[t] = r;
        codes |= uint32_t(1 + d) << (8 * t);
        ++n;
    }
    if (!qo.q) return;
    if ((j + k) & 1) codes |= QUAD_ODD;
    if (((j >> 1) + (k >> 1)) & 1) codes |= QUAD_PARENT_ODD;
    const int c = (i0 + MG_OX) + (j + 1) * qo.sy0 + (k + 1) * qo.sz0;
    const int pc = qo.sy1 ? (2 * Q + MG_OX) + ((j >> 1) + 1) * qo.sy1 + ((k >> 1) + 1) * qo.sz1 : 0;
    qo.q[nq] = make_int4(c, int(codes), pc, int(e0));
    qo.rhs[nq] = make_float4(rq[0], rq[1], rq[2], rq[3]);
}

// ---------------------------------------------------------------- projection
// UFunctor/VFunctor/WFunctor (FluidSolver3D.cu:2072-2336) for one face between
// cells L and R: a SOLID/BODY side gets a ghost pressure that makes the face
// velocity equal to the wall velocity (0 or the rigid-body velocity).
__device__ __forceinline__ float project_face(float vel, uint8_t lL, uint8_t lR, float pL, float pR, float vb,
                                              float scale, float inv) {
    const bool fL = (lL == FLUID || lL == AIR), fR = (lR == FLUID || lR == AIR);
    float p0, p1;
    if (fL && fR) { p0 = pL; p1 = pR; }
    else if (solidish(lL)) { float s = lL == BODY ? vb : 0.0f; p0 = pR - inv * (vel - s); p1 = pR; }
    else if (solidish(lR)) { float s = lR == BODY ? vb : 0.0f; p0 = pL; p1 = pL + inv * (vel - s); }
    else { p0 = pL; p1 = pR; }
    return vel - scale * (p1 - p0);
}

__device__ __forceinline__ float p_at(const float* __restrict__ p, const Dims& g, int i, int j, int k) {
    if (i < 0 || i >= g.W || j < 0 || j >= g.H || k < 0 || k >= g.D) return 0.0f;
    return p[i + j * g.W + k * g.W * g.H];
}

__global__ void k_project(float* __restrict__ u, float* __restrict__ v, float* __restrict__ w,
                          const float* __restrict__ p, const uint8_t* __restrict__ lab, Dims g, float scale, float inv,
                          BodyKin body, const int* __restrict__ guard) {
    if (solve_failed(guard)) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z;
    const int W = g.W, H = g.H, D = g.D;
    if (i > W || j > H || k > D) return;
    const float dx = g.dx;
    const uint8_t lc = label_at(lab, g, i, j, k);
    // A face between two AIR cells keeps its velocity exactly (the pressure is
    // zero off the fluid: vel - scale * (0 - 0) is vel), so it is neither read
    // nor written; in a dam break most faces are such.
    const uint8_t lx = label_at(lab, g, i - 1, j, k), ly = label_at(lab, g, i, j - 1, k),
                  lz = label_at(lab, g, i, j, k - 1);
    const bool air = lc == AIR;
    const float pc = p_at(p, g, i, j, k);
    if (j < H && k < D && !(air && lx == AIR)) {
        int64_t id = int64_t(i) + int64_t(j) * (W + 1) + int64_t(k) * (W + 1) * H;
        float vb = body.active ? body_vel_at(body, make_float3(float(i) * dx, (float(j) + 0.5f) * dx, (float(k) + 0.5f) * dx)).x : 0.0f;
        u[id] = project_face(u[id], lx, lc, p_at(p, g, i - 1, j, k), pc, vb, scale, inv);
    }
    if (i < W && k < D && !(air && ly == AIR)) {
        int64_t id = int64_t(i) + int64_t(j) * W + int64_t(k) * W * (H + 1);
        float vb = body.active ? body_vel_at(body, make_float3((float(i) + 0.5f) * dx, float(j) * dx, (float(k) + 0.5f) * dx)).y : 0.0f;
        v[id] = project_face(v[id], ly, lc, p_at(p, g, i, j - 1, k), pc, vb, scale, inv);
    }
    if (i < W && j < H && !(air && lz == AIR)) {
        int64_t id = int64_t(i) + int64_t(j) * W + int64_t(k) * W * H;
        float vb = body.active ? body_vel_at(body, make_float3((float(i) + 0.5f) * dx, (float(j) + 0.5f) * dx, float(k) * dx)).z : 0.0f;
        w[id] = project_face(w[id], lz, lc, p_at(p, g, i, j, k - 1), pc, vb, scale, inv);
    }
}

// ---------------------------------------------------------------- CSR CG (FP64)
// Jacobi-preconditioned CG on a symmetric matrix stored as its upper triangle,
// y = U x + U^T x - diag(U) x, as one cooperative launch.
//
// Bound: latency.  A solve of 64,000 unknowns touches 4 MB, all of it in L2,
// so its time is the number of dependent steps.  As separate kernels with the
// scalars read back (ten launches and three host waits per iteration) 40^3
// unknowns to 1e-12 (202 iterations) took 18.0 ms on a B200; this kernel takes
// 1.52 ms, 7.5 us per iteration.  An iteration is two passes and two grid
// barriers:
//   pass 1 forms the row's new direction d = z + beta d_old, and its
//     neighbours' with the same fused multiply-add (so d needs no pass of its
//     own and no barrier between it and the product), adds the row's products
//     into q with FP64 reductions, and sums (d, A d) from the products it
//     makes: an entry (i, c) off the diagonal counts twice;
//   pass 2 updates x, r, z of the row, clears its q, and sums (r, z), (r, r).
// d is double-buffered, because pass 1 reads the old directions of other rows
// while their owners write the new ones.
constexpr int CSR_THREADS = 512;

struct CsrCgArgs {
    int n, check, maxit;
    double tol;
    const int *off, *cols;
    const double *vals, *b;
    double *x, *dg, *r, *z, *q, *d[2];
    double* part;  // [2][2][gridDim.x]
    CsrCtl* ctl;
};

// +0 computed from v, so that its store waits for the load of v (a store of a
// constant to an address with a load in flight stalls in the memory pipeline).
__device__ __forceinline__ double zero_after(double v) { return fmin(fabs(v), 0.0); }

// Entries e .. e + CSR_BATCH - 1 of a row that ends at e1; c = -1 past its end.
// A batch's loads are issued together; four hold a row of the 7-point operator.
// The first row's first batch stays in registers for the whole solve (the
// barriers' acquires empty L1); entry by entry, a row took one L2 round trip
// for each of them (2.03 ms for the solve above).
constexpr int CSR_BATCH = 4;
struct Entries {
    int c[CSR_BATCH];
    double v[CSR_BATCH];
};
__device__ __forceinline__ void load_entries(const CsrCgArgs& a, int e, int e1, Entries& k) {
#pragma unroll
    for (int u = 0; u < CSR_BATCH; ++u) {
        k.c[u] = e + u < e1 ? __ldg(a.cols + e + u) : -1;
        k.v[u] = e + u < e1 ? __ldg(a.vals + e + u) : 0.0;
    }
}

__global__ void __launch_bounds__(CSR_THREADS) k_csr_cg(CsrCgArgs a) {
    const int nb = int(gridDim.x);
    const int t0 = int(blockIdx.x) * CSR_THREADS + threadIdx.x, st = nb * CSR_THREADS;
    CsrCtl* ctl = a.ctl;
    int red = 0;
    auto reduce = [&](double (&v)[2]) {
        return grid_reduce(v, a.part + (red++ & 1) * 2 * nb, &ctl->bar, nb, &ctl->status);
    };
    if (a.check) {
        // row offsets start at 0 and never decrease; then the columns, whose loop bounds that makes safe
        for (int i = t0; i < a.n; i += st)
            if ((i == 0 && a.off[0] != 0) || a.off[i + 1] < a.off[i]) ctl->bad_off = 1;
        if (!grid_barrier(&ctl->bar, unsigned(nb), &ctl->status)) return;
        if (__ldcg(&ctl->bad_off)) return;
        for (int i = t0; i < a.n; i += st)
            for (int e = a.off[i]; e < a.off[i + 1]; ++e)
                if (a.cols[e] < 0 || a.cols[e] >= a.n) ctl->bad_col = 1;
        if (!grid_barrier(&ctl->bar, unsigned(nb), &ctl->status)) return;
        if (__ldcg(&ctl->bad_col)) return;
    }
    double sum[2] = {0.0, 0.0};
    for (int i = t0; i < a.n; i += st) {
        double d = 1.0;
        for (int e = a.off[i]; e < a.off[i + 1]; ++e)
            if (a.cols[e] == i) d = a.vals[e];
        const double r = a.b[i], z = r / d;
        a.dg[i] = d;
        a.r[i] = r;
        a.z[i] = z;
        a.x[i] = 0.0;
        a.q[i] = 0.0;
        a.d[1][i] = 0.0;
        sum[0] += r * z;
        sum[1] += r * r;
    }
    // the thread's first row: offsets and entries, -1 past its end
    int e_first = 0, e_last = 0;
    Entries first;
    if (t0 < a.n) {
        e_first = a.off[t0];
        e_last = a.off[t0 + 1];
        load_entries(a, e_first, e_last, first);
    }
    if (!reduce(sum)) return;
    double rz = sum[0], rr = sum[1], beta = 0.0;
    const double bb = rr;
    int it = 0;
    while (bb > 0.0 && rr > a.tol * a.tol * bb && it < a.maxit) {
        double* dn = a.d[it & 1];
        const double* dold = a.d[(it & 1) ^ 1];
        sum[0] = sum[1] = 0.0;
        for (int i = t0; i < a.n; i += st) {
            const bool f = i == t0;
            const int e0 = f ? e_first : __ldg(a.off + i), e1 = f ? e_last : __ldg(a.off + i + 1);
            double di = 0.0, s = 0.0, pair = 0.0, own = 0.0;
            for (int e = e0;; e += CSR_BATCH) {
                Entries k = first;
                if (!(f && e == e0)) load_entries(a, e, e1, k);
                double zc[CSR_BATCH], dc[CSR_BATCH];
#pragma unroll
                for (int u = 0; u < CSR_BATCH; ++u) {
                    const int c = k.c[u] < 0 ? i : k.c[u];
                    zc[u] = a.z[c];
                    dc[u] = dold[c];
                }
                if (e == e0) di = __fma_rn(beta, dold[i], a.z[i]);
#pragma unroll
                for (int u = 0; u < CSR_BATCH; ++u) {
                    if (k.c[u] < 0) continue;
                    if (k.c[u] == i) {
                        own += k.v[u] * di;
                        continue;
                    }
                    const double t = k.v[u] * __fma_rn(beta, dc[u], zc[u]);
                    s += t;
                    pair += t;
                    atomicAdd(&a.q[k.c[u]], k.v[u] * di);
                }
                if (e + CSR_BATCH >= e1) break;
            }
            dn[i] = di;
            atomicAdd(&a.q[i], s + own);
            sum[0] += di * (own + 2.0 * pair);
        }
        if (!reduce(sum)) return;
        if (!(sum[0] > 0.0)) break;
        const double alpha = rz / sum[0];
        sum[0] = sum[1] = 0.0;
        for (int i = t0; i < a.n; i += st) {
            const double q = __ldcg(a.q + i);  // summed in L2
            const double r = a.r[i] - alpha * q, z = r / a.dg[i];
            a.x[i] += alpha * dn[i];
            a.r[i] = r;
            a.z[i] = z;
            a.q[i] = zero_after(q);
            sum[0] += r * z;
            sum[1] += r * r;
        }
        if (!reduce(sum)) return;
        beta = sum[0] / rz;
        rz = sum[0];
        rr = sum[1];
        ++it;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        ctl->iters = it;
        ctl->rr = rr;
        ctl->bb = bb;
    }
}

__global__ void k_csr_reset(CsrCtl* ctl, unsigned limit) {
    ctl->bar.count = 0;
    ctl->bar.limit = limit;
    ctl->bar.gave_up = nullptr;
    ctl->status = DEV_OK;
    ctl->bad_off = ctl->bad_col = 0;
    ctl->iters = 0;
    ctl->rr = ctl->bb = 0.0;
}

}  // namespace

// ---------------------------------------------------------------- launchers

static int quad_tiles(Dims g) {
    const int64_t nq = int64_t((g.W + 3) / 4) * g.H * g.D;
    return int((nq + SCAN_BLOCK - 1) / SCAN_BLOCK);
}
// Two rows of tile counts, each from a multiple of four (k_scan_rows reads vectors).
int pressure_tiles(Dims g) { return 2 * ((quad_tiles(g) + 3) & ~3); }

void launch_pressure_setup(const uint8_t* labels, const float* u, const float* v, const float* w, Dims g, float dt,
                           BodyKin body, const float* rhs_dense, float* p, PressureBufs& pb, const MgBufs* mg,
                           unsigned wait_polls, cudaStream_t st) {
    const int ntiles = quad_tiles(g), stride = pressure_tiles(g) / 2;
    const float scale = (1000.0f * g.dx) / dt;  // rho*dx/dt, FluidSolver3D.cu:1520
    QuadOut qo{};
    if (mg && mg->L > 0) {
        qo.q = mg->q[0];
        qo.rhs = mg->rhs;
        qo.sy0 = mg->lv[0].sy; qo.sz0 = mg->lv[0].sz;
        if (mg->L > 1) { qo.sy1 = mg->lv[1].sy; qo.sz1 = mg->lv[1].sz; }
    }
    int* nq = qo.q ? mg->nq : nullptr;
    k_fluid_tiles<<<ntiles, SCAN_BLOCK, 0, st>>>(labels, g, p, pb.tile_sums, stride, pb.bar, pb.out, wait_polls, nq);
    k_scan_rows<<<2, 1024, 0, st>>>(pb.tile_sums, ntiles, stride, pb.nf, nq);
    k_fluid_build<<<ntiles, SCAN_BLOCK, 0, st>>>(labels, u, v, w, g, scale, body, rhs_dense, pb.tile_sums, stride,
                                                 pb.fidx, pb.diag, pb.b, qo);
}

void launch_project(float* u, float* v, float* w, const float* p, const uint8_t* labels, Dims g, float dt, BodyKin b,
                    cudaStream_t st, const int* guard) {
    const float scale = dt / (1000.0f * g.dx);  // dt/(rho*dx), FluidSolver3D.cu:2341
    const float inv = 1.0f / scale;
    dim3 blk(32, 8, 1);
    dim3 grd((g.W + 1 + 31) / 32, (g.H + 1 + 7) / 8, g.D + 1);
    k_project<<<grd, blk, 0, st>>>(u, v, w, p, labels, g, scale, inv, b, guard);
}

int launch_csr_cg(int n, const int* off, const int* cols, const double* vals, const double* b, double* x, double* work,
                  int64_t stride, double* part, CsrCtl* ctl, int check, double tol, int maxit, cudaStream_t st,
                  unsigned wait_polls) {
    static DeviceMemo memo;
    const int resident = memo.get([](int dev) {
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        return std::min(sms, kCsrMaxBlocks);
    });
    // One row per thread while that fits one CTA per SM (a one-CTA grid's barrier is a block barrier).
    const int nb = std::max(1, std::min(resident, (n - 1) / CSR_THREADS + 1));
    k_csr_reset<<<1, 1, 0, st>>>(ctl, wait_polls);
    CsrCgArgs a{};
    a.n = n; a.check = check; a.maxit = maxit; a.tol = tol;
    a.off = off; a.cols = cols; a.vals = vals; a.b = b; a.x = x;
    double** v[kCsrVectors] = {&a.dg, &a.r, &a.z, &a.q, &a.d[0], &a.d[1]};
    for (int i = 0; i < kCsrVectors; ++i) *v[i] = work + i * stride;
    a.part = part;
    a.ctl = ctl;
    void* args[] = {&a};
    return int(cudaLaunchCooperativeKernel((const void*)k_csr_cg, dim3(nb), dim3(CSR_THREADS), args, 0, st));
}

int csr_cg_solve(int n, const int* offsets, const int* cols, const double* vals, const double* b, double* x, double tol,
                 int maxit, int* iters, double* relres, cudaStream_t st, unsigned wait_polls) {
    const size_t nnz = size_t(offsets[n]), N = size_t(n);
    // one allocation: doubles (values, b, x, the work vectors), the partials and the control block, then the integers
    const size_t nd = nnz + (2 + kCsrVectors) * N;
    const size_t bytes = sizeof(double) * (nd + kCsrPartials) + sizeof(CsrCtl) + sizeof(int) * (N + 1 + nnz);
    unsigned char* base = nullptr;
    cudaError_t e = cudaMalloc(&base, bytes);
    if (e != cudaSuccess) return FP_ERR_CUDA;
    double* d_vals = reinterpret_cast<double*>(base);
    double *d_b = d_vals + nnz, *d_x = d_b + N, *work = d_x + N;
    double* part = d_vals + nd;
    CsrCtl* ctl = reinterpret_cast<CsrCtl*>(part + kCsrPartials);
    int* d_off = reinterpret_cast<int*>(ctl + 1);
    int* d_cols = d_off + N + 1;
    auto ck = [&](cudaError_t r) { if (r != cudaSuccess && e == cudaSuccess) e = r; };
    ck(cudaMemcpyAsync(d_off, offsets, sizeof(int) * (N + 1), cudaMemcpyHostToDevice, st));
    ck(cudaMemcpyAsync(d_cols, cols, sizeof(int) * nnz, cudaMemcpyHostToDevice, st));
    ck(cudaMemcpyAsync(d_vals, vals, sizeof(double) * nnz, cudaMemcpyHostToDevice, st));
    ck(cudaMemcpyAsync(d_b, b, sizeof(double) * N, cudaMemcpyHostToDevice, st));
    if (e == cudaSuccess)
        ck(cudaError_t(launch_csr_cg(n, d_off, d_cols, d_vals, d_b, d_x, work, int64_t(N), part, ctl, 0, tol, maxit, st,
                                     wait_polls)));
    CsrCtl h{};
    ck(cudaMemcpyAsync(&h, ctl, sizeof h, cudaMemcpyDeviceToHost, st));
    ck(cudaStreamSynchronize(st));
    const bool gave_up = e == cudaSuccess && h.status != DEV_OK;
    if (e == cudaSuccess && !gave_up) {
        ck(cudaMemcpyAsync(x, d_x, sizeof(double) * N, cudaMemcpyDeviceToHost, st));
        ck(cudaStreamSynchronize(st));
    }
    cudaFree(base);
    if (gave_up) return FP_ERR_TIMEOUT;
    if (e != cudaSuccess) return FP_ERR_CUDA;
    if (iters) *iters = h.iters;
    if (relres) *relres = h.bb > 0 ? sqrt(h.rr / h.bb) : 0.0;
    return FP_OK;
}

}  // namespace fp
