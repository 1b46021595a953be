// kernels_mg.cu -- multigrid-preconditioned conjugate gradients for the
// pressure Poisson system (FP_SOLVER_PCG_MG).
//
// Same system as the reference's cuDSS solve (FluidSolver3D.cu:1815-2062): unit
// 7-point operator over FLUID cells, AIR = Dirichlet 0, SOLID/BODY and
// out-of-domain = Neumann.  Preconditioner: one geometric multigrid V-cycle.
//   * Levels coarsen by 2 per axis; a coarse cell is AIR if any child is AIR,
//     else FLUID if any child is FLUID, else SOLID (Dirichlet priority), and
//     carries the rediscretised unit operator of its labels.
//   * Restriction sums the FLUID children's residuals and scales by 1/4 (3D)
//     or 1/2 (2D); prolongation adds the coarse value to every FLUID child.
//     With these transfers R*A*P equals the coarse unit operator, and P is a
//     multiple of R^T.
//   * Smoother: red-black Gauss-Seidel over-relaxed by MG_SOR, red then black
//     going down, black then red coming up (two pairs on the finest level by
//     default, one on the other grid-wide levels, two on the block levels);
//     the coarsest level does the same symmetric sweeps.  The V-cycle is
//     therefore a symmetric positive definite preconditioner.  After the black
//     sweep only red cells carry a residual, so restriction sums the red
//     children.  The coarse correction is scaled by omega.
// Layout: every level is a padded grid whose rows are a multiple of four cells
// apart and start four cells in (MG_OX), so that four cells of a row -- a quad
// -- are one aligned 16-byte vector and both halos of a row are the zero gap
// before the next one.  Grid-wide levels are walked as lists of the quads that
// hold a FLUID cell: a sweep of a quad is eight loads (its row of x, b, the four
// neighbouring rows, one cell at each end), where cell by cell it took 36, and
// the issue of those loads is what a phase waited for: with one cell per
// thread a level-0 sweep took 3.2 us at 485,000 FLUID cells and 9.8 at 2.2 M,
// against 2.6 and 7.2.  A thread's first quads stay in shared memory (slot_of).
// Code length counts as much as loads: a phase runs once between two grid
// barriers, so its instructions are fetched as it goes, and the phases are short
// functions, one quad a trip, rather than unrolled and inlined.
// Per solve, a cell per thread and trip against quads: dam break 64 x 64 187 and
// 132 us, 128^3 849 and 730, pool 160^3 2350 and 1700, 256 x 128 x 256 2047 and
// 1460, at the same iterations; 123, 698, 1648 and 1395 with the block levels'
// stage as it is now.
// Levels with more than MG_BLOCK_CELLS cells are swept by the whole grid with a
// grid barrier between sweeps; every block then does the remaining coarse
// levels on its own shared-memory copy with __syncthreads only (labels
// coarsened there at kernel start; the first block level's b and x copied in
// per cycle) and prolongs from that copy, so the stage costs no grid barrier
// of its own (one block alone, with a copy-out and a barrier, was 1.5 us per
// iteration slower at 128^3).  A level of 8000 cells (160^3) done so instead of
// grid-wide took 1884 instead of 1648 us per solve.  Block levels take
// MG_NU_BLOCK sweep pairs:
// two instead of one took the 128^3 dam break from 10.85 to 10.1 iterations
// per warm-started solve (1.030 to 0.985 ms); two pairs on the grid-wide
// levels as well reached 8.9 iterations, but their extra grid barriers made
// the solve slower (1.067 ms).  The whole PCG (flexible, in the Chronopoulos-Gear
// form, optionally started from a guess) runs in one persistent cooperative
// launch with the bounded grid barrier.  Precision split: the V-cycle works in
// FP32; the Krylov vectors (x, r, p, s; stored by quads) and all dot products
// are FP64, so the recurrence residual tracks the true residual down to the
// 1e-6 target without restarts.
#include <algorithm>

#include "device_memo.hpp"
#include "kernels.hpp"
#include "pcg_common.cuh"

namespace fp {

namespace {

// One CTA per SM, 128 registers a thread.  Per solve of the four scenes above:
// 384 threads 133, 791, 1852 and 1582 us, 512 132, 730, 1700 and 1457, 640 138,
// 783, 1672 and 1388 (with 96 registers, some spilled): 512 is the best or near it.
constexpr int MG_THREADS = 512;
// Red-black sweep pairs before and after the coarse correction on the
// grid-wide levels below the finest (MG_NU_GRID) and on the block levels
// above the coarsest (MG_NU_BLOCK); build tunables.
#ifndef MG_NU_GRID
#define MG_NU_GRID 1
#endif
#ifndef MG_NU_BLOCK
#define MG_NU_BLOCK 2
#endif
// Symmetric sweep pairs on the coarsest level (build tunable).
#ifndef MG_NU_COARSE
#define MG_NU_COARSE 2
#endif
// Scale of the coarse-grid correction (build tunable).
#ifndef MG_OMEGA
#define MG_OMEGA 1.7f
#endif
// Over-relaxation of every red-black Gauss-Seidel update (pre- and
// post-smoothing alike, so the cycle stays symmetric): x <- x + w (y - x),
// y = (b + neighbours) / d.  1 is plain Gauss-Seidel.  With two sweep pairs
// on the block levels, 1.2 (and a coarse correction scaled by 1.7) took the
// 128^3 dam break from 10.83 to 10.35 iterations per warm-started solve and
// from 12.9 to 12.1 from x = 0 (mean of 40 steps), against 1.1 and 1.8; 1.15
// gave 10.48 and 12.5, 1.25 (with 1.8) 11.1.
#ifndef MG_SOR_VALUE
#define MG_SOR_VALUE 1.2f
#endif
constexpr float MG_SOR = MG_SOR_VALUE;
// The same on the coarser levels (build tunable MG_SOR_COARSE_VALUE).
#ifndef MG_SOR_COARSE_VALUE
#define MG_SOR_COARSE_VALUE MG_SOR_VALUE
#endif
constexpr float MG_SORC = MG_SOR_COARSE_VALUE;

struct MgArgs {
    int L, G;                    // levels; levels [0, G) are grid-wide
    int smem;                    // bytes of the shared-memory copies of levels [G, L); 0: none
    float rscale;                // restriction scale (1/4 in 3D, 1/2 in 2D)
    float omega;                 // over-relaxation of the coarse-grid correction
    int nu_coarse;               // symmetric sweep pairs on the coarsest level
    int nu0;                     // red-black sweep pairs before and after on level 0
    int nu_grid;                 // ... on the other grid-wide levels
    int nu_block;                // ... on the block levels above the coarsest
    MgLevel lv[MG_MAX_LEVELS];
    const int4* q[MG_MAX_LEVELS];  // quad lists of levels [0, max(G, 1)) (QUAD_* entries)
    const int* nq;               // their lengths
    const float4* rhs;           // right-hand side by level-0 quad (zero off the fluid)
    // FP64 Krylov vectors by quad: the first two cells of quad n at [n], the last two at [cap + n]
    double2 *p, *s, *xs, *r, *w;
    int cap;
    double* xd;                  // level-0 grid for the FP64 solution, zero between solves
    const float* guess;          // dense W x H x D guess, or null
    int guess_dir;               // the guess is the first search direction (the network's)
    float* pout;                 // dense W x H x D pressure out (zero off the fluid already)
    double* red;                 // [2] out: ||rhs - A x||^2 and ||rhs||^2 of the solution, in FP64
    double* part;
    GridBar* bar;
    int* status;
    PcgOut* out;
    double tol;
    int maxit;
};

__host__ __device__ __forceinline__ int lv_index(const MgLevel& L, int i, int j, int k) {
    return (i + MG_OX) + (j + 1) * L.sy + (k + 1) * L.sz;
}
// Cells of a level's padded grid (vector loads at its end stay inside).
__host__ __device__ __forceinline__ int npad(const MgLevel& L) { return L.sz * (L.D + 2) + 2 * MG_OX; }
__device__ __forceinline__ int lv_diag(const MgLevel& L, int c) {
    const uint8_t* l = L.lab;
    const int o[6] = {1, -1, L.sy, -L.sy, L.sz, -L.sz};
    int d = 0;
#pragma unroll
    for (int m = 0; m < 6; ++m) { const uint8_t v = l[c + o[m]]; d += (v == FLUID || v == AIR); }
    return d;
}
__device__ __forceinline__ float lv_nbsum(const MgLevel& L, int c) {
    const float* x = L.x;
    return (x[c + 1] + x[c - 1]) + (x[c + L.sy] + x[c - L.sy]) + (x[c + L.sz] + x[c - L.sz]);
}
__device__ __forceinline__ int lv_cell(const MgLevel& L, int t, int& i, int& j, int& k) {
    i = t % L.W; j = (t / L.W) % L.H; k = t / (L.W * L.H);
    return lv_index(L, i, j, k);
}

// 1 / d of the diagonals d = 1..6 by code 1 + d; 0 for codes 0 and 1 (a FLUID
// cell with no FLUID or AIR neighbour takes x = 0).
__shared__ float s_rcp[8];
// Over-relaxed Gauss-Seidel value y = (b + nb) / d of a FLUID cell.  The
// division is a multiplication by the rounded reciprocal: one more rounding, in
// the FP32 preconditioner only.
__device__ __forceinline__ float gs_value(float xo, float b, float nb, int dc, float w) {
    const float y = (b + nb) * s_rcp[dc];
    return dc > 1 ? xo + w * (y - xo) : (dc == 1 ? 0.0f : xo);
}
// ---- operations over quad lists ----
// A thread's quads are n = t0 + q * stride for trips q = 0, 1, ..., one at a
// time: a grid-wide phase's code is cold when it starts, and at 512 threads its
// length costs more than a second quad's loads in flight gain (two quads a
// trip: 0.83 against 0.72 ms for a warm-started 128^3 solve, 1.83 against 1.56
// for 256 x 128 x 256).
struct Quad {
    int c;       // index of the first cell
    uint32_t k;  // four codes (1 + diagonal, 0: not FLUID) and parity bits
    int pc;      // index of its first cells' parent on the next level
};
// The first trips' quads of the grid-wide levels, kept in shared memory for the
// whole solve: two on levels 0 and 1, one on levels 2 and 3 (in each thread's
// own column; only the thread itself reads them).
constexpr int SLOTS = 6;
__shared__ int s_qc[SLOTS * MG_THREADS], s_qp[SLOTS * MG_THREADS];
__shared__ uint32_t s_qk[SLOTS * MG_THREADS];
__shared__ int s_nq[MG_MAX_LEVELS];  // the lists' lengths
__device__ __forceinline__ int slot_of(int l) { return l < 2 ? 2 * l : l + 2; }  // first slot of level l
__device__ __forceinline__ int slots_of(int l) { return l < 2 ? 2 : (l <= 3 ? 1 : 0); }
// Codes and parity bits of a list entry (level 0's carries its codes).
__device__ __forceinline__ uint32_t codes_of(const MgLevel& L, int l, const int4& e) {
    return l == 0 ? uint32_t(e.y) : *reinterpret_cast<const uint32_t*>(L.code + e.x) | (uint32_t(e.y) & QUAD_PAR);
}
// Fills the slots of levels [l0, l1) (the codes must be complete).
__device__ __forceinline__ void fill_slots(const MgArgs& a, int l0, int l1, int t0, int st) {
    for (int l = l0; l < min(l1, 4); ++l)
        for (int u = 0; u < slots_of(l); ++u) {
            const int n = t0 + u * st, at = (slot_of(l) + u) * MG_THREADS + threadIdx.x;
            if (n >= s_nq[l]) continue;
            const int4 e = a.q[l][n];
            s_qc[at] = e.x;
            s_qk[at] = codes_of(a.lv[l], l, e);
            s_qp[at] = e.z;
        }
}
// Calls f(quad, n) for each of the thread's quads of level l; the entry of the
// next one is on its way meanwhile.
template <class Fn>
__device__ __forceinline__ void for_quads(const MgArgs& a, int l, Fn f) {
    const int st = gridDim.x * MG_THREADS, nq = s_nq[l], slots = slots_of(l);
    const int4* list = a.q[l];
    int n = blockIdx.x * MG_THREADS + threadIdx.x, at = slot_of(l) * MG_THREADS + threadIdx.x, q = 0;
    int4 next = make_int4(0, 0, 0, 0);
    if (slots == 0 && n < nq) next = list[n];
#pragma unroll 1
    for (; n < nq; n += st, ++q, at += MG_THREADS) {
        Quad Q;
        if (q < slots) Q = Quad{s_qc[at], s_qk[at], s_qp[at]};
        else Q = Quad{next.x, codes_of(a.lv[l], l, next), next.z};
        if (q + 1 >= slots && n + st < nq) next = list[n + st];
        f(Q, n);
    }
}
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float2 ld2(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ int code_at(uint32_t k, int e) { return int((k >> (8 * e)) & 7u); }

// Gauss-Seidel update of the FLUID cells of one colour (0 red: even i + j + k)
// of a quad: cells 0, 2 or 1, 3.
__device__ __forceinline__ void sweep_quad(const MgLevel& L, const Quad& Q, int color, float w) {
    float* X = L.x + Q.c;
    const float4 x = ld4(X), yp = ld4(X + L.sy), ym = ld4(X - L.sy), zp = ld4(X + L.sz), zm = ld4(X - L.sz);
    const float xl = X[-1], xr = X[4];
    const float4 b = ld4(L.b + Q.c);
    const bool odd = (((Q.k >> 7) & 1u) ^ uint32_t(color)) != 0u;
    const float nba = ((odd ? x.z : x.y) + (odd ? x.x : xl)) + ((odd ? yp.y : yp.x) + (odd ? ym.y : ym.x)) +
                      ((odd ? zp.y : zp.x) + (odd ? zm.y : zm.x));
    const float nbb = ((odd ? xr : x.w) + (odd ? x.z : x.y)) + ((odd ? yp.w : yp.z) + (odd ? ym.w : ym.z)) +
                      ((odd ? zp.w : zp.z) + (odd ? zm.w : zm.z));
    const float va = gs_value(odd ? x.y : x.x, odd ? b.y : b.x, nba, code_at(Q.k, odd ? 1 : 0), w);
    const float vb = gs_value(odd ? x.w : x.z, odd ? b.w : b.z, nbb, code_at(Q.k, odd ? 3 : 2), w);
    // the other colour's cells keep their values: this thread alone owns the quad
    *reinterpret_cast<float4*>(X) = odd ? make_float4(x.x, va, x.z, vb) : make_float4(va, x.y, vb, x.w);
}
// Restriction into the listed cells of level Cl fused with that level's first
// sweep: b_coarse = scale * sum over the red FLUID children of (b - A x), then
// x_coarse = b/d on red FLUID cells, 0 on black ones.  After the black sweep
// the black residuals vanish, so only the red children (offsets with an even
// coordinate sum) are summed, in k, j, i order.  One thread per coarse cell;
// its 2 x 2 x 2 children are four aligned pairs.  Children beyond an odd-sized
// level are halo cells with code 0; those in z would have neighbours beyond
// the grid, so they are not read.
__device__ __forceinline__ void restrict_quads(const MgLevel& F, const MgLevel& Cl, float scale, const int4* list,
                                               int nq, int t0, int st) {
    for (int t = t0; t < 4 * nq; t += st) {
        const int4 E = list[t >> 2];
        const int e = t & 3, cc = E.x + e, r0 = E.w + 2 * e, r1 = r0 + F.sy, r2 = r0 + F.sz, r3 = r1 + F.sz;
        const bool kk = (uint32_t(E.y) & QUAD_Z) != 0u;
        const int dc = Cl.code[cc];
        const float* X = F.x;
        const float2 x0 = ld2(X + r0), x1 = ld2(X + r1);
        const float a0 = X[r0 - 1], a1 = X[r0 - F.sy], a2 = X[r0 - F.sz];
        const float b0 = X[r1 + 2], b1 = X[r1 + 1 + F.sy], b2 = X[r1 + 1 - F.sz];
        const int d0 = F.code[r0], d1 = F.code[r1 + 1];
        const float f0 = F.b[r0], f1 = F.b[r1 + 1];
        float2 x2 = make_float2(0.0f, 0.0f), x3 = x2;
        float c0 = 0.0f, c1 = 0.0f, c2 = 0.0f, g0 = 0.0f, g1 = 0.0f, g2 = 0.0f, f2 = 0.0f, f3 = 0.0f;
        int d2 = 0, d3 = 0;
        if (kk) {
            x2 = ld2(X + r2); x3 = ld2(X + r3);
            c0 = X[r2 + 2]; c1 = X[r2 + 1 - F.sy]; c2 = X[r2 + 1 + F.sz];
            g0 = X[r3 - 1]; g1 = X[r3 + F.sy]; g2 = X[r3 + F.sz];
            d2 = F.code[r2 + 1]; d3 = F.code[r3];
            f2 = F.b[r2 + 1]; f3 = F.b[r3];
        }
        if (dc == 0) continue;
        auto res = [](int d, float bv, float xv, float nb) { return d > 0 ? bv - (float(d - 1) * xv - nb) : 0.0f; };
        float s = res(d0, f0, x0.x, (x0.y + a0) + (x1.x + a1) + (x2.x + a2));
        s += res(d1, f1, x1.y, (b0 + x1.x) + (b1 + x0.y) + (x3.y + b2));
        s += res(d2, f2, x2.y, (c0 + x2.x) + (x3.y + c1) + (c2 + x0.y));
        s += res(d3, f3, x3.x, (x3.y + g0) + (g1 + x2.x) + (g2 + x1.x));
        s *= scale;
        const bool red = ((uint32_t(E.y) >> 7) & 1u) == uint32_t(e & 1);
        Cl.b[cc] = s;
        Cl.x[cc] = red ? gs_value(0.0f, s, 0.0f, dc, MG_SORC) : 0.0f;
    }
}
// The last (red) sweep of a coarse level fused with the prolongation of its
// result: every FLUID fine cell with a FLUID parent adds omega * (parent's
// value), where a red parent's value is its Gauss-Seidel update (recomputed
// by each of its children from the final black neighbours, with the same
// arithmetic, so all eight see the same bits) and a black parent's is final.
// The coarse x is not needed after this, so it is not written back.  A quad's
// four cells have two parents, an aligned pair.
__device__ __forceinline__ void prolong_quad(const MgLevel& F, const MgLevel& Cl, float omega, const Quad& Q) {
    const float* X = Cl.x + Q.pc;
    float4 f = ld4(F.x + Q.c);
    const int d = *reinterpret_cast<const uint16_t*>(Cl.code + Q.pc), d0 = d & 0xFF, d1 = d >> 8;
    const float2 x = ld2(X), yp = ld2(X + Cl.sy), ym = ld2(X - Cl.sy), zp = ld2(X + Cl.sz), zm = ld2(X - Cl.sz);
    const float xl = X[-1], xr = X[2];
    const float2 b = ld2(Cl.b + Q.pc);
    const bool odd = (Q.k & QUAD_PARENT_ODD) != 0u;  // the first parent is black
    // the one parent that is red
    const float nb = odd ? (xr + x.x) + (yp.y + ym.y) + (zp.y + zm.y) : (x.y + xl) + (yp.x + ym.x) + (zp.x + zm.x);
    const float v = gs_value(odd ? x.y : x.x, odd ? b.y : b.x, nb, odd ? d1 : d0, MG_SORC);
    const float v0 = odd ? x.x : v, v1 = odd ? v : x.y;
    if (d0 > 0) {
        if (code_at(Q.k, 0)) f.x = f.x + omega * v0;
        if (code_at(Q.k, 1)) f.y = f.y + omega * v0;
    }
    if (d1 > 0) {
        if (code_at(Q.k, 2)) f.z = f.z + omega * v1;
        if (code_at(Q.k, 3)) f.w = f.w + omega * v1;
    }
    *reinterpret_cast<float4*>(F.x + Q.c) = f;
}
// Codes of the listed quads of a level from its labels (zero elsewhere).
__device__ __forceinline__ void codes_quads(const MgLevel& L, const int4* list, int nq, int t0, int st) {
    for (int n = t0; n < nq; n += st) {
        const int c = list[n].x;
        uint32_t k = 0;
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (L.lab[c + e] == FLUID) k |= uint32_t(1 + lv_diag(L, c + e)) << (8 * e);
        *reinterpret_cast<uint32_t*>(L.code + c) = k;
    }
}

// ---- dense operations over a (t0, stride) share of a level: the block levels
// in global memory, and the restriction into the first block level ----
// They read the level's code (FLUID: 1 + diagonal, else 0) instead of labels,
// and issue a cell's loads together, masked by the code afterwards: every
// load is of an interior cell or its halo, so it stays in bounds.
// Gauss-Seidel update of one FLUID cell (code dc > 0).
__device__ __forceinline__ void gs_update(const MgLevel& L, int c) {
    const int dc = L.code[c];
    const float bv = L.b[c], nb = lv_nbsum(L, c), xo = L.x[c];
    if (dc > 0) L.x[c] = gs_value(xo, bv, nb, dc, MG_SORC);
}
// Gauss-Seidel update of the FLUID cells of one colour.
__device__ void op_sweep(const MgLevel& L, int color, int t0, int stride) {
    const int n = L.W * L.H * L.D;
    for (int t = t0; t < n; t += stride) {
        int i, j, k;
        const int c = lv_cell(L, t, i, j, k);
        if (((i + j + k) & 1) == color) gs_update(L, c);
    }
}
// Residual b - A x of fine cell c if it is FLUID, else 0.
__device__ __forceinline__ float fine_residual(const MgLevel& F, int c) {
    const int dc = F.code[c];
    const float bv = F.b[c], xv = F.x[c], nb = lv_nbsum(F, c);
    return dc > 0 ? bv - (float(dc - 1) * xv - nb) : 0.0f;
}
// restrict_quads' operation over every cell of Cl (x and b zero off the fluid).
// A child beyond an odd-sized fine level (every 2D level in z) is skipped: its
// stencil would leave the padded grid.
__device__ void op_restrict_first(const MgLevel& F, const MgLevel& Cl, float scale, int t0, int stride) {
    const int n = Cl.W * Cl.H * Cl.D;
    for (int t = t0; t < n; t += stride) {
        int I, J, K;
        const int cc = lv_cell(Cl, t, I, J, K);
        const int dc = Cl.code[cc];
        float s = 0.0f, xv = 0.0f;
        if (dc > 0) {
            const bool ii = 2 * I + 1 < F.W, jj = 2 * J + 1 < F.H, kk = 2 * K + 1 < F.D;
            const int c0 = lv_index(F, 2 * I, 2 * J, 2 * K);
            s += fine_residual(F, c0);
            if (ii && jj) s += fine_residual(F, c0 + 1 + F.sy);
            if (ii && kk) s += fine_residual(F, c0 + 1 + F.sz);
            if (jj && kk) s += fine_residual(F, c0 + F.sy + F.sz);
            s *= scale;
            if (((I + J + K) & 1) == 0) xv = gs_value(0.0f, s, 0.0f, dc, MG_SORC);
        }
        Cl.b[cc] = s;
        Cl.x[cc] = xv;
    }
}
// prolong_quad's operation on one cell, and over every FLUID cell of F.
__device__ __forceinline__ void prolong_one(const MgLevel& F, int c, const MgLevel& Cl, float omega, int i, int j,
                                            int k) {
    const int I = i >> 1, J = j >> 1, K = k >> 1;
    const int cc = lv_index(Cl, I, J, K);
    const int dc = Cl.code[cc];
    const float xc = Cl.x[cc], bc = Cl.b[cc], nb = lv_nbsum(Cl, cc), xf = F.x[c];
    if (dc == 0) return;
    const float v = ((I + J + K) & 1) != 0 ? xc : gs_value(xc, bc, nb, dc, MG_SORC);
    F.x[c] = xf + omega * v;
}
__device__ void op_prolong_red(const MgLevel& F, const MgLevel& Cl, float omega, int t0, int stride) {
    const int n = F.W * F.H * F.D;
    for (int t = t0; t < n; t += stride) {
        int i, j, k;
        const int c = lv_cell(F, t, i, j, k);
        if (F.code[c] != 0) prolong_one(F, c, Cl, omega, i, j, k);
    }
}

// Codes of the interior cells of a dense level from its labels.
__device__ void op_codes(const MgLevel& L, int t0, int stride) {
    const int n = L.W * L.H * L.D;
    for (int t = t0; t < n; t += stride) {
        int i, j, k;
        const int c = lv_cell(L, t, i, j, k);
        L.code[c] = L.lab[c] == FLUID ? uint8_t(1 + lv_diag(L, c)) : uint8_t(0);
    }
}

// Coarse label of cell t of level Cl, with Dirichlet priority: AIR if any
// child is AIR, else FLUID if any child is FLUID, else SOLID.
__device__ __forceinline__ void coarsen_cell(const MgLevel& F, const MgLevel& Cl, int t) {
    int I, J, K;
    const int cc = lv_cell(Cl, t, I, J, K);
    bool air = false, fluid = false;
    for (int c3 = 0; c3 < 2; ++c3)
        for (int b3 = 0; b3 < 2; ++b3)
            for (int a3 = 0; a3 < 2; ++a3) {
                const int i = 2 * I + a3, j = 2 * J + b3, k = 2 * K + c3;
                if (i >= F.W || j >= F.H || k >= F.D) continue;
                const uint8_t l = F.lab[lv_index(F, i, j, k)];
                air |= l == AIR;
                fluid |= l == FLUID;
            }
    Cl.lab[cc] = air ? AIR : (fluid ? FLUID : SOLID);
}

// ---- the block stage: levels [G, L) solved by each block on its own copy ----
// Shared-memory form.  Per level: x and b as FP32 padded grids; code (FLUID:
// 1 + diagonal, else 0) as bytes; ent, the level's FLUID cells (red ones from
// the front, black ones from the back; padded index | parent's padded index
// on the next level << 16) and kid (first child's padded index on the level
// above).  Built once per solve at kernel start, the labels in x's place;
// afterwards each operation walks a FLUID list (no index decoding, no label
// tests).  Only FLUID cells are written, so every other cell stays zero.
struct BlkLevel {
    MgLevel m;            // dims, strides and the x, b, lab pointers
    uint8_t* code;
    uint32_t* ent;
    uint16_t* kid;
    int x, b, ocode;      // where x, b (floats) and code (bytes) start in mg_smem
    int oent, okid;       // ... and the entries (words, half-words)
    int cells;            // interior cells
    int nred, nblack;     // FLUID cells of each colour
};

__host__ __device__ __forceinline__ int mg_cells(const MgLevel& L) { return L.W * L.H * L.D; }
// Bytes of the block levels [G, L): every level's two FP32 grids (padded cells
// rounded up to 4), then the entries and, below level G, kid (cells rounded up
// to 4 and 8), then the codes (padded cells rounded up to 16).  The same walk
// sizes the launch and places the arrays (block_levels_init).
__host__ __device__ __forceinline__ int mg_smem_bytes(const MgLevel* lv, int G, int L) {
    int by = 0;
    for (int l = G; l < L; ++l) {
        by += 8 * ((npad(lv[l]) + 3) & ~3) + 4 * ((mg_cells(lv[l]) + 3) & ~3) + ((npad(lv[l]) + 15) & ~15);
        if (l > G) by += 2 * ((mg_cells(lv[l]) + 7) & ~7);
    }
    return by;
}

extern __shared__ __align__(16) unsigned char mg_smem[];
__shared__ BlkLevel s_lv[MG_MAX_LEVELS];  // the block levels
__shared__ int s_levels, s_tiny;          // one past the deepest level with FLUID cells; first level for one warp

// Each block at kernel start.  Sets the number of levels that carry FLUID
// cells (at least G + 1): the deepest of them is the cycle's coarsest level.
__device__ void block_levels_init(const MgArgs& a) {
    const int G = a.G, L = a.L, t0 = threadIdx.x, st = blockDim.x;
    BlkLevel* S = s_lv;
    if (t0 == 0) {
        int at = 0;  // bytes
        for (int l = G; l < L; ++l) {
            const int n4 = (npad(a.lv[l]) + 3) & ~3;
            S[l].m = a.lv[l];
            S[l].x = at / 4; S[l].b = at / 4 + n4;
            S[l].m.x = reinterpret_cast<float*>(mg_smem + at);
            S[l].m.b = S[l].m.x + n4;
            S[l].m.lab = mg_smem + at;
            at += 8 * n4;
        }
        for (int l = G; l < L; ++l) {
            S[l].ent = reinterpret_cast<uint32_t*>(mg_smem + at);
            S[l].oent = at / 4;
            at += 4 * ((mg_cells(a.lv[l]) + 3) & ~3);
        }
        for (int l = G; l < L; ++l) {
            S[l].kid = reinterpret_cast<uint16_t*>(mg_smem + at);
            S[l].okid = at / 2;
            if (l > G) at += 2 * ((mg_cells(a.lv[l]) + 7) & ~7);
        }
        for (int l = G; l < L; ++l) {
            S[l].code = S[l].m.code = mg_smem + at;
            S[l].ocode = at;
            at += (npad(a.lv[l]) + 15) & ~15;
            S[l].cells = mg_cells(a.lv[l]);
            S[l].nred = S[l].nblack = 0;
        }
    }
    uint4* z = reinterpret_cast<uint4*>(mg_smem);
    for (int i = t0; i < a.smem / 16; i += st) z[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    {
        // whole vectors (the grid and its copy are allocated up to a multiple of 16 bytes)
        const uint4* src = reinterpret_cast<const uint4*>(a.lv[G].lab);
        uint4* dst = reinterpret_cast<uint4*>(S[G].m.lab);
        for (int c = t0; c < (npad(a.lv[G]) + 15) / 16; c += st) dst[c] = src[c];
    }
    __syncthreads();
    for (int l = G + 1; l < L; ++l) {
        for (int t = t0; t < S[l].cells; t += st) coarsen_cell(S[l - 1].m, S[l].m, t);
        __syncthreads();
    }
    for (int l = G; l < L; ++l) {
        BlkLevel& B = S[l];
        // (every lane of a warp takes part: one atomic per warp and colour)
        for (int base = 0; base < B.cells; base += st) {
            const int t = base + t0;
            int i = 0, j = 0, k = 0;
            const int c = lv_cell(B.m, min(t, B.cells - 1), i, j, k);
            const bool fl = t < B.cells && B.m.lab[c] == FLUID, black = ((i + j + k) & 1) != 0;
            const unsigned mr = __ballot_sync(0xffffffffu, fl && !black), mb = __ballot_sync(0xffffffffu, fl && black);
            const int lane = t0 & 31;
            int at = 0;
            if (lane == 0 && mr) at = atomicAdd(&B.nred, __popc(mr));
            if (lane == 1 && mb) at = atomicAdd(&B.nblack, __popc(mb));
            const int r0 = __shfl_sync(0xffffffffu, at, 0), b0 = __shfl_sync(0xffffffffu, at, 1);
            if (!fl) continue;
            B.code[c] = uint8_t(1 + lv_diag(B.m, c));
            const unsigned below = (1u << lane) - 1u;
            const int slot = black ? B.cells - 1 - (b0 + __popc(mb & below)) : r0 + __popc(mr & below);
            const int pc = l + 1 < L ? lv_index(S[l + 1].m, i >> 1, j >> 1, k >> 1) : 0;
            B.ent[slot] = uint32_t(c) | (uint32_t(pc) << 16);
            if (l > G) B.kid[slot] = uint16_t(lv_index(S[l - 1].m, 2 * i, 2 * j, 2 * k));
        }
    }
    __syncthreads();
    for (int l = G; l < L; ++l)  // x again
        for (int c = t0; c < (npad(S[l].m) + 3) / 4; c += st) S[l].m.x[c] = 0.0f;
    if (t0 == 0) {
        int n = G + 1;
        for (int l = G; l < L; ++l)
            if (S[l].nred + S[l].nblack > 0) n = l + 1;
        s_levels = n;
        s_tiny = n;
        while (s_tiny > G + 1 && max(S[s_tiny - 1].nred, S[s_tiny - 1].nblack) <= 32) --s_tiny;
    }
    __syncthreads();
}

// The stage's operations, by the whole block or (WARP) by its first warp.  All
// addresses are offsets into mg_smem, so that its loads are shared-memory loads.
template <bool WARP>
__device__ __forceinline__ void bl_sync() {
    if (WARP) __syncwarp();
    else __syncthreads();
}
template <bool WARP>
__device__ __forceinline__ int bl_stride() { return WARP ? 32 : MG_THREADS; }
__device__ __forceinline__ float* bl_f() { return reinterpret_cast<float*>(mg_smem); }
__device__ __forceinline__ const uint32_t* bl_w() { return reinterpret_cast<const uint32_t*>(mg_smem); }

// Slot of the t-th FLUID cell of level B (red ones first).
__device__ __forceinline__ int bl_slot(const BlkLevel& B, int t) {
    return t < B.nred ? t : B.cells - B.nblack + (t - B.nred);
}
// One cell, with what its updates need; c < 0: none.
struct BlkCell {
    int c, d;  // d: code
    float x, b;
};
__device__ __forceinline__ BlkCell bl_cell(const BlkLevel& B, int color, int t) {
    BlkCell q{-1, 0, 0.0f, 0.0f};
    if (t < (color == 0 ? B.nred : B.nblack)) {
        q.c = int(bl_w()[B.oent + (color == 0 ? t : B.cells - B.nblack + t)] & 0xFFFFu);
        q.x = bl_f()[B.x + q.c];
        q.b = bl_f()[B.b + q.c];
        q.d = mg_smem[B.ocode + q.c];
    }
    return q;
}
__device__ __forceinline__ float bl_nbsum(int at, int sy, int sz) {
    const float* x = bl_f() + at;
    return (x[1] + x[-1]) + (x[sy] + x[-sy]) + (x[sz] + x[-sz]);
}
// n Gauss-Seidel sweeps of alternating colours, black first.  Up to a cell of
// each colour per thread, those cells stay in registers over all sweeps; more
// are read again in each.
template <bool WARP>
__device__ __noinline__ void bl_smooth(int l, int n) {
    const BlkLevel& B = s_lv[l];
    const int t0 = threadIdx.x, st = bl_stride<WARP>(), X = B.x, sy = B.m.sy, sz = B.m.sz;
    auto update = [&](BlkCell& q) {
        q.x = gs_value(q.x, q.b, bl_nbsum(X + q.c, sy, sz), q.d, MG_SORC);
        bl_f()[X + q.c] = q.x;
    };
    if (WARP || max(B.nred, B.nblack) <= st) {
        BlkCell r = bl_cell(B, 0, t0), k = bl_cell(B, 1, t0);
#pragma unroll 1
        for (int e = 0; e < n; ++e) {
            if (e & 1) {
                if (r.c >= 0) update(r);
            } else {
                if (k.c >= 0) update(k);
            }
            bl_sync<WARP>();
        }
    } else {
        for (int e = 0; e < n; ++e) {
            const int color = (e & 1) ^ 1, m = color == 0 ? B.nred : B.nblack;
            for (int t = t0; t < m; t += st) {
                BlkCell q = bl_cell(B, color, t);
                update(q);
            }
            bl_sync<WARP>();
        }
    }
}
// Restriction of level l into l + 1 fused with that level's first sweep: b =
// scale * (sum of the red FLUID children's residuals; after a black sweep the
// black ones vanish), x = b/d on red cells, 0 on black ones.  The first child
// of a cell has even coordinates, so it and its three diagonal neighbours are
// the red ones.
template <bool WARP>
__device__ __noinline__ void bl_restrict(int l, float scale) {
    const BlkLevel &F = s_lv[l], &C = s_lv[l + 1];
    const int n = C.nred + C.nblack, sy = F.m.sy, sz = F.m.sz;
    const int off[4] = {0, sy + 1, sz + 1, sz + sy};
    for (int t = threadIdx.x; t < n; t += bl_stride<WARP>()) {
        const int slot = bl_slot(C, t);
        const int cc = int(bl_w()[C.oent + slot] & 0xFFFFu);
        const int f = reinterpret_cast<const uint16_t*>(mg_smem)[C.okid + slot];
        float s = 0.0f;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const int c = f + off[m], d = mg_smem[F.ocode + c];
            if (d > 0) s += bl_f()[F.b + c] - (float(d - 1) * bl_f()[F.x + c] - bl_nbsum(F.x + c, sy, sz));
        }
        s *= scale;
        bl_f()[C.b + cc] = s;
        bl_f()[C.x + cc] = t < C.nred ? gs_value(0.0f, s, 0.0f, mg_smem[C.ocode + cc], MG_SORC) : 0.0f;
    }
    bl_sync<WARP>();
}
// Prolongation: every FLUID cell of level l adds omega * its parent's x when the
// parent is FLUID (the parent level's red cells are already swept).
template <bool WARP>
__device__ __noinline__ void bl_prolong(int l, float omega) {
    const BlkLevel &F = s_lv[l], &C = s_lv[l + 1];
    const int n = F.nred + F.nblack;
    for (int t = threadIdx.x; t < n; t += bl_stride<WARP>()) {
        const uint32_t e = bl_w()[F.oent + bl_slot(F, t)];
        const int c = int(e & 0xFFFFu), pc = int(e >> 16);
        if (mg_smem[C.ocode + pc] > 0) bl_f()[F.x + c] += omega * bl_f()[C.x + pc];
    }
    bl_sync<WARP>();
}
// Levels [l, lend) going down, and [lbeg, l] coming up, whose last red sweep the
// stage leaves out on its first level, first.
template <bool WARP>
__device__ __forceinline__ void bl_down(const MgArgs& a, int l, int lend) {
#pragma unroll 1
    for (; l < lend; ++l) {
        bl_smooth<WARP>(l, 2 * a.nu_block - 1);
        bl_restrict<WARP>(l, a.rscale);
    }
}
template <bool WARP>
__device__ __forceinline__ void bl_up(const MgArgs& a, int l, int lbeg, int first) {
#pragma unroll 1
    for (; l >= lbeg; --l) {
        bl_prolong<WARP>(l, a.omega);
        bl_smooth<WARP>(l, 2 * a.nu_block - (l == first));
    }
}
template <bool WARP>
__device__ __forceinline__ void bl_coarsest(const MgArgs& a, int l, int first) {
    bl_smooth<WARP>(l, 2 * a.nu_coarse - 1);
    bl_smooth<WARP>(l, 2 * a.nu_coarse - (l == first));
}

// V-cycle over the shared-memory levels [l0, s_levels) by one block.  Level l0's
// first sweep is already done: the grid-wide restriction wrote its b and x,
// which are copied in.  The stage stops after level l0's last black sweep: the
// final red sweep of level l0 is the grid-wide prolongation into level l0 - 1,
// which recomputes it from this block's copy.  Some forty short steps, each
// waiting for the one before, so bound by a step's latency: registers over a
// level's sweeps, shared-memory addresses, and one warp without block barriers
// on the levels of at most 32 cells a colour (s_tiny on).  With the prolongation
// and the barrier after it, 8.8 us a cycle for 64 x 64 and 9.9 for 128^3, against
// 13.1 and 13.4 with a list walk per sweep, residuals stored before they were
// summed, and block barriers throughout.
__device__ __noinline__ void block_vcycle_smem(const MgArgs& a, int l0) {
    const BlkLevel& B0 = s_lv[l0];
    const MgLevel& G0 = a.lv[l0];
    for (int t = threadIdx.x; t < B0.nred + B0.nblack; t += MG_THREADS) {
        const int c = int(bl_w()[B0.oent + bl_slot(B0, t)] & 0xFFFFu);
        bl_f()[B0.b + c] = G0.b[c];
        bl_f()[B0.x + c] = G0.x[c];
    }
    __syncthreads();
    const int lc = s_levels - 1, lt = s_tiny, lb = min(lt, lc);
    bl_down<false>(a, l0, lb);
    if (lt > lc) {
        bl_coarsest<false>(a, lc, l0);
    } else {
        if (threadIdx.x < 32) {
            bl_down<true>(a, lt, lc);
            bl_coarsest<true>(a, lc, l0);
            bl_up<true>(a, lc - 1, lt, l0);
        }
        __syncthreads();
    }
    bl_up<false>(a, lb - 1, l0, l0);
    // the prolongation that follows reads level l0 from this block's copy
}

// Global-memory form (the block levels do not fit in shared memory, or the
// hierarchy has one level): V-cycle over levels [l0, L) of a.lv by block 0.
// Level l0's first sweep is already done (fused into the step that wrote its
// right-hand side).  With l0 > 0 the stage stops after level l0's last black
// sweep: the final red sweep of level l0 is the grid-wide prolongation into
// level l0 - 1, which recomputes it.  With l0 == 0 it finishes level 0 itself.
__device__ __noinline__ void block_vcycle_global(const MgArgs& a, int l0) {
    const int t0 = threadIdx.x, st = blockDim.x;
    for (int l = l0; l < a.L - 1; ++l) {
        op_sweep(a.lv[l], 1, t0, st); __syncthreads();
        for (int e = 1; e < (l == 0 ? a.nu0 : a.nu_block); ++e) {
            op_sweep(a.lv[l], 0, t0, st); __syncthreads();
            op_sweep(a.lv[l], 1, t0, st); __syncthreads();
        }
        op_restrict_first(a.lv[l], a.lv[l + 1], a.rscale, t0, st); __syncthreads();
    }
    const int lc = a.L - 1;
    const MgLevel& C = a.lv[lc];
    op_sweep(C, 1, t0, st); __syncthreads();
    for (int it = 1; it < a.nu_coarse; ++it) {
        op_sweep(C, 0, t0, st); __syncthreads();
        op_sweep(C, 1, t0, st); __syncthreads();
    }
    for (int it = 0; it < a.nu_coarse; ++it) {
        op_sweep(C, 1, t0, st); __syncthreads();
        if (it + 1 < a.nu_coarse || lc == 0) {
            op_sweep(C, 0, t0, st); __syncthreads();
        } else if (lc > l0) {
            op_prolong_red(a.lv[lc - 1], C, a.omega, t0, st); __syncthreads();
        }
    }
    for (int l = lc - 1; l >= l0; --l) {
        for (int e = 1; e < (l == 0 ? a.nu0 : a.nu_block); ++e) {
            op_sweep(a.lv[l], 1, t0, st); __syncthreads();
            op_sweep(a.lv[l], 0, t0, st); __syncthreads();
        }
        op_sweep(a.lv[l], 1, t0, st); __syncthreads();
        if (l == 0) {
            op_sweep(a.lv[0], 0, t0, st); __syncthreads();
        } else if (l > l0) {
            op_prolong_red(a.lv[l - 1], a.lv[l], a.omega, t0, st); __syncthreads();
        }
    }
}

// The grid-wide operations of the cycle.  Functions of their own, not inlined
// at each of their places in it: the cycle's code then stays in the instruction
// cache.
__device__ __noinline__ void grid_sweep(const MgArgs& a, int l, int color) {
    const float w = l == 0 ? MG_SOR : MG_SORC;
    const MgLevel& L = a.lv[l];
    for_quads(a, l, [&](const Quad& Q, int) { sweep_quad(L, Q, color, w); });
}
__device__ __noinline__ void grid_restrict(const MgArgs& a, int l, int G) {
    const int t0 = blockIdx.x * MG_THREADS + threadIdx.x, st = gridDim.x * MG_THREADS;
    if (l + 1 < G) restrict_quads(a.lv[l], a.lv[l + 1], a.rscale, a.q[l + 1], s_nq[l + 1], t0, st);
    else op_restrict_first(a.lv[l], a.lv[l + 1], a.rscale, t0, st);
}
__device__ __noinline__ void grid_prolong(const MgArgs& a, int lf, const MgLevel* Cp) {
    const MgLevel& F = a.lv[lf];
    const MgLevel C = *Cp;
    for_quads(a, lf, [&](const Quad& Q, int) { prolong_quad(F, C, a.omega, Q); });
}

// z = V-cycle(r) with r = lv[0].b, z = lv[0].x.  The caller has already done
// the first (red) sweep of level 0 (z = w b/d on red FLUID cells, 0 on black
// ones) and a grid barrier since.  Ends with a grid barrier; returns false if
// a barrier timed out.  Grid-wide levels take four barriers each with one
// sweep pair (level 0 two more per extra pair): black sweep, restriction (with
// the next level's first sweep), black sweep, red sweep (with the
// prolongation into the finer level).
__device__ bool vcycle(const MgArgs& a) {
    const unsigned nb = gridDim.x;
    const int G = min(a.G, a.L - 1);
    auto sweep = [&](int l, int color) {
        grid_sweep(a, l, color);
        return grid_barrier(a.bar, nb, a.status);
    };
#pragma unroll 1
    for (int l = 0; l < G; ++l) {
        // pre-smoothing (red, black)^nu (nu = nu0 on level 0, else nu_grid); the
        // first red sweep is fused upstream
        const int n = 2 * (l == 0 ? a.nu0 : a.nu_grid) - 1;
#pragma unroll 1
        for (int e = 0; e < n; ++e)
            if (!sweep(l, (e & 1) ^ 1)) return false;
        grid_restrict(a, l, G);
        if (!grid_barrier(a.bar, nb, a.status)) return false;
    }
    if (a.smem) {
        // Every block runs the block levels on its own shared-memory copy (the
        // same arithmetic, so the same bits) and prolongs from that copy: no
        // grid barrier and no copy-out between the stage and the prolongation.
        block_vcycle_smem(a, G);
        grid_prolong(a, G - 1, &s_lv[G].m);
        if (!grid_barrier(a.bar, nb, a.status)) return false;
    } else {
        if (blockIdx.x == 0) block_vcycle_global(a, G);
        if (!grid_barrier(a.bar, nb, a.status)) return false;
        if (G > 0) {  // level G's last red sweep, fused with its prolongation into level G - 1
            grid_prolong(a, G - 1, &a.lv[G]);
            if (!grid_barrier(a.bar, nb, a.status)) return false;
        }
    }
#pragma unroll 1
    for (int l = G - 1; l >= 0; --l) {
        // post-smoothing (black, red)^nu, the reverse of the pre-smoothing; the
        // first red sweep was fused with the prolongation, the last red sweep
        // with the next prolongation
        const int n = 2 * (l == 0 ? a.nu0 : a.nu_grid) - 1;
#pragma unroll 1
        for (int e = 0; e < n; ++e)
            if (!sweep(l, (e & 1) ^ 1)) return false;
        if (l == 0) grid_sweep(a, 0, 0);
        else grid_prolong(a, l - 1, &a.lv[l]);
        if (!grid_barrier(a.bar, nb, a.status)) return false;
    }
    return true;
}

// Level-0 first sweep value of one cell with code dc: b/d on red FLUID cells, else 0.
__device__ __forceinline__ float first_red0(float b, int dc, bool red) {
    return red ? gs_value(0.0f, b, 0.0f, dc, MG_SOR) : 0.0f;
}
// b0 and the first sweep's z of one quad from its residual.
__device__ __forceinline__ void start_cycle(const MgLevel& F, int c, uint32_t k, float4 b) {
    const bool odd = ((k >> 7) & 1u) != 0u;
    *reinterpret_cast<float4*>(F.b + c) = b;
    *reinterpret_cast<float4*>(F.x + c) =
        make_float4(first_red0(b.x, code_at(k, 0), !odd), first_red0(b.y, code_at(k, 1), odd),
                    first_red0(b.z, code_at(k, 2), !odd), first_red0(b.w, code_at(k, 3), odd));
}

struct D4 {
    double v[4];
};
__device__ __forceinline__ D4 ldq(const double2* p, int cap, int n) {
    const double2 a = p[n], b = p[cap + n];
    return D4{{a.x, a.y, b.x, b.y}};
}
__device__ __forceinline__ void stq(double2* p, int cap, int n, const D4& d) {
    p[n] = make_double2(d.v[0], d.v[1]);
    p[cap + n] = make_double2(d.v[2], d.v[3]);
}
// A z at the four cells of a quad exactly (FP32 values summed in FP64), 0 off the fluid; zc: z itself.
__device__ __forceinline__ D4 apply_quad(const MgLevel& F, int c, uint32_t k, float4& zc) {
    const float* z = F.x + c;
    zc = ld4(z);
    const float4 yp = ld4(z + F.sy), ym = ld4(z - F.sy), zp = ld4(z + F.sz), zm = ld4(z - F.sz);
    const float xl = z[-1], xr = z[4];
    auto at = [&](int e, float v, float r, float l, float a, float b, float f, float g) {
        const int dc = code_at(k, e);
        const double s = (double(r) + double(l)) + (double(a) + double(b)) + (double(f) + double(g));
        return dc > 0 ? double(dc - 1) * double(v) - s : 0.0;
    };
    return D4{{at(0, zc.x, zc.y, xl, yp.x, ym.x, zp.x, zm.x), at(1, zc.y, zc.z, zc.x, yp.y, ym.y, zp.y, zm.y),
               at(2, zc.z, zc.w, zc.y, yp.z, ym.z, zp.z, zm.z), at(3, zc.w, xr, zc.z, yp.w, ym.w, zp.w, zm.w)}};
}

__global__ void __launch_bounds__(MG_THREADS, 1) k_pcg_mg(const __grid_constant__ MgArgs a) {
    note_solve(&a.out->t_begin);
    const int nb = int(gridDim.x);
    const int t0 = blockIdx.x * MG_THREADS + threadIdx.x, st = nb * MG_THREADS;
    const MgLevel& F = a.lv[0];
    if (threadIdx.x < MG_MAX_LEVELS) s_nq[threadIdx.x] = a.nq[threadIdx.x];
    if (threadIdx.x < 8) s_rcp[threadIdx.x] = threadIdx.x > 1 ? 1.0f / float(threadIdx.x - 1) : 0.0f;
    __syncthreads();
    const int nq = s_nq[0], cap = a.cap, G = min(a.G, a.L - 1);
    const int4* list = a.q[0];
    int red = 0;  // reductions so far (the partial buffers alternate)
    auto sum = [&](double (&v)[3]) {
        return grid_reduce(v, a.part + (red++ & 1) * 3 * nb, a.bar, nb, a.status);
    };
    if (a.smem) block_levels_init(a);  // every block: its own copy

    // level codes: the listed quads of the grid-wide levels (zero elsewhere,
    // restored at the end), the other levels over all their cells
    for (int l = 1; l < G; ++l) codes_quads(a.lv[l], a.q[l], s_nq[l], t0, st);
    for (int l = max(G, 1); l <= (a.smem ? G : a.L - 1); ++l) op_codes(a.lv[l], t0, st);
    fill_slots(a, 0, 1, t0, st);
    // r = rhs, the level-0 codes, and the guess (kept as the FP32 values z) or
    // the V-cycle's right-hand side and first sweep
    double v[3] = {0.0, 0.0, 0.0};
    for (int n = t0; n < nq; n += st) {
        const int4 e = list[n];
        const uint32_t k = uint32_t(e.y);
        const float4 bf = a.rhs[n];
        const D4 r{{double(bf.x), double(bf.y), double(bf.z), double(bf.w)}};
        *reinterpret_cast<uint32_t*>(F.code + e.x) = k & QUAD_CODES;
        stq(a.r, cap, n, r);
#pragma unroll
        for (int m = 0; m < 4; ++m) v[0] += r.v[m] * r.v[m];
        if (a.guess) {
            float g[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                g[m] = code_at(k, m) ? a.guess[e.w + m] : 0.0f;
                if (!a.guess_dir && !isfinite(g[m])) g[m] = 0.0f;
            }
            *reinterpret_cast<float4*>(F.x + e.x) = make_float4(g[0], g[1], g[2], g[3]);
        } else {
            stq(a.xs, cap, n, D4{{0.0, 0.0, 0.0, 0.0}});
            start_cycle(F, e.x, k, bf);
        }
    }
    // With a guess g the solve's first flexible-CG step uses g as its
    // preconditioned residual: z0 = g, p0 = z0, alpha0 = (r0, z0) / (p0, A p0)
    // -- the energy-optimal scaling: the A-norm error of alpha0 g is never
    // above that of x = 0 -- and x1 = alpha0 g.  For the network's
    // guess N(b) (the learned preconditioner), p0, A p0, gamma0 = (r0, z0) and
    // (p0, A p0) stay in the recurrence, so the next direction (from the
    // V-cycle) is made A-conjugate to p0 by the Polak-Ribiere beta.  The
    // previous step's pressure restarts the recurrence instead: kept in it, it
    // cost iterations (11.2 against 10.8 per warm-started solve at 128^3).
    bool dir0 = false;
    double gam0 = 0.0, alpha0 = 0.0, den0 = 0.0;
    if (!sum(v)) return;
    fill_slots(a, 1, G, t0, st);
    const double bb = v[0];
    double rr = bb;
    if (a.guess) {
        v[0] = v[1] = v[2] = 0.0;
        for_quads(a, 0, [&](const Quad& Q, int n) {
            const int c = Q.c;
            const uint32_t k = Q.k;
            float4 g;
            const D4 s = apply_quad(F, c, k, g), r = ldq(a.r, cap, n);
            const double gd[4] = {double(g.x), double(g.y), double(g.z), double(g.w)};
            stq(a.s, cap, n, s);
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                v[0] += gd[m] * r.v[m];
                v[1] += gd[m] * s.v[m];
            }
        });
        if (!sum(v)) return;
        const double alpha = (v[1] > 0.0 && isfinite(v[0] / v[1])) ? v[0] / v[1] : 0.0;
        dir0 = alpha != 0.0 && a.guess_dir;
        gam0 = v[0]; alpha0 = alpha; den0 = v[1];
        v[0] = v[1] = v[2] = 0.0;
        for_quads(a, 0, [&](const Quad& Q, int n) {
            const int c = Q.c;
            const uint32_t k = Q.k;
            const float4 g = ld4(F.x + c);
            const D4 s = ldq(a.s, cap, n);
            D4 r = ldq(a.r, cap, n), x{{double(g.x), double(g.y), double(g.z), double(g.w)}};
            if (a.guess_dir) stq(a.p, cap, n, x);  // p0 = g; s holds A p0
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                x.v[m] *= alpha;
                r.v[m] = r.v[m] - alpha * s.v[m];
                v[0] += r.v[m] * r.v[m];
            }
            stq(a.xs, cap, n, x);
            stq(a.r, cap, n, r);
            start_cycle(F, c, k, make_float4(float(r.v[0]), float(r.v[1]), float(r.v[2]), float(r.v[3])));
        });
        if (!sum(v)) return;
        rr = v[0];
    }
    const double rr0 = rr;
    const double thr = a.tol * a.tol * bb;
    // Flexible preconditioned CG in the Chronopoulos-Gear form: after the
    // V-cycle one pass forms w = A z, gamma = (r, z), delta = (z, w) and
    // zeta = (z, s_old); one more updates p = z + beta p, s = w + beta s
    // (= A p), x += alpha p, r -= alpha s and starts the next cycle.  beta is
    // the Polak-Ribiere choice (z, r - r_old) / gamma_old = -alpha_old zeta /
    // gamma_old, and (p, A p) = delta + 2 beta zeta + beta^2 (p, A p)_old holds
    // for any beta, so alpha = gamma / (p, A p) needs no symmetry of the
    // V-cycle (over-relaxed smoothing makes it slightly non-symmetric).  Two
    // grid-wide passes per iteration besides the cycle.
    double gam = 0.0, gam_old = gam0, alpha_old = dir0 ? alpha0 : 1.0, den_old = dir0 ? den0 : 1.0;
    int it = 0, stt = DEV_OK;
    while (rr > thr && bb > 0.0) {
        if (it >= a.maxit) { stt = DEV_MAXIT; break; }
        if (!vcycle(a)) return;  // z = M^-1 r
        const bool coupled = it > 0 || dir0;  // a previous direction to conjugate against
        v[0] = v[1] = v[2] = 0.0;
        for_quads(a, 0, [&](const Quad& Q, int n) {
            const int c = Q.c;
            const uint32_t k = Q.k;
            float4 zf;
            const D4 r = ldq(a.r, cap, n);
            D4 s{{0.0, 0.0, 0.0, 0.0}};
            if (coupled) s = ldq(a.s, cap, n);
            const D4 w = apply_quad(F, c, k, zf);
            const double z[4] = {double(zf.x), double(zf.y), double(zf.z), double(zf.w)};
            stq(a.w, cap, n, w);
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                v[0] += r.v[m] * z[m];
                v[1] += z[m] * w.v[m];
                v[2] += z[m] * s.v[m];
            }
        });
        if (!sum(v)) return;
        gam = v[0];
        if (isnan(v[0]) || isnan(v[1]) || isnan(v[2])) { stt = DEV_NAN; break; }
        const double beta = coupled ? -alpha_old * v[2] / gam_old : 0.0;
        const double den = coupled ? v[1] + beta * (2.0 * v[2] + beta * den_old) : v[1];
        if (!(den > 0.0)) { stt = DEV_BREAKDOWN; break; }
        const double alpha = gam / den;
        v[0] = v[1] = v[2] = 0.0;
        for_quads(a, 0, [&](const Quad& Q, int n) {
            const int c = Q.c;
            const uint32_t k = Q.k;
            const float4 zf = ld4(F.x + c);
            const D4 w = ldq(a.w, cap, n);
            D4 x = ldq(a.xs, cap, n), r = ldq(a.r, cap, n);
            D4 p{{double(zf.x), double(zf.y), double(zf.z), double(zf.w)}}, s = w;
            if (coupled) {
                const D4 po = ldq(a.p, cap, n), so = ldq(a.s, cap, n);
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    p.v[m] = p.v[m] + beta * po.v[m];
                    s.v[m] = w.v[m] + beta * so.v[m];
                }
            }
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                x.v[m] = x.v[m] + alpha * p.v[m];
                r.v[m] = r.v[m] - alpha * s.v[m];
                v[0] += r.v[m] * r.v[m];
            }
            stq(a.p, cap, n, p);
            stq(a.s, cap, n, s);
            stq(a.xs, cap, n, x);
            stq(a.r, cap, n, r);
            start_cycle(F, c, k, make_float4(float(r.v[0]), float(r.v[1]), float(r.v[2]), float(r.v[3])));
        });
        if (!sum(v)) return;
        rr = v[0];
        ++it;
        if (isnan(rr)) { stt = DEV_NAN; break; }
        gam_old = gam;
        alpha_old = alpha;
        den_old = den;
    }
    // The true residual of the FP64 solution, ||rhs - A x||^2 and ||rhs||^2,
    // then the dense solution; zero the work grids at the listed quads so the
    // next solve starts from zero whatever cells are fluid.
    for_quads(a, 0, [&](const Quad& Q, int n) {
        const int c = Q.c;
        const D4 x = ldq(a.xs, cap, n);
        double2* X = reinterpret_cast<double2*>(a.xd + c);
        X[0] = make_double2(x.v[0], x.v[1]);
        X[1] = make_double2(x.v[2], x.v[3]);
    });
    if (!grid_barrier(a.bar, unsigned(nb), a.status)) return;
    v[0] = v[1] = v[2] = 0.0;
    for_quads(a, 0, [&](const Quad& Q, int n) {
        const int c = Q.c;
        const uint32_t k = Q.k;
        const float4 bf = a.rhs[n];
        const float b[4] = {bf.x, bf.y, bf.z, bf.w};
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const int dc = code_at(k, m);
            if (dc == 0) continue;
            const double* x = a.xd + c + m;
            const double ax = double(dc - 1) * x[0] -
                              ((x[1] + x[-1]) + (x[F.sy] + x[-F.sy]) + (x[F.sz] + x[-F.sz]));
            const double bv = double(b[m]), e = bv - ax;
            v[0] += e * e;
            v[1] += bv * bv;
        }
    });
    if (!sum(v)) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) { a.red[0] = v[0]; a.red[1] = v[1]; }
    for (int n = t0; n < nq; n += st) {
        const int4 e = list[n];
        const uint32_t k = uint32_t(e.y);
        const D4 x = ldq(a.xs, cap, n);
#pragma unroll
        for (int m = 0; m < 4; ++m)
            if (code_at(k, m)) a.pout[e.w + m] = float(x.v[m]);
        double2* X = reinterpret_cast<double2*>(a.xd + e.x);
        X[0] = X[1] = make_double2(0.0, 0.0);
        *reinterpret_cast<float4*>(F.x + e.x) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        *reinterpret_cast<uint32_t*>(F.code + e.x) = 0u;
    }
    for (int l = 1; l < G; ++l)
        for (int n = t0; n < s_nq[l]; n += st) {
            const int c = a.q[l][n].x;
            *reinterpret_cast<float4*>(a.lv[l].x + c) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            *reinterpret_cast<uint32_t*>(a.lv[l].code + c) = 0u;
        }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.out->iters = it;
        atomicCAS(a.status, DEV_OK, stt);
        a.out->rr = rr;
        a.out->bb = bb;
        a.out->rz = gam;
        a.out->rr0 = rr0;
        note_solve(&a.out->t_end);
    }
}

// Labels of level Cl from the finer level's, with Dirichlet priority (AIR if
// any child AIR, else FLUID if any child FLUID, else SOLID; BODY, like SOLID,
// is neither), one thread per quad, and the list of the quads that hold a
// FLUID cell (one atomic per block, in no fixed order: every use of the list
// treats its quads independently).  raw: the finer level is the cell labels
// themselves (W x H x D, no padding).  *nlist must be zero before the launch.
constexpr int COARSEN_THREADS = 256;
template <bool RAW>
__global__ void __launch_bounds__(COARSEN_THREADS) k_coarsen(const uint8_t* __restrict__ raw, MgLevel F, MgLevel Cl,
                                                             MgLevel next, int4* __restrict__ list,
                                                             int* __restrict__ nlist) {
    const int nqr = (Cl.W + 3) >> 2;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = t < nqr * Cl.H * Cl.D;
    bool listed = false;
    int4 entry = make_int4(0, 0, 0, 0);
    if (in) {
        const int r = t / nqr, Q = t - r * nqr, K = r / Cl.H, J = r - K * Cl.H;
        uint32_t air = 0, fluid = 0;  // a byte per coarse cell
#pragma unroll
        for (int c3 = 0; c3 < 2; ++c3)
#pragma unroll
            for (int b3 = 0; b3 < 2; ++b3) {
                const int j = 2 * J + b3, k = 2 * K + c3;
                if (j >= F.H || k >= F.D) continue;
                const uint8_t* row = RAW ? raw + int64_t(8 * Q) + int64_t(j) * F.W + int64_t(k) * F.W * F.H
                                         : F.lab + lv_index(F, 8 * Q, j, k);
#pragma unroll
                for (int m = 0; m < 8; ++m) {
                    // (a padded row reads its zero gap, SOLID, beyond the last cell)
                    if (8 * Q + m >= F.W) break;
                    const uint8_t l = row[m];
                    if (l == AIR) air |= 1u << (8 * (m >> 1));
                    if (l == FLUID) fluid |= 1u << (8 * (m >> 1));
                }
            }
        uint32_t lab = 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const uint32_t m = 1u << (8 * e);
            const uint32_t v = (air & m) ? uint32_t(AIR) : (fluid & m) ? uint32_t(FLUID) : uint32_t(SOLID);
            lab |= v << (8 * e);
            listed |= v == uint32_t(FLUID);
        }
        const int cc = lv_index(Cl, 4 * Q, J, K);
        *reinterpret_cast<uint32_t*>(Cl.lab + cc) = lab;
        uint32_t par = ((J + K) & 1) ? QUAD_ODD : 0u;
        if (((J >> 1) + (K >> 1)) & 1) par |= QUAD_PARENT_ODD;
        if (2 * K + 1 < F.D) par |= QUAD_Z;
        entry = make_int4(cc, int(par), next.W ? lv_index(next, 2 * Q, J >> 1, K >> 1) : 0,
                          lv_index(F, 8 * Q, 2 * J, 2 * K));
    }
    if (!list) return;  // uniform across the block
    __shared__ int s_off[COARSEN_THREADS / 32];
    __shared__ int s_base;
    const unsigned m = __ballot_sync(0xffffffffu, listed);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) s_off[wid] = __popc(m);
    __syncthreads();
    if (threadIdx.x == 0) {
        int tot = 0;
        for (int w = 0; w < COARSEN_THREADS / 32; ++w) { const int c = s_off[w]; s_off[w] = tot; tot += c; }
        s_base = tot > 0 ? atomicAdd(nlist, tot) : 0;
    }
    __syncthreads();
    if (listed) list[s_base + s_off[wid] + __popc(m & ((1u << lane) - 1u))] = entry;
}

}  // namespace

int mg_npad(const MgLevel& L) { return (npad(L) + 15) & ~15; }

int mg_levels_for(int W, int H, int D, MgLevel* lv) {
    int L = 0;
    int w = W, h = H, d = D;
    while (L < MG_MAX_LEVELS) {
        lv[L].W = w; lv[L].H = h; lv[L].D = d;
        lv[L].sy = ((w + 3) & ~3) + MG_OX;
        lv[L].sz = lv[L].sy * (h + 2);
        ++L;
        if (w <= 2 && h <= 2 && d <= 2) break;
        w = (w + 1) / 2; h = (h + 1) / 2; d = (d + 1) / 2;
    }
    return L;
}

int mg_max_blocks() {
    static DeviceMemo memo;
    return memo.get([](int dev) {
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaFuncSetAttribute(k_pcg_mg, cudaFuncAttributeMaxDynamicSharedMemorySize, MG_SMEM_BUDGET);
        return sms;
    });
}

int mg_split(const MgLevel* lv, int L, int* smem_bytes) {
    *smem_bytes = 0;
    if (L <= 1) return 0;
    int G = 1;  // level 0 is always swept grid-wide on its list
    for (int l = 0; l < L; ++l)
        if (int64_t(lv[l].W) * lv[l].H * lv[l].D > MG_BLOCK_CELLS) G = std::max(G, l + 1);
    for (G = std::min(G, L - 1); G < L; ++G) {
        const int b = mg_smem_bytes(lv, G, L);
        // the FLUID lists hold padded indices in 16 bits
        if (b <= MG_SMEM_BUDGET && npad(lv[G]) <= 65535) { *smem_bytes = b; return G; }
    }
    return L - 1;  // not even the coarsest level fits: the block levels stay in global memory
}

int launch_mg_setup(const uint8_t* labels, const MgBufs& m, cudaStream_t st) {
    int smem = 0;
    const int G = mg_split(m.lv, m.L, &smem);
    const int last = smem ? G : m.L - 1;  // deeper shared-memory levels: coarsened by the solver kernel
    for (int l = 1; l <= last; ++l) {
        const MgLevel& C = m.lv[l];
        const int n = ((C.W + 3) >> 2) * C.H * C.D, nb = (n + COARSEN_THREADS - 1) / COARSEN_THREADS;
        const MgLevel next = l + 1 < m.L ? m.lv[l + 1] : MgLevel{};
        int4* list = l < G ? m.q[l] : nullptr;
        if (l == 1) k_coarsen<true><<<nb, COARSEN_THREADS, 0, st>>>(labels, m.lv[0], C, next, list, m.nq + l);
        else k_coarsen<false><<<nb, COARSEN_THREADS, 0, st>>>(nullptr, m.lv[l - 1], C, next, list, m.nq + l);
    }
    return last;
}

int launch_pcg_mg(Dims g, PressureBufs& pb, const MgBufs& m, double tol, int maxit, const float* guess, int guess_dir,
                  int nu0, float* pout, cudaStream_t st) {
    // One block per 4096 cells, at most one per SM: a small grid waits at
    // cheaper barriers (one block: __syncthreads).
    const int64_t want = (g.nc() + 4095) / 4096;
    const int nb = int(std::max<int64_t>(1, std::min<int64_t>(mg_max_blocks(), want)));
    MgArgs a{};
    a.L = m.L;
    a.G = mg_split(m.lv, m.L, &a.smem);
    for (int l = 0; l < m.L; ++l) { a.lv[l] = m.lv[l]; a.q[l] = m.q[l]; }
    a.nq = m.nq;
    a.rscale = g.D > 1 ? 0.25f : 0.5f;
    // The piecewise-constant prolongation underestimates the coarse correction;
    // scaling it by 1.7 roughly halves the PCG iterations (29 -> 15 at 128^3,
    // 31 -> 14 at 256^2 in a float64 model of this V-cycle).  Any omega > 0
    // keeps the preconditioner symmetric; in that model PCG converged for
    // every omega up to 2 on dam-break, pool and random-box scenes.  With the
    // over-relaxed smoother, 1.8 was as fast as 1.9 on the dam break and
    // faster on random boxes (14 against 15 iterations); with two sweep pairs
    // on the block levels and SOR 1.2, 1.7 is best (1.9: 10.55, 2.0: 10.75
    // iterations per warm-started solve at 128^3).
    a.omega = MG_OMEGA;
    a.nu_coarse = MG_NU_COARSE;
    a.nu0 = std::max(1, nu0);
    a.nu_grid = MG_NU_GRID;
    a.nu_block = MG_NU_BLOCK;
    a.rhs = m.rhs;
    a.p = m.p; a.s = m.s; a.xs = m.xs; a.r = m.r; a.w = m.w;
    a.cap = m.cap;
    a.xd = m.xd;
    a.guess = guess; a.guess_dir = guess_dir;
    a.pout = pout;
    a.red = pb.red;
    a.part = pb.part; a.bar = pb.bar; a.status = &pb.out->status; a.out = pb.out;
    a.tol = tol; a.maxit = maxit;
    void* args[] = {&a};
    cudaError_t e =
        cudaLaunchCooperativeKernel((const void*)k_pcg_mg, dim3(nb), dim3(MG_THREADS), args, size_t(a.smem), st);
    return e == cudaSuccess ? 0 : int(e);
}

}  // namespace fp
