// kernels_pcg.cu -- the plain and the mixed-precision pressure solvers
// (FP_SOLVER_PCG, FP_SOLVER_PCG_MIXED and the refinement of
// FP_SOLVER_PCG_LEARNED_MIXED), each one cooperative launch per solve.
//
// Same system as the reference's cuDSS solve (FluidSolver3D.cu:1815-2062): the
// unit 7-point operator over FLUID cells, never stored: A d at a FLUID cell is
// diag d - the sum of d over its FLUID neighbours.
//
// Jacobi-preconditioned conjugate gradients in the Chronopoulos-Gear form:
//   s_i = w_i + b_i s_{i-1}; p_i = u_i + b_i p_{i-1}; x += a_i p_i;
//   r_{i+1} = r_i - a_i s_i; u = M^-1 r; w_{i+1} = A u_{i+1};
//   g = (r,u), d = (w,u); b = g_new/g; a = g_new/(d - b g_new/a_old).
// Vectors in T (FP64, or FP32 inside the refinement), the three sums always in
// FP64, reduced in a fixed order (grid_reduce).  Each CTA owns a contiguous
// range of the FLUID list, so the x and y neighbours of its cells mostly lie
// in the same CTA.  Two forms of the iteration, with the same arithmetic:
//
//   one cell per thread (cg_one): everything a cell owns stays in registers,
//     r, w and s go to padded grids that alternate between iterations, and
//     each thread recomputes its neighbours' r_{i+1} from them, so one grid
//     barrier per iteration both publishes the vectors and completes the
//     sums.  The neighbours' loads do not depend on the sums and overlap them.
//     Bound by latency: a barrier, an L2 round trip and the reduction.
//     3.4 us per FP64 iteration at 25,800 FLUID cells and 3.2 per FP32 one at
//     51,300 (6.3 and 5.4 when every vector came from memory each time and
//     the sums went through a two-level tree).
//   more cells (cg_many): a CTA's x, r, p, s and w live in its shared memory
//     (what does not fit, in global memory) and only u crosses CTAs, through
//     one padded grid: 6 neighbour loads per cell in place of 18 at the price
//     of a second barrier.  Recomputing neighbours is bound by those loads:
//     17.2 us per FP64 iteration at 625,000 FLUID cells and 12.1 per FP32 one
//     at 483,000, against 9.4 and 7.3 here, of which the two barriers take
//     about 3.4 us.
//
// The solution's FP64 residual, the dense pressure and the clean-up of the
// work grids (zero between solves, whatever cells were fluid) are part of the
// launch, and so is the whole refinement loop of the mixed solver.
#include <algorithm>

#include "device_memo.hpp"
#include "kernels.hpp"
#include "pcg_common.cuh"

namespace fp {

namespace {

// One CTA per SM of 512 threads with 128 registers each.  768 and 1024 threads
// run cg_many within 5 % of it either way (3.79 against 3.82-3.96 ms for the
// FP32 solve below) but cg_one spills (0.76 and 1.07 against 0.55 ms).
constexpr int PCG_THREADS = 512;
constexpr int PCG_UNR = 4;        // cells per thread whose loads are issued together
// Dynamic shared memory for the vectors of cg_many.
constexpr int PCG_SMEM = 200 * 1024;
template <class T>
constexpr int cell_bytes() { return 5 * int(sizeof(T)) + 5; }  // x, r, p, s, w, index and diagonal

__device__ __forceinline__ float fmaT(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fmaT(double a, double b, double c) { return __fma_rn(a, b, c); }

struct PcgArgs {
    int W, H, sy, sz;    // interior width and height, padded strides
    const int* nf;
    const int* fidx;     // padded dense index of the n-th FLUID cell
    const uint8_t* diag; // compact diagonal
    const float* b;      // compact right-hand side
    const float* x0;     // mixed: compact initial guess, or null
    float* bin;          // mixed: compact right-hand side of an inner solve
    void* R[2];          // padded grids of T, zero between solves
    void* Wv[2];
    void* S[2];
    void* invd;
    void* P;             // compact
    void* X;             // compact
    double* x64;         // mixed: compact FP64 iterate
    double* xd;          // padded FP64 iterate, zero between solves
    float* pout;         // dense W x H x D pressure
    double* red;         // [2] ||b - A x||^2, ||b||^2
    double* part;        // [2][3][nblocks]
    GridBar* bar;
    int* status;
    PcgOut* out;
    double tol;
    int maxit;
    int cap;             // cells per CTA in shared memory
};

// A CTA's share of the FLUID list and its place in the reductions.
struct Share {
    int nb, n0, m;  // CTAs, first cell, number of cells
    int red;        // reductions so far (the partial buffers alternate)
};
template <int N, class Mid>
__device__ __forceinline__ bool reduce(const PcgArgs& a, Share& h, double (&v)[N], Mid mid) {
    return grid_reduce(v, a.part + (h.red++ & 1) * 3 * h.nb, a.bar, h.nb, a.status, mid);
}
template <int N>
__device__ __forceinline__ bool reduce(const PcgArgs& a, Share& h, double (&v)[N]) {
    return reduce(a, h, v, [] {});
}

// The scalars of the recurrence, the same in every thread.
struct Cg {
    double gam, alpha, beta, rr, bb, thr;
    int it, st;
    // the first sums: alpha_0; false: stop
    __device__ __forceinline__ bool start(const double (&v)[3], double tol) {
        gam = v[0]; rr = bb = v[2];
        thr = tol * tol * bb;
        alpha = v[1] > 0.0 ? gam / v[1] : 0.0;
        beta = 0.0;
        it = 0;
        st = DEV_OK;
        if (bb > 0.0 && !(v[1] > 0.0)) st = isnan(v[1]) ? DEV_NAN : DEV_BREAKDOWN;
        return st == DEV_OK && rr > thr && bb > 0.0;
    }
    __device__ __forceinline__ bool capped(int maxit) {
        if (it < maxit) return false;
        st = DEV_MAXIT;
        return true;
    }
    // the sums after an update; false: stop
    __device__ __forceinline__ bool next(const double (&v)[3]) {
        ++it;
        rr = v[2];
        if (isnan(v[0]) || isnan(v[1]) || isnan(v[2])) { st = DEV_NAN; return false; }
        if (rr <= thr) return false;
        beta = v[0] / gam;
        const double den = v[1] - beta * v[0] / alpha;
        if (!(den > 0.0) || !(v[0] > 0.0)) { st = DEV_BREAKDOWN; return false; }
        alpha = v[0] / den;
        gam = v[0];
        return true;
    }
};

// Shared memory: cg_many's vectors, and 1/d of the diagonals d = 0..6 (0 for
// d = 0, a cell without neighbours) in both precisions.
extern __shared__ __align__(16) unsigned char pcg_smem[];
__shared__ double s_inv64[8];
__shared__ float s_inv32[8];
__device__ __forceinline__ double inv_of(int d, double) { return s_inv64[d]; }
__device__ __forceinline__ float inv_of(int d, float) { return s_inv32[d]; }

// CG of A x = rhs with at most one cell per thread; x to a.X.  Returns false
// if a barrier gave up.
template <class T>
__device__ bool cg_one(const PcgArgs& a, Share& h, const float* rhs, double tol, int maxit, Cg& cg) {
    const bool ok = int(threadIdx.x) < h.m;
    const int n = h.n0 + int(threadIdx.x);
    // an idle thread reads around interior cell (0,0,0): in bounds, its result dropped
    const int c = ok ? a.fidx[n] : 1 + a.sy + a.sz;
    const int dg = ok ? a.diag[n] : 0;
    const int offs[6] = {1, -1, a.sy, -a.sy, a.sz, -a.sz};
    T* const R0 = static_cast<T*>(a.R[0]);
    T* const invd = static_cast<T*>(a.invd);
    const T inv = inv_of(dg, T(0));
    T r = ok ? T(rhs[n]) : T(0), u = r * inv, s = T(0), p = T(0), x = T(0);
    if (ok) {
        R0[c] = r;
        invd[c] = inv;
        static_cast<T*>(a.S[0])[c] = T(0);
    }
    if (!grid_barrier(a.bar, unsigned(h.nb), a.status)) return false;
    T iq[6], nbs = T(0);
#pragma unroll
    for (int o = 0; o < 6; ++o) {
        iq[o] = invd[c + offs[o]];
        nbs += R0[c + offs[o]] * iq[o];
    }
    T w = T(dg) * u - nbs;
    if (ok) static_cast<T*>(a.Wv[0])[c] = w;
    int cur = 0;
    T rq[6], wq[6], sq[6];
    auto fetch = [&] {
        const T* R = static_cast<const T*>(a.R[cur]) + c;
        const T* Wc = static_cast<const T*>(a.Wv[cur]) + c;
        const T* S = static_cast<const T*>(a.S[cur]) + c;
#pragma unroll
        for (int o = 0; o < 6; ++o) { rq[o] = R[offs[o]]; wq[o] = Wc[offs[o]]; sq[o] = S[offs[o]]; }
    };
    double v[3];
    auto sums = [&] {
        v[0] = ok ? double(r) * double(u) : 0.0;
        v[1] = ok ? double(w) * double(u) : 0.0;
        v[2] = ok ? double(r) * double(r) : 0.0;
    };
    sums();
    if (!reduce(a, h, v, fetch)) return false;
    bool go = cg.start(v, tol);
    while (go && !cg.capped(maxit)) {
        const T al = T(cg.alpha), be = T(cg.beta);
        s = fmaT(be, s, w);
        p = fmaT(be, p, u);
        x = fmaT(al, p, x);
        r = fmaT(-al, s, r);
        u = r * inv;
        nbs = T(0);
#pragma unroll
        for (int o = 0; o < 6; ++o) nbs += fmaT(-al, fmaT(be, sq[o], wq[o]), rq[o]) * iq[o];
        w = T(dg) * u - nbs;
        cur ^= 1;
        if (ok) {
            static_cast<T*>(a.R[cur])[c] = r;
            static_cast<T*>(a.Wv[cur])[c] = w;
            static_cast<T*>(a.S[cur])[c] = s;
        }
        sums();
        if (!reduce(a, h, v, fetch)) return false;
        go = cg.next(v);
    }
    if (ok) static_cast<T*>(a.X)[n] = x;
    return true;
}

// A CTA's vectors: cells [0, cap) in shared memory, the rest in the compact
// global arrays.  l counts the CTA's cells; the global pointers start at its
// first one.
template <class T>
struct Own {
    T *x, *r, *p, *s, *w;
    int* c;
    uint8_t* d;
};

// CG of A x = rhs with any number of cells; x to a.X.
template <class T>
__device__ bool cg_many(const PcgArgs& a, Share& h, const float* rhs, double tol, int maxit, Cg& cg) {
    const int tid = threadIdx.x, ms = min(h.m, a.cap);
    Own<T> S;  // shared
    S.x = reinterpret_cast<T*>(pcg_smem);
    S.r = S.x + a.cap; S.p = S.r + a.cap; S.s = S.p + a.cap; S.w = S.s + a.cap;
    S.c = reinterpret_cast<int*>(S.w + a.cap);
    S.d = reinterpret_cast<uint8_t*>(S.c + a.cap);
    Own<T> G;  // global (c and d are read only)
    G.x = static_cast<T*>(a.X) + h.n0;
    G.p = static_cast<T*>(a.P) + h.n0;
    G.r = static_cast<T*>(a.R[1]) + h.n0;
    G.s = static_cast<T*>(a.S[0]) + h.n0;
    G.w = static_cast<T*>(a.Wv[0]) + h.n0;
    G.c = const_cast<int*>(a.fidx) + h.n0;
    G.d = const_cast<uint8_t*>(a.diag) + h.n0;
    T* const U = static_cast<T*>(a.R[0]);
    const int sy = a.sy, sz = a.sz;
    for (int l = tid; l < h.m; l += PCG_THREADS) {
        const int c = G.c[l];
        const uint8_t d = G.d[l];
        const T r = T(rhs[h.n0 + l]);
        const Own<T>& o = l < ms ? S : G;
        if (l < ms) { S.c[l] = c; S.d[l] = d; }
        o.x[l] = o.p[l] = o.s[l] = T(0);
        o.r[l] = r;
        U[c] = r * inv_of(d, T(0));
    }
    if (!grid_barrier(a.bar, unsigned(h.nb), a.status)) return false;
    double v[3];
    // w = A u and the three sums over cells [l0, l1) of o
    auto apply = [&](const Own<T>& o, int l0, int l1) {
        for (int base = l0 + tid; base < l1; base += PCG_UNR * PCG_THREADS) {
            T nbs[PCG_UNR], r[PCG_UNR];
            int d[PCG_UNR];
#pragma unroll
            for (int q = 0; q < PCG_UNR; ++q) {
                const int l = min(base + q * PCG_THREADS, l1 - 1);
                const T* up = U + o.c[l];
                r[q] = o.r[l];
                d[q] = o.d[l];
                nbs[q] = up[1];
                nbs[q] += up[-1];
                nbs[q] += up[sy];
                nbs[q] += up[-sy];
                nbs[q] += up[sz];
                nbs[q] += up[-sz];
            }
#pragma unroll
            for (int q = 0; q < PCG_UNR; ++q) {
                const int l = base + q * PCG_THREADS;
                if (l >= l1) break;
                const T u = r[q] * inv_of(d[q], T(0)), w = T(d[q]) * u - nbs[q];
                o.w[l] = w;
                v[0] += double(r[q]) * double(u);
                v[1] += double(w) * double(u);
                v[2] += double(r[q]) * double(r[q]);
            }
        }
    };
    auto update = [&](const Own<T>& o, int l0, int l1, T al, T be) {
        for (int l = l0 + tid; l < l1; l += PCG_THREADS) {
            const T inv = inv_of(o.d[l], T(0)), r = o.r[l];
            const T s = fmaT(be, o.s[l], o.w[l]);
            const T p = fmaT(be, o.p[l], r * inv);
            o.x[l] = fmaT(al, p, o.x[l]);
            const T rn = fmaT(-al, s, r);
            o.s[l] = s;
            o.p[l] = p;
            o.r[l] = rn;
            U[o.c[l]] = rn * inv;
        }
    };
    auto sums = [&] {
        v[0] = v[1] = v[2] = 0.0;
        apply(S, 0, ms);
        if (h.m > ms) apply(G, ms, h.m);
        return reduce(a, h, v);
    };
    if (!sums()) return false;
    bool go = cg.start(v, tol);
    while (go && !cg.capped(maxit)) {
        const T al = T(cg.alpha), be = T(cg.beta);
        update(S, 0, ms, al, be);
        if (h.m > ms) update(G, ms, h.m, al, be);
        if (!grid_barrier(a.bar, unsigned(h.nb), a.status)) return false;
        if (!sums()) return false;
        go = cg.next(v);
    }
    for (int l = tid; l < ms; l += PCG_THREADS) G.x[l] = S.x[l];
    for (int l = ms + tid; l < h.m; l += PCG_THREADS) G.r[l] = G.s[l] = G.w[l] = T(0);
    return true;
}

// A x of the padded FP64 iterate at a FLUID cell.
__device__ __forceinline__ double apply64(const PcgArgs& a, int c, int d) {
    const double* x = a.xd + c;
    return double(d) * x[0] - (x[1] + x[-1] + x[a.sy] + x[-a.sy] + x[a.sz] + x[-a.sz]);
}
// ||b - A xd||^2 and ||b||^2 over the grid; r (if not null) receives the residual in FP32.
__device__ __forceinline__ bool residual64(const PcgArgs& a, Share& h, float* r, double (&v)[2]) {
    v[0] = v[1] = 0.0;
    for (int l = threadIdx.x; l < h.m; l += PCG_THREADS) {
        const int n = h.n0 + l;
        const double b = double(a.b[n]), e = b - apply64(a, a.fidx[n], a.diag[n]);
        if (r) r[n] = float(e);
        v[0] += e * e;
        v[1] += b * b;
    }
    return reduce(a, h, v);
}
// The pressure out and the padded grids back to zero at the CTA's cells (after
// a reduction: no CTA reads them any more).
template <class T>
__device__ __forceinline__ void finish(const PcgArgs& a, const Share& h, const double* x) {
    for (int l = threadIdx.x; l < h.m; l += PCG_THREADS) {
        const int n = h.n0 + l, c = a.fidx[n];
        const int i = c % a.sy - 1, j = (c / a.sy) % (a.H + 2) - 1, k = c / a.sz - 1;
        a.pout[(int64_t(k) * a.H + j) * a.W + i] = float(x[n]);
        a.xd[c] = 0.0;
        static_cast<T*>(a.invd)[c] = T(0);
        for (int t = 0; t < 2; ++t) {
            static_cast<T*>(a.R[t])[c] = T(0);
            static_cast<T*>(a.Wv[t])[c] = T(0);
            static_cast<T*>(a.S[t])[c] = T(0);
        }
    }
}
__device__ __forceinline__ void report(const PcgArgs& a, int iters, int outer, int st, double rr, double bb, double rz,
                                       double rr0, const double (&res)[2]) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    a.out->iters = iters;
    a.out->outer = outer;
    atomicCAS(a.status, DEV_OK, st);  // never masks a timeout recorded by another CTA
    a.out->rr = rr;
    a.out->bb = bb;
    a.out->rz = rz;
    a.out->rr0 = rr0;
    a.red[0] = res[0];
    a.red[1] = res[1];
    note_solve(&a.out->t_end);
}

__device__ __forceinline__ Share share_of(const PcgArgs& a, bool& one) {
    if (threadIdx.x < 8) {
        s_inv64[threadIdx.x] = threadIdx.x ? 1.0 / double(threadIdx.x) : 0.0;
        s_inv32[threadIdx.x] = threadIdx.x ? 1.0f / float(threadIdx.x) : 0.0f;
    }
    __syncthreads();
    const int nf = *a.nf, nb = int(gridDim.x), chunk = (nf + nb - 1) / nb;
    const int n0 = min(nf, int(blockIdx.x) * chunk);
    one = chunk <= PCG_THREADS;
    return Share{nb, n0, min(nf, n0 + chunk) - n0, 0};
}

// The FP64 solver: CG from x = 0, then the true residual of its solution.
__global__ void __launch_bounds__(PCG_THREADS) k_pcg64(PcgArgs a) {
    note_solve(&a.out->t_begin);
    bool one;
    Share h = share_of(a, one);
    Cg cg;
    if (!(one ? cg_one<double>(a, h, a.b, a.tol, a.maxit, cg) : cg_many<double>(a, h, a.b, a.tol, a.maxit, cg))) return;
    const double* X = static_cast<const double*>(a.X);
    for (int l = threadIdx.x; l < h.m; l += PCG_THREADS) a.xd[a.fidx[h.n0 + l]] = X[h.n0 + l];
    if (!grid_barrier(a.bar, unsigned(h.nb), a.status)) return;
    double v[2];
    if (!residual64(a, h, nullptr, v)) return;
    finish<double>(a, h, X);
    report(a, cg.it, 1, cg.st, cg.rr, cg.bb, cg.gam, cg.bb, v);
}

// The mixed-precision solver: r = b - A x in FP64, A c = r by FP32 CG to a
// loose tolerance, x += c, until ||r|| <= tol ||b||.
__global__ void __launch_bounds__(PCG_THREADS) k_pcg_mixed(PcgArgs a) {
    note_solve(&a.out->t_begin);
    bool one;
    Share h = share_of(a, one);
    const int tid = threadIdx.x;
    double v[2] = {0.0, 0.0};
    if (a.x0) {
        // start at alpha x0, alpha = (x0, b) / (x0, A x0): the A-norm error is never above that of x = 0
        for (int l = tid; l < h.m; l += PCG_THREADS) a.xd[a.fidx[h.n0 + l]] = double(a.x0[h.n0 + l]);
        if (!grid_barrier(a.bar, unsigned(h.nb), a.status)) return;
        for (int l = tid; l < h.m; l += PCG_THREADS) {
            const int n = h.n0 + l;
            const double x = double(a.x0[n]);
            v[0] += x * double(a.b[n]);
            v[1] += x * apply64(a, a.fidx[n], a.diag[n]);
        }
        if (!reduce(a, h, v)) return;
        const double alpha = (v[1] > 0.0 && isfinite(v[0] / v[1])) ? v[0] / v[1] : 0.0;
        for (int l = tid; l < h.m; l += PCG_THREADS) {
            const int n = h.n0 + l;
            a.x64[n] = a.xd[a.fidx[n]] = double(a.x0[n]) * alpha;
        }
        if (!grid_barrier(a.bar, unsigned(h.nb), a.status)) return;
        if (!residual64(a, h, a.bin, v)) return;
    } else {
        for (int l = tid; l < h.m; l += PCG_THREADS) {
            const int n = h.n0 + l;
            const float b = a.b[n];
            a.x64[n] = 0.0;
            a.bin[n] = b;
            v[1] += double(b) * double(b);
        }
        if (!reduce(a, h, v)) return;
        v[0] = v[1];
    }
    const double bb = v[1], rr0 = v[0];
    double relres = bb > 0.0 ? sqrt(v[0] / bb) : 0.0;
    int outer = 0, total = 0, st = DEV_OK;
    Cg cg{};
    while (relres > a.tol && outer < 12 && total < a.maxit) {
        // enough to land below tol after this update, but not below what FP32 vectors can resolve
        const double inner_tol = fmin(0.1, fmax(2e-4, 0.5 * a.tol / relres));
        const int left = a.maxit - total;
        if (!(one ? cg_one<float>(a, h, a.bin, inner_tol, left, cg) : cg_many<float>(a, h, a.bin, inner_tol, left, cg)))
            return;
        const float* C = static_cast<const float*>(a.X);
        for (int l = tid; l < h.m; l += PCG_THREADS) {
            const int n = h.n0 + l;
            const double x = a.x64[n] + double(C[n]);
            a.x64[n] = x;
            a.xd[a.fidx[n]] = x;
        }
        if (!grid_barrier(a.bar, unsigned(h.nb), a.status)) return;
        if (!residual64(a, h, a.bin, v)) return;
        total += cg.it;
        ++outer;
        if (cg.st == DEV_NAN) { st = DEV_NAN; break; }
        const double nr = bb > 0.0 ? sqrt(v[0] / bb) : 0.0;
        const bool better = nr < relres;
        relres = nr;
        if (!better) { st = DEV_BREAKDOWN; break; }  // refinement stalled
    }
    if (relres > a.tol && st == DEV_OK) st = DEV_MAXIT;
    finish<float>(a, h, a.x64);
    v[1] = bb;
    report(a, total, outer, st, v[0], bb, cg.gam, rr0, v);
}

__global__ void k_reset_pcg(GridBar* bar, int* status, unsigned limit) {
    bar->count = 0;
    bar->limit = limit;
    *status = DEV_OK;
}

template <class K>
int launch(K kern, int bytes_per_cell, Dims g, PressureBufs& pb, const float* x0, double tol, int maxit, float* pout,
           cudaStream_t st) {
    // One CTA per 1024 cells of the grid, at most one per SM: with up to half
    // of the cells FLUID a small system has one cell per thread, and a
    // one-CTA grid's barrier is a block barrier.
    const int64_t nc = g.nc();
    const int nb = int(std::max<int64_t>(1, std::min<int64_t>(pcg_max_blocks(), (nc + 1023) / 1024)));
    PcgArgs a{};
    a.W = g.W; a.H = g.H; a.sy = g.W + 2; a.sz = (g.W + 2) * (g.H + 2);
    a.nf = pb.nf; a.fidx = pb.fidx; a.diag = pb.diag; a.b = pb.b; a.x0 = x0; a.bin = pb.bin;
    for (int i = 0; i < 2; ++i) { a.R[i] = pb.R[i]; a.Wv[i] = pb.Wv[i]; a.S[i] = pb.S[i]; }
    a.invd = pb.invd; a.P = pb.P; a.X = pb.X; a.x64 = pb.x64; a.xd = pb.xd;
    a.pout = pout; a.red = pb.red; a.part = pb.part; a.bar = pb.bar; a.status = &pb.out->status; a.out = pb.out;
    a.tol = tol; a.maxit = maxit;
    // shared memory for at most a CTA's share of a grid full of FLUID cells (a multiple of 16, so that every
    // vector is aligned); less of it leaves more of the SM's memory to L1
    const int64_t most = (nc + nb - 1) / nb;
    a.cap = most <= PCG_THREADS ? 0 : int(std::min<int64_t>(PCG_SMEM / bytes_per_cell, most + 15)) & ~15;
    void* args[] = {&a};
    const cudaError_t e = cudaLaunchCooperativeKernel((const void*)kern, dim3(nb), dim3(PCG_THREADS), args,
                                                      size_t(a.cap) * bytes_per_cell, st);
    return e == cudaSuccess ? 0 : int(e);
}

}  // namespace

int pcg_max_blocks() {
    static DeviceMemo memo;
    return memo.get([](int dev) {
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaFuncSetAttribute(k_pcg64, cudaFuncAttributeMaxDynamicSharedMemorySize, PCG_SMEM);
        cudaFuncSetAttribute(k_pcg_mixed, cudaFuncAttributeMaxDynamicSharedMemorySize, PCG_SMEM);
        return sms;
    });
}

void launch_reset_barrier(GridBar* bar, int* status, unsigned wait_polls, cudaStream_t st) {
    k_reset_pcg<<<1, 1, 0, st>>>(bar, status, wait_polls);
}

int launch_pcg(Dims g, PressureBufs& pb, double tol, int maxit, float* pout, cudaStream_t st) {
    return launch(k_pcg64, cell_bytes<double>(), g, pb, nullptr, tol, maxit, pout, st);
}

int launch_pcg_mixed(Dims g, PressureBufs& pb, const float* x0, double tol, int maxit, float* pout, cudaStream_t st) {
    return launch(k_pcg_mixed, cell_bytes<float>(), g, pb, x0, tol, maxit, pout, st);
}

}  // namespace fp
