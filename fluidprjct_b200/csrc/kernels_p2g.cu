// kernels_p2g.cu -- particle-to-grid transfer on the MAC grid.
//
// Restates particlesToGrid (FluidSolver3D.cu:438-685): per particle, 8
// trilinear weights per velocity component (base index floor(r - offset),
// clamped; fractions clamped to [0,1]; faces outside the grid skipped), then
// u = num/den where den > 1e-8, else 0.  The epilogue also performs
// saveVelocities (:399-415, u* = u before gravity) and applyForces
// (:700-761, gravity on every face with the x > (float)INT_MIN test).
//
// B200 design: particles are sorted by cell, and each CTA owns a brick of
// BX x BY x BZ cells with one group of BX * BY threads per velocity component.
// A thread walks a cell's (contiguous) particles once and sums its component's
// contributions to the 2 x 3 x 3 faces the cell can reach in registers; the
// group then adds them into shared-memory accumulators covering the faces the
// brick's cells reach, one face offset at a time: distinct cells write
// distinct faces at the same offset, so plain adds between group barriers do
// (an FP32 shared-memory atomic is a compare-and-swap loop).  Each brick adds
// its accumulated (num, den) pairs into a global FP32 pair array with one
// vector reduction per face, so every particle is walked once per component (a
// brick that instead re-walks a one-cell halo to own its faces outright walks
// each particle 1.76 times on average for 16 x 8 x 8 bricks); empty bricks
// return at once.  A second, elementwise kernel divides, saves and adds
// gravity, and zeroes the pair array for the next step.
//
// Bound by the L1 data pipe (81 % busy: a lane's 16-byte loads lie a cell's
// particles apart) and by the latency of those loads, so by occupancy.
// Staging a slab's particles in shared memory for all three components halved
// the pipe's work but took a third more instructions (152 us at 128^3).  The
// accumulate kernel takes 131 us for the 128^3 dam break (3.8 M particles), 319
// for the 160^3 pool (11 M, dx not a power of two), 488 for the 256 x 128 x 256
// tank (17.5 M) and 14.4 for a 50^3 box; with a hardware barrier in place of the
// one-warp groups' __syncwarp 135, 323, 510 and 15.  With hardware barriers, and
// x / dx still a division: this split 136, 412, 508 and 19; one thread per cell
// for all three components in turn, with shared-memory atomics, 138, 420, 567
// and 33 (a small grid's bricks then leave most of the chip idle); 8 x 8 x 4
// bricks 141, 430, 561 and 23 at five CTAs of 192 per SM, 165, 504 and 650 at
// four.
#include "kernels.hpp"

namespace fp {

namespace {

// Packed FP32 pairs (sm_100's f32x2 FMA/mul/add): two lanes of one 64-bit
// register, each an IEEE FP32 operation rounded to nearest.
__device__ __forceinline__ float2 f2_fma(float2 a, float2 b, float2 c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(d)
        : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)),
          "l"(*reinterpret_cast<unsigned long long*>(&c)));
    return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ float2 f2_mul(float2 a, float2 b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;"
        : "=l"(d)
        : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)));
    return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ float2 f2_add(float2 a, float2 b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;"
        : "=l"(d)
        : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)));
    return *reinterpret_cast<float2*>(&d);
}

// Sums one velocity component of the particles [q0, q1) of cell (ci, cj, ck)
// over the 2 x 3 x 3 faces that cell can reach (2 along the component's own
// axis): an and ad hold num and den, pair = the component axis' two faces,
// index = p slot + 3 q slot of the other two axes.  COMP selects the component.
// The reference's base indices (AccumulateVelocities::operator(),
// FluidSolver3D.cu:469-574) follow from the cell, which is floor(r) clamped to
// the grid: along the own axis the base face is the cell's own, or the next one
// beyond the grid's far edge; along the others it is the face below the cell or
// the cell's own.  Weights are (wx*wy)*wz as in the reference; the two faces
// along the component's axis are one packed pair, so each particle costs 12
// packed multiplies and 9 packed FMAs and adds per component.  num accumulates
// vel*wgt with one fused multiply-add (the reference rounds the product first;
// its float atomics already leave the last bits of the sums order-dependent).
// The particle's velocity component COMP.
template <int COMP>
__device__ __forceinline__ float comp_of(const float4& v) { return COMP == 0 ? v.x : (COMP == 1 ? v.y : v.z); }

template <int COMP, bool P2>
__device__ __forceinline__ void sum_cell(const float4* __restrict__ pos, const float4* __restrict__ vel, int q0, int q1,
                                         int ci, int cj, int ck, const Dims& g, float2 (&an)[9], float2 (&ad)[9]) {
    const int co = COMP == 0 ? ci : (COMP == 1 ? cj : ck), cp = COMP == 0 ? cj : ci, cq = COMP == 2 ? cj : ck;
    const float fo = float(co), fe = float(COMP == 0 ? g.W : (COMP == 1 ? g.H : g.D)), fp = float(cp), fq = float(cq);
    const float tp = cp > 0 ? fp : -INFINITY, tq = cq > 0 ? fq : -INFINITY;
#pragma unroll
    for (int m = 0; m < 9; ++m) { an[m] = make_float2(0.0f, 0.0f); ad[m] = make_float2(0.0f, 0.0f); }
    // (unrolling this walk by 2 or 4 measured slower: the larger code missed
    // in the instruction cache; prefetching the next particle gained 1 us)
    for (int q = q0; q < q1; ++q) {
        const float4 P = pos[q];
        const float vc = comp_of<COMP>(vel[q]);
        const float rx = to_grid<P2>(P.x, g), ry = to_grid<P2>(P.y, g), rz = to_grid<P2>(P.z, g);
        const float ro = COMP == 0 ? rx : (COMP == 1 ? ry : rz), rp = (COMP == 0 ? ry : rx) - 0.5f,
                    rq = (COMP == 2 ? ry : rz) - 0.5f;
        const bool past = ro >= fe, lp = rp < tp, lq = rq < tq;
        const float wo = __saturatef(ro - (past ? fe : fo)), wp = __saturatef(rp - (lp ? fp - 1.0f : fp)),
                    wq = __saturatef(rq - (lq ? fq - 1.0f : fq));
        const float2 w2 = past ? make_float2(0.0f, 1.0f - wo) : make_float2(1.0f - wo, wo);
        const float p3[3] = {lp ? 1.0f - wp : 0.0f, lp ? wp : 1.0f - wp, lp ? 0.0f : wp};
        const float q3[3] = {lq ? 1.0f - wq : 0.0f, lq ? wq : 1.0f - wq, lq ? 0.0f : wq};
        const float2 vv = make_float2(vc, vc);
        // (wx * wy) * wz, as in the reference
#pragma unroll
        for (int b = 0; b < 3; ++b)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                float2 w;
                if (COMP == 2) w = f2_mul(make_float2(p3[b] * q3[c], p3[b] * q3[c]), w2);
                else w = f2_mul(f2_mul(w2, make_float2(p3[b], p3[b])), make_float2(q3[c], q3[c]));
                an[b + 3 * c] = f2_fma(vv, w, an[b + 3 * c]);
                ad[b + 3 * c] = f2_add(ad[b + 3 * c], w);
            }
    }
}

// CTAs per SM that the register budget must allow (P2G_MIN_BLOCKS, a build
// tunable): the walk over a cell's particles waits on their loads, so
// occupancy decides.  At 64 registers, ten CTAs of 96 threads.
#ifndef P2G_MIN_BLOCKS
#define P2G_MIN_BLOCKS 10
#endif

// The faces around a brick: one more than its cells on each side of every axis
// (one less is reached along a component's own axis).
template <int BX, int BY, int BZ>
struct Reach {
    static constexpr int X = BX + 2, Y = BY + 2, Z = BZ + 2, N = X * Y * Z;
};

// Barrier of one component's group of N threads.  The lanes come out of walks of
// different lengths: a group of one warp synchronises as a warp, a larger one by
// the form of the barrier that does not need its warps converged.
template <int COMP, int N>
__device__ __forceinline__ void group_sync() {
    if constexpr (N == 32) __syncwarp();
    else asm volatile("barrier.sync %0, %1;\n" ::"n"(COMP + 1), "n"(N) : "memory");
}

// One component of a brick, by the BX * BY threads of one group: thread t
// takes cell (t % BX, t / BX) of every z slab in turn.
template <int COMP, int BX, int BY, int BZ, bool P2>
__device__ __forceinline__ void brick_component(const float4* __restrict__ pos, const float4* __restrict__ vel,
                                                const int* __restrict__ start, const Dims& g, int i0, int j0, int k0,
                                                float2* s_acc) {
    using R = Reach<BX, BY, BZ>;
    const int t = int(threadIdx.x) % (BX * BY), lx = t % BX, ly = t / BX, ci = i0 + lx, cj = j0 + ly;
    const bool in = ci < g.W && cj < g.H;
#pragma unroll 1
    for (int lz = 0; lz < BZ; ++lz) {
        const int ck = k0 + lz, c = ci + cj * g.W + ck * g.W * g.H;
        const bool ok = in && ck < g.D;
        const int q0 = ok ? start[c] : 0, q1 = ok ? start[c + 1] : 0;
        float2 an[9], ad[9];
        sum_cell<COMP, P2>(pos, vel, q0, q1, ci, cj, ck, g, an, ad);
        float2* s = s_acc + COMP * R::N + lx + ly * R::X + lz * R::X * R::Y;
#pragma unroll
        for (int m = 0; m < 9; ++m)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int o1 = m % 3, o2 = m / 3;
                const int ox = COMP == 0 ? e : o1, oy = COMP == 1 ? e : (COMP == 0 ? o1 : o2), oz = COMP == 2 ? e : o2;
                // a face that none of the cell's particles reaches has weight 0 here, and a num of 0 times
                // their velocities: NaN for one that is not finite, so it is left out
                const float den = e ? ad[m].y : ad[m].x;
                if (den != 0.0f) {
                    float2& f = s[ox + oy * R::X + oz * R::X * R::Y];
                    const float2 v = f;
                    f = make_float2(v.x + (e ? an[m].y : an[m].x), v.y + den);
                }
                group_sync<COMP, BX * BY>();
            }
    }
}

// Pass 1: one CTA per brick.  acc holds (num, den) pairs for the u, v and w
// faces back to back ([nu | nv | nw]); it is zero on entry except for what
// other bricks of this launch add.
template <int BX, int BY, int BZ, bool P2>
__global__ void __launch_bounds__(3 * BX * BY, P2G_MIN_BLOCKS) k_p2g_accum(const float4* __restrict__ pos,
                                                                           const float4* __restrict__ vel,
                                                                           const int* __restrict__ start, Dims g,
                                                                           float2* __restrict__ acc) {
    using R = Reach<BX, BY, BZ>;
    constexpr int NT = 3 * BX * BY;
    static_assert(BX * BY % 32 == 0, "a group is whole warps");
    __shared__ float2 s_acc[3 * R::N];

    const int W = g.W, H = g.H, D = g.D;
    const int nbx = (W + BX - 1) / BX, nby = (H + BY - 1) / BY;
    const int bid = blockIdx.x;
    const int i0 = (bid % nbx) * BX, j0 = ((bid / nbx) % nby) * BY, k0 = (bid / (nbx * nby)) * BZ;

    bool any = false;
    for (int t = threadIdx.x; t < BX * BY * BZ; t += NT) {
        const int i = i0 + t % BX, j = j0 + (t / BX) % BY, k = k0 + t / (BX * BY);
        if (i >= W || j >= H || k >= D) continue;
        const int c = i + j * W + k * W * H;
        any |= start[c + 1] > start[c];
    }
    if (!__syncthreads_or(any)) return;  // no particle: nothing to add
    for (int t = threadIdx.x; t < 3 * R::N; t += NT) s_acc[t] = make_float2(0.0f, 0.0f);
    __syncthreads();
    const int grp = int(threadIdx.x) / (BX * BY);
    if (grp == 0) brick_component<0, BX, BY, BZ, P2>(pos, vel, start, g, i0, j0, k0, s_acc);
    else if (grp == 1) brick_component<1, BX, BY, BZ, P2>(pos, vel, start, g, i0, j0, k0, s_acc);
    else brick_component<2, BX, BY, BZ, P2>(pos, vel, start, g, i0, j0, k0, s_acc);
    __syncthreads();

    // Add the reached faces inside the grid into acc (one 8-byte vector
    // reduction per face); faces outside the grid are dropped, as the
    // reference skips them.
    const int64_t nu = g.nu(), nv = g.nv();
    for (int t = threadIdx.x; t < 3 * R::N; t += NT) {
        const float2 f = s_acc[t];
        if (f.y == 0.0f) continue;
        const int a = t / R::N, r = t - a * R::N;
        const int fi = i0 + r % R::X - (a != 0), fj = j0 + (r / R::X) % R::Y - (a != 1),
                  fk = k0 + r / (R::X * R::Y) - (a != 2);
        const int nx = W + (a == 0), ny = H + (a == 1), nz = D + (a == 2);
        if (fi < 0 || fi >= nx || fj < 0 || fj >= ny || fk < 0 || fk >= nz) continue;
        const int64_t idx = (a == 0 ? 0 : a == 1 ? nu : nu + nv) + int64_t(fi) + int64_t(fj) * nx + int64_t(fk) * nx * ny;
        atomicAdd(&acc[idx], f);
    }
}

// Pass 2, over every face: num/den (ComputeVelocityFunc :598-605), u* <- u, u +=
// dt*g (the x > (float)INT_MIN test of applyForces), and acc <- 0 where it is
// not 0 already: most faces of a scene are away from its particles, and their
// pair needs no store.  Bound by memory, so a thread loads all its pairs before
// it uses any: 22.9 us at 128^3, 41 at 160^3 and 84 for 256 x 128 x 256 (500 MB),
// against 29, 55 and 114 face by face, and 31, 57 and 114 as a launch per
// component that stored every pair.
struct FinishArgs {
    int64_t end[3];  // faces of u; of u and v; of all
    float g[3];
    float *dst[3], *sav[3];
};
constexpr int FINISH_THREADS = 256, FINISH_FACES = 4;
template <bool FUSED>
__global__ void __launch_bounds__(FINISH_THREADS) k_p2g_finish(float2* __restrict__ acc, float dt, FinishArgs f) {
    const int64_t t0 = int64_t(blockIdx.x) * (FINISH_THREADS * FINISH_FACES) + threadIdx.x;
    float2 a[FINISH_FACES];
#pragma unroll
    for (int m = 0; m < FINISH_FACES; ++m) {
        const int64_t t = t0 + m * FINISH_THREADS;
        a[m] = t < f.end[2] ? acc[t] : make_float2(0.0f, 0.0f);
    }
#pragma unroll
    for (int m = 0; m < FINISH_FACES; ++m) {
        const int64_t t = t0 + m * FINISH_THREADS;
        if (t >= f.end[2]) return;
        const int c = t < f.end[0] ? 0 : (t < f.end[1] ? 1 : 2);
        const int64_t i = c == 0 ? t : t - (c == 1 ? f.end[0] : f.end[1]);
        float* dst = c == 0 ? f.dst[0] : (c == 1 ? f.dst[1] : f.dst[2]);
        if (a[m].x != 0.0f || a[m].y != 0.0f) acc[t] = make_float2(0.0f, 0.0f);
        float val = 0.0f;
        if (a[m].y > 1e-8f) val = a[m].x / a[m].y;
        if (FUSED) {
            float* sav = c == 0 ? f.sav[0] : (c == 1 ? f.sav[1] : f.sav[2]);
            const float gc = c == 0 ? f.g[0] : (c == 1 ? f.g[1] : f.g[2]);
            sav[i] = val;
            dst[i] = (val > -2147483648.0f) ? val + dt * gc : val;
        } else {
            dst[i] = val;
        }
    }
}

// applyForces alone (phase-by-phase mode): x > (float)INT_MIN ? x + dt*a : x.
__global__ void k_forces(float* __restrict__ a, int64_t n, float dt, float acc) {
    int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= n) return;
    float x = a[t];
    a[t] = (x > -2147483648.0f) ? x + dt * acc : x;
}

__global__ void k_copy(const float* __restrict__ s, float* __restrict__ d, int64_t n) {
    int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t < n) d[t] = s[t];
}

}  // namespace

// Brick shape and CTA size (build tunables).
#ifndef P2G_BRICK_X
#define P2G_BRICK_X 8
#define P2G_BRICK_Y 4
#define P2G_BRICK_Z 4
#endif
constexpr int P2G_BX = P2G_BRICK_X, P2G_BY = P2G_BRICK_Y, P2G_BZ = P2G_BRICK_Z, P2G_NT = 3 * P2G_BX * P2G_BY;

void launch_p2g(const float4* pos, const float4* vel, const int* start, Dims g, float dt, float3 gravity,
                float2* acc, float* u, float* v, float* w, float* us, float* vs, float* ws, int fused_forces,
                cudaStream_t st) {
    const int nb = ((g.W + P2G_BX - 1) / P2G_BX) * ((g.H + P2G_BY - 1) / P2G_BY) * ((g.D + P2G_BZ - 1) / P2G_BZ);
    if (g.idx != 0.0f) k_p2g_accum<P2G_BX, P2G_BY, P2G_BZ, true><<<nb, P2G_NT, 0, st>>>(pos, vel, start, g, acc);
    else k_p2g_accum<P2G_BX, P2G_BY, P2G_BZ, false><<<nb, P2G_NT, 0, st>>>(pos, vel, start, g, acc);
    const FinishArgs f{{g.nu(), g.nu() + g.nv(), g.nu() + g.nv() + g.nw()},
                       {gravity.x, gravity.y, gravity.z}, {u, v, w}, {us, vs, ws}};
    constexpr int per = FINISH_THREADS * FINISH_FACES;
    const unsigned nb2 = unsigned((f.end[2] + per - 1) / per);
    if (fused_forces) k_p2g_finish<true><<<nb2, FINISH_THREADS, 0, st>>>(acc, dt, f);
    else k_p2g_finish<false><<<nb2, FINISH_THREADS, 0, st>>>(acc, dt, f);
}

void launch_forces(float* u, float* v, float* w, Dims g, float dt, float3 gravity, cudaStream_t st) {
    k_forces<<<unsigned((g.nu() + 255) / 256), 256, 0, st>>>(u, g.nu(), dt, gravity.x);
    k_forces<<<unsigned((g.nv() + 255) / 256), 256, 0, st>>>(v, g.nv(), dt, gravity.y);
    k_forces<<<unsigned((g.nw() + 255) / 256), 256, 0, st>>>(w, g.nw(), dt, gravity.z);
}

void launch_copy(const float* src, float* dst, int64_t n, cudaStream_t st) {
    if (n > 0) k_copy<<<unsigned((n + 255) / 256), 256, 0, st>>>(src, dst, n);
}

}  // namespace fp
