// The fused per-step sweep: one CTA advances a TX x TY tile of interior
// cells by one time step.
//
// It restates, in one pass over shared memory, the reference Advance
// (MUSCL_Scheme.cpp:6-152 / MHM_Scheme.cpp:5-203 / Godunov_Scheme.cpp:6-140):
// face reconstruction, MHM predictor, X and Y Riemann solves, the X update
// followed by the Y update (both from the old state), restricted to fluid
// cells; then the CFL maxima (ComputeDt.cpp:28-49) and the mass sum
// (CaculateMass.cpp:27-38) of the new state, folded into the epilogue.
//
// The reference's Y solver shares its output slot with the X solver
// (MUSCL/EQDefine.H:35-36) and skips the store in some branches; the
// kernel keeps both face fluxes in shared memory and takes the X-face flux
// of the same cell where the reference would have left it in place.
//
// The tile body (sweep_tile64) is shared by two frames: sweep_kernel (one
// case, one CTA per active tile) and the persistent batched kernel of
// batch.cu (many cases, CTAs loop over one tile table).
#pragma once

#include <atomic>

#include "internal.h"
#include "physics.cuh"
#include "physics_fast64.cuh"
#include "tile_faces.cuh"
#include "tma.cuh"

namespace ibtfo {

__device__ __forceinline__ void atomic_max_nonneg(unsigned long long *addr, double v)
{
    // non-negative doubles order like their bit patterns
    atomicMax(addr, (unsigned long long)__double_as_longlong(v));
}

// the partial mass sums a step's last block adds up: `n` of them, or those of
// `n` 32x16 tiles in `parts` parts each, which are added in the tree of
// tile_mass_32x16: four FINE_X x FINE_Y tiles (lower row first), or two 32x8 ones
struct MassPartials
{
    double *p;
    unsigned n;
    int parts;
    unsigned at;   // where the block's own sum goes
};

__device__ __forceinline__ double mass_partial(const MassPartials &m, unsigned b)
{
    const volatile double *p = m.p;
    if (m.parts == 1)
        return p[b];
    if (m.parts == 2)
        return p[2 * (size_t)b] + p[2 * (size_t)b + 1];
    static_assert(TILE_X == 2 * FINE_X && FAST_TILE_Y == 2 * FINE_Y, "four fine tiles in a 32x16 tile");
    const volatile double *q = p + 4 * (size_t)b;
    return (q[0] + q[1]) + (q[2] + q[3]);
}

// Commit one block's (max a, max |u|, max |v|, mass, nan count), held by
// thread 0, to the step's device state; the last of the case's `nblocks`
// blocks to finish computes the next dt and advances the reference loop
// accounting.  Deterministic: the mass partials are summed in a fixed order
// (256 interleaved sums, then a tree) whichever block finishes last and
// however many threads it has.  Called by every
// thread of the block.  A first RK2 stage (`first_stage`) commits nothing:
// its last block only hands the stage's buffer to the boundary pass.
template <int NT>
__device__ __forceinline__ void block_commit_finalize(double a, double u, double v, double m, int n, DevState *st,
                                                      const MassPartials &mp, const GridDesc &g, bool step_accounting,
                                                      bool set_start, unsigned nblocks, bool first_stage = false)
{
    __shared__ bool last;
    if (first_stage)
    {
        if (threadIdx.x == 0)
        {
            __threadfence();
            unsigned t = atomicAdd(&st->ticket, 1u);
            if (t == nblocks - 1)
            {
                volatile DevState *vs = st;
                vs->cur = vs->cur ^ 1;
                vs->fill_pending = 1;
                vs->ticket = 0u;
                __threadfence();
            }
        }
        return;
    }
    if (threadIdx.x == 0)
    {
        if (a > 0) atomic_max_nonneg(&st->amax_bits, a);
        if (u > 0) atomic_max_nonneg(&st->umax_bits, u);
        if (v > 0) atomic_max_nonneg(&st->vmax_bits, v);
        if (n) atomicAdd(&st->nan_step, n);
        mp.p[mp.at] = m;
        __threadfence();
        unsigned t = atomicAdd(&st->ticket, 1u);
        last = (t == nblocks - 1);
    }
    __syncthreads();
    if (!last)
        return;
    __threadfence();
    // fixed-order sum of the mass partials
    constexpr int SUMS = 256;
    __shared__ double msum[SUMS];
    for (int q = threadIdx.x; q < SUMS; q += NT)
    {
        double s = 0.0;
        for (unsigned b = q; b < mp.n; b += SUMS)
            s += mass_partial(mp, b);
        msum[q] = s;
    }
    __syncthreads();
    for (int h = SUMS / 2; h > 0; h >>= 1)
    {
        for (int q = threadIdx.x; q < h; q += NT)
            msum[q] += msum[q + h];
        __syncthreads();
    }
    if (threadIdx.x == 0)
    {
        volatile DevState *vs = st;
        double a_max = __longlong_as_double((long long)vs->amax_bits);
        double u_max = __longlong_as_double((long long)vs->umax_bits);
        double v_max = __longlong_as_double((long long)vs->vmax_bits);
        // ComputeDt.cpp:49
        double dt_new = g.cfl * g.dx / (a_max + ((u_max < v_max) ? v_max : u_max));
        vs->last_amax = a_max;
        vs->last_umax = u_max;
        vs->last_vmax = v_max;
        vs->dt = dt_new;
        vs->mass = msum[0];
        if (set_start)
            vs->mass_start = msum[0];
        if (step_accounting)
        {
            vs->now_t = vs->now_t + dt_new; // Test/Sod/Sod.cpp:176
            vs->iter = vs->iter + 1;
            vs->cur = vs->cur ^ 1;
            vs->fill_pending = 1;
        }
        vs->nan_cells = vs->nan_step;
        vs->nan_step = 0;
        if (vs->nan_cells)
            vs->status |= STATUS_NAN; // sticky: some step held a NaN
        vs->amax_bits = 0ull;
        vs->umax_bits = 0ull;
        vs->vmax_bits = 0ull;
        vs->ticket = 0u;
        __threadfence();
    }
    __syncthreads(); // msum and `last` are reused by the next tile of a persistent CTA
}

// Second RK2 stage: the cell's new state is 0.5 (U0 + w), w the advanced
// first-stage state and U0 the state at the start of the step, which the
// output buffer still holds at this cell (RK2.cpp:41-43 without the
// reference's stride mix-up; the first stage never writes that buffer)
__device__ __forceinline__ void rk2_average(const double *V, long long o, long long P, double v[4])
{
#pragma unroll
    for (int k = 0; k < 4; k++)
        v[k] = 0.5 * (V[k * P + o] + v[k]);
}

// Per-thread CFL maxima, mass and NaN count of the cells a thread updated.
// The sound speed enters as its square (a2max); the block takes one square
// root of the maximum, which equals the maximum of the roots (the root is
// monotone and correctly rounded; NaN and negative squares drop out of both).
// The mass of a 32x16 tile's lower and upper eight rows is kept apart.
struct CellStats
{
    double amax = 0.0, a2max = 0.0, umax = 0.0, vmax = 0.0, mass = 0.0, mass_upper = 0.0;
    int nans = 0;
};

// max(m, x) for m >= 0 as fmax gives it (NaN and negative x leave m), with
// the compare on the integer pipe: non-negative doubles order like their bits
__device__ __forceinline__ double max_nonneg(double m, double x)
{
    const long long bm = __double_as_longlong(m), bx = __double_as_longlong(x);
    return (bx > bm && bx <= 0x7ff0000000000000LL) ? x : m;
}

// The mass of a 32x16 tile, added as a tree over its 8x8 blocks: in a block
// the columns in pairs, fours and eights, then the rows likewise; then the
// four blocks of each half, then the halves.  A sum of the same cells swept
// as 16x8 or 32x8 tiles (mass_partial) has the same bits.  Warp w holds rows w
// (mass) and w + 8 (mass_upper; zero in a 32x8 tile), lane c column c; thread 0
// receives the sum.
__device__ __forceinline__ double tile_mass_32x16(double lower, double upper)
{
    __shared__ double col[2][4][8], half[2];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1)
    {
        lower += __shfl_xor_sync(0xffffffffu, lower, o);
        upper += __shfl_xor_sync(0xffffffffu, upper, o);
    }
    if ((lane & 7) == 0)
    {
        col[0][lane >> 3][w] = lower;
        col[1][lane >> 3][w] = upper;
    }
    __syncthreads();
    if (w < 2)
    {
        double v = col[w][lane >> 3][lane & 7];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
            v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0)
            half[w] = v;
    }
    __syncthreads();
    return half[0] + half[1];
}

// The mass of a 16x8 tile: threads 0..127 hold its cells, row-major (a warp
// two rows of 16); the others take no part.  Thread 0 receives the sum.
__device__ __forceinline__ double tile_mass_16x8(double v)
{
    static_assert(FINE_X == 16 && FINE_Y == 8, "two 8x8 blocks");
    __shared__ double part[2][4]; // block, pair of rows
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (w < 4)
    {
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) // the columns of a block
            v += __shfl_xor_sync(0xffffffffu, v, o);
        v += __shfl_xor_sync(0xffffffffu, v, 16); // the warp's two rows
        if ((lane & 7) == 0 && lane < 16)
            part[lane >> 3][w] = v;
    }
    __syncthreads();
    if (threadIdx.x != 0)
        return 0.0;
    return ((part[0][0] + part[0][1]) + (part[0][2] + part[0][3])) +
           ((part[1][0] + part[1][1]) + (part[1][2] + part[1][3]));
}

// The sum of 256 threads' values: per warp, lanes 16 apart, then 8, 4, 2, 1;
// then the warps in order (thread 0 receives it).  The partial sums are
// gathered after each level, so that a level takes as many FP64 warp
// instructions as it has sums (16 for the block; 47 with every lane of every
// warp adding at every level).
__device__ __forceinline__ double block_sum_256(double v)
{
    __shared__ double part[256];
    const int t = threadIdx.x;
    part[t] = v;
    __syncthreads();
    if (t < 128)
        v = part[(t >> 4) * 32 + (t & 15)] + part[(t >> 4) * 32 + (t & 15) + 16];
    __syncthreads();
    if (t < 128)
        part[t] = v;
    __syncthreads();
    if (t < 64)
        v = part[(t >> 3) * 16 + (t & 7)] + part[(t >> 3) * 16 + (t & 7) + 8];
    __syncthreads();
    if (t < 64)
        part[t] = v;
    __syncthreads();
    if (t < 32)
    {
        v = part[(t >> 2) * 8 + (t & 3)] + part[(t >> 2) * 8 + (t & 3) + 4];
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        double m = v; // lane 4 w: the sum of warp w
        for (int w = 1; w < 8; w++)
            m += __shfl_sync(0xffffffffu, v, 4 * w);
        v = m;
    }
    return v;
}

// Block-wide FP64 reduction of the per-thread statistics, then
// block_commit_finalize.  CELLS: the warps that hold updated cells come first
// (a block with more threads than cells).
// HALF: a 32x8 tile added as a half of a 32x16 one.
template <int NT, int TX = 0, int TY = 0, bool HALF = false>
__device__ __forceinline__ void block_reduce_finalize(CellStats cs, DevState *st, const MassPartials &mp,
                                                      const GridDesc &g, bool step_accounting, bool set_start,
                                                      unsigned nblocks, bool first_stage = false)
{
    if (first_stage)
    {
        __syncthreads(); // every thread of the block has stored its cells
        block_commit_finalize<NT>(0, 0, 0, 0, 0, st, mp, g, false, false, nblocks, true);
        return;
    }
    static_assert(!HALF || (TX == 32 && TY == 8 && NT == 256), "rows by warps");
    constexpr bool TREE = (TX == 32 && TY == 16 && NT == 256) || (TX == FINE_X && TY == FINE_Y) || HALF;
    constexpr int CELLS = TX * TY ? TX * TY : NT;
    constexpr int NW = (CELLS < NT ? CELLS : NT) / 32; // warps with cells
    __shared__ double red[5][NW];
    __shared__ int rnan[NW];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double m = 0.0;
    if constexpr (TREE && TX == 32)
        m = tile_mass_32x16(cs.mass, cs.mass_upper);
    if constexpr (TREE && TX == FINE_X)
        m = tile_mass_16x8(cs.mass);
    if constexpr (!TREE && TX * TY > NT)
        cs.mass += cs.mass_upper;
    constexpr bool GATHER = !TREE && NT == 256 && NW == 8;
    if constexpr (GATHER)
        m = block_sum_256(cs.mass);
    if (wid < NW)
    {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
        {
            cs.amax = max_nonneg(cs.amax, __shfl_xor_sync(0xffffffffu, cs.amax, o));
            cs.a2max = max_nonneg(cs.a2max, __shfl_xor_sync(0xffffffffu, cs.a2max, o));
            cs.umax = max_nonneg(cs.umax, __shfl_xor_sync(0xffffffffu, cs.umax, o));
            cs.vmax = max_nonneg(cs.vmax, __shfl_xor_sync(0xffffffffu, cs.vmax, o));
            if (!TREE && !GATHER)
                cs.mass += __shfl_xor_sync(0xffffffffu, cs.mass, o);
            cs.nans += __shfl_xor_sync(0xffffffffu, cs.nans, o);
        }
        if (lane == 0)
        {
            red[0][wid] = cs.amax;
            red[1][wid] = cs.umax;
            red[2][wid] = cs.vmax;
            red[3][wid] = cs.mass;
            red[4][wid] = cs.a2max;
            rnan[wid] = cs.nans;
        }
    }
    __syncthreads();
    double a = 0.0, u = 0.0, v = 0.0;
    int n = 0;
    if (threadIdx.x == 0)
    {
        double a2 = red[4][0];
        a = red[0][0], u = red[1][0], v = red[2][0];
        n = rnan[0];
        if (!TREE && !GATHER)
            m = red[3][0];
        for (int w = 1; w < NW; w++)
        {
            a = max_nonneg(a, red[0][w]);
            a2 = max_nonneg(a2, red[4][w]);
            u = max_nonneg(u, red[1][w]);
            v = max_nonneg(v, red[2][w]);
            if (!TREE && !GATHER)
                m += red[3][w];
            n += rnan[w];
        }
        a = max_nonneg(a, sqrt_rn(a2));
    }
    block_commit_finalize<NT>(a, u, v, m, n, st, mp, g, step_accounting, set_start, nblocks);
}

// any of four values NaN, tested on the integer pipe
__device__ __forceinline__ int any_nan4(const double v[4])
{
    const long long inf = 0x7ff0000000000000LL;
    return (magnitude_bits(v[0]) > inf || magnitude_bits(v[1]) > inf || magnitude_bits(v[2]) > inf ||
            magnitude_bits(v[3]) > inf)
               ? 1
               : 0;
}

// CFL and mass contributions of one fluid cell of the new state
// (ComputeDt.cpp:38-45, CaculateMass.cpp:36)
__device__ __forceinline__ void cell_stats(const double v[4], double gam, double dx, double dy, CellStats &cs,
                                           double &mass)
{
    double rho = v[0];
    const Divisor by_rho = divisor(rho);
    double u = divide_rn(v[1], by_rho);
    double w = divide_rn(v[2], by_rho);
    double p = (gam - 1) * (v[3] - 0.5 * rho * (u * u + w * w));
    cs.a2max = max_nonneg(cs.a2max, divide_rn(gam * p, by_rho)); // pow(gam p / rho, 0.5) taken once per block
    cs.umax = max_nonneg(cs.umax, magnitude(u));
    cs.vmax = max_nonneg(cs.vmax, magnitude(w));
    mass += v[0] * dx * dy;
    cs.nans += any_nan4(v);
}

// the same statistics from the cell's velocity and internal energy (fp64_fast)
__device__ __forceinline__ void cell_stats_fast(const double v[4], const Cell64 &c, const GasConst<double> &K,
                                                double dxdy, CellStats &cs, double &mass)
{
    cs.a2max = max_nonneg(cs.a2max, K.ggm1 * (c.ir * c.ei));
    cs.umax = max_nonneg(cs.umax, magnitude(c.u));
    cs.vmax = max_nonneg(cs.vmax, magnitude(c.v));
    mass += v[0] * dxdy;
    cs.nans += any_nan4(v);
}

// shared memory of one FP64 tile: the tile plus two halo cells each side,
// X faces (i+1/2, j) for i in [i0-1, i0+TX), j in [j0-1, j0+TY), Y faces
// (i, j+1/2) for i in [i0, i0+TX), j in [j0-1, j0+TY)
template <int TX, int TY>
struct SweepSmem64
{
    double sU[4][TY + 4][TX + 4];
    double sF[4][TY + 1][TX + 1];
    double sG[4][TY + 1][TX];
    double sC[4]; // fp64_fast: dt/dx, dt/dy, dt/(2dx), dt/(2dy), computed once per tile
    unsigned char sKeep[TY + 1][TX];
    TileFaces<TX, TY> tf; // the faces some fluid cell of the tile reads
};

// Advance the tile whose first interior cell is (i0, j0) from U into V and
// accumulate the statistics of the updated cells.  All NT threads call it.
// stage 2 (the second RK2 stage) stores 0.5 (V + the advanced state) instead,
// V holding the state at the start of the step; stage 1 gathers no statistics.
// With `tmap` the tile and halo are staged by one bulk tensor copy (the box
// starts at column i0 - 2, which must be a multiple of 2); a copy that does
// not complete within the bounded wait sets STATUS_STALL in *status and the
// tile is staged element-wise.
template <int SCH, int RIE, int LIM, int FAST, int TX, int TY, int NT>
__device__ __forceinline__ void sweep_tile64(SweepSmem64<TX, TY> &s, const GridDesc &g, const double *__restrict__ U,
                                             double *__restrict__ V, const uint8_t *__restrict__ type, int i0, int j0,
                                             double dt, CellStats &cs, int stage = 0,
                                             const CUtensorMap *tmap = nullptr, int *status = nullptr,
                                             bool interior = false)
{
    constexpr int WX = TX + 4, WY = TY + 4;
    const long long P = g.plane;
    const int pitch = g.pitch;
    const int tid = threadIdx.x;
    constexpr bool FASTPHYS = FAST || safeguarded(RIE); // faces evaluated by physics_fast64.cuh
    if (FASTPHYS && tid == 0)
    {
        s.sC[0] = dt * g.idx;
        s.sC[1] = dt * g.idy;
        s.sC[2] = 0.5 * s.sC[0];
        s.sC[3] = 0.5 * s.sC[1];
    }

    bool staged = false;
    __shared__ uint64_t bar;
    if (tmap)
    {
        if (tid == 0)
            mbar_init(&bar, 1);
        __syncthreads();
        if (tid == 0)
        {
            mbar_expect_tx(&bar, (unsigned)sizeof(s.sU));
            tma_load_3d(&s.sU[0][0][0], tmap, i0 - 2, j0 - 2, 0, &bar);
        }
    }
    // cell flags and the face list while the copy is in flight
    tile_faces_build<TX, TY, NT>(s.tf, s.sKeep, g, type, i0, j0, interior);
    if (tmap)
    {
        staged = __syncthreads_and(mbar_wait(&bar, 0));
        // a copy that missed the bounded wait: the step is reported as failed
        // (STATUS_STALL makes the host return IBTFO_ETIMEOUT); the tile is
        // staged element-wise and, before the CTA leaves the tile, the copy is
        // waited for once more, so that a late copy lands while this CTA
        // still owns the shared memory (it brings the values staged here)
        if (!staged && tid == 0 && status)
            atomicOr(status, STATUS_STALL);
    }
    // stage the tile and its halo (always inside the padded array: ng >= 2),
    // one index computation per cell for the four planes
    if (!staged)
    {
        for (int q = tid; q < WX * WY; q += NT)
        {
            const int ly = q / WX, lx = q - ly * WX;
            const int gi = i0 - 2 + lx, gj = j0 - 2 + ly;
            double v[4] = {0.0, 0.0, 0.0, 0.0};
            if (gi < g.M && gj < g.N)
            {
                const double *src = U + (long long)gj * pitch + gi;
#pragma unroll
                for (int k = 0; k < 4; k++)
                    v[k] = src[k * P];
            }
#pragma unroll
            for (int k = 0; k < 4; k++)
                s.sU[k][ly][lx] = v[k];
        }
        stores_before_copies(); // a batch's next tile
    }
    __syncthreads();

    const double gam = g.gamma;
    const GasConst<double> K(g);
    const double hx2 = FASTPHYS ? s.sC[2] : 0.0, hy2 = FASTPHYS ? s.sC[3] : 0.0; // MHM predictor of physics_fast64.cuh
    // X faces of the tile's rows (sF rows 1..TY) and all Y faces; the X faces
    // of the row below the tile (sF row 0) follow below, where needed
    constexpr int NXF = TileFaces<TX, TY>::NXF;
    const int nfaces = s.tf.n;
    for (int t = tid; t < nfaces; t += NT)
    {
        const int q = tile_face(s.tf, t);
        double c0[4], c1[4], c2[4], c3[4], f[4];
        if (q < NXF)
        {
            int r, fc;
            x_face_of<TX, TY>(q, r, fc);
#pragma unroll
            for (int k = 0; k < 4; k++)
            {
                c0[k] = s.sU[k][r + 1][fc];
                c1[k] = s.sU[k][r + 1][fc + 1];
                c2[k] = s.sU[k][r + 1][fc + 2];
                c3[k] = s.sU[k][r + 1][fc + 3];
            }
            if (FASTPHYS)
                face64<SCH, RIE, LIM, 1>(c0, c1, c2, c3, K, hx2, f, nullptr);
            else
                x_face<SCH, RIE, LIM>(c0, c1, c2, c3, g, dt, f);
#pragma unroll
            for (int k = 0; k < 4; k++)
                s.sF[k][r][fc] = f[k];
        }
        else
        {
            int r, c;
            y_face_of<TX, TY>(q, r, c);
#pragma unroll
            for (int k = 0; k < 4; k++)
            {
                c0[k] = s.sU[k][r][c + 2];
                c1[k] = s.sU[k][r + 1][c + 2];
                c2[k] = s.sU[k][r + 2][c + 2];
                c3[k] = s.sU[k][r + 3][c + 2];
            }
            double stray = 0.0;
            int keep = FASTPHYS ? face64<SCH, RIE, LIM, 2>(c0, c1, c2, c3, K, hy2, f, &stray)
                                : y_face<SCH, RIE, LIM>(c0, c1, c2, c3, g, dt, f, &stray);
            if constexpr (RIE == PVRS)
            {
                // the reference's PVRS stray store from cell 7 c' + 2 into this face's
                // energy flux (physics.cuh, pvrs_stray_source)
                const long long lin = (long long)g.M * (j0 - 1 + r) + (i0 + c);
                const long long src = 7 * lin + 2;
                double sv;
                if (i0 + c < g.M && src < (long long)g.M * g.N &&
                    pvrs_stray_source<SCH, LIM>(U, P, pitch, g.M, g.N, g.ng, gam, dt, g.dx, g.dy,
                                                (int)(src % g.M), (int)(src / g.M), &sv))
                {
                    f[3] = sv;
                    keep &= ~8;
                }
            }
#pragma unroll
            for (int k = 0; k < 4; k++)
                s.sG[k][r][c] = f[k];
            s.sKeep[r][c] = (unsigned char)keep;
        }
    }
    __syncthreads();
    // a Y face (i, j - 1/2) that kept the X-face flux of its slot, as the
    // reference's Y solver does in some branches, reads the X face
    // (i + 1/2, j - 1): solved here where the list did not (always for the
    // row below the tile)
    for (int q = tid; q < TX * TY; q += NT)
    {
        const int r = q / TX, c = q - r * TX, fc = c + 1;
        if (!s.sKeep[r][c] || x_face_listed(s.tf, r, fc))
            continue;
        double c0[4], c1[4], c2[4], c3[4], f[4];
#pragma unroll
        for (int k = 0; k < 4; k++)
        {
            c0[k] = s.sU[k][r + 1][fc];
            c1[k] = s.sU[k][r + 1][fc + 1];
            c2[k] = s.sU[k][r + 1][fc + 2];
            c3[k] = s.sU[k][r + 1][fc + 3];
        }
        if (FASTPHYS)
            face64<SCH, RIE, LIM, 1>(c0, c1, c2, c3, K, hx2, f, nullptr);
        else
            x_face<SCH, RIE, LIM>(c0, c1, c2, c3, g, dt, f);
#pragma unroll
        for (int k = 0; k < 4; k++)
            s.sF[k][r][fc] = f[k];
    }
    __syncthreads();

    // update (X then Y, MUSCL_Scheme.cpp:74-88 and :136-150) on fluid cells
    for (int cell = tid; cell < TX * TY; cell += NT)
    {
        const int c = cell % TX, r = cell / TX;
        const int i = i0 + c, j = j0 + r;
        if (tile_cell_fluid(s.tf, r, c))
        {
            const int kp = s.sKeep[r + 1][c], km = s.sKeep[r][c];
            const double lx = FAST ? s.sC[0] : 0.0, ly = FAST ? s.sC[1] : 0.0;
            double v[4];
#pragma unroll
            for (int k = 0; k < 4; k++)
            {
                double gp = ((kp >> k) & 1) ? s.sF[k][r + 1][c + 1] : s.sG[k][r + 1][c];
                double gm = ((km >> k) & 1) ? s.sF[k][r][c + 1] : s.sG[k][r][c];
                if (FAST)
                {
                    double x = s.sU[k][r + 2][c + 2] - lx * (s.sF[k][r + 1][c + 1] - s.sF[k][r + 1][c]);
                    v[k] = x - ly * (gp - gm);
                }
                else
                {
                    double x = s.sU[k][r + 2][c + 2] -
                               divide_rn(dt * (s.sF[k][r + 1][c + 1] - s.sF[k][r + 1][c]), g.by_dx);
                    v[k] = x - divide_rn(dt * (gp - gm), g.by_dy);
                }
            }
            Cell64 cl;
            if constexpr (FASTPHYS)
                if (safeguarded(RIE) || stage == 0)
                    cl = cell64(v);
            if constexpr (safeguarded(RIE))
                pressure_floor64(v, cl);
            if (stage == 2)
            {
                rk2_average(V, (long long)j * pitch + i, P, v);
                if constexpr (FAST)
                    cl = cell64(v);
            }
#pragma unroll
            for (int k = 0; k < 4; k++)
                V[k * P + (long long)j * pitch + i] = v[k];
            if (stage == 1)
                continue;
            // the rows of a tile's upper half are the threads' second cells
            double &mass = (cell < NT) ? cs.mass : cs.mass_upper;
            if (FAST)
                cell_stats_fast(v, cl, K, g.dxdy, cs, mass);
            else
                cell_stats(v, gam, g.dx, g.dy, cs, mass);
        }
    }
    // a copy that missed the first wait is waited for once more (bounded);
    // the barrier is then released for the next tile of a persistent CTA
    if (tmap && tid == 0 && (staged || mbar_wait(&bar, 0)))
        mbar_inval(&bar);
}

// threads of a sweep CTA: one per cell of a 32x8 tile, one for two cells of a 32x16 tile
template <int TX>
constexpr int sweep_threads()
{
    return TX == FINE_X ? FINE_THREADS : TILE_X * TILE_Y;
}
// CTAs per SM the registers are fitted to
template <int RIE, int FAST, int TX>
constexpr int sweep_ctas()
{
    if (RIE == PVRS)
        return 1;
    if (TX == FINE_X)
        return 5;
    return 3;
}

// one case: one CTA per active tile of TX x TY cells.  32x16 tiles in 80
// registers (3 CTAs per SM, 59 KB of shared memory each): with fp64_fast HLL
// 4% faster than 512 threads per tile; HLL_Toro, which had two CTAs of 106
// registers, gains 3% (vortex 1024^2 MHM + RK2 9.47 -> 9.15 ms for eight steps
// when it was changed, a sixth of it from calls in place of if-converted rare
// paths); the strict form: capi.cu, FINE_PARENTS.
template <int SCH, int RIE, int LIM, int FAST, int TX, int TY>
__global__ void __launch_bounds__(sweep_threads<TX>(), sweep_ctas<RIE, FAST, TX>())
    sweep_kernel(const __grid_constant__ SweepArgs a)
{
    constexpr int NT = sweep_threads<TX>();
    extern __shared__ __align__(128) unsigned char smem_raw[];
    auto &s = *reinterpret_cast<SweepSmem64<TX, TY> *>(smem_raw);

    const GridDesc &g = a.g;
    DevState *st = a.st;
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0)
        st->fill_pending = 0;
    // reference loop condition, Test/Sod/Sod.cpp:123
    if (a.guard && !(st->now_t < a.t_end && st->iter < a.max_iter))
        return;
    const double dt = st->dt;
    const int cur = st->cur;
    const double *U = cur ? a.buf1 : a.buf0;
    double *V = cur ? a.buf0 : a.buf1;
    // tiles without fluid cells are skipped: nothing in them is updated or
    // counted by the reference (updates, ComputeDt and CaculateMass all test
    // the cell type), so the launch covers the active tiles only
    const unsigned bid = a.tile0 + blockIdx.x;
    const unsigned tile = a.tiles[bid];
    const int i0 = g.ng + tile_ix(tile) * TX;
    const int j0 = g.ng + tile_jy(tile) * TY;
    const bool interior = (tile & TILE_INTERIOR) != 0;
    CellStats cs;
    sweep_tile64<SCH, RIE, LIM, FAST, TX, TY, NT>(s, g, U, V, a.type, i0, j0, dt, cs, a.stage,
                                                  a.tma ? &a.tmap[cur] : nullptr, &st->status, interior);
    const unsigned nblocks = a.nblocks ? a.nblocks : gridDim.x;
    // a tile's sum has its place by 32x16 tile in the order of the case's list,
    // whatever tiles are swept in whatever order (the row bands of the
    // host-array step: a.slot), so that the mass has the same bits
    constexpr int PARTS = (TX == FINE_X) ? 4 : (RIE == PVRS) ? 2 : 1;
    const MassPartials mp{a.partial, a.slot ? a.nparents : nblocks, a.slot ? PARTS : 1, a.slot ? a.slot[bid] : bid};
    block_reduce_finalize<NT, TX, TY, PARTS == 2>(cs, st, mp, g, true, false, nblocks, a.stage == 1);
}

template <int SCH, int RIE, int LIM, int FAST, int TX, int TY>
void launch_sweep(const SweepArgs &a, int grid, cudaStream_t s)
{
    sweep_kernel<SCH, RIE, LIM, FAST, TX, TY><<<grid, sweep_threads<TX>(), sizeof(SweepSmem64<TX, TY>), s>>>(a);
}

// The launcher of one instantiation.  A 32 x FAST_TILE_Y tile's shared memory
// (59 KB) exceeds the default 48 KB limit: the limit is raised on the current
// device, once per device, when a case picks the launcher (outside any
// stream capture).
template <int SCH, int RIE, int LIM, int FAST, int TX, int TY>
SweepLaunch prepared_sweep_launcher()
{
    constexpr int smem = (int)sizeof(SweepSmem64<TX, TY>);
    if (smem > 48 * 1024)
    {
        static std::atomic<unsigned long long> ready{0};
        int dev = 0;
        cudaGetDevice(&dev);
        const unsigned long long bit = 1ull << (dev & 63);
        if (!(ready.load() & bit))
        {
            cudaFuncSetAttribute(sweep_kernel<SCH, RIE, LIM, FAST, TX, TY>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
            ready.fetch_or(bit);
        }
    }
    return &launch_sweep<SCH, RIE, LIM, FAST, TX, TY>;
}

template <int SCH, int RIE, int FAST>
SweepLaunch select_sweep_tile(bool vl, bool fine)
{
    constexpr int TY = (RIE != PVRS) ? FAST_TILE_Y : TILE_Y;
    if (fine)
        return vl ? prepared_sweep_launcher<SCH, RIE, VANLEER, FAST, FINE_X, FINE_Y>()
                  : prepared_sweep_launcher<SCH, RIE, MINMOD, FAST, FINE_X, FINE_Y>();
    return vl ? prepared_sweep_launcher<SCH, RIE, VANLEER, FAST, TILE_X, TY>()
              : prepared_sweep_launcher<SCH, RIE, MINMOD, FAST, TILE_X, TY>();
}

// the sweep of one scheme in strict FP64 (FAST = 0) or fp64_fast over 32x16
// tiles (with PVRS 32x8), or (fine) over FINE_X x FINE_Y tiles
template <int SCH, int FAST>
SweepLaunch select_sweep(int riemann, int limiter, bool fine)
{
    const bool vl = (limiter == VANLEER);
    switch (riemann)
    {
    case PVRS: return select_sweep_tile<SCH, PVRS, FAST>(vl, fine);
    case SW: return select_sweep_tile<SCH, SW, FAST>(vl, fine);
    case HLLCT: return select_sweep_tile<SCH, HLLCT, FAST>(vl, fine);
    case HLLT: return select_sweep_tile<SCH, HLLT, FAST>(vl, fine);
    default: return select_sweep_tile<SCH, HLL, FAST>(vl, fine);
    }
}

} // namespace ibtfo
