// The persistent batched sweep: CTAs (a fixed grid of resident CTAs) walk
// one tile table that holds the active tiles of every case of a batch.  Each
// tile runs the same tile body as the one-case kernels (sweep_tile64 /
// sweep_tile32), so a case advances bit for bit as it does alone with the
// same tile shape; its statistics go to its own device state, and the last
// of its tiles to finish computes its next dt (per-case dt and loop
// accounting, Test/Sod/Sod.cpp:123-176).  Cases whose loop has ended
// (now_t >= t_end or iter >= max_iter) are skipped tile by tile.
#pragma once

#include "sweep_f32_impl.cuh"
#include "sweep_impl.cuh"

namespace ibtfo {

template <int SCH, int RIE, int LIM, int PREC, int TX, int TY>
__global__ void __launch_bounds__(f32_threads<SCH, RIE, PREC>(), (PREC == 2 && RIE == HLLT) ? 3 : 1)
    batch_sweep_kernel(const BatchHeader *__restrict__ h, int stage)
{
    constexpr int NT = f32_threads<SCH, RIE, PREC>();
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int ntiles = h->ntiles;
    // the FP32 difference form stages its next tile while it commits the last
    __shared__ uint64_t bar;
    TileStager ts{&bar, 0u, false, false};
    if constexpr (PREC == 2 && RIE == HLLT)
    {
        if (threadIdx.x == 0)
            mbar_init(&bar, 1);
        __syncthreads();
    }
    // the copy of the first tile from `t` on whose case still runs
    const auto next_box = [&](int t) {
        StageBox b{};
        for (; t < ntiles; t += gridDim.x)
        {
            const BatchTile e = h->tiles[t];
            const SweepArgs &a = h->cases[e.z].s;
            if (!(a.st->now_t < a.t_end && a.st->iter < a.max_iter))
                continue;
            if (!a.tma || TX != TILE_X || TY != FAST_TILE_Y)
                break;
            const int cur = a.st->cur;
            b.map = &a.tmap[cur];
            tensormap_acquire(b.map);
            if (stage == 2)
            {
                b.vmap = &a.tmap[cur ^ 1];
                tensormap_acquire(b.vmap);
            }
            b.x = a.g.ng + tile_ix(e.x) * TX - 2;
            b.y = a.g.ng + tile_jy(e.x) * TY - 2;
            break;
        }
        return b;
    };
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x)
    {
        const BatchTile e = h->tiles[t];
        const BatchCase &bc = h->cases[e.z];
        const SweepArgs &a = bc.s;
        DevState *st = a.st;
        if (e.y == 0 && threadIdx.x == 0)
            st->fill_pending = 0;
        // the case's tiles of this launch all read the same state: its
        // accounting changes only when the last of them has finished
        if (!(st->now_t < a.t_end && st->iter < a.max_iter))
            continue;
        const double dt = st->dt;
        const int cur = st->cur;
        const GridDesc &g = a.g;
        const int i0 = g.ng + tile_ix(e.x) * TX;
        const int j0 = g.ng + tile_jy(e.x) * TY;
        const bool interior = (e.x & TILE_INTERIOR) != 0;
        // the case's own tensor maps describe boxes of its one-case tiles
        // (32x16 except under PVRS): the 32x16 shape stages tiles with them
        const CUtensorMap *tm = nullptr;
        if constexpr (TX == TILE_X && TY == FAST_TILE_Y && RIE != PVRS)
            if (a.tma)
            {
                tm = &a.tmap[cur];
                if (threadIdx.x == 0 && !ts.issued)
                {
                    tensormap_acquire(tm);
                    if (stage == 2)
                        tensormap_acquire(&a.tmap[cur ^ 1]);
                }
            }
        int *status = tm ? &st->status : nullptr;
        if constexpr (PREC == 2)
        {
            const float *U = reinterpret_cast<const float *>(cur ? a.buf1 : a.buf0);
            float *V = reinterpret_cast<float *>(cur ? a.buf0 : a.buf1);
            CellStats32 cs;
            if constexpr (RIE == HLLT)
                sweep_tile32_delta<SCH, RIE, LIM, TX, TY, NT>(*reinterpret_cast<SweepSmem32D<TX, TY> *>(smem_raw), g,
                                                              U, V, a.type, i0, j0, dt, cs, stage,
                                                              StageBox{tm, stage == 2 ? &a.tmap[cur ^ 1] : nullptr,
                                                                       i0 - 2, j0 - 2},
                                                              ts, [&] { return next_box(t + gridDim.x); }, status,
                                                              interior);
            else
                sweep_tile32<SCH, RIE, LIM, TX, TY, NT>(*reinterpret_cast<SweepSmem32<TX, TY> *>(smem_raw), g, U, V,
                                                        a.type, i0, j0, dt, cs, stage, tm, status, interior);
            block_reduce_finalize32<NT>(cs, st, a.partial, g, (unsigned)bc.ntiles, e.y, stage == 1);
        }
        else
        {
            auto &s = *reinterpret_cast<SweepSmem64<TX, TY> *>(smem_raw);
            const double *U = cur ? a.buf1 : a.buf0;
            double *V = cur ? a.buf0 : a.buf1;
            CellStats cs;
            sweep_tile64<SCH, RIE, LIM, 1, TX, TY, NT>(s, g, U, V, a.type, i0, j0, dt, cs, stage, tm, status,
                                                       interior);
            block_reduce_finalize<NT, TX, TY>(cs, st, {a.partial, (unsigned)bc.ntiles, 1, e.y}, g, true, false,
                                              (unsigned)bc.ntiles, stage == 1);
        }
    }
}

template <int SCH, int RIE, int LIM, int PREC, int TX, int TY>
struct BatchVariant
{
    static constexpr size_t smem()
    {
        return PREC == 2 ? sizeof(Smem32<RIE, TX, TY>) : sizeof(SweepSmem64<TX, TY>);
    }
    static void launch(const BatchHeader *h, int grid, cudaStream_t s, int stage)
    {
        batch_sweep_kernel<SCH, RIE, LIM, PREC, TX, TY><<<grid, f32_threads<SCH, RIE, PREC>(), smem(), s>>>(h, stage);
    }
    static int prepare()
    {
        auto k = batch_sweep_kernel<SCH, RIE, LIM, PREC, TX, TY>;
        if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem()) != cudaSuccess)
            return 0;
        int n = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, f32_threads<SCH, RIE, PREC>(), smem()) != cudaSuccess)
            return 0;
        return n;
    }
};

template <int SCH, int RIE, int LIM, int PREC>
BatchKernel batch_kernel_shape(int shape)
{
    switch (shape)
    {
    case SHAPE_32x16:
        return {&BatchVariant<SCH, RIE, LIM, PREC, 32, 16>::launch, &BatchVariant<SCH, RIE, LIM, PREC, 32, 16>::prepare};
    case SHAPE_64x8:
        return {&BatchVariant<SCH, RIE, LIM, PREC, 64, 8>::launch, &BatchVariant<SCH, RIE, LIM, PREC, 64, 8>::prepare};
    default:
        return {&BatchVariant<SCH, RIE, LIM, PREC, 32, 8>::launch, &BatchVariant<SCH, RIE, LIM, PREC, 32, 8>::prepare};
    }
}

// every (Riemann solver, limiter) of one scheme and precision; PVRS has no
// FP32 form
template <int SCH, int PREC>
BatchKernel batch_kernel_scheme(int riemann, int limiter, int shape)
{
    const bool vl = (limiter == VANLEER);
    switch (riemann)
    {
    case PVRS:
        if constexpr (PREC == 2)
            return {nullptr, nullptr};
        else
            return vl ? batch_kernel_shape<SCH, PVRS, VANLEER, PREC>(shape)
                      : batch_kernel_shape<SCH, PVRS, MINMOD, PREC>(shape);
    case SW:
        return vl ? batch_kernel_shape<SCH, SW, VANLEER, PREC>(shape) : batch_kernel_shape<SCH, SW, MINMOD, PREC>(shape);
    case HLLCT:
        return vl ? batch_kernel_shape<SCH, HLLCT, VANLEER, PREC>(shape)
                  : batch_kernel_shape<SCH, HLLCT, MINMOD, PREC>(shape);
    case HLLT:
        return vl ? batch_kernel_shape<SCH, HLLT, VANLEER, PREC>(shape)
                  : batch_kernel_shape<SCH, HLLT, MINMOD, PREC>(shape);
    default:
        return vl ? batch_kernel_shape<SCH, HLL, VANLEER, PREC>(shape) : batch_kernel_shape<SCH, HLL, MINMOD, PREC>(shape);
    }
}

} // namespace ibtfo
