// Sums over the particles of the sort cells around a fluid cell, by one warp,
// in the order of the reference's loops.
//
// The porosity kernels visit the particles of 27 (Darcy) or 125
// (Navier-Stokes) cells around each cell, one thread per cell in the
// reference: several hundred visits in a chain, and only the cells inside the
// packing have any.  Here a warp takes a cell: the lanes visit 32 particles at
// a time and queue, in visiting order, those that contribute; the queue is
// evaluated 32 at a time, and one lane per sum adds the terms in that order
// (leaving out a zero changes nothing in a sum that started at +0), so the sums
// are the same bits.  Blocks of 8 warps take 32 fluid cells: cells with no
// particle around them, most of a consolidation's grid, are found with one lane
// each and need no warp.
#pragma once

#include "dem_device.cuh"

namespace sphb {

// Scratch of a warp of gather_cells.
struct GatherScratch {
    double term[5 * 32];
    uint32_t queue[64];      // sorted index | periodic shift code << 28
};

// Visits the particles of the `ncell` cells that cell_at(l, cx, cy, cz) names
// (coordinates before wrapping; false: none), in the order of l and of the sort.  near(i,
// dm): whether particle i, with periodic shift dm, contributes; eval(i, dm, t)
// computes its five terms.  Lane c < 5 returns sum c; sum 0 starts at `first`
// and its terms are subtracted with `neg`.
template <class Cell, class Near, class Eval>
__device__ __forceinline__ double gather_cells(const DevParams &P, const DevState &S, unsigned ncell,
                                               double first, bool neg, GatherScratch &W, Cell &&cell_at,
                                               Near &&near, Eval &&eval)
{
    constexpr unsigned ALL = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31u;
    double acc = lane == 0 ? first : 0.0;
    unsigned queued = 0;
    auto flush = [&](unsigned n) {   // the first n <= 32 entries of the queue
        __syncwarp();
        if (lane < n) {
            const uint32_t e = W.queue[lane];
            double t[5];
            eval(e & 0x0fffffffu, dm_decode(P, (uint8_t)(e >> 28)), t);
#pragma unroll
            for (int c = 0; c < 5; ++c) W.term[c * 32 + lane] = t[c];
        }
        __syncwarp();
        if (lane < 5u)
            for (unsigned q = 0; q < n; ++q) {
                const double v = W.term[lane * 32u + q];
                acc += neg && lane == 0u ? -v : v;
            }
        __syncwarp();
    };
    for (unsigned g = 0; g < ncell; g += 32u) {
        unsigned start = 0, count = 0, code = 0;
        int cx, cy, cz, sx, sy;
        if (g + lane < ncell && cell_at(g + lane, cx, cy, cz) && wrap_cell(P, cx, cy, cz, sx, sy)) {
            const unsigned cell = (unsigned)cx + (unsigned)cy * P.num[0] + (P.num[0] * P.num[1]) * (unsigned)cz;
            const unsigned s = S.cell_start[cell];
            if (s != 0xffffffffu) {
                start = s;
                count = S.cell_end[cell] - s;
                code = dm_encode(sx, sy);
            }
        }
        if (!__any_sync(ALL, count != 0u)) continue;
        const unsigned end = warp_inclusive_sum(count);
        const unsigned total = __shfl_sync(ALL, end, 31);
        const unsigned base = start - (end - count);   // visit number -> sorted index
        for (unsigned r0 = 0; r0 < total; r0 += 32u) {
            const unsigned item = r0 + lane;
            // the cell of this visit: the number of cells whose visits end before it
            unsigned l = 0;
#pragma unroll
            for (unsigned step = 16; step; step >>= 1) {
                const unsigned e = __shfl_sync(ALL, end, l + step - 1u);
                if (e <= item) l += step;
            }
            l &= 31u;
            const unsigned i = __shfl_sync(ALL, base, l) + item, c = __shfl_sync(ALL, code, l);
            const bool hit = item < total && near(i, dm_decode(P, (uint8_t)c));
            const unsigned m = __ballot_sync(ALL, hit);
            if (hit) W.queue[queued + __popc(m & ((1u << lane) - 1u))] = i | c << 28;
            queued += __popc(m);
            if (queued >= 32u) {
                flush(32u);
                queued -= 32u;
                // the rest moves to the front: written by the lanes that hold it
                // alone, before any lane queues behind it
                const uint32_t e = W.queue[32u + lane];
                __syncwarp();
                if (lane < queued) W.queue[lane] = e;
                __syncwarp();
            }
        }
    }
    if (queued) flush(queued);
    return acc;
}

// For the 32 cells base .. base + 31 of a block of 8 warps (n cells in all):
// which have a particle in one of the cells that cell_at(cell, l, ...) names.
template <class Cell>
__device__ __forceinline__ unsigned cells_with_particles(const DevParams &P, const DevState &S, unsigned base,
                                                         unsigned n, unsigned ncell, Cell &&cell_at)
{
    __shared__ unsigned found;
    const unsigned lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) found = 0u;
    __syncthreads();
    bool any = false;
    if (base + lane < n)
        for (unsigned l = w; l < ncell; l += 8u) {
            int cx, cy, cz, sx, sy;
            if (cell_at(base + lane, l, cx, cy, cz) && wrap_cell(P, cx, cy, cz, sx, sy))
                any |= S.cell_start[(unsigned)cx + (unsigned)cy * P.num[0] +
                                    (P.num[0] * P.num[1]) * (unsigned)cz] != 0xffffffffu;
        }
    const unsigned m = __ballot_sync(0xffffffffu, any);
    if (lane == 0 && m) atomicOr(&found, m);
    __syncthreads();
    return found;
}

}  // namespace sphb
