// Strips of a mesh of one level: index helpers of the fused step kernels
// (fcb_step_adv.cuh, fcb_step_split.cuh) and the choice of their size.
//
// Why strips: a patch of mx cells a side sweeps mx + 4 columns over mx + 7 rows (ghost
// cells, pipeline), 1.8 cells of work per cell at mx = 16 and 2.8 at mx = 8; a strip of
// 121 columns over 241 rows 1.07.  Swirl advection, level 8, mx = 16, one step on B200:
// FP64 0.508 ms with fused patches, 0.369 ms in strips with the same kernel (0.274 ms
// with a kernel made for them, fcb_step_adv.cuh); mixed 0.375, 0.272 and 0.196 ms;
// shallow water, 1024 x 1024 cells: 0.139 (mx = 32), 0.178 (16), 0.214 ms (8) in patches
// and a ghost fill of 0.02 to 0.03 ms, 0.120 ms in strips.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "fcb_device.h"

namespace fcb {

namespace {

// Strip form (ghost-exchange fusion on a mesh of one level): the mesh is cut into
// strips of columns and rows without regard to patch edges, and a strip is swept
// like one large patch.  The ghost update that precedes a step on such a mesh
// (fclaw2d_ghost_update_async, one rank) only copies neighbours' interior cells
// (fclaw2d_clawpatch46_fort_copy_face/_corner) and applies the physical boundary
// conditions (clawpack46_bc2_default.f) left, right, bottom, top, each over the whole
// band; so the cell left of a patch's first column is simply the previous column
// of the mesh, and outside the domain a cell takes column 1 / mx (extrapolation),
// the mirrored column (wall, component 2 negated) or the opposite side
// (periodic); rows likewise with component 3.
//
// Mesh column or row k of [-2, n + 2) -> the one inside that holds its value.
__device__ __forceinline__ int strip_inside(int k, int n, int bc_lo, int bc_hi, bool& wall) {
    wall = false;
    if (k < 0) {
        if (bc_lo == 3) { wall = true; return -1 - k; }
        return bc_lo == 0 ? k + n : 0;
    }
    if (k >= n) {
        if (bc_hi == 3) { wall = true; return 2 * n - 1 - k; }
        return bc_hi == 0 ? k - n : n - 1;
    }
    return k;
}

// Slot of the patch that holds mesh cell (x, y), inside the domain.
__device__ __forceinline__ int strip_slot(const StripArgs& g, int x, int y) {
    return __ldg(g.grid + ((y >> g.lg) << g.lgp) + (x >> g.lg));
}

// Offset of mesh cell (x, y) in its slot.
__device__ __forceinline__ int strip_cell(const StripArgs& g, int x, int y) {
    const int mask = (1 << g.lg) - 1;
    return ((y & mask) + 2) * g.nxp + (x & mask) + 2;
}

// Stored aux (component k) of mesh cell (x, y) of [-2, n + 2)^2: outside the domain
// the edge patch's own ghost aux (aux is a function of the cell centre, set in
// the ghost cells too).
__device__ __forceinline__ double strip_aux(const StepArgs& a, int x, int y, int k) {
    const StripArgs& g = a.strip;
    const int px = min(max(x, 0), g.n - 1) >> g.lg, py = min(max(y, 0), g.n - 1) >> g.lg;
    const int slot = __ldg(g.grid + (py << g.lgp) + px);
    return a.aux[(int64_t)slot * a.aux_stride + (k * g.nxp + y - (py << g.lg) + 2) * g.nxp + (x - (px << g.lg) + 2)];
}

constexpr int kStripRowsMax = 2048;  // bounds a strip's tables in shared memory

// Strip width and height of a mesh of n x n cells for strips of at most `most`
// columns on a chip that holds per_wave of them at once.  A strip of h rows
// takes h + extra row-iterations (ghost rows, pipeline), so few tall strips do the
// least work and many short ones finish soonest: of the heights that give 1, 2, ...
// full waves, the one whose waves x iterations is least.
inline void strip_plan(StripArgs& g, int most, int per_wave, int extra) {
    g.nsx = (g.n + most - 1) / most;
    g.w = (g.n + g.nsx - 1) / g.nsx;
    g.nsx = (g.n + g.w - 1) / g.w;
    long best = -1;
    for (int waves = 1; waves <= 64; ++waves) {
        const int nsy = std::max(1, (int)((long)waves * per_wave / g.nsx));
        const int h = std::max(std::min(g.n, 2), (g.n + nsy - 1) / nsy);
        if (h > kStripRowsMax) continue;
        const long ctas = (long)g.nsx * ((g.n + h - 1) / h);
        const long cost = (ctas + per_wave - 1) / per_wave * (h + extra);
        if (best < 0 || cost < best) {
            best = cost;
            g.h = h;
        }
    }
    g.nsy = (g.n + g.h - 1) / g.h;
}

}  // namespace

}  // namespace fcb
