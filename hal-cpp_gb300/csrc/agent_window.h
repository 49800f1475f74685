// agent_window.h -- the cells of an agent's force window as runs of cells.
//
// The CPU backend visits the window's cells x-major then y, each index taken
// modulo its side where that axis wraps (CpuAgentForceBackend2D.cpp:112-175).
// Cells of one row are consecutive, and so are their agents' slots, so a row is
// one run of cells, or two where its y-range passes the edge.  Host and device
// code, so that the index arithmetic can be checked without a GPU.
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define HAL_WINDOW_FN __host__ __device__ __forceinline__
#else
#define HAL_WINDOW_FN inline
#endif

namespace halcuda
{
    // i modulo dim, in [0, dim).
    HAL_WINDOW_FN int32_t WrapIndex(int32_t i, int32_t dim)
    {
        if (i < 0 || i >= dim)
        {
            i %= dim;
            i += (i < 0) ? dim : 0;
        }
        return i;
    }

    // The rows xStart .. xEnd - 1 of a window, each with the cells yStart ..
    // yEnd - 1, as `runs` runs: run j is cells [cell, cell + count).
    struct WindowRuns
    {
        int32_t runs;    // 0: no cells
        int32_t perRow;  // 1, or 2 where the y-range passes the edge
        int32_t y0;      // the y-range reduced into the grid: `first` cells from y0 on,
        int32_t first;   // and `over` cells from 0 on
        int32_t over;
        bool fits;       // the y-range is no longer than the side, so the runs are the whole window

        // On an axis that does not wrap the range lies within the grid.  An
        // agent may lie anywhere (the binning clamps it), so that a window may
        // lie wholly outside, by any number of sides: it is reduced first, and
        // only then cut at the edge.
        HAL_WINDOW_FN void Set(int32_t xStart, int32_t xEnd, int32_t yStart, int32_t yEnd, int32_t yDim)
        {
            // (unsigned: the bounds may be the ends of int32's range)
            const uint32_t rows = static_cast<uint32_t>(xEnd) - static_cast<uint32_t>(xStart);
            const uint32_t cells = static_cast<uint32_t>(yEnd) - static_cast<uint32_t>(yStart);
            runs = 0;
            perRow = 1;
            y0 = first = over = 0;
            fits = true;
            if (xEnd <= xStart || yEnd <= yStart)
            {
                return;
            }
            if (cells > static_cast<uint32_t>(yDim) || rows > (uint32_t(1) << 29))
            {
                fits = false;
                return;
            }
            y0 = WrapIndex(yStart, yDim);
            const int32_t n = static_cast<int32_t>(cells), left = yDim - y0;
            first = (n < left) ? n : left;
            over = n - first;
            perRow = (over > 0) ? 2 : 1;
            runs = static_cast<int32_t>(rows) * perRow;
        }

        // Run j (0 <= j < runs), in the visiting order.
        HAL_WINDOW_FN void Run(int32_t j, int32_t xStart, int32_t xDim, int32_t yDim, int32_t &cell,
                               int32_t &count) const
        {
            const bool second = perRow == 2 && (j & 1) != 0;
            const int32_t row = WrapIndex(xStart + (perRow == 2 ? j >> 1 : j), xDim);
            cell = row * yDim + (second ? 0 : y0);
            count = second ? over : first;
        }
    };
}
