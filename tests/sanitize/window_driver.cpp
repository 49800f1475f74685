// Host-code driver run under AddressSanitizer and UndefinedBehaviorSanitizer
// (tests/test_agent_window.py): the runs of cells that a force window is walked
// as (hal-cpp_gb300/csrc/agent_window.h) against the cells that the CPU backend
// visits, in its order, for windows inside, across and wholly outside the grid.
// Every run's two offsets are read from an array of the grid's size.
#include "agent_window.h"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <vector>

namespace
{
    int32_t Mod(int64_t i, int32_t dim)
    {
        const int32_t m = static_cast<int32_t>(i % dim);
        return m < 0 ? m + dim : m;
    }
}

int main()
{
    using namespace halcuda;
    const int32_t sides[] = {1, 2, 3, 5, 7, 8, 24, 64};
    const double radii[] = {1e-3, 0.75, 1.0, 1.5, 2.0, 3.5, 6.0};
    long windows = 0, runsSeen = 0;
    for (int32_t xDim : sides)
    {
        for (int32_t yDim : sides)
        {
            std::vector<int32_t> offsets(static_cast<size_t>(xDim) * yDim + 1);
            for (size_t c = 0; c < offsets.size(); c++)
            {
                offsets[c] = static_cast<int32_t>(c);  // one agent per cell
            }
            for (double R : radii)
            {
                const auto at = [&](int32_t dim) {
                    return std::vector<double>{-1e9,      -1000.0,   -3.0 * dim,   -dim - 3.0, -dim - 0.5, -5.5,
                                               -R - 1.0,  -R,        -0.5,         0.0,        0.25 * dim, 0.5 * dim,
                                               dim - 0.5, 1.0 * dim, dim + R,      dim + 0.25, dim + R + 2, 2.0 * dim + 1,
                                               3.0 * dim, 1e6 + 0.5, 2147483520.0, 1e12,       -1e12};
                };
                for (int wrap = 0; wrap < 4; wrap++)
                {
                    for (double x : at(xDim))
                    {
                        for (double y : at(yDim))
                        {
                            const auto cast = [](double v) {
                                return static_cast<int32_t>(std::min(std::max(v, -2147483648.0), 2147483647.0));
                            };
                            int32_t x0 = cast(std::floor(x - R)), x1 = cast(std::ceil(x + R));
                            int32_t y0 = cast(std::floor(y - R)), y1 = cast(std::ceil(y + R));
                            if (!(wrap & 1))
                            {
                                x0 = std::max(x0, 0);
                                x1 = std::min(x1, xDim);
                            }
                            if (!(wrap & 2))
                            {
                                y0 = std::max(y0, 0);
                                y1 = std::min(y1, yDim);
                            }
                            std::vector<int32_t> want, got;
                            for (int64_t i = x0; i < x1; i++)
                            {
                                for (int64_t j = y0; j < y1; j++)
                                {
                                    want.push_back(Mod(i, xDim) * yDim + Mod(j, yDim));
                                }
                            }
                            WindowRuns w;
                            w.Set(x0, x1, y0, y1, yDim);
                            windows++;
                            if (!w.fits)
                            {
                                // only what does not fit may be refused
                                if (static_cast<int64_t>(y1) - y0 <= yDim)
                                {
                                    std::printf("refused: %d x %d, R %g, (%g, %g)\n", xDim, yDim, R, x, y);
                                    return 1;
                                }
                                continue;
                            }
                            for (int32_t j = 0; j < w.runs; j++)
                            {
                                int32_t cell, count;
                                w.Run(j, x0, xDim, yDim, cell, count);
                                for (int32_t q = offsets.at(static_cast<size_t>(cell));
                                     q < offsets.at(static_cast<size_t>(cell + count)); q++)
                                {
                                    got.push_back(q);
                                }
                                runsSeen++;
                            }
                            if (got != want)
                            {
                                std::printf("cells differ: %d x %d, R %g, (%g, %g), wrap %d\n", xDim, yDim, R, x, y, wrap);
                                return 1;
                            }
                        }
                    }
                }
            }
        }
    }
    std::printf("ok %ld windows, %ld runs\n", windows, runsSeen);
    return 0;
}
