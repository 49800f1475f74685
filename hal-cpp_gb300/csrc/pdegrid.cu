// pdegrid.cu -- a device-resident Hal::PDEGrid2D (include/Hal/Grids/PDEGrid2D.h).
//
// PDEGrid2D keeps a committed field and a delta buffer: Get reads the field,
// Set/Add/Mul/Scale and the PDE operators accumulate into the deltas, and
// Update commits them (PDEGrid2D.h:17-186).  This handle keeps both buffers in
// HBM in FP64 and reproduces every call bit for bit:
//   * per-cell operations arrive as lists (from the host, or one per agent of
//     an agent handle's last binning); entries of one cell are applied by one
//     thread in list order, so repeated cells accumulate exactly as a loop of
//     single calls does;
//   * the explicit stencils are the FP64 functors of the interface path
//     (IEEE operations in the reference's order);
//   * DiffusionADI is the reference's Thomas solve per line
//     (include/Hal/Pde/ADIequations.h:225-337, TdmaSolver.h:26-120) in FP64.
//     Its matrix is the same for every line of a sweep, so the modified
//     diagonal, the elimination multipliers and, on a periodic axis, the
//     Sherman-Morrison vector are computed once on the host with the
//     reference's operations; each line then runs the right-hand-side part
//     of the elimination and the back substitution, one thread per line, in
//     the reference's order.  The x-sweep reads its lines across the
//     contiguous y index (coalesced); its output is transposed so that the
//     y-sweep reads coalesced too, and the y-sweep's result is transposed
//     back while it is added into the deltas.
#include "common.cuh"
#include "adi64.h"
#include "stencil64.cuh"
#include "agents_wells.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <limits>
#include <map>
#include <memory>
#include <numeric>
#include <vector>

using namespace halcuda::stencil64;

namespace halcuda
{
    namespace
    {
        // ---- per-cell operations (PDEGrid2D.h:88-140) ---------------------
        constexpr int kOpSet = HAL_CUDA_CELL_SET;
        constexpr int kOpAdd = HAL_CUDA_CELL_ADD;
        constexpr int kOpMul = HAL_CUDA_CELL_MUL;
        constexpr int kOpScale = HAL_CUDA_CELL_SCALE;

        // One operation on a cell's delta d given its committed value f:
        // Set d = v - f, Add d += v, Mul d += f * v, Scale d += f * (v - 1).
        __device__ __forceinline__ double ApplyOp(int op, double d, double f, double v)
        {
            switch (op)
            {
            case kOpSet:
                return __dsub_rn(v, f);
            case kOpAdd:
                return __dadd_rn(d, v);
            case kOpMul:
                return __dadd_rn(d, __dmul_rn(f, v));
            default:
                return __dadd_rn(d, __dmul_rn(f, __dsub_rn(v, 1.0)));
            }
        }

        // Runs of a cell-sorted operation list: run r covers entries
        // [runStart[r], runStart[r + 1]) of one cell, in list order.
        __global__ void ApplyRuns(const int32_t *__restrict__ cells, const int8_t *__restrict__ ops,
                                  const double *__restrict__ vals, const int32_t *__restrict__ runStart, int32_t nRuns,
                                  const double *__restrict__ f, double *__restrict__ deltas)
        {
            const int32_t r = blockIdx.x * blockDim.x + threadIdx.x;
            if (r >= nRuns)
            {
                return;
            }
            const int32_t s = runStart[r], e = runStart[r + 1];
            const int64_t c = cells[s];
            const double fc = f[c];
            double d = deltas[c];
            for (int32_t k = s; k < e; k++)
            {
                d = ApplyOp(ops[k], d, fc, vals[k]);
            }
            deltas[c] = d;
        }

        // One operation per agent of a binning, each at its agent's cell, in
        // agent index order within a cell (the bucket order): the thread of
        // the first slot of each occupied cell applies the cell's agents.
        __global__ void ApplyAgents(const int32_t *__restrict__ offsets, const int32_t *__restrict__ bucket,
                                    const int32_t *__restrict__ cellOf, int32_t n, int op, double value,
                                    const double *__restrict__ perAgent, const double *__restrict__ f,
                                    double *__restrict__ deltas)
        {
            const int32_t s = blockIdx.x * blockDim.x + threadIdx.x;
            if (s >= n)
            {
                return;
            }
            const int32_t c = cellOf[bucket[s]];
            if (offsets[c] != s)
            {
                return;
            }
            const int32_t e = offsets[c + 1];
            const double fc = f[c];
            double d = deltas[c];
            for (int32_t k = s; k < e; k++)
            {
                d = ApplyOp(op, d, fc, perAgent != nullptr ? perAgent[bucket[k]] : value);
            }
            deltas[c] = d;
        }

        // SetAll / AddAll / MulAll (PDEGrid2D.h:188-217): the operation at
        // every cell, the value a scalar or (SetAll(pVals)) one per cell.
        __global__ void ApplyAll(int op, double value, const double *__restrict__ perCell, int64_t n,
                                 const double *__restrict__ f, double *__restrict__ deltas)
        {
            for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
                 i += static_cast<int64_t>(gridDim.x) * blockDim.x)
            {
                deltas[i] = ApplyOp(op, deltas[i], f[i], perCell != nullptr ? perCell[i] : value);
            }
        }

        // Update (PDEGrid2D.h:178-186): field += deltas, deltas = 0.
        __global__ void Commit(int64_t n, double *__restrict__ f, double *__restrict__ deltas)
        {
            for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
                 i += static_cast<int64_t>(gridDim.x) * blockDim.x)
            {
                f[i] = __dadd_rn(f[i], deltas[i]);
                deltas[i] = 0.0;
            }
        }

        // A value-form SetAll / AddAll / MulAll deferred to the Update right
        // after it, in one pass: deltas = op(deltas, field, value), then
        // field += deltas and deltas = 0, the two kernels' operations in
        // their order.
        __global__ void ApplyAllCommit(int op, double value, int64_t n, double *__restrict__ f,
                                       double *__restrict__ deltas)
        {
            for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
                 i += static_cast<int64_t>(gridDim.x) * blockDim.x)
            {
                const double fi = f[i];
                const double d = ApplyOp(op, deltas[i], fi, value);
                f[i] = __dadd_rn(fi, d);
                deltas[i] = 0.0;
            }
        }

        // SetNonNegative (PDEGrid2D.h:244-255): Set(i, 0) where f + d < 0.
        __global__ void NonNegative(int64_t n, const double *__restrict__ f, double *__restrict__ deltas)
        {
            for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
                 i += static_cast<int64_t>(gridDim.x) * blockDim.x)
            {
                if (__dadd_rn(f[i], deltas[i]) < 0.0)
                {
                    deltas[i] = __dsub_rn(0.0, f[i]);
                }
            }
        }

        __global__ void Gather(const int32_t *__restrict__ cells, int64_t n, const double *__restrict__ f,
                               double *__restrict__ out)
        {
            const int64_t k = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
            if (k < n)
            {
                out[k] = f[cells[k]];
            }
        }

        // ---- reductions: GetMax, GetMin, GetAvg, MaxDelta, MaxDeltaScaled ----
        // GetMax keeps max = (f < max) ? max : f over the cells in order, so
        // of equal values (+0 and -0 compare equal) the last one is kept; the
        // reduction carries the index to keep the same one.  GetMin likewise.
        struct Extreme
        {
            double v;
            int64_t i;
        };

        __device__ __forceinline__ Extreme MaxOf(Extreme a, Extreme b)  // a before b or after: by index
        {
            if (a.v < b.v)
            {
                return b;
            }
            if (b.v < a.v)
            {
                return a;
            }
            return (a.i > b.i) ? a : b;
        }

        __device__ __forceinline__ Extreme MinOf(Extreme a, Extreme b)
        {
            if (b.v < a.v)
            {
                return b;
            }
            if (a.v < b.v)
            {
                return a;
            }
            return (a.i > b.i) ? a : b;
        }

        constexpr int kRedThreads = 256;
        constexpr int kRedBlocks = 592;  // 4 per SM on 148-152 SMs

        // Per block: the extremes of its cells, the sum of the field (in a
        // fixed order, so the result is deterministic), max |d| and max
        // |d / (|f| + offset)|.  Partials go to out[block]; the host combines
        // them in block order.
        struct RedPartial
        {
            double maxV, minV, sum, maxDelta, maxScaled;
            long long maxI, minI;
        };

        __global__ void __launch_bounds__(kRedThreads) Reduce(int64_t n, const double *__restrict__ f,
                                                              const double *__restrict__ deltas, double offset,
                                                              bool scaled, RedPartial *__restrict__ out)
        {
            const int64_t chunk = (n + gridDim.x - 1) / gridDim.x;
            const int64_t lo = blockIdx.x * chunk;
            const int64_t hi = (lo + chunk < n) ? lo + chunk : n;
            Extreme mx = {-INFINITY, -1}, mn = {INFINITY, -1};
            double sum = 0.0, md = 0.0, ms = 0.0;
            for (int64_t i = lo + threadIdx.x; i < hi; i += blockDim.x)
            {
                const double fv = f[i];
                const double dv = deltas[i];
                mx = MaxOf(mx, Extreme{fv, i});
                mn = MinOf(mn, Extreme{fv, i});
                sum = __dadd_rn(sum, fv);
                md = fmax(md, fabs(dv));
                if (scaled)
                {
                    ms = fmax(ms, fabs(__ddiv_rn(dv, __dadd_rn(fabs(fv), offset))));
                }
            }
            __shared__ RedPartial sh[kRedThreads];
            sh[threadIdx.x] = RedPartial{mx.v, mn.v, sum, md, ms, mx.i, mn.i};
            __syncthreads();
            for (int w = kRedThreads / 2; w > 0; w >>= 1)
            {
                if (threadIdx.x < w)
                {
                    RedPartial a = sh[threadIdx.x], b = sh[threadIdx.x + w];
                    const Extreme xm = MaxOf(Extreme{a.maxV, a.maxI}, Extreme{b.maxV, b.maxI});
                    const Extreme xn = MinOf(Extreme{a.minV, a.minI}, Extreme{b.minV, b.minI});
                    a.maxV = xm.v;
                    a.maxI = xm.i;
                    a.minV = xn.v;
                    a.minI = xn.i;
                    a.sum = __dadd_rn(a.sum, b.sum);
                    a.maxDelta = fmax(a.maxDelta, b.maxDelta);
                    a.maxScaled = fmax(a.maxScaled, b.maxScaled);
                    sh[threadIdx.x] = a;
                }
                __syncthreads();
            }
            if (threadIdx.x == 0)
            {
                out[blockIdx.x] = sh[0];
            }
        }

        // GradientX/GradientY (PDEGrid2D.h:257-285) at query points:
        // DisplacedField(x+1) - DisplacedField(x-1), off-grid the cell's own
        // value (reflecting) or a boundary value.
        __device__ __forceinline__ double DisplacedField(const double *f, int32_t a, int32_t b, bool alongX,
                                                         int32_t xDim, int32_t yDim, bool wrap, double oob)
        {
            const int32_t dim = alongX ? xDim : yDim;
            int32_t v = alongX ? a : b;
            if (v < 0 || v >= dim)
            {
                if (!wrap)
                {
                    return oob;
                }
                v %= dim;
                v = (v < 0) ? v + dim : v;
            }
            return alongX ? f[static_cast<int64_t>(v) * yDim + b] : f[static_cast<int64_t>(a) * yDim + v];
        }

        __global__ void Gradients(const int32_t *__restrict__ xs, const int32_t *__restrict__ ys, int64_t n,
                                  const double *__restrict__ f, int32_t xDim, int32_t yDim, int32_t wrapX,
                                  int32_t wrapY, int32_t useBoundary, double boundary, double *__restrict__ gx,
                                  double *__restrict__ gy)
        {
            const int64_t k = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
            if (k >= n)
            {
                return;
            }
            const int32_t x = xs[k], y = ys[k];
            const double own = f[static_cast<int64_t>(x) * yDim + y];
            const double oob = useBoundary ? boundary : own;
            gx[k] = __dsub_rn(DisplacedField(f, x + 1, y, true, xDim, yDim, wrapX != 0, oob),
                              DisplacedField(f, x - 1, y, true, xDim, yDim, wrapX != 0, oob));
            gy[k] = __dsub_rn(DisplacedField(f, x, y + 1, false, xDim, yDim, wrapY != 0, oob),
                              DisplacedField(f, x, y - 1, false, xDim, yDim, wrapY != 0, oob));
        }

        // ---- ADI in FP64 ----------------------------------------------------
        // The line-independent part of one sweep's Thomas solve.
        struct LinePlan64Dev
        {
            const double *ws;    // elimination multipliers (index 0 unused)
            const double *bs;    // modified diagonal
            const double *zs;    // periodic: the Sherman-Morrison solution
            const double2 *bh;   // (bs[i], RN(1 / bs[i])): DivByPlan's b and yHi
            const int2 *lo;      // RN(1 / bs[i]) - yHi as (FP32 mantissa bits, exponent)
            double off;          // the off-diagonal -r/2
            double vEnd;         // periodic: beta / gamma
            double onePlusVz;    // periodic: 1 + (zs[0] + zs[L-1] * vEnd)
            int32_t L;
            int32_t periodic;
            int32_t fastDiv;     // every bs[i] in [2^-20, 2^20]: DivByPlan is exact
            // split solve (below): segments per line (1: not split), elements
            // per segment, the back substitution's multipliers off / bs[i]
            // negated, and each segment's products of the negated ws and of g
            int32_t segs, segLen;
            const double *g;
            const double *segP;
            const double *segQ;
            int32_t *ctl;        // SegCtl, then each 32 lines' walks: elimination, back substitution
            int32_t mendBudget;  // cycles of walks up to which segments are the faster
        };

        // A split plan's record, in ctl: sweeps left to solve serially, how many
        // the next time, and of the current sweep the most cycles that the walks
        // of any 32 lines took (the longest of step 3 and 4, and all of step 5)
        // and the CTAs that have reported.
        enum SegCtl : int
        {
            kCtlSkip = 0,
            kCtlPeriod = 1,
            kCtlWorst = 2,
            kCtlReported = 3,
            kCtlCount = 4
        };
        __host__ __device__ __forceinline__ int32_t CtlLines(int32_t lines) { return (lines + 31) / 32; }
        constexpr int32_t kSegMinPeriod = 4, kSegMaxPeriod = 32;
        // cycles that mending an element takes (1820 of 2048 elements of a back
        // substitution: 425 us)
        constexpr int32_t kMendFwd = 160, kMendBwd = 480;

        // ImplicitBoundarySource (ADIequations.h:198-220) at position i of a
        // line of length L; 0 on a wrapped axis.
        __device__ __forceinline__ double ImplicitSource(int32_t i, int32_t L, bool wrap, double r, double lo,
                                                         double hi)
        {
            if (wrap)
            {
                return 0.0;
            }
            double source = 0.0;
            if (i == 0)
            {
                source = __dadd_rn(source, lo);
            }
            if (i == L - 1)
            {
                source = __dadd_rn(source, hi);
            }
            return __dmul_rn(__dmul_rn(__dmul_rn(source, 2.0), r), 0.5);
        }

        // Difference to a cross-axis neighbour n of a line of length dim:
        // on the grid, wrapped, a doubled Dirichlet ghost, or 0.
        __device__ __forceinline__ double CrossDelta(const double *v, double c, int32_t n, int32_t dim, bool wrap,
                                                     int64_t base, int64_t stride, const double *ghost, int64_t gi)
        {
            return DeltaTerm64(v, c, n, dim, wrap, base, stride, ghost, gi);
        }

        // An approximation of n * yLo, for DivByPlan, without FP64
        // instructions: yLo = mLo * 2^eLo with mLo an FP32 value in +-[1, 2]
        // (0 for yLo = 0, with eLo very negative); n's top 20 mantissa bits
        // times mLo in FP32, the exponents added as integers.  Within 1e-5
        // of n * yLo relative, or 0 where n is +-0 or subnormal or the
        // product is below 2^-1022.
        __device__ __forceinline__ double ApproxTimesLo(double n, float mLo, int32_t eLo)
        {
            const uint32_t hi = static_cast<uint32_t>(__double2hiint(n));
            const int32_t en = static_cast<int32_t>((hi >> 20) & 0x7ffu);
            const float fn = __uint_as_float(0x3f800000u | ((hi & 0xfffffu) << 3));
            const uint32_t pb = __float_as_uint(fn * mLo);
            const int32_t te = en + eLo + static_cast<int32_t>((pb >> 23) & 0xffu) - 127;
            const uint32_t tHi = ((hi ^ pb) & 0x80000000u) | (static_cast<uint32_t>(te) << 20) | ((pb & 0x7fffffu) >> 3);
            const bool ok = te > 0 && en != 0;
            return __hiloint2double(ok ? static_cast<int32_t>(tHi) : 0, ok ? static_cast<int32_t>(pb << 29) : 0);
        }

        // n / b rounded to nearest, bit-equal to __ddiv_rn(n, b) for every n
        // that PlanDivisionOutOfRange accepts, from the plan's reciprocal of
        // b as a double-word: yHi = RN(1/b) and yLo = RN(1/b - yHi) (|yLo| <=
        // 2^-53 |yHi|).  With t within half of n*yLo (ApproxTimesLo's is
        // within 1e-5), n*yHi + t is within 2^-54 |n/b| of n/b, so q =
        // RN(n*yHi + t) is one of the two doubles around n/b (faithful); its
        // remainder n - b*q is then exact under an FMA, and RN(q + rem*yHi)
        // is the correctly rounded quotient by Markstein's theorem (P.
        // Markstein, "Computation of elementary functions on the IBM RISC
        // System/6000 processor", IBM J. Res. Dev. 34(1), 1990: y within half
        // an ulp of 1/b, q within one ulp of n/b).  The argument needs no
        // intermediate to underflow or overflow: the plan allows b in
        // [2^-20, 2^20] only (fastDiv), and n must lie in [2^-900, 2^900) in
        // magnitude.  n = +0 gives +0 (t = 0, q = +0, rem = +0, for b > 0);
        // n = -0 would give +0 too, so PlanDivisionOutOfRange refuses it.
        // Three dependent FP64 operations instead of a division's longer
        // sequence; hal_cuda_check_plan_division compares the two.
        __device__ __forceinline__ double DivByPlan(double n, double2 bh, int2 lo)
        {
            const double t = ApproxTimesLo(n, __int_as_float(lo.x), lo.y);
            const double q = __fma_rn(n, bh.y, t);
            const double rem = __fma_rn(-bh.x, q, n);
            return __fma_rn(rem, bh.y, q);
        }

        // Nonzero when DivByPlan may not be exact for the numerator n: -0,
        // subnormal, nonzero below 2^-900 or from 2^900 in magnitude, inf or
        // NaN.  Integer operations only, off the FP64 chain.
        __device__ __forceinline__ uint32_t PlanDivisionOutOfRange(double n)
        {
            const uint32_t hi = static_cast<uint32_t>(__double2hiint(n));
            const uint32_t e = (hi >> 20) & 0x7ffu;
            const bool plusZero = (hi | static_cast<uint32_t>(__double2loint(n))) == 0u;
            return ((e - 123u) > (1922u - 123u) && !plusZero) ? 1u : 0u;
        }

        // ExplicitDiffusionY2ADI / X2ADI (src/Pde/ADIequations.cpp:19-47 and
        // the Dirichlet forms, include/Hal/Pde/ADIequations.h:54-94): the cell
        // plus half the rate times the sum s of its two cross-axis differences,
        // c + (s * r) * 0.5.  With t = RN(s * r), t / 2 is exact unless it is
        // subnormal, and rides on the addition (HalfStep); HalfInexact says
        // where it may not be, and HalfStepExact keeps the operations apart.
        __device__ __forceinline__ double HalfStep(double c, double t)
        {
            return __fma_rn(t, 0.5, c);
        }

        __device__ __forceinline__ uint32_t HalfInexact(double t)
        {
            const uint32_t hi = static_cast<uint32_t>(__double2hiint(t)) & 0x7fffffffu;
            return (hi < 0x00200000u && (hi | static_cast<uint32_t>(__double2loint(t))) != 0u) ? 1u : 0u;
        }

        // Not inlined: the compiler would issue it, predicated off, for every
        // cell, and a predicated-off FP64 instruction still takes the pipe.
        __device__ __noinline__ double HalfStepExact(double c, double t)
        {
            return __dadd_rn(c, __dmul_rn(t, 0.5));
        }

        constexpr int kRhsCells = 4;  // consecutive lines of one thread

        // Right-hand side of one sweep at every cell (i, line) of lines laid
        // out v[i * lines + line]: for the x-sweep ExplicitDiffusionY2ADI
        // (ADIequations.h:316-324, Dirichlet :351-362), for the y-sweep
        // ExplicitDiffusionX2ADI (ADIequations.h:325-336, Dirichlet :363-377)
        // -- the cell plus half the rate times its two cross-axis differences,
        // to line + 1 then line - 1 -- plus, with a ghost table,
        // ImplicitBoundarySource along the line.  crossGhost[L + i] /
        // crossGhost[i] are the ghosts beyond line lines-1 / line 0 of row i;
        // alongLo[line] / alongLo[lines + line] those before element 0 / after
        // element L-1 of a line (null: zero-flux).
        // Bound by FP64 issue: six operations per cell took 51 us at 2048^2.  A
        // thread takes kRhsCells lines and shares each difference between the
        // two cells it separates (negated, which is exact), and the product by
        // 1/2 rides on the last addition: 4.25 operations, 38 us.  (The
        // negation of a zero difference changes the sign of the sum's zero,
        // which the addition to a cell of the same value does not see.)
        __global__ void AdiRhs64(const double *__restrict__ v, double *__restrict__ rhs, int32_t L, int32_t lines,
                                 int32_t wrapCross, int32_t wrapAlong, const double *__restrict__ crossGhost,
                                 const double *__restrict__ alongLo, double r)
        {
            constexpr int C = kRhsCells;
            const int32_t line0 = (blockIdx.x * blockDim.x + threadIdx.x) * C;
            if (line0 >= lines)
            {
                return;
            }
            const bool whole = line0 + C <= lines;
            const bool vec = whole && (lines & 1) == 0;  // 16-byte aligned pairs
            const int32_t n = min(C, lines - line0);
            for (int32_t i = blockIdx.y; i < L; i += gridDim.y)
            {
                const int64_t row = static_cast<int64_t>(i) * lines;
                const double *q = v + row + line0;
                double c[C];
                if (vec)
                {
#pragma unroll
                    for (int k = 0; k < C; k += 2)
                    {
                        const double2 t = __ldg(reinterpret_cast<const double2 *>(q + k));
                        c[k] = t.x;
                        c[k + 1] = t.y;
                    }
                }
                else
                {
#pragma unroll
                    for (int k = 0; k < C; k++)
                    {
                        c[k] = __ldg(q + min(k, n - 1));
                    }
                }
                // up: difference to the line after the cell; dn: to the one
                // before it, of the first cell
                double up[C];
                double dn;
#pragma unroll
                for (int k = 0; k < C - 1; k++)
                {
                    up[k] = __dsub_rn(c[k + 1], c[k]);
                }
                if (line0 > 0)
                {
                    dn = __dsub_rn(__ldg(q - 1), c[0]);
                }
                else
                {
                    dn = CrossDelta(v, c[0], -1, lines, wrapCross != 0, row, 1, crossGhost, i);
                }
                if (whole && line0 + C < lines)
                {
                    up[C - 1] = __dsub_rn(__ldg(q + C), c[C - 1]);
                }
                else
                {
                    // the grid's last cell is c[n - 1]
                    const double last =
                        CrossDelta(v, c[C - 1], lines, lines, wrapCross != 0, row, 1, crossGhost, L + i);
#pragma unroll
                    for (int k = 0; k < C; k++)
                    {
                        up[k] = (k == n - 1) ? last : up[k];
                    }
                }
                double s[C], t[C];
                uint32_t rare = 0;
#pragma unroll
                for (int k = 0; k < C; k++)
                {
                    t[k] = __dmul_rn(__dadd_rn(up[k], k == 0 ? dn : -up[k - 1]), r);
                    s[k] = HalfStep(c[k], t[k]);
                    rare |= HalfInexact(t[k]);
                }
                if (rare != 0)
                {
#pragma unroll
                    for (int k = 0; k < C; k++)
                    {
                        s[k] = HalfStepExact(c[k], t[k]);
                    }
                }
                if (alongLo != nullptr && !wrapAlong && (i == 0 || i == L - 1))
                {
#pragma unroll
                    for (int k = 0; k < C; k++)
                    {
                        if (k < n)
                        {
                            s[k] = __dadd_rn(s[k], ImplicitSource(i, L, false, r, alongLo[line0 + k],
                                                                  alongLo[lines + line0 + k]));
                        }
                    }
                }
                else if (alongLo != nullptr && (wrapAlong || __double2hiint(r) >= 0))
                {
                    // the source is +0: adding it only turns -0 into +0
#pragma unroll
                    for (int k = 0; k < C; k++)
                    {
                        s[k] = (__double_as_longlong(s[k]) == __double_as_longlong(-0.0)) ? 0.0 : s[k];
                    }
                }
                double *o = rhs + row + line0;
                if (vec)
                {
#pragma unroll
                    for (int k = 0; k < C; k += 2)
                    {
                        *reinterpret_cast<double2 *>(o + k) = make_double2(s[k], s[k + 1]);
                    }
                }
                else
                {
#pragma unroll
                    for (int k = 0; k < C; k++)
                    {
                        if (k < n)
                        {
                            o[k] = s[k];
                        }
                    }
                }
            }
        }

        constexpr int kChainFwd = 16;  // elements loaded ahead in the elimination
        constexpr int kChainBwd = 8;   // ... and in the back substitution
        constexpr int kChainFix = 8;   // ... and where the elimination is checked

        // Thomas solve of one line per thread, TdmaSolver::TDMA
        // (TdmaSolver.h:26-66) in its operations and order, over the
        // right-hand sides in d (element i of a line at d[i * lines + line]):
        // elimination in place, d[i] = d[i] - ws[i] * d[i - 1], then back
        // substitution x[i] = (d[i] - off * x[i + 1]) / bs[i] into out.
        // A warp's FP64 instruction costs tens of cycles on this part however
        // many lanes it runs, and a line is one dependent chain, so the chain
        // is all a thread does: AdiRhs64 computes the right-hand sides, the
        // transposes apply the periodic correction, each loop loads the next
        // batch of elements while it works on the current one, and the
        // divisions use the plan's reciprocals (DivByPlan, FAST).  A periodic
        // line (TDMAperiodic, TdmaSolver.h:96-119) leaves its factor (y0 +
        // yL * vEnd) / (1 + vz) in factor[line].
        template <bool FAST>
        __device__ __forceinline__ void ChainLine(double *__restrict__ d, double *__restrict__ out,
                                                  const LinePlan64Dev &pl, int32_t lines, int32_t line,
                                                  double *__restrict__ factor)
        {
            const int32_t L = pl.L;
            auto at = [&](int32_t i) { return static_cast<int64_t>(i) * lines + line; };

            double rc[kChainFwd], wc[kChainFwd];
#pragma unroll
            for (int k = 0; k < kChainFwd; k++)
            {
                const int32_t i = min(k, L - 1);
                rc[k] = __ldcg(d + at(i));
                wc[k] = __ldg(pl.ws + i);
            }
            double prev = 0.0;
            for (int32_t i0 = 0; i0 < L; i0 += kChainFwd)
            {
                double rn[kChainFwd], wn[kChainFwd];
#pragma unroll
                for (int k = 0; k < kChainFwd; k++)
                {
                    const int32_t i = min(i0 + kChainFwd + k, L - 1);
                    rn[k] = __ldcg(d + at(i));
                    wn[k] = __ldg(pl.ws + i);
                }
#pragma unroll
                for (int k = 0; k < kChainFwd; k++)
                {
                    const int32_t i = i0 + k;
                    if (i < L)
                    {
                        prev = (i == 0) ? rc[k] : __dsub_rn(rc[k], __dmul_rn(wc[k], prev));
                        d[at(i)] = prev;
                    }
                }
#pragma unroll
                for (int k = 0; k < kChainFwd; k++)
                {
                    rc[k] = rn[k];
                    wc[k] = wn[k];
                }
            }

            // FAST: a numerator outside DivByPlan's range is only recorded
            // here, and the line is solved again with IEEE divisions below
            // (a test in the loop would put its branch on the chain)
            uint32_t redo = 0;
            double x = FAST ? DivByPlan(prev, pl.bh[L - 1], pl.lo[L - 1]) : __ddiv_rn(prev, pl.bs[L - 1]);
            if (FAST)
            {
                redo |= PlanDivisionOutOfRange(prev);
            }
            out[at(L - 1)] = x;
            double xLast = x;
            double dc[kChainBwd];
            double2 bc[kChainBwd];
            int2 lc[kChainBwd];
#pragma unroll
            for (int k = 0; k < kChainBwd; k++)
            {
                const int32_t i = max(L - 2 - k, 0);
                dc[k] = __ldcg(d + at(i));
                bc[k] = FAST ? __ldg(pl.bh + i) : make_double2(__ldg(pl.bs + i), 0.0);
                lc[k] = FAST ? __ldg(pl.lo + i) : make_int2(0, 0);
            }
            for (int32_t i0 = L - 2; i0 >= 0; i0 -= kChainBwd)
            {
                double dn[kChainBwd];
                double2 bn[kChainBwd];
                int2 ln[kChainBwd];
#pragma unroll
                for (int k = 0; k < kChainBwd; k++)
                {
                    const int32_t i = max(i0 - kChainBwd - k, 0);
                    dn[k] = __ldcg(d + at(i));
                    bn[k] = FAST ? __ldg(pl.bh + i) : make_double2(__ldg(pl.bs + i), 0.0);
                    ln[k] = FAST ? __ldg(pl.lo + i) : make_int2(0, 0);
                }
#pragma unroll
                for (int k = 0; k < kChainBwd; k++)
                {
                    const int32_t i = i0 - k;
                    if (i >= 0)
                    {
                        const double num = __dsub_rn(dc[k], __dmul_rn(pl.off, x));
                        x = FAST ? DivByPlan(num, bc[k], lc[k]) : __ddiv_rn(num, bc[k].x);
                        if (FAST)
                        {
                            redo |= PlanDivisionOutOfRange(num);
                        }
                        out[at(i)] = x;
                    }
                }
#pragma unroll
                for (int k = 0; k < kChainBwd; k++)
                {
                    dc[k] = dn[k];
                    bc[k] = bn[k];
                    lc[k] = ln[k];
                }
            }
            if (FAST && redo != 0)
            {
                x = __ddiv_rn(prev, pl.bs[L - 1]);
                out[at(L - 1)] = x;
                xLast = x;
                for (int32_t i = L - 2; i >= 0; i--)
                {
                    x = __ddiv_rn(__dsub_rn(__ldcg(d + at(i)), __dmul_rn(pl.off, x)), pl.bs[i]);
                    out[at(i)] = x;
                }
            }
            if (pl.periodic)
            {
                // x is now y0 (element 0), xLast yL (element L - 1)
                const double vy = __dadd_rn(x, __dmul_rn(xLast, pl.vEnd));
                factor[line] = __ddiv_rn(vy, pl.onePlusVz);
            }
        }

        template <bool FAST>
        __global__ void __launch_bounds__(32) AdiChain64(double *__restrict__ d, double *__restrict__ out,
                                                          LinePlan64Dev pl, int32_t lines,
                                                          double *__restrict__ factor)
        {
            const int32_t line = blockIdx.x * blockDim.x + threadIdx.x;
            if (line < lines)
            {
                ChainLine<FAST>(d, out, pl, lines, line, factor);
            }
        }

        // ---- the same solve, each line split into segments ------------------
        // One thread per line is one dependent FP64 chain of 2 + 5
        // instructions per element, 64 cycles each: 580 us for 2048 lines of
        // 2048 on 64 warps, while the chip could issue from 608.  Split into
        // segments, the chains of a line run side by side and still give the
        // serial chain's bits:
        //   1. AdiSegEnds: every segment's elimination from a zero start (one
        //      FMA per element).  With the segments' products of -ws, which
        //      the plan holds, these give every segment's incoming value to
        //      within a few ulps (a relative error also where the solution
        //      decays along the line: sums of one sign do not cancel);
        //   2. AdiSegElim: the elimination in the reference's operations from
        //      that value.  The recurrence contracts (|ws| < 1), so two
        //      trajectories a few ulps apart round to the same value after
        //      some tens of elements and are one from there on;
        //   3. AdiSegFix: from the end of the segment before, which has met
        //      the serial trajectory by then, the elements again until one
        //      comes out bit-equal to what is stored: from there the segment
        //      is the serial one.  A segment that ends without such a meeting
        //      marks its line.  Then the back substitution's segments from a
        //      zero start, as in 1;
        //   4. AdiSegBack and AdiSegBackFix: the same for the back
        //      substitution;
        //   5. of each 32 lines, the CTA that is the last to be done with step 3
        //      (4) mends the marked lines, from segment to segment: a segment
        //      that was entered with another value than the line now holds is
        //      walked again, until it meets what is stored.
        // Every element is thus either checked against the serial recurrence
        // or follows from one that was: equality is bitwise, so zeros' signs,
        // infinities and NaN end in a marked line at worst.
        // Lines are marked where trajectories an ulp apart stay apart: on
        // constant data, where each has its own rounded fixed point (a uniform
        // field's back substitution), and where the right-hand side is zero, so
        // that a relative difference neither grows nor shrinks (the tails of a
        // point or a step in an empty field).  Where mending them costs more than
        // the segments save, the sweep is slower than one chain a line, so the
        // device keeps a record per plan (SegCtl) and solves the next sweeps
        // serially, in AdiSegEnds: 4, then 8, 16, 32 between attempts.  The bits
        // are the same either way.
        // us per sweep at r = 5, the right-hand sides and the transpose included,
        // one chain a line / here: random values in 2048^2 659 / 177 (19 segments
        // a line; FP64 issue needs 79 for the ten operations per element), in
        // 512^2 161 / 72, in 256^2 87 / 72; a uniform field, over forty sweeps, in
        // 2048^2 659 / 663, in 512^2 161 / 165, in 256^2 87 / 92.

        __device__ __forceinline__ bool SameBits(double a, double b)
        {
            return __double_as_longlong(a) == __double_as_longlong(b);
        }

        // A load that stays where it is written, ahead of its use (the compiler
        // moves others down to it, past the walks' tests).
        __device__ __forceinline__ double LdAhead(const double *p)
        {
            double v;
            asm volatile("ld.global.cg.f64 %0, [%1];" : "=d"(v) : "l"(p));
            return v;
        }

        // e[i] = d[i] - ws[i] * e[i - 1] over elements [a, b) of a line, from
        // prev (unused at i = 0), in the reference's operations; prev becomes
        // the last value.  at(i): the element's offset.  CHECK: the warp stops
        // after a batch by which every lane had a batch whose last element came
        // out bit-equal to the stored one, since the trajectories are one from
        // where they meet; whether the lane's did.  (Nothing on the chain tests
        // anything, and the lanes stay together: with a test per element, or
        // lanes that stop by themselves, the walk took three times as long.)
        template <bool CHECK, int B, typename At>
        __device__ __forceinline__ bool ElimWalk(const double *__restrict__ d, double *__restrict__ e,
                                                 const LinePlan64Dev &pl, int32_t a, int32_t b, double &prev, At at,
                                                 int32_t *batches = nullptr)
        {
            bool met = false;
            double rc[B], wc[B], oc = 0.0;  // oc: the batch's last element as stored
#pragma unroll
            for (int k = 0; k < B; k++)
            {
                const int32_t i = min(a + k, b - 1);
                rc[k] = LdAhead(d + at(i));
                wc[k] = __ldg(pl.ws + i);
            }
            if (CHECK)
            {
                oc = LdAhead(e + at(min(a + B - 1, b - 1)));
                __syncwarp();  // (a line may be on two lanes)
            }
            for (int32_t i0 = a; i0 < b; i0 += B)
            {
                double rn[B], wn[B], on = 0.0;
#pragma unroll
                for (int k = 0; k < B; k++)
                {
                    const int32_t i = min(i0 + B + k, b - 1);
                    rn[k] = LdAhead(d + at(i));
                    wn[k] = __ldg(pl.ws + i);
                }
                if (CHECK)
                {
                    on = LdAhead(e + at(min(i0 + 2 * B - 1, b - 1)));
                }
#pragma unroll
                for (int k = 0; k < B; k++)
                {
                    const int32_t i = i0 + k;
                    if (i < b)
                    {
                        prev = (i == 0) ? rc[k] : __dsub_rn(rc[k], __dmul_rn(wc[k], prev));
                        e[at(i)] = prev;
                    }
                }
                if (batches != nullptr)
                {
                    (*batches)++;
                }
                if (CHECK)
                {
                    met = met || SameBits(prev, oc);
                    if (__all_sync(0xffffffffu, met))
                    {
                        break;
                    }
                }
                oc = on;
#pragma unroll
                for (int k = 0; k < B; k++)
                {
                    rc[k] = rn[k];
                    wc[k] = wn[k];
                }
            }
            return met;
        }

        // The exact quotient num / bs[i] for any numerator.
        __device__ __forceinline__ double DivExact(double num, double2 bh, int2 lo)
        {
            return PlanDivisionOutOfRange(num) ? __ddiv_rn(num, bh.x) : DivByPlan(num, bh, lo);
        }

        // Elements i1, i1 - 1, .. i0 of the back substitution from x, with
        // numerators that DivByPlan does not take; *again: there was one.  Not
        // inlined (HalfStepExact).
        __device__ __noinline__ double BackSlow(const double *e, double *out, const double2 *bh, const int2 *lo,
                                                double off, int32_t L, int32_t i1, int32_t i0, double x,
                                                int32_t lines, int32_t line, bool *again)
        {
            constexpr int B = 8;
            double ev[B];
            double2 bv[B];
            int2 lv[B];
#pragma unroll
            for (int k = 0; k < B; k++)
            {
                const int32_t i = max(i1 - k, i0);
                ev[k] = __ldcg(e + static_cast<int64_t>(i) * lines + line);
                bv[k] = __ldg(bh + i);
                lv[k] = __ldg(lo + i);
            }
            uint32_t rare = 0;
#pragma unroll
            for (int k = 0; k < B; k++)
            {
                const int32_t i = i1 - k;
                if (i >= i0)
                {
                    const double num = (i == L - 1) ? ev[k] : __dsub_rn(ev[k], __dmul_rn(off, x));
                    rare |= PlanDivisionOutOfRange(num);
                    x = DivExact(num, bv[k], lv[k]);
                    out[static_cast<int64_t>(i) * lines + line] = x;
                }
            }
            *again = rare != 0;
            return x;
        }

        // x[i] = (e[i] - off * x[i + 1]) / bs[i] over [a, b) downwards, from x
        // (unused at i = L - 1), in the reference's operations; x becomes x[a].
        // A batch that has a numerator outside DivByPlan's range is computed
        // again with the division chosen per element (a branch on the chain),
        // and so are the next ones until a batch has none.  CHECK as in
        // ElimWalk.
        template <bool CHECK>
        __device__ __forceinline__ bool BackWalk(const double *__restrict__ e, double *__restrict__ out,
                                                 const LinePlan64Dev &pl, int32_t lines, int32_t line, int32_t a,
                                                 int32_t b, double &x, int32_t *batches = nullptr)
        {
            constexpr int B = kChainBwd;
            static_assert(B == 8, "BackSlow's batch");
            auto at = [&](int32_t i) { return static_cast<int64_t>(i) * lines + line; };
            bool slow = false, met = false;
            double dc[B], oc = 0.0;
            double2 bc[B];
            int2 lc[B];
#pragma unroll
            for (int k = 0; k < B; k++)
            {
                const int32_t i = max(b - 1 - k, a);
                dc[k] = __ldcg(e + at(i));
                bc[k] = __ldg(pl.bh + i);
                lc[k] = __ldg(pl.lo + i);
            }
            if (CHECK)
            {
                oc = LdAhead(out + at(max(b - B, a)));
                __syncwarp();
            }
            for (int32_t i0 = b - 1; i0 >= a; i0 -= B)
            {
                double dn[B], on = 0.0;
                double2 bn[B];
                int2 ln[B];
#pragma unroll
                for (int k = 0; k < B; k++)
                {
                    const int32_t i = max(i0 - B - k, a);
                    dn[k] = __ldcg(e + at(i));
                    bn[k] = __ldg(pl.bh + i);
                    ln[k] = __ldg(pl.lo + i);
                }
                if (CHECK)
                {
                    on = LdAhead(out + at(max(i0 - 2 * B + 1, a)));
                }
                const double x0 = x;
                uint32_t rare = slow ? 1u : 0u;
                if (!slow)
                {
#pragma unroll
                    for (int k = 0; k < B; k++)
                    {
                        const int32_t i = i0 - k;
                        if (i >= a)
                        {
                            const double num = (i == pl.L - 1) ? dc[k] : __dsub_rn(dc[k], __dmul_rn(pl.off, x));
                            x = DivByPlan(num, bc[k], lc[k]);
                            rare |= PlanDivisionOutOfRange(num);
                            out[at(i)] = x;
                        }
                    }
                }
                if (rare != 0)
                {
                    x = BackSlow(e, out, pl.bh, pl.lo, pl.off, pl.L, i0, max(i0 - B + 1, a), x0, lines, line, &slow);
                }
                if (batches != nullptr)
                {
                    (*batches)++;
                }
                if (CHECK)
                {
                    met = met || SameBits(x, oc);
                    if (__all_sync(0xffffffffu, met))
                    {
                        break;
                    }
                }
                oc = on;
#pragma unroll
                for (int k = 0; k < B; k++)
                {
                    dc[k] = dn[k];
                    bc[k] = bn[k];
                    lc[k] = ln[k];
                }
            }
            return met;
        }

        // Whether the CTA (one warp: 32 lines of one segment) is the last of its
        // lines' CTAs to come here, and may read what the others wrote.  No CTA
        // waits for another.  arrived: one count per 32 lines, zero between
        // kernels.
        __device__ __forceinline__ bool LastOfLines(int32_t *__restrict__ arrived)
        {
            __threadfence();
            __syncwarp();
            int32_t before = 0;
            if (threadIdx.x == 0)
            {
                before = atomicAdd(arrived + blockIdx.x, 1);
            }
            before = __shfl_sync(0xffffffffu, before, 0);
            if (before != static_cast<int32_t>(gridDim.y) - 1)
            {
                return false;
            }
            if (threadIdx.x == 0)
            {
                arrived[blockIdx.x] = 0;
            }
            __threadfence();
            return true;
        }

        __device__ __forceinline__ bool Serial(const LinePlan64Dev &pl)
        {
            return __ldcg(pl.ctl + kCtlSkip) > 0;
        }

        // Step 1 (segments 0 .. segs - 2): y[seg * lines + line].  In a serial
        // sweep the first segment's CTAs solve their lines whole.
        __global__ void __launch_bounds__(32) AdiSegEnds(double *__restrict__ d, LinePlan64Dev pl, int32_t lines,
                                                          double *__restrict__ y, double *__restrict__ out,
                                                          double *__restrict__ factor)
        {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            const int32_t line = blockIdx.x * 32 + threadIdx.x, seg = blockIdx.y;
            if (line >= lines)
            {
                return;
            }
            if (Serial(pl))
            {
                if (seg == 0)
                {
                    ChainLine<true>(d, out, pl, lines, line, factor);
                }
                return;
            }
            const int32_t a = seg * pl.segLen, b = a + pl.segLen;
            auto at = [&](int32_t i) { return static_cast<int64_t>(i) * lines + line; };
            double v = 0.0;
            double rc[kChainFwd], wc[kChainFwd];
#pragma unroll
            for (int k = 0; k < kChainFwd; k++)
            {
                const int32_t i = min(a + k, b - 1);
                rc[k] = __ldcg(d + at(i));
                wc[k] = __ldg(pl.ws + i);
            }
            for (int32_t i0 = a; i0 < b; i0 += kChainFwd)
            {
                double rn[kChainFwd], wn[kChainFwd];
#pragma unroll
                for (int k = 0; k < kChainFwd; k++)
                {
                    const int32_t i = min(i0 + kChainFwd + k, b - 1);
                    rn[k] = __ldcg(d + at(i));
                    wn[k] = __ldg(pl.ws + i);
                }
#pragma unroll
                for (int k = 0; k < kChainFwd; k++)
                {
                    if (i0 + k < b)
                    {
                        v = __fma_rn(-wc[k], v, rc[k]);
                    }
                }
#pragma unroll
                for (int k = 0; k < kChainFwd; k++)
                {
                    rc[k] = rn[k];
                    wc[k] = wn[k];
                }
            }
            y[static_cast<int64_t>(seg) * lines + line] = v;
        }

        // Step 2: e over every segment; ends[seg * lines + line] = its last.
        __global__ void __launch_bounds__(32) AdiSegElim(const double *__restrict__ d, double *__restrict__ e,
                                                          LinePlan64Dev pl, int32_t lines,
                                                          const double *__restrict__ y, double *__restrict__ ends)
        {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            const int32_t line = blockIdx.x * 32 + threadIdx.x, seg = blockIdx.y;
            if (line >= lines)
            {
                return;
            }
            const bool serial = Serial(pl);
            const int32_t a = seg * pl.segLen, b = min(a + pl.segLen, pl.L);
            double prev = 0.0;
            for (int32_t q = 0; q < seg; q++)
            {
                prev = __fma_rn(__ldg(pl.segP + q), prev, __ldcg(y + static_cast<int64_t>(q) * lines + line));
            }
            if (serial)
            {
                return;
            }
            ElimWalk<false, kChainFwd>(d, e, pl, a, b, prev,
                                       [&](int32_t i) { return static_cast<int64_t>(i) * lines + line; });
            ends[static_cast<int64_t>(seg) * lines + line] = prev;
        }

        // Step 3; z[seg * lines + line]: segments 1 .. segs - 1 of the back
        // substitution from a zero start (of a marked line from values that may
        // be an ulp off: they only estimate).
        __global__ void __launch_bounds__(32) AdiSegFix(const double *__restrict__ d, double *__restrict__ e,
                                                         LinePlan64Dev pl, int32_t lines,
                                                         const double *__restrict__ ends, double *__restrict__ z,
                                                         int32_t *__restrict__ marks, int32_t *__restrict__ arrived)
        {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            if (Serial(pl))
            {
                return;
            }
            // (lanes past the last line repeat it: the walks take the whole warp)
            const int32_t line = min(static_cast<int32_t>(blockIdx.x * 32 + threadIdx.x), lines - 1);
            const int32_t seg = blockIdx.y + 1;
            const int32_t a = seg * pl.segLen, b = min(a + pl.segLen, pl.L);
            auto at = [&](int32_t i) { return static_cast<int64_t>(i) * lines + line; };
            int32_t batches = 0;
            double prev = __ldcg(ends + static_cast<int64_t>(seg - 1) * lines + line);
            if (!ElimWalk<true, kChainFix>(d, e, pl, a, b, prev, at, &batches) && seg < pl.segs - 1)
            {
                marks[line] = 1;
            }
            double v = 0.0;
            for (int32_t i0 = b - 1; i0 >= a; i0 -= kChainBwd)
            {
                double ev[kChainBwd], gv[kChainBwd];
#pragma unroll
                for (int k = 0; k < kChainBwd; k++)
                {
                    const int32_t i = max(i0 - k, a);
                    ev[k] = __dmul_rn(__ldcg(e + at(i)), __ldg(&pl.bh[i].y));
                    gv[k] = __ldg(pl.g + i);
                }
#pragma unroll
                for (int k = 0; k < kChainBwd; k++)
                {
                    if (i0 - k >= a)
                    {
                        v = __fma_rn(gv[k], v, ev[k]);
                    }
                }
            }
            z[static_cast<int64_t>(seg) * lines + line] = v;
            int32_t *walked = pl.ctl + kCtlCount + blockIdx.x;
            if (threadIdx.x == 0)
            {
                atomicMax(walked, batches);
            }
            if (!LastOfLines(arrived))
            {
                return;
            }
            // step 5 of the elimination
            const bool marked = __any_sync(0xffffffffu, __ldcg(marks + line) != 0);
            marks[line] = 0;
            batches = 0;
            for (int32_t q = 1; marked && q < pl.segs; q++)
            {
                const int32_t qa = q * pl.segLen;
                prev = __ldcg(e + at(qa - 1));
                if (__any_sync(0xffffffffu,
                               !SameBits(prev, __ldcg(ends + static_cast<int64_t>(q - 1) * lines + line))))
                {
                    ElimWalk<true, kChainFix>(d, e, pl, qa, min(qa + pl.segLen, pl.L), prev, at, &batches);
                }
            }
            if (threadIdx.x == 0)
            {
                *walked = kMendFwd * kChainFix * (__ldcg(walked) + batches);
            }
        }

        // Step 4: the back substitution; starts[seg * lines + line] = its x[a].
        __global__ void __launch_bounds__(32) AdiSegBack(const double *__restrict__ e, double *__restrict__ out,
                                                          LinePlan64Dev pl, int32_t lines,
                                                          const double *__restrict__ z, double *__restrict__ starts)
        {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            const int32_t line = blockIdx.x * 32 + threadIdx.x, seg = blockIdx.y;
            if (line >= lines)
            {
                return;
            }
            const bool serial = Serial(pl);
            const int32_t a = seg * pl.segLen, b = min(a + pl.segLen, pl.L);
            double x = 0.0;
            for (int32_t q = pl.segs - 1; q > seg; q--)
            {
                x = __fma_rn(__ldg(pl.segQ + q), x, __ldcg(z + static_cast<int64_t>(q) * lines + line));
            }
            if (serial)
            {
                return;
            }
            BackWalk<false>(e, out, pl, lines, line, a, b, x);
            starts[static_cast<int64_t>(seg) * lines + line] = x;
        }

        // With a periodic line's factor (see AdiChain64).
        __global__ void __launch_bounds__(32) AdiSegBackFix(const double *__restrict__ e, double *__restrict__ out,
                                                             LinePlan64Dev pl, int32_t lines,
                                                             const double *__restrict__ starts,
                                                             int32_t *__restrict__ marks,
                                                             int32_t *__restrict__ arrived, double *__restrict__ factor)
        {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            if (Serial(pl))
            {
                return;
            }
            const int32_t line = min(static_cast<int32_t>(blockIdx.x * 32 + threadIdx.x), lines - 1);
            const int32_t seg = blockIdx.y;
            const int32_t a = seg * pl.segLen, b = a + pl.segLen;
            int32_t batches = 0;
            double x = __ldcg(starts + static_cast<int64_t>(seg + 1) * lines + line);
            if (!BackWalk<true>(e, out, pl, lines, line, a, b, x, &batches) && seg > 0)
            {
                marks[line] = 1;
            }
            int32_t *walked = pl.ctl + kCtlCount + blockIdx.x;
            batches = __reduce_max_sync(0xffffffffu, batches);
            if (threadIdx.x == 0)
            {
                atomicMax(walked + CtlLines(lines), batches);
            }
            if (!LastOfLines(arrived))
            {
                return;
            }
            // step 5 of the back substitution
            auto at = [&](int32_t i) { return static_cast<int64_t>(i) * lines + line; };
            const bool marked = __any_sync(0xffffffffu, __ldcg(marks + line) != 0);
            marks[line] = 0;
            batches = 0;
            for (int32_t q = pl.segs - 2; marked && q >= 0; q--)
            {
                const int32_t qb = (q + 1) * pl.segLen;
                x = __ldcg(out + at(qb));
                if (__any_sync(0xffffffffu,
                               !SameBits(x, __ldcg(starts + static_cast<int64_t>(q + 1) * lines + line))))
                {
                    BackWalk<true>(e, out, pl, lines, line, q * pl.segLen, qb, x, &batches);
                }
            }
            if (pl.periodic)
            {
                const double vy = __dadd_rn(__ldcg(out + at(0)), __dmul_rn(__ldcg(out + at(pl.L - 1)), pl.vEnd));
                factor[line] = __ddiv_rn(vy, pl.onePlusVz);
            }
            // the record
            if (threadIdx.x == 0)
            {
                int32_t *ctl = pl.ctl;
                int32_t *back = walked + CtlLines(lines);
                atomicMax(ctl + kCtlWorst, __ldcg(walked) + kMendBwd * kChainBwd * (__ldcg(back) + batches));
                *walked = *back = 0;
                __threadfence();
                if (atomicAdd(ctl + kCtlReported, 1) == static_cast<int32_t>(gridDim.x) - 1)
                {
                    const bool late = atomicExch(ctl + kCtlWorst, 0) > pl.mendBudget;
                    const int32_t period = late ? ctl[kCtlPeriod] : 0;
                    ctl[kCtlReported] = 0;
                    ctl[kCtlPeriod] = late ? min(2 * period, kSegMaxPeriod) : kSegMinPeriod;
                    ctl[kCtlSkip] = late ? period + 1 : 0;  // (the transpose of this sweep counts one)
                }
            }
        }

        // The sweeps' division (DivByPlan, or __ddiv_rn where
        // PlanDivisionOutOfRange says so) against __ddiv_rn for every num[i]
        // and divisor j (bh[j], lo[j]: its plan entries); the count of
        // differing bit patterns goes to *bad.
        __global__ void CheckPlanDivision(const double *__restrict__ num, int64_t nNum, const double2 *__restrict__ bh,
                                          const int2 *__restrict__ lo, int32_t nDen, unsigned long long *bad)
        {
            for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < nNum;
                 i += static_cast<int64_t>(gridDim.x) * blockDim.x)
            {
                const double n = num[i];
                unsigned long long c = 0;
                for (int32_t j = 0; j < nDen; j++)
                {
                    const double a = __ddiv_rn(n, bh[j].x);
                    const double b = PlanDivisionOutOfRange(n) ? __ddiv_rn(n, bh[j].x) : DivByPlan(n, bh[j], lo[j]);
                    c += (__double_as_longlong(a) != __double_as_longlong(b)) ? 1ull : 0ull;
                }
                if (c != 0)
                {
                    atomicAdd(bad, c);
                }
            }
        }

        // Tiled transpose of a rows x cols FP64 array: out[c * rows + r] =
        // in[r * cols + c].  With deltas, instead deltas[c * rows + r] +=
        // in[r * cols + c] - f[c * rows + r] (the y-sweep's commit into the
        // deltas, ADIequations.h:331-335).  With fac, each input first takes
        // the periodic correction of its line c at element r, in - fac[c] *
        // zs[r] (TDMAperiodic's ys - factor * zs, TdmaSolver.h:115-118).
        template <bool COMMIT>
        __global__ void Transpose64(const double *__restrict__ in, double *__restrict__ out, int32_t rows,
                                    int32_t cols, const double *__restrict__ f, const double *__restrict__ fac,
                                    const double *__restrict__ zs, int32_t *__restrict__ ctl)
        {
            __shared__ double tile[32][33];
            if (ctl != nullptr && blockIdx.x + blockIdx.y + threadIdx.x + threadIdx.y == 0 && ctl[kCtlSkip] > 0)
            {
                ctl[kCtlSkip]--;
            }
            const int32_t c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
            for (int j = threadIdx.y; j < 32; j += blockDim.y)
            {
                const int32_t r = r0 + j, c = c0 + threadIdx.x;
                if (r < rows && c < cols)
                {
                    double v = in[static_cast<int64_t>(r) * cols + c];
                    if (fac != nullptr)
                    {
                        v = __dsub_rn(v, __dmul_rn(fac[c], zs[r]));
                    }
                    tile[j][threadIdx.x] = v;
                }
            }
            __syncthreads();
            for (int j = threadIdx.y; j < 32; j += blockDim.y)
            {
                const int32_t c = c0 + j, r = r0 + threadIdx.x;
                if (r < rows && c < cols)
                {
                    const int64_t o = static_cast<int64_t>(c) * rows + r;
                    if constexpr (COMMIT)
                    {
                        out[o] = __dadd_rn(out[o], __dsub_rn(tile[threadIdx.x][j], f[o]));
                    }
                    else
                    {
                        out[o] = tile[threadIdx.x][j];
                    }
                }
            }
        }

        inline unsigned Blocks(int64_t n, int t)
        {
            const int64_t b = (n + t - 1) / t;
            return static_cast<unsigned>(b < 1 ? 1 : (b > 2147483647 ? 2147483647 : b));
        }

        inline unsigned StrideBlocks(int64_t n)
        {
            return static_cast<unsigned>(std::min<int64_t>(std::max<int64_t>((n + 255) / 256, 1), 152 * 16));
        }

        // ---- host side of the ADI plan -------------------------------------
        // TdmaSolver::TDMA's elimination (TdmaSolver.h:26-66) applied to the
        // coefficients alone, in its operations: bs[i] = b_i - ws[i] * c,
        // ws[i] = a / bs[i - 1], with ADISolveRow's coefficients
        // (ADIequations.h:225-270): off-diagonal -r/2; diagonal 1 - w * off,
        // w = 2 plus endAdjust (+1 Dirichlet, -1 zero-flux) at each end; on a
        // wrapped axis TDMAperiodic's adjusted ends (TdmaSolver.h:68-95).
        // This file is compiled without floating-point contraction on the
        // host, so each operation rounds as the reference's does.
        struct LinePlan64Host
        {
            std::vector<double> ws, bs, zs;
            std::vector<double2> bh;
            std::vector<int2> lo;
            double off = 0, vEnd = 0, onePlusVz = 0;
            bool periodic = false;
            bool fastDiv = false;
            int32_t segs = 1, segLen = 0, mendBudget = 0;
            std::vector<double> g, segP, segQ;
        };

        // DivByPlan's entries for the divisor b: (b, hi) with hi = RN(1/b),
        // and lo = RN(1/b - hi) as an FP32 mantissa in +-[1, 2) (its bits)
        // and an exponent; 1 - b*hi is exact under an FMA, so lo = RN((1 -
        // b*hi) / b).  A lo below 2^-200 |hi| counts as 0 (its product with
        // any n is far below half an ulp of n/b).
        void PlanReciprocal(double b, double2 *bh, int2 *lo)
        {
            const double hi = 1.0 / b;
            const double l = std::fma(-b, hi, 1.0) / b;
            *bh = make_double2(b, hi);
            *lo = make_int2(0, -4096);
            if (l != 0.0 && std::fabs(l) >= std::ldexp(std::fabs(hi), -200))
            {
                int e = 0;
                const double fr = std::frexp(l, &e);  // l = fr * 2^e, |fr| in [0.5, 1)
                const float m = static_cast<float>(fr * 2.0);
                int32_t bits = 0;
                std::memcpy(&bits, &m, sizeof(bits));
                *lo = make_int2(bits, e - 1);
            }
        }

        // b in [2^-20, 2^20], where DivByPlan is exact for every n that
        // PlanDivisionOutOfRange accepts (the matrices of a diffusion rate
        // r >= 0 have diagonals of at least 1).
        bool PlanDivisorInRange(double b)
        {
            return b >= 0x1p-20 && b <= 0x1p20;
        }

        // Reciprocals of the modified diagonal and whether DivByPlan may
        // replace the back substitution's divisions.
        void AddReciprocals(LinePlan64Host &p)
        {
            const size_t n = p.bs.size();
            p.bh.assign(n, make_double2(0.0, 0.0));
            p.lo.assign(n, make_int2(0, 0));
            p.fastDiv = true;
            for (size_t i = 0; i < n; i++)
            {
                p.fastDiv = p.fastDiv && PlanDivisorInRange(p.bs[i]);
            }
            for (size_t i = 0; p.fastDiv && i < n; i++)
            {
                PlanReciprocal(p.bs[i], &p.bh[i], &p.lo[i]);
            }
        }

        struct PlanCoeffs
        {
            double off;
            double endAdjust;
            bool periodic, adjusted;
            double gamma, alpha, beta;
            int32_t len;

            double BRaw(int32_t i) const
            {
                if (periodic)
                {
                    return 1 - 2 * off;
                }
                double weight = 2.0;
                if (i == 0)
                {
                    weight += endAdjust;
                }
                if (i == len - 1)
                {
                    weight += endAdjust;
                }
                return 1 - weight * off;
            }

            double B(int32_t i) const
            {
                if (adjusted)
                {
                    if (i == 0)
                    {
                        return BRaw(i) - gamma;
                    }
                    if (i == len - 1)
                    {
                        return BRaw(i) - (alpha * beta) / gamma;
                    }
                }
                return BRaw(i);
            }
        };

        // The elimination's coefficients (ws, bs) of a matrix.
        void Eliminate(const PlanCoeffs &k, std::vector<double> &ws, std::vector<double> &bs)
        {
            const int32_t n = k.len;
            ws.assign(static_cast<size_t>(n), 0.0);
            bs.assign(static_cast<size_t>(n), 0.0);
            bs[0] = k.B(0);
            for (int32_t i = 1; i < n; i++)
            {
                bs[i] = k.B(i);
                ws[i] = k.off / bs[i - 1];
                bs[i] = bs[i] - ws[i] * k.off;
            }
        }

        // TDMA of one right-hand side with given coefficients (host).
        void SolveHost(const PlanCoeffs &k, const std::vector<double> &ws, const std::vector<double> &bs,
                       const std::vector<double> &rhs, std::vector<double> &out)
        {
            const int32_t n = k.len;
            std::vector<double> ds(rhs);
            for (int32_t i = 1; i < n; i++)
            {
                ds[i] = ds[i] - ws[i] * ds[i - 1];
            }
            out.assign(static_cast<size_t>(n), 0.0);
            double x = ds[n - 1] / bs[n - 1];
            out[n - 1] = x;
            for (int32_t i = n - 2; i >= 0; i--)
            {
                x = (ds[i] - k.off * x) / bs[i];
                out[i] = x;
            }
        }

        LinePlan64Host BuildPlan64(int32_t len, double r, bool wrap, bool dirichlet)
        {
            LinePlan64Host p;
            PlanCoeffs k{};
            k.off = -r / 2.0;
            k.len = len;
            p.off = k.off;
            if (wrap)
            {
                k.periodic = true;
                const double gamma = -k.B(0);
                k.gamma = gamma;
                k.alpha = k.off;
                k.beta = k.off;
                k.adjusted = true;
                Eliminate(k, p.ws, p.bs);
                std::vector<double> us(static_cast<size_t>(len), 0.0);
                for (int32_t i = 0; i < len; i++)
                {
                    us[i] = (i == 0) ? gamma : ((i == len - 1) ? k.alpha : 0.0);
                }
                SolveHost(k, p.ws, p.bs, us, p.zs);
                p.vEnd = k.beta / gamma;
                const double vz = p.zs[0] + p.zs[len - 1] * p.vEnd;
                p.onePlusVz = 1 + vz;
                p.periodic = true;
                AddReciprocals(p);
                return p;
            }
            k.endAdjust = dirichlet ? 1.0 : -1.0;
            Eliminate(k, p.ws, p.bs);
            p.zs.assign(static_cast<size_t>(len), 0.0);
            AddReciprocals(p);
            return p;
        }

        constexpr int32_t kSegMaxWarps = 1216;  // 152 SMs x 4 FP64 pipes x 2
        constexpr int32_t kSegMinLen = 64;
        constexpr int32_t kSegMinLine = 232;
        constexpr int32_t kSegMinCount = 3;

        // Segments of a line's split solve, for `lines` lines.  As many as
        // give every FP64 pipe two warps, which cover each other's loads (the
        // kernels of a 2048^2 sweep: 161 us with one warp per pipe, 122 us
        // with two, 118 us with three, and the whole tick no faster than with
        // two); segments of at least kSegMinLen elements (shorter ones spend
        // more on their launches and meetings than the chain saves), and each
        // long enough that a trajectory's error falls below 2^-64 of itself
        // over it: otherwise, for large rates, segments would end before they
        // meet the serial one.  One segment: the serial chain, also where only
        // two segments would do (they cost more than the chain where they meet
        // late: 2048^2 at r = 500 1010 against 660 us per sweep) and for lines
        // below kSegMinLine, whose chain costs less than the segments' launches
        // (four ticks, chain / segments: 200^2 574 / 696 us, 240^2 673 / 634, 320^2
        // 868 / 639).
        void AddSegments(LinePlan64Host &p, int32_t lines)
        {
            const int32_t L = static_cast<int32_t>(p.bs.size());
            const int32_t warps = (lines + 31) / 32;
            p.segs = 1;
            p.segLen = L;
            if (!p.fastDiv)
            {
                return;
            }
            p.g.assign(static_cast<size_t>(L), 0.0);
            for (int32_t i = 0; i < L; i++)
            {
                p.g[static_cast<size_t>(i)] = -p.off * p.bh[static_cast<size_t>(i)].y;
            }
            const int32_t most = L < kSegMinLine ? 1 : std::min(kSegMaxWarps / warps, L / kSegMinLen);
            for (int32_t segs = most; segs >= kSegMinCount; segs--)
            {
                const int32_t len = (L + segs - 1) / segs;
                const int32_t n = (L + len - 1) / len;
                std::vector<double> P(static_cast<size_t>(n), 1.0), Q(static_cast<size_t>(n), 1.0);
                bool ok = true;
                for (int32_t q = 0; q < n; q++)
                {
                    for (int32_t i = q * len; i < std::min(L, (q + 1) * len); i++)
                    {
                        P[static_cast<size_t>(q)] *= -p.ws[static_cast<size_t>(i)];
                        Q[static_cast<size_t>(q)] *= p.g[static_cast<size_t>(i)];
                    }
                    ok = ok && (q == n - 1 || (std::fabs(P[static_cast<size_t>(q)]) <= 0x1p-64 &&
                                               std::fabs(Q[static_cast<size_t>(q)]) <= 0x1p-64));
                }
                if (ok && n >= kSegMinCount)
                {
                    p.segs = n;
                    p.segLen = len;
                    // what the chain takes less the segments' kernels, as
                    // measured (cycles): 586 per element (2048: 580 us), and 831
                    // per segment's element and warp that shares a pipe, and
                    // 72000 (2048^2 122 us, 512^2 65 us; at least the walks of
                    // ordinary fields)
                    const double perPipe = std::max(1.0, static_cast<double>(n) * warps / 608.0);
                    p.mendBudget =
                        static_cast<int32_t>(std::max(20000.0, 586.0 * L - 831.0 * len * perPipe - 72000.0));
                    p.segP = P;
                    p.segQ = Q;
                    return;
                }
            }
        }

        // Launches a kernel of the split solve, which waits for the one before
        // at its start; none triggers its successor early, so that its CTAs come
        // to SMs that have been left (us per sweep without / with: random 512^2
        // 82 / 72, 2048^2 193 / 182).
        template <typename... KArgs, typename... Args>
        void ChainedSeg(void (*kernel)(KArgs...), dim3 grid, cudaStream_t s, Args... args)
        {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = grid;
            cfg.blockDim = dim3(32);
            cfg.stream = s;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            at[0].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
        }

        struct PlanBuf64
        {
            DevBuf<double> buf;  // the plan's arrays
            DevBuf<int32_t> ctl; // of a split plan
            LinePlan64Dev dev;
        };
    }

    struct PdeGrid
    {
        int32_t xDim = 0, yDim = 0;
        int32_t wrapX = 0, wrapY = 0;
        int32_t updateCt = 0;
        // a value-form *All call not yet run (see Prepare)
        bool pendingAll = false;
        int32_t pendingOp = 0;
        double pendingValue = 0.0;
        int device = 0;
        StreamSlot stream;
        DevBuf<double> f, d;
        Adi64 adi64;                     // DiffusionADI (plans and scratch)
        DevBuf<double> a0, a1, a2;       // uploaded per-cell arrays (rates, velocities)
        DevBuf<double> g0, g1, g2;       // uploaded ghost tables
        DevBuf<RedPartial> red;
        HostBuf<RedPartial> redHost;
        DevBuf<int32_t> ic0, ic1;        // uploaded index lists
        DevBuf<int8_t> iops;
        DevBuf<double> ivals, iout, iout2;
        cudaEvent_t evA = nullptr, evB = nullptr;

        int64_t Length() const
        {
            return static_cast<int64_t>(xDim) * yDim;
        }

        int Init(int32_t x, int32_t y, int32_t wx, int32_t wy)
        {
            xDim = x;
            yDim = y;
            wrapX = wx;
            wrapY = wy;
            device = CurrentDevice();
            HAL_TRY(CudaStatus(cudaSetDevice(device), "cudaSetDevice"));
            HAL_TRY(stream.Create("cudaStreamCreate"));
            HAL_TRY(f.Alloc(static_cast<size_t>(Length()), "cudaMalloc(pdegrid field)"));
            HAL_TRY(d.Alloc(static_cast<size_t>(Length()), "cudaMalloc(pdegrid deltas)"));
            HAL_TRY(CudaStatus(cudaMemset(f.p, 0, static_cast<size_t>(Length()) * sizeof(double)), "cudaMemset"));
            HAL_TRY(CudaStatus(cudaMemset(d.p, 0, static_cast<size_t>(Length()) * sizeof(double)), "cudaMemset"));
            HAL_TRY(red.Alloc(kRedBlocks, "cudaMalloc(reduction)"));
            HAL_TRY(redHost.Reserve(kRedBlocks, "cudaMallocHost(reduction)"));
            HAL_TRY(CudaStatus(cudaEventCreateWithFlags(&evA, cudaEventDisableTiming), "cudaEventCreate"));
            HAL_TRY(CudaStatus(cudaEventCreateWithFlags(&evB, cudaEventDisableTiming), "cudaEventCreate"));
            return HAL_CUDA_OK;
        }

        ~PdeGrid()
        {
            if (evA != nullptr)
            {
                cudaEventDestroy(evA);
            }
            if (evB != nullptr)
            {
                cudaEventDestroy(evB);
            }
        }

        // Copies n values of host array h into device buffer b (grown to
        // at least n), on the handle's stream.
        template <typename T>
        int Upload(DevBuf<T> &b, const T *h, size_t n, const char *what)
        {
            if (b.n < n || b.p == nullptr)
            {
                HAL_TRY(CudaStatus(cudaStreamSynchronize(stream.Get()), what));
                HAL_TRY(b.Alloc(n, what));
            }
            if (n > 0)
            {
                HAL_TRY(CudaStatus(cudaMemcpyAsync(b.p, h, n * sizeof(T), cudaMemcpyHostToDevice, stream.Get()),
                                   what));
            }
            return HAL_CUDA_OK;
        }

        template <typename T>
        int Ensure(DevBuf<T> &b, size_t n, const char *what)
        {
            if (b.n < n || b.p == nullptr)
            {
                HAL_TRY(CudaStatus(cudaStreamSynchronize(stream.Get()), what));
                HAL_TRY(b.Alloc(n, what));
            }
            return HAL_CUDA_OK;
        }

        int GhostTable(const double *ghost, DevBuf<double> &buf, const double **out)
        {
            *out = nullptr;
            if (ghost != nullptr)
            {
                HAL_TRY(Upload(buf, ghost, 2 * (static_cast<size_t>(xDim) + yDim), "cudaMemcpy(ghost)"));
                *out = buf.p;
            }
            return HAL_CUDA_OK;
        }

        // Internal::Diffusion2DADI (ADIequations.h:306-337, Dirichlet
        // :339-378): deltas += v - f.
        int Adi(double r, const double *ghostHost)
        {
            const double *g = nullptr;
            HAL_TRY(GhostTable(ghostHost, g0, &g));
            return adi64.Run(f.p, d.p, xDim, yDim, wrapX, wrapY, r, g, stream.Get());
        }

        int Sync(const char *who)
        {
            return CudaStatus(cudaStreamSynchronize(stream.Get()), who);
        }
    };

    // ---- Adi64 -------------------------------------------------------------
    struct Adi64::Impl
    {
        DevBuf<double> wA, wB, vB, dS;  // scratch (grown on first use)
        DevBuf<double> fac;             // periodic factors of the current sweep's lines
        DevBuf<double> segA, segB;      // split solve: values at the segments' ends
        DevBuf<int32_t> marks;          // split solve: lines to mend, CTAs arrived (zero between kernels)
        std::map<std::string, std::unique_ptr<PlanBuf64>> plans;

        int Ensure(DevBuf<double> &b, size_t n, cudaStream_t s, const char *what)
        {
            if (b.n < n || b.p == nullptr)
            {
                HAL_TRY(CudaStatus(cudaStreamSynchronize(s), what));
                HAL_TRY(b.Alloc(n, what));
            }
            return HAL_CUDA_OK;
        }

        // (each axis has its own, with its own record)
        int Plan(char axis, int32_t L, int32_t lines, double r, bool wrap, bool dirichlet, LinePlan64Dev *out)
        {
            char key[96];
            snprintf(key, sizeof(key), "%c%d|%d|%a|%d|%d", axis, L, lines, r, wrap ? 1 : 0,
                     (dirichlet && !wrap) ? 1 : 0);
            auto it = plans.find(key);
            if (it == plans.end())
            {
                LinePlan64Host h = BuildPlan64(L, r, wrap, dirichlet);
                AddSegments(h, lines);
                auto pb = std::make_unique<PlanBuf64>();
                // layout (in doubles): bh [2L], lo [L], ws [L], bs [L], zs [L],
                // and of a split line g [L], segP [segs], segQ [segs]
                const size_t Ls = static_cast<size_t>(L);
                const size_t split = h.segs > 1 ? Ls + 2 * static_cast<size_t>(h.segs) : 0;
                std::vector<double> all(6 * Ls + split, 0.0);
                if (split > 0)
                {
                    std::copy(h.g.begin(), h.g.end(), all.begin() + 6 * Ls);
                    std::copy(h.segP.begin(), h.segP.end(), all.begin() + 7 * Ls);
                    std::copy(h.segQ.begin(), h.segQ.end(), all.begin() + 7 * Ls + h.segs);
                }
                std::memcpy(all.data(), h.bh.data(), sizeof(double2) * Ls);
                std::memcpy(all.data() + 2 * Ls, h.lo.data(), sizeof(int2) * Ls);
                std::copy(h.ws.begin(), h.ws.end(), all.begin() + 3 * Ls);
                std::copy(h.bs.begin(), h.bs.end(), all.begin() + 4 * Ls);
                std::copy(h.zs.begin(), h.zs.end(), all.begin() + 5 * Ls);
                HAL_TRY(pb->buf.Alloc(all.size(), "cudaMalloc(ADI plan)"));
                HAL_TRY(CudaStatus(cudaMemcpy(pb->buf.p, all.data(), all.size() * sizeof(double),
                                              cudaMemcpyHostToDevice),
                                   "cudaMemcpy(ADI plan)"));
                pb->dev.bh = reinterpret_cast<const double2 *>(pb->buf.p);
                pb->dev.lo = reinterpret_cast<const int2 *>(pb->buf.p + 2 * Ls);
                pb->dev.ws = pb->buf.p + 3 * Ls;
                pb->dev.bs = pb->buf.p + 4 * Ls;
                pb->dev.zs = pb->buf.p + 5 * Ls;
                pb->dev.fastDiv = h.fastDiv ? 1 : 0;
                pb->dev.off = h.off;
                pb->dev.vEnd = h.vEnd;
                pb->dev.onePlusVz = h.onePlusVz;
                pb->dev.L = L;
                pb->dev.periodic = h.periodic ? 1 : 0;
                pb->dev.segs = h.segs;
                pb->dev.segLen = h.segLen;
                pb->dev.g = pb->buf.p + 6 * Ls;
                pb->dev.segP = pb->buf.p + 7 * Ls;
                pb->dev.segQ = pb->buf.p + 7 * Ls + h.segs;
                pb->dev.ctl = nullptr;
                pb->dev.mendBudget = h.mendBudget;
                if (h.segs > 1)
                {
                    std::vector<int32_t> ctl(kCtlCount + 2 * static_cast<size_t>(CtlLines(lines)), 0);
                    ctl[kCtlPeriod] = kSegMinPeriod;
                    HAL_TRY(pb->ctl.Alloc(ctl.size(), "cudaMalloc(ADI plan)"));
                    HAL_TRY(CudaStatus(cudaMemcpy(pb->ctl.p, ctl.data(), ctl.size() * sizeof(int32_t),
                                                  cudaMemcpyHostToDevice), "cudaMemcpy(ADI plan)"));
                    pb->dev.ctl = pb->ctl.p;
                }
                it = plans.emplace(key, std::move(pb)).first;
            }
            *out = it->second->dev;
            return HAL_CUDA_OK;
        }
    };

    Adi64::Adi64() : m_impl(new Impl())
    {
    }

    Adi64::~Adi64() = default;

    int Adi64::Run(const double *f, double *deltas, int32_t xDim, int32_t yDim, int32_t wrapX, int32_t wrapY,
                   double r, const double *g, cudaStream_t s)
    {
        Impl &m = *m_impl;
        const size_t n = static_cast<size_t>(xDim) * static_cast<size_t>(yDim);
        HAL_TRY(m.Ensure(m.wA, n, s, "cudaMalloc(ADI scratch)"));
        HAL_TRY(m.Ensure(m.wB, n, s, "cudaMalloc(ADI scratch)"));
        HAL_TRY(m.Ensure(m.vB, n, s, "cudaMalloc(ADI scratch)"));
        HAL_TRY(m.Ensure(m.dS, n, s, "cudaMalloc(ADI scratch)"));
        LinePlan64Dev px, py;
        HAL_TRY(m.Plan('x', xDim, yDim, r, wrapX != 0, g != nullptr, &px));
        HAL_TRY(m.Plan('y', yDim, xDim, r, wrapY != 0, g != nullptr, &py));
        // per sweep: the right-hand sides on every SM, the chains one line
        // per thread and one warp per block (the lines spread over the most
        // SMs), then the transpose that applies the periodic correction
        const size_t nFac = static_cast<size_t>(std::max(xDim, yDim));
        HAL_TRY(m.Ensure(m.fac, nFac, s, "cudaMalloc(ADI scratch)"));
        const int T = 32;
        const dim3 tb(32, 8);
        // threads for one row of lines in whole warps, at most 256 a block
        const auto rhsThreads = [](int32_t lines) {
            return std::min(256, ((lines + kRhsCells - 1) / kRhsCells + 31) / 32 * 32);
        };
        const auto rhsGrid = [&](int32_t lines, int32_t L) {
            return dim3(Blocks(lines, rhsThreads(lines) * kRhsCells),
                        static_cast<unsigned>(std::min<int32_t>(std::max<int32_t>(L, 1), 65535)));
        };
        const size_t nSeg = static_cast<size_t>(std::max(static_cast<int64_t>(px.segs) * yDim,
                                                         static_cast<int64_t>(py.segs) * xDim));
        if (px.segs > 1 || py.segs > 1)
        {
            HAL_TRY(m.Ensure(m.segA, nSeg, s, "cudaMalloc(ADI scratch)"));
            HAL_TRY(m.Ensure(m.segB, nSeg, s, "cudaMalloc(ADI scratch)"));
            const size_t nMarks = nFac + Blocks(static_cast<int64_t>(nFac), T);  // and the counts of arrived CTAs
            if (m.marks.n != nMarks || m.marks.p == nullptr)
            {
                HAL_TRY(CudaStatus(cudaStreamSynchronize(s), "cudaMalloc(ADI scratch)"));
                HAL_TRY(m.marks.Alloc(nMarks, "cudaMalloc(ADI scratch)"));
                HAL_TRY(CudaStatus(cudaMemsetAsync(m.marks.p, 0, nMarks * sizeof(int32_t), s), "ADI scratch"));
            }
        }
        // e: a scratch array that the sweep does not use otherwise (the split
        // solve keeps the right-hand sides)
        const auto chain = [&](const LinePlan64Dev &pl, int32_t lines, double *out, double *e) {
            if (pl.segs > 1)
            {
                const unsigned b = Blocks(lines, T), segs = static_cast<unsigned>(pl.segs);
                ChainedSeg(AdiSegEnds, dim3(b, segs - 1), s, m.dS.p, pl, lines, m.segA.p, out, m.fac.p);
                ChainedSeg(AdiSegElim, dim3(b, segs), s, m.dS.p, e, pl, lines, m.segA.p, m.segB.p);
                ChainedSeg(AdiSegFix, dim3(b, segs - 1), s, m.dS.p, e, pl, lines, m.segB.p, m.segA.p, m.marks.p,
                           m.marks.p + nFac);
                ChainedSeg(AdiSegBack, dim3(b, segs), s, e, out, pl, lines, m.segA.p, m.segB.p);
                ChainedSeg(AdiSegBackFix, dim3(b, segs - 1), s, e, out, pl, lines, m.segB.p, m.marks.p,
                           m.marks.p + nFac, m.fac.p);
                CountLaunch(4);
            }
            else if (pl.fastDiv)
            {
                AdiChain64<true><<<Blocks(lines, T), T, 0, s>>>(m.dS.p, out, pl, lines, m.fac.p);
            }
            else
            {
                AdiChain64<false><<<Blocks(lines, T), T, 0, s>>>(m.dS.p, out, pl, lines, m.fac.p);
            }
        };
        AdiRhs64<<<rhsGrid(yDim, xDim), rhsThreads(yDim), 0, s>>>(f, m.dS.p, xDim, yDim, wrapY, wrapX,
                                                        g ? g + 2 * static_cast<size_t>(yDim) : nullptr, g, r);
        chain(px, yDim, m.wA.p, m.vB.p);
        Transpose64<false><<<dim3((yDim + 31) / 32, (xDim + 31) / 32), tb, 0, s>>>(
            m.wA.p, m.wB.p, xDim, yDim, nullptr, px.periodic ? m.fac.p : nullptr, px.zs, px.ctl);
        AdiRhs64<<<rhsGrid(xDim, yDim), rhsThreads(xDim), 0, s>>>(m.wB.p, m.dS.p, yDim, xDim, wrapX, wrapY, g,
                                                        g ? g + 2 * static_cast<size_t>(yDim) : nullptr, r);
        chain(py, xDim, m.vB.p, m.wA.p);
        Transpose64<true><<<dim3((xDim + 31) / 32, (yDim + 31) / 32), tb, 0, s>>>(
            m.vB.p, deltas, yDim, xDim, f, py.periodic ? m.fac.p : nullptr, py.zs, py.ctl);
        CountLaunch(6);
        return LaunchStatus("DiffusionADI (FP64)");
    }
}

struct hal_cuda_pdegrid : public halcuda::PdeGrid
{
};

namespace
{
    using halcuda::CudaStatus;
    using halcuda::LaunchStatus;

    // Every entry point starts here.  A pending value-form *All call
    // (hal_cuda_pdegrid_apply_all) runs first, unless the caller is the
    // Update that takes it over (flush false).
    int Prepare(hal_cuda_pdegrid *h, const char *who, bool flush = true)
    {
        HAL_REQUIRE(h != nullptr, "%s: handle is NULL", who);
        HAL_TRY(CudaStatus(cudaSetDevice(h->device), "cudaSetDevice"));
        if (flush && h->pendingAll)
        {
            h->pendingAll = false;
            const int64_t n = h->Length();
            halcuda::ApplyAll<<<halcuda::StrideBlocks(n), 256, 0, h->stream.Get()>>>(
                h->pendingOp, h->pendingValue, nullptr, n, h->f.p, h->d.p);
            halcuda::CountLaunch();
            HAL_TRY(LaunchStatus(who));
        }
        return HAL_CUDA_OK;
    }
}

extern "C" int hal_cuda_pdegrid_create(int32_t xDim, int32_t yDim, int32_t wrapX, int32_t wrapY,
                                       hal_cuda_pdegrid **out)
{
    HAL_REQUIRE(out != nullptr, "hal_cuda_pdegrid_create: out is NULL");
    *out = nullptr;
    HAL_REQUIRE(xDim > 0 && yDim > 0, "hal_cuda_pdegrid_create: dimensions must be positive");
    HAL_REQUIRE(static_cast<int64_t>(xDim) * yDim <= INT32_MAX,
                "hal_cuda_pdegrid_create: xDim*yDim exceeds int32 (PDEGrid2D indexes cells with int32_t)");
    hal_cuda_pdegrid *h = new (std::nothrow) hal_cuda_pdegrid();
    if (h == nullptr)
    {
        halcuda::SetError("hal_cuda_pdegrid_create: out of host memory");
        return HAL_CUDA_ENOMEM;
    }
    const int rc = h->Init(xDim, yDim, wrapX != 0, wrapY != 0);
    if (rc != HAL_CUDA_OK)
    {
        delete h;
        return rc;
    }
    *out = h;
    return HAL_CUDA_OK;
}

extern "C" int hal_cuda_pdegrid_destroy(hal_cuda_pdegrid *h)
{
    if (h != nullptr)
    {
        cudaSetDevice(h->device);
        cudaStreamSynchronize(h->stream.Get());
        delete h;
    }
    return HAL_CUDA_OK;
}

extern "C" int hal_cuda_pdegrid_set_state(hal_cuda_pdegrid *h, const double *field, const double *deltas,
                                          int32_t updateCt)
{
    HAL_TRY(Prepare(h, "hal_cuda_pdegrid_set_state"));
    HAL_REQUIRE(field != nullptr, "PDEGrid::SetState arrays must match the grid length");
    cudaStream_t s = h->stream.Get();
    const size_t bytes = static_cast<size_t>(h->Length()) * sizeof(double);
    HAL_TRY(CudaStatus(cudaMemcpyAsync(h->f.p, field, bytes, cudaMemcpyHostToDevice, s), "cudaMemcpy(field)"));
    HAL_TRY(CudaStatus(deltas != nullptr ? cudaMemcpyAsync(h->d.p, deltas, bytes, cudaMemcpyHostToDevice, s)
                                         : cudaMemsetAsync(h->d.p, 0, bytes, s),
                       "cudaMemcpy(deltas)"));
    h->updateCt = updateCt;
    return h->Sync("hal_cuda_pdegrid_set_state");
}

extern "C" int hal_cuda_pdegrid_get_state(hal_cuda_pdegrid *h, double *field, double *deltas, int32_t *updateCt)
{
    HAL_TRY(Prepare(h, "hal_cuda_pdegrid_get_state"));
    cudaStream_t s = h->stream.Get();
    const size_t bytes = static_cast<size_t>(h->Length()) * sizeof(double);
    halcuda::PopulateOutput(field, bytes);
    halcuda::PopulateOutput(deltas, bytes);
    if (field != nullptr)
    {
        HAL_TRY(CudaStatus(cudaMemcpyAsync(field, h->f.p, bytes, cudaMemcpyDeviceToHost, s), "cudaMemcpy(field)"));
    }
    if (deltas != nullptr)
    {
        HAL_TRY(CudaStatus(cudaMemcpyAsync(deltas, h->d.p, bytes, cudaMemcpyDeviceToHost, s), "cudaMemcpy(deltas)"));
    }
    if (updateCt != nullptr)
    {
        *updateCt = h->updateCt;
    }
    return h->Sync("hal_cuda_pdegrid_get_state");
}

extern "C" int hal_cuda_pdegrid_apply(hal_cuda_pdegrid *h, const int32_t *ops, int32_t op, const int32_t *cells,
                                      const double *values, double value, int64_t n)
{
    const char *who = "hal_cuda_pdegrid_apply";
    HAL_TRY(Prepare(h, who));
    HAL_REQUIRE(n >= 0, "%s: negative count", who);
    if (n == 0)
    {
        return HAL_CUDA_OK;
    }
    HAL_REQUIRE(cells != nullptr, "%s: cells is NULL", who);
    HAL_REQUIRE(ops != nullptr || (op >= HAL_CUDA_CELL_SET && op <= HAL_CUDA_CELL_SCALE), "%s: unknown operation %d",
                who, op);
    const int64_t len = h->Length();
    // stable order by cell: entries of a cell keep their list order
    std::vector<int64_t> order(static_cast<size_t>(n));
    std::iota(order.begin(), order.end(), int64_t(0));
    for (int64_t k = 0; k < n; k++)
    {
        HAL_REQUIRE(cells[k] >= 0 && cells[k] < len, "%s: cell %d outside the grid of %lld cells", who, cells[k],
                    static_cast<long long>(len));
        if (ops != nullptr)
        {
            HAL_REQUIRE(ops[k] >= HAL_CUDA_CELL_SET && ops[k] <= HAL_CUDA_CELL_SCALE, "%s: unknown operation %d", who,
                        ops[k]);
        }
    }
    std::stable_sort(order.begin(), order.end(), [&](int64_t a, int64_t b) { return cells[a] < cells[b]; });
    std::vector<int32_t> sc(static_cast<size_t>(n));
    std::vector<int8_t> so(static_cast<size_t>(n));
    std::vector<double> sv(static_cast<size_t>(n));
    std::vector<int32_t> runs;
    for (int64_t k = 0; k < n; k++)
    {
        const int64_t e = order[static_cast<size_t>(k)];
        sc[k] = cells[e];
        so[k] = static_cast<int8_t>(ops != nullptr ? ops[e] : op);
        sv[k] = values != nullptr ? values[e] : value;
        if (k == 0 || sc[k] != sc[k - 1])
        {
            runs.push_back(static_cast<int32_t>(k));
        }
    }
    runs.push_back(static_cast<int32_t>(n));
    const int32_t nRuns = static_cast<int32_t>(runs.size()) - 1;
    HAL_TRY(h->Upload(h->ic0, sc.data(), sc.size(), "cudaMemcpy(cells)"));
    HAL_TRY(h->Upload(h->iops, so.data(), so.size(), "cudaMemcpy(ops)"));
    HAL_TRY(h->Upload(h->ivals, sv.data(), sv.size(), "cudaMemcpy(values)"));
    HAL_TRY(h->Upload(h->ic1, runs.data(), runs.size(), "cudaMemcpy(runs)"));
    halcuda::ApplyRuns<<<halcuda::Blocks(nRuns, 256), 256, 0, h->stream.Get()>>>(
        h->ic0.p, h->iops.p, h->ivals.p, h->ic1.p, nRuns, h->f.p, h->d.p);
    halcuda::CountLaunch();
    HAL_TRY(LaunchStatus(who));
    // the host lists are copied out before this call returns
    return h->Sync(who);
}

extern "C" int hal_cuda_pdegrid_apply_agents(hal_cuda_pdegrid *h, hal_cuda_agents *agents, int32_t op, double value,
                                             const double *perAgent)
{
    const char *who = "hal_cuda_pdegrid_apply_agents";
    HAL_TRY(Prepare(h, who));
    HAL_REQUIRE(agents != nullptr, "%s: agents is NULL", who);
    HAL_REQUIRE(op >= HAL_CUDA_CELL_SET && op <= HAL_CUDA_CELL_SCALE, "%s: unknown operation %d", who, op);
    const halcuda::AgentBinsView v = halcuda::AgentsBins(agents);
    HAL_REQUIRE(v.xDim == h->xDim && v.yDim == h->yDim, "%s: agent grid %dx%d differs from the field %dx%d", who,
                v.xDim, v.yDim, h->xDim, h->yDim);
    HAL_REQUIRE(v.device == h->device, "%s: the agents live on another device", who);
    if (v.n == 0)
    {
        return HAL_CUDA_OK;
    }
    cudaStream_t s = h->stream.Get();
    const double *pa = nullptr;
    if (perAgent != nullptr)
    {
        HAL_TRY(h->Upload(h->ivals, perAgent, static_cast<size_t>(v.n), "cudaMemcpy(per-agent values)"));
        pa = h->ivals.p;
    }
    // the agents' last binning completes before, and their next one starts
    // after, this grid's use of it
    HAL_TRY(CudaStatus(cudaEventRecord(h->evA, v.stream), "cudaEventRecord"));
    HAL_TRY(CudaStatus(cudaStreamWaitEvent(s, h->evA, 0), "cudaStreamWaitEvent"));
    halcuda::ApplyAgents<<<halcuda::Blocks(v.n, 256), 256, 0, s>>>(v.offsets, v.bucket, v.cellOf, v.n, op, value, pa,
                                                                   h->f.p, h->d.p);
    halcuda::CountLaunch();
    HAL_TRY(LaunchStatus(who));
    HAL_TRY(CudaStatus(cudaEventRecord(h->evB, s), "cudaEventRecord"));
    HAL_TRY(CudaStatus(cudaStreamWaitEvent(v.stream, h->evB, 0), "cudaStreamWaitEvent"));
    if (perAgent != nullptr)
    {
        return h->Sync(who);  // the host values are read before the call returns
    }
    return HAL_CUDA_OK;
}

extern "C" int hal_cuda_pdegrid_apply_all(hal_cuda_pdegrid *h, int32_t op, double value, const double *perCell)
{
    const char *who = "hal_cuda_pdegrid_apply_all";
    HAL_TRY(Prepare(h, who));
    HAL_REQUIRE(op >= HAL_CUDA_CELL_SET && op <= HAL_CUDA_CELL_SCALE, "%s: unknown operation %d", who, op);
    cudaStream_t s = h->stream.Get();
    const int64_t n = h->Length();
    if (perCell == nullptr)
    {
        // deferred: the next call runs it first, and an Update right after
        // it runs it in its own pass (ApplyAllCommit)
        h->pendingAll = true;
        h->pendingOp = op;
        h->pendingValue = value;
        return HAL_CUDA_OK;
    }
    HAL_TRY(h->Upload(h->a0, perCell, static_cast<size_t>(n), "cudaMemcpy(values)"));
    const double *pc = h->a0.p;
    halcuda::ApplyAll<<<halcuda::StrideBlocks(n), 256, 0, s>>>(op, value, pc, n, h->f.p, h->d.p);
    halcuda::CountLaunch();
    HAL_TRY(LaunchStatus(who));
    return h->Sync(who);
}

extern "C" int hal_cuda_pdegrid_update(hal_cuda_pdegrid *h)
{
    HAL_TRY(Prepare(h, "hal_cuda_pdegrid_update", false));
    const int64_t n = h->Length();
    if (h->pendingAll)
    {
        h->pendingAll = false;
        halcuda::ApplyAllCommit<<<halcuda::StrideBlocks(n), 256, 0, h->stream.Get()>>>(
            h->pendingOp, h->pendingValue, n, h->f.p, h->d.p);
    }
    else
    {
        halcuda::Commit<<<halcuda::StrideBlocks(n), 256, 0, h->stream.Get()>>>(n, h->f.p, h->d.p);
    }
    halcuda::CountLaunch();
    h->updateCt++;
    return LaunchStatus("hal_cuda_pdegrid_update");
}

extern "C" int hal_cuda_pdegrid_set_non_negative(hal_cuda_pdegrid *h)
{
    HAL_TRY(Prepare(h, "hal_cuda_pdegrid_set_non_negative"));
    const int64_t n = h->Length();
    halcuda::NonNegative<<<halcuda::StrideBlocks(n), 256, 0, h->stream.Get()>>>(n, h->f.p, h->d.p);
    halcuda::CountLaunch();
    return LaunchStatus("hal_cuda_pdegrid_set_non_negative");
}

extern "C" int hal_cuda_pdegrid_get_cells(hal_cuda_pdegrid *h, const int32_t *cells, int64_t n, double *out)
{
    const char *who = "hal_cuda_pdegrid_get_cells";
    HAL_TRY(Prepare(h, who));
    HAL_REQUIRE(n >= 0 && (n == 0 || (cells != nullptr && out != nullptr)), "%s: NULL array", who);
    if (n == 0)
    {
        return HAL_CUDA_OK;
    }
    const int64_t len = h->Length();
    for (int64_t k = 0; k < n; k++)
    {
        HAL_REQUIRE(cells[k] >= 0 && cells[k] < len, "%s: cell %d outside the grid", who, cells[k]);
    }
    cudaStream_t s = h->stream.Get();
    HAL_TRY(h->Upload(h->ic0, cells, static_cast<size_t>(n), "cudaMemcpy(cells)"));
    HAL_TRY(h->Ensure(h->iout, static_cast<size_t>(n), "cudaMalloc(values)"));
    halcuda::Gather<<<halcuda::Blocks(n, 256), 256, 0, s>>>(h->ic0.p, n, h->f.p, h->iout.p);
    halcuda::CountLaunch();
    HAL_TRY(LaunchStatus(who));
    HAL_TRY(CudaStatus(cudaMemcpyAsync(out, h->iout.p, static_cast<size_t>(n) * sizeof(double), cudaMemcpyDeviceToHost,
                                       s),
                       "cudaMemcpy(values)"));
    return h->Sync(who);
}

extern "C" int hal_cuda_pdegrid_gradient(hal_cuda_pdegrid *h, const int32_t *xs, const int32_t *ys, int64_t n,
                                         int32_t useBoundary, double boundaryValue, double *gradX, double *gradY)
{
    const char *who = "hal_cuda_pdegrid_gradient";
    HAL_TRY(Prepare(h, who));
    HAL_REQUIRE(n >= 0 && (n == 0 || (xs != nullptr && ys != nullptr && gradX != nullptr && gradY != nullptr)),
                "%s: NULL array", who);
    if (n == 0)
    {
        return HAL_CUDA_OK;
    }
    for (int64_t k = 0; k < n; k++)
    {
        HAL_REQUIRE(xs[k] >= 0 && xs[k] < h->xDim && ys[k] >= 0 && ys[k] < h->yDim, "%s: point (%d, %d) outside the grid",
                    who, xs[k], ys[k]);
    }
    cudaStream_t s = h->stream.Get();
    HAL_TRY(h->Upload(h->ic0, xs, static_cast<size_t>(n), "cudaMemcpy(points)"));
    HAL_TRY(h->Upload(h->ic1, ys, static_cast<size_t>(n), "cudaMemcpy(points)"));
    HAL_TRY(h->Ensure(h->iout, static_cast<size_t>(n), "cudaMalloc(gradients)"));
    HAL_TRY(h->Ensure(h->iout2, static_cast<size_t>(n), "cudaMalloc(gradients)"));
    halcuda::Gradients<<<halcuda::Blocks(n, 256), 256, 0, s>>>(h->ic0.p, h->ic1.p, n, h->f.p, h->xDim, h->yDim,
                                                               h->wrapX, h->wrapY, useBoundary, boundaryValue,
                                                               h->iout.p, h->iout2.p);
    halcuda::CountLaunch();
    HAL_TRY(LaunchStatus(who));
    const size_t bytes = static_cast<size_t>(n) * sizeof(double);
    HAL_TRY(CudaStatus(cudaMemcpyAsync(gradX, h->iout.p, bytes, cudaMemcpyDeviceToHost, s), "cudaMemcpy(gradients)"));
    HAL_TRY(CudaStatus(cudaMemcpyAsync(gradY, h->iout2.p, bytes, cudaMemcpyDeviceToHost, s), "cudaMemcpy(gradients)"));
    return h->Sync(who);
}

extern "C" int hal_cuda_pdegrid_stats(hal_cuda_pdegrid *h, double denomOffset, double *stats)
{
    const char *who = "hal_cuda_pdegrid_stats";
    HAL_TRY(Prepare(h, who));
    HAL_REQUIRE(stats != nullptr, "%s: stats is NULL", who);
    cudaStream_t s = h->stream.Get();
    const int64_t n = h->Length();
    const bool scaled = !std::isnan(denomOffset);
    halcuda::Reduce<<<halcuda::kRedBlocks, halcuda::kRedThreads, 0, s>>>(n, h->f.p, h->d.p, denomOffset, scaled,
                                                                         h->red.p);
    halcuda::CountLaunch();
    HAL_TRY(LaunchStatus(who));
    HAL_TRY(CudaStatus(cudaMemcpyAsync(h->redHost.p, h->red.p, halcuda::kRedBlocks * sizeof(halcuda::RedPartial),
                                       cudaMemcpyDeviceToHost, s),
                       "cudaMemcpy(reduction)"));
    HAL_TRY(h->Sync(who));
    // combine the blocks in order (the same rules as within a block)
    double maxV = -INFINITY, minV = INFINITY, sum = 0.0, md = 0.0, ms = 0.0;
    long long maxI = -1, minI = -1;
    for (int b = 0; b < halcuda::kRedBlocks; b++)
    {
        const halcuda::RedPartial &p = h->redHost.p[b];
        if (maxV < p.maxV || (!(p.maxV < maxV) && p.maxI > maxI))
        {
            maxV = p.maxV;
            maxI = p.maxI;
        }
        if (p.minV < minV || (!(minV < p.minV) && p.minI > minI))
        {
            minV = p.minV;
            minI = p.minI;
        }
        sum += p.sum;
        md = std::fmax(md, p.maxDelta);
        ms = std::fmax(ms, p.maxScaled);
    }
    // GetMax / GetMin start from lowest() / max() (PDEGrid2D.h:142-164),
    // which an all -inf (+inf) field never replaces
    const double lowest = -std::numeric_limits<double>::max();
    const double highest = std::numeric_limits<double>::max();
    stats[0] = (maxV < lowest) ? lowest : maxV;
    stats[1] = (highest < minV) ? highest : minV;
    stats[2] = sum / static_cast<double>(n);
    stats[3] = md;
    stats[4] = scaled ? ms : NAN;
    return HAL_CUDA_OK;
}

namespace
{
    // A stencil of stencil64.cuh over the whole grid, into the deltas.
    template <class Cell>
    int RunCells(hal_cuda_pdegrid *h, const Cell &cell, const char *who)
    {
        halcuda::stencil64::Cells64Kernel<<<halcuda::stencil64::Cells64Grid(h->xDim, h->yDim), 256, 0,
                                            h->stream.Get()>>>(cell, h->xDim, h->yDim);
        halcuda::CountLaunch();
        HAL_TRY(LaunchStatus(who));
        // host arrays (rates, velocities, ghost tables) were copied
        // asynchronously from the caller's memory: finish before returning
        return h->Sync(who);
    }

    int SignOf(double v)
    {
        return (v > 0) ? 1 : ((v < 0) ? -1 : 0);
    }
}

extern "C" int hal_cuda_pdegrid_diffusion(hal_cuda_pdegrid *h, double diffCoef, const double *ghost)
{
    const char *who = "hal_cuda_pdegrid_diffusion";
    HAL_TRY(Prepare(h, who));
    HAL_REQUIRE(!(diffCoef > 0.25), "Diffusion rate above stable maximum value of 0.25");
    const double *g = nullptr;
    HAL_TRY(h->GhostTable(ghost, h->g0, &g));
    const halcuda::stencil64::Diffuse64Cell cell{h->f.p, h->d.p, g, diffCoef, h->xDim, h->yDim, h->wrapX, h->wrapY};
    return RunCells(h, cell, who);
}

extern "C" int hal_cuda_pdegrid_diffusion_var(hal_cuda_pdegrid *h, const double *ratesX, const double *ratesY)
{
    const char *who = "hal_cuda_pdegrid_diffusion_var";
    HAL_TRY(Prepare(h, who));
    HAL_REQUIRE(ratesX != nullptr && ratesY != nullptr, "%s: NULL rate array", who);
    const size_t n = static_cast<size_t>(h->Length());
    HAL_TRY(h->Upload(h->a0, ratesX, n, "cudaMemcpy(rates)"));
    HAL_TRY(h->Upload(h->a1, ratesY, n, "cudaMemcpy(rates)"));
    const halcuda::stencil64::DiffuseVar64Cell cell{h->f.p, h->d.p, h->a0.p, h->a1.p, h->xDim, h->yDim, h->wrapX,
                                                    h->wrapY};
    return RunCells(h, cell, who);
}

extern "C" int hal_cuda_pdegrid_diffusion_adi(hal_cuda_pdegrid *h, double diffRate, const double *ghost)
{
    const char *who = "hal_cuda_pdegrid_diffusion_adi";
    HAL_TRY(Prepare(h, who));
    HAL_TRY(h->Adi(diffRate, ghost));
    return ghost != nullptr ? h->Sync(who) : HAL_CUDA_OK;
}

extern "C" int hal_cuda_pdegrid_advection(hal_cuda_pdegrid *h, double xVel, double yVel, const double *ghost)
{
    const char *who = "hal_cuda_pdegrid_advection";
    HAL_TRY(Prepare(h, who));
    HAL_REQUIRE(!((std::fabs(xVel) + std::fabs(yVel)) > 0.5),
                "Advection rate component sum above stable maximum value of 0.5");
    const double *g = nullptr;
    HAL_TRY(h->GhostTable(ghost, h->g0, &g));
    const halcuda::stencil64::Advect64Cell cell{h->f.p, h->d.p, g, xVel, yVel, h->xDim, h->yDim, h->wrapX, h->wrapY,
                                                SignOf(xVel), SignOf(yVel)};
    return RunCells(h, cell, who);
}

extern "C" int hal_cuda_pdegrid_advection_var(hal_cuda_pdegrid *h, const double *xVels, const double *yVels,
                                              const double *ghost, const double *ghostXVel, const double *ghostYVel)
{
    const char *who = "hal_cuda_pdegrid_advection_var";
    HAL_TRY(Prepare(h, who));
    HAL_REQUIRE(xVels != nullptr && yVels != nullptr, "%s: NULL velocity array", who);
    const size_t n = static_cast<size_t>(h->Length());
    HAL_TRY(h->Upload(h->a0, xVels, n, "cudaMemcpy(velocities)"));
    HAL_TRY(h->Upload(h->a1, yVels, n, "cudaMemcpy(velocities)"));
    const double *g = nullptr, *gx = nullptr, *gy = nullptr;
    HAL_TRY(h->GhostTable(ghost, h->g0, &g));
    HAL_TRY(h->GhostTable(ghostXVel, h->g1, &gx));
    HAL_TRY(h->GhostTable(ghostYVel, h->g2, &gy));
    const halcuda::stencil64::AdvectVar64Cell cell{h->f.p, h->d.p, h->a0.p, h->a1.p, g, gx, gy,
                                                   h->xDim, h->yDim, h->wrapX, h->wrapY};
    return RunCells(h, cell, who);
}

extern "C" int hal_cuda_pdegrid_sync(hal_cuda_pdegrid *h)
{
    HAL_TRY(Prepare(h, "hal_cuda_pdegrid_sync"));
    return h->Sync("hal_cuda_pdegrid_sync");
}

extern "C" void *hal_cuda_pdegrid_stream(hal_cuda_pdegrid *h)
{
    return h ? static_cast<void *>(h->stream.Get()) : nullptr;
}

extern "C" int hal_cuda_pdegrid_set_stream(hal_cuda_pdegrid *h, void *stream)
{
    HAL_TRY(Prepare(h, "hal_cuda_pdegrid_set_stream"));  // a pending *All runs on the old stream
    h->stream.Set(stream);
    return HAL_CUDA_OK;
}

extern "C" int hal_cuda_pdegrid_dims(hal_cuda_pdegrid *h, int32_t *dims)
{
    HAL_REQUIRE(h != nullptr && dims != nullptr, "hal_cuda_pdegrid_dims: NULL argument");
    dims[0] = h->xDim;
    dims[1] = h->yDim;
    dims[2] = h->wrapX;
    dims[3] = h->wrapY;
    dims[4] = h->updateCt;
    return HAL_CUDA_OK;
}

extern "C" int hal_cuda_check_plan_division(const double *num, int64_t nNum, const double *den, int32_t nDen,
                                            int64_t *mismatches)
{
    using namespace halcuda;
    HAL_REQUIRE(num != nullptr && den != nullptr && mismatches != nullptr,
                "hal_cuda_check_plan_division: NULL argument");
    HAL_REQUIRE(nNum >= 0 && nDen >= 0, "hal_cuda_check_plan_division: negative count");
    std::vector<double2> bh(static_cast<size_t>(nDen));
    std::vector<int2> lo(static_cast<size_t>(nDen));
    for (int32_t j = 0; j < nDen; j++)
    {
        HAL_REQUIRE(PlanDivisorInRange(den[j]),
                    "hal_cuda_check_plan_division: divisor %d (%g) outside [2^-20, 2^20]", j, den[j]);
        PlanReciprocal(den[j], &bh[j], &lo[j]);
    }
    HAL_TRY(CudaStatus(cudaSetDevice(CurrentDevice()), "cudaSetDevice"));
    DevBuf<double> dNum;
    DevBuf<double2> dBh;
    DevBuf<int2> dLo;
    DevBuf<unsigned long long> dBad;
    HAL_TRY(dNum.Alloc(static_cast<size_t>(std::max<int64_t>(nNum, 1)), "cudaMalloc(division check)"));
    HAL_TRY(dBh.Alloc(static_cast<size_t>(std::max<int32_t>(nDen, 1)), "cudaMalloc(division check)"));
    HAL_TRY(dLo.Alloc(static_cast<size_t>(std::max<int32_t>(nDen, 1)), "cudaMalloc(division check)"));
    HAL_TRY(dBad.Alloc(1, "cudaMalloc(division check)"));
    HAL_TRY(CudaStatus(cudaMemcpy(dNum.p, num, sizeof(double) * nNum, cudaMemcpyHostToDevice), "cudaMemcpy"));
    HAL_TRY(CudaStatus(cudaMemcpy(dBh.p, bh.data(), sizeof(double2) * bh.size(), cudaMemcpyHostToDevice),
                       "cudaMemcpy"));
    HAL_TRY(CudaStatus(cudaMemcpy(dLo.p, lo.data(), sizeof(int2) * lo.size(), cudaMemcpyHostToDevice),
                       "cudaMemcpy"));
    HAL_TRY(CudaStatus(cudaMemset(dBad.p, 0, sizeof(unsigned long long)), "cudaMemset"));
    if (nNum > 0 && nDen > 0)
    {
        CheckPlanDivision<<<StrideBlocks(nNum), 256>>>(dNum.p, nNum, dBh.p, dLo.p, nDen, dBad.p);
        CountLaunch();
        HAL_TRY(LaunchStatus("CheckPlanDivision"));
    }
    unsigned long long bad = 0;
    HAL_TRY(CudaStatus(cudaMemcpy(&bad, dBad.p, sizeof(bad), cudaMemcpyDeviceToHost), "cudaMemcpy"));
    *mismatches = static_cast<int64_t>(bad);
    return HAL_CUDA_OK;
}
