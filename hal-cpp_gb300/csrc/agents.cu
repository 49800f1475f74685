// agents.cu -- cell-bucket agent forces (IAgentForceBackend2D) on sm_103a.
//
// The CPU backend (src/Agents/CpuAgentForceBackend2D.cpp:66-176) runs four
// serial passes: count agents per cell, exclusive prefix into offsets, stable
// scatter of agent indices, and a per-agent scan of the surrounding cells
// summing a linear spring force.  Here each pass is data-parallel:
//   BinCount     one thread per agent: clamped cell, atomic count, arrival rank
//   scan         reduce-then-scan over the cells (at most three launches, no spin
//                waits; in a resident run the move before adds up the tiles: 20k
//                agents in 256^2 17.9 -> 16.5 us per tick, 200k in 1024^2 36.4 ->
//                33.9, 400k in 2048^2 52.9 -> 49.5)
//   Scatter      agent -> offsets[cell] + arrival rank (order within a cell is
//                the atomic arrival order, not yet the CPU's)
//   Stabilize    one thread per arrival-order slot: its agent counts the
//                lower-indexed agents of its cell, which gives exactly the
//                CPU's slot; it writes the final bucket and a cell-sorted copy
//                of positions and radii
//   Forces       one thread per sorted slot walks the cell window x-major then
//                y, and each cell's slots in order -- the CPU's summation
//                order -- and writes the agent's velocity delta.
// The binning is integer work and matches the CPU bit for bit: the cell of a
// position is floored in the precision the caller gave it (FP64 on the
// interface path, as the CPU does; FP32 on the resident path, where the CPU
// fed the same float32 values bins identically).  The force sum runs in FP32
// on the resident path and in FP64 with IEEE round-to-nearest operations (no
// contraction) on the FP64 interface path, where positions stay FP64 end to
// end and the result matches the CPU backend bit for bit.
#include "common.cuh"
#include "agent_window.h"
#include "agents_wells.h"

#include <cmath>
#include <type_traits>

namespace halcuda
{
    namespace
    {
        // Scan tiles of 4096 cells: 256 threads, each with 16 cells in four
        // 16-byte groups, so every thread has four loads in flight.
        constexpr int kScanThreads = 256;
        constexpr int kScanGroups = 4;
        constexpr int kScanItems = 4 * kScanGroups;
        constexpr int kScanTile = kScanThreads * kScanItems;
        // tiles whose prefix ScanApplySum forms itself (4.19M cells)
        constexpr int kScanSumTiles = kAgentScanSumTiles;

        // Position pairs in the precision of the path: float2 on the FP32
        // resident path, double2 on the FP64 interface path.
        template <typename T>
        struct Vec2;
        template <>
        struct Vec2<float>
        {
            using Type = float2;
            __device__ static float2 Make(float x, float y) { return make_float2(x, y); }
        };
        template <>
        struct Vec2<double>
        {
            using Type = double2;
            __device__ static double2 Make(double x, double y) { return make_double2(x, y); }
        };
        template <typename T>
        using V2 = typename Vec2<T>::Type;

        // AgentForceCellCoord (CpuAgentForceBackend2D.cpp:14-27): the floor is
        // taken in the precision of the positions, as the CPU takes it in FP64.
        __device__ __forceinline__ int32_t Floor32(float v) { return static_cast<int32_t>(floorf(v)); }
        __device__ __forceinline__ int32_t Floor32(double v) { return static_cast<int32_t>(floor(v)); }

        template <typename TP>
        __device__ __forceinline__ int32_t CellCoord(TP v, int32_t dim)
        {
            int32_t c = Floor32(v);
            c = (c < 0) ? 0 : c;
            c = (c >= dim) ? dim - 1 : c;
            return c;
        }

        // Programmatic dependent launch (LaunchChained): the next kernel of a
        // dispatch may be scheduled once every CTA of this one has started;
        // each kernel waits for its predecessor to complete before it touches
        // any buffer (both are no-ops in a plain launch).
        __device__ __forceinline__ void ChainEntry()
        {
            asm volatile("griddepcontrol.launch_dependents;");
            asm volatile("griddepcontrol.wait;" ::: "memory");
        }

        template <typename TP>
        __global__ void BinCount(const TP *__restrict__ pos, int32_t n, int32_t xDim, int32_t yDim,
                                 V2<TP> *__restrict__ posF, int32_t *__restrict__ cellOf,
                                 int32_t *__restrict__ arrival, int32_t *__restrict__ counts)
        {
            ChainEntry();
            int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
            if (i >= n)
            {
                return;
            }
            const TP px = pos[2 * static_cast<int64_t>(i)];
            const TP py = pos[2 * static_cast<int64_t>(i) + 1];
            if (posF != nullptr)  // null when the positions are already V2-aligned
            {
                posF[i] = Vec2<TP>::Make(px, py);
            }
            int32_t c = CellCoord(px, xDim) * yDim + CellCoord(py, yDim);
            cellOf[i] = c;
            arrival[i] = atomicAdd(counts + c, 1);
        }

        // A kernel of the agent dispatch, launched with programmatic stream
        // serialization so that its launch overlaps its predecessor's tail
        // (the kernels start with ChainEntry).
        template <typename... KArgs, typename... Args>
        void LaunchChained(void (*kernel)(KArgs...), unsigned grid, unsigned block, cudaStream_t s, Args... args)
        {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(grid);
            cfg.blockDim = dim3(block);
            cfg.dynamicSmemBytes = 0;
            cfg.stream = s;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            at[0].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
        }

        // The same kernels launched after their predecessor is complete, for
        // work that differs much between CTAs: CTAs that start early fill the
        // SMs that the ending kernel leaves, and a few SMs then hold the heavy
        // ones (ForcesGroup64 with a pile of 2586 agents: 2.9 against 1.5 ms).
        template <typename... KArgs, typename... Args>
        void LaunchAfter(void (*kernel)(KArgs...), unsigned grid, unsigned block, cudaStream_t s, Args... args)
        {
            kernel<<<grid, block, 0, s>>>(static_cast<KArgs>(args)...);
        }

        // Adds the calling lanes' agents to the sums of their cells' scan tiles,
        // one atomic per tile a warp meets (neighbouring slots share most).
        __device__ __forceinline__ void AddToTiles(int32_t *__restrict__ tileSums, int32_t cell)
        {
            const int32_t tile = cell / kScanTile;
            const uint32_t same = __match_any_sync(__activemask(), tile);
            if (static_cast<int>(threadIdx.x & 31) == __ffs(same) - 1)
            {
                atomicAdd(tileSums + tile, __popc(same));
            }
        }

        // Inclusive warp scan.
        __device__ __forceinline__ int32_t WarpScan(int32_t v, int lane)
        {
#pragma unroll
            for (int d = 1; d < 32; d <<= 1)
            {
                int32_t t = __shfl_up_sync(0xffffffffu, v, d);
                if (lane >= d)
                {
                    v += t;
                }
            }
            return v;
        }

        // Exclusive block scan of one value per thread; returns the block total.
        __device__ __forceinline__ int32_t BlockExclusiveScan(int32_t v, int32_t &excl)
        {
            __shared__ int32_t warpSums[32];
            const int lane = threadIdx.x & 31;
            const int warp = threadIdx.x >> 5;
            const int nwarps = blockDim.x >> 5;
            int32_t inc = WarpScan(v, lane);
            if (lane == 31)
            {
                warpSums[warp] = inc;
            }
            __syncthreads();
            if (warp == 0)
            {
                int32_t s = (lane < nwarps) ? warpSums[lane] : 0;
                int32_t si = WarpScan(s, lane);
                if (lane < nwarps)
                {
                    warpSums[lane] = si - s;  // exclusive prefix of the warp sums
                }
            }
            __syncthreads();
            excl = inc - v + warpSums[warp];
            __shared__ int32_t s_total;
            if (threadIdx.x == blockDim.x - 1)
            {
                s_total = excl + v;
            }
            __syncthreads();
            const int32_t total = s_total;
            __syncthreads();
            return total;
        }

        // Pass 1 of the scan: per-tile sums.
        // Four consecutive cells [base, base + 4): one 16-byte access when the
        // four are in range and aligned, element by element otherwise.
        __device__ __forceinline__ bool Vec4Ok(const int32_t *p, int64_t base, int64_t C)
        {
            return base + 4 <= C && ((reinterpret_cast<uintptr_t>(p + base) & 15u) == 0u);
        }

        __device__ __forceinline__ void LoadItems(const int32_t *__restrict__ p, int64_t base, int64_t C,
                                                  int32_t *v)
        {
            if (Vec4Ok(p, base, C))
            {
                const int4 t = *reinterpret_cast<const int4 *>(p + base);
                v[0] = t.x;
                v[1] = t.y;
                v[2] = t.z;
                v[3] = t.w;
                return;
            }
#pragma unroll
            for (int q = 0; q < 4; q++)
            {
                v[q] = (base + q < C) ? p[base + q] : 0;
            }
        }

        __device__ __forceinline__ void StoreItems(int32_t *__restrict__ p, int64_t base, int64_t C, const int32_t *v)
        {
            if (Vec4Ok(p, base, C))
            {
                *reinterpret_cast<int4 *>(p + base) = make_int4(v[0], v[1], v[2], v[3]);
                return;
            }
#pragma unroll
            for (int q = 0; q < 4; q++)
            {
                if (base + q < C)
                {
                    p[base + q] = v[q];
                }
            }
        }

        // The tile sum needs no order: group g of a thread is cells tile +
        // g * 1024 + 4 * thread, so each warp's loads are contiguous.
        __global__ void __launch_bounds__(kScanThreads) ScanReduce(const int32_t *__restrict__ counts, int64_t C,
                                                                   int32_t *__restrict__ tileSums)
        {
            ChainEntry();
            const int64_t tile0 = static_cast<int64_t>(blockIdx.x) * kScanTile;
            int32_t v[kScanItems];
#pragma unroll
            for (int g = 0; g < kScanGroups; g++)
            {
                LoadItems(counts, tile0 + g * (4 * kScanThreads) + 4 * threadIdx.x, C, v + 4 * g);
            }
            int32_t s = 0;
#pragma unroll
            for (int q = 0; q < kScanItems; q++)
            {
                s += v[q];
            }
            int32_t excl;
            int32_t total = BlockExclusiveScan(s, excl);
            if (threadIdx.x == 0)
            {
                tileSums[blockIdx.x] = total;
            }
        }

        // Pass 2: exclusive scan of the tile sums by one CTA (looping over
        // chunks of kScanThreads).
        __global__ void __launch_bounds__(kScanThreads) ScanTiles(int32_t *__restrict__ tileSums, int32_t nTiles)
        {
            ChainEntry();
            int32_t carry = 0;
            for (int32_t base = 0; base < nTiles; base += kScanThreads)
            {
                int32_t idx = base + threadIdx.x;
                int32_t v = (idx < nTiles) ? tileSums[idx] : 0;
                int32_t excl;
                int32_t total = BlockExclusiveScan(v, excl);
                if (idx < nTiles)
                {
                    tileSums[idx] = carry + excl;
                }
                carry += total;
            }
        }

        // The counts are cleared by the scan as it reads them, writing only the
        // 4-cell groups that hold a count; a memset before the binning clears
        // counts not known to be zero.  With every group written, clearing in
        // the scan had measured 3.5x slower than a memset at 109M cells; with
        // only the occupied groups it is faster at both measured sizes (4.19M
        // cells, 1M agents: 119.2 -> 115.0 us per dispatch; 109M cells, 5.2M
        // agents: agent pass 0.818 -> 0.772 ms).

        // The cells of a thread of passes 3: kScanItems consecutive cells
        // from tile + thread * kScanItems (in order, for the exclusive scan),
        // loaded as four 16-byte groups.  With `clear` the groups holding a
        // count are written back as zeros (most cells are empty, and an empty
        // group is already cleared).
        __device__ __forceinline__ void LoadThreadCells(int32_t *__restrict__ counts, int64_t base, int64_t C,
                                                        bool clear, int32_t (&v)[kScanItems])
        {
#pragma unroll
            for (int g = 0; g < kScanGroups; g++)
            {
                LoadItems(counts, base + 4 * g, C, v + 4 * g);
            }
            if (clear)
            {
#pragma unroll
                for (int g = 0; g < kScanGroups; g++)
                {
                    if ((v[4 * g] | v[4 * g + 1] | v[4 * g + 2] | v[4 * g + 3]) != 0)
                    {
                        const int32_t zeros[4] = {0, 0, 0, 0};
                        StoreItems(counts, base + 4 * g, C, zeros);
                    }
                }
            }
        }

        // The thread's exclusive offsets from its first one, stored as four
        // 16-byte groups.
        __device__ __forceinline__ void StoreThreadOffsets(int32_t *__restrict__ offsets, int64_t base, int64_t C,
                                                           int32_t first, const int32_t (&v)[kScanItems])
        {
            int32_t o[kScanItems];
            o[0] = first;
#pragma unroll
            for (int q = 1; q < kScanItems; q++)
            {
                o[q] = o[q - 1] + v[q - 1];
            }
#pragma unroll
            for (int g = 0; g < kScanGroups; g++)
            {
                StoreItems(offsets, base + 4 * g, C, o + 4 * g);
            }
        }

        // Pass 3: tile-local exclusive scan plus the tile prefix -> offsets.
        // With CLEAR it also zeroes the counts it has read (only the groups
        // holding one), so the next binning starts from zero without a memset.
        template <bool CLEAR>
        __global__ void __launch_bounds__(kScanThreads) ScanApply(int32_t *__restrict__ counts, int64_t C,
                                                                  const int32_t *__restrict__ tilePrefix,
                                                                  int32_t *__restrict__ offsets, int32_t n)
        {
            ChainEntry();
            const int64_t base = static_cast<int64_t>(blockIdx.x) * kScanTile + threadIdx.x * kScanItems;
            int32_t v[kScanItems];
            LoadThreadCells(counts, base, C, CLEAR, v);
            int32_t s = 0;
#pragma unroll
            for (int q = 0; q < kScanItems; q++)
            {
                s += v[q];
            }
            int32_t excl;
            BlockExclusiveScan(s, excl);
            StoreThreadOffsets(offsets, base, C, tilePrefix[blockIdx.x] + excl, v);
            if (blockIdx.x == 0 && threadIdx.x == 0)
            {
                offsets[C] = n;
            }
        }

        // Passes 2 and 3 in one launch, for grids of at most kScanSumTiles
        // tiles: each CTA reduces the tile sums before its own (a few per
        // thread) into its tile's prefix, then runs ScanApply<true>'s tile
        // scan.  This saves the single-CTA ScanTiles launch between them.
        __global__ void __launch_bounds__(kScanThreads) ScanApplySum(int32_t *__restrict__ counts, int64_t C,
                                                                     const int32_t *__restrict__ tileSums,
                                                                     int32_t *__restrict__ offsets, int32_t n)
        {
            ChainEntry();
            int32_t before = 0;
            for (int32_t t = static_cast<int32_t>(threadIdx.x); t < static_cast<int32_t>(blockIdx.x);
                 t += kScanThreads)
            {
                before += tileSums[t];
            }
            int32_t unused;
            const int32_t prefix = BlockExclusiveScan(before, unused);  // the block total
            const int64_t base = static_cast<int64_t>(blockIdx.x) * kScanTile + threadIdx.x * kScanItems;
            int32_t v[kScanItems];
            LoadThreadCells(counts, base, C, true, v);
            int32_t sum = 0;
#pragma unroll
            for (int q = 0; q < kScanItems; q++)
            {
                sum += v[q];
            }
            int32_t excl;
            BlockExclusiveScan(sum, excl);
            StoreThreadOffsets(offsets, base, C, prefix + excl, v);
            if (blockIdx.x == 0 && threadIdx.x == 0)
            {
                offsets[C] = n;
            }
        }

        // With tileSums it also clears the nTiles tile sums, which the scan has
        // used: the resident step's move adds to them.
        __global__ void Scatter(const int32_t *__restrict__ cellOf, const int32_t *__restrict__ arrival,
                                const int32_t *__restrict__ offsets, int32_t n, int32_t *__restrict__ bucketTmp,
                                int32_t *__restrict__ tileSums, int32_t nTiles)
        {
            ChainEntry();
            int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
            if (tileSums != nullptr)
            {
                for (int32_t t = i; t < nTiles; t += static_cast<int32_t>(gridDim.x * blockDim.x))
                {
                    tileSums[t] = 0;
                }
            }
            if (i >= n)
            {
                return;
            }
            bucketTmp[offsets[cellOf[i]] + arrival[i]] = i;
        }

        // The CPU scatters in agent-index order (CpuAgentForceBackend2D.cpp:
        // 100-109), so an agent's slot within its cell is the number of
        // lower-indexed agents in the same cell.
        template <typename TP, typename TR>
        __global__ void Stabilize(const int32_t *__restrict__ cellOf, const int32_t *__restrict__ offsets,
                                  const int32_t *__restrict__ bucketTmp, const V2<TP> *__restrict__ posF,
                                  const TR *__restrict__ rad, int32_t n, int32_t *__restrict__ bucket,
                                  V2<TP> *__restrict__ sPos, TR *__restrict__ sRad)
        {
            ChainEntry();
            // thread -> arrival-order slot q: its agent i, then i's stable
            // slot in the same cell (neighbouring threads share a cell's
            // offsets and bucket range, and their writes land near q)
            const int32_t q = blockIdx.x * blockDim.x + threadIdx.x;
            if (q >= n)
            {
                return;
            }
            const int32_t i = bucketTmp[q];
            const int32_t c = cellOf[i];
            const int32_t s = offsets[c];
            const int32_t e = offsets[c + 1];
            int32_t rank = 0;
            for (int32_t t = s; t < e; t++)
            {
                rank += (bucketTmp[t] < i) ? 1 : 0;
            }
            const int32_t slot = s + rank;
            bucket[slot] = i;
            sPos[slot] = posF[i];
            sRad[slot] = rad[i];
        }

        // Stable order within each cell (the CPU's scatter in agent index
        // order, CpuAgentForceBackend2D.cpp:100-109), one thread per
        // arrival-order slot q: its agent i, whose position gives its cell
        // again (no cell-array gather), goes to slot s + (number of
        // lower-indexed agents of the cell).  Neighbouring threads share a
        // cell's offsets and range of arrival-ordered indices, and the writes
        // land within the cell's own slots.
        template <typename TP, typename TR>
        __global__ void StabilizeSlots(const int32_t *__restrict__ offsets, const int32_t *__restrict__ bucketTmp,
                                       const V2<TP> *__restrict__ pos, const TR *__restrict__ rad, int32_t n,
                                       int32_t xDim, int32_t yDim, int32_t *__restrict__ bucket,
                                       V2<TP> *__restrict__ sPos, TR *__restrict__ sRad)
        {
            ChainEntry();
            const int32_t q = blockIdx.x * blockDim.x + threadIdx.x;
            if (q >= n)
            {
                return;
            }
            const int32_t i = bucketTmp[q];
            const V2<TP> p = pos[i];
            const TR r = rad[i];
            const int32_t c = CellCoord(p.x, xDim) * yDim + CellCoord(p.y, yDim);
            const int32_t s = offsets[c];
            const int32_t e = offsets[c + 1];
            int32_t rank = 0;
            for (int32_t t = s; t < e; t++)
            {
                rank += (bucketTmp[t] < i) ? 1 : 0;
            }
            const int32_t slot = s + rank;
            bucket[slot] = i;
            sPos[slot] = p;
            sRad[slot] = r;
        }

        // IEEE-exact FP64 helpers (no contraction) and their FP32 twins.
        __device__ __forceinline__ double Add(double a, double b) { return __dadd_rn(a, b); }
        __device__ __forceinline__ double Sub(double a, double b) { return __dsub_rn(a, b); }
        __device__ __forceinline__ double Mul(double a, double b) { return __dmul_rn(a, b); }
        __device__ __forceinline__ double Div(double a, double b) { return __ddiv_rn(a, b); }
        __device__ __forceinline__ double Sqrt(double a) { return __dsqrt_rn(a); }
        __device__ __forceinline__ float Add(float a, float b) { return __fadd_rn(a, b); }
        __device__ __forceinline__ float Sub(float a, float b) { return __fsub_rn(a, b); }
        __device__ __forceinline__ float Mul(float a, float b) { return __fmul_rn(a, b); }
        __device__ __forceinline__ double Abs(double a) { return fabs(a); }
        __device__ __forceinline__ float Abs(float a) { return fabsf(a); }

        // AgentForceDisp (CpuAgentForceBackend2D.cpp:30-45).
        template <typename T>
        __device__ __forceinline__ T Disp(T a, T b, T dimF, bool wrap)
        {
            T d = Sub(b, a);
            if (wrap && Abs(d) > Mul(dimF, T(0.5)))
            {
                d = (a > b) ? Add(d, dimF) : Sub(d, dimF);
            }
            return d;
        }

        // The agent grid's displacement GridGeometry2D::DispX/DispY
        // (src/Grids/GridGeometry2D.cpp:132-150) of p2 seen from p1: on a
        // wrapped axis DispWrap (src/MathUtil.cpp:363-379) shifts one end by
        // the axis length before subtracting, so it rounds differently from
        // AgentForceDisp.
        template <typename T>
        __device__ __forceinline__ T DispGrid(T p1, T p2, T dimF, bool wrap)
        {
            if (wrap && Abs(Sub(p1, p2)) > Mul(dimF, T(0.5)))
            {
                return (p1 > p2) ? Sub(Add(p2, dimF), p1) : Sub(p2, Add(p1, dimF));
            }
            return Sub(p2, p1);
        }

        // Overlap force laws: the overlapFun(touchDist, other) of
        // SphericalAgent2D::SumForces (include/Hal/Agents/SphericalAgent2D.h:
        // 74-102) as a law kind and its parameters.
        constexpr int kLawLinear = HAL_CUDA_FORCE_LINEAR;
        constexpr int kLawClamped = HAL_CUDA_FORCE_LINEAR_CLAMPED;
        constexpr int kLawPower = HAL_CUDA_FORCE_POWER;

        template <typename T>
        struct LawParams
        {
            T scale;
            T exponent;
        };

        __device__ __forceinline__ double Pow(double a, double b) { return pow(a, b); }
        __device__ __forceinline__ float Pow(float a, float b) { return powf(a, b); }

        template <int LAW, typename T>
        __device__ __forceinline__ T OverlapForce(T touch, const LawParams<T> &lp)
        {
            if constexpr (LAW == kLawLinear)
            {
                // springConstant * touchDist (CpuAgentForceBackend2D.cpp:165)
                return Mul(lp.scale, touch);
            }
            else if constexpr (LAW == kLawClamped)
            {
                // no force unless overlapping, then Hooke's law
                // (examples/OffLatticeExample.cpp:147-154)
                return (touch < T(0)) ? T(0) : Mul(lp.scale, touch);
            }
            else
            {
                // pow(scale * touchDist, exponent) (examples/Chemotaxis.cpp:128-130)
                return Pow(Mul(lp.scale, touch), lp.exponent);
            }
        }

        // The FP32 force of a pair at displacement (xComp, yComp): whether it
        // is within 0 < d < R, the force and its product with 1/d.  1/d comes
        // from rsqrt (d^2 = 0 gives NaN, which fails both tests like the CPU's
        // d > 0).
        template <int LAW>
        __device__ __forceinline__ bool PairScale32(float xComp, float yComp, float radSum, float R,
                                                    const LawParams<float> &lp, float &force, float &scale)
        {
            const float d2 = fmaf(xComp, xComp, __fmul_rn(yComp, yComp));
            const float inv = rsqrtf(d2);
            const float dist = __fmul_rn(d2, inv);
            force = 0.0f;
            scale = 0.0f;
            if (!((dist < R) && (dist > 0.0f)))
            {
                return false;
            }
            force = OverlapForce<LAW>(__fsub_rn(radSum, dist), lp);
            scale = __fmul_rn(inv, force);
            return true;
        }

        // The linear law's term without a branch, so that several candidates'
        // chains interleave: (x, y, scale) with v - (x, y) * scale the pair's
        // contribution, all 0 where the pair has none.  Subtracting such a
        // term adds -0, which leaves every v as it is.
        __device__ __forceinline__ bool PairTerm32(bool valid, float dx, float dy, float radSum, float R, float k,
                                                   float &x, float &y, float &scale)
        {
            const float d2 = fmaf(dx, dx, __fmul_rn(dy, dy));
            const float inv = rsqrtf(d2);
            const float dist = __fmul_rn(d2, inv);
            const float sc = __fmul_rn(inv, __fmul_rn(k, __fsub_rn(radSum, dist)));
            const bool near = valid && dist < R && dist > 0.0f;
            x = near ? dx : 0.0f;
            y = near ? dy : 0.0f;
            scale = near ? sc : 0.0f;
            return near;
        }

        // Windows of this many candidates are walked run by run (WalkRuns32).
        constexpr int32_t kLongWindow = 64;

        // One neighbour's contribution (CpuAgentForceBackend2D.cpp:153-169,
        // SphericalAgent2D.h:83-98): the displacement to pj, and for
        // 0 < d < R the force law's force along it, subtracted from (vx, vy);
        // with SUM a positive force is added to sum.
        template <typename T, int LAW, bool SUM, bool GRID>
        __device__ __forceinline__ void PairStep(T px, T py, T rad, V2<T> pj, T radj, T R, const LawParams<T> &lp,
                                                 T xDimF, T yDimF, int32_t wrapX, int32_t wrapY, T &vx, T &vy,
                                                 T &sum)
        {
            T xComp, yComp;
            if constexpr (GRID)
            {
                xComp = DispGrid(px, pj.x, xDimF, wrapX != 0);
                yComp = DispGrid(py, pj.y, yDimF, wrapY != 0);
            }
            else
            {
                xComp = Disp(px, pj.x, xDimF, wrapX != 0);
                yComp = Disp(py, pj.y, yDimF, wrapY != 0);
            }
            if constexpr (std::is_same<T, double>::value)
            {
                // IEEE operations in the CPU's order: bit-exact
                const T dist = Sqrt(Add(Mul(xComp, xComp), Mul(yComp, yComp)));
                if ((dist < R) && (dist > T(0)))
                {
                    const T touchDist = Sub(Add(rad, radj), dist);
                    const T force = OverlapForce<LAW>(touchDist, lp);
                    vx = Sub(vx, Mul(Div(xComp, dist), force));
                    vy = Sub(vy, Mul(Div(yComp, dist), force));
                    if constexpr (SUM)
                    {
                        if (force > T(0))
                        {
                            sum = Add(sum, Abs(force));
                        }
                    }
                }
            }
            else
            {
                T force, scale;
                if (PairScale32<LAW>(xComp, yComp, rad + radj, R, lp, force, scale))
                {
                    vx = fmaf(-xComp, scale, vx);
                    vy = fmaf(-yComp, scale, vy);
                    if constexpr (SUM)
                    {
                        if (force > T(0))
                        {
                            sum += force;
                        }
                    }
                }
            }
        }

        // One agent's force sum: its velocity after the neighbours' forces
        // (or the deltas, from zero) and the sum of its positive forces.
        template <typename T>
        struct ForceAcc
        {
            V2<T> v;
            T sum;
        };

        // The FP32 linear law over the slots of up to four runs [rs, re), one
        // after another in order, added to (vx, vy).  The terms of a group of
        // candidates are formed side by side, without branches, after the
        // loads of the whole group.  A long walk (a dense cluster, a pile at an
        // edge) is bound by its one thread's instructions and goes run by run,
        // without the choice of the run per candidate; a short one keeps the
        // runs joined, where groups cut short at each run's end would cost more.
        // Measured on GB300, 1M agents in 2048^2, 30% in a cluster, the force
        // pass, branches per pair / here: cluster inside 38 / 37 us, clipped at
        // an edge 66 / 51 us, at a corner 394 / 294 us (groups of eight in the
        // long walk were 5% slower there).
        __device__ __forceinline__ void WalkRuns32(const int32_t (&rs)[4], const int32_t (&re)[4], int32_t slot,
                                                   float2 pf, float rad, const float2 *__restrict__ sPos,
                                                   const float *__restrict__ sRad, float R, float k, float xDimF,
                                                   float yDimF, int32_t wrapX, int32_t wrapY, float &vx, float &vy)
        {
            const int32_t c1 = re[0] - rs[0];
            const int32_t c2 = c1 + (re[1] - rs[1]);
            const int32_t c3 = c2 + (re[2] - rs[2]);
            const int32_t total = c3 + (re[3] - rs[3]);
            constexpr int G = 4;
            auto add = [&](const int32_t(&q)[G], const float2(&pj)[G], const float(&rj)[G])
            {
                float x[G], y[G], sc[G];
#pragma unroll
                for (int u = 0; u < G; u++)
                {
                    PairTerm32(q[u] >= 0 && q[u] != slot, Disp(pf.x, pj[u].x, xDimF, wrapX != 0),
                               Disp(pf.y, pj[u].y, yDimF, wrapY != 0), __fadd_rn(rad, rj[u]), R, k, x[u], y[u], sc[u]);
                }
#pragma unroll
                for (int u = 0; u < G; u++)
                {
                    vx = fmaf(-x[u], sc[u], vx);
                    vy = fmaf(-y[u], sc[u], vy);
                }
            };
            if (total >= kLongWindow)
            {
#pragma unroll 1
                for (int r = 0; r < 4; r++)
                {
                    const int32_t q0 = r == 0 ? rs[0] : (r == 1 ? rs[1] : (r == 2 ? rs[2] : rs[3]));
                    const int32_t q1 = r == 0 ? re[0] : (r == 1 ? re[1] : (r == 2 ? re[2] : re[3]));
                    for (int32_t qb = q0; qb < q1; qb += G)
                    {
                        int32_t q[G];
                        float2 pj[G];
                        float rj[G];
#pragma unroll
                        for (int u = 0; u < G; u++)
                        {
                            const int32_t at = min(qb + u, q1 - 1);
                            q[u] = (qb + u < q1) ? at : -1;
                            pj[u] = sPos[at];
                            rj[u] = sRad[at];
                        }
                        add(q, pj, rj);
                    }
                }
                return;
            }
            for (int32_t k0 = 0; k0 < total; k0 += G)
            {
                int32_t q[G];
                float2 pj[G];
                float rj[G];
#pragma unroll
                for (int u = 0; u < G; u++)
                {
                    const int32_t at = k0 + u;
                    q[u] = (at >= total) ? -1
                           : (at < c1)   ? rs[0] + at
                           : (at < c2)   ? rs[1] + (at - c1)
                           : (at < c3)   ? rs[2] + (at - c2)
                                         : rs[3] + (at - c3);
                    pj[u] = pf;
                    rj[u] = rad;
                    if (q[u] >= 0)
                    {
                        pj[u] = sPos[q[u]];
                        rj[u] = sRad[q[u]];
                    }
                }
                add(q, pj, rj);
            }
        }

        // Pass 4 (CpuAgentForceBackend2D.cpp:112-175) for the agent in sorted
        // slot `slot`; offsets are the cell offsets of its grid.  Starting
        // from v0, each neighbour j within range subtracts (disp/d)*force,
        // force = LAW(touchDist); with SUM the positive forces are summed as
        // SumForces returns them.  GRID visits each cell's agents in
        // descending index order with the agent grid's displacement, which is
        // SphericalAgent2D::SumForces on an AgentGrid2D whose agents were
        // created in index order (each square's list is newest first,
        // AgentPT2D.h:200-241); otherwise the order is the CPU backend's
        // (ascending index within a cell).
        template <typename T, int LAW, bool SUM, bool GRID>
        __device__ __forceinline__ ForceAcc<T> ForceSlotLaw(const int32_t slot, const int32_t *__restrict__ offsets,
                                                            const V2<T> *__restrict__ sPos,
                                                            const T *__restrict__ sRad, double interactionRad, T R,
                                                            const LawParams<T> lp, int32_t xDim, int32_t yDim,
                                                            int32_t wrapX, int32_t wrapY, V2<T> v0)
        {
            const V2<T> pf = sPos[slot];
            const T px = pf.x;
            const T py = pf.y;
            const T rad = sRad[slot];
            // window bounds in FP64, as the CPU computes them
            int32_t xStart = static_cast<int32_t>(floor(static_cast<double>(pf.x) - interactionRad));
            int32_t xEnd = static_cast<int32_t>(ceil(static_cast<double>(pf.x) + interactionRad));
            int32_t yStart = static_cast<int32_t>(floor(static_cast<double>(pf.y) - interactionRad));
            int32_t yEnd = static_cast<int32_t>(ceil(static_cast<double>(pf.y) + interactionRad));
            // off-grid cells of a non-wrapped axis are skipped anyway
            if (!wrapX)
            {
                xStart = max(xStart, 0);
                xEnd = min(xEnd, xDim);
            }
            if (!wrapY)
            {
                yStart = max(yStart, 0);
                yEnd = min(yEnd, yDim);
            }
            const T xDimF = static_cast<T>(xDim);
            const T yDimF = static_cast<T>(yDim);
            T vx = v0.x, vy = v0.y;
            T sum = T(0);
            // one candidate slot q of the window, in the CPU's visiting order
            auto visit = [&](int32_t q) {
                if (q == slot)
                {
                    return;
                }
                PairStep<T, LAW, SUM, GRID>(px, py, rad, sPos[q], sRad[q], R, lp, xDimF, yDimF, wrapX, wrapY, vx,
                                            vy, sum);
            };
            auto result = [&]() {
                ForceAcc<T> acc;
                acc.v.x = vx;
                acc.v.y = vy;
                acc.sum = sum;
                return acc;
            };
            if constexpr (GRID)
            {
                // cell by cell, each cell's slots from last to first
                for (int32_t xSq = xStart; xSq < xEnd; xSq++)
                {
                    int32_t retX = xSq;
                    if (retX < 0 || retX >= xDim)
                    {
                        retX %= xDim;  // only reached on a wrapped axis (clamped otherwise)
                        retX = (retX < 0) ? retX + xDim : retX;
                    }
                    for (int32_t ySq = yStart; ySq < yEnd; ySq++)
                    {
                        int32_t retY = ySq;
                        if (retY < 0 || retY >= yDim)
                        {
                            retY %= yDim;
                            retY = (retY < 0) ? retY + yDim : retY;
                        }
                        const int32_t cell = retX * yDim + retY;
                        const int32_t s = __ldg(offsets + cell);
                        const int32_t e = __ldg(offsets + cell + 1);
                        for (int32_t q = e - 1; q >= s; q--)
                        {
                            visit(q);
                        }
                    }
                }
                return result();
            }
            // Common case: a window of at most four rows whose y-range does
            // not wrap, so each row is one run of cells.  All rows' offset
            // pairs are loaded before the first candidate, which shortens the
            // chain of dependent loads; the visiting order is unchanged.
            const int32_t nRows = xEnd - xStart;
            if (nRows > 0 && nRows <= 4 && yStart >= 0 && yEnd <= yDim && yEnd > yStart)
            {
                int32_t rs[4], re[4];
#pragma unroll
                for (int j = 0; j < 4; j++)
                {
                    rs[j] = 0;
                    re[j] = 0;
                    if (j < nRows)
                    {
                        int32_t retX = xStart + j;
                        if (retX < 0 || retX >= xDim)
                        {
                            retX %= xDim;  // only reached on a wrapped axis (clamped otherwise)
                            retX = (retX < 0) ? retX + xDim : retX;
                        }
                        const int32_t cell = retX * yDim + yStart;
                        rs[j] = __ldg(offsets + cell);
                        re[j] = __ldg(offsets + cell + (yEnd - yStart));
                    }
                }
                if constexpr (std::is_same<T, float>::value && LAW == kLawLinear && !SUM)
                {
                    WalkRuns32(rs, re, slot, pf, rad, sPos, sRad, R, lp.scale, xDimF, yDimF, wrapX, wrapY, vx, vy);
                    return result();
                }
                // The rows' runs, one after another, form one sequence of
                // candidates in the visiting order; it is walked in groups of
                // kGroup whose loads are issued before any of them is used, so
                // a thread waits for one round trip per group, not per
                // candidate.
                constexpr int kGroup = 4;
                const int32_t c1 = re[0] - rs[0];
                const int32_t c2 = c1 + (re[1] - rs[1]);
                const int32_t c3 = c2 + (re[2] - rs[2]);
                const int32_t total = c3 + (re[3] - rs[3]);
                for (int32_t k0 = 0; k0 < total; k0 += kGroup)
                {
                    int32_t qs[kGroup];
                    V2<T> pj[kGroup];
                    T rj[kGroup];
#pragma unroll
                    for (int u = 0; u < kGroup; u++)
                    {
                        const int32_t k = k0 + u;
                        qs[u] = (k >= total) ? -1
                                : (k < c1)   ? rs[0] + k
                                : (k < c2)   ? rs[1] + (k - c1)
                                : (k < c3)   ? rs[2] + (k - c2)
                                             : rs[3] + (k - c3);
                        if (qs[u] >= 0)
                        {
                            pj[u] = sPos[qs[u]];
                            rj[u] = sRad[qs[u]];
                        }
                    }
#pragma unroll
                    for (int u = 0; u < kGroup; u++)
                    {
                        if (qs[u] >= 0 && qs[u] != slot)
                        {
                            PairStep<T, LAW, SUM, GRID>(px, py, rad, pj[u], rj[u], R, lp, xDimF, yDimF, wrapX, wrapY,
                                                        vx, vy, sum);
                        }
                    }
                }
                return result();
            }
            for (int32_t xSq = xStart; xSq < xEnd; xSq++)
            {
                int32_t retX = xSq;
                const bool inX = (retX >= 0) && (retX < xDim);
                if (!inX)
                {
                    if (!wrapX)
                    {
                        continue;
                    }
                    retX %= xDim;
                    retX = (retX < 0) ? retX + xDim : retX;
                }
                // The cells (retX, ySq) for consecutive ySq are consecutive
                // cell indices, and their agents consecutive bucket slots, so
                // the row is walked as runs of cells that do not wrap: two
                // offset loads per run, the same visiting order as cell by
                // cell (the CPU's order).
                for (int32_t ySq = yStart; ySq < yEnd;)
                {
                    int32_t retY = ySq;
                    if (retY < 0 || retY >= yDim)
                    {
                        retY %= yDim;  // only reached on a wrapped axis (clamped otherwise)
                        retY = (retY < 0) ? retY + yDim : retY;
                    }
                    const int32_t run = min(yEnd - ySq, yDim - retY);
                    ySq += run;
                    const int32_t cell = retX * yDim + retY;
                    const int32_t s = __ldg(offsets + cell);
                    const int32_t e = __ldg(offsets + cell + run);
                    for (int32_t q = s; q < e; q++)
                    {
                        visit(q);
                    }
                }
            }
            return result();
        }

        // The CPU backend's pass 4: linear law, velocity deltas from zero.
        template <typename T>
        __device__ __forceinline__ V2<T> ForceSlot(const int32_t slot, const int32_t *__restrict__ offsets,
                                                   const V2<T> *__restrict__ sPos, const T *__restrict__ sRad,
                                                   double interactionRad, T R, T k, int32_t xDim, int32_t yDim,
                                                   int32_t wrapX, int32_t wrapY)
        {
            LawParams<T> lp;
            lp.scale = k;
            lp.exponent = T(1);
            return ForceSlotLaw<T, kLawLinear, false, false>(slot, offsets, sPos, sRad, interactionRad, R, lp, xDim,
                                                             yDim, wrapX, wrapY, Vec2<T>::Make(T(0), T(0)))
                .v;
        }

        template <typename TV, typename TVec>
        __device__ __forceinline__ void StoreDelta(TV *__restrict__ vel, int32_t i, TVec d)
        {
            vel[2 * static_cast<int64_t>(i)] = static_cast<TV>(d.x);
            vel[2 * static_cast<int64_t>(i) + 1] = static_cast<TV>(d.y);
        }

        // Pass 4 over cell-sorted slots: one thread per slot.  With velIn the
        // sum starts from the agent's velocity (SumForces adds to xVel/yVel),
        // otherwise from zero (the interface's velocity deltas); with SUM the
        // agent's sum of positive forces goes to sums.
        // WALLS: neither axis wraps (a compile-time 0 for both wrap flags, so
        // the displacement's wrap test leaves the per-candidate code).
        template <typename T, typename TV, int LAW = kLawLinear, bool SUM = false, bool GRID = false,
                  bool WALLS = false>
        __global__ void Forces(const int32_t *__restrict__ bucket, const int32_t *__restrict__ offsets,
                               const V2<T> *__restrict__ sPos, const T *__restrict__ sRad, int32_t n,
                               double interactionRad, T R, LawParams<T> lp, int32_t xDim, int32_t yDim,
                               int32_t wrapX, int32_t wrapY, TV *vel, T *__restrict__ sums, const TV *velIn)
        {
            ChainEntry();
            const int32_t slot = blockIdx.x * blockDim.x + threadIdx.x;
            if (slot >= n)
            {
                return;
            }
            const int32_t i = bucket[slot];
            V2<T> v0 = Vec2<T>::Make(T(0), T(0));
            if (velIn != nullptr)
            {
                v0 = Vec2<T>::Make(static_cast<T>(velIn[2 * static_cast<int64_t>(i)]),
                                   static_cast<T>(velIn[2 * static_cast<int64_t>(i) + 1]));
            }
            const ForceAcc<T> acc = ForceSlotLaw<T, LAW, SUM, GRID>(slot, offsets, sPos, sRad, interactionRad, R, lp,
                                                                    xDim, yDim, WALLS ? 0 : wrapX, WALLS ? 0 : wrapY,
                                                                    v0);
            StoreDelta(vel, i, acc.v);
            if constexpr (SUM)
            {
                sums[i] = acc.sum;
            }
        }

        // SphericalAgent2D's per-tick update after its forces
        // (include/Hal/Agents/SphericalAgent2D.h:133-162) in FP32, each IEEE
        // operation rounded to nearest with no contraction:
        //   vel += delta;  CapVelocity(maxVel) when maxVel >= 0;
        //   ForceMove: MoveSafePT(pos + vel) (AgentPT2D.h:157-186): a point
        //     on the grid is taken as is; otherwise each wrapped axis wraps
        //     (Wrap, src/MathUtil.cpp:48-53) and each closed axis whose new
        //     coordinate left [0, dim) keeps the old one;
        //   ApplyFriction(friction): vel *= friction.
        struct MoveParams
        {
            float friction;
            float maxVel;  // < 0: no cap
            float xDimF, yDimF;
            int32_t wrapX, wrapY;
        };

        __device__ __forceinline__ float WrapCoord(float v, float dim)
        {
            const float m = fmodf(v, dim);
            return (m < 0.0f) ? __fadd_rn(dim, m) : m;
        }

        __device__ __forceinline__ void MoveAgent(const MoveParams &mp, float2 &p, float2 &v)
        {
            if (mp.maxVel >= 0.0f)
            {
                const float maxVelSq = __fmul_rn(mp.maxVel, mp.maxVel);
                const float normSq = __fadd_rn(__fmul_rn(v.x, v.x), __fmul_rn(v.y, v.y));
                if (normSq > maxVelSq)
                {
                    const float conv = __fdiv_rn(mp.maxVel, __fsqrt_rn(normSq));
                    v.x = __fmul_rn(v.x, conv);
                    v.y = __fmul_rn(v.y, conv);
                }
            }
            float nx = __fadd_rn(p.x, v.x);
            float ny = __fadd_rn(p.y, v.y);
            const bool in = nx >= 0.0f && nx < mp.xDimF && ny >= 0.0f && ny < mp.yDimF;
            if (!in)
            {
                if (mp.wrapX)
                {
                    nx = WrapCoord(nx, mp.xDimF);
                }
                else if (!(nx >= 0.0f && nx < mp.xDimF))
                {
                    nx = p.x;
                }
                if (mp.wrapY)
                {
                    ny = WrapCoord(ny, mp.yDimF);
                }
                else if (!(ny >= 0.0f && ny < mp.yDimF))
                {
                    ny = p.y;
                }
            }
            p.x = nx;
            p.y = ny;
            v.x = __fmul_rn(v.x, mp.friction);
            v.y = __fmul_rn(v.y, mp.friction);
        }

        // Forces of the resident step with the move fused in: the slot's
        // agent adds its delta to its velocity and moves.  Positions are read
        // from the cell-sorted copy, so writing the agent-order positions
        // here races with no other thread.  With counts set, the moved agent
        // is also counted into its new cell, BinCount's work for the next
        // tick (cell, arrival rank): this tick's scan cleared the counts, and
        // its scatter has read the previous cells and ranks.
        template <int LAW = kLawLinear, bool SUM = false, bool WALLS = false>
        __global__ void ForcesMove(const int32_t *__restrict__ bucket, const int32_t *__restrict__ offsets,
                                   const float2 *__restrict__ sPos, const float *__restrict__ sRad, int32_t n,
                                   double interactionRad, float R, LawParams<float> lp, int32_t xDim, int32_t yDim,
                                   MoveParams mp, float *__restrict__ deltas, float2 *__restrict__ pos,
                                   float2 *__restrict__ velocity, float *__restrict__ sums,
                                   int32_t *__restrict__ cellOf, int32_t *__restrict__ arrival,
                                   int32_t *__restrict__ counts, int32_t *__restrict__ tileSums)
        {
            ChainEntry();
            const int32_t slot = blockIdx.x * blockDim.x + threadIdx.x;
            if (slot >= n)
            {
                return;
            }
            const int32_t i = bucket[slot];
            // in flight during the sums (200k agents 34 -> 25 us per step, 400k 50 ->
            // 45, 1M 91 -> 89)
            float2 v = velocity[i];
            const ForceAcc<float> acc = ForceSlotLaw<float, LAW, SUM, false>(
                slot, offsets, sPos, sRad, interactionRad, R, lp, xDim, yDim, WALLS ? 0 : mp.wrapX,
                WALLS ? 0 : mp.wrapY, make_float2(0.f, 0.f));
            const V2<float> d = acc.v;
            StoreDelta(deltas, i, d);
            if constexpr (SUM)
            {
                sums[i] = acc.sum;
            }
            float2 p = sPos[slot];
            v.x = __fadd_rn(v.x, d.x);
            v.y = __fadd_rn(v.y, d.y);
            MoveAgent(mp, p, v);
            pos[i] = p;
            velocity[i] = v;
            if (counts != nullptr)
            {
                const int32_t c = CellCoord(p.x, xDim) * yDim + CellCoord(p.y, yDim);
                cellOf[i] = c;
                arrival[i] = atomicAdd(counts + c, 1);
                AddToTiles(tileSums, c);
            }
        }


        // ---- few agents: eight lanes per agent ------------------------------
        // With one thread per agent, 20000 agents are a warp per scheduler, and
        // the tick waits for the longest chain: the agents of a dense cluster
        // walk their window's candidates (60 and more) one after another, 13 of
        // the step's 24 us.  Here a group of kGroupLanes lanes takes an agent:
        // each lane finds one run of the window's cells, the lanes evaluate
        // that many candidates at a time, and the terms are then added in the
        // candidates' order by every lane (a candidate out of range adds -0),
        // so the sum is ForceSlotLaw's, bit for bit.  A window of more runs
        // takes several rounds (a radius of 4 has nine rows, a radius of 2 at a
        // wrapped edge five of two runs; us per step with such windows left to
        // one lane's walk / in rounds: 20k agents in 256^2, radius 4, 161 / 48
        // with a cluster, 37 / 19 uniform; 90k in 512^2, wrapped, 110 / 43).  It
        // issues more instructions per pair than one thread per agent does:
        // GroupPerAgent says where it pays.  Leaving only the agents of long
        // windows to groups, in a second launch, cost 3 us per 1M-agent step and
        // lost up to 2x where many agents had long windows.
        constexpr int kGroupLanes = 8;

        // floor(v - r) and ceil(v + r) as the CPU takes them, in FP64.  For an
        // integer r the FP32 floor and ceiling give the same (v is exact, and
        // the FP64 sum exact, for the magnitudes below; nearer zero the sum can
        // round onto an integer) without FP64 instructions on the chain.
        __device__ __forceinline__ void WindowOf(float v, double r, bool intR, int32_t &lo, int32_t &hi)
        {
            const float a = fabsf(v);
            if (intR && (a == 0.0f || (a >= 0x1p-28f && a < 0x1p24f)))
            {
                const int32_t ri = static_cast<int32_t>(static_cast<float>(r));
                lo = static_cast<int32_t>(floorf(v)) - ri;
                hi = static_cast<int32_t>(ceilf(v)) + ri;
            }
            else
            {
                lo = static_cast<int32_t>(floor(static_cast<double>(v) - r));
                hi = static_cast<int32_t>(ceil(static_cast<double>(v) + r));
            }
        }

        // The force sum (linear law, from zero) of the agent in slot `slot`
        // (live: there is one), on every lane of its group.  All lanes of the
        // warp call it.
        __device__ __forceinline__ float2 ForceSlotGroup(const int32_t slot, const bool live,
                                                         const int32_t *__restrict__ offsets,
                                                         const float2 *__restrict__ sPos,
                                                         const float *__restrict__ sRad, double interactionRad,
                                                         bool intR, float R, const LawParams<float> lp, int32_t xDim,
                                                         int32_t yDim, int32_t wrapX, int32_t wrapY)
        {
            constexpr int G = kGroupLanes;
            const int j = threadIdx.x & (G - 1);
            const float2 pf = sPos[slot];
            const float rad = sRad[slot];
            int32_t xStart, xEnd, yStart, yEnd;
            WindowOf(pf.x, interactionRad, intR, xStart, xEnd);
            WindowOf(pf.y, interactionRad, intR, yStart, yEnd);
            if (!wrapX)
            {
                xStart = max(xStart, 0);
                xEnd = min(xEnd, xDim);
            }
            if (!wrapY)
            {
                yStart = max(yStart, 0);
                yEnd = min(yEnd, yDim);
            }
            // the window as runs of cells, in the visiting order, eight a round, a
            // lane's each
            WindowRuns win;
            win.Set(xStart, xEnd, yStart, yEnd, yDim);
            const int32_t runs = (live && win.fits) ? win.runs : 0;
            const float xDimF = static_cast<float>(xDim), yDimF = static_cast<float>(yDim);
            float vx = 0.0f, vy = 0.0f;
            auto rounds = [&](auto xTag, auto yTag)
            {
                constexpr bool WX = decltype(xTag)::value, WY = decltype(yTag)::value;
                int32_t r0 = 0;
                do
                {
                    int32_t s0 = 0, len = 0;
                    if (r0 + j < runs)
                    {
                        int32_t cell, count;
                        win.Run(r0 + j, xStart, xDim, yDim, cell, count);
                        s0 = __ldg(offsets + cell);
                        len = __ldg(offsets + cell + count) - s0;
                    }
                    // candidate k is slot k + shift[r] of the first run r with k < end[r]
                    int32_t end[G], shift[G];
                    int32_t total = 0;
#pragma unroll
                    for (int r = 0; r < G; r++)
                    {
                        shift[r] = __shfl_sync(0xffffffffu, s0, r, G) - total;
                        total += __shfl_sync(0xffffffffu, len, r, G);
                        end[r] = total;
                    }
                    const int32_t most = __reduce_max_sync(0xffffffffu, total);
                    auto candidate = [&](int32_t k, int32_t &q, float2 &pj, float &rj)
                    {
                        q = -1;
                        if (k < total)
                        {
                            int32_t sh = shift[G - 1];
#pragma unroll
                            for (int r = G - 2; r >= 0; r--)
                            {
                                sh = (k < end[r]) ? shift[r] : sh;
                            }
                            q = k + sh;
                            pj = sPos[q];
                            rj = sRad[q];
                        }
                    };
                    int32_t q;
                    float2 pj = make_float2(0.0f, 0.0f);
                    float rj = 0.0f;
                    candidate(j, q, pj, rj);
#pragma unroll 2
                    for (int32_t k0 = 0; k0 < most; k0 += G)
                    {
                        // the next round's loads, in flight during this one's sums
                        int32_t qn;
                        float2 pn = make_float2(0.0f, 0.0f);
                        float rn = 0.0f;
                        candidate(k0 + G + j, qn, pn, rn);
                        float x, y, scale;
                        const bool near = PairTerm32(
                            q >= 0 && q != slot, Disp(pf.x, pj.x, xDimF, WX), Disp(pf.y, pj.y, yDimF, WY),
                            __fadd_rn(rad, rj), R, lp.scale, x, y, scale);
                        // the terms, in the candidates' order, on every lane (walking
                        // only the ones in range took more instructions than it saved)
                        if (__any_sync(0xffffffffu, near))
                        {
#pragma unroll
                            for (int t = 0; t < G; t++)
                            {
                                const float sc = __shfl_sync(0xffffffffu, scale, t, G);
                                vx = fmaf(-__shfl_sync(0xffffffffu, x, t, G), sc, vx);
                                vy = fmaf(-__shfl_sync(0xffffffffu, y, t, G), sc, vy);
                            }
                        }
                        q = qn;
                        pj = pn;
                        rj = rn;
                    }
                    r0 += G;
                } while (__any_sync(0xffffffffu, r0 < runs));
            };
            // A window clear of the edge cells holds only agents that lie in its
            // cells (an edge cell also holds those outside the grid), less than
            // half a side away: no displacement wraps.  (The loop's form matters
            // where windows are long: 50k agents in 256^2, wrapped, 30% in a
            // cluster, us per step with the wrap's test on every candidate 216,
            // without 190, and two candidates a trip 163; 20k 37, 34, 31.)
            const bool clear = xStart > 0 && xEnd < xDim && yStart > 0 && yEnd < yDim && xEnd - xStart < xDim / 2 &&
                               yEnd - yStart < yDim / 2;
            const bool flat = __all_sync(0xffffffffu, clear);
            const std::true_type yes;
            const std::false_type no;
            if (flat || !(wrapX || wrapY))
            {
                rounds(no, no);
            }
            else if (wrapX && wrapY)
            {
                rounds(yes, yes);
            }
            else if (wrapX)
            {
                rounds(yes, no);
            }
            else
            {
                rounds(no, yes);
            }
            if (!win.fits && live)
            {
                // a y-range longer than the side: one lane's walk for all
                const ForceAcc<float> acc = ForceSlotLaw<float, kLawLinear, false, false>(
                    slot, offsets, sPos, sRad, interactionRad, R, lp, xDim, yDim, wrapX, wrapY,
                    make_float2(0.0f, 0.0f));
                vx = acc.v.x;
                vy = acc.v.y;
            }
            return make_float2(vx, vy);
        }

        // Forces and ForcesMove (linear law, no sums) with a group per agent.
        template <bool WALLS>
        __global__ void ForcesGroup(const int32_t *__restrict__ bucket, const int32_t *__restrict__ offsets,
                                    const float2 *__restrict__ sPos, const float *__restrict__ sRad, int32_t n,
                                    double interactionRad, bool intR, float R, LawParams<float> lp, int32_t xDim,
                                    int32_t yDim, int32_t wrapX, int32_t wrapY, float *__restrict__ vel)
        {
            ChainEntry();
            const int32_t at = (blockIdx.x * blockDim.x + threadIdx.x) / kGroupLanes;
            const bool live = at < n;
            const int32_t slot = live ? at : n - 1;
            const float2 d = ForceSlotGroup(slot, live, offsets, sPos, sRad, interactionRad, intR, R, lp, xDim, yDim,
                                            WALLS ? 0 : wrapX, WALLS ? 0 : wrapY);
            if (live && (threadIdx.x & (kGroupLanes - 1)) == 0)
            {
                StoreDelta(vel, bucket[slot], d);
            }
        }

        // One agent's forces and move, by its group.
        template <bool WALLS>
        __device__ __forceinline__ void MoveSlotGroup(const int32_t slot, const bool live,
                                                      const int32_t *__restrict__ bucket,
                                                      const int32_t *__restrict__ offsets,
                                                      const float2 *__restrict__ sPos, const float *__restrict__ sRad,
                                                      double interactionRad, bool intR, float R, LawParams<float> lp,
                                                      int32_t xDim, int32_t yDim, const MoveParams &mp,
                                                      float *__restrict__ deltas, float2 *__restrict__ pos,
                                                      float2 *__restrict__ velocity, int32_t *__restrict__ cellOf,
                                                      int32_t *__restrict__ arrival, int32_t *__restrict__ counts,
                                                      int32_t *__restrict__ tileSums)
        {
            const bool lead = live && (threadIdx.x & (kGroupLanes - 1)) == 0;
            // the move's inputs, in flight during the sums
            const int32_t i = bucket[slot];
            float2 v = lead ? velocity[i] : make_float2(0.0f, 0.0f);
            const float2 d = ForceSlotGroup(slot, live, offsets, sPos, sRad, interactionRad, intR, R, lp, xDim, yDim,
                                            WALLS ? 0 : mp.wrapX, WALLS ? 0 : mp.wrapY);
            if (!lead)
            {
                return;
            }
            StoreDelta(deltas, i, d);
            float2 p = sPos[slot];
            v.x = __fadd_rn(v.x, d.x);
            v.y = __fadd_rn(v.y, d.y);
            MoveAgent(mp, p, v);
            pos[i] = p;
            velocity[i] = v;
            const int32_t c = CellCoord(p.x, xDim) * yDim + CellCoord(p.y, yDim);
            cellOf[i] = c;
            arrival[i] = atomicAdd(counts + c, 1);
            AddToTiles(tileSums, c);
        }

        template <bool WALLS>
        __global__ void ForcesMoveGroup(const int32_t *__restrict__ bucket, const int32_t *__restrict__ offsets,
                                        const float2 *__restrict__ sPos, const float *__restrict__ sRad, int32_t n,
                                        double interactionRad, bool intR, float R, LawParams<float> lp, int32_t xDim,
                                        int32_t yDim, MoveParams mp, float *__restrict__ deltas,
                                        float2 *__restrict__ pos, float2 *__restrict__ velocity,
                                        int32_t *__restrict__ cellOf, int32_t *__restrict__ arrival,
                                        int32_t *__restrict__ counts, int32_t *__restrict__ tileSums)
        {
            ChainEntry();
            const int32_t at = (blockIdx.x * blockDim.x + threadIdx.x) / kGroupLanes;
            const bool live = at < n;
            const int32_t slot = live ? at : n - 1;
            MoveSlotGroup<WALLS>(slot, live, bucket, offsets, sPos, sRad, interactionRad, intR, R, lp, xDim, yDim, mp,
                                 deltas, pos, velocity, cellOf, arrival, counts, tileSums);
        }

        // ---- FP64 forces: a group of lanes per agent, only near pairs in FP64 --
        // The FP64 pipe bounds the interface's FP64 sums (a warp's FP64
        // instruction holds its pipe for 64 cycles, about 35 of them per pair
        // with the square root and the divisions), and a thread per agent gives
        // a dense cluster's long walks to a few warps.  Here eight lanes take an
        // agent's candidates; each first compares an FP32 distance, made from
        // the positions' bits without FP64 instructions and with its error
        // bound on the safe side, and only the pairs that may be in range are
        // queued.  Full queues of pairs then go through the FP64 operations, one
        // pair per lane, and the terms are subtracted in the visiting order: the
        // same operations on the same values as a thread's walk, bit for bit.
        // A group takes up to four agents, one after another, once there are
        // enough of them, so that a sparse grid's few pairs still fill the lanes.
        // A CTA is one warp: the agents' walks differ much, and small CTAs spread
        // them (20k in 256^2 at R = 2: CTAs of 128 threads 215, of 32 180 us).
        // Measured on GB300, the interface's FP64 call, thread per agent / here
        // (us): 50k agents in 256^2, 30% in a cluster, 380 / 157 (the kernel 298
        // / 86), the cluster clipped at a corner, with 2586 agents in one cell,
        // 8360 / 1480; 5k in 100 x 77 207 / 67; 200k in 1024^2 453 / 283 with a
        // cluster, 253 / 211 uniform; 20k in 256^2 at R = 2 632 / 180.  One agent
        // a group throughout: 200k uniform 288; up to eight from 20k on: 50k 198,
        // 200k with a cluster 359.  Two agents a group already from kPairSparse on
        // where a window holds fewer than two of a uniform population: 50k uniform
        // in 512^2, wrapped, 111 with a thread per agent, 120 with one agent a
        // group, 106 with two (a cluster clipped at a corner 348 / 161 / 169).
        constexpr int kPairQueue = 32;  // pairs an agent's queue holds (a power of two)
        constexpr int kPairDrain = 16;  // a queue this long is worked off
        constexpr int kPairThreads = 32;
        constexpr int32_t kPairGroups = 152 * 256;  // groups that fill the chip
        constexpr int32_t kPairPerGroup = 4;        // agents a group takes, one after another, at most
        constexpr int32_t kPairSparse = 40000;

        // The FP32 value nearest towards zero of v, by its bits: zero below the
        // normal range, NaN for what FP32 cannot hold (and for NaN itself).
        __device__ __forceinline__ float Truncated(double v)
        {
            const int32_t hi = __double2hiint(v);
            const uint32_t lo = static_cast<uint32_t>(__double2loint(v));
            const uint32_t mag = static_cast<uint32_t>(hi) & 0x7fffffffu;
            uint32_t f = __funnelshift_l(lo, mag - 0x38000000u, 3);
            f = (mag < 0x38100000u) ? 0u : f;
            f = (mag >= 0x47f00000u) ? 0x7fffffffu : f;
            return __uint_as_float(f | (static_cast<uint32_t>(hi) & 0x80000000u));
        }

        template <bool WALLS>
        __global__ void __launch_bounds__(kPairThreads)
            ForcesGroup64(const int32_t *__restrict__ bucket, const int32_t *__restrict__ offsets,
                          const double2 *__restrict__ sPos, const double *__restrict__ sRad, int32_t n,
                          int32_t perGroup, double interactionRad, LawParams<double> lp, int32_t xDim, int32_t yDim,
                          int32_t wrapX, int32_t wrapY, double *vel, const double *velIn)
        {
            constexpr int G = kGroupLanes;
            __shared__ int2 queue[kPairThreads / G][kPairQueue];  // (agent's slot, neighbour's slot)
            __shared__ double2 terms[kPairThreads / G][G];
            __shared__ int32_t owner[kPairThreads / G][G];
            ChainEntry();
            const int j = threadIdx.x & (G - 1);
            const int group = threadIdx.x / G;
            const int64_t first = (static_cast<int64_t>(blockIdx.x) * kPairThreads + threadIdx.x) / G * perGroup;
            const bool odd = (j & 1) != 0;
            if (WALLS)
            {
                wrapX = wrapY = 0;
            }
            const float xDimF = static_cast<float>(xDim), yDimF = static_cast<float>(yDim);
            const double xDimD = xDim, yDimD = yDim;
            const float rF = __double2float_ru(interactionRad);
            const uint64_t rBits = static_cast<uint64_t>(__double_as_longlong(interactionRad));
            int32_t head = 0, tail = 0;  // the queue's pairs [head, tail), modulo its size
            int32_t cur = -1;            // the agent whose sum v holds (its slot)
            double v = 0.0;              // even lanes: the x sum, odd lanes: the y sum
            auto start = [&](int32_t slot) {
                return velIn == nullptr ? 0.0 : velIn[2 * static_cast<int64_t>(bucket[slot]) + (odd ? 1 : 0)];
            };
            auto store = [&](int32_t slot, double sum) {
                if (j < 2)
                {
                    vel[2 * static_cast<int64_t>(bucket[slot]) + j] = sum;
                }
            };

            // up to eight queued pairs, in order
            auto drain = [&]() {
                __syncwarp();
                const bool valid = j < tail - head;
                const int2 pair = valid ? queue[group][(head + j) & (kPairQueue - 1)] : make_int2(-1, -1);
                head += min(tail - head, G);
                double2 t = make_double2(0.0, 0.0);
                if (valid)
                {
                    const double2 p = sPos[pair.x];
                    const double2 pj = sPos[pair.y];
                    const double radSum = Add(sRad[pair.x], sRad[pair.y]);
                    const double x = Disp(p.x, pj.x, xDimD, wrapX != 0);
                    const double y = Disp(p.y, pj.y, yDimD, wrapY != 0);
                    const double dist = Sqrt(Add(Mul(x, x), Mul(y, y)));
                    // 0 < dist < R by the bits of non-negative values (NaN's are larger)
                    const uint64_t dBits = static_cast<uint64_t>(__double_as_longlong(dist));
                    if (dBits != 0 && dBits < rBits)
                    {
                        const double force = OverlapForce<kLawLinear>(Sub(radSum, dist), lp);
                        t.x = Mul(Div(x, dist), force);
                        t.y = Mul(Div(y, dist), force);
                    }
                }
                terms[group][j] = t;
                owner[group][j] = pair.x;
                __syncwarp();
#pragma unroll
                for (int u = 0; u < G; u++)
                {
                    const int32_t o = owner[group][u];
                    if (o >= 0 && o != cur)
                    {
                        if (cur >= 0)
                        {
                            store(cur, v);
                        }
                        cur = o;
                        v = start(o);
                    }
                    // (subtracting the zero of a pair out of range changes nothing)
                    v = Sub(v, reinterpret_cast<const double *>(&terms[group][u])[odd ? 1 : 0]);
                }
                __syncwarp();
            };

            for (int32_t a = 0; a < perGroup; a++)
            {
                const bool live = first + a < n;
                const int32_t slot = live ? static_cast<int32_t>(first + a) : n - 1;
                const double2 p = sPos[slot];
                const int32_t before = tail;
                // window bounds in FP64, as the CPU computes them, one per lane:
                // floor(x - R), ceil(x + R), floor(y - R), ceil(y + R)
                int32_t bound;
                {
                    const double c = (j & 2) ? p.y : p.x;
                    const double b = __dadd_rn(c, odd ? interactionRad : -interactionRad);
                    bound = static_cast<int32_t>(odd ? ceil(b) : floor(b));
                }
                int32_t xStart = __shfl_sync(0xffffffffu, bound, 0, G), xEnd = __shfl_sync(0xffffffffu, bound, 1, G);
                int32_t yStart = __shfl_sync(0xffffffffu, bound, 2, G), yEnd = __shfl_sync(0xffffffffu, bound, 3, G);
                if (!wrapX)
                {
                    xStart = max(xStart, 0);
                    xEnd = min(xEnd, xDim);
                }
                if (!wrapY)
                {
                    yStart = max(yStart, 0);
                    yEnd = min(yEnd, yDim);
                }
                const float pxF = Truncated(p.x), pyF = Truncated(p.y);
                // |error| of an FP32 distance: per axis the coordinates'
                // truncation (2^-23 of each), the difference's and the wrap's
                // roundings (2^-24 of |a| + |b| and of |a| + |b| + dim), twice
                // that where only one precision wraps: below
                // 4.8e-7 (|a| + |b| + dim)
                const float own = 6e-7f * (fabsf(pxF) + fabsf(pyF) + xDimF + yDimF) + 1e-30f;

                // The window as runs of cells, in the visiting order: a round
                // takes up to eight runs (one per row, two where a wrapped
                // y-range crosses the edge; the y-range may wrap more than once).
                const bool some = live && xEnd > xStart && yEnd > yStart;
                int32_t row = xStart, yAt = yStart;  // the next run
                while (__any_sync(0xffffffffu, some && row < xEnd))
                {
                    int32_t s0 = 0, len = 0;
#pragma unroll 1
                    for (int r = 0; r < G && some && row < xEnd; r++)
                    {
                        int32_t retX = row;
                        if (retX < 0 || retX >= xDim)
                        {
                            retX %= xDim;  // only reached on a wrapped axis (clamped otherwise)
                            retX = (retX < 0) ? retX + xDim : retX;
                        }
                        int32_t retY = yAt;
                        if (retY < 0 || retY >= yDim)
                        {
                            retY %= yDim;
                            retY = (retY < 0) ? retY + yDim : retY;
                        }
                        const int32_t run = min(yEnd - yAt, yDim - retY);
                        if (r == j)
                        {
                            const int32_t cell = retX * yDim + retY;
                            s0 = __ldg(offsets + cell);
                            len = __ldg(offsets + cell + run) - s0;
                        }
                        yAt += run;
                        if (yAt >= yEnd)
                        {
                            yAt = yStart;
                            row++;
                        }
                    }
                    __syncwarp();
                    // candidate k is slot k + shift[r] of the first run r with k < end[r]
                    int32_t end[G], shift[G];
                    int32_t total = 0;
#pragma unroll
                    for (int r = 0; r < G; r++)
                    {
                        shift[r] = __shfl_sync(0xffffffffu, s0, r, G) - total;
                        total += __shfl_sync(0xffffffffu, len, r, G);
                        end[r] = total;
                    }
                    const int32_t most = __reduce_max_sync(0xffffffffu, total);
                    for (int32_t k0 = 0; k0 < most; k0 += G)
                    {
                        const int32_t k = k0 + j;
                        int32_t q = shift[G - 1];
#pragma unroll
                        for (int r = G - 2; r >= 0; r--)
                        {
                            q = (k < end[r]) ? shift[r] : q;
                        }
                        q += k;
                        // the pairs that may be in range join the queue, in the lanes' order
                        bool pass = false;
                        if (k < total && q != slot)
                        {
                            const double2 pj = sPos[q];
                            const float qx = Truncated(pj.x), qy = Truncated(pj.y);
                            const float x = Disp(pxF, qx, xDimF, wrapX != 0);
                            const float y = Disp(pyF, qy, yDimF, wrapY != 0);
                            const float reach = rF + (own + 6e-7f * (fabsf(qx) + fabsf(qy)));
                            // not greater: a NaN passes to the FP64 test; agents on
                            // one spot (a pile at a clipped edge) are no pair
                            const bool same = __double_as_longlong(pj.x) == __double_as_longlong(p.x) &&
                                              __double_as_longlong(pj.y) == __double_as_longlong(p.y);
                            pass = !same && !(x * x + y * y > reach * reach * 1.00001f);
                        }
                        const uint32_t mine =
                            (__ballot_sync(0xffffffffu, pass) >> (threadIdx.x & 24)) & ((1u << G) - 1u);
                        if (pass)
                        {
                            queue[group][(tail + __popc(mine & ((1u << j) - 1u))) & (kPairQueue - 1)] =
                                make_int2(slot, q);
                        }
                        tail += __popc(mine);
                        while (__any_sync(0xffffffffu, tail - head >= kPairDrain))
                        {
                            drain();
                        }
                    }
                }
                if (live && tail == before)
                {
                    store(slot, start(slot));  // no neighbour near
                }
            }
            while (__any_sync(0xffffffffu, tail > head))
            {
                drain();
            }
            if (cur >= 0)
            {
                store(cur, v);
            }
        }

        // ---- many independent wells in one pass ------------------------------
        // Agents of all wells are concatenated, and so are the cells of the
        // wells that have agents (well w's cells start at cellBase); the
        // count, scan, scatter and stable-rank passes then run unchanged over
        // the concatenation, and each agent's window walks its own well.  With
        // motion the move counts the agents for the next pass, as the resident
        // step does, and the pass starts at the scan: 427k agents in 48 wells,
        // 71.5 -> 65.0 us per pass.

        __device__ __forceinline__ int32_t WellBin(const AgentWellDev &wd, float px, float py)
        {
            return static_cast<int32_t>(wd.binBase) + (CellCoord(px, wd.xDim) >> wd.binShift) * wd.binsY +
                   (CellCoord(py, wd.yDim) >> wd.binShift);
        }

        __global__ void BinCountWells(const float *__restrict__ pos, const int32_t *__restrict__ wellOf,
                                      const AgentWellDev *__restrict__ wells, int32_t n,
                                      int32_t *__restrict__ binOf, int32_t *__restrict__ arrival,
                                      int32_t *__restrict__ counts)
        {
            ChainEntry();
            const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
            if (i >= n)
            {
                return;
            }
            const AgentWellDev wd = wells[wellOf[i]];
            const float px = pos[2 * static_cast<int64_t>(i)];
            const float py = pos[2 * static_cast<int64_t>(i) + 1];
            const int32_t b = WellBin(wd, px, py);
            binOf[i] = b;
            arrival[i] = atomicAdd(counts + b, 1);
        }

        // The order within a coarse bin: by cell, then by agent index (the
        // per-cell binning's order for each cell).  The agent at
        // arrival-order slot q counts the agents of its bin before it.
        __global__ void StabilizeWells(const int32_t *__restrict__ offsets, const int32_t *__restrict__ bucketTmp,
                                       const float2 *__restrict__ posF, const float *__restrict__ rad,
                                       const int32_t *__restrict__ wellOf, const AgentWellDev *__restrict__ wells,
                                       int32_t n, int32_t *__restrict__ bucket, float2 *__restrict__ sPos,
                                       float *__restrict__ sRad, int32_t *__restrict__ sCell)
        {
            ChainEntry();
            const int32_t q = blockIdx.x * blockDim.x + threadIdx.x;
            if (q >= n)
            {
                return;
            }
            const int32_t i = bucketTmp[q];
            const AgentWellDev wd = wells[wellOf[q]];  // the slots go well by well, as the agents do
            const float2 p = posF[i];
            const float r = rad[i];
            const int32_t c = CellCoord(p.x, wd.xDim) * wd.yDim + CellCoord(p.y, wd.yDim);
            const int32_t b = WellBin(wd, p.x, p.y);
            const int32_t s = offsets[b];
            const int32_t e = offsets[b + 1];
            int32_t rank = 0;
            for (int32_t t = s; t < e; t++)
            {
                const int32_t j = bucketTmp[t];
                int32_t cj = c;  // one cell per bin: the bin's agents share it
                if (wd.binShift != 0)
                {
                    const float2 pj = posF[j];
                    cj = CellCoord(pj.x, wd.xDim) * wd.yDim + CellCoord(pj.y, wd.yDim);
                }
                rank += (cj < c || (cj == c && j < i)) ? 1 : 0;
            }
            const int32_t slot = s + rank;
            bucket[slot] = i;
            sPos[slot] = p;
            sRad[slot] = r;
            sCell[slot] = c;
        }

        // Pass 4 of one well's agent over the coarse bins: the window's cells
        // x-major then y, each cell's agents (a run of its bin, in index
        // order), so the visiting order and the sum are those of ForceSlot
        // on the well's own per-cell bins.
        __device__ __forceinline__ V2<float> ForceSlotWell(const int32_t slot, const int32_t *__restrict__ offsets,
                                                           const float2 *__restrict__ sPos,
                                                           const float *__restrict__ sRad,
                                                           const int32_t *__restrict__ sCell, double interactionRad,
                                                           bool intR, float R, float k, const AgentWellDev &wd)
        {
            const float2 pf = sPos[slot];
            const float rad = sRad[slot];
            const int32_t xDim = wd.xDim, yDim = wd.yDim;
            int32_t xStart, xEnd, yStart, yEnd;
            WindowOf(pf.x, interactionRad, intR, xStart, xEnd);
            WindowOf(pf.y, interactionRad, intR, yStart, yEnd);
            if (!wd.wrapX)
            {
                xStart = max(xStart, 0);
                xEnd = min(xEnd, xDim);
            }
            if (!wd.wrapY)
            {
                yStart = max(yStart, 0);
                yEnd = min(yEnd, yDim);
            }
            LawParams<float> lp;
            lp.scale = k;
            lp.exponent = 1.0f;
            const float xDimF = static_cast<float>(xDim);
            const float yDimF = static_cast<float>(yDim);
            float vx = 0.0f, vy = 0.0f, sum = 0.0f;
            const int32_t sh = wd.binShift;
            const int32_t nRows = xEnd - xStart;
            if (sh == 0 && nRows > 0 && nRows <= 4 && yStart >= 0 && yEnd <= yDim && yEnd > yStart)
            {
                // One cell per bin and a window whose y-range does not wrap:
                // each window row is one run of consecutive bins, so one
                // stretch of slots.  All rows' bounds are loaded before the
                // first candidate (WalkRuns32).  The visiting order is unchanged.
                // (Walking the coarser bins' stretches the same way, with a
                // filter for the other cells' agents, took as long as the walk
                // below: fewer chained loads, more candidates.)
                int32_t rs[4], re[4];
#pragma unroll
                for (int j = 0; j < 4; j++)
                {
                    rs[j] = 0;
                    re[j] = 0;
                    if (j < nRows)
                    {
                        int32_t retX = xStart + j;
                        if (retX < 0 || retX >= xDim)
                        {
                            retX %= xDim;  // only reached on a wrapped axis (clamped otherwise)
                            retX = (retX < 0) ? retX + xDim : retX;
                        }
                        const int32_t bin = static_cast<int32_t>(wd.binBase) + retX * wd.binsY + yStart;
                        rs[j] = __ldg(offsets + bin);
                        re[j] = __ldg(offsets + bin + (yEnd - yStart));
                    }
                }
                WalkRuns32(rs, re, slot, pf, rad, sPos, sRad, R, lp.scale, xDimF, yDimF, wd.wrapX, wd.wrapY, vx, vy);
                return make_float2(vx, vy);
            }
            const int32_t bs = 1 << sh;
            for (int32_t xSq = xStart; xSq < xEnd; xSq++)
            {
                int32_t retX = xSq;
                if (retX < 0 || retX >= xDim)
                {
                    retX %= xDim;  // only reached on a wrapped axis (clamped otherwise)
                    retX = (retX < 0) ? retX + xDim : retX;
                }
                const int32_t binRow = static_cast<int32_t>(wd.binBase) + (retX >> sh) * wd.binsY;
                // the row's window cells as runs that stay in one bin and do
                // not wrap: a run's cells are consecutive cell indices, so its
                // agents are one stretch of the bin's (cell, index) order
                for (int32_t ySq = yStart; ySq < yEnd;)
                {
                    int32_t retY = ySq;
                    if (retY < 0 || retY >= yDim)
                    {
                        retY %= yDim;  // only reached on a wrapped axis (clamped otherwise)
                        retY = (retY < 0) ? retY + yDim : retY;
                    }
                    const int32_t by = retY >> sh;
                    const int32_t binEnd = min((by + 1) * bs, yDim);  // first y past the bin
                    const int32_t run = min(yEnd - ySq, binEnd - retY);
                    ySq += run;
                    const int32_t cLo = retX * yDim + retY;
                    const int32_t cHi = cLo + run - 1;
                    const int32_t s = __ldg(offsets + binRow + by);
                    const int32_t e = __ldg(offsets + binRow + by + 1);
                    for (int32_t t = s; t < e; t++)
                    {
                        const int32_t ct = __ldg(sCell + t);
                        if (ct > cHi)
                        {
                            break;  // the bin is ordered by cell
                        }
                        if (ct >= cLo && t != slot)
                        {
                            PairStep<float, kLawLinear, false, false>(pf.x, pf.y, rad, sPos[t], sRad[t], R, lp, xDimF,
                                                                      yDimF, wd.wrapX, wd.wrapY, vx, vy, sum);
                        }
                    }
                }
            }
            return make_float2(vx, vy);
        }

        __global__ void ForcesWells(const int32_t *__restrict__ bucket, const int32_t *__restrict__ offsets,
                                    const float2 *__restrict__ sPos, const float *__restrict__ sRad,
                                    const int32_t *__restrict__ sCell, const int32_t *__restrict__ wellOf,
                                    const AgentWellDev *__restrict__ wells, int32_t n, double interactionRad,
                                    bool intR, float R, float k, float *__restrict__ vel)
        {
            ChainEntry();
            const int32_t slot = blockIdx.x * blockDim.x + threadIdx.x;
            if (slot >= n)
            {
                return;
            }
            const int32_t i = bucket[slot];
            const AgentWellDev wd = wells[wellOf[slot]];  // the slots go well by well, as the agents do
            StoreDelta(vel, i, ForceSlotWell(slot, offsets, sPos, sRad, sCell, interactionRad, intR, R, k, wd));
        }

        // ForcesWells with each agent's SphericalAgent2D update fused, moved
        // within its own well (its sizes and wrap flags).
        __global__ void ForcesWellsMove(const int32_t *__restrict__ bucket, const int32_t *__restrict__ offsets,
                                        const float2 *__restrict__ sPos, const float *__restrict__ sRad,
                                        const int32_t *__restrict__ sCell, const int32_t *__restrict__ wellOf,
                                        const AgentWellDev *__restrict__ wells, int32_t n, double interactionRad,
                                        bool intR, float R, float k, float friction, float maxVel, float *__restrict__ vel,
                                        float2 *__restrict__ pos, float2 *__restrict__ velocity,
                                        int32_t *__restrict__ binOf, int32_t *__restrict__ arrival,
                                        int32_t *__restrict__ counts, int32_t *__restrict__ tileSums)
        {
            ChainEntry();
            const int32_t slot = blockIdx.x * blockDim.x + threadIdx.x;
            if (slot >= n)
            {
                return;
            }
            const int32_t i = bucket[slot];
            float2 v = velocity[i];  // in flight during the sums (48 wells: 98 ticks 11.2 -> 9.7 ms)
            const AgentWellDev wd = wells[wellOf[slot]];  // the slots go well by well, as the agents do
            const V2<float> d = ForceSlotWell(slot, offsets, sPos, sRad, sCell, interactionRad, intR, R, k, wd);
            StoreDelta(vel, i, d);
            MoveParams mp;
            mp.friction = friction;
            mp.maxVel = maxVel;
            mp.xDimF = static_cast<float>(wd.xDim);
            mp.yDimF = static_cast<float>(wd.yDim);
            mp.wrapX = wd.wrapX;
            mp.wrapY = wd.wrapY;
            float2 p = sPos[slot];
            v.x = __fadd_rn(v.x, d.x);
            v.y = __fadd_rn(v.y, d.y);
            MoveAgent(mp, p, v);
            pos[i] = p;
            velocity[i] = v;
            // BinCountWells' work for the next pass: this one's scan cleared the
            // counts, its scatter the tile sums
            const int32_t nb = WellBin(wd, p.x, p.y);
            binOf[i] = nb;
            arrival[i] = atomicAdd(counts + nb, 1);
            AddToTiles(tileSums, nb);
        }
    }

    // Whether WindowOf may take the FP32 form for this radius.
    inline bool IntegerRadius(double r)
    {
        return r >= 0.0 && r <= 0x1p20 && r == std::floor(r);
    }

    // The agents of a uniform population that a window holds.
    inline double WindowAgents(int32_t n, int64_t cells, double R)
    {
        return static_cast<double>(n) / static_cast<double>(cells) * (2.0 * R + 1.0) * (2.0 * R + 1.0);
    }

    // Whether a force pass (step: with the move) takes a group of lanes per
    // agent.  A thread per agent costs the longest window's chain, a group its
    // instructions, n times: the group pays while the windows are long for the
    // number of agents.  Their length is known as the candidates that a uniform
    // population has in one, m = n / cells * (2 R + 1)^2; where the agents
    // cluster, windows are longer and the group gains more.  Measured on GB300,
    // us per step thread / group, uniform, and with 30% in a cluster:
    //   R = 1    5k in 256^2 (m 0.7)  12.2 / 12.5   13.9 / 12.8
    //           20k in 1024^2 (0.2)   15.5 / 18.0   16.0 / 18.0
    //           20k in 256^2 (2.7)    14.4 / 16.8   19.9 / 17.0
    //           50k in 512^2 (1.7)    16.6 / 23.4   19.1 / 24.1
    //           50k in 256^2 (6.9)    17.0 / 23.6   27.4 / 25.4
    //   R = 2   50k in 2048^2 (0.3)   23.6 / 26.6   24.2 / 25.3
    //           50k in 512^2 (4.8)    19.6 / 24.4   31.1 / 25.9
    //           90k in 512^2 (8.6)    24.1 / 32.5   46.4 / 37.3
    //   R = 3.5 90k in 512^2 (22)     36.6 / 34.2   154 / 68
    // The lines lie where a uniform population is no slower than it was with one
    // thread per agent and branches per pair (us: step, 20k in 256^2 at R = 1 17.7,
    // 50k 21.5, 90k in 512^2 at R = 2 30.5; a pass without the move gained less
    // with a thread per agent: 20k in 256^2 18.3, thread 17.7, group 20.1).  On a
    // wrapped axis a thread's test of the wrap per candidate costs more and they
    // lie further out (step, R = 1, 50k in 256^2, uniform: 25.9 before, thread
    // 22.0, group 23.4; with a cluster 43.8, 32.3 and 26.5).
    inline bool GroupPerAgent(int32_t n, int64_t cells, double R, bool walls, bool step)
    {
        const double m = WindowAgents(n, cells, R);
        if (R >= 2.0)
        {
            const int32_t most = (R >= 3.0 || !walls) ? 100000 : (step ? 70000 : 60000);
            return n <= most && n <= m * (step ? 50000.0 : 25000.0);
        }
        return n <= (walls ? (step ? 30000 : 12000) : 55000) && n <= m * 8000.0;
    }

    struct ForceLawSpec
    {
        int kind = kLawLinear;
        double scale = 0.0;
        double exponent = 1.0;
        bool sums = false;  // write each agent's sum of positive forces
        bool grid = false;  // the agent grid's order and displacement (FP64)

        static ForceLawSpec Linear(double k)
        {
            ForceLawSpec l;
            l.scale = k;
            return l;
        }
    };

    struct Agents
    {
        int32_t xDim = 0, yDim = 0, maxAgents = 0;
        int64_t C = 0;
        int32_t n = 0;          // agents of the last upload
        int device = 0;
        StreamSlot stream;
        DevBuf<float> pos32, rad32, vel32;
        DevBuf<float2> velState;  // the agents' own velocities (xVel, yVel) of the resident step
        DevBuf<double> pos64, rad64, vel64;
        DevBuf<float2> sPos;
        DevBuf<double2> sPosD;  // FP64 interface path
        DevBuf<float> sRad32;
        DevBuf<double> sRad64;
        DevBuf<int32_t> cellOf, arrival, counts, offsets, tileSums, bucketTmp, bucket;
        DevBuf<float> sums32;    // per-agent sums of positive forces (FP32 path)
        DevBuf<double> sums64;   // the same, FP64 path
        bool sumsValid = false;  // sums32 holds the last dispatch's or step's sums
        int32_t nTiles = 0;
        bool countsDirty = true;  // counts not known to be zero (cleared by each scan)
        // counts, cellOf, arrival and tileSums hold the binning of the current
        // pos32, counted by the last resident step's force kernel as it moved
        // the agents: the next FP32 binning skips its count pass and the
        // scan's first
        bool binsPrecounted = false;

        // pos32 changed by other means than the resident step: the precounted
        // bins are stale and the counts must be cleared before a binning
        void DropPrecount()
        {
            if (binsPrecounted)
            {
                binsPrecounted = false;
                countsDirty = true;
            }
        }

        int Init(int32_t x, int32_t y, int32_t maxN)
        {
            xDim = x;
            yDim = y;
            maxAgents = maxN;
            C = static_cast<int64_t>(x) * y;
            device = CurrentDevice();
            HAL_TRY(CudaStatus(cudaSetDevice(device), "cudaSetDevice"));
            HAL_TRY(stream.Create("cudaStreamCreate"));
            size_t m = static_cast<size_t>(maxN > 0 ? maxN : 1);
            HAL_TRY(pos32.Alloc(2 * m, "cudaMalloc(agents)"));
            HAL_TRY(rad32.Alloc(m, "cudaMalloc(agents)"));
            HAL_TRY(vel32.Alloc(2 * m, "cudaMalloc(agents)"));
            HAL_TRY(velState.Alloc(m, "cudaMalloc(agents)"));
            HAL_TRY(CudaStatus(cudaMemset(velState.p, 0, m * sizeof(float2)), "cudaMemset"));
            HAL_TRY(sPos.Alloc(m, "cudaMalloc(agents)"));
            HAL_TRY(sRad32.Alloc(m, "cudaMalloc(agents)"));
            HAL_TRY(cellOf.Alloc(m, "cudaMalloc(agents)"));
            HAL_TRY(arrival.Alloc(m, "cudaMalloc(agents)"));
            HAL_TRY(bucketTmp.Alloc(m, "cudaMalloc(agents)"));
            HAL_TRY(bucket.Alloc(m, "cudaMalloc(agents)"));
            HAL_TRY(counts.Alloc(static_cast<size_t>(C), "cudaMalloc(bins)"));
            HAL_TRY(offsets.Alloc(static_cast<size_t>(C) + 1, "cudaMalloc(bins)"));
            nTiles = static_cast<int32_t>((C + kScanTile - 1) / kScanTile);
            HAL_TRY(tileSums.Alloc(static_cast<size_t>(nTiles), "cudaMalloc(bins)"));

            HAL_TRY(CudaStatus(cudaMemset(offsets.p, 0, (static_cast<size_t>(C) + 1) * sizeof(int32_t)), "cudaMemset"));
            return HAL_CUDA_OK;
        }

        V2<float> *SortedPosBuf(float) { return sPos.p; }
        V2<double> *SortedPosBuf(double) { return sPosD.p; }

        // Bins n agents (positions of type TP, interleaved x,y, in one of the
        // handle's own device buffers) and sorts radii of type TR alongside.
        // With ev != nullptr, records an event after each stage (count, scan,
        // scatter, stabilize) for profiling.
        template <typename TP, typename TR>
        int Bin(const TP *pos, const TR *rad, TR *sRad, cudaStream_t s, cudaEvent_t *ev = nullptr)
        {
            // the resident step's force kernel already counted these positions
            const bool pre = binsPrecounted && static_cast<const void *>(pos) == static_cast<const void *>(pos32.p);
            if (!pre)
            {
                DropPrecount();
            }
            binsPrecounted = false;
            if (countsDirty && !pre)
            {
                // a previous binning stopped before its scan cleared the counts
                HAL_TRY(CudaStatus(cudaMemsetAsync(counts.p, 0, static_cast<size_t>(C) * sizeof(int32_t), s),
                                   "cudaMemsetAsync(counts)"));
            }
            countsDirty = true;
            const int T = 256;
            unsigned ablocks = static_cast<unsigned>((n + T - 1) / T);
            if (n > 0 && !pre)
            {
                LaunchChained(BinCount<TP>, ablocks, T, s, pos, n, xDim, yDim, static_cast<V2<TP> *>(nullptr),
                              cellOf.p, arrival.p, counts.p);
                CountLaunch();
            }
            if (ev)
            {
                cudaEventRecord(ev[0], s);
            }
            if (!pre)
            {
                // (the move that counted the agents has added up the tiles too)
                LaunchChained(ScanReduce, nTiles, kScanThreads, s, counts.p, C, tileSums.p);
                CountLaunch();
            }
            if (nTiles <= kScanSumTiles)
            {
                LaunchChained(ScanApplySum, nTiles, kScanThreads, s, counts.p, C, tileSums.p, offsets.p, n);
                CountLaunch();
            }
            else
            {
                LaunchChained(ScanTiles, 1u, kScanThreads, s, tileSums.p, nTiles);
                LaunchChained(ScanApply<true>, nTiles, kScanThreads, s, counts.p, C, tileSums.p, offsets.p, n);
                CountLaunch(2);
            }
            countsDirty = (cudaPeekAtLastError() != cudaSuccess);
            if (ev)
            {
                cudaEventRecord(ev[1], s);
            }
            if (n > 0)
            {
                LaunchChained(Scatter, ablocks, T, s, cellOf.p, arrival.p, offsets.p, n, bucketTmp.p, tileSums.p, nTiles);
                CountLaunch();
            }
            if (ev)
            {
                cudaEventRecord(ev[2], s);
            }
            if (n > 0)
            {
                // pos is the handle's own device buffer (cudaMalloc'd, so
                // aligned for V2<TP>)
                LaunchChained(StabilizeSlots<TP, TR>, ablocks, T, s, offsets.p, bucketTmp.p,
                              reinterpret_cast<const V2<TP> *>(pos), rad, n, xDim, yDim, bucket.p, SortedPosBuf(TP()),
                              sRad);
                CountLaunch();
            }
            if (ev)
            {
                cudaEventRecord(ev[3], s);
            }
            return LaunchStatus("agent binning");
        }

        // Pass 4 with force law `law`: velocity deltas (from zero, or from
        // velIn) into vel, and with law.sums each agent's sum of positive
        // forces into sums.  law.grid (FP64 only) selects the agent grid's
        // visiting order and displacement.
        template <typename T, typename TV>
        int Force(const T *sRad, double R, const ForceLawSpec &law, bool wrapX, bool wrapY, TV *vel, T *sums,
                  const TV *velIn, cudaStream_t s)
        {
            if (n == 0)
            {
                return HAL_CUDA_OK;
            }
            const int T_ = 128;
            const unsigned blocks = static_cast<unsigned>((n + T_ - 1) / T_);
            LawParams<T> lp;
            lp.scale = static_cast<T>(law.scale);
            lp.exponent = static_cast<T>(law.exponent);
            auto go = [&](auto kernel) {
                LaunchChained(kernel, blocks, T_, s, bucket.p, offsets.p, SortedPosBuf(T()), sRad, n, R,
                              static_cast<T>(R), lp, xDim, yDim, static_cast<int32_t>(wrapX),
                              static_cast<int32_t>(wrapY), vel, sums, velIn);
            };
            const bool grid = std::is_same<T, double>::value && law.grid;
            switch (law.kind * 4 + (law.sums ? 2 : 0) + (grid ? 1 : 0))
            {
            case 0:
                // the interface's law on a grid with walls: the wrap tests compiled out
                if constexpr (std::is_same<T, float>::value)
                {
                    if (GroupPerAgent(n, C, R, !wrapX && !wrapY, false) && velIn == nullptr)
                    {
                        const unsigned groups =
                            static_cast<unsigned>((static_cast<int64_t>(n) * kGroupLanes + T_ - 1) / T_);
                        LaunchChained(!wrapX && !wrapY ? ForcesGroup<true> : ForcesGroup<false>, groups, T_, s, bucket.p,
                                      offsets.p, SortedPosBuf(T()), sRad, n, R, IntegerRadius(R), static_cast<T>(R), lp,
                                      xDim, yDim, static_cast<int32_t>(wrapX), static_cast<int32_t>(wrapY), vel);
                        break;
                    }
                    if (!wrapX && !wrapY)
                    {
                        go(Forces<T, TV, kLawLinear, false, false, true>);
                        break;
                    }
                }
                if constexpr (std::is_same<T, double>::value && std::is_same<TV, double>::value)
                {
                    // (few agents a window: kPairSparse; and chained, 2 to 9 us of
                    // 100, since no CTA's work is long enough to gather on an SM)
                    const bool sparse = WindowAgents(n, C, R) < 2.0;
                    const int32_t least = sparse && n >= kPairSparse ? 2 : 1;
                    const int32_t perGroup = std::min(std::max(n / kPairGroups, least), kPairPerGroup);
                    const int64_t groups = (static_cast<int64_t>(n) + perGroup - 1) / perGroup;
                    const auto launch = [&](auto start) {
                        start(!wrapX && !wrapY ? ForcesGroup64<true> : ForcesGroup64<false>,
                              static_cast<unsigned>((groups * kGroupLanes + kPairThreads - 1) / kPairThreads),
                              kPairThreads, s, bucket.p, offsets.p, SortedPosBuf(T()), sRad, n, perGroup, R + 0.0, lp,
                              xDim, yDim, static_cast<int32_t>(wrapX), static_cast<int32_t>(wrapY), vel, velIn);
                    };
                    if (sparse)
                    {
                        launch([](auto... args) { LaunchChained(args...); });
                    }
                    else
                    {
                        launch([](auto... args) { LaunchAfter(args...); });
                    }
                    break;
                }
                go(Forces<T, TV, kLawLinear, false, false>);
                break;
            case 1: go(Forces<T, TV, kLawLinear, false, true>); break;
            case 2: go(Forces<T, TV, kLawLinear, true, false>); break;
            case 3: go(Forces<T, TV, kLawLinear, true, true>); break;
            case 4: go(Forces<T, TV, kLawClamped, false, false>); break;
            case 5: go(Forces<T, TV, kLawClamped, false, true>); break;
            case 6: go(Forces<T, TV, kLawClamped, true, false>); break;
            case 7: go(Forces<T, TV, kLawClamped, true, true>); break;
            case 8: go(Forces<T, TV, kLawPower, false, false>); break;
            case 9: go(Forces<T, TV, kLawPower, false, true>); break;
            case 10: go(Forces<T, TV, kLawPower, true, false>); break;
            default: go(Forces<T, TV, kLawPower, true, true>); break;
            }
            CountLaunch();
            return LaunchStatus("agent forces");
        }

        // The interface's pass 4: linear law, deltas from zero.
        template <typename T, typename TV>
        int Force(const T *sRad, double R, double k, bool wrapX, bool wrapY, TV *vel, cudaStream_t s)
        {
            return Force<T, TV>(sRad, R, ForceLawSpec::Linear(k), wrapX, wrapY, vel, static_cast<T *>(nullptr),
                                static_cast<const TV *>(nullptr), s);
        }

        // Buffer of the FP32 force sums, allocated on first use.
        int SumsBuf32(float **out)
        {
            if (sums32.p == nullptr)
            {
                HAL_TRY(sums32.Alloc(static_cast<size_t>(maxAgents > 0 ? maxAgents : 1), "cudaMalloc(force sums)"));
            }
            *out = sums32.p;
            return HAL_CUDA_OK;
        }
    };

    const int32_t *AgentsCellOffsets(const hal_cuda_agents *a, int32_t *xDim, int32_t *yDim);
}

namespace
{
    // One resident tick of the agents: bin, then forces with the move fused.
    int StepOnce(halcuda::Agents &a, double R, const halcuda::ForceLawSpec &law, const halcuda::MoveParams &mp,
                 cudaStream_t s)
    {
        using namespace halcuda;
        HAL_TRY((a.Bin<float, float>(a.pos32.p, a.rad32.p, a.sRad32.p, s)));
        if (a.n == 0)
        {
            return HAL_CUDA_OK;
        }
        float *sums = nullptr;
        if (law.sums)
        {
            HAL_TRY(a.SumsBuf32(&sums));
        }
        const int T = 128;
        const unsigned blocks = static_cast<unsigned>((a.n + T - 1) / T);
        LawParams<float> lp;
        lp.scale = static_cast<float>(law.scale);
        lp.exponent = static_cast<float>(law.exponent);
        // the force kernel counts the moved agents into their new cells (the
        // next binning's count pass); this binning's scan cleared the counts
        auto go = [&](auto kernel) {
            LaunchChained(kernel, blocks, T, s, a.bucket.p, a.offsets.p, a.sPos.p, a.sRad32.p, a.n, R,
                          static_cast<float>(R), lp, a.xDim, a.yDim, mp, a.vel32.p,
                          reinterpret_cast<float2 *>(a.pos32.p), a.velState.p, sums, a.cellOf.p, a.arrival.p,
                          a.counts.p, a.tileSums.p);
        };
        const bool walls = !mp.wrapX && !mp.wrapY;
        if (law.kind == kLawLinear && !law.sums && GroupPerAgent(a.n, a.C, R, walls, true))
        {
            const unsigned groups = static_cast<unsigned>((static_cast<int64_t>(a.n) * kGroupLanes + T - 1) / T);
            LaunchChained(walls ? ForcesMoveGroup<true> : ForcesMoveGroup<false>, groups, T, s, a.bucket.p, a.offsets.p,
                          a.sPos.p, a.sRad32.p, a.n, R, IntegerRadius(R), static_cast<float>(R), lp, a.xDim, a.yDim, mp,
                          a.vel32.p, reinterpret_cast<float2 *>(a.pos32.p), a.velState.p, a.cellOf.p, a.arrival.p,
                          a.counts.p, a.tileSums.p);
        }
        else
        switch (law.kind * 2 + (law.sums ? 1 : 0))
        {
        case 0:
            if (walls)
            {
                go(ForcesMove<kLawLinear, false, true>);  // walls: the wrap tests compiled out
            }
            else
            {
                go(ForcesMove<kLawLinear, false>);
            }
            break;
        case 1: go(ForcesMove<kLawLinear, true>); break;
        case 2: go(ForcesMove<kLawClamped, false>); break;
        case 3: go(ForcesMove<kLawClamped, true>); break;
        case 4: go(ForcesMove<kLawPower, false>); break;
        default: go(ForcesMove<kLawPower, true>); break;
        }
        CountLaunch();
        const int rc = LaunchStatus("agent forces and move");
        a.binsPrecounted = (rc == HAL_CUDA_OK);
        a.countsDirty = (rc != HAL_CUDA_OK);
        return rc;
    }
}

using halcuda::Agents;

struct hal_cuda_agents : public Agents
{
};

namespace halcuda
{
    AgentBinsView AgentsBins(const hal_cuda_agents *a)
    {
        AgentBinsView v;
        v.offsets = a->offsets.p;
        v.bucket = a->bucket.p;
        v.cellOf = a->cellOf.p;
        v.n = a->n;
        v.xDim = a->xDim;
        v.yDim = a->yDim;
        v.device = a->device;
        v.stream = a->stream.Get();
        return v;
    }

    const int32_t *AgentsCellOffsets(const hal_cuda_agents *a, int32_t *xDim, int32_t *yDim)
    {
        *xDim = a->xDim;
        *yDim = a->yDim;
        return a->offsets.p;
    }
}

extern "C" int hal_cuda_agents_create(int32_t xDim, int32_t yDim, int32_t maxAgents, hal_cuda_agents **out)
{
    HAL_REQUIRE(out != nullptr, "hal_cuda_agents_create: out is NULL");
    *out = nullptr;
    HAL_REQUIRE(xDim > 0 && yDim > 0, "hal_cuda_agents_create: dimensions must be positive");
    HAL_REQUIRE(static_cast<int64_t>(xDim) * yDim < (int64_t(1) << 31) - 1,
                "hal_cuda_agents_create: xDim*yDim exceeds int32");
    HAL_REQUIRE(maxAgents >= 0, "hal_cuda_agents_create: negative capacity");
    hal_cuda_agents *h = new (std::nothrow) hal_cuda_agents();
    if (h == nullptr)
    {
        halcuda::SetError("hal_cuda_agents_create: out of host memory");
        return HAL_CUDA_ENOMEM;
    }
    int rc = h->Init(xDim, yDim, maxAgents);
    if (rc != HAL_CUDA_OK)
    {
        delete h;
        return rc;
    }
    *out = h;
    return HAL_CUDA_OK;
}

extern "C" int hal_cuda_agents_destroy(hal_cuda_agents *h)
{
    if (h != nullptr)
    {
        cudaSetDevice(h->device);
        cudaStreamSynchronize(h->stream.Get());
        delete h;
    }
    return HAL_CUDA_OK;
}

namespace
{
    // The cell window spans about 2R cells per axis; a wrapped axis walks all
    // of it, so the radius is bounded to keep every launch short.
    constexpr double kMaxInteractionRad = 1048576.0;

    bool RadiusOk(double r)
    {
        return std::isfinite(r) && r >= 0.0 && r <= kMaxInteractionRad;
    }
}

namespace
{
    // A hal_cuda_force_law checked and turned into a spec; sums as given.
    int LawFrom(const hal_cuda_force_law *law, bool sums, const char *who, halcuda::ForceLawSpec *out)
    {
        HAL_REQUIRE(law != nullptr, "%s: law is NULL", who);
        HAL_REQUIRE(law->kind == HAL_CUDA_FORCE_LINEAR || law->kind == HAL_CUDA_FORCE_LINEAR_CLAMPED ||
                        law->kind == HAL_CUDA_FORCE_POWER,
                    "%s: unknown force law kind %d", who, law->kind);
        HAL_REQUIRE(std::isfinite(law->scale), "%s: the law's scale must be finite", who);
        HAL_REQUIRE(law->kind != HAL_CUDA_FORCE_POWER || std::isfinite(law->exponent),
                    "%s: the law's exponent must be finite", who);
        out->kind = law->kind;
        out->scale = law->scale;
        out->exponent = (law->kind == HAL_CUDA_FORCE_POWER) ? law->exponent : 1.0;
        out->sums = sums;
        out->grid = false;
        return HAL_CUDA_OK;
    }

    // The FP64 interface path's buffers, allocated on its first call.
    int Ensure64(hal_cuda_agents *h)
    {
        if (h->sPosD.p == nullptr)  // the last of the FP64 buffers: all or none are allocated
        {
            size_t m = static_cast<size_t>(h->maxAgents > 0 ? h->maxAgents : 1);
            HAL_TRY(h->pos64.Alloc(2 * m, "cudaMalloc(agents64)"));
            HAL_TRY(h->rad64.Alloc(m, "cudaMalloc(agents64)"));
            HAL_TRY(h->vel64.Alloc(2 * m, "cudaMalloc(agents64)"));
            HAL_TRY(h->sRad64.Alloc(m, "cudaMalloc(agents64)"));
            HAL_TRY(h->sPosD.Alloc(m, "cudaMalloc(agents64)"));
        }
        return HAL_CUDA_OK;
    }
}

extern "C" int hal_cuda_accumulate_forces(hal_cuda_agents *h, const double *positions, int64_t posLen,
                                          const double *radii, int64_t radLen, double *velocityDeltas,
                                          double interactionRad, double springConstant, int32_t xDim, int32_t yDim,
                                          int32_t wrapX, int32_t wrapY)
{
    HAL_TRACE();
    HAL_REQUIRE(h != nullptr, "hal_cuda_accumulate_forces: handle is NULL");
    HAL_REQUIRE(xDim == h->xDim && yDim == h->yDim,
                "CudaAgentForceBackend2D::AccumulateForces called with dimensions differing from construction");
    HAL_REQUIRE(posLen == 2 * radLen && radLen >= 0,
                "CudaAgentForceBackend2D::AccumulateForces: positions must hold two values per radius");
    HAL_REQUIRE(radLen <= h->maxAgents,
                "CudaAgentForceBackend2D::AccumulateForces called with more agents than the construction-time capacity");
    HAL_REQUIRE(radLen == 0 || (positions != nullptr && radii != nullptr && velocityDeltas != nullptr),
                "hal_cuda_accumulate_forces: NULL array");
    HAL_REQUIRE(RadiusOk(interactionRad), "hal_cuda_accumulate_forces: interactionRad %g outside [0, %g]",
                interactionRad, kMaxInteractionRad);
    using namespace halcuda;
    HAL_TRY(CudaStatus(cudaSetDevice(h->device), "cudaSetDevice"));
    HAL_TRY(Ensure64(h));
    cudaStream_t s = h->stream.Get();
    h->n = static_cast<int32_t>(radLen);
    if (h->n > 0)
    {
        HAL_TRY(CudaStatus(cudaMemcpyAsync(h->pos64.p, positions, posLen * sizeof(double), cudaMemcpyHostToDevice, s),
                           "cudaMemcpy(positions)"));
        HAL_TRY(CudaStatus(cudaMemcpyAsync(h->rad64.p, radii, radLen * sizeof(double), cudaMemcpyHostToDevice, s),
                           "cudaMemcpy(radii)"));
    }
    HAL_TRY((h->Bin<double, double>(h->pos64.p, h->rad64.p, h->sRad64.p, s)));
    HAL_TRY((h->Force<double, double>(h->sRad64.p, interactionRad, springConstant, wrapX != 0, wrapY != 0,
                                      h->vel64.p, s)));
    if (h->n > 0)
    {
        HAL_TRY(CudaStatus(cudaMemcpyAsync(velocityDeltas, h->vel64.p, posLen * sizeof(double), cudaMemcpyDeviceToHost, s),
                           "cudaMemcpy(velocityDeltas)"));
    }
    return CudaStatus(cudaStreamSynchronize(s), "hal_cuda_accumulate_forces");
}

extern "C" int hal_cuda_sum_forces(hal_cuda_agents *h, const double *positions, const double *radii, int64_t n,
                                   const double *velocities, double *velocitiesOut, double *forceSums,
                                   double interactionRad, const hal_cuda_force_law *law, int32_t order,
                                   int32_t xDim, int32_t yDim, int32_t wrapX, int32_t wrapY)
{
    HAL_TRACE();
    const char *who = "hal_cuda_sum_forces";
    HAL_REQUIRE(h != nullptr, "%s: handle is NULL", who);
    HAL_REQUIRE(xDim == h->xDim && yDim == h->yDim,
                "CudaAgentForceBackend2D::SumForces called with dimensions differing from construction");
    HAL_REQUIRE(n >= 0 && n <= h->maxAgents,
                "CudaAgentForceBackend2D::SumForces called with more agents than the construction-time capacity");
    HAL_REQUIRE(n == 0 || (positions != nullptr && radii != nullptr && velocitiesOut != nullptr),
                "%s: NULL array", who);
    HAL_REQUIRE(RadiusOk(interactionRad), "%s: interactionRad %g outside [0, %g]", who, interactionRad,
                kMaxInteractionRad);
    HAL_REQUIRE(order == HAL_CUDA_ORDER_BACKEND || order == HAL_CUDA_ORDER_AGENTGRID, "%s: unknown order %d", who,
                order);
    halcuda::ForceLawSpec spec;
    HAL_TRY(LawFrom(law, forceSums != nullptr, who, &spec));
    spec.grid = (order == HAL_CUDA_ORDER_AGENTGRID);
    using namespace halcuda;
    HAL_TRY(CudaStatus(cudaSetDevice(h->device), "cudaSetDevice"));
    HAL_TRY(Ensure64(h));
    if (forceSums != nullptr && h->sums64.p == nullptr)
    {
        HAL_TRY(h->sums64.Alloc(static_cast<size_t>(h->maxAgents > 0 ? h->maxAgents : 1), "cudaMalloc(force sums)"));
    }
    cudaStream_t s = h->stream.Get();
    h->n = static_cast<int32_t>(n);
    h->sumsValid = false;  // the FP32 sums are not this call's
    const size_t bytes2 = 2 * static_cast<size_t>(n) * sizeof(double);
    if (n > 0)
    {
        HAL_TRY(CudaStatus(cudaMemcpyAsync(h->pos64.p, positions, bytes2, cudaMemcpyHostToDevice, s),
                           "cudaMemcpy(positions)"));
        HAL_TRY(CudaStatus(cudaMemcpyAsync(h->rad64.p, radii, static_cast<size_t>(n) * sizeof(double),
                                           cudaMemcpyHostToDevice, s), "cudaMemcpy(radii)"));
        if (velocities != nullptr)
        {
            HAL_TRY(CudaStatus(cudaMemcpyAsync(h->vel64.p, velocities, bytes2, cudaMemcpyHostToDevice, s),
                               "cudaMemcpy(velocities)"));
        }
    }
    HAL_TRY((h->Bin<double, double>(h->pos64.p, h->rad64.p, h->sRad64.p, s)));
    // velocities in place: each thread reads and writes only its own agent
    HAL_TRY((h->Force<double, double>(h->sRad64.p, interactionRad, spec, wrapX != 0, wrapY != 0, h->vel64.p,
                                      forceSums != nullptr ? h->sums64.p : nullptr,
                                      velocities != nullptr ? h->vel64.p : nullptr, s)));
    if (n > 0)
    {
        HAL_TRY(CudaStatus(cudaMemcpyAsync(velocitiesOut, h->vel64.p, bytes2, cudaMemcpyDeviceToHost, s),
                           "cudaMemcpy(velocities)"));
        if (forceSums != nullptr)
        {
            HAL_TRY(CudaStatus(cudaMemcpyAsync(forceSums, h->sums64.p, static_cast<size_t>(n) * sizeof(double),
                                               cudaMemcpyDeviceToHost, s), "cudaMemcpy(force sums)"));
        }
    }
    return CudaStatus(cudaStreamSynchronize(s), who);
}

extern "C" int hal_cuda_agents_upload(hal_cuda_agents *h, const float *positions, const float *radii, int32_t n)
{
    HAL_REQUIRE(h != nullptr, "hal_cuda_agents_upload: handle is NULL");
    HAL_REQUIRE(n >= 0 && n <= h->maxAgents, "AgentForceKernel2D::UploadAgents: agent count %d outside [0, %d]", n,
                h->maxAgents);
    HAL_REQUIRE(n == 0 || (positions != nullptr && radii != nullptr), "hal_cuda_agents_upload: NULL array");
    using namespace halcuda;
    HAL_TRY(CudaStatus(cudaSetDevice(h->device), "cudaSetDevice"));
    cudaStream_t s = h->stream.Get();
    h->DropPrecount();
    h->n = n;
    if (n > 0)
    {
        HAL_TRY(CudaStatus(cudaMemcpyAsync(h->pos32.p, positions, 2 * static_cast<size_t>(n) * sizeof(float),
                                           cudaMemcpyHostToDevice, s), "cudaMemcpy(positions)"));
        HAL_TRY(CudaStatus(cudaMemcpyAsync(h->rad32.p, radii, static_cast<size_t>(n) * sizeof(float),
                                           cudaMemcpyHostToDevice, s), "cudaMemcpy(radii)"));
        HAL_TRY(CudaStatus(cudaMemsetAsync(h->velState.p, 0, static_cast<size_t>(n) * sizeof(float2), s),
                           "cudaMemsetAsync(velocities)"));
    }
    return CudaStatus(cudaStreamSynchronize(s), "hal_cuda_agents_upload");
}

extern "C" int hal_cuda_agents_set_velocities(hal_cuda_agents *h, const float *velocities, int32_t n)
{
    HAL_REQUIRE(h != nullptr, "hal_cuda_agents_set_velocities: handle is NULL");
    HAL_REQUIRE(n == h->n, "hal_cuda_agents_set_velocities: %d agents given, %d uploaded", n, h->n);
    using namespace halcuda;
    HAL_TRY(CudaStatus(cudaSetDevice(h->device), "cudaSetDevice"));
    cudaStream_t s = h->stream.Get();
    if (n > 0)
    {
        const size_t bytes = static_cast<size_t>(n) * sizeof(float2);
        HAL_TRY(CudaStatus(velocities != nullptr
                               ? cudaMemcpyAsync(h->velState.p, velocities, bytes, cudaMemcpyHostToDevice, s)
                               : cudaMemsetAsync(h->velState.p, 0, bytes, s),
                           "hal_cuda_agents_set_velocities"));
    }
    return CudaStatus(cudaStreamSynchronize(s), "hal_cuda_agents_set_velocities");
}

extern "C" int hal_cuda_agents_get_state(hal_cuda_agents *h, float *positions, float *velocities, int32_t n)
{
    HAL_REQUIRE(h != nullptr, "hal_cuda_agents_get_state: handle is NULL");
    HAL_REQUIRE(n == h->n, "hal_cuda_agents_get_state: %d agents requested, %d uploaded", n, h->n);
    using namespace halcuda;
    HAL_TRY(CudaStatus(cudaSetDevice(h->device), "cudaSetDevice"));
    cudaStream_t s = h->stream.Get();
    const size_t bytes = static_cast<size_t>(n) * sizeof(float2);
    PopulateOutput(positions, bytes);
    PopulateOutput(velocities, bytes);
    if (n > 0 && positions != nullptr)
    {
        HAL_TRY(CudaStatus(cudaMemcpyAsync(positions, h->pos32.p, bytes, cudaMemcpyDeviceToHost, s),
                           "cudaMemcpy(positions)"));
    }
    if (n > 0 && velocities != nullptr)
    {
        HAL_TRY(CudaStatus(cudaMemcpyAsync(velocities, h->velState.p, bytes, cudaMemcpyDeviceToHost, s),
                           "cudaMemcpy(velocities)"));
    }
    return CudaStatus(cudaStreamSynchronize(s), "hal_cuda_agents_get_state");
}

namespace halcuda
{
    // ---- resident steps inside another handle's run (hal_cuda_adi_run_coupled)

    int CoupledStepBegin(hal_cuda_agents *h, const CoupledStep &st, cudaStream_t s)
    {
        HAL_REQUIRE(h != nullptr, "hal_cuda_adi_run_coupled: agent handle is NULL");
        HAL_REQUIRE(RadiusOk(st.interactionRad), "hal_cuda_adi_run_coupled: interactionRad %g outside [0, %g]",
                    st.interactionRad, kMaxInteractionRad);
        HAL_REQUIRE(std::isfinite(st.springConstant), "hal_cuda_adi_run_coupled: springConstant must be finite");
        HAL_REQUIRE(std::isfinite(st.friction), "hal_cuda_adi_run_coupled: friction must be finite");
        HAL_REQUIRE(!std::isnan(st.maxVel), "hal_cuda_adi_run_coupled: maxVel is NaN");
        HAL_TRY(CudaStatus(cudaSetDevice(h->device), "cudaSetDevice"));
        // the agent handle's own queued work comes first
        cudaStream_t own = h->stream.Get();
        if (own != s)
        {
            cudaEvent_t ev = nullptr;
            HAL_TRY(CudaStatus(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming), "cudaEventCreate"));
            cudaError_t e = cudaEventRecord(ev, own);
            if (e == cudaSuccess)
            {
                e = cudaStreamWaitEvent(s, ev, 0);
            }
            cudaEventDestroy(ev);
            HAL_TRY(CudaStatus(e, "hal_cuda_adi_run_coupled: stream order"));
        }
        // every replayed tick starts from counts that hold the current
        // positions' binning (the previous tick's force kernel counted them)
        if (!h->binsPrecounted && h->n > 0)
        {
            if (h->countsDirty)
            {
                HAL_TRY(CudaStatus(cudaMemsetAsync(h->counts.p, 0, static_cast<size_t>(h->C) * sizeof(int32_t), s),
                                   "cudaMemsetAsync(counts)"));
            }
            const int T = 256;
            BinCount<float><<<static_cast<unsigned>((h->n + T - 1) / T), T, 0, s>>>(
                h->pos32.p, h->n, h->xDim, h->yDim, static_cast<float2 *>(nullptr), h->cellOf.p, h->arrival.p,
                h->counts.p);
            ScanReduce<<<static_cast<unsigned>(h->nTiles), kScanThreads, 0, s>>>(h->counts.p, h->C, h->tileSums.p);
            CountLaunch(2);
            HAL_TRY(LaunchStatus("agent binning"));
            h->binsPrecounted = true;
            h->countsDirty = false;
        }
        h->sumsValid = false;
        return HAL_CUDA_OK;
    }

    int CoupledStepOnce(hal_cuda_agents *h, const CoupledStep &st, int32_t wrapX, int32_t wrapY, cudaStream_t s)
    {
        MoveParams mp;
        mp.friction = static_cast<float>(st.friction);
        mp.maxVel = (st.maxVel < 0 || std::isinf(st.maxVel)) ? -1.0f : static_cast<float>(st.maxVel);
        mp.xDimF = static_cast<float>(h->xDim);
        mp.yDimF = static_cast<float>(h->yDim);
        mp.wrapX = wrapX != 0;
        mp.wrapY = wrapY != 0;
        return StepOnce(*h, st.interactionRad, ForceLawSpec::Linear(st.springConstant), mp, s);
    }

    int CoupledStepEnd(hal_cuda_agents *h, cudaStream_t s)
    {
        // the agent handle's later work waits for the run
        cudaStream_t own = h->stream.Get();
        if (own == s)
        {
            return HAL_CUDA_OK;
        }
        cudaEvent_t ev = nullptr;
        HAL_TRY(CudaStatus(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming), "cudaEventCreate"));
        cudaError_t e = cudaEventRecord(ev, s);
        if (e == cudaSuccess)
        {
            e = cudaStreamWaitEvent(own, ev, 0);
        }
        cudaEventDestroy(ev);
        return CudaStatus(e, "hal_cuda_adi_run_coupled: stream order");
    }

    int32_t CoupledAgentCount(const hal_cuda_agents *h)
    {
        return h->n;
    }

    bool CoupledBinsPrecounted(const hal_cuda_agents *h)
    {
        return h->binsPrecounted;
    }
}

namespace
{
    int StepCommon(hal_cuda_agents *h, int32_t ticks, double interactionRad, const halcuda::ForceLawSpec &law,
                   int32_t wrapX, int32_t wrapY, double friction, double maxVel, const char *who)
    {
        HAL_REQUIRE(h != nullptr, "%s: handle is NULL", who);
        HAL_REQUIRE(ticks >= 0, "%s: ticks must be >= 0", who);
        HAL_REQUIRE(RadiusOk(interactionRad), "%s: interactionRad %g outside [0, %g]", who, interactionRad,
                    kMaxInteractionRad);
        HAL_REQUIRE(std::isfinite(friction), "%s: friction must be finite", who);
        HAL_REQUIRE(!std::isnan(maxVel), "%s: maxVel is NaN", who);
        using namespace halcuda;
        HAL_TRY(CudaStatus(cudaSetDevice(h->device), "cudaSetDevice"));
        cudaStream_t s = h->stream.Get();
        MoveParams mp;
        mp.friction = static_cast<float>(friction);
        mp.maxVel = (maxVel < 0 || std::isinf(maxVel)) ? -1.0f : static_cast<float>(maxVel);
        mp.xDimF = static_cast<float>(h->xDim);
        mp.yDimF = static_cast<float>(h->yDim);
        mp.wrapX = wrapX != 0;
        mp.wrapY = wrapY != 0;
        h->sumsValid = false;
        for (int32_t t = 0; t < ticks; t++)
        {
            HAL_TRY(StepOnce(*h, interactionRad, law, mp, s));
        }
        h->sumsValid = law.sums && ticks > 0;
        return HAL_CUDA_OK;
    }

    int DispatchCommon(hal_cuda_agents *h, double interactionRad, const halcuda::ForceLawSpec &law, int32_t wrapX,
                       int32_t wrapY, const char *who)
    {
        HAL_REQUIRE(h != nullptr, "%s: handle is NULL", who);
        HAL_REQUIRE(RadiusOk(interactionRad), "%s: interactionRad %g outside [0, %g]", who, interactionRad,
                    kMaxInteractionRad);
        using namespace halcuda;
        HAL_TRY(CudaStatus(cudaSetDevice(h->device), "cudaSetDevice"));
        cudaStream_t s = h->stream.Get();
        h->sumsValid = false;
        HAL_TRY((h->Bin<float, float>(h->pos32.p, h->rad32.p, h->sRad32.p, s)));
        float *sums = nullptr;
        if (law.sums)
        {
            HAL_TRY(h->SumsBuf32(&sums));
        }
        HAL_TRY((h->Force<float, float>(h->sRad32.p, interactionRad, law, wrapX != 0, wrapY != 0, h->vel32.p, sums,
                                        static_cast<const float *>(nullptr), s)));
        h->sumsValid = law.sums;
        return HAL_CUDA_OK;
    }
}

extern "C" int hal_cuda_agents_step(hal_cuda_agents *h, int32_t ticks, double interactionRad, double springConstant,
                                    int32_t wrapX, int32_t wrapY, double friction, double maxVel)
{
    HAL_TRACE();
    return StepCommon(h, ticks, interactionRad, halcuda::ForceLawSpec::Linear(springConstant), wrapX, wrapY, friction,
                      maxVel, "hal_cuda_agents_step");
}

extern "C" int hal_cuda_agents_step_law(hal_cuda_agents *h, int32_t ticks, double interactionRad,
                                        const hal_cuda_force_law *law, int32_t withSums, int32_t wrapX,
                                        int32_t wrapY, double friction, double maxVel)
{
    HAL_TRACE();
    halcuda::ForceLawSpec spec;
    HAL_TRY(LawFrom(law, withSums != 0, "hal_cuda_agents_step_law", &spec));
    return StepCommon(h, ticks, interactionRad, spec, wrapX, wrapY, friction, maxVel, "hal_cuda_agents_step_law");
}

extern "C" int hal_cuda_agents_dispatch(hal_cuda_agents *h, double interactionRad, double springConstant,
                                        int32_t wrapX, int32_t wrapY)
{
    HAL_TRACE();
    return DispatchCommon(h, interactionRad, halcuda::ForceLawSpec::Linear(springConstant), wrapX, wrapY,
                          "hal_cuda_agents_dispatch");
}

extern "C" int hal_cuda_agents_dispatch_law(hal_cuda_agents *h, double interactionRad, const hal_cuda_force_law *law,
                                            int32_t withSums, int32_t wrapX, int32_t wrapY)
{
    HAL_TRACE();
    halcuda::ForceLawSpec spec;
    HAL_TRY(LawFrom(law, withSums != 0, "hal_cuda_agents_dispatch_law", &spec));
    return DispatchCommon(h, interactionRad, spec, wrapX, wrapY, "hal_cuda_agents_dispatch_law");
}

extern "C" int hal_cuda_agents_get_force_sums(hal_cuda_agents *h, float *forceSums, int32_t n)
{
    HAL_REQUIRE(h != nullptr, "hal_cuda_agents_get_force_sums: handle is NULL");
    HAL_REQUIRE(n == h->n, "hal_cuda_agents_get_force_sums: %d agents requested, %d uploaded", n, h->n);
    HAL_REQUIRE(n == 0 || forceSums != nullptr, "hal_cuda_agents_get_force_sums: NULL array");
    HAL_REQUIRE(h->sumsValid || n == 0,
                "hal_cuda_agents_get_force_sums: the last dispatch or step did not compute force sums");
    using namespace halcuda;
    HAL_TRY(CudaStatus(cudaSetDevice(h->device), "cudaSetDevice"));
    cudaStream_t s = h->stream.Get();
    if (n > 0)
    {
        HAL_TRY(CudaStatus(cudaMemcpyAsync(forceSums, h->sums32.p, static_cast<size_t>(n) * sizeof(float),
                                           cudaMemcpyDeviceToHost, s), "cudaMemcpy(force sums)"));
    }
    return CudaStatus(cudaStreamSynchronize(s), "hal_cuda_agents_get_force_sums");
}

extern "C" int hal_cuda_agents_download(hal_cuda_agents *h, float *velocityDeltas, int32_t n)
{
    HAL_REQUIRE(h != nullptr, "hal_cuda_agents_download: handle is NULL");
    HAL_REQUIRE(n == h->n, "hal_cuda_agents_download: %d agents requested, %d uploaded", n, h->n);
    HAL_REQUIRE(n == 0 || velocityDeltas != nullptr, "hal_cuda_agents_download: NULL array");
    using namespace halcuda;
    HAL_TRY(CudaStatus(cudaSetDevice(h->device), "cudaSetDevice"));
    cudaStream_t s = h->stream.Get();
    if (n > 0)
    {
        HAL_TRY(CudaStatus(cudaMemcpyAsync(velocityDeltas, h->vel32.p, 2 * static_cast<size_t>(n) * sizeof(float),
                                           cudaMemcpyDeviceToHost, s), "cudaMemcpy(velocityDeltas)"));
    }
    return CudaStatus(cudaStreamSynchronize(s), "hal_cuda_agents_download");
}

extern "C" int hal_cuda_agents_get_bins(hal_cuda_agents *h, int32_t *cellOffsets, int32_t *bucketAgents)
{
    HAL_REQUIRE(h != nullptr, "hal_cuda_agents_get_bins: handle is NULL");
    using namespace halcuda;
    HAL_TRY(CudaStatus(cudaSetDevice(h->device), "cudaSetDevice"));
    cudaStream_t s = h->stream.Get();
    if (cellOffsets != nullptr)
    {
        HAL_TRY(CudaStatus(cudaMemcpyAsync(cellOffsets, h->offsets.p, (static_cast<size_t>(h->C) + 1) * sizeof(int32_t),
                                           cudaMemcpyDeviceToHost, s), "cudaMemcpy(offsets)"));
    }
    if (bucketAgents != nullptr && h->n > 0)
    {
        HAL_TRY(CudaStatus(cudaMemcpyAsync(bucketAgents, h->bucket.p, static_cast<size_t>(h->n) * sizeof(int32_t),
                                           cudaMemcpyDeviceToHost, s), "cudaMemcpy(bucket)"));
    }
    return CudaStatus(cudaStreamSynchronize(s), "hal_cuda_agents_get_bins");
}

extern "C" int hal_cuda_agents_sync(hal_cuda_agents *h)
{
    HAL_REQUIRE(h != nullptr, "hal_cuda_agents_sync: handle is NULL");
    HAL_TRY(halcuda::CudaStatus(cudaSetDevice(h->device), "cudaSetDevice"));
    return halcuda::CudaStatus(cudaStreamSynchronize(h->stream.Get()), "hal_cuda_agents_sync");
}

extern "C" void *hal_cuda_agents_stream(hal_cuda_agents *h)
{
    return h ? static_cast<void *>(h->stream.Get()) : nullptr;
}

extern "C" int hal_cuda_agents_set_stream(hal_cuda_agents *h, void *stream)
{
    HAL_REQUIRE(h != nullptr, "hal_cuda_agents_set_stream: handle is NULL");
    h->stream.Set(stream);
    return HAL_CUDA_OK;
}

extern "C" int hal_cuda_agents_profile(hal_cuda_agents *h, int32_t iters, double interactionRad, double springConstant,
                                       int32_t wrapX, int32_t wrapY, float *ms)
{
    HAL_REQUIRE(h != nullptr && ms != nullptr, "hal_cuda_agents_profile: NULL argument");
    HAL_REQUIRE(iters > 0, "hal_cuda_agents_profile: iters must be positive");
    HAL_REQUIRE(RadiusOk(interactionRad), "hal_cuda_agents_profile: interactionRad out of range");
    using namespace halcuda;
    HAL_TRY(CudaStatus(cudaSetDevice(h->device), "cudaSetDevice"));
    cudaStream_t s = h->stream.Get();
    cudaEvent_t ev[6];
    for (auto &e : ev)
    {
        HAL_TRY(CudaStatus(cudaEventCreate(&e), "cudaEventCreate"));
    }
    double acc[6] = {0, 0, 0, 0, 0, 0};
    int rc = HAL_CUDA_OK;
    for (int32_t t = 0; t < iters && rc == HAL_CUDA_OK; t++)
    {
        cudaEventRecord(ev[5], s);
        rc = h->Bin<float, float>(h->pos32.p, h->rad32.p, h->sRad32.p, s, ev);
        if (rc == HAL_CUDA_OK)
        {
            rc = h->Force<float, float>(h->sRad32.p, interactionRad, springConstant, wrapX != 0, wrapY != 0,
                                        h->vel32.p, s);
        }
        cudaEventRecord(ev[4], s);
        if (rc == HAL_CUDA_OK)
        {
            rc = CudaStatus(cudaEventSynchronize(ev[4]), "hal_cuda_agents_profile");
        }
        if (rc != HAL_CUDA_OK)
        {
            break;
        }
        float t0 = 0, t1 = 0, t2 = 0, t3 = 0, t4 = 0, tall = 0;
        cudaEventElapsedTime(&t0, ev[5], ev[0]);
        cudaEventElapsedTime(&t1, ev[0], ev[1]);
        cudaEventElapsedTime(&t2, ev[1], ev[2]);
        cudaEventElapsedTime(&t3, ev[2], ev[3]);
        cudaEventElapsedTime(&t4, ev[3], ev[4]);
        cudaEventElapsedTime(&tall, ev[5], ev[4]);
        acc[0] += t0;
        acc[1] += t1;
        acc[2] += t2;
        acc[3] += t3;
        acc[4] += t4;
        acc[5] += tall;
    }
    for (auto &e : ev)
    {
        cudaEventDestroy(e);
    }
    HAL_TRY(rc);
    for (int q = 0; q < 6; q++)
    {
        ms[q] = static_cast<float>(acc[q] / iters);
    }
    return HAL_CUDA_OK;
}

// ---------------------------------------------------------------------------
// Agent forces without allocation.
//
// Some callers cannot call cudaMalloc: a host framework that reserves its
// device memory in its own pool at start-up and forbids cudaMalloc/cudaFree in
// its step loop (both synchronise the whole device and stall the framework's
// other streams), or a plugin whose host budgets device memory and hands it
// only pointers to inputs and outputs.  For them this entry point runs the same
// binning and force kernels as hal_cuda_agents_dispatch with every piece of
// scratch taken from one file-scope device array of fixed size, so it needs no
// handle and allocates nothing.  The caller passes device pointers to the
// positions, radii and velocity deltas.
//
// The array is a static __device__ variable: every GPU that loads this library
// holds it (HAL_CUDA_NOALLOC_SCRATCH_BYTES) until the process exits.  In host
// code its name is only a host-side stand-in, so its device address is looked
// up once per device with cudaGetSymbolAddress, with that device current,
// on the first call made on that device.  All calls share it and it keeps the
// last call's contents; the cell counts, the only part that must start at
// zero, are cleared on the caller's stream at the start of each call.
// ---------------------------------------------------------------------------
#include <cuda.h>
#include <mutex>

namespace
{
    constexpr size_t kNoAllocMaxAgents = HAL_CUDA_NOALLOC_MAX_AGENTS;
    constexpr size_t kNoAllocMaxCells = HAL_CUDA_NOALLOC_MAX_CELLS;
    constexpr size_t kNoAllocMaxTiles = (kNoAllocMaxCells + halcuda::kScanTile - 1) / halcuda::kScanTile;

    constexpr size_t Round256(size_t b)
    {
        return (b + 255) / 256 * 256;
    }

    // Byte offsets of the regions of the scratch array (each 256-byte aligned).
    constexpr size_t kOffPosF = 0;
    constexpr size_t kOffSPos = kOffPosF + Round256(kNoAllocMaxAgents * sizeof(float2));
    constexpr size_t kOffSRad = kOffSPos + Round256(kNoAllocMaxAgents * sizeof(float2));
    constexpr size_t kOffCellOf = kOffSRad + Round256(kNoAllocMaxAgents * sizeof(float));
    constexpr size_t kOffArrival = kOffCellOf + Round256(kNoAllocMaxAgents * sizeof(int32_t));
    constexpr size_t kOffBucketTmp = kOffArrival + Round256(kNoAllocMaxAgents * sizeof(int32_t));
    constexpr size_t kOffBucket = kOffBucketTmp + Round256(kNoAllocMaxAgents * sizeof(int32_t));
    constexpr size_t kOffCounts = kOffBucket + Round256(kNoAllocMaxAgents * sizeof(int32_t));
    constexpr size_t kOffOffsets = kOffCounts + Round256(kNoAllocMaxCells * sizeof(int32_t));
    constexpr size_t kOffTileSums = kOffOffsets + Round256((kNoAllocMaxCells + 1) * sizeof(int32_t));
    constexpr size_t kNoAllocBytes = kOffTileSums + Round256(kNoAllocMaxTiles * sizeof(int32_t));
    static_assert(kNoAllocBytes <= HAL_CUDA_NOALLOC_SCRATCH_BYTES, "no-alloc scratch regions exceed the stated size");

    static __device__ __align__(256) unsigned char gNoAllocScratch[HAL_CUDA_NOALLOC_SCRATCH_BYTES];

    constexpr int kNoAllocMaxDevices = 64;
    std::mutex gNoAllocMutex;
    unsigned char *gNoAllocAddr[kNoAllocMaxDevices] = {};
    // The CUDA context each cached address belongs to (its unique id,
    // cuCtxGetId).  After cudaDeviceReset the runtime creates a new primary
    // context, loads this module again and the array may sit elsewhere; a
    // changed id makes the next call look the address up again.
    unsigned long long gNoAllocCtx[kNoAllocMaxDevices] = {};

    using CtxGetCurrentFn = CUresult (*)(CUcontext *);
    using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long *);

    // Id of the calling thread's current context (0 when it cannot be read).
    unsigned long long CurrentContextId()
    {
        static CtxGetCurrentFn s_getCurrent = nullptr;
        static CtxGetIdFn s_getId = nullptr;
        static bool s_resolved = false;
        if (!s_resolved)
        {
            void *fn = nullptr;
            cudaDriverEntryPointQueryResult q;
            if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &fn, 12000, cudaEnableDefault, &q) ==
                    cudaSuccess && q == cudaDriverEntryPointSuccess)
            {
                s_getCurrent = reinterpret_cast<CtxGetCurrentFn>(fn);
            }
            fn = nullptr;
            if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &fn, 12000, cudaEnableDefault, &q) == cudaSuccess &&
                q == cudaDriverEntryPointSuccess)
            {
                s_getId = reinterpret_cast<CtxGetIdFn>(fn);
            }
            s_resolved = true;
        }
        CUcontext ctx = nullptr;
        unsigned long long id = 0;
        if (s_getCurrent == nullptr || s_getId == nullptr || s_getCurrent(&ctx) != CUDA_SUCCESS || ctx == nullptr ||
            s_getId(ctx, &id) != CUDA_SUCCESS)
        {
            return 0;
        }
        return id;
    }

    // Device address of gNoAllocScratch on the current device `dev`; looked
    // up on the first call on that device, and again whenever the device's
    // context has changed since (a cudaDeviceReset in between).
    int NoAllocScratch(int dev, unsigned char **out)
    {
        if (dev < 0 || dev >= kNoAllocMaxDevices)
        {
            halcuda::SetError("hal_cuda_agents_forces_noalloc: device ordinal %d not supported", dev);
            return HAL_CUDA_EDEVICE;
        }
        std::lock_guard<std::mutex> lock(gNoAllocMutex);
        // an id of 0 (no context yet, or the driver cannot say) never
        // matches, so the address is looked up then
        void *p = nullptr;
        const unsigned long long ctx = CurrentContextId();
        if (gNoAllocAddr[dev] == nullptr || ctx == 0 || ctx != gNoAllocCtx[dev])
        {
            HAL_TRY(halcuda::CudaStatus(cudaGetSymbolAddress(&p, gNoAllocScratch),
                                        "cudaGetSymbolAddress(no-alloc scratch)"));
            gNoAllocAddr[dev] = static_cast<unsigned char *>(p);
            gNoAllocCtx[dev] = CurrentContextId();
        }
        *out = gNoAllocAddr[dev];
        return HAL_CUDA_OK;
    }

    // The pointer must be device (or managed) memory reachable from `dev`.
    bool OnDevice(const void *p, int dev)
    {
        cudaPointerAttributes a{};
        if (cudaPointerGetAttributes(&a, p) != cudaSuccess)
        {
            cudaGetLastError();
            return false;
        }
        return a.type == cudaMemoryTypeManaged || (a.type == cudaMemoryTypeDevice && a.device == dev);
    }
}

extern "C" int hal_cuda_agents_forces_noalloc(const float *positions, const float *radii, int32_t n,
                                              float *velocityDeltas, double interactionRad, double springConstant,
                                              int32_t xDim, int32_t yDim, int32_t wrapX, int32_t wrapY, void *stream)
{
    HAL_REQUIRE(xDim > 0 && yDim > 0, "hal_cuda_agents_forces_noalloc: dimensions must be positive");
    HAL_REQUIRE(static_cast<int64_t>(xDim) * yDim <= static_cast<int64_t>(kNoAllocMaxCells),
                "hal_cuda_agents_forces_noalloc: grid %d x %d has more than %d cells, the no-alloc limit",
                xDim, yDim, HAL_CUDA_NOALLOC_MAX_CELLS);
    HAL_REQUIRE(n >= 0 && static_cast<size_t>(n) <= kNoAllocMaxAgents,
                "hal_cuda_agents_forces_noalloc: agent count %d outside [0, %d], the no-alloc limit", n,
                HAL_CUDA_NOALLOC_MAX_AGENTS);
    HAL_REQUIRE(RadiusOk(interactionRad), "hal_cuda_agents_forces_noalloc: interactionRad %g outside [0, %g]",
                interactionRad, kMaxInteractionRad);
    HAL_REQUIRE(n == 0 || (positions != nullptr && radii != nullptr && velocityDeltas != nullptr),
                "hal_cuda_agents_forces_noalloc: NULL array");
    using namespace halcuda;
    int dev = 0;
    HAL_TRY(CudaStatus(cudaGetDevice(&dev), "cudaGetDevice"));
    HAL_REQUIRE(n == 0 || (OnDevice(positions, dev) && OnDevice(radii, dev) && OnDevice(velocityDeltas, dev)),
                "hal_cuda_agents_forces_noalloc: positions, radii and velocityDeltas must be device memory of "
                "the current device %d", dev);
    unsigned char *base = nullptr;
    HAL_TRY(NoAllocScratch(dev, &base));
    if (n == 0)
    {
        return HAL_CUDA_OK;
    }
    float2 *posF = reinterpret_cast<float2 *>(base + kOffPosF);
    float2 *sPos = reinterpret_cast<float2 *>(base + kOffSPos);
    float *sRad = reinterpret_cast<float *>(base + kOffSRad);
    int32_t *cellOf = reinterpret_cast<int32_t *>(base + kOffCellOf);
    int32_t *arrival = reinterpret_cast<int32_t *>(base + kOffArrival);
    int32_t *bucketTmp = reinterpret_cast<int32_t *>(base + kOffBucketTmp);
    int32_t *bucket = reinterpret_cast<int32_t *>(base + kOffBucket);
    int32_t *counts = reinterpret_cast<int32_t *>(base + kOffCounts);
    int32_t *offsets = reinterpret_cast<int32_t *>(base + kOffOffsets);
    int32_t *tileSums = reinterpret_cast<int32_t *>(base + kOffTileSums);

    const int64_t C = static_cast<int64_t>(xDim) * yDim;
    const unsigned nTiles = static_cast<unsigned>((C + kScanTile - 1) / kScanTile);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    HAL_TRY(CudaStatus(cudaMemsetAsync(counts, 0, static_cast<size_t>(C) * sizeof(int32_t), s),
                       "cudaMemsetAsync(no-alloc counts)"));
    const int T = 256;
    const unsigned ablocks = static_cast<unsigned>((n + T - 1) / T);
    BinCount<float><<<ablocks, T, 0, s>>>(positions, n, xDim, yDim, posF, cellOf, arrival, counts);
    ScanReduce<<<nTiles, kScanThreads, 0, s>>>(counts, C, tileSums);
    ScanTiles<<<1, kScanThreads, 0, s>>>(tileSums, static_cast<int32_t>(nTiles));
    ScanApply<false><<<nTiles, kScanThreads, 0, s>>>(counts, C, tileSums, offsets, n);
    Scatter<<<ablocks, T, 0, s>>>(cellOf, arrival, offsets, n, bucketTmp, nullptr, 0);
    Stabilize<float, float><<<ablocks, T, 0, s>>>(cellOf, offsets, bucketTmp, posF, radii, n, bucket, sPos, sRad);
    const int TF = 128;
    LawParams<float> lp;
    lp.scale = static_cast<float>(springConstant);
    lp.exponent = 1.0f;
    Forces<float, float><<<static_cast<unsigned>((n + TF - 1) / TF), TF, 0, s>>>(
        bucket, offsets, sPos, sRad, n, interactionRad, static_cast<float>(interactionRad), lp, xDim, yDim,
        wrapX != 0, wrapY != 0, velocityDeltas, static_cast<float *>(nullptr), static_cast<const float *>(nullptr));
    CountLaunch(7);
    return LaunchStatus("hal_cuda_agents_forces_noalloc");
}

namespace halcuda
{
    int32_t AgentScanTiles(int64_t cells)
    {
        return static_cast<int32_t>((cells + kScanTile - 1) / kScanTile);
    }

    int LaunchCountWells(const AgentWellsArgs &a, cudaStream_t s)
    {
        const int T = 256;
        LaunchChained(BinCountWells, static_cast<unsigned>((a.n + T - 1) / T), T, s, a.pos, a.wellOf, a.wells, a.n,
                      a.cellOf, a.arrival, a.counts);
        LaunchChained(ScanReduce, static_cast<unsigned>(AgentScanTiles(a.cells)), kScanThreads, s, a.counts, a.cells,
                      a.tileSums);
        CountLaunch(2);
        return LaunchStatus("agent wells count");
    }

    int LaunchBinWells(const AgentWellsArgs &a, cudaStream_t s)
    {
        if (a.n <= 0)
        {
            return HAL_CUDA_OK;
        }
        if (!a.counted)
        {
            HAL_TRY(LaunchCountWells(a, s));
        }
        const int T = 256;
        const unsigned ablocks = static_cast<unsigned>((a.n + T - 1) / T);
        const int32_t nTiles = AgentScanTiles(a.cells);
        // the scan clears the counts it has read
        if (nTiles <= kScanSumTiles)
        {
            LaunchChained(ScanApplySum, nTiles, kScanThreads, s, a.counts, a.cells, a.tileSums, a.offsets, a.n);
        }
        else
        {
            LaunchChained(ScanTiles, 1u, kScanThreads, s, a.tileSums, nTiles);
            LaunchChained(ScanApply<true>, nTiles, kScanThreads, s, a.counts, a.cells, a.tileSums, a.offsets, a.n);
            CountLaunch();
        }
        LaunchChained(Scatter, ablocks, T, s, a.cellOf, a.arrival, a.offsets, a.n, a.bucketTmp, a.tileSums, nTiles);
        LaunchChained(StabilizeWells, ablocks, T, s, a.offsets, a.bucketTmp, reinterpret_cast<const float2 *>(a.pos),
                      a.rad, a.wellOf, a.wells, a.n, a.bucket, a.sPos, a.sRad, a.sCell);
        CountLaunch(3);
        return LaunchStatus("agent wells bins");
    }

    int LaunchForceWells(const AgentWellsArgs &a, cudaStream_t s)
    {
        if (a.n <= 0)
        {
            return HAL_CUDA_OK;
        }
        const int TF = (a.forceThreads == 64 || a.forceThreads == 256) ? a.forceThreads : 128;
        const unsigned fblocks = static_cast<unsigned>((a.n + TF - 1) / TF);
        if (a.velState != nullptr)
        {
            LaunchChained(ForcesWellsMove, fblocks, TF, s, a.bucket, a.offsets, a.sPos, a.sRad, a.sCell, a.wellOf,
                          a.wells, a.n, a.interactionRad, IntegerRadius(a.interactionRad), a.R, a.k, a.friction,
                          a.maxVel, a.vel, a.posOut, a.velState, a.cellOf, a.arrival, a.counts, a.tileSums);
        }
        else
        {
            LaunchChained(ForcesWells, fblocks, TF, s, a.bucket, a.offsets, a.sPos, a.sRad, a.sCell, a.wellOf,
                          a.wells, a.n, a.interactionRad, IntegerRadius(a.interactionRad), a.R, a.k, a.vel);
        }
        CountLaunch();
        return LaunchStatus("agent wells");
    }

    int LaunchAgentWells(const AgentWellsArgs &a, cudaStream_t s)
    {
        HAL_TRY(LaunchBinWells(a, s));
        return LaunchForceWells(a, s);
    }
}
