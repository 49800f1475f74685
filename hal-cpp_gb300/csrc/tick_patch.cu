// tick_patch.cu -- several explicit ticks per launch, the field in registers.
//
// What bounds one tick per launch (TickKernel, diffusion.cu): a tick does about
// ten FP32 operations per cell and moves 8 bytes, so a large field is bound by
// the L2 or HBM (6.5 us per 2048^2 tick, 26 us per 4096^2 tick) and a small one
// by its launches and load latency (5.2 us per 256^2 tick with a Dirichlet edge
// and point sources).  Here a warp loads a patch of 32 * V columns x R rows once,
// keeps it in registers for up to HK ticks and stores the part that no patch
// edge has reached: R - 2 HK rows, and HK columns less on either side.  A lane
// owns V columns of every row, so the neighbours in x are its own registers and
// those in y one shuffle away; no shared memory, and no warp waits for another.
// Patches overlap by the halo, which costs redundant work (1.7x to 2.5x of the
// cells at the shapes below) instead of memory passes.
//
// Rows i and i + R/2 of a column share a 64-bit register pair, so that the FP32
// arithmetic is packed (f32x2): the FP32 pipe does the same work in half the
// instructions, which leaves issue slots for the shuffles.  The differences are
// shared between the two cells they separate: f[x+1] - f[x] is one cell's lower
// difference and, negated exactly, the next one's upper.  So every cell's result
// is TickKernel's, bit for bit.
//
// Shapes (TickPatchShapeFor), measured on GB300, us per tick without / with a
// dense source, in a graph:
//
//   V  R HK | 256^2        512^2        1024^2       2048^2       4096^2
//   1 40  8 | 0.59 / 0.58  0.77 / 0.85  1.58 / 1.74  5.2 / 5.8    19.7 / 22.8
//   2 24  4 | 0.76 / 0.84  1.04 / 1.22  1.04 / 1.19  2.88 / 3.36  11.1 / 14.2
//   2 32  6 | 0.70 / 0.83  0.94 / 1.10  1.06 / 1.21  3.01 / 3.44  11.1 / 13.3
//   2 32  8 | 0.63 / 0.74  0.90 / 1.03  1.26 / 1.45  3.66 / 4.20  13.4 / 15.3
//
// Small fields take the narrow patches, whose many warps and long runs of ticks
// hide the launch and load latency; large ones the wide patches, which recompute
// less.  The two cross near 2^19 cells.  The large shape spends half of its time
// on the FP32 pipe and the rest on the loads and stores around the ticks.
#include "common.cuh"
#include "tick_params.h"

#include <cstdint>

namespace halcuda
{
    namespace
    {
        constexpr int kPatchWarps = 4;  // warps per CTA (independent of one another)

        // Two FP32 values in one 64-bit register pair, and the packed FP32
        // arithmetic of sm_100 and later: each half rounds as the scalar
        // operation does.
        using Pair = unsigned long long;

        __device__ __forceinline__ Pair Pack(float lo, float hi)
        {
            Pair r;
            asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
            return r;
        }

        __device__ __forceinline__ void Unpack(Pair a, float &lo, float &hi)
        {
            asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a));
        }

        __device__ __forceinline__ Pair Fma2(Pair a, Pair b, Pair c)
        {
            Pair r;
            asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
            return r;
        }

        __device__ __forceinline__ Pair Add2(Pair a, Pair b)
        {
            Pair r;
            asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
            return r;
        }

        __device__ __forceinline__ Pair Mul2(Pair a, Pair b)
        {
            Pair r;
            asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
            return r;
        }

        // a - b (the product by -1 is exact)
        __device__ __forceinline__ Pair Sub2(Pair a, Pair b, Pair minusOne)
        {
            return Fma2(b, minusOne, a);
        }

        // V values of a lane at q (consecutive columns, 4 * V-byte aligned
        // when VEC), or one by one at q[col[k]].
        // FIELD: what the launch before may have written, through the L2 (the
        // read-only path is for data that no kernel in flight writes).
        template <int V, bool VEC, bool FIELD>
        __device__ __forceinline__ void LoadCells(const float *__restrict__ q, const int32_t (&col)[V], float (&v)[V])
        {
            if constexpr (VEC && V == 2)
            {
                const float2 *at = reinterpret_cast<const float2 *>(q + col[0]);
                const float2 t = FIELD ? __ldcg(at) : __ldg(at);
                v[0] = t.x;
                v[1] = t.y;
            }
            else
            {
#pragma unroll
                for (int k = 0; k < V; k++)
                {
                    v[k] = FIELD ? __ldcg(q + col[k]) : __ldg(q + col[k]);
                }
            }
        }

        template <int V, int R, int HK, int SRC, bool ADV, bool VEC, bool EDGE>
        __device__ __forceinline__ void Patch(const TickPatchParams &p, const float *__restrict__ sA,
                                              const float *__restrict__ sB, const int32_t x0, const int32_t yBeg,
                                              const bool topEdge, const bool botEdge, const bool leftEdge,
                                              const bool rightEdge)
        {
            static_assert(R % 2 == 0 && R / 2 > HK, "the seam of the two halves lies among the stored rows");
            constexpr int N = R / 2;
            constexpr int HL = (HK + V - 1) / V;  // lanes of halo on either side
            const int32_t lane = static_cast<int32_t>(threadIdx.x & 31u);
            const int32_t y0 = yBeg + lane * V;
            const Pair m1 = Pack(-1.0f, -1.0f);

            // columns that the lane's cells are read from
            int32_t col[V];
            // off a closed grid: the cells keep their values
            const bool held = EDGE && ((leftEdge && lane < HL) || (rightEdge && lane >= 32 - HL));
#pragma unroll
            for (int k = 0; k < V; k++)
            {
                int32_t c = y0 + k;
                if constexpr (EDGE)
                {
                    c += c < 0 ? p.yDim : 0;
                    c -= c >= p.yDim ? p.yDim : 0;
                }
                col[k] = c;
            }
            // grid row of patch row r
            auto gridRow = [&](int r)
            {
                int32_t x = x0 - HK + r;
                if constexpr (EDGE)
                {
                    x += x < 0 ? p.xDim : 0;
                    x -= x >= p.xDim ? p.xDim : 0;
                }
                return x;
            };
            auto rowOf = [&](const float *__restrict__ a, int r) { return a + static_cast<int64_t>(gridRow(r)) * p.yDim; };

            Pair f[N][V];
            {
                float lo[N][V], hi[N][V];
#pragma unroll
                for (int i = 0; i < N; i++)
                {
                    LoadCells<V, VEC, true>(rowOf(p.f, i), col, lo[i]);
                    LoadCells<V, VEC, true>(rowOf(p.f, i + N), col, hi[i]);
                }
#pragma unroll
                for (int i = 0; i < N; i++)
                {
#pragma unroll
                    for (int k = 0; k < V; k++)
                    {
                        f[i][k] = Pack(lo[i][k], hi[i][k]);
                    }
                }
            }
            // the first source stays in registers, the second (point sources
            // beside a dense one) is read each tick
            const float on = held ? 0.0f : 1.0f;
            Pair sa[SRC > 0 ? N : 1][V];
            if constexpr (SRC > 0)
            {
#pragma unroll
                for (int i = 0; i < N; i++)
                {
                    float lo[V], hi[V];
                    LoadCells<V, VEC, false>(rowOf(sA, i), col, lo);
                    LoadCells<V, VEC, false>(rowOf(sA, i + N), col, hi);
#pragma unroll
                    for (int k = 0; k < V; k++)
                    {
                        sa[i][k] = Pack(EDGE ? lo[k] * on : lo[k], EDGE ? hi[k] * on : hi[k]);
                    }
                }
            }
            if constexpr (EDGE)
            {
                if (held)
                {
                    // the boundary values beside the first or last column (or
                    // zeros, whose differences have weight 0)
                    const float *g = lane < HL ? p.ghost.ylo : p.ghost.yhi;
                    const int kg = lane < HL ? V - 1 : 0;
#pragma unroll
                    for (int i = 0; i < N; i++)
                    {
                        const float lo = g != nullptr ? __ldg(g + gridRow(i)) : 0.0f;
                        const float hi = g != nullptr ? __ldg(g + gridRow(i + N)) : 0.0f;
#pragma unroll
                        for (int k = 0; k < V; k++)
                        {
                            f[i][k] = k == kg ? Pack(lo, hi) : 0ull;
                        }
                    }
                }
            }
            // the rows just beyond a closed x edge hold the boundary values
            // (or zeros, whose differences have weight 0)
            float gTop[V], gBot[V];
#pragma unroll
            for (int k = 0; k < V; k++)
            {
                gTop[k] = (topEdge && p.ghost.xlo != nullptr) ? __ldg(p.ghost.xlo + col[k]) : 0.0f;
                gBot[k] = (botEdge && p.ghost.xlo != nullptr) ? __ldg(p.ghost.xhi + col[k]) : 0.0f;
            }
            constexpr int iTop = HK - 1;       // row -1: lower half of pair iTop
            constexpr int iBot = R - HK - N;   // row xDim: upper half of pair iBot
            auto hold = [&](int i)
            {
                if (i == iTop && topEdge)
                {
#pragma unroll
                    for (int k = 0; k < V; k++)
                    {
                        float lo, hi;
                        Unpack(f[i][k], lo, hi);
                        f[i][k] = Pack(gTop[k], hi);
                    }
                }
                if (i == iBot && botEdge)
                {
#pragma unroll
                    for (int k = 0; k < V; k++)
                    {
                        float lo, hi;
                        Unpack(f[i][k], lo, hi);
                        f[i][k] = Pack(lo, gBot[k]);
                    }
                }
            };
            if constexpr (EDGE)
            {
                hold(iTop);
                hold(iBot);
            }
            const float edge = p.ghost.xlo != nullptr ? 2.0f : 0.0f;
            const Pair wTop = Pack(topEdge ? edge : 1.0f, 1.0f);
            const Pair wBot = Pack(1.0f, botEdge ? edge : 1.0f);
            const float wlf = (EDGE && leftEdge && lane == HL) ? edge : 1.0f;
            const float wrf = (EDGE && rightEdge && lane == 31 - HL) ? edge : 1.0f;
            const Pair wl = Pack(wlf, wlf), wr = Pack(wrf, wrf);
            // a held cell's weights are 0: its change is too
            const Pair r2 = Pack(p.r * on, p.r * on), nd = Pack(p.negDecay * on, p.negDecay * on);
            const Pair kDn = Pack(p.kDn * on, p.kDn * on), kUpN = Pack(-p.kUp * on, -p.kUp * on);
            const Pair kYp = Pack(p.kYp * on, p.kYp * on), kYmN = Pack(-p.kYm * on, -p.kYm * on);

#pragma unroll 1
            for (int t = 0; t < p.ticks; t++)
            {
                // differences across the seam between the halves
                Pair up[V], seam[V];
#pragma unroll
                for (int k = 0; k < V; k++)
                {
                    float a, b, c, d;
                    Unpack(f[0][k], a, b);
                    Unpack(f[N - 1][k], c, d);
                    const float s = b - c;
                    up[k] = Pack(0.0f, s);
                    seam[k] = Pack(s, 0.0f);
                }
#pragma unroll
                for (int i = 0; i < N; i++)
                {
                    Pair dn[V], e[V + 1];
#pragma unroll
                    for (int k = 0; k < V; k++)
                    {
                        dn[k] = (i < N - 1) ? Sub2(f[i + 1 < N ? i + 1 : i][k], f[i][k], m1) : seam[k];
                        if (EDGE && i == iTop)
                        {
                            dn[k] = Mul2(dn[k], wTop);
                        }
                        if (EDGE && i == iBot - 1)
                        {
                            dn[k] = Mul2(dn[k], wBot);
                        }
                    }
                    {
                        float a, b, c, d;
                        Unpack(f[i][V - 1], a, b);
                        Unpack(f[i][0], c, d);
                        const Pair left = Pack(__shfl_up_sync(0xffffffffu, a, 1), __shfl_up_sync(0xffffffffu, b, 1));
                        const Pair right = Pack(__shfl_down_sync(0xffffffffu, c, 1), __shfl_down_sync(0xffffffffu, d, 1));
                        e[0] = Sub2(f[i][0], left, m1);
                        e[V] = Sub2(right, f[i][V - 1], m1);
                        if constexpr (EDGE)
                        {
                            e[0] = Mul2(e[0], wl);
                            e[V] = Mul2(e[V], wr);
                        }
                    }
#pragma unroll
                    for (int k = 1; k < V; k++)
                    {
                        e[k] = Sub2(f[i][k], f[i][k - 1], m1);
                    }
                    float bLo[V], bHi[V];
                    if constexpr (SRC > 1)
                    {
                        LoadCells<V, VEC, false>(rowOf(sB, i), col, bLo);
                        LoadCells<V, VEC, false>(rowOf(sB, i + N), col, bHi);
                    }
#pragma unroll
                    for (int k = 0; k < V; k++)
                    {
                        Pair d;
                        if constexpr (ADV)
                        {
                            Pair s = Mul2(dn[k], kDn);
                            s = Fma2(up[k], kUpN, s);
                            s = Fma2(e[k + 1], kYp, s);
                            s = Fma2(e[k], kYmN, s);
                            d = Fma2(f[i][k], nd, s);
                        }
                        else
                        {
                            Pair s = Sub2(dn[k], up[k], m1);
                            s = Add2(e[k + 1], s);
                            s = Sub2(s, e[k], m1);
                            d = Mul2(s, r2);
                            d = Fma2(f[i][k], nd, d);
                        }
                        if constexpr (SRC > 0)
                        {
                            d = Add2(d, sa[i][k]);
                        }
                        if constexpr (SRC > 1)
                        {
                            d = Add2(d, Pack(EDGE ? bLo[k] * on : bLo[k], EDGE ? bHi[k] * on : bHi[k]));
                        }
                        up[k] = dn[k];
                        f[i][k] = Add2(f[i][k], d);
                    }
                    if constexpr (EDGE)
                    {
                        hold(i);
                    }
                }
            }

            if (lane < HL || lane >= 32 - HL)
            {
                return;
            }
            auto store = [&](int r, const float (&v)[V])
            {
                if (r < HK || r >= R - HK)
                {
                    return;
                }
                float *q = p.out + static_cast<int64_t>(x0 - HK + r) * p.yDim + y0;
                if constexpr (VEC && V == 2)
                {
                    *reinterpret_cast<float2 *>(q) = make_float2(v[0], v[1]);
                }
                else
                {
#pragma unroll
                    for (int k = 0; k < V; k++)
                    {
                        q[k] = v[k];
                    }
                }
            };
#pragma unroll
            for (int i = 0; i < N; i++)
            {
                float lo[V], hi[V];
#pragma unroll
                for (int k = 0; k < V; k++)
                {
                    Unpack(f[i][k], lo[k], hi[k]);
                }
                store(i, lo);
                store(i + N, hi);
            }
        }

        // The part of a patch that is stored.
        template <int V, int R, int HK>
        struct Shape
        {
            static constexpr int kHaloCols = (HK + V - 1) / V * V;
            static constexpr int kCols = 32 * V - 2 * kHaloCols;
            static constexpr int kRows = R - 2 * HK;
        };

        template <int V, int R, int HK, int SRC, bool ADV, bool VEC>
        __global__ void __launch_bounds__(32 * kPatchWarps, V > 1 ? 3 : 1) TickPatch(TickPatchParams p)
        {
            // Chained as TickKernel is: the next launch may be scheduled once
            // every CTA of this one has started, and waits for its completion.
            asm volatile("griddepcontrol.launch_dependents;");
            asm volatile("griddepcontrol.wait;" ::: "memory");
            using S = Shape<V, R, HK>;
            const int32_t w = static_cast<int32_t>(blockIdx.x) * kPatchWarps + static_cast<int32_t>(threadIdx.x >> 5);
            if (w >= p.windows * p.strips)
            {
                return;
            }
            const int32_t win = w % p.windows, strip = w / p.windows;
            const int32_t yIn = TickPatchStart(win, p.windows, S::kCols, S::kHaloCols, p.yDim);
            const int32_t x0 = TickPatchStart(strip, p.strips, S::kRows, HK, p.xDim);
            const int32_t yBeg = yIn - S::kHaloCols;
            // point sources: only the patches that hold one read them
            const float *pts = (SRC > 0 && p.pts != nullptr && __ldg(p.flags + w) != 0) ? p.pts : nullptr;
            const float *sA = (SRC == 1 && p.src == nullptr) ? pts : p.src;
            const bool interior = yBeg >= 0 && yBeg + 32 * V <= p.yDim && x0 >= HK && x0 - HK + R <= p.xDim;
            const bool top = !p.wrapX && x0 == 0, bot = !p.wrapX && x0 + S::kRows == p.xDim;
            const bool left = !p.wrapY && yIn == 0, right = !p.wrapY && yIn + S::kCols == p.yDim;
            if (SRC == 2 && pts != nullptr)
            {
                Patch<V, R, HK, 2, ADV, VEC, true>(p, sA, pts, x0, yBeg, top, bot, left, right);
            }
            else if (SRC > 0 && sA != nullptr)
            {
                if (interior)
                {
                    Patch<V, R, HK, SRC == 0 ? 0 : 1, ADV, VEC, false>(p, sA, nullptr, x0, yBeg, false, false, false, false);
                }
                else
                {
                    Patch<V, R, HK, SRC == 0 ? 0 : 1, ADV, VEC, true>(p, sA, nullptr, x0, yBeg, top, bot, left, right);
                }
            }
            else if (SRC < 2)
            {
                if (interior)
                {
                    Patch<V, R, HK, 0, ADV, VEC, false>(p, nullptr, nullptr, x0, yBeg, false, false, false, false);
                }
                else
                {
                    Patch<V, R, HK, 0, ADV, VEC, true>(p, nullptr, nullptr, x0, yBeg, top, bot, left, right);
                }
            }
        }

        template <int V, int R, int HK, bool VEC>
        const void *KernelOf(int src, bool adv)
        {
            switch (2 * src + (adv ? 1 : 0))
            {
            case 0:
                return reinterpret_cast<const void *>(TickPatch<V, R, HK, 0, false, VEC>);
            case 1:
                return reinterpret_cast<const void *>(TickPatch<V, R, HK, 0, true, VEC>);
            case 2:
                return reinterpret_cast<const void *>(TickPatch<V, R, HK, 1, false, VEC>);
            case 3:
                return reinterpret_cast<const void *>(TickPatch<V, R, HK, 1, true, VEC>);
            case 4:
                return reinterpret_cast<const void *>(TickPatch<V, R, HK, 2, false, VEC>);
            default:
                return reinterpret_cast<const void *>(TickPatch<V, R, HK, 2, true, VEC>);
            }
        }

        constexpr int kSmallRows = 40, kSmallHalo = 8;  // V = 1
        constexpr int kLargeRows = 24, kLargeHalo = 4;  // V = 2
        // Up to this many cells the narrow patches are the faster ones (the
        // table above).
        constexpr int64_t kSmallCells = int64_t(1) << 19;

        TickPatchShape MakeShape(int vec, int rows, int halo, int32_t xDim, int32_t yDim)
        {
            TickPatchShape s;
            s.vec = vec;
            s.patchRows = rows;
            s.halo = halo;
            s.haloCols = (halo + vec - 1) / vec * vec;
            s.cols = 32 * vec - 2 * s.haloCols;
            s.rows = rows - 2 * halo;
            // a whole patch must fit the grid: then no window but the first
            // and the last reaches beyond an edge, and a wrapped index needs
            // one correction
            if (xDim >= rows && yDim >= 32 * vec)
            {
                s.windows = (yDim + s.cols - 1) / s.cols;
                s.strips = (xDim + s.rows - 1) / s.rows;
            }
            return s;
        }
    }

    TickPatchShape TickPatchShapeFor(int32_t xDim, int32_t yDim)
    {
        const TickPatchShape small = MakeShape(1, kSmallRows, kSmallHalo, xDim, yDim);
        const TickPatchShape large = MakeShape(2, kLargeRows, kLargeHalo, xDim, yDim);
        const bool preferSmall = static_cast<int64_t>(xDim) * yDim <= kSmallCells;
        if (preferSmall)
        {
            return small.windows > 0 ? small : large;
        }
        return large.windows > 0 ? large : small;
    }

    int LaunchTickPatch(const TickPatchShape &shape, TickPatchParams &p, bool adv, cudaStream_t s)
    {
        p.windows = shape.windows;
        p.strips = shape.strips;
        const int src = (p.src != nullptr && p.pts != nullptr) ? 2 : ((p.src != nullptr || p.pts != nullptr) ? 1 : 0);
        const void *k = nullptr;
        if (shape.vec == 1)
        {
            k = KernelOf<1, kSmallRows, kSmallHalo, true>(src, adv);
        }
        else if (p.yDim % 2 == 0)
        {
            k = KernelOf<2, kLargeRows, kLargeHalo, true>(src, adv);
        }
        else
        {
            k = KernelOf<2, kLargeRows, kLargeHalo, false>(src, adv);
        }
        const int64_t warps = static_cast<int64_t>(p.windows) * p.strips;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(static_cast<unsigned>((warps + kPatchWarps - 1) / kPatchWarps));
        cfg.blockDim = dim3(32 * kPatchWarps);
        cfg.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        void *args[] = {&p};
        return CudaStatus(cudaLaunchKernelExC(&cfg, k, args), "TickPatch launch");
    }
}
