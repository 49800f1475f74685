// adjoint.cu -- variable-rate ADI (a rate D per cell) and the gradient of a
// field loss by reverse-mode differentiation, with checkpoints.
//
// The reference has no variable-rate ADI and no gradient code.  The step is
// defined from HAL's variable-rate explicit stencil Internal::Diffusion2(...,
// pDiffRatesX, pDiffRatesY, ...) (src/Pde/PDEequations.cpp:199-230): the
// face between cells j and j+1 of a line carries cell j's rate, a non-wrapped
// edge has no face, and L is the face-weighted Laplacian along a line:
//   w  = (I - Lx/2)^-1 (I + Ly/2) f            x-sweep  (FwdLines<M, false>)
//   v  = (I - Ly/2)^-1 (I + Lx/2) w            y-sweep  (FwdLines<M, true>)
//   f' = f + (((v - f) + f*(-decay)) + src)    PDEGrid2D tick order
// For a constant rate this is Internal::Diffusion2DADI plus the tick.
//
// Gradient of loss = 1/2 |f_T - target|^2.  I - L/2 and I + L/2 are
// symmetric, so with gbar the adjoint of a step's output:
//   b2bar = (I - Ly/2)^-1 gbar;        wbar = (I + Lx/2) b2bar
//   b1bar = (I - Lx/2)^-1 wbar;        fbar = (I + Ly/2) b1bar - decay gbar
//   dsrc += gbar;   ddecay -= <gbar, f>
//   dD[owner of face] += -1/2 (p_j+1 - p_j)(q_j+1 - q_j) for the pairs
//   (b2bar, v) and (b1bar, f) on y-faces, (b2bar, w) and (b1bar, w) on x-faces
// Two kernels per backward step: BwdY applies the previous step's (I + Ly/2)
// and then this step's y-solve (both along y), BwdX the x-stencil and x-solve.
// States are recomputed segment by segment from checkpoints every k steps,
// each segment on a second stream while the one after it is differentiated.
//
// What bounds a step.  A field is 1 MB at 512^2: a step's kernels move a few MB
// through the L2, a microsecond or two, and are bound by latency: the launch,
// the loads, the solve's dependent chain, the stores.  Parallel cyclic
// reduction of every line in shared memory took nine stages of two barriers
// (12 us a forward kernel, 13 to 16 us a backward one).  But the rates do not
// change between the steps of a call, so each line is factored once per call, in FP64
// (Factor), and a step only runs the right-hand side through the factors:
//   - a warp solves one line, a lane M consecutive positions of it in
//     registers: Thomas with the precomputed multipliers (fw, ib, cb) over the
//     lane's first M - 1 positions, the last one being a separator;
//   - the separators' tridiagonal system (one per lane) by cyclic reduction
//     over shuffles with precomputed multipliers (five stages, no division);
//   - x = z - s_left p - s_right q with the precomputed coupling vectors;
//   - a wrapped line is split as T + u v^T (TdmaSolver::TDMAperiodic's form,
//     include/Hal/Pde/TdmaSolver.h:68-120): x = y - (y_0 + bog y_n-1) zf with
//     zf precomputed.
// No barriers but one, for the transposed write-out: a CTA's four lines leave
// through shared memory as 16-byte pieces, in the layout in which the next
// kernel's lines are contiguous.  The kernels are chained by programmatic
// launches; everything that does not come from the kernel just before
// (factors, rates, kept states, accumulators) is loaded before the wait for it.
// A run of steps between checkpoints is replayed from a small CUDA graph.
// Measured at 512^2, 500 steps, zero-flux: forward 3.2 ms (12.3 ms with the
// reductions), gradient with checkpoints every 22 steps 8.5 ms (28.8 ms); its
// error against 64 bits is unchanged (1.5e-6 for dL/dD).  What is left per
// kernel is latency: 1.7 us of it is there on a 64^2 field too.
//
// Layout: "by y" arrays are x * ldY + y (HAL's order), "by x" arrays y * ldX +
// x; ldX and ldY are the sides rounded up to multiples of 4 and the padding
// holds zeros, so every line is read and written in 16-byte pieces.
#include "common.cuh"

#include <algorithm>
#include <cmath>
#include <map>
#include <string>
#include <type_traits>
#include <utility>
#include <vector>

namespace halcuda
{
    namespace
    {
        constexpr int kMaxAdjLine = HAL_CUDA_ADJOINT_MAX_SIDE;
        constexpr int kAdjLines = 4;  // lines (warps) per CTA: a 16-byte piece of the transposed write-out
        constexpr unsigned kAll = 0xffffffffu;

        // Coefficient vectors of a factored line (kCoefZ on wrapped axes only).
        enum AdjCoef : int
        {
            kCoefFw = 0,
            kCoefIb = 1,
            kCoefCb = 2,
            kCoefP = 3,
            kCoefQ = 4,
            kCoefZ = 5
        };

        // Per-lane values of a factored line: the separator stages' multipliers
        // (five below, five above), the reciprocal of its reduced diagonal, the
        // separator row's off-diagonals, and a wrapped line's beta / gamma.
        enum AdjExt : int
        {
            kExtLo = 0,
            kExtHi = 5,
            kExtBinv = 10,
            kExtA = 11,
            kExtC = 12,
            kExtBog = 13,
            kExtCount = 14
        };

        // One axis of the grid: lines of n positions, nl of them.
        struct Axis
        {
            int32_t n, nl;
            int32_t ld;                   // row stride of arrays whose rows are this axis's lines
            int32_t ldT;                  // row stride of the other layout
            int32_t wrap, wrapCross;
            const float *D;               // rates, line by line
            const float *coef;            // [line][coef][M / 4][32 lanes][4]
            const float *ext;             // [line][kExtCount][32]
        };

        __device__ __forceinline__ void WaitForPredecessor()
        {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            // the next kernel may start loading what this one does not write:
            // whatever it reads before its own wait was complete before this
            // kernel's predecessor had finished
            asm volatile("griddepcontrol.launch_dependents;");
        }

        // The lane's M positions of a line (0 beyond the row).  Through the
        // L2: rows written by kernels of the same chain.
        template <int M>
        __device__ __forceinline__ void LoadRow(const float *__restrict__ row, int32_t ld, int lane, float (&v)[M])
        {
#pragma unroll
            for (int q = 0; q < M / 4; q++)
            {
                const int32_t pos = lane * M + 4 * q;
                float4 t = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (pos < ld)
                {
                    t = __ldcg(reinterpret_cast<const float4 *>(row + pos));
                }
                v[4 * q] = t.x;
                v[4 * q + 1] = t.y;
                v[4 * q + 2] = t.z;
                v[4 * q + 3] = t.w;
            }
        }

        template <int M>
        __device__ __forceinline__ void StoreRow(float *__restrict__ row, int32_t ld, int lane, const float (&v)[M])
        {
#pragma unroll
            for (int q = 0; q < M / 4; q++)
            {
                const int32_t pos = lane * M + 4 * q;
                if (pos < ld)
                {
                    *reinterpret_cast<float4 *>(row + pos) =
                        make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                }
            }
        }

        // row += v
        template <int M>
        __device__ __forceinline__ void AddRow(float *__restrict__ row, int32_t ld, int lane, const float (&v)[M])
        {
            float t[M];
            LoadRow<M>(row, ld, lane, t);
#pragma unroll
            for (int i = 0; i < M; i++)
            {
                t[i] += v[i];
            }
            StoreRow<M>(row, ld, lane, t);
        }

        // A line's factors in registers.
        template <int M>
        struct Factors
        {
            float fw[M], ib[M], cb[M], p[M], q[M];
            float lo[5], hi[5], binv, a, c;

            __device__ __forceinline__ void Load(const Axis &ax, int32_t line, int lane)
            {
                const int nc = ax.wrap ? 6 : 5;
                const float4 *base = reinterpret_cast<const float4 *>(ax.coef) +
                                     static_cast<int64_t>(line) * nc * (M / 4) * 32 + lane;
                auto vec = [&](int k, float (&v)[M])
                {
#pragma unroll
                    for (int j = 0; j < M / 4; j++)
                    {
                        const float4 t = __ldg(base + (k * (M / 4) + j) * 32);
                        v[4 * j] = t.x;
                        v[4 * j + 1] = t.y;
                        v[4 * j + 2] = t.z;
                        v[4 * j + 3] = t.w;
                    }
                };
                vec(kCoefFw, fw);
                vec(kCoefIb, ib);
                vec(kCoefCb, cb);
                vec(kCoefP, p);
                vec(kCoefQ, q);
                const float *e = ax.ext + static_cast<int64_t>(line) * kExtCount * 32 + lane;
#pragma unroll
                for (int t = 0; t < 5; t++)
                {
                    lo[t] = __ldg(e + (kExtLo + t) * 32);
                    hi[t] = __ldg(e + (kExtHi + t) * 32);
                }
                binv = __ldg(e + kExtBinv * 32);
                a = __ldg(e + kExtA * 32);
                c = __ldg(e + kExtC * 32);
            }
        };

        // Position n-1's value of a row (its lane's register li).
        template <int M>
        __device__ __forceinline__ float LastOf(const float (&u)[M], int li, int lastLane)
        {
            float v = 0.0f;
#pragma unroll
            for (int i = 0; i < M; i++)
            {
                v = (i == li) ? u[i] : v;
            }
            return __shfl_sync(kAll, v, lastLane);
        }

        // (I - L/2)^-1 d in place, from the line's factors.
        template <int M>
        __device__ __forceinline__ void Solve(const Axis &ax, const Factors<M> &k, int32_t line, int lane, float (&d)[M])
        {
#pragma unroll
            for (int i = 1; i < M - 1; i++)
            {
                d[i] = fmaf(-k.fw[i], d[i - 1], d[i]);
            }
            d[M - 2] *= k.ib[M - 2];
#pragma unroll
            for (int i = M - 3; i >= 0; i--)
            {
                d[i] = fmaf(-k.cb[i], d[i + 1], d[i] * k.ib[i]);
            }
            // the separator's equation with the lane's and the next lane's
            // positions eliminated (a missing neighbour's multiplier is 0)
            const float next = __shfl_down_sync(kAll, d[0], 1);
            float r = fmaf(-k.c, next, fmaf(-k.a, d[M - 2], d[M - 1]));
#pragma unroll
            for (int t = 0; t < 5; t++)
            {
                const float lo = __shfl_up_sync(kAll, r, 1 << t);
                const float hi = __shfl_down_sync(kAll, r, 1 << t);
                r = fmaf(k.lo[t], lo, fmaf(k.hi[t], hi, r));
            }
            const float s = r * k.binv;
            const float sl = __shfl_up_sync(kAll, s, 1);
#pragma unroll
            for (int i = 0; i < M - 1; i++)
            {
                d[i] = fmaf(-sl, k.p[i], fmaf(-s, k.q[i], d[i]));
            }
            d[M - 1] = s;
            if (ax.wrap)
            {
                const float bog = __ldg(ax.ext + (static_cast<int64_t>(line) * kExtCount + kExtBog) * 32 + lane);
                const float y0 = __shfl_sync(kAll, d[0], 0);
                const float yn = LastOf<M>(d, ax.n - 1 - lane * M, (ax.n - 1) / M);
                const float f = fmaf(bog, yn, y0);
                const float4 *z = reinterpret_cast<const float4 *>(ax.coef) +
                                  (static_cast<int64_t>(line) * 6 + kCoefZ) * (M / 4) * 32 + lane;
#pragma unroll
                for (int j = 0; j < M / 4; j++)
                {
                    const float4 t = __ldg(z + j * 32);
                    d[4 * j] = fmaf(-f, t.x, d[4 * j]);
                    d[4 * j + 1] = fmaf(-f, t.y, d[4 * j + 1]);
                    d[4 * j + 2] = fmaf(-f, t.z, d[4 * j + 2]);
                    d[4 * j + 3] = fmaf(-f, t.w, d[4 * j + 3]);
                }
            }
        }

        // The rates of a line as face weights: face (j, j+1) carries e[j], 0
        // at the last position (a wrapped line's last face is its own, eW).
        template <int M>
        __device__ __forceinline__ void MaskLast(float (&e)[M], int li)
        {
#pragma unroll
            for (int i = 0; i < M; i++)
            {
                e[i] = (i == li) ? 0.0f : e[i];
            }
        }

        // out = L u along the line.
        template <int M>
        __device__ __forceinline__ void LapAlong(const Axis &ax, const float (&u)[M], const float (&e)[M], float eW,
                                                 int lane, float (&out)[M])
        {
            float dif[M];
            const float next = __shfl_down_sync(kAll, u[0], 1);
#pragma unroll
            for (int i = 0; i < M; i++)
            {
                dif[i] = (i < M - 1 ? u[i < M - 1 ? i + 1 : i] : next) - u[i];
            }
            float below = __shfl_up_sync(kAll, e[M - 1] * dif[M - 1], 1);
            below = lane == 0 ? 0.0f : below;
#pragma unroll
            for (int i = 0; i < M; i++)
            {
                out[i] = fmaf(e[i], dif[i], i > 0 ? -e[i > 0 ? i - 1 : 0] * dif[i > 0 ? i - 1 : 0] : -below);
            }
            if (ax.wrap)
            {
                const int li = ax.n - 1 - lane * M;
                const float u0 = __shfl_sync(kAll, u[0], 0);
                const float un = LastOf<M>(u, li, (ax.n - 1) / M);
                const float fw = eW * (u0 - un);
                out[0] -= lane == 0 ? fw : 0.0f;
#pragma unroll
                for (int i = 0; i < M; i++)
                {
                    out[i] += (i == li) ? fw : 0.0f;
                }
            }
        }

        // acc[j] += -1/2 (p_j+1 - p_j)(q_j+1 - q_j), the gradient of the face
        // above position j.
        template <int M>
        __device__ __forceinline__ void AddFaceGrad(const Axis &ax, const float (&p)[M], const float (&q)[M], int lane,
                                                    float (&acc)[M])
        {
            const int li = ax.n - 1 - lane * M;
            const float pn = __shfl_down_sync(kAll, p[0], 1), qn = __shfl_down_sync(kAll, q[0], 1);
#pragma unroll
            for (int i = 0; i < M; i++)
            {
                const float dp = (i < M - 1 ? p[i < M - 1 ? i + 1 : i] : pn) - p[i];
                const float dq = (i < M - 1 ? q[i < M - 1 ? i + 1 : i] : qn) - q[i];
                // li and beyond: no face (or the wrapped one below)
                acc[i] = (i < li) ? fmaf(-0.5f * dp, dq, acc[i]) : acc[i];
            }
            if (ax.wrap && ax.n > 1)
            {
                const int last = (ax.n - 1) / M;
                const float p0 = __shfl_sync(kAll, p[0], 0), q0 = __shfl_sync(kAll, q[0], 0);
                const float pl = LastOf<M>(p, li, last), ql = LastOf<M>(q, li, last);
                const float g = -0.5f * (p0 - pl) * (q0 - ql);
#pragma unroll
                for (int i = 0; i < M; i++)
                {
                    acc[i] += (i == li) ? g : 0.0f;
                }
            }
        }

        // The CTA's lines, transposed, into out (row stride ax.ldT): four lines
        // of one position are one 16-byte piece.  Chunks of M positions sit M +
        // 4 floats apart, so that the lanes' 16-byte writes meet no bank
        // conflicts.  Lines beyond the last write the zeros of the padding.
        template <int M>
        __device__ __forceinline__ void StoreTransposed(const Axis &ax, float (&tile)[kAdjLines][32 * (M + 4)],
                                                        int32_t line0, bool live, int lane, const float (&v)[M],
                                                        float *__restrict__ out)
        {
            float *mine = tile[threadIdx.x >> 5] + lane * (M + 4);
#pragma unroll
            for (int q = 0; q < M / 4; q++)
            {
                *reinterpret_cast<float4 *>(mine + 4 * q) =
                    live ? make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3])
                         : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
            __syncthreads();
            for (int32_t pos = threadIdx.x; pos < ax.n; pos += 32 * kAdjLines)
            {
                const int at = pos / M * (M + 4) + pos % M;
                *reinterpret_cast<float4 *>(out + static_cast<int64_t>(pos) * ax.ldT + line0) =
                    make_float4(tile[0][at], tile[1][at], tile[2][at], tile[3][at]);
            }
        }

        // One sweep of a forward step over the lines of an axis, in residual
        // form: u + (I - L/2)^-1 (L + Lcross) u / 2, so that the solve's
        // rounding scales with the step's change, not the field.
        // x-sweep (COMMIT false): in = f by x; out = w by y (transposed), keep =
        // w by x (or null).  y-sweep (COMMIT true): in = w by y, f by y; out =
        // f' by x (transposed), fOut = f' by y, keep = v by y (or null).
        template <int M, bool COMMIT>
        __global__ void __launch_bounds__(32 * kAdjLines)
            FwdLines(Axis ax, const float *__restrict__ in, const float *__restrict__ f, const float *__restrict__ src,
                     const float *__restrict__ par, float *__restrict__ out, float *__restrict__ fOut,
                     float *__restrict__ keep)
        {
            __shared__ __align__(16) float tile[kAdjLines][32 * (M + 4)];
            const int lane = threadIdx.x & 31;
            const int32_t line0 = blockIdx.x * kAdjLines;
            const bool live = line0 + static_cast<int32_t>(threadIdx.x >> 5) < ax.nl;
            const int32_t line = min(line0 + static_cast<int32_t>(threadIdx.x >> 5), ax.nl - 1);
            const int li = ax.n - 1 - lane * M;
            const bool hasUp = line + 1 < ax.nl || (ax.wrapCross && ax.nl > 1);
            const bool hasDn = line > 0 || (ax.wrapCross && ax.nl > 1);
            const int64_t up = hasUp ? (line + 1 < ax.nl ? line + 1 : 0) : line;
            const int64_t dn = hasDn ? (line > 0 ? line - 1 : ax.nl - 1) : line;
            Factors<M> k;
            k.Load(ax, line, lane);
            float e[M], eDn[M], f0[COMMIT ? M : 1], sv[COMMIT ? M : 1];
            LoadRow<M>(ax.D + line * static_cast<int64_t>(ax.ld), ax.ld, lane, e);
            LoadRow<M>(ax.D + dn * ax.ld, ax.ld, lane, eDn);
            const float eW = ax.wrap ? __ldcg(ax.D + static_cast<int64_t>(line) * ax.ld + ax.n - 1) : 0.0f;
            if constexpr (COMMIT)
            {
                LoadRow<M>(f + line * static_cast<int64_t>(ax.ld), ax.ld, lane, f0);
                if (src != nullptr)
                {
                    LoadRow<M>(src + line * static_cast<int64_t>(ax.ld), ax.ld, lane, sv);
                }
            }
            const float negDecay = COMMIT ? __ldg(par + 1) : 0.0f;
            WaitForPredecessor();
            float c[M], d[M];
            {
                float uu[M], ud[M];
                LoadRow<M>(in + line * static_cast<int64_t>(ax.ld), ax.ld, lane, c);
                LoadRow<M>(in + up * ax.ld, ax.ld, lane, uu);
                LoadRow<M>(in + dn * ax.ld, ax.ld, lane, ud);
                const float wu = hasUp ? 1.0f : 0.0f, wd = hasDn ? 1.0f : 0.0f;
#pragma unroll
                for (int i = 0; i < M; i++)
                {
                    uu[i] = fmaf(wd * eDn[i], ud[i] - c[i], wu * e[i] * (uu[i] - c[i]));
                }
                MaskLast<M>(e, li);
                LapAlong<M>(ax, c, e, eW, lane, d);
#pragma unroll
                for (int i = 0; i < M; i++)
                {
                    d[i] = 0.5f * (uu[i] + d[i]);
                }
            }
            Solve<M>(ax, k, line, lane, d);
            if constexpr (COMMIT)
            {
                float fn[M];
#pragma unroll
                for (int i = 0; i < M; i++)
                {
                    // v - f = (w - f) + e: both small, so the commit keeps the
                    // field's precision
                    float delta = (c[i] - f0[i]) + d[i];
                    delta = fmaf(f0[i], negDecay, delta);
                    delta = src != nullptr ? delta + sv[i] : delta;
                    fn[i] = f0[i] + delta;
                    d[i] = c[i] + d[i];
                }
                if (live)
                {
                    StoreRow<M>(fOut + line * static_cast<int64_t>(ax.ld), ax.ld, lane, fn);
                    if (keep != nullptr)
                    {
                        StoreRow<M>(keep + line * static_cast<int64_t>(ax.ld), ax.ld, lane, d);
                    }
                }
                StoreTransposed<M>(ax, tile, line0, live, lane, fn, out);
            }
            else
            {
#pragma unroll
                for (int i = 0; i < M; i++)
                {
                    d[i] = c[i] + d[i];
                }
                if (live && keep != nullptr)
                {
                    StoreRow<M>(keep + line * static_cast<int64_t>(ax.ld), ax.ld, lane, d);
                }
                StoreTransposed<M>(ax, tile, line0, live, lane, d, out);
            }
        }

        // s + x and its rounding error (Knuth's two-sum).
        __device__ __forceinline__ float TwoSum(float &s, float x)
        {
            const float t = __fadd_rn(s, x);
            const float b = __fsub_rn(t, s);
            const float e = __fadd_rn(__fsub_rn(s, __fsub_rn(t, b)), __fsub_rn(x, b));
            s = t;
            return e;
        }

        // The power of two, as its exponent, that brings the largest of |v| into
        // [1, 2) (or next to it at the ends of the range).
        template <int M>
        __device__ __forceinline__ int Exponent(const float (&v)[M], bool &finite)
        {
            float m = 0.0f;
#pragma unroll
            for (int i = 0; i < M; i++)
            {
                m = fmaxf(m, fabsf(v[i]));
                finite = finite && v[i] == v[i];  // (fmaxf leaves NaN out)
            }
            const int e = static_cast<int>(__float_as_uint(m) >> 23);
            finite = finite && e < 255;
            return min(max(e, 1), 253) - 127;
        }

        // sum - <g, f> over a lane's positions.  An FP64 instruction holds its
        // pipe for 64 cycles, conversions included: M products summed in FP64 made
        // a step of a 300 x 700 gradient 2.5 us longer.  Here the operands are
        // scaled by powers of two so that no product leaves FP32's range, each
        // product is a pair of floats and the sum three, all without error but
        // the third's (2^-72 of the largest term), and only their total is added
        // in FP64: fewer roundings than a sum in FP64 throughout.
        template <int M>
        __device__ __forceinline__ double SubDot(double sum, const float (&g)[M], const float (&f)[M])
        {
            bool finite = true;
            const int eg = Exponent<M>(g, finite), ef = Exponent<M>(f, finite);
            if (!finite)
            {
#pragma unroll 1
                for (int i = 0; i < M; i++)
                {
                    float a = 0.0f, b = 0.0f;
#pragma unroll
                    for (int k = 0; k < M; k++)
                    {
                        a = (k == i) ? g[k] : a;
                        b = (k == i) ? f[k] : b;
                    }
                    sum = fma(-static_cast<double>(a), static_cast<double>(b), sum);
                }
                return sum;
            }
            const float kg = __uint_as_float(static_cast<uint32_t>(127 - eg) << 23);
            const float kf = __uint_as_float(static_cast<uint32_t>(127 - ef) << 23);
            float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f;
#pragma unroll
            for (int i = 0; i < M; i++)
            {
                const float a = __fmul_rn(g[i], kg), b = __fmul_rn(f[i], kf);
                const float p = __fmul_rn(a, b);
                const float e = TwoSum(s0, p);
                s2 = __fadd_rn(s2, TwoSum(s1, __fmaf_rn(a, b, -p)));
                s2 = __fadd_rn(s2, TwoSum(s1, e));
            }
            const double t = (static_cast<double>(s2) + static_cast<double>(s1)) + static_cast<double>(s0);
            return fma(-t, __hiloint2double((1023 + eg + ef) << 20, 0), sum);
        }

        enum BwdYMode : int
        {
            kBwdFirst = 0,  // gbar given (the last step's output adjoint)
            kBwdNext = 1,   // gbar = (I + Ly/2) b1bar - decay gbarPrev
            kBwdTail = 2    // the y-stencil part of kBwdNext only (after step 0)
        };

        // Backward along y for step t: [gbar from step t+1] then the y-solve.
        // All arrays by y, but b2bar, which leaves by x.  ddecay's sum is FP64,
        // one per lane and line.  A step's term, -<gbar of t, f_t>, is added by
        // the launch of step t-1 (the tail for step 0), whose gPrev and fNext are
        // its factors and are loaded before the wait: the sum may run while the
        // kernel before does, off the step's critical path.
        template <int M>
        __global__ void __launch_bounds__(32 * kAdjLines)
            BwdY(Axis ax, int mode, const float *__restrict__ par,
                 const float *__restrict__ b1bar,  // step t+1's x-solve adjoint (kBwdNext/Tail)
                 const float *__restrict__ gPrev,  // adjoint of f_t+2 (kBwdNext/Tail), or gbar (kBwdFirst)
                 const float *__restrict__ fNext,  // f_t+1 (kBwdNext/Tail)
                 const float *__restrict__ vT,     // v_t
                 float *__restrict__ gOut,         // adjoint of f_t+1 (gbar of step t)
                 float *__restrict__ b2bar, float *__restrict__ dD, float *__restrict__ dS,
                 double *__restrict__ dDecay)
        {
            __shared__ __align__(16) float tile[kAdjLines][32 * (M + 4)];
            const int lane = threadIdx.x & 31;
            const int32_t line0 = blockIdx.x * kAdjLines;
            const bool live = line0 + static_cast<int32_t>(threadIdx.x >> 5) < ax.nl;
            const int32_t line = min(line0 + static_cast<int32_t>(threadIdx.x >> 5), ax.nl - 1);
            const int64_t row = line * static_cast<int64_t>(ax.ld);
            Factors<M> k;
            k.Load(ax, line, lane);
            float e[M], g[M], acc[M], q[M], t[M];
            LoadRow<M>(ax.D + row, ax.ld, lane, e);
            const float eW = ax.wrap ? __ldcg(ax.D + row + ax.n - 1) : 0.0f;
            MaskLast<M>(e, ax.n - 1 - lane * M);
            const float decay = __ldg(par);
            LoadRow<M>(gPrev + row, ax.ld, lane, g);
            LoadRow<M>(fNext + row, ax.ld, lane, q);
            // this step's terms of dD, small beside the sum so far
#pragma unroll
            for (int i = 0; i < M; i++)
            {
                acc[i] = 0.0f;
            }
            if (mode != kBwdFirst && live)
            {
                double *at = dDecay + static_cast<int64_t>(line) * 32 + lane;
                *at = SubDot<M>(__ldcg(at), g, q);
            }
            WaitForPredecessor();
            if (mode != kBwdFirst)
            {
                float b[M];
                LoadRow<M>(b1bar + row, ax.ld, lane, b);
                LapAlong<M>(ax, b, e, eW, lane, t);
#pragma unroll
                for (int i = 0; i < M; i++)
                {
                    g[i] = fmaf(0.5f, t[i], b[i]) - decay * g[i];
                }
                AddFaceGrad<M>(ax, b, q, lane, acc);
                if (mode == kBwdTail)
                {
                    if (live)
                    {
                        AddRow<M>(dD + row, ax.ld, lane, acc);
                    }
                    return;
                }
            }
            // residual form: b2bar = gbar + (I - Ly/2)^-1 (Ly gbar) / 2
            float d[M];
            LapAlong<M>(ax, g, e, eW, lane, d);
#pragma unroll
            for (int i = 0; i < M; i++)
            {
                d[i] *= 0.5f;
            }
            Solve<M>(ax, k, line, lane, d);
            // the accumulators' rows, in flight during the write-out (the
            // factors' registers are free now)
            float sD[M], sS[M];
            LoadRow<M>(vT + row, ax.ld, lane, q);
            LoadRow<M>(dD + row, ax.ld, lane, sD);
            LoadRow<M>(dS + row, ax.ld, lane, sS);
#pragma unroll
            for (int i = 0; i < M; i++)
            {
                d[i] += g[i];
            }
            StoreTransposed<M>(ax, tile, line0, live, lane, d, b2bar);
            AddFaceGrad<M>(ax, d, q, lane, acc);
            if (!live)
            {
                return;
            }
            StoreRow<M>(gOut + row, ax.ld, lane, g);
#pragma unroll
            for (int i = 0; i < M; i++)
            {
                sD[i] += acc[i];
                sS[i] += g[i];
            }
            StoreRow<M>(dD + row, ax.ld, lane, sD);
            StoreRow<M>(dS + row, ax.ld, lane, sS);
        }

        // Backward along x for step t: wbar = (I + Lx/2) b2bar, b1bar = (I - Lx/2)^-1 wbar.
        // All arrays by x, but b1bar, which leaves by y.
        template <int M>
        __global__ void __launch_bounds__(32 * kAdjLines)
            BwdX(Axis ax, const float *__restrict__ b2bar, const float *__restrict__ wT, float *__restrict__ b1bar,
                 float *__restrict__ dD)
        {
            __shared__ __align__(16) float tile[kAdjLines][32 * (M + 4)];
            const int lane = threadIdx.x & 31;
            const int32_t line0 = blockIdx.x * kAdjLines;
            const bool live = line0 + static_cast<int32_t>(threadIdx.x >> 5) < ax.nl;
            const int32_t line = min(line0 + static_cast<int32_t>(threadIdx.x >> 5), ax.nl - 1);
            const int64_t row = line * static_cast<int64_t>(ax.ld);
            Factors<M> k;
            k.Load(ax, line, lane);
            float e[M], w[M], acc[M], b[M], l[M], d[M];
            LoadRow<M>(ax.D + row, ax.ld, lane, e);
            const float eW = ax.wrap ? __ldcg(ax.D + row + ax.n - 1) : 0.0f;
            MaskLast<M>(e, ax.n - 1 - lane * M);
            LoadRow<M>(wT + row, ax.ld, lane, w);
#pragma unroll
            for (int i = 0; i < M; i++)
            {
                acc[i] = 0.0f;
            }
            WaitForPredecessor();
            LoadRow<M>(b2bar + row, ax.ld, lane, b);
            LapAlong<M>(ax, b, e, eW, lane, l);
            // residual form: b1bar = wbar + (I - Lx/2)^-1 (Lx wbar) / 2, with
            // Lx wbar = Lx b2bar + Lx (Lx b2bar) / 2
            LapAlong<M>(ax, l, e, eW, lane, d);
#pragma unroll
            for (int i = 0; i < M; i++)
            {
                d[i] = 0.5f * fmaf(0.5f, d[i], l[i]);
            }
            Solve<M>(ax, k, line, lane, d);
            float sD[M];
            LoadRow<M>(dD + row, ax.ld, lane, sD);
#pragma unroll
            for (int i = 0; i < M; i++)
            {
                d[i] += fmaf(0.5f, l[i], b[i]);
            }
            StoreTransposed<M>(ax, tile, line0, live, lane, d, b1bar);
            AddFaceGrad<M>(ax, b, w, lane, acc);
            AddFaceGrad<M>(ax, d, w, lane, acc);
            if (live)
            {
#pragma unroll
                for (int i = 0; i < M; i++)
                {
                    sD[i] += acc[i];
                }
                StoreRow<M>(dD + row, ax.ld, lane, sD);
            }
        }

        // ---- the factors -----------------------------------------------------

        // 1 / b by Newton's iteration from the hardware's approximation (20
        // bits, then 40, then all but the last rounding), for finite b >= 1 and
        // thereabouts.  An IEEE division is three times as long a chain of FP64
        // instructions, and the factors leave in FP32.
        __device__ __forceinline__ double Reciprocal(double b)
        {
            double y;
            asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
            y = fma(fma(-b, y, 1.0), y, y);
            return fma(fma(-b, y, 1.0), y, y);
        }

        // Factors every line of an axis (one warp a line, FP64): see the top of
        // this file.  Positions beyond the line are rows of the identity.  Bound
        // by its chains of FP64 instructions, 64 cycles and more each: us per
        // axis of 64^2 / 512^2 / 1024^2 with IEEE divisions 19 / 29 / 80, so 11 /
        // 23 / 63, and the axes run side by side.  (A call of one step still pays
        // more for its factors than it gains: forward 64^2 77 us against 54 with
        // the reductions, even from some 8 steps on; gradients from 2 or 3.)
        template <int M>
        __global__ void __launch_bounds__(32 * kAdjLines) Factor(Axis ax, float *__restrict__ coef, float *__restrict__ ext)
        {
            const int lane = threadIdx.x & 31;
            const int32_t line = blockIdx.x * kAdjLines + static_cast<int32_t>(threadIdx.x >> 5);
            if (line >= ax.nl)
            {
                return;
            }
            const float *D = ax.D + static_cast<int64_t>(line) * ax.ld;
            const int32_t n = ax.n;
            // a wrapped pair has two faces between its cells, a wrapped single
            // cell couples only to itself (L = 0); longer wrapped lines are
            // split as T + u v^T
            const bool split = ax.wrap && n >= 3;
            const double eW = split ? static_cast<double>(D[n - 1]) : 0.0;
            // a face's coefficient -D/2 is exact in FP32 (but for the sum of a
            // wrapped pair's two faces)
            auto half = [&](int32_t j)  // -1/2 of face (j, j+1) within the line
            {
                if (j < 0 || j >= n - 1)
                {
                    return 0.0;
                }
                const double h = static_cast<double>(-0.5f * D[j]);
                return (ax.wrap && n == 2) ? h - 0.5 * static_cast<double>(D[1]) : h;
            };
            const double a0 = -0.5 * eW;  // row 0's coefficient of x_n-1, and row n-1's of x_0
            const double gamma = -(1.0 - a0 - half(0));
            double a[M], b[M], c[M];
            double before = half(lane * M - 1);
#pragma unroll
            for (int i = 0; i < M; i++)
            {
                const int32_t j = lane * M + i;
                const double here = half(j);
                a[i] = (j < n) ? before : 0.0;
                c[i] = here;
                b[i] = 1.0 - (a[i] + c[i]);
                if (split && j == 0)
                {
                    b[i] = b[i] - a0 - gamma;
                }
                if (split && j == n - 1)
                {
                    b[i] = b[i] - a0 - a0 * a0 / gamma;
                }
                before = here;
            }
            double fw[M], ib[M], cb[M], p[M], q[M];
            double bp = b[0];
            fw[0] = 0.0;
            ib[0] = Reciprocal(bp);
#pragma unroll
            for (int i = 1; i < M - 1; i++)
            {
                fw[i] = a[i] * ib[i - 1];
                bp = b[i] - fw[i] * c[i - 1];
                ib[i] = Reciprocal(bp);
            }
#pragma unroll
            for (int i = 0; i < M - 1; i++)
            {
                cb[i] = (i < M - 2) ? c[i] * ib[i] : 0.0;
            }
            fw[M - 1] = ib[M - 1] = cb[M - 1] = 0.0;
            // p = A^-1 (a_0 e_0), q = A^-1 (c_M-2 e_M-2)
            p[0] = a[0];
#pragma unroll
            for (int i = 1; i < M - 1; i++)
            {
                p[i] = -fw[i] * p[i - 1];
            }
            q[M - 2] = c[M - 2] * ib[M - 2];
            p[M - 2] *= ib[M - 2];
#pragma unroll
            for (int i = M - 3; i >= 0; i--)
            {
                p[i] = p[i] * ib[i] - cb[i] * p[i + 1];
                q[i] = -cb[i] * q[i + 1];
            }
            p[M - 1] = q[M - 1] = 0.0;
            const double as = a[M - 1], cs = lane < 31 ? c[M - 1] : 0.0;
            const double pn = __shfl_down_sync(kAll, p[0], 1), qn = __shfl_down_sync(kAll, q[0], 1);
            double A = -as * p[M - 2], B = b[M - 1] - as * q[M - 2] - cs * pn, C = -cs * qn;
            double lo[5], hi[5];
#pragma unroll
            for (int t = 0; t < 5; t++)
            {
                const int s = 1 << t;
                const double al = __shfl_up_sync(kAll, A, s), bl = __shfl_up_sync(kAll, B, s),
                             cl = __shfl_up_sync(kAll, C, s);
                const double ar = __shfl_down_sync(kAll, A, s), br = __shfl_down_sync(kAll, B, s),
                             cr = __shfl_down_sync(kAll, C, s);
                lo[t] = lane >= s ? -A * Reciprocal(bl) : 0.0;
                hi[t] = lane + s < 32 ? -C * Reciprocal(br) : 0.0;
                B += (lane >= s ? lo[t] * cl : 0.0) + (lane + s < 32 ? hi[t] * ar : 0.0);
                A = lane >= s ? lo[t] * al : 0.0;
                C = lane + s < 32 ? hi[t] * cr : 0.0;
            }
            const double binv = Reciprocal(B);
            const int nc = ax.wrap ? 6 : 5;
            float *o = coef + static_cast<int64_t>(line) * nc * M * 32 + 4 * lane;
            auto put = [&](int k, const double (&v)[M])
            {
#pragma unroll
                for (int i = 0; i < M; i++)
                {
                    o[(k * (M / 4) + i / 4) * 128 + (i & 3)] = static_cast<float>(v[i]);
                }
            };
            put(kCoefFw, fw);
            put(kCoefIb, ib);
            put(kCoefCb, cb);
            put(kCoefP, p);
            put(kCoefQ, q);
            double bog = 0.0;
            if (ax.wrap)
            {
                double z[M];
#pragma unroll
                for (int i = 0; i < M; i++)
                {
                    z[i] = 0.0;
                }
                if (split)
                {
                    // T z = u = (gamma, 0, .., 0, a0)
                    bog = a0 / gamma;
#pragma unroll
                    for (int i = 0; i < M; i++)
                    {
                        const int32_t j = lane * M + i;
                        z[i] = (j == 0) ? gamma : ((j == n - 1) ? a0 : 0.0);
                    }
#pragma unroll
                    for (int i = 1; i < M - 1; i++)
                    {
                        z[i] -= fw[i] * z[i - 1];
                    }
                    z[M - 2] *= ib[M - 2];
#pragma unroll
                    for (int i = M - 3; i >= 0; i--)
                    {
                        z[i] = z[i] * ib[i] - cb[i] * z[i + 1];
                    }
                    double r = z[M - 1] - as * z[M - 2] - cs * __shfl_down_sync(kAll, z[0], 1);
#pragma unroll
                    for (int t = 0; t < 5; t++)
                    {
                        const double rl = __shfl_up_sync(kAll, r, 1 << t), rr = __shfl_down_sync(kAll, r, 1 << t);
                        r += lo[t] * rl + hi[t] * rr;
                    }
                    const double s = r * binv;
                    double sl = __shfl_up_sync(kAll, s, 1);
                    sl = lane == 0 ? 0.0 : sl;
#pragma unroll
                    for (int i = 0; i < M - 1; i++)
                    {
                        z[i] -= sl * p[i] + s * q[i];
                    }
                    z[M - 1] = s;
                    double zn = 0.0;
#pragma unroll
                    for (int i = 0; i < M; i++)
                    {
                        zn = (lane * M + i == n - 1) ? z[i] : zn;
                    }
                    zn = __shfl_sync(kAll, zn, (n - 1) / M);
                    const double inv = 1.0 / (1.0 + __shfl_sync(kAll, z[0], 0) + bog * zn);
#pragma unroll
                    for (int i = 0; i < M; i++)
                    {
                        z[i] *= inv;
                    }
                }
                put(kCoefZ, z);
            }
            float *x = ext + static_cast<int64_t>(line) * kExtCount * 32 + lane;
#pragma unroll
            for (int t = 0; t < 5; t++)
            {
                x[(kExtLo + t) * 32] = static_cast<float>(lo[t]);
                x[(kExtHi + t) * 32] = static_cast<float>(hi[t]);
            }
            x[kExtBinv * 32] = static_cast<float>(binv);
            x[kExtA * 32] = static_cast<float>(as);
            x[kExtC * 32] = static_cast<float>(cs);
            x[kExtBog * 32] = static_cast<float>(bog);
        }

        // ---- the rest of a call --------------------------------------------

        constexpr int kLossThreads = 256;
        constexpr int kLossBlocks = 1024;

        __device__ __forceinline__ double BlockSum(double v, double *sred)
        {
            for (int o = 16; o > 0; o >>= 1)
            {
                v += __shfl_down_sync(kAll, v, o);
            }
            const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
            __syncthreads();
            if (lane == 0)
            {
                sred[warp] = v;
            }
            __syncthreads();
            double t = 0.0;
            if (threadIdx.x == 0)
            {
                for (int k = 0; k < static_cast<int>((blockDim.x + 31) / 32); k++)
                {
                    t += sred[k];
                }
            }
            return t;
        }

        // part[block] = sum of 1/2 (f - target)^2; gbar = f - target.
        __global__ void __launch_bounds__(kLossThreads)
            LossGrad(int64_t n, const float *__restrict__ f, const float *__restrict__ target,
                     float *__restrict__ gbar, double *__restrict__ part)
        {
            __shared__ double sred[32];
            double acc = 0.0;
            for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
                 i += static_cast<int64_t>(gridDim.x) * blockDim.x)
            {
                const float r = f[i] - target[i];
                if (gbar != nullptr)
                {
                    gbar[i] = r;
                }
                acc += 0.5 * static_cast<double>(r) * static_cast<double>(r);
            }
            const double t = BlockSum(acc, sred);
            if (threadIdx.x == 0)
            {
                part[blockIdx.x] = t;
            }
        }

        // acc[0] = sum of part; acc[1] = sum of dDecay (one CTA, a fixed order).
        // (256 threads for the parts alone, 3 to 5 us; 1024 with the sums, 16384
        // of them at 512^2: 8 us, 17 with 256)
        __global__ void __launch_bounds__(1024)
            Totals(const double *__restrict__ part, int32_t nPart, const double *__restrict__ dDecay, int64_t nDecay,
                   double *__restrict__ acc)
        {
            __shared__ double sred[32];
            double a = 0.0, b = 0.0;
            // (the first 256 threads, so that the loss has one order of summing)
            for (int32_t i = threadIdx.x; threadIdx.x < 256 && i < nPart; i += 256)
            {
                a += part[i];
            }
            for (int64_t i = threadIdx.x; i < nDecay; i += blockDim.x)
            {
                b += dDecay[i];
            }
            a = BlockSum(a, sred);
            b = nDecay > 0 ? BlockSum(b, sred) : 0.0;
            if (threadIdx.x == 0)
            {
                acc[0] = a;
                acc[1] = b;
            }
        }

        // out[c * ldOut + r] (+)= in[r * ldIn + c], rows x cols.
        template <bool ADD>
        __global__ void TransposeRows(const float *__restrict__ in, int32_t ldIn, float *__restrict__ out, int32_t ldOut,
                                      int32_t rows, int32_t cols)
        {
            __shared__ float tile[32][33];
            const int32_t r0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
            for (int32_t k = threadIdx.y; k < 32; k += blockDim.y)
            {
                const int32_t r = r0 + k, c = c0 + threadIdx.x;
                if (r < rows && c < cols)
                {
                    tile[k][threadIdx.x] = in[static_cast<int64_t>(r) * ldIn + c];
                }
            }
            __syncthreads();
            for (int32_t k = threadIdx.y; k < 32; k += blockDim.y)
            {
                const int32_t c = c0 + k, r = r0 + threadIdx.x;
                if (r < rows && c < cols)
                {
                    float *o = out + static_cast<int64_t>(c) * ldOut + r;
                    *o = ADD ? *o + tile[threadIdx.x][k] : tile[threadIdx.x][k];
                }
            }
        }

        // Positions per lane of a line: M = 4 * ceil(n / 128).
        constexpr int32_t LaneLen(int32_t n)
        {
            return (n + 127) / 128 * 4;
        }

        // Calls fn with M as a compile-time constant.
        template <typename Fn>
        auto WithLaneLen(int32_t m, Fn fn)
        {
            switch (m / 4)
            {
            case 1:
                return fn(std::integral_constant<int, 4>());
            case 2:
                return fn(std::integral_constant<int, 8>());
            case 3:
                return fn(std::integral_constant<int, 12>());
            case 4:
                return fn(std::integral_constant<int, 16>());
            case 5:
                return fn(std::integral_constant<int, 20>());
            case 6:
                return fn(std::integral_constant<int, 24>());
            case 7:
                return fn(std::integral_constant<int, 28>());
            default:
                return fn(std::integral_constant<int, 32>());
            }
        }

        // Launches `kernel`, as a programmatic dependent of the kernel before
        // it in the stream if chained.
        template <typename... P, typename... A>
        int LaunchChained(void (*kernel)(P...), int32_t nl, bool chained, cudaStream_t s, A... args)
        {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(static_cast<unsigned>((nl + kAdjLines - 1) / kAdjLines));
            cfg.blockDim = dim3(32 * kAdjLines);
            cfg.stream = s;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            at[0].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = at;
            cfg.numAttrs = chained ? 1 : 0;
            return CudaStatus(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...), "adjoint launch");
        }
    }

    struct Adjoint
    {
        int device = 0;
        StreamSlot stream;
        int32_t xDim = 0, yDim = 0, ldX = 0, ldY = 0;
        Axis axX{}, axY{};                  // x-lines (by x) and y-lines (by y)
        int64_t n = 0;                      // cells
        size_t nA = 0, nB = 0;              // padded array sizes, by y and by x
        int32_t steps = 0, every = 1;
        bool keepAll = false;               // checkpoint interval 0: every state kept, nothing recomputed
        bool hasProblem = false;
        // by y: the problem, the fields, the adjoints (but b2), the y-faces'
        // part of dL/dD
        DevBuf<float> f0, target, D, src, work[2], wA, gA, gB, b1, dD, dS;
        DevBuf<float> ckpt;                 // checkpoints: one field every `every` steps
        DevBuf<float> segF[2], segV[2];     // states of a segment, double-buffered
        // by x: the rates, the current field, b2, the x-faces' part of dL/dD,
        // and the w of a segment
        DevBuf<float> DT, fB, b2, dDT;
        DevBuf<float> segW[2];
        StreamSlot recomputeStream;         // recomputes segment s-1 while segment s is differentiated
        DevBuf<float> coefX, extX, coefY, extY;
        DevBuf<float> par;                  // decay, -decay
        DevBuf<double> dDecay;              // BwdY's sums
        DevBuf<double> part, acc;           // the loss's partial sums; [0] loss, [1] d loss / d decay
        float msForward = 0.0f, msGradient = 0.0f;
        // runs of steps as graphs (the pointers are the problem's): see Replay
        std::map<std::string, cudaGraphExec_t> graphs;

        cudaEvent_t factored = nullptr;     // the y-lines' factors, made on recomputeStream

        ~Adjoint()
        {
            DropGraphs();
            if (factored != nullptr)
            {
                cudaEventDestroy(factored);
            }
        }

        void DropGraphs()
        {
            for (auto &g : graphs)
            {
                cudaGraphExecDestroy(g.second);
            }
            graphs.clear();
        }

        int32_t Segments() const
        {
            return (steps + every - 1) / every;
        }

        int Init(int32_t xd, int32_t yd, int32_t wrapX, int32_t wrapY)
        {
            device = CurrentDevice();
            HAL_TRY(CudaStatus(cudaSetDevice(device), "cudaSetDevice"));
            // the backward (and the forward) on the highest-priority stream,
            // the overlapped recomputation on the lowest: recompute CTAs take
            // the SMs the critical path leaves free
            int least = 0, greatest = 0;
            HAL_TRY(CudaStatus(cudaDeviceGetStreamPriorityRange(&least, &greatest), "cudaDeviceGetStreamPriorityRange"));
            HAL_TRY(stream.Create("cudaStreamCreate", greatest));
            HAL_TRY(recomputeStream.Create("cudaStreamCreate", least));
            HAL_TRY(CudaStatus(cudaEventCreateWithFlags(&factored, cudaEventDisableTiming), "cudaEventCreate"));
            xDim = xd;
            yDim = yd;
            ldX = (xDim + 3) & ~3;
            ldY = (yDim + 3) & ~3;
            n = static_cast<int64_t>(xDim) * yDim;
            nA = static_cast<size_t>(xDim) * ldY;
            nB = static_cast<size_t>(yDim) * ldX;
            for (DevBuf<float> *b : {&f0, &target, &D, &src, &work[0], &work[1], &wA, &gA, &gB, &b1, &dD, &dS})
            {
                HAL_TRY(Zeroed(*b, nA));
            }
            for (DevBuf<float> *b : {&DT, &fB, &b2, &dDT})
            {
                HAL_TRY(Zeroed(*b, nB));
            }
            const size_t mx = static_cast<size_t>(LaneLen(xDim)), my = static_cast<size_t>(LaneLen(yDim));
            HAL_TRY(coefX.Alloc(static_cast<size_t>(yDim) * (wrapX ? 6 : 5) * mx * 32, "cudaMalloc(adjoint)"));
            HAL_TRY(coefY.Alloc(static_cast<size_t>(xDim) * (wrapY ? 6 : 5) * my * 32, "cudaMalloc(adjoint)"));
            HAL_TRY(extX.Alloc(static_cast<size_t>(yDim) * kExtCount * 32, "cudaMalloc(adjoint)"));
            HAL_TRY(extY.Alloc(static_cast<size_t>(xDim) * kExtCount * 32, "cudaMalloc(adjoint)"));
            HAL_TRY(par.Alloc(2, "cudaMalloc(adjoint)"));
            HAL_TRY(dDecay.Alloc(static_cast<size_t>(xDim) * 32, "cudaMalloc(adjoint)"));
            HAL_TRY(part.Alloc(kLossBlocks, "cudaMalloc(adjoint)"));
            HAL_TRY(acc.Alloc(2, "cudaMalloc(adjoint)"));
            axX = Axis{xDim, yDim, ldX, ldY, wrapX != 0, wrapY != 0, DT.p, coefX.p, extX.p};
            axY = Axis{yDim, xDim, ldY, ldX, wrapY != 0, wrapX != 0, D.p, coefY.p, extY.p};
            return HAL_CUDA_OK;
        }

        // A zeroed buffer: the padding stays zero from here on.
        static int Zeroed(DevBuf<float> &b, size_t count)
        {
            HAL_TRY(b.Alloc(count, "cudaMalloc(adjoint)"));
            return CudaStatus(cudaMemset(b.p, 0, count * sizeof(float)), "cudaMemset(adjoint)");
        }

        // Host arrays (xDim x yDim) to and from the padded "by y" layout.
        // (as one run of bytes where nothing is padded)
        int ToDevice(float *d, const float *h, cudaStream_t s, const char *what) const
        {
            if (ldY == yDim)
            {
                return CudaStatus(cudaMemcpyAsync(d, h, nA * sizeof(float), cudaMemcpyHostToDevice, s), what);
            }
            return CudaStatus(cudaMemcpy2DAsync(d, ldY * sizeof(float), h, yDim * sizeof(float), yDim * sizeof(float),
                                                static_cast<size_t>(xDim), cudaMemcpyHostToDevice, s), what);
        }

        int ToHost(float *h, const float *d, cudaStream_t s, const char *what) const
        {
            if (ldY == yDim)
            {
                return CudaStatus(cudaMemcpyAsync(h, d, nA * sizeof(float), cudaMemcpyDeviceToHost, s), what);
            }
            return CudaStatus(cudaMemcpy2DAsync(h, yDim * sizeof(float), d, ldY * sizeof(float), yDim * sizeof(float),
                                                static_cast<size_t>(xDim), cudaMemcpyDeviceToHost, s), what);
        }

        int CopyField(float *to, const float *from, cudaStream_t s) const
        {
            return CudaStatus(cudaMemcpyAsync(to, from, nA * sizeof(float), cudaMemcpyDeviceToDevice, s),
                              "cudaMemcpy(field)");
        }

        // out (by x) = in (by y)
        int ByX(const float *in, float *out, cudaStream_t s) const
        {
            TransposeRows<false><<<dim3((xDim + 31) / 32, (yDim + 31) / 32), dim3(32, 8), 0, s>>>(in, ldY, out, ldX,
                                                                                                  xDim, yDim);
            CountLaunch();
            return LaunchStatus("adjoint transpose");
        }

        // One forward step fIn -> fOut (by y; fB holds fIn by x and then
        // fOut); the step's w is kept in wKeep and its v in vKeep when they
        // are set.  chained: the kernel before it on s may be overlapped.
        int LaunchFwd(const float *fIn, float *fOut, float *wKeep, float *vKeep, const float *srcp, bool chained,
                      cudaStream_t s)
        {
            HAL_TRY(WithLaneLen(LaneLen(xDim), [&](auto m) {
                return LaunchChained(FwdLines<m(), false>, yDim, chained, s, axX, fB.p, nullptr, nullptr, par.p, wA.p,
                                     nullptr, wKeep);
            }));
            HAL_TRY(WithLaneLen(LaneLen(yDim), [&](auto m) {
                return LaunchChained(FwdLines<m(), true>, xDim, true, s, axY, wA.p, fIn, srcp, par.p, fB.p, fOut, vKeep);
            }));
            CountLaunch(2);
            return HAL_CUDA_OK;
        }

        int LaunchBwdY(int mode, const float *gPrev, const float *fNext, const float *vT, float *gOut, bool chained,
                       cudaStream_t s)
        {
            CountLaunch();
            return WithLaneLen(LaneLen(yDim), [&](auto m) {
                return LaunchChained(BwdY<m()>, xDim, chained, s, axY, mode, par.p, b1.p, gPrev, fNext, vT, gOut,
                                     b2.p, dD.p, dS.p, dDecay.p);
            });
        }

        int LaunchBwdX(const float *wT, cudaStream_t s)
        {
            CountLaunch();
            return WithLaneLen(LaneLen(xDim), [&](auto m) {
                return LaunchChained(BwdX<m()>, yDim, true, s, axX, b2.p, wT, b1.p, dDT.p);
            });
        }

        // Enqueues on s what `body(s)` enqueues (`kernels` of them), replayed from
        // a graph of that key: a launch of a run of steps instead of one per
        // kernel.
        template <typename Body>
        int Replay(const std::string &key, int64_t kernels, cudaStream_t s, Body body)
        {
            auto it = graphs.find(key);
            if (it == graphs.end())
            {
                HAL_TRY(CudaStatus(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal), "cudaStreamBeginCapture"));
                const int rc = body(s);
                cudaGraph_t g = nullptr;
                const cudaError_t e = cudaStreamEndCapture(s, &g);
                if (rc == HAL_CUDA_OK)
                {
                    CountLaunch(-kernels);  // counted by each replay
                }
                if (rc != HAL_CUDA_OK || e != cudaSuccess)
                {
                    if (g != nullptr)
                    {
                        cudaGraphDestroy(g);
                    }
                    return rc != HAL_CUDA_OK ? rc : CudaStatus(e, "cudaStreamEndCapture");
                }
                cudaGraphExec_t x = nullptr;
                const cudaError_t ei = cudaGraphInstantiate(&x, g, 0);
                cudaGraphDestroy(g);
                HAL_TRY(CudaStatus(ei, "cudaGraphInstantiate"));
                it = graphs.emplace(key, x).first;
            }
            CountLaunch(kernels);
            return CudaStatus(cudaGraphLaunch(it->second, s), "cudaGraphLaunch");
        }

        // `count` steps between the work fields, from work[c]; returns the
        // field's index.
        int RunPlain(int &c, int32_t count, const float *srcp, cudaStream_t s)
        {
            const int c0 = c;
            c ^= count & 1;
            const auto body = [&](cudaStream_t t)
            {
                int k = c0;
                for (int32_t i = 0; i < count; i++)
                {
                    HAL_TRY(LaunchFwd(work[k].p, work[k ^ 1].p, nullptr, nullptr, srcp, i > 0, t));
                    k ^= 1;
                }
                return static_cast<int>(HAL_CUDA_OK);
            };
            return Run("F" + std::to_string(c0) + "." + std::to_string(count) + (srcp ? "s" : ""), count, count, s, body);
        }

        // The states of `count` steps in buffer b, from its first field (fB
        // holds it by x).
        int RunStates(int b, int32_t count, const float *srcp, cudaStream_t s)
        {
            const auto body = [&](cudaStream_t t)
            {
                for (int32_t i = 0; i < count; i++)
                {
                    const size_t k = static_cast<size_t>(i);
                    HAL_TRY(LaunchFwd(segF[b].p + k * nA, segF[b].p + (k + 1) * nA, segW[b].p + k * nB,
                                      segV[b].p + k * nA, srcp, i > 0, t));
                }
                return static_cast<int>(HAL_CUDA_OK);
            };
            return Run("S" + std::to_string(b) + "." + std::to_string(count) + (srcp ? "s" : ""), count, count, s, body);
        }

        // Reverse steps over the `count` states in buffer b; g: the index of
        // the latest adjoint (0: gA, 1: gB).
        int RunBackward(int b, int32_t count, int &g, bool first, cudaStream_t s)
        {
            const int g0 = g;
            g ^= count & 1;
            const auto body = [&](cudaStream_t t)
            {
                int cur = g0;
                for (int32_t i = count - 1; i >= 0; i--)
                {
                    const size_t k = static_cast<size_t>(i);
                    const float *gc = cur == 0 ? gA.p : gB.p;
                    float *gn = cur == 0 ? gB.p : gA.p;
                    const bool lead = i == count - 1;
                    HAL_TRY(LaunchBwdY(first && lead ? kBwdFirst : kBwdNext, gc, segF[b].p + (k + 1) * nA,
                                       segV[b].p + k * nA, gn, !lead, t));
                    HAL_TRY(LaunchBwdX(segW[b].p + k * nB, t));
                    cur ^= 1;
                }
                return static_cast<int>(HAL_CUDA_OK);
            };
            return Run("B" + std::to_string(b) + "." + std::to_string(g0) + "." + std::to_string(count) +
                           (first ? "f" : ""),
                       first ? steps : count, count, s, body);
        }

        // A run of steps of two kernels each: whole segments (`repeated` as long
        // as a run that the call repeats) from a graph; runs that occur once in
        // a call (every state kept, the last segment) launch by launch, which
        // takes the host less than capturing them.
        template <typename Body>
        int Run(const std::string &key, int32_t repeated, int32_t count, cudaStream_t s, Body body)
        {
            if (repeated != Chunk())
            {
                return body(s);
            }
            return Replay(key, 2 * static_cast<int64_t>(count), s, body);
        }

        // Steps of a run that a call repeats.
        int32_t Chunk() const
        {
            return keepAll || Segments() <= 2 ? kPlainChunk : every;
        }
        static constexpr int32_t kPlainChunk = 16;  // a forward pass without checkpoints

        // Uploads a call's inputs and factors its lines (timed from begin).
        int Prepare(const float *hD, double decay, const float *hSrc, bool &useSrc, cudaEvent_t begin, cudaStream_t s)
        {
            HAL_TRY(ToDevice(D.p, hD, s, "cudaMemcpy(D)"));
            HAL_TRY(ByX(D.p, DT.p, s));
            useSrc = (hSrc != nullptr);
            if (useSrc)
            {
                HAL_TRY(ToDevice(src.p, hSrc, s, "cudaMemcpy(src)"));
            }
            const float hp[2] = {static_cast<float>(decay), static_cast<float>(-decay)};
            HAL_TRY(CudaStatus(cudaMemcpyAsync(par.p, hp, sizeof(hp), cudaMemcpyHostToDevice, s), "cudaMemcpy(decay)"));
            HAL_TRY(CudaStatus(cudaEventRecord(begin, s), "cudaEventRecord"));
            if (steps == 0)
            {
                return HAL_CUDA_OK;
            }
            // the axes side by side
            cudaStream_t rs = recomputeStream.Get();
            HAL_TRY(CudaStatus(cudaStreamWaitEvent(rs, begin, 0), "cudaStreamWaitEvent"));
            HAL_TRY(WithLaneLen(LaneLen(yDim), [&](auto m) {
                return LaunchChained(Factor<m()>, xDim, false, rs, axY, coefY.p, extY.p);
            }));
            HAL_TRY(CudaStatus(cudaEventRecord(factored, rs), "cudaEventRecord"));
            HAL_TRY(WithLaneLen(LaneLen(xDim), [&](auto m) {
                return LaunchChained(Factor<m()>, yDim, false, s, axX, coefX.p, extX.p);
            }));
            HAL_TRY(CudaStatus(cudaStreamWaitEvent(s, factored, 0), "cudaStreamWaitEvent"));
            CountLaunch(2);
            return HAL_CUDA_OK;
        }

        int LaunchLoss(const float *fT, float *gbar, cudaStream_t s)
        {
            const int64_t cells = static_cast<int64_t>(nA);
            LossGrad<<<LossParts(), kLossThreads, 0, s>>>(cells, fT, target.p, gbar, part.p);
            CountLaunch();
            return LaunchStatus("adjoint loss");
        }

        int LossParts() const
        {
            return static_cast<int>(
                std::min<int64_t>((static_cast<int64_t>(nA) + kLossThreads - 1) / kLossThreads, kLossBlocks));
        }

        int LaunchTotals(bool decayToo, cudaStream_t s)
        {
            Totals<<<1, decayToo ? 1024 : 256, 0, s>>>(part.p, LossParts(), dDecay.p, decayToo ? static_cast<int64_t>(xDim) * 32 : 0,
                                      acc.p);
            CountLaunch();
            return LaunchStatus("adjoint totals");
        }

        int EnqueueForward(bool useSrc, const float *&fT, cudaStream_t s)
        {
            HAL_TRY(CopyField(work[0].p, f0.p, s));
            HAL_TRY(ByX(f0.p, fB.p, s));
            int c = 0;
            for (int32_t t = 0; t < steps;)
            {
                const int32_t k = std::min(Chunk(), steps - t);
                HAL_TRY(RunPlain(c, k, useSrc ? src.p : nullptr, s));
                t += k;
            }
            fT = work[c].p;
            HAL_TRY(LaunchLoss(fT, nullptr, s));
            return LaunchTotals(false, s);
        }

        int RunForward(const float *hD, double decay, const float *hSrc, double *loss, float *hFT)
        {
            cudaStream_t s = stream.Get();
            bool useSrc = false;
            cudaEvent_t e0, e1;
            HAL_TRY(CudaStatus(cudaEventCreate(&e0), "cudaEventCreate"));
            HAL_TRY(CudaStatus(cudaEventCreate(&e1), "cudaEventCreate"));
            int rc = Prepare(hD, decay, hSrc, useSrc, e0, s);
            const float *fT = nullptr;
            if (rc == HAL_CUDA_OK)
            {
                rc = EnqueueForward(useSrc, fT, s);
            }
            cudaEventRecord(e1, s);
            double h[2] = {0, 0};
            if (rc == HAL_CUDA_OK)
            {
                rc = CudaStatus(cudaMemcpyAsync(h, acc.p, 2 * sizeof(double), cudaMemcpyDeviceToHost, s),
                                "cudaMemcpy(loss)");
            }
            if (rc == HAL_CUDA_OK && hFT != nullptr)
            {
                rc = ToHost(hFT, fT, s, "cudaMemcpy(f_T)");
            }
            if (rc == HAL_CUDA_OK)
            {
                rc = CudaStatus(cudaStreamSynchronize(s), "adjoint forward");
            }
            if (rc == HAL_CUDA_OK)
            {
                cudaEventElapsedTime(&msForward, e0, e1);
                *loss = h[0];
            }
            cudaEventDestroy(e0);
            cudaEventDestroy(e1);
            return rc;
        }

        // Events of a checkpointed gradient.
        struct Events
        {
            cudaEvent_t ready = nullptr, recDone[2] = {nullptr, nullptr}, bwdDone[2] = {nullptr, nullptr};

            int Create()
            {
                for (cudaEvent_t *e : {&ready, &recDone[0], &recDone[1], &bwdDone[0], &bwdDone[1]})
                {
                    HAL_TRY(CudaStatus(cudaEventCreateWithFlags(e, cudaEventDisableTiming), "cudaEventCreate"));
                }
                return HAL_CUDA_OK;
            }

            ~Events()
            {
                for (cudaEvent_t e : {ready, recDone[0], recDone[1], bwdDone[0], bwdDone[1]})
                {
                    if (e != nullptr)
                    {
                        cudaEventDestroy(e);
                    }
                }
            }
        };

        // Every state of the run kept: one forward pass, no recomputation.
        int EnqueueKept(const float *srcp, int &g, cudaStream_t s)
        {
            HAL_TRY(CopyField(segF[0].p, f0.p, s));
            HAL_TRY(ByX(f0.p, fB.p, s));
            HAL_TRY(RunStates(0, steps, srcp, s));
            HAL_TRY(LaunchLoss(segF[0].p + static_cast<size_t>(steps) * nA, gA.p, s));
            return steps > 0 ? RunBackward(0, steps, g, true, s) : static_cast<int>(HAL_CUDA_OK);
        }

        // Segments are differentiated last to first.  Segment s-1 is
        // recomputed from its checkpoint on a second stream into the other
        // buffer while segment s is differentiated; events order each
        // buffer's writer (recompute) and reader (backward).  The forward pass
        // keeps checkpoints, and writes the states of the last two segments
        // (one per buffer) as it goes, so the backward starts without waiting
        // for a recomputation.
        int EnqueueCheckpointed(const float *srcp, int &g, Events &ev, cudaStream_t s, cudaStream_t rs)
        {
            const int32_t S = Segments();
            const int32_t firstKept = std::max(S - 2, 0);
            const auto length = [&](int32_t seg) { return std::min(steps - seg * every, every); };
            HAL_TRY(CopyField(work[0].p, f0.p, s));
            HAL_TRY(ByX(f0.p, fB.p, s));
            const float *fCur = work[0].p;
            int c = 0;
            for (int32_t seg = 0; seg < S; seg++)
            {
                HAL_TRY(CopyField(ckpt.p + static_cast<size_t>(seg) * nA, fCur, s));
                if (seg >= firstKept)
                {
                    HAL_TRY(CopyField(segF[seg & 1].p, fCur, s));
                    HAL_TRY(RunStates(seg & 1, length(seg), srcp, s));
                    fCur = segF[seg & 1].p + static_cast<size_t>(length(seg)) * nA;
                }
                else
                {
                    HAL_TRY(RunPlain(c, every, srcp, s));
                    fCur = work[c].p;
                }
            }
            HAL_TRY(LaunchLoss(fCur, gA.p, s));
            // the checkpoints are written by the forward pass on s
            HAL_TRY(CudaStatus(cudaEventRecord(ev.ready, s), "cudaEventRecord"));
            HAL_TRY(CudaStatus(cudaStreamWaitEvent(rs, ev.ready, 0), "cudaStreamWaitEvent"));
            for (int32_t seg = S - 1; seg >= 0; seg--)
            {
                const int32_t next = seg - 1;
                if (next >= 0 && next < firstKept)
                {
                    // the buffer's previous reader is the backward of segment next+2
                    const int b = next & 1;
                    HAL_TRY(CudaStatus(cudaStreamWaitEvent(rs, ev.bwdDone[b], 0), "cudaStreamWaitEvent"));
                    HAL_TRY(CopyField(segF[b].p, ckpt.p + static_cast<size_t>(next) * nA, rs));
                    HAL_TRY(ByX(segF[b].p, fB.p, rs));
                    HAL_TRY(RunStates(b, every, srcp, rs));
                    HAL_TRY(CudaStatus(cudaEventRecord(ev.recDone[b], rs), "cudaEventRecord"));
                }
                const int b = seg & 1;
                if (seg < firstKept)
                {
                    HAL_TRY(CudaStatus(cudaStreamWaitEvent(s, ev.recDone[b], 0), "cudaStreamWaitEvent"));
                }
                HAL_TRY(RunBackward(b, length(seg), g, seg == S - 1, s));
                HAL_TRY(CudaStatus(cudaEventRecord(ev.bwdDone[b], s), "cudaEventRecord"));
            }
            return HAL_CUDA_OK;
        }

        int EnqueueGradient(bool useSrc, Events &ev, cudaStream_t s)
        {
            HAL_TRY(CudaStatus(cudaMemsetAsync(dD.p, 0, nA * sizeof(float), s), "cudaMemset(dD)"));
            HAL_TRY(CudaStatus(cudaMemsetAsync(dDT.p, 0, nB * sizeof(float), s), "cudaMemset(dD)"));
            HAL_TRY(CudaStatus(cudaMemsetAsync(dS.p, 0, nA * sizeof(float), s), "cudaMemset(dS)"));
            HAL_TRY(CudaStatus(cudaMemsetAsync(dDecay.p, 0, static_cast<size_t>(xDim) * 32 * sizeof(double), s),
                               "cudaMemset(dDecay)"));
            const float *srcp = useSrc ? src.p : nullptr;
            int g = 0;
            if (keepAll)
            {
                HAL_TRY(EnqueueKept(srcp, g, s));
            }
            else
            {
                HAL_TRY(EnqueueCheckpointed(srcp, g, ev, s, recomputeStream.Get()));
            }
            if (steps > 0)
            {
                // the y-stencil part of step 0's (I + Ly/2) b1bar: its D terms
                // (buffer 0 holds segment 0's states)
                HAL_TRY(LaunchBwdY(kBwdTail, g == 0 ? gA.p : gB.p, segF[0].p, segV[0].p, g == 0 ? gB.p : gA.p, false,
                                   s));
            }
            // the x-faces' part of dL/dD
            TransposeRows<true><<<dim3((yDim + 31) / 32, (xDim + 31) / 32), dim3(32, 8), 0, s>>>(dDT.p, ldX, dD.p, ldY,
                                                                                                 yDim, xDim);
            CountLaunch();
            HAL_TRY(LaunchStatus("adjoint dD"));
            return LaunchTotals(true, s);
        }

        int RunGradient(const float *hD, double decay, const float *hSrc, double *loss, float *hgD, double *hgK,
                        float *hgS)
        {
            cudaStream_t s = stream.Get();
            bool useSrc = false;
            cudaEvent_t e0, e1;
            HAL_TRY(CudaStatus(cudaEventCreate(&e0), "cudaEventCreate"));
            HAL_TRY(CudaStatus(cudaEventCreate(&e1), "cudaEventCreate"));
            Events ev;
            int rc = ev.Create();
            if (rc == HAL_CUDA_OK)
            {
                rc = Prepare(hD, decay, hSrc, useSrc, e0, s);
            }
            if (rc == HAL_CUDA_OK)
            {
                rc = EnqueueGradient(useSrc, ev, s);
            }
            if (rc != HAL_CUDA_OK)
            {
                // s follows every recomputation only when all of it was enqueued
                cudaStreamSynchronize(recomputeStream.Get());
            }
            cudaEventRecord(e1, s);
            double h[2] = {0, 0};
            if (rc == HAL_CUDA_OK)
            {
                rc = CudaStatus(cudaMemcpyAsync(h, acc.p, 2 * sizeof(double), cudaMemcpyDeviceToHost, s),
                                "cudaMemcpy(loss)");
            }
            if (rc == HAL_CUDA_OK && hgD != nullptr)
            {
                rc = ToHost(hgD, dD.p, s, "cudaMemcpy(dD)");
            }
            if (rc == HAL_CUDA_OK && hgS != nullptr)
            {
                rc = ToHost(hgS, dS.p, s, "cudaMemcpy(dS)");
            }
            if (rc == HAL_CUDA_OK)
            {
                rc = CudaStatus(cudaStreamSynchronize(s), "adjoint gradient");
            }
            if (rc == HAL_CUDA_OK)
            {
                cudaEventElapsedTime(&msGradient, e0, e1);
                *loss = h[0];
                if (hgK != nullptr)
                {
                    *hgK = h[1];
                }
            }
            cudaEventDestroy(e0);
            cudaEventDestroy(e1);
            return rc;
        }
    };
}

using halcuda::Adjoint;

struct hal_cuda_adjoint : public Adjoint
{
};

extern "C" int hal_cuda_adjoint_create(int32_t xDim, int32_t yDim, int32_t wrapX, int32_t wrapY,
                                       hal_cuda_adjoint **out)
{
    HAL_REQUIRE(out != nullptr, "hal_cuda_adjoint_create: out is NULL");
    *out = nullptr;
    HAL_REQUIRE(xDim >= 1 && yDim >= 1 && xDim <= halcuda::kMaxAdjLine && yDim <= halcuda::kMaxAdjLine,
                "hal_cuda_adjoint_create: grid %d x %d, sides must be in [1, %d]", xDim, yDim, halcuda::kMaxAdjLine);
    hal_cuda_adjoint *h = new (std::nothrow) hal_cuda_adjoint();
    if (h == nullptr)
    {
        halcuda::SetError("hal_cuda_adjoint_create: out of host memory");
        return HAL_CUDA_ENOMEM;
    }
    int rc = h->Init(xDim, yDim, wrapX, wrapY);
    if (rc != HAL_CUDA_OK)
    {
        delete h;
        return rc;
    }
    *out = h;
    return HAL_CUDA_OK;
}

extern "C" int hal_cuda_adjoint_destroy(hal_cuda_adjoint *h)
{
    if (h != nullptr)
    {
        cudaSetDevice(h->device);
        cudaStreamSynchronize(h->stream.Get());
        cudaStreamSynchronize(h->recomputeStream.Get());
        delete h;
    }
    return HAL_CUDA_OK;
}

extern "C" int hal_cuda_adjoint_set_problem(hal_cuda_adjoint *h, const float *f0, const float *target, int64_t len,
                                            int32_t steps, int32_t checkpointEvery)
{
    HAL_REQUIRE(h != nullptr && f0 != nullptr && target != nullptr, "hal_cuda_adjoint_set_problem: NULL argument");
    HAL_REQUIRE(len == h->n, "hal_cuda_adjoint_set_problem: length %lld, grid holds %lld cells",
                static_cast<long long>(len), static_cast<long long>(h->n));
    HAL_REQUIRE(steps >= 0, "hal_cuda_adjoint_set_problem: negative step count");
    HAL_REQUIRE(checkpointEvery >= 0, "hal_cuda_adjoint_set_problem: negative checkpoint interval");
    using namespace halcuda;
    HAL_TRY(CudaStatus(cudaSetDevice(h->device), "cudaSetDevice"));
    // (a call that failed may have left work in flight)
    HAL_TRY(CudaStatus(cudaStreamSynchronize(h->stream.Get()), "hal_cuda_adjoint_set_problem"));
    h->DropGraphs();
    h->hasProblem = false;
    h->steps = steps;
    h->keepAll = (checkpointEvery == 0);
    h->every = h->keepAll ? std::max(steps, 1) : std::min(checkpointEvery, std::max(steps, 1));
    HAL_TRY(h->ckpt.Alloc(h->nA * static_cast<size_t>(std::max(h->Segments(), 1)), "cudaMalloc(checkpoints)"));
    // one segment buffer when every state is kept or there is one segment,
    // two (recompute of one overlapping the backward of the other) otherwise
    const int nBuf = (h->keepAll || h->Segments() <= 1) ? 1 : 2;
    for (int b = 0; b < 2; b++)
    {
        if (b < nBuf)
        {
            // (whole arrays are written before they are read, padding included)
            HAL_TRY(h->segF[b].Alloc(h->nA * static_cast<size_t>(h->every + 1), "cudaMalloc(segment)"));
            HAL_TRY(h->segW[b].Alloc(h->nB * static_cast<size_t>(h->every), "cudaMalloc(segment)"));
            HAL_TRY(h->segV[b].Alloc(h->nA * static_cast<size_t>(h->every), "cudaMalloc(segment)"));
        }
        else
        {
            h->segF[b].Free();
            h->segW[b].Free();
            h->segV[b].Free();
        }
    }
    cudaStream_t s = h->stream.Get();
    HAL_TRY(h->ToDevice(h->f0.p, f0, s, "cudaMemcpy(f0)"));
    HAL_TRY(h->ToDevice(h->target.p, target, s, "cudaMemcpy(target)"));
    HAL_TRY(CudaStatus(cudaStreamSynchronize(s), "hal_cuda_adjoint_set_problem"));
    h->hasProblem = true;
    return HAL_CUDA_OK;
}

extern "C" int hal_cuda_adjoint_forward(hal_cuda_adjoint *h, const float *D, double decay, const float *src,
                                        double *loss, float *fT)
{
    HAL_TRACE();
    HAL_REQUIRE(h != nullptr && D != nullptr && loss != nullptr, "hal_cuda_adjoint_forward: NULL argument");
    HAL_REQUIRE(h->hasProblem, "hal_cuda_adjoint_forward: call hal_cuda_adjoint_set_problem first");
    HAL_REQUIRE(std::isfinite(decay), "hal_cuda_adjoint_forward: decay %g", decay);
    HAL_TRY(halcuda::CudaStatus(cudaSetDevice(h->device), "cudaSetDevice"));
    return h->RunForward(D, decay, src, loss, fT);
}

extern "C" int hal_cuda_adjoint_gradient(hal_cuda_adjoint *h, const float *D, double decay, const float *src,
                                         double *loss, float *gradD, double *gradDecay, float *gradSrc)
{
    HAL_TRACE();
    HAL_REQUIRE(h != nullptr && D != nullptr && loss != nullptr, "hal_cuda_adjoint_gradient: NULL argument");
    HAL_REQUIRE(h->hasProblem, "hal_cuda_adjoint_gradient: call hal_cuda_adjoint_set_problem first");
    HAL_REQUIRE(std::isfinite(decay), "hal_cuda_adjoint_gradient: decay %g", decay);
    HAL_TRY(halcuda::CudaStatus(cudaSetDevice(h->device), "cudaSetDevice"));
    return h->RunGradient(D, decay, src, loss, gradD, gradDecay, gradSrc);
}

extern "C" int hal_cuda_adjoint_times(hal_cuda_adjoint *h, float *msForward, float *msGradient)
{
    HAL_REQUIRE(h != nullptr && msForward != nullptr && msGradient != nullptr, "hal_cuda_adjoint_times: NULL argument");
    *msForward = h->msForward;
    *msGradient = h->msGradient;
    return HAL_CUDA_OK;
}
