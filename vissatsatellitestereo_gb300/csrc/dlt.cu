// (a)+(b) RPC projection and the RPC -> perspective fit:
//   RPCModel.projection        lib/rpc_model.py:160-168
//   solve_perspective          lib/solve_perspective.py:82-126  (+ factorize :38-79)
//   check_perspective_error    lib/check_error.py:37-121
//   the per-view loop          camera_approx.py:166-189
//
// The fit solves the reference's problem -- the unit vector p minimising |A p| for the
// 2N x 12 DLT matrix A -- without forming A.  A^T A only depends on 40 point moments
// (sum X X^T weighted by 1, c, r, c^2 + r^2 with X = [x y z 1]), so one streaming pass
// accumulates them in coordinates centred and scaled per view (FP32 sums over at most 16
// points per thread and across a warp, FP64 beyond).  The 12x12 problem is then solved in
// FP64 by inverse iteration on the normalised Gram matrix, with the centring/scaling map M
// applied exactly, so the minimiser is the reference's un-normalised one.  Factorisation is
// a positive-diagonal RQ (Gram-Schmidt from the last row), which is unique and equals the
// reference's sign-fixed scipy RQ.
//
// GB300 executes FP64 arithmetic, FP64 compares and every conversion instruction on a
// narrow pipe (~1/64 of FP32), so the per-point passes use integer bit manipulation for
// conversions and double-float (two-FP32) arithmetic where FP32 is not accurate enough.
#include <algorithm>
#include <math.h>

#include "common.cuh"
#include "rpc.cuh"

namespace vs {
namespace {

// ---------------------------------------------------------------------------------------
// (a) projection
// ---------------------------------------------------------------------------------------
// A block's camera in shared memory, by arithmetic.
template <int MODE>
struct CameraOf {
    using type = RpcFast;
};
template <>
struct CameraOf<VS_PROJ_EXACT> {
    using type = RpcExact;
};

template <int MODE>
__global__ void __launch_bounds__(256) rpc_project_kernel(const VsRpcCamera *__restrict__ cams,
                                                          const double *__restrict__ lat,
                                                          const double *__restrict__ lon,
                                                          const double *__restrict__ alt, long long n,
                                                          long long stride, double *__restrict__ col,
                                                          double *__restrict__ row,
                                                          uint8_t *__restrict__ keep) {
    constexpr bool kExact = MODE == VS_PROJ_EXACT;
    __shared__ typename CameraOf<MODE>::type cam;
    const int c = blockIdx.y;
    if constexpr (kExact) load_exact(cams + c, cam);
    else prepare_fast(cams[c], cam);
    const double *la = lat + c * stride, *lo = lon + c * stride, *al = alt + c * stride;
    double *oc = col + c * n, *orow = row + c * n;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        double cc, rr;
        bool k;
        if constexpr (kExact) {
            project_exact(cam, __ldcs(la + i), __ldcs(lo + i), __ldcs(al + i), cc, rr);
            k = cc >= 0.0 && rr >= 0.0 && cc < cam.cam.width && rr < cam.cam.height;
        } else {
            df dc, dr;
            project_fast(cam, split_double(__ldcs(la + i)), split_double(__ldcs(lo + i)),
                         split_double(__ldcs(al + i)), dc, dr);
            cc = df_to_double(dc);
            rr = df_to_double(dr);
            k = df_ge0(dc) && df_ge0(dr) && df_lt(dc, cam.width) && df_lt(dr, cam.height);
        }
        __stcs(oc + i, cc);
        __stcs(orow + i, rr);
        if (keep) keep[c * n + i] = k;
    }
}

// ---------------------------------------------------------------------------------------
// (b) fit: normalisation, moments, solve
// ---------------------------------------------------------------------------------------
// Per-view normalisation: X' = (X - centre) / s, c' = (col - c0) / sp, r' = (row - r0) / sp
struct Norm {
    double cx, cy, cz, s, c0, r0, sp;
};

// Points sampled per view for the normalisation box: each sample costs a DRAM sector per
// coordinate array, and 8192 of them bound the data's extent well enough for scaling.
constexpr int kBoxSamples = 8192;

__device__ __forceinline__ double finite_or(double v, double fallback) {
    return (isfinite(v)) ? v : fallback;
}

// Per-view normalisation in the forms the per-point kernels use.
struct NormF {
    df cx, cy, cz, inv_s, c0, r0, inv_sp;
    float sp;
};

__device__ __forceinline__ NormF make_normf(const Norm &nm) {
    NormF f;
    f.cx = df_from_double(nm.cx);
    f.cy = df_from_double(nm.cy);
    f.cz = df_from_double(nm.cz);
    f.inv_s = df_from_double(1.0 / nm.s);
    f.c0 = df_from_double(nm.c0);
    f.r0 = df_from_double(nm.r0);
    f.inv_sp = df_from_double(1.0 / nm.sp);
    f.sp = static_cast<float>(nm.sp);
    return f;
}

// Normalisation of one view from its sampled box.  For the fused camera path the pixel frame
// is the RPC's own (colOff/rowOff, larger scale).
__device__ __forceinline__ void make_norm(const unsigned long long *b, const VsRpcCamera *cam, Norm &nm) {
    double mx[5], mn[5];
    for (int j = 0; j < 5; ++j) {
        mx[j] = b[j] ? double_from_key(b[j]) : 0.0;
        mn[j] = b[5 + j] ? double_from_key(~b[5 + j]) : 0.0;
    }
    nm.cx = finite_or(0.5 * (mn[0] + mx[0]), 0.0);
    nm.cy = finite_or(0.5 * (mn[1] + mx[1]), 0.0);
    nm.cz = finite_or(0.5 * (mn[2] + mx[2]), 0.0);
    double s = fmax(fmax(mx[0] - mn[0], mx[1] - mn[1]), mx[2] - mn[2]) * 0.5;
    nm.s = (s > 0.0 && isfinite(s)) ? s : 1.0;
    if (cam) {
        nm.c0 = cam->col_off;
        nm.r0 = cam->row_off;
        nm.sp = fmax(fabs(cam->col_scale), fabs(cam->row_scale));
        if (!(nm.sp > 0.0) || !isfinite(nm.sp)) nm.sp = 1.0;
    } else {
        nm.c0 = finite_or(0.5 * (mn[3] + mx[3]), 0.0);
        nm.r0 = finite_or(0.5 * (mn[4] + mx[4]), 0.0);
        double sp = fmax(mx[3] - mn[3], mx[4] - mn[4]) * 0.5;
        nm.sp = (sp > 0.0 && isfinite(sp)) ? sp : 1.0;
    }
}

// The box of one view: order-preserving keys of the largest values, then of the smallest (the
// keys' complements), and the number of blocks that have added theirs.  All zero to begin with.
struct Box {
    unsigned long long key[10];
    unsigned done, pad;
};

// Min/max of x, y, z (and col, row when given) over a strided sample of the kept points, and
// from them the view's normalisation: any centre and scale serve, it only has to keep the
// moments well scaled.  The last block of a view to add its box computes the normalisation, which was
// a launch of its own.  (50 views: 35 us of strided sectors; neither fewer blocks, nor one atomic per
// block, nor four samples in flight per thread changes that.)
__global__ void __launch_bounds__(256) bbox_kernel(const double *__restrict__ x, const double *__restrict__ y,
                                                   const double *__restrict__ z, long long xyz_stride,
                                                   const double *__restrict__ col, const double *__restrict__ row,
                                                   const uint8_t *__restrict__ keep, long long n, long long step,
                                                   const VsRpcCamera *__restrict__ cams, Box *__restrict__ boxes,
                                                   Norm *__restrict__ norm, NormF *__restrict__ normf) {
    __shared__ unsigned long long best[10];
    chain_wait();
    const int v = blockIdx.y;
    const double *src[5] = {x + v * xyz_stride, y + v * xyz_stride, z + v * xyz_stride, col ? col + v * n : nullptr,
                            row ? row + v * n : nullptr};
    if (threadIdx.x < 10) best[threadIdx.x] = 0ull;
    __syncthreads();
    unsigned long long hi[5], lo[5];
#pragma unroll
    for (int j = 0; j < 5; ++j) hi[j] = lo[j] = 0ull;
    for (long long i = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) * step; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x * step) {
        if (keep && !keep[v * n + i]) continue;
#pragma unroll
        for (int j = 0; j < 5; ++j) {
            if (!src[j]) continue;
            const unsigned long long k = key_from_double(src[j][i]);
            hi[j] = max(hi[j], k);
            lo[j] = max(lo[j], ~k);
        }
    }
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        if (!src[j]) continue;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            hi[j] = max(hi[j], __shfl_xor_sync(0xffffffffu, hi[j], off));
            lo[j] = max(lo[j], __shfl_xor_sync(0xffffffffu, lo[j], off));
        }
        if ((threadIdx.x & 31) == 0) {
            atomicMax(best + j, hi[j]);
            atomicMax(best + 5 + j, lo[j]);
        }
    }
    __syncthreads();
    Box &box = boxes[v];
    if (threadIdx.x < 10 && best[threadIdx.x]) {
        atomicMax(box.key + threadIdx.x, best[threadIdx.x]);
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(&box.done, 1u) != gridDim.x - 1) return;
    __threadfence();
    unsigned long long k[10];
    for (int j = 0; j < 10; ++j) k[j] = atomicAdd(box.key + j, 0ull);
    Norm nm;
    make_norm(k, cams ? cams + v : nullptr, nm);
    norm[v] = nm;
    normf[v] = make_normf(nm);     // once per view: the per-point kernels read it (no FP64 there)
}

constexpr int kMom = 40;            // 4 weights x 10 unique entries of X X^T
constexpr int kSlots = 41;          // + kept-point count
constexpr int kMomThreads = 128;
constexpr int kChunk = 16;          // points per thread (FP32 partial sums)

// Accumulates one point's 40 moment terms into FP32 partial sums held as FP32x2 pairs:
// ma[k] = (m[k], m[10 + k]) with weights (1, c), mb[k] = (m[20 + k], m[30 + k]) with
// weights (r, c^2 + r^2) -- one FFMA2 per pair; 1 * e + m is exactly the plain sum, so
// every lane rounds as the scalar accumulation does.
__device__ __forceinline__ void add_moments(float2 (&ma)[10], float2 (&mb)[10], float x, float y, float z, float c,
                                            float r) {
    const float xx = x * x, xy = x * y, xz = x * z, yy = y * y, yz = y * z, zz = z * z;
    const float e[10] = {xx, xy, xz, x, yy, yz, y, zz, z, 1.0f};
    const float2 wa = make_float2(1.0f, c), wb = make_float2(r, __fmaf_rn(c, c, r * r));
#pragma unroll
    for (int k = 0; k < 10; ++k) {
        const float2 ek = make_float2(e[k], e[k]);
        ma[k] = __ffma2_rn(wa, ek, ma[k]);
        mb[k] = __ffma2_rn(wb, ek, mb[k]);
    }
}

// Warp sums in FP32, warps combined in FP64 in a fixed order (deterministic):
// partial[kSlots] of this block.
__device__ __forceinline__ void store_block_moments(float (&m)[kMom], float count, double *partial, double *red) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // moments 0..31: a reduce-scatter -- at the step of offset h a lane keeps the half of
    // its remaining sums selected by lane bit h and adds its partner's copy of that half --
    // so lane l ends with the warp sum of moment l after 31 shuffles instead of 160.  Each
    // sum is formed as own + partner's at every step, as the butterfly below forms it, so
    // the values are the butterfly's bit for bit.
#pragma unroll
    for (int h = 16; h > 0; h >>= 1) {
        const bool up = (lane & h) != 0;
#pragma unroll
        for (int j = 0; j < h; ++j) {
            const float send = up ? m[j] : m[j + h];
            const float keep = up ? m[j + h] : m[j];
            m[j] = keep + __shfl_xor_sync(0xffffffffu, send, h);
        }
    }
    // moments 32..39 and the count: butterflies (every lane ends with the sum)
#pragma unroll
    for (int k = 32; k < kMom; ++k)
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) m[k] += __shfl_xor_sync(0xffffffffu, m[k], off);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) count += __shfl_xor_sync(0xffffffffu, count, off);
    red[warp * kSlots + lane] = f32_to_f64(m[0]);
    if (lane == 0) {
#pragma unroll
        for (int k = 32; k < kMom; ++k) red[warp * kSlots + k] = f32_to_f64(m[k]);
        red[warp * kSlots + kMom] = f32_to_f64(count);
    }
    __syncthreads();
    if (threadIdx.x < kSlots) {
        double s = 0.0;
        for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) s += red[w * kSlots + threadIdx.x];
        partial[threadIdx.x] = s;
    }
}

// Normalised coordinates of one kept point from FP64 ENU and double-float pixels (FP32 is
// enough here: the rounding acts like data noise of ~1e-4 px that the fit averages out).
__device__ __forceinline__ void normalised_point(const NormF &nf, long long X, long long Y, long long Z, df c, df r,
                                                 float &px, float &py, float &pz, float &pc, float &pr) {
    const df x = split_double(__longlong_as_double(X)), y = split_double(__longlong_as_double(Y)),
             z = split_double(__longlong_as_double(Z));
    px = ((x.hi - nf.cx.hi) + (x.lo - nf.cx.lo)) * nf.inv_s.hi;
    py = ((y.hi - nf.cy.hi) + (y.lo - nf.cy.lo)) * nf.inv_s.hi;
    pz = ((z.hi - nf.cz.hi) + (z.lo - nf.cz.lo)) * nf.inv_s.hi;
    pc = ((c.hi - nf.c0.hi) + (c.lo - nf.c0.lo)) * nf.inv_sp.hi;
    pr = ((r.hi - nf.r0.hi) + (r.lo - nf.r0.lo)) * nf.inv_sp.hi;
}

// A block's next contiguous span of an array, on its way to L2 (16-byte pieces only).
__device__ __forceinline__ void prefetch_l2(const void *p, long long bytes) {
    bytes &= ~15ll;
    if (bytes > 0 && (reinterpret_cast<unsigned long long>(p) & 15) == 0)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(static_cast<unsigned>(bytes)) : "memory");
}

// Moments of the kept points of view v.  Block b owns points [b * 128 * kChunk, ...);
// (col, row) come as FP64 arrays (drop-in fit) or as the double-floats of the projection
// pass (fused camera path, in-image mask from the image size).
//
// Latency-bound: 40 bytes and 200 instructions per point, and 80 accumulators and inputs per thread
// leave 20 warps per SM.  So one thread sends the block's 80 KB on its way to L2 at the start, and
// each thread loads its next two points before it adds the current two.  50 x 800,000 points (1.6 GB,
// 240 us of HBM time): 400 us with the loads at the head of each group, 336 us so.  (Of the whole fit's
// 1996 us the prefetch alone takes off 46, two points ahead alone 43, both 67; one point ahead at six
// blocks per SM, with the prefetch, 61.)
__global__ void __launch_bounds__(kMomThreads, 5) moments_kernel(
    const double *__restrict__ x, const double *__restrict__ y, const double *__restrict__ z, long long xyz_stride,
    const double *__restrict__ col, const double *__restrict__ row, const float4 *__restrict__ colrow,
    const uint8_t *__restrict__ keep, const float *__restrict__ wh, long long n, const NormF *__restrict__ normf,
    double *__restrict__ partial) {
    __shared__ double red[(kMomThreads / 32) * kSlots];
    chain_wait();
    const int v = blockIdx.y;
    const NormF nf = normf[v];
    const double *xv = x + v * xyz_stride, *yv = y + v * xyz_stride, *zv = z + v * xyz_stride;
    const float w = wh ? wh[2 * v] : 0.f, h = wh ? wh[2 * v + 1] : 0.f;
    float2 ma[10], mb[10];
#pragma unroll
    for (int k = 0; k < 10; ++k) ma[k] = mb[k] = make_float2(0.0f, 0.0f);
    float count = 0.0f;
    const long long base = static_cast<long long>(blockIdx.x) * kMomThreads * kChunk + threadIdx.x;
    if (threadIdx.x == 0) {
        const long long cnt = min(static_cast<long long>(kMomThreads * kChunk), n - base);
        prefetch_l2(xv + base, 8 * cnt);
        prefetch_l2(yv + base, 8 * cnt);
        prefetch_l2(zv + base, 8 * cnt);
        if (colrow) {
            prefetch_l2(colrow + static_cast<long long>(v) * n + base, 16 * cnt);
        } else {
            prefetch_l2(col + v * n + base, 8 * cnt);
            prefetch_l2(row + v * n + base, 8 * cnt);
        }
    }
    constexpr int kAhead = 2;
    // coordinates as raw 64-bit patterns: double-typed registers would be moved and
    // selected by FP64 instructions, which GB300 runs on a narrow pipe
    long long X[kAhead], Y[kAhead], Z[kAhead];
    float4 cr[kAhead];
    unsigned kp[kAhead];
    auto load = [&](int j0) {
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const long long i = base + static_cast<long long>(j0 + u) * kMomThreads;
            kp[u] = 0;
            X[u] = Y[u] = Z[u] = 0;
            cr[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (j0 + u < kChunk && i < n) {
                X[u] = __ldg(reinterpret_cast<const long long *>(xv) + i);
                Y[u] = __ldg(reinterpret_cast<const long long *>(yv) + i);
                Z[u] = __ldg(reinterpret_cast<const long long *>(zv) + i);
                if (colrow) {
                    cr[u] = colrow[static_cast<long long>(v) * n + i];
                    kp[u] = 1;
                } else {
                    kp[u] = !keep || keep[v * n + i];
                    const df c = split_double(col[v * n + i]), r = split_double(row[v * n + i]);
                    cr[u] = make_float4(c.hi, c.lo, r.hi, r.lo);
                }
            }
        }
    };
    load(0);
#pragma unroll 1
    for (int j0 = 0; j0 < kChunk; j0 += kAhead) {
        float px[kAhead], py[kAhead], pz[kAhead], pc[kAhead], pr[kAhead];
        bool ok[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const df c = {cr[u].x, cr[u].y}, r = {cr[u].z, cr[u].w};
            ok[u] = kp[u] && (!colrow || (df_ge0(c) && df_ge0(r) && df_lt(c, w) && df_lt(r, h)));
            normalised_point(nf, X[u], Y[u], Z[u], c, r, px[u], py[u], pz[u], pc[u], pr[u]);
        }
        load(j0 + kAhead);
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            if (!ok[u]) continue;
            add_moments(ma, mb, px[u], py[u], pz[u], pc[u], pr[u]);
            count += 1.0f;
        }
    }
    float m[kMom];
#pragma unroll
    for (int k = 0; k < 10; ++k) {
        m[k] = ma[k].x;
        m[10 + k] = ma[k].y;
        m[20 + k] = mb[k].x;
        m[30 + k] = mb[k].y;
    }
    store_block_moments(m, count, partial + (static_cast<long long>(v) * gridDim.x + blockIdx.x) * kSlots, red);
}

// Double-float form of every view's camera, prepared once per call (one block per view)
// rather than by every projection block.
__global__ void __launch_bounds__(64) prepare_views_kernel(const VsRpcCamera *__restrict__ cams,
                                                           RpcFast *__restrict__ fast, float *__restrict__ wh) {
    const int v = blockIdx.x;
    chain_wait();
    prepare_fast(cams[v], fast[v]);
    if (threadIdx.x == 0) {
        wh[2 * v] = fast[v].width;
        wh[2 * v + 1] = fast[v].height;
    }
}

// Projection pass of the fused camera path: (col, row) of every grid point through view
// v's RPC camera as double-floats.
template <int MODE>
__global__ void __launch_bounds__(256) project_view_kernel(const VsRpcCamera *__restrict__ cams,
                                                           const RpcFast *__restrict__ fasts,
                                                           const double *__restrict__ lat,
                                                           const double *__restrict__ lon,
                                                           const double *__restrict__ alt, long long n,
                                                           long long stride, float4 *__restrict__ colrow) {
    constexpr bool kExact = MODE == VS_PROJ_EXACT;
    __shared__ typename CameraOf<MODE>::type cam;
    const int v = blockIdx.y;
    chain_wait();
    if constexpr (kExact) {
        load_exact(cams + v, cam);
    } else {
        const unsigned *src = reinterpret_cast<const unsigned *>(fasts + v);
        unsigned *dst = reinterpret_cast<unsigned *>(&cam);
        for (int i = threadIdx.x; i < static_cast<int>(sizeof(RpcFast) / 4); i += blockDim.x) dst[i] = src[i];
        __syncthreads();
    }
    const long long off = v * stride;
    const long long step = static_cast<long long>(gridDim.x) * blockDim.x;
    // the next point's coordinates (raw 64-bit patterns) are loaded before the current
    // point's few hundred instructions, so their latency is hidden behind them
    const long long *la = reinterpret_cast<const long long *>(lat + off);
    const long long *lo = reinterpret_cast<const long long *>(lon + off);
    const long long *al = reinterpret_cast<const long long *>(alt + off);
    long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    long long a0 = 0, a1 = 0, a2 = 0;
    if (i < n) {
        a0 = __ldcs(la + i);
        a1 = __ldcs(lo + i);
        a2 = __ldcs(al + i);
    }
    for (; i < n; i += step) {
        long long b0 = 0, b1 = 0, b2 = 0;
        if (i + step < n) {
            b0 = __ldcs(la + i + step);
            b1 = __ldcs(lo + i + step);
            b2 = __ldcs(al + i + step);
        }
        df dc, dr;
        if constexpr (kExact) {
            double cc, rr;
            project_exact(cam, __longlong_as_double(a0), __longlong_as_double(a1), __longlong_as_double(a2), cc, rr);
            dc = split_double(cc);
            dr = split_double(rr);
        } else {
            project_fast(cam, split_double(__longlong_as_double(a0)), split_double(__longlong_as_double(a1)),
                         split_double(__longlong_as_double(a2)), dc, dr);
        }
        colrow[static_cast<long long>(v) * n + i] = make_float4(dc.hi, dc.lo, dr.hi, dr.lo);
        a0 = b0;
        a1 = b1;
        a2 = b2;
    }
}

// ---- 12x12 solve (one warp per view; FP64) ---------------------------------------------
// The exact map M between normalised (q) and original (p) camera vectors: q1 = T^T(p1 - c0
// p3)/sp, q2 = T^T(p2 - r0 p3)/sp, q3 = T^T p3, T = [[s,0,0,cx],[0,s,0,cy],[0,0,s,cz],[0,0,0,1]].
//
// One warp: FP64 latency and divisions are all of its time, so lane l < 12 holds component l of the
// vectors (component i = l mod 4 of row b = l / 4) and row l of the factor, and the divisions,
// which were one after the other in one lane, run side by side; those by a pivot or a scale, which
// repeat each iteration, use its reciprocal (div_known: 4 operations, the same bits).  Every
// element sees the operations of the serial form in its order.  One view: 175 us, 95 us, most of it
// FP64 latency (59 cycles an operation, 600 a division or square root).

// A divisor and whether its quotients may take the reciprocal form.
struct LaneDivisor {
    Divisor d;
    bool known;
};
// Exponent within 2^+-160 (no zero): div_known has the bits of the division.
__device__ __forceinline__ bool mid_range(double v) {
    return ((static_cast<unsigned>(__double2hiint(v)) >> 20) & 0x7ffu) - (1023u - 160u) <= 320u;
}
__device__ __forceinline__ LaneDivisor lane_divisor(double v) {
    LaneDivisor r;
    r.known = mid_range(v);
    r.d = divisor_of(v);
    return r;
}
__device__ __forceinline__ double lane_div(double v, const LaneDivisor &d) {
    if (__all_sync(0xffffffffu, d.known && mid_range(v))) return div_known(v, d.d);
    return __ddiv_rn(v, d.d.d);
}
__device__ __forceinline__ double lane_get(double v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }

// u = M^-T v, component by component: rows 0 and 1 are sp T^-1 v_b, row 2 is T^-1 (v_2 + c0 v_0 + r0 v_1).
__device__ __forceinline__ double solve_mt(const Norm &m, const LaneDivisor &ds, int b, int i, double v) {
    const double v0 = lane_get(v, i), v1 = lane_get(v, 4 + i);
    const double t0 = lane_get(v, 3), t1 = lane_get(v, 7), t2 = lane_get(v, 11);
    const double wi = b < 2 ? v : __fma_rn(m.r0, v1, __fma_rn(m.c0, v0, v));
    const double w3 = b == 0 ? t0 : (b == 1 ? t1 : __fma_rn(m.r0, t1, __fma_rn(m.c0, t0, t2)));
    const double c = i == 0 ? m.cx : (i == 1 ? m.cy : m.cz);
    const double q = lane_div(__fma_rn(-c, w3, wi), ds);
    const double u = i < 3 ? q : wi;
    return b < 2 ? __dmul_rn(u, m.sp) : u;
}
// u = M^-1 v: row 2 is T^-T v_2, rows 0 and 1 are T^-T (sp v_b + {c0, r0} v_2).
__device__ __forceinline__ double solve_m(const Norm &m, const LaneDivisor &ds, int b, int i, double v) {
    const double v2 = lane_get(v, 8 + i);
    const double w = b == 2 ? v : __fma_rn(m.sp, v, __dmul_rn(b == 0 ? m.c0 : m.r0, v2));
    const double q = lane_div(w, ds);
    const double q0 = lane_get(q, 4 * b), q1 = lane_get(q, 4 * b + 1), q2 = lane_get(q, 4 * b + 2);
    return i < 3 ? q : __fma_rn(-m.cz, q2, __fma_rn(-m.cy, q1, __fma_rn(-m.cx, q0, w)));
}

__device__ double det3(const double *a) {
    return a[0] * (a[4] * a[8] - a[5] * a[7]) - a[1] * (a[3] * a[8] - a[5] * a[6]) +
           a[2] * (a[3] * a[7] - a[4] * a[6]);
}

__device__ __forceinline__ bool isclose(double a, double b) {   // numpy defaults
    return fabs(a - b) <= 1e-8 + 1e-5 * fabs(b);
}

// rotation -> quaternion (w, x, y, z), M. Day's branch-on-trace method applied to R^T
// (the convention of pyquaternion's Quaternion(matrix=R), camera_approx.py:178)
__device__ void quaternion(const double *R, double *q) {
    double m[9];
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) m[3 * i + j] = R[3 * j + i];
    double t;
    if (m[8] < 0) {
        if (m[0] > m[4]) {
            t = 1 + m[0] - m[4] - m[8];
            q[0] = m[5] - m[7]; q[1] = t; q[2] = m[1] + m[3]; q[3] = m[6] + m[2];
        } else {
            t = 1 - m[0] + m[4] - m[8];
            q[0] = m[6] - m[2]; q[1] = m[1] + m[3]; q[2] = t; q[3] = m[5] + m[7];
        }
    } else {
        if (m[0] < -m[4]) {
            t = 1 - m[0] - m[4] + m[8];
            q[0] = m[1] - m[3]; q[1] = m[6] + m[2]; q[2] = m[5] + m[7]; q[3] = t;
        } else {
            t = 1 + m[0] + m[4] + m[8];
            q[0] = t; q[1] = m[5] - m[7]; q[2] = m[6] - m[2]; q[3] = m[1] - m[3];
        }
    }
    const double f = 0.5 / sqrt(t);
    for (int i = 0; i < 4; ++i) q[i] *= f;
}

// The camera of one view in shared memory.
struct CameraSmem {
    double P[12], K[9], R[9], t[3], u[12], q[12];
};

// Positive-diagonal RQ of the left 3x3 block of P by Gram-Schmidt from the last row (with
// one re-orthogonalisation), then the reference's normalisations.  The whole warp runs the scalar
// parts; lanes share the divisions.  Returns a status; s.K, s.R, s.t are zero unless set.
__device__ int factorize(CameraSmem &s, int lane) {
    double P[12], K[9], R[9];
    for (int i = 0; i < 12; ++i) P[i] = s.P[i];
    const double *a0 = P, *a1 = P + 4, *a2 = P + 8;
    double r0[3], r1[3], r2[3], u[3];
    auto unit = [&](const double *a, double n, double *r) {        // r = a / n
        const double q = (lane == 0 ? a[0] : (lane == 1 ? a[1] : a[2])) / n;
        for (int i = 0; i < 3; ++i) r[i] = lane_get(q, i);
    };
    for (int i = 0; i < 9; ++i) K[i] = 0.0;
    auto store = [&](int st) {
        __syncwarp();
        if (lane < 9) {
            double k = 0.0, r = 0.0;
            for (int i = 0; i < 9; ++i) k = lane == i ? K[i] : k, r = lane == i ? R[i] : r;
            s.K[lane] = k;
            s.R[lane] = r;
        }
        __syncwarp();
        return st;
    };
    for (int i = 0; i < 9; ++i) R[i] = 0.0;
    double n2 = sqrt(a2[0] * a2[0] + a2[1] * a2[1] + a2[2] * a2[2]);
    if (!(n2 > 0.0) || !isfinite(n2)) return store(VS_ERR_DEGENERATE);
    unit(a2, n2, r2);
    K[8] = n2;
    double k12 = a1[0] * r2[0] + a1[1] * r2[1] + a1[2] * r2[2];
    for (int i = 0; i < 3; ++i) u[i] = a1[i] - k12 * r2[i];
    double d = u[0] * r2[0] + u[1] * r2[1] + u[2] * r2[2];
    for (int i = 0; i < 3; ++i) u[i] -= d * r2[i];
    k12 += d;
    double n1 = sqrt(u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
    if (!(n1 > 0.0)) return store(VS_ERR_DEGENERATE);
    unit(u, n1, r1);
    K[4] = n1;
    K[5] = k12;
    double k02 = a0[0] * r2[0] + a0[1] * r2[1] + a0[2] * r2[2];
    double k01 = a0[0] * r1[0] + a0[1] * r1[1] + a0[2] * r1[2];
    for (int i = 0; i < 3; ++i) u[i] = a0[i] - k02 * r2[i] - k01 * r1[i];
    double d2 = u[0] * r2[0] + u[1] * r2[1] + u[2] * r2[2];
    double d1 = u[0] * r1[0] + u[1] * r1[1] + u[2] * r1[2];
    for (int i = 0; i < 3; ++i) u[i] -= d2 * r2[i] + d1 * r1[i];
    k02 += d2;
    k01 += d1;
    double n0 = sqrt(u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
    if (!(n0 > 0.0)) return store(VS_ERR_DEGENERATE);
    unit(u, n0, r0);
    K[0] = n0;
    K[1] = k01;
    K[2] = k02;
    for (int i = 0; i < 3; ++i) R[i] = r0[i], R[3 + i] = r1[i], R[6 + i] = r2[i];
    // K /= K[2,2], P /= K[2,2]: lanes 0..11 P, 12..20 K
    {
        const double sc = K[8];
        double x = sc;
        for (int i = 0; i < 12; ++i) x = lane == i ? P[i] : x;
        for (int i = 0; i < 9; ++i) x = lane == 12 + i ? K[i] : x;
        x /= sc;
        for (int i = 0; i < 12; ++i) P[i] = lane_get(x, i);
        for (int i = 0; i < 9; ++i) K[i] = lane_get(x, 12 + i);
    }
    if (det3(R) < 0.0) {
        for (int i = 0; i < 9; ++i) R[i] = -R[i];
        for (int i = 0; i < 12; ++i) P[i] = -P[i];
    }
    // t = K^-1 P[:, 3] (upper triangular)
    double t[3];
    t[2] = P[11] / K[8];
    t[1] = __dsub_rn(P[7], __dmul_rn(K[5], t[2])) / K[4];
    t[0] = __dsub_rn(__dsub_rn(P[3], __dmul_rn(K[1], t[1])), __dmul_rn(K[2], t[2])) / K[0];
    store(VS_OK);
    if (lane < 3) s.t[lane] = lane == 0 ? t[0] : (lane == 1 ? t[1] : t[2]);
    __syncwarp();
    // the reference's assertions: det R ~ 1 and K [R | t] ~ P
    if (!isclose(det3(R), 1.0)) return VS_ERR_FACTORIZE;
    bool near = true;
    if (lane < 12) {
        const int i = lane / 4, j = lane - 4 * i;
        double kr = 0.0, p = 0.0;
        for (int l = 0; l < 3; ++l) kr += s.K[3 * i + l] * (j < 3 ? s.R[3 * l + j] : s.t[l]);
        for (int k = 0; k < 12; ++k) p = lane == k ? P[k] : p;
        near = isclose(p, kr);
    }
    return __all_sync(0xffffffffu, near) ? VS_OK : VS_ERR_FACTORIZE;
}

// What the error pass needs of one view's camera: the camera in the normalised frame
// (q = M p, rescaled) as double-floats, the normalisation, and K^-1.
struct ErrCam {
    df q[12];
    float2 q01_hi[4], q01_lo[4];   // rows 0 and 1 of q paired, for the packed dot products
    NormF nf;
    float qscale;      // q = qscale * M p
    float kinv[9];
    float w, h;
    int ok;
};

// One warp fills a view's ErrCam from the camera in s.K, s.R, s.t (lanes 0..11: element (i, j) of
// the 3x4 matrices; the divisions side by side).
__device__ void make_errcam(CameraSmem &s, const Norm &nm, const NormF &nf, float w, float h, int ok, ErrCam &ec,
                            int lane) {
    const int l = min(lane, 11), i = l / 4, j = l - 4 * i;
    {
        double p = 0.0;
        for (int k = 0; k < 3; ++k) p += s.K[3 * i + k] * (j < 3 ? s.R[3 * k + j] : s.t[k]);
        __syncwarp();
        if (lane < 12) s.P[lane] = p;
        __syncwarp();
    }
    {
        const double *p = s.P + 4 * i;                 // T^T p_i
        const double last = nm.cx * p[0] + nm.cy * p[1] + nm.cz * p[2] + p[3];
        const double u = j < 3 ? nm.s * p[j] : last;
        if (lane < 12) s.u[lane] = u;
        __syncwarp();
    }
    const double uij = s.u[l], u2j = s.u[8 + j];
    const double off = i == 0 ? nm.c0 : nm.r0;
    const double quo = (uij - off * u2j) / nm.sp;
    const double q = i < 2 ? quo : u2j;
    double mx = fmax(0.0, fabs(q));
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, d));
    const double sc = (mx > 0.0 && isfinite(mx)) ? 1.0 / mx : 1.0;
    const df qd = df_from_double(q * sc);
    const float hi1 = __shfl_sync(0xffffffffu, qd.hi, (l + 4) & 15), lo1 = __shfl_sync(0xffffffffu, qd.lo, (l + 4) & 15);
    if (lane < 12) ec.q[lane] = qd;
    if (lane < 4) {
        ec.q01_hi[lane] = make_float2(qd.hi, hi1);
        ec.q01_lo[lane] = make_float2(qd.lo, lo1);
    }
    // K^-1 by cofactors: entry (r, c) = (K[a] K[b] - K[c] K[d]) / det
    const double a = s.K[0], b = s.K[1], c = s.K[2], d = s.K[3], e = s.K[4], f = s.K[5], g = s.K[6], hh = s.K[7],
                 i9 = s.K[8];
    const double det = a * (e * i9 - f * hh) - b * (d * i9 - f * g) + c * (d * hh - e * g);
    const double ki[9] = {e * i9 - f * hh, c * hh - b * i9, b * f - c * e, f * g - d * i9, a * i9 - c * g,
                          c * d - a * f,   d * hh - e * g,  b * g - a * hh, a * e - b * d};
    double x = det;
    for (int k = 0; k < 9; ++k) x = lane == k ? ki[k] : x;
    x /= det;
    if (lane < 9) ec.kinv[lane] = static_cast<float>(x);
    if (lane == 0) {
        ec.qscale = static_cast<float>(sc);
        ec.nf = nf;
        ec.w = w;
        ec.h = h;
        ec.ok = ok;
    }
}

// One CTA per view: sum the block partials in a fixed order, solve, factorise.
__global__ void __launch_bounds__(64) solve_kernel(const double *__restrict__ partial, int n_blocks,
                                                   const Norm *__restrict__ norm, const NormF *__restrict__ normf,
                                                   const VsRpcCamera *__restrict__ cams, double *__restrict__ K_out,
                                                   double *__restrict__ R_out, double *__restrict__ t_out,
                                                   double *__restrict__ params, ErrCam *__restrict__ errcam,
                                                   int32_t *__restrict__ status) {
    __shared__ double mom[kSlots];
    chain_wait();
    const int v = blockIdx.x;
    if (threadIdx.x < kSlots) {
        double s = 0.0;
        const double *p = partial + static_cast<long long>(v) * n_blocks * kSlots + threadIdx.x;
        int b = 0;
        for (; b + 16 <= n_blocks; b += 16) {           // one chain of sums; its loads 16 at a time
            double x[16];
#pragma unroll
            for (int k = 0; k < 16; ++k) x[k] = p[(b + k) * kSlots];
#pragma unroll
            for (int k = 0; k < 16; ++k) s += x[k];
        }
        for (; b < n_blocks; ++b) s += p[b * kSlots];
        mom[threadIdx.x] = s;
    }
    __syncthreads();
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x, l = min(lane, 11), bl = l >> 2, il = l & 3;   // lanes 12.. repeat lane 11
    __shared__ double L[12][13];
    __shared__ CameraSmem cam;
    const Norm nm = norm[v];
    if (lane < 9) cam.K[lane] = cam.R[lane] = 0.0;
    if (lane < 3) cam.t[lane] = 0.0;
    int st = mom[kMom] < 6.0 ? VS_ERR_DEGENERATE : VS_OK;
    if (st == VS_OK) {
        // row l of the normalised Gram matrix G = [[S0,0,-Sc],[0,S0,-Sr],[-Sc,-Sr,Sq]], S* symmetric
        double g[12];
        const int ent[4] = {0, 3, 5, 6};               // entry (a, b >= a) of a 10-vector: ent[a] + b
        double dmax = 0.0;
#pragma unroll
        for (int j = 0; j < 12; ++j) {
            const int bj = j >> 2, ij = j & 3, lo = min(il, ij), hi = max(il, ij);
            const double *m = mom + ((lo == 0 ? ent[0] : (lo == 1 ? ent[1] : (lo == 2 ? ent[2] : ent[3]))) + hi);
            const int other = min(bl, bj);             // 0: column block, 1: row block, when just one is block 2
            g[j] = bl == bj ? (bl < 2 ? m[0] : m[30]) : (max(bl, bj) < 2 ? 0.0 : (other == 0 ? -m[10] : -m[20]));
            dmax = fmax(dmax, l == j ? g[j] : 0.0);
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) dmax = fmax(dmax, __shfl_xor_sync(0xffffffffu, dmax, d));
        // Cholesky G = L L^T, column by column (a non-positive pivot -- an exactly
        // consistent system -- is floored; the inverse iteration then lands on the null vector).
        // Every lane forms the pivot; each element loses its products in the order of the columns.
        const double floor_piv = dmax * 1e-30 + 1e-300;
        double diag = 1.0;
#pragma unroll
        for (int k = 0; k < 12; ++k) {
            double d = lane_get(g[k], k);
            d = d > floor_piv ? d : floor_piv;
            d = sqrt(d);
            g[k] = l == k ? d : g[k] / d;
            diag = l == k ? d : diag;
#pragma unroll
            for (int j = k + 1; j < 12; ++j) g[j] = __fma_rn(-g[k], lane_get(g[k], j), g[j]);
        }
        if (lane < 12)
#pragma unroll
            for (int j = 0; j < 12; ++j) L[lane][j] = g[j];
        __syncwarp();
        double col[12];
#pragma unroll
        for (int j = 0; j < 12; ++j) col[j] = L[j][l];
        const LaneDivisor pivot = lane_divisor(diag), scale = lane_divisor(nm.s);
        double p = 0.28867513459481287;                // 1/sqrt(12)
#pragma unroll 1
        for (int it = 0; it < 6; ++it) {
            double sum = solve_mt(nm, scale, bl, il, p), x = 0.0;
            // L w = u: lane i subtracts w[j] L[i][j] as each w[j] is formed
#pragma unroll
            for (int j = 0; j < 12; ++j) {
                const double t = lane_div(sum, pivot), wj = lane_get(t, j);
                x = l == j ? t : x;
                sum = l > j ? __fma_rn(-g[j], wj, sum) : sum;
            }
            // L^T u = w
            sum = x;
#pragma unroll
            for (int j = 11; j >= 0; --j) {
                const double t = lane_div(sum, pivot), uj = lane_get(t, j);
                x = l == j ? t : x;
                sum = l < j ? __fma_rn(-col[j], uj, sum) : sum;
            }
            const double pp = solve_m(nm, scale, bl, il, x);
            double nrm = 0.0;
#pragma unroll
            for (int i = 0; i < 12; ++i) {
                const double y = lane_get(pp, i);
                nrm = __fma_rn(y, y, nrm);
            }
            p = __dmul_rn(pp, 1.0 / sqrt(nrm));
        }
        if (lane < 12) cam.P[lane] = p;
        __syncwarp();
        st = __all_sync(0xffffffffu, isfinite(p)) ? factorize(cam, lane) : VS_ERR_DEGENERATE;
    }
    __syncwarp();
    const double *K = cam.K, *R = cam.R, *t = cam.t;
    if (lane < 9) K_out[v * 9 + lane] = K[lane], R_out[v * 9 + lane] = R[lane];
    if (lane < 3) t_out[v * 3 + lane] = t[lane];
    if (lane == 0) status[v] = st;
    if (params) {
        double q[4] = {0, 0, 0, 0};
        if (st == VS_OK) quaternion(R, q);
        double *o = params + v * VS_CAMERA_PARAMS;
        if (lane == 0) {
            o[0] = cams ? cams[v].width : 0.0;
            o[1] = cams ? cams[v].height : 0.0;
            o[2] = K[0]; o[3] = K[4]; o[4] = K[2]; o[5] = K[5]; o[6] = K[1];
            o[7] = q[0]; o[8] = q[1]; o[9] = q[2]; o[10] = q[3];
            o[11] = t[0]; o[12] = t[1]; o[13] = t[2];
        }
    }
    if (errcam)
        make_errcam(cam, nm, normf[v], cams ? static_cast<float>(cams[v].width) : 0.f,
                    cams ? static_cast<float>(cams[v].height) : 0.f, st == VS_OK, errcam[v], lane);
}

// ---------------------------------------------------------------------------------------
// error statistics (check_perspective_error)
// ---------------------------------------------------------------------------------------
// ErrCam for given K, R, t (the drop-in statistics entry), a warp per view
__global__ void __launch_bounds__(32) errcam_kernel(const double *K, const double *R, const double *t,
                                                    const Norm *norm, const NormF *normf, ErrCam *ec) {
    __shared__ CameraSmem s;
    chain_wait();
    const int v = blockIdx.x, lane = threadIdx.x;
    if (lane < 9) s.K[lane] = K[9 * v + lane], s.R[lane] = R[9 * v + lane];
    if (lane < 3) s.t[lane] = t[3 * v + lane];
    __syncwarp();
    make_errcam(s, norm[v], normf[v], 0.f, 0.f, 1, ec[v], lane);
}

// Radix selection over the float bits of the per-point errors (non-negative floats, so
// the bits order like the values), 11 + 11 + 10 bits.  Targets per view: 0/1 = the
// low/high middle order statistic of the pixel errors, 2/3 = of the metric errors.
__host__ __device__ constexpr int digit_bits(int pass) { return pass == 2 ? 10 : 11; }
__host__ __device__ constexpr int digit_shift(int pass) { return pass == 0 ? 21 : (pass == 1 ? 10 : 0); }
constexpr int kBins = 2048;

struct ErrWs {
    unsigned *keys;          // [2][V][n] float bits of the per-point errors (kept points only)
    double *sums;            // [V][blocks][3]: pixel sum, metric sum, count
    unsigned *maxk;          // [V][2]; maxk and hist are cleared as one range
    unsigned *hist;          // [V][2][kBins] of the leading digit (pixel, metric), then for each
                             // later digit [V][4][kBins] (one per target)
    size_t cleared;          // bytes from maxk to the end of hist
    unsigned *sel;           // [V][4][2]: prefix, rank
    __device__ unsigned *digit_hist(int pass, int V, int v) const {
        return pass == 0 ? hist + static_cast<long long>(v) * 2 * kBins
                         : hist + (2ll * V + 4ll * (pass - 1) * V + 4ll * v) * kBins;
    }
};

constexpr int kErrThreads = 256;

// Inclusive sum over the lanes up to this one.
__device__ __forceinline__ unsigned warp_scan(unsigned x, int lane) {
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const unsigned u = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += u;
    }
    return x;
}

// Picks digit `pass` of the four targets of one view: one block per view, one warp per target.
// Pass 0 reads the two histograms the error kernel built (pixel, metric) and starts from the
// ranks; later passes read one histogram per target, except that the high target shares its
// low partner's while their prefixes agree.  A warp takes its bins in two looks -- all bins, a run
// per lane, then the run that holds the rank -- instead of 32 bins at a time, each a trip to L2 (12
// to 43 us, 6 to 8 now).  The last pass also writes the view's statistics, which, like the
// ranks, were launches that summed the blocks' partials one by one (17 + 29 us for 210 blocks).
// (A step by the last block of the pass before it saves a launch and costs every block a fence
// behind its histogram's atomics: 50 us more for 50 views.)
constexpr int kStepThreads = 128;

__global__ void __launch_bounds__(kStepThreads) select_step_kernel(ErrWs w, int n_blocks, int pass,
                                                                   double *__restrict__ err) {
    const int v = blockIdx.x, V = gridDim.x;
    const int t = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __shared__ double part[3][kStepThreads / 32];
    __shared__ unsigned pre[4];
    chain_wait();
    double total[3] = {0.0, 0.0, 0.0};       // pixel sum, metric sum, count
    if (pass != 1) {
        for (int b = threadIdx.x; b < n_blocks; b += kStepThreads)
#pragma unroll
            for (int q = 0; q < 3; ++q) total[q] += w.sums[(static_cast<long long>(v) * n_blocks + b) * 3 + q];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) total[q] += __shfl_xor_sync(0xffffffffu, total[q], off);
            if (lane == 0) part[q][t] = total[q];
        }
    }
    unsigned *sel = w.sel + 2 * (v * 4 + t);
    if (lane == 0) pre[t] = pass == 0 ? 0u : sel[0];
    __syncthreads();
    if (pass != 1)
#pragma unroll
        for (int q = 0; q < 3; ++q) total[q] = ((part[q][0] + part[q][1]) + part[q][2]) + part[q][3];
    const unsigned long long n = static_cast<unsigned long long>(total[2]);
    const unsigned k = pass == 0 ? (n ? static_cast<unsigned>((t & 1) ? n / 2 : (n - 1) / 2) : 0u) : sel[1];
    const int which = pass == 0 ? t >> 1 : ((t & 1) && pre[t] == pre[t ^ 1] ? t ^ 1 : t);
    const unsigned *hist = w.digit_hist(pass, V, v) + which * kBins;
    const int bins = 1 << digit_bits(pass), run = bins / 32;
    unsigned c = 0;
    const uint4 *mine = reinterpret_cast<const uint4 *>(hist + lane * run);
#pragma unroll 8
    for (int i = 0; i < run / 4; ++i) {
        const uint4 x = mine[i];
        c += (x.x + x.y) + (x.z + x.w);
    }
    unsigned incl = warp_scan(c, lane);
    const unsigned hit = __ballot_sync(0xffffffffu, incl > k);
    int digit = bins - 1;
    unsigned skip;
    if (hit) {
        const int seg = __ffs(hit) - 1;
        unsigned below = __shfl_sync(0xffffffffu, incl - c, seg);
        digit = seg * run;
        for (int i = 0; i < run; i += 32) {          // one or two looks
            const unsigned x = hist[seg * run + i + lane], in = warp_scan(x, lane);
            const unsigned h2 = __ballot_sync(0xffffffffu, below + in > k);
            if (h2) {
                digit = seg * run + i + __ffs(h2) - 1;
                below += __shfl_sync(0xffffffffu, in - x, __ffs(h2) - 1);
                break;
            }
            below += __shfl_sync(0xffffffffu, in, 31);
        }
        skip = below;
    } else {                     // rank beyond the counts (no kept points): the last bin
        skip = __shfl_sync(0xffffffffu, incl, 31) - hist[bins - 1];
    }
    const unsigned chosen = pre[t] | (static_cast<unsigned>(digit) << digit_shift(pass));
    __syncthreads();                                     // every pre[] has been read
    if (lane == 0) {
        sel[0] = chosen;
        sel[1] = k - skip;
        pre[t] = chosen;
    }
    if (pass < 2) return;
    __syncthreads();
    if (threadIdx.x < 2) {
        const int q = threadIdx.x;
        const double cnt = total[2], lo = __uint_as_float(pre[2 * q]), hi = __uint_as_float(pre[2 * q + 1]);
        const double nan = __longlong_as_double(0x7ff8000000000000ll);
        double *o = err + v * VS_ERROR_STATS + 3 * q;
        o[0] = cnt > 0 ? (q ? total[1] : total[0]) / cnt : nan;
        o[1] = cnt > 0 ? ((0.0 + lo) + hi) / 2.0 : nan;
        o[2] = cnt > 0 ? static_cast<double>(__uint_as_float(w.maxk[2 * v + q])) : nan;
    }
}

// compensated dot product of a double-float 4-vector with (x, y, z, 1), FP32 exact inputs
__device__ __forceinline__ df dot2(const df *q, float x, float y, float z) {
    df p0 = two_prod(q[0].hi, x), p1 = two_prod(q[1].hi, y), p2 = two_prod(q[2].hi, z);
    float err = __fmaf_rn(q[0].lo, x, p0.lo) + __fmaf_rn(q[1].lo, y, p1.lo) + __fmaf_rn(q[2].lo, z, p2.lo) + q[3].lo;
    df s = two_sum(p0.hi, p1.hi);
    err += s.lo;
    s = two_sum(s.hi, p2.hi);
    err += s.lo;
    s = two_sum(s.hi, q[3].hi);
    err += s.lo;
    return fast_two_sum(s.hi, err);
}

// dot2 for rows 0 and 1 of q at once (FP32x2 lanes; each lane performs dot2's operations)
__device__ __forceinline__ df2 dot2_rows01(const ErrCam &ec, float x, float y, float z) {
    const float2 X = f2s(x), Y = f2s(y), Z = f2s(z), nX = f2s(-x), nY = f2s(-y), nZ = f2s(-z);
    const float2 h0 = ec.q01_hi[0], h1 = ec.q01_hi[1], h2 = ec.q01_hi[2];
    const df2 p0 = {__fmul2_rn(h0, X), __ffma2_rn(h0, X, __fmul2_rn(h0, nX))};
    const df2 p1 = {__fmul2_rn(h1, Y), __ffma2_rn(h1, Y, __fmul2_rn(h1, nY))};
    const df2 p2 = {__fmul2_rn(h2, Z), __ffma2_rn(h2, Z, __fmul2_rn(h2, nZ))};
    float2 err = __fadd2_rn(__fadd2_rn(__fadd2_rn(__ffma2_rn(ec.q01_lo[0], X, p0.lo), __ffma2_rn(ec.q01_lo[1], Y, p1.lo)),
                                       __ffma2_rn(ec.q01_lo[2], Z, p2.lo)),
                            ec.q01_lo[3]);
    df2 s = two_sum2(p0.hi, p1.hi);
    err = __fadd2_rn(err, s.lo);
    s = two_sum2(s.hi, p2.hi);
    err = __fadd2_rn(err, s.lo);
    s = two_sum2(s.hi, ec.q01_hi[3]);
    err = __fadd2_rn(err, s.lo);
    return fast_two_sum2(s.hi, err);
}

// Per kept point: pixel reprojection error and metric inverse-projection error, written
// as float bits for the median selection, plus block sums/maxima and the histogram of
// the leading digit.
//  * reprojection: in the fit's normalised frame, with the ENU point rounded to FP32
//    (|error| <~ 1e-4 px): h = q.X' by compensated dot products, residual
//    (h0 - c' h2) / h2 with c' the double-float normalised observation;
//  * inverse projection: the reference's |scale*ray - cam| is the distance from the
//    camera-frame point to the ray d = K^-1 [c r 1].  The point lies on the ray through
//    its own projection, cam = h2 K^-1 [c^ r^ 1], so the distance is
//    |h2| |delta x d| / |d| with delta = K^-1 [c^ - c, r^ - r, 0]: the pixel residual
//    enters directly and nothing of the camera's ~1e5-1e6 m depth cancels.
__global__ void __launch_bounds__(kErrThreads, 4) error_points_kernel(
    const double *__restrict__ x, const double *__restrict__ y, const double *__restrict__ z, long long xyz_stride,
    const double *__restrict__ col, const double *__restrict__ row, const float4 *__restrict__ colrow,
    const uint8_t *__restrict__ keep, long long n, const ErrCam *__restrict__ cams, ErrWs w) {
    __shared__ ErrCam ec;
    __shared__ double red[3][kErrThreads / 32];
    __shared__ unsigned hist[2][kBins];
    chain_wait();
    const int v = blockIdx.y;
    const int V = gridDim.y;
    if (threadIdx.x == 0) ec = cams[v];
    for (int i = threadIdx.x; i < 2 * kBins; i += blockDim.x) (&hist[0][0])[i] = 0;
    __syncthreads();
    float ps = 0.0f, is = 0.0f, cnt = 0.0f;
    unsigned pmax = 0, imax = 0;
    const double *xv = x + v * xyz_stride, *yv = y + v * xyz_stride, *zv = z + v * xyz_stride;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        // the point's coordinates are requested with its pixels, not after the in-image
        // test on them: one memory round trip per point instead of two
        const long long RX = __ldg(reinterpret_cast<const long long *>(xv) + i);
        const long long RY = __ldg(reinterpret_cast<const long long *>(yv) + i);
        const long long RZ = __ldg(reinterpret_cast<const long long *>(zv) + i);
        df c, r;
        bool k;
        if (colrow) {
            const float4 cr = colrow[static_cast<long long>(v) * n + i];
            c = {cr.x, cr.y};
            r = {cr.z, cr.w};
            k = df_ge0(c) && df_ge0(r) && df_lt(c, ec.w) && df_lt(r, ec.h);
        } else {
            c = split_double(col[v * n + i]);
            r = split_double(row[v * n + i]);
            k = keep ? keep[v * n + i] != 0 : true;
        }
        unsigned pk = 0xffffffffu, ik = 0xffffffffu;
        if (k && ec.ok) {
            float X, Y, Z, cf_, rf_;
            normalised_point(ec.nf, RX, RY, RZ, c, r, X, Y, Z, cf_, rf_);
            // rows 0 and 1 of the camera (h0, h1) and the observations (c, r) travel as FP32x2
            // pairs; every lane performs the scalar double-float operations
            const df2 h01 = dot2_rows01(ec, X, Y, Z);
            const df h2 = dot2(ec.q + 8, X, Y, Z);
            // observation in the normalised frame as a double-float: (c - c0) / sp
            const df2 crn = df_mul2(df_add2({f2(c.hi, r.hi), f2(c.lo, r.lo)},
                                            {f2(-ec.nf.c0.hi, -ec.nf.r0.hi), f2(-ec.nf.c0.lo, -ec.nf.r0.lo)}),
                                    {f2s(ec.nf.inv_sp.hi), f2s(ec.nf.inv_sp.lo)}, f2s(-ec.nf.inv_sp.hi));
            const df2 ncr = df_add2(h01, df_mul2({sub2(f2s(0.0f), crn.hi), sub2(f2s(0.0f), crn.lo)},
                                                 {f2s(h2.hi), f2s(h2.lo)}, f2s(-h2.hi)));
            const float h2f = h2.hi + h2.lo;
            const float2 nsum = __fadd2_rn(ncr.hi, ncr.lo);
            const float dc = ec.nf.sp * (nsum.x / h2f), dr = ec.nf.sp * (nsum.y / h2f);
            const float pe = sqrtf(__fmaf_rn(dr, dr, dc * dc));
            const float *ki = ec.kinv;
            const float cf = c.hi, rf = r.hi;
            const float d0 = __fmaf_rn(ki[0], cf, __fmaf_rn(ki[1], rf, ki[2]));
            const float d1 = __fmaf_rn(ki[3], cf, __fmaf_rn(ki[4], rf, ki[5]));
            const float d2 = __fmaf_rn(ki[6], cf, __fmaf_rn(ki[7], rf, ki[8]));
            const float e0 = __fmaf_rn(ki[0], dc, ki[1] * dr);
            const float e1 = __fmaf_rn(ki[3], dc, ki[4] * dr);
            const float e2 = __fmaf_rn(ki[6], dc, ki[7] * dr);
            const float x0 = e1 * d2 - e2 * d1, x1 = e2 * d0 - e0 * d2, x2 = e0 * d1 - e1 * d0;
            const float hz = fabsf(h2f / ec.qscale);
            const float ie = hz * sqrtf((x0 * x0 + x1 * x1 + x2 * x2) / (d0 * d0 + d1 * d1 + d2 * d2));
            ps += pe;
            is += ie;
            cnt += 1.0f;
            pk = __float_as_uint(pe);
            ik = __float_as_uint(ie);
            pmax = max(pmax, pk);
            imax = max(imax, ik);
            atomicAdd(&hist[0][pk >> digit_shift(0)], 1u);
            atomicAdd(&hist[1][ik >> digit_shift(0)], 1u);
        }
        w.keys[static_cast<long long>(v) * n + i] = pk;
        w.keys[(static_cast<long long>(V) + v) * n + i] = ik;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        ps += __shfl_xor_sync(0xffffffffu, ps, off);
        is += __shfl_xor_sync(0xffffffffu, is, off);
        cnt += __shfl_xor_sync(0xffffffffu, cnt, off);
        pmax = max(pmax, __shfl_xor_sync(0xffffffffu, pmax, off));
        imax = max(imax, __shfl_xor_sync(0xffffffffu, imax, off));
    }
    const int warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        red[0][warp] = f32_to_f64(ps);
        red[1][warp] = f32_to_f64(is);
        red[2][warp] = f32_to_f64(cnt);
        if (pmax) atomicMax(w.maxk + 2 * v, pmax);
        if (imax) atomicMax(w.maxk + 2 * v + 1, imax);
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        double s = 0.0;
        for (int i = 0; i < kErrThreads / 32; ++i) s += red[threadIdx.x][i];
        w.sums[(static_cast<long long>(v) * gridDim.x + blockIdx.x) * 3 + threadIdx.x] = s;
    }
    for (int i = threadIdx.x; i < 2 * kBins; i += blockDim.x) {
        const unsigned c = (&hist[0][0])[i];
        if (c) atomicAdd(w.digit_hist(0, V, v) + i, c);
    }
}

// Histograms of digit `pass` (1, 2) of the keys matching each target's prefix.  Issue-bound at 94
// instructions per point with four masked compares and as many histograms whether the targets of a
// pair differ or not: now each thread has 4 points' keys in flight and compares them with
// its pair's one prefix unless the pair has split, in as many blocks as the SMs hold (a block
// clears and adds 8192 bins).  50 x 800,000 points: 125 us a pass, 77 us.
constexpr int kHistThreads = 256, kHistAhead = 4;

__global__ void __launch_bounds__(kHistThreads) select_hist_kernel(ErrWs w, long long n, int pass) {
    __shared__ unsigned h[4][kBins];
    chain_wait();
    const int v = blockIdx.y, V = gridDim.y;
    const int shift = digit_shift(pass), top = shift + digit_bits(pass);
    const unsigned dmask = (1u << digit_bits(pass)) - 1u;
    unsigned pre[4];
    for (int t = 0; t < 4; ++t) pre[t] = w.sel[2 * (v * 4 + t)] >> top;
    const bool split[2] = {pre[0] != pre[1], pre[2] != pre[3]};
    for (int t = 0; t < 4; ++t)
        if (!(t & 1) || split[t >> 1])
            for (int i = threadIdx.x; i < kBins; i += kHistThreads) h[t][i] = 0;
    __syncthreads();
    const unsigned *kp = w.keys + static_cast<long long>(v) * n, *kq = w.keys + (static_cast<long long>(V) + v) * n;
    const long long step = static_cast<long long>(gridDim.x) * kHistThreads * kHistAhead;
    for (long long i = static_cast<long long>(blockIdx.x) * kHistThreads * kHistAhead + threadIdx.x; i < n; i += step) {
        unsigned k[2][kHistAhead];
#pragma unroll
        for (int u = 0; u < kHistAhead; ++u) {
            const long long j = i + u * kHistThreads;
            k[0][u] = j < n ? __ldcs(kp + j) : 0xffffffffu;      // as a point that is not kept
            k[1][u] = j < n ? __ldcs(kq + j) : 0xffffffffu;
        }
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int u = 0; u < kHistAhead; ++u) {
                const unsigned head = k[q][u] >> top, digit = (k[q][u] >> shift) & dmask;
                if (head == pre[2 * q]) atomicAdd(&h[2 * q][digit], 1u);
                if (split[q] && head == pre[2 * q + 1]) atomicAdd(&h[2 * q + 1][digit], 1u);
            }
    }
    __syncthreads();
    unsigned *out = w.digit_hist(pass, V, v);
    for (int t = 0; t < 4; ++t)
        if (!(t & 1) || split[t >> 1])
            for (int i = threadIdx.x; i < kBins; i += kHistThreads) {
                const unsigned c = h[t][i];
                if (c) atomicAdd(out + t * kBins + i, c);
            }
}

int err_blocks(long long n) {
    long long want = ceil_div(n, kErrThreads * 4);
    return static_cast<int>(std::max<long long>(1, std::min<long long>(want, sm_count() * 2LL)));
}

// Blocks per view of a histogram pass: at least 16 points per thread, at most two rounds of
// what the SMs hold over all views.
int hist_blocks(long long n, int V) {
    const long long most = std::max<long long>(1, ceil_div(sm_count() * 12LL, V));
    return static_cast<int>(std::max<long long>(1, std::min<long long>(ceil_div(n, kHistThreads * 16), most)));
}

ErrWs carve_err(Carver &cv, int V, long long n, int blocks) {
    ErrWs w;
    w.keys = cv.take<unsigned>(2 * static_cast<size_t>(V) * n);
    w.sums = cv.take<double>(static_cast<size_t>(V) * blocks * 3);
    w.maxk = cv.take<unsigned>(2 * static_cast<size_t>(V));
    w.hist = cv.take<unsigned>(static_cast<size_t>(V) * 10 * kBins);
    w.cleared = reinterpret_cast<char *>(w.hist + static_cast<size_t>(V) * 10 * kBins) - reinterpret_cast<char *>(w.maxk);
    w.sel = cv.take<unsigned>(static_cast<size_t>(V) * 8);
    return w;
}

int clear_async(void *p, size_t bytes, cudaStream_t st) {
    if (cudaMemsetAsync(p, 0, bytes, st) == cudaSuccess) return VS_OK;
    set_error("cudaMemsetAsync failed");
    return VS_ERR_CUDA;
}

// w.maxk .. w.hist have been cleared.
int run_error_stats(const double *x, const double *y, const double *z, long long xyz_stride, const double *col,
                    const double *row, const float4 *colrow, const uint8_t *keep, int V, long long n,
                    const ErrCam *cams, double *err, ErrWs &w, cudaStream_t st) {
    const int blocks = err_blocks(n);
    int s;
    if (n > 0) {
        launch_chained(error_points_kernel, dim3(blocks, V), kErrThreads, 0, st, x, y, z, xyz_stride, col, row, colrow, keep, n,
                                                                      cams, w);
        VS_LAUNCH_CHECK("error_points_kernel");
    } else if ((s = clear_async(w.sums, sizeof(double) * V * blocks * 3, st)) != VS_OK) {
        return s;
    }
    for (int pass = n > 0 ? 0 : 2; pass < 3; ++pass) {
        if (pass > 0 && n > 0) {
            launch_chained(select_hist_kernel, dim3(hist_blocks(n, V), V), kHistThreads, 0, st, w, n, pass);
            VS_LAUNCH_CHECK("select_hist_kernel");
        }
        launch_chained(select_step_kernel, V, kStepThreads, 0, st, w, blocks, pass, err);
        VS_LAUNCH_CHECK("select_step_kernel");
    }
    return VS_OK;
}

int mom_blocks(long long n) {
    return static_cast<int>(std::max<long long>(1, ceil_div(n, static_cast<long long>(kMomThreads) * kChunk)));
}

long long box_step(long long n) { return std::max<long long>(1, n / kBoxSamples); }

int box_blocks(long long n) {
    long long samples = ceil_div(n, box_step(n));
    return static_cast<int>(std::max<long long>(1, std::min<long long>(ceil_div(samples, 256), 64)));
}

struct FitWs {
    Box *box;
    Norm *norm;
    NormF *normf;
    double *partial;
    ErrCam *errcam;
    float4 *colrow;
    float *wh;
    RpcFast *fast;
};

FitWs carve_fit(Carver &cv, int V, long long n, bool fused) {
    FitWs f;
    f.box = cv.take<Box>(V);
    f.norm = cv.take<Norm>(V);
    f.normf = cv.take<NormF>(V);
    f.partial = cv.take<double>(static_cast<size_t>(V) * mom_blocks(n) * kSlots);
    f.errcam = cv.take<ErrCam>(V);
    f.colrow = fused ? cv.take<float4>(static_cast<size_t>(V) * n) : nullptr;
    f.wh = cv.take<float>(2 * static_cast<size_t>(V));
    f.fast = fused ? cv.take<RpcFast>(V) : nullptr;
    return f;
}

// f.box has been cleared.
int launch_norm(const double *x, const double *y, const double *z, long long xyz_stride, const double *col,
                const double *row, const uint8_t *keep, const VsRpcCamera *cams, int V, long long n, FitWs &f,
                cudaStream_t st) {
    launch_chained(bbox_kernel, dim3(box_blocks(n), V), 256, 0, st, x, y, z, xyz_stride, col, row, keep, n, box_step(n), cams,
                                                          f.box, f.norm, f.normf);
    VS_LAUNCH_CHECK("bbox_kernel");
    return VS_OK;
}

int launch_moments(const double *x, const double *y, const double *z, long long xyz_stride, const double *col,
                   const double *row, const float4 *colrow, const uint8_t *keep, int V, long long n, FitWs &f,
                   cudaStream_t st) {
    launch_chained(moments_kernel, dim3(mom_blocks(n), V), kMomThreads, 0, st, x, y, z, xyz_stride, col, row, colrow, keep,
                   colrow ? f.wh : nullptr, n, f.normf, f.partial);
    return check_launch("moments_kernel");
}

}  // namespace
}  // namespace vs

using namespace vs;

extern "C" int vs_rpc_project(const VsRpcCamera *cams, int n_cams, const double *lat, const double *lon,
                              const double *alt, int64_t n, int64_t point_stride, double *col, double *row,
                              uint8_t *keep, int mode, void *stream) {
    VS_REQUIRE(n_cams > 0 && n_cams <= 65535 && n >= 0 && point_stride >= 0, "vs_rpc_project: bad sizes");
    VS_REQUIRE(mode == VS_PROJ_EXACT || mode == VS_PROJ_FAST, "vs_rpc_project: bad mode %d", mode);
    if (n == 0) return VS_OK;
    VS_REQUIRE(cams && lat && lon && alt && col && row, "vs_rpc_project: null pointer");
    // The exact form is bound by each SM's FP64 pipe, so few points are spread over all SMs:
    // 1999 points in blocks of 256 took 26 us on 8 SMs, in blocks of 32 on 63 SMs 14 us.
    // The fast form is bound by each block's preparation of its camera, which the threads share: 100 points 6.5 us
    // in a block of 256, 8.3 in blocks of 32; 2000 points 6.9 and 8.3, 10,000 8.1 and 8.4.  Above 128 points
    // per SM blocks of 64 spread them better: 20,000 points 8.3 us with 256, 7.4 with 64.
    const int sms = sm_count();
    const long long points = n * n_cams;
    const int few = mode == VS_PROJ_EXACT ? 32 : 256;
    const int threads = points >= 512LL * sms ? 256 : (points >= 128LL * sms ? 64 : few);
    const long long want = ceil_div(n, threads);
    const long long cap = std::max(1LL, sms * (2048LL / threads) / n_cams + 1);
    // even shares: every thread of a full grid takes as many points as any other, +-1
    const long long rounds = ceil_div(want, cap);
    const dim3 grid(static_cast<unsigned>(ceil_div(want, rounds)), n_cams);
    cudaStream_t st = as_stream(stream);
    if (mode == VS_PROJ_EXACT)
        rpc_project_kernel<VS_PROJ_EXACT><<<grid, threads, 0, st>>>(cams, lat, lon, alt, n, point_stride, col, row, keep);
    else
        rpc_project_kernel<VS_PROJ_FAST><<<grid, threads, 0, st>>>(cams, lat, lon, alt, n, point_stride, col, row, keep);
    VS_LAUNCH_CHECK("rpc_project_kernel");
    return VS_OK;
}

extern "C" size_t vs_dlt_fit_workspace_size(int n_views, int64_t n) {
    if (n_views <= 0 || n < 0) return 0;
    Carver cv(nullptr);
    carve_fit(cv, n_views, n, false);
    return cv.used + 256;
}

extern "C" int vs_dlt_fit(const double *x, const double *y, const double *z, int64_t xyz_stride, const double *col,
                          const double *row, const uint8_t *keep, int n_views, int64_t n, double *K, double *R,
                          double *t, int32_t *status, void *workspace, size_t workspace_bytes, void *stream) {
    VS_REQUIRE(n_views > 0 && n_views <= 65535 && n >= 0 && xyz_stride >= 0, "vs_dlt_fit: bad sizes");
    VS_REQUIRE(x && y && z && col && row && K && R && t && status && workspace, "vs_dlt_fit: null pointer");
    const size_t need = vs_dlt_fit_workspace_size(n_views, n);
    if (workspace_bytes < need) {
        set_error("vs_dlt_fit: workspace %zu < %zu bytes", workspace_bytes, need);
        return VS_ERR_WORKSPACE;
    }
    cudaStream_t st = as_stream(stream);
    Carver cv(workspace);
    FitWs f = carve_fit(cv, n_views, n, false);
    int s = clear_async(f.box, sizeof(Box) * n_views, st);
    if (s != VS_OK) return s;
    s = launch_norm(x, y, z, xyz_stride, col, row, keep, nullptr, n_views, n, f, st);
    if (s != VS_OK) return s;
    const int blocks = mom_blocks(n);
    if ((s = launch_moments(x, y, z, xyz_stride, col, row, nullptr, keep, n_views, n, f, st)) != VS_OK) return s;
    launch_chained(solve_kernel, n_views, 64, 0, st, f.partial, blocks, f.norm, f.normf, nullptr, K, R, t, nullptr,
                   nullptr, status);
    VS_LAUNCH_CHECK("solve_kernel");
    return VS_OK;
}

extern "C" size_t vs_perspective_error_workspace_size(int n_views, int64_t n) {
    if (n_views <= 0 || n < 0) return 0;
    Carver cv(nullptr);
    carve_fit(cv, n_views, 0, false);
    carve_err(cv, n_views, n, err_blocks(n));
    return cv.used + 256;
}

extern "C" int vs_perspective_error(const double *x, const double *y, const double *z, int64_t xyz_stride,
                                    const double *col, const double *row, const uint8_t *keep, int n_views,
                                    int64_t n, const double *K, const double *R, const double *t, double *err,
                                    void *workspace, size_t workspace_bytes, void *stream) {
    VS_REQUIRE(n_views > 0 && n_views <= 65535 && n >= 0 && xyz_stride >= 0, "vs_perspective_error: bad sizes");
    VS_REQUIRE(x && y && z && col && row && K && R && t && err && workspace, "vs_perspective_error: null pointer");
    const size_t need = vs_perspective_error_workspace_size(n_views, n);
    if (workspace_bytes < need) {
        set_error("vs_perspective_error: workspace %zu < %zu bytes", workspace_bytes, need);
        return VS_ERR_WORKSPACE;
    }
    cudaStream_t st = as_stream(stream);
    Carver cv(workspace);
    FitWs f = carve_fit(cv, n_views, 0, false);
    ErrWs w = carve_err(cv, n_views, n, err_blocks(n));
    int s = clear_async(f.box, sizeof(Box) * n_views, st);
    if (s == VS_OK) s = clear_async(w.maxk, w.cleared, st);
    if (s != VS_OK) return s;
    s = launch_norm(x, y, z, xyz_stride, col, row, keep, nullptr, n_views, n, f, st);
    if (s != VS_OK) return s;
    launch_chained(errcam_kernel, n_views, 32, 0, st, K, R, t, f.norm, f.normf, f.errcam);
    VS_LAUNCH_CHECK("errcam_kernel");
    return run_error_stats(x, y, z, xyz_stride, col, row, nullptr, keep, n_views, n, f.errcam, err, w, st);
}

extern "C" size_t vs_camera_approx_workspace_size(int n_views, int64_t n) {
    if (n_views <= 0 || n < 0) return 0;
    Carver cv(nullptr);
    carve_fit(cv, n_views, n, true);
    cv.take<double>(static_cast<size_t>(n_views) * 9);    // K
    cv.take<double>(static_cast<size_t>(n_views) * 9);    // R
    cv.take<double>(static_cast<size_t>(n_views) * 3);    // t
    carve_err(cv, n_views, n, err_blocks(n));
    return cv.used + 256;
}

extern "C" int vs_camera_approx_perspective(const VsRpcCamera *cams, int n_views, const double *lat,
                                            const double *lon, const double *alt, const double *x, const double *y,
                                            const double *z, int64_t n, int64_t point_stride, int proj_mode,
                                            double *params, double *err, int32_t *status, void *workspace,
                                            size_t workspace_bytes, void *stream) {
    VS_REQUIRE(n_views > 0 && n_views <= 65535 && n >= 0 && point_stride >= 0,
               "vs_camera_approx_perspective: bad sizes");
    VS_REQUIRE(proj_mode == VS_PROJ_EXACT || proj_mode == VS_PROJ_FAST, "vs_camera_approx_perspective: bad mode");
    VS_REQUIRE(cams && lat && lon && alt && x && y && z && params && status && workspace,
               "vs_camera_approx_perspective: null pointer");
    const size_t need = vs_camera_approx_workspace_size(n_views, n);
    if (workspace_bytes < need) {
        set_error("vs_camera_approx_perspective: workspace %zu < %zu bytes", workspace_bytes, need);
        return VS_ERR_WORKSPACE;
    }
    cudaStream_t st = as_stream(stream);
    Carver cv(workspace);
    FitWs f = carve_fit(cv, n_views, n, true);
    double *K = cv.take<double>(static_cast<size_t>(n_views) * 9);
    double *R = cv.take<double>(static_cast<size_t>(n_views) * 9);
    double *t = cv.take<double>(static_cast<size_t>(n_views) * 3);
    ErrWs ew = carve_err(cv, n_views, n, err_blocks(n));
    // the clears first, so that nothing comes between the kernels of the chain
    int s = clear_async(f.box, sizeof(Box) * n_views, st);
    if (s == VS_OK && err) s = clear_async(ew.maxk, ew.cleared, st);
    if (s != VS_OK) return s;
    // ENU box (sampled) -> normalisation; pixel frame from each RPC
    s = launch_norm(x, y, z, point_stride, nullptr, nullptr, nullptr, cams, n_views, n, f, st);
    if (s != VS_OK) return s;
    const int blocks = mom_blocks(n);
    launch_chained(prepare_views_kernel, n_views, 64, 0, st, cams, f.fast, f.wh);
    VS_LAUNCH_CHECK("prepare_views_kernel");
    if (n > 0) {
        // many short blocks: three fit an SM, and 3.5 rounds of long ones left the last half empty
        // (50 x 800,000 points: 8 blocks per SM in all 646 us, 48 per SM 620 us, 96 the same)
        const unsigned pg = static_cast<unsigned>(std::min<long long>(ceil_div(n, 256), sm_count() * 48LL / n_views + 8));
        if (proj_mode == VS_PROJ_EXACT)
            launch_chained(project_view_kernel<VS_PROJ_EXACT>, dim3(pg, n_views), 256, 0, st, cams, f.fast, lat, lon, alt, n,
                                                                                  point_stride, f.colrow);
        else
            launch_chained(project_view_kernel<VS_PROJ_FAST>, dim3(pg, n_views), 256, 0, st, cams, f.fast, lat, lon, alt, n,
                                                                                 point_stride, f.colrow);
        VS_LAUNCH_CHECK("project_view_kernel");
    }
    if ((s = launch_moments(x, y, z, point_stride, nullptr, nullptr, f.colrow, nullptr, n_views, n, f, st)) != VS_OK)
        return s;
    launch_chained(solve_kernel, n_views, 64, 0, st, f.partial, blocks, f.norm, f.normf, cams, K, R, t, params, f.errcam,
                   status);
    VS_LAUNCH_CHECK("solve_kernel");
    if (!err) return VS_OK;
    return run_error_stats(x, y, z, point_stride, nullptr, nullptr, f.colrow, nullptr, n_views, n, f.errcam, err, ew,
                           st);
}
