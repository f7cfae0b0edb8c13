// RPCModel.inverse_projection (lib/rpc_model.py:170-249) for many cameras and points.
//
// The reference iterates all points of one camera together: from lon = lat = -1 (in the
// normalised frame) it projects the point and two finite-difference neighbours (steps 2,
// then 0.1), moves lon/lat by the projections of the image residual on the two difference
// vectors, and stops when EVERY point reprojects within sqrt(1e-18) of its target.  A
// point's result therefore depends on its camera's global iteration count.  Every FP64
// operation is the reference's (no contraction into FMA), so the results are bit-identical.
//
// The global count is found without a host round trip per iteration.  It is at least the
// largest over the points of the first iteration at which that point has converged, so
//   1. inverse_first_kernel iterates each warp's points, in registers, until every one of them has
//      converged once, keeps their state and posts that iteration (a maximum per camera);
//   2. inverse_advance_kernel takes every point on to the posted maximum and counts the points
//      that have left convergence again;
//   3. inverse_result_kernel writes the results, unless a point of the call was found unconverged: a
//      call that fails leaves its outputs as they were.
// No such point: done, with one host synchronisation.  Otherwise the camera goes on one iteration at
// a time (2 and 3, target + 1).  Every point runs each iteration once either way.  A launch does 32
// iterations at most; cameras that need more go on from the saved state.
#include <algorithm>
#include <vector>

#include "common.cuh"
#include "rpc.cuh"

namespace vs {
namespace {

// The kernels are bound by the FP64 pipe (19 sums and a share of the quotients per polynomial),
// which every SM has its own of: small blocks spread the points evenly over the SMs (90,001
// points: blocks of 64 hold every SM to within 8% of the mean load, blocks of 256 to 30%), and
// registers for 12 of them on an SM (whole calls, for 8, 10, 12 and 16: 90,001 points 560, 462, 471 and 477 us; four
// cameras of 30,000 points 681, 687, 664 and 639 us, of 300,000 points 5.73, 5.37, 5.40 and 5.62 ms).
// 90,001 points with the products on the FP64 pipe and a host synchronisation per iteration took 1111 us.
constexpr int kInvThreads = 64;
constexpr int kStateFields = 11;   // lon lat x0 y0 x1 y1 x2 y2 c_col c_row c_alt

struct InvState {
    double *f[kStateFields];
    int *k;                        // iterations done
};

// The three projections of an iteration share the products of the coordinates they share (the
// same values: the compiler computes each once), 364 of 540 per iteration.
struct Factor3 {
    Factor a, b, c;
};
struct Prod3 {
    Prod a, b, c;
};
struct Double3 {
    double a, b, c;
};
__device__ __forceinline__ Prod3 operator*(const RpcCoef &k, const Factor3 &f) { return {k * f.a, k * f.b, k * f.c}; }
__device__ __forceinline__ Prod3 operator*(const Prod3 &p, const Factor3 &f) {
    return {p.a * f.a, p.b * f.b, p.c * f.c};
}
__device__ __forceinline__ Double3 value(const Prod3 &p) { return {value(p.a), value(p.b), value(p.c)}; }
__device__ __forceinline__ Double3 sum(const Double3 &p, const Double3 &q) {
    return {da(p.a, q.a), da(p.b, q.b), da(p.c, q.c)};
}

// poly_factors at three points.
__device__ __forceinline__ Double3 poly_factors3(const RpcCoef *c, const Factor3 &x, const Factor3 &y,
                                                 const Factor3 &z) {
    const double c0 = value(c[0]);
    Double3 out{c0, c0, c0};
    out = sum(out, sum(sum(value(c[1] * y), value(c[2] * x)), value(c[3] * z)));
    out = sum(out, sum(sum(value(c[4] * y * x), value(c[5] * y * z)), value(c[6] * x * z)));
    out = sum(out, sum(sum(value(c[7] * y * y), value(c[8] * x * x)), value(c[9] * z * z)));
    out = sum(out, value(c[10] * x * y * z));
    out = sum(out, value(c[11] * y * y * y));
    out = sum(out, sum(sum(value(c[12] * y * x * x), value(c[13] * y * z * z)),
                     value(c[14] * y * y * x)));
    out = sum(out, value(c[15] * x * x * x));
    out = sum(out, sum(sum(value(c[16] * x * z * z), value(c[17] * y * y * z)),
                     value(c[18] * x * x * z)));
    out = sum(out, value(c[19] * z * z * z));
    return out;
}

__device__ __forceinline__ Double3 poly3(const RpcExact &s, int q, bool fast, const Factor3 &fx, const Factor3 &fy,
                                         const Factor3 &fz, const Double3 &x, const Double3 &y, double z) {
    if (fast) return poly_factors3(s.coef + 20 * q, fx, fy, fz);
    const double *c = s.cam.row_num + 20 * q;      // the camera's polynomials follow one another
    return {poly_exact(c, x.a, y.a, z), poly_exact(c, x.b, y.b, z), poly_exact(c, x.c, y.c, z)};
}

// the reference's three projections: at (lat, lon), (lat, lon + eps), (lat + eps, lon)
__device__ __forceinline__ void frames(const RpcExact &s, double lat, double lon, double alt, double eps,
                                       double (&o)[6]) {
    const double lon_e = __dadd_rn(lon, eps), lat_e = __dadd_rn(lat, eps);
    const Double3 x{lat, lat, lat_e}, y{lon, lon_e, lon};
    const bool fast = s.moderate && moderate(lat) && moderate(lat_e) && moderate(lon) && moderate(lon_e) && moderate(alt);
    const Factor3 fx{factor_of(lat), factor_of(lat), factor_of(lat_e)}, fy{factor_of(lon), factor_of(lon_e), factor_of(lon)};
    const Factor3 fz{factor_of(alt), factor_of(alt), factor_of(alt)};
#pragma unroll 1
    for (int axis = 0; axis < 2; ++axis) {         // rows, then columns
        Double3 num{0.0, 0.0, 0.0}, den{0.0, 0.0, 0.0};
#pragma unroll 1
        for (int d = 0; d < 2; ++d) {
            num = den;
            den = poly3(s, 2 * axis + d, fast, fx, fy, fz, x, y, alt);
        }
        const double q0 = __ddiv_rn(num.a, den.a), q1 = __ddiv_rn(num.b, den.b), q2 = __ddiv_rn(num.c, den.c);
        if (axis == 0) {
            o[1] = q0;
            o[3] = q1;
            o[5] = q2;
        } else {
            o[0] = q0;
            o[2] = q1;
            o[4] = q2;
        }
    }
}

// (x0 - c_col)^2 + (y0 - c_row)^2 < 1e-18 (false for NaN)
__device__ __forceinline__ bool converged(double x0, double y0, double cc, double cr) {
    const double dx = __dsub_rn(x0, cc), dy = __dsub_rn(y0, cr);
    return __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)) < 1e-18;
}

// One point: its position, projections and target in the normalised frame.
struct InvPoint {
    double lon, lat, o[6], cc, cr, ca;
};

// Iteration k (0-based) of one point.
__device__ __forceinline__ void inverse_iteration(const RpcExact &s, int k, InvPoint &p) {
    const double e1x = __dsub_rn(p.o[2], p.o[0]), e1y = __dsub_rn(p.o[3], p.o[1]);
    const double e2x = __dsub_rn(p.o[4], p.o[0]), e2y = __dsub_rn(p.o[5], p.o[1]);
    const double ux = __dsub_rn(p.cc, p.o[0]), uy = __dsub_rn(p.cr, p.o[1]);
    const double a1 = __ddiv_rn(__dadd_rn(__dmul_rn(ux, e1x), __dmul_rn(uy, e1y)),
                                __dadd_rn(__dmul_rn(e1x, e1x), __dmul_rn(e1y, e1y)));
    const double a2 = __ddiv_rn(__dadd_rn(__dmul_rn(ux, e2x), __dmul_rn(uy, e2y)),
                                __dadd_rn(__dmul_rn(e2x, e2x), __dmul_rn(e2y, e2y)));
    const double eps = k == 0 ? 2.0 : 0.1;
    p.lon = __dadd_rn(p.lon, __dmul_rn(a1, eps));
    p.lat = __dadd_rn(p.lat, __dmul_rn(a2, eps));
    frames(s, p.lat, p.lon, p.ca, 0.1, p.o);
}

__device__ __forceinline__ InvPoint load_point(const InvState &st, long long s) {
    InvPoint p;
    p.lon = st.f[0][s];
    p.lat = st.f[1][s];
#pragma unroll
    for (int q = 0; q < 6; ++q) p.o[q] = st.f[2 + q][s];
    p.cc = st.f[8][s];
    p.cr = st.f[9][s];
    p.ca = st.f[10][s];
    return p;
}

__device__ __forceinline__ void save_point(const InvState &st, long long s, const InvPoint &p, int k) {
    st.f[0][s] = p.lon;
    st.f[1][s] = p.lat;
#pragma unroll
    for (int q = 0; q < 6; ++q) st.f[2 + q][s] = p.o[q];
    st.f[8][s] = p.cc;
    st.f[9][s] = p.cr;
    st.f[10][s] = p.ca;
    st.k[s] = k;
}

// Iterations of a point in one launch.  A launch's time is then bounded whatever the caller's
// max_iter is (a point that never converges, a NaN, runs to max_iter); image points take 5 to 13.
constexpr int kInvBurst = 32;
constexpr int kUnfinished = 1, kBehind = 2;      // flags of InvCounters::state
constexpr int kAdvance = 1, kResume = 2;         // values of InvCounters::run

// Per camera: the largest posted iteration; whether a point has not converged yet (kUnfinished) or has
// not come to the posted iteration (kBehind); the points that do not reproject within the bound at the
// posted iteration; and whether the camera goes on.  open: set if there is any such point in the call.
struct InvCounters {
    int *target, *state, *count, *open, *run;
};

// Iterations up to `limit` of a warp's points (RESUME: of cameras with unfinished points, from the saved
// state), until every one of them has converged once.  The points of a warp share their count, which is
// saved complemented for a point that has not converged yet.  grid (points, cameras).
template <bool RESUME>
__global__ void __launch_bounds__(kInvThreads, 12) inverse_first_kernel(
    const VsRpcCamera *__restrict__ cams, const double *__restrict__ col, const double *__restrict__ row,
    const double *__restrict__ alt, long long n, long long stride, int limit, InvState st, InvCounters ct) {
    __shared__ RpcExact cam;
    const int c = blockIdx.y;
    if (RESUME && ct.run[c] != kResume) return;
    load_exact(cams + c, cam);
    const long long i = blockIdx.x * static_cast<long long>(kInvThreads) + threadIdx.x;
    const bool in = i < n;
    InvPoint p;
    bool done;
    int k = 0;
    if (RESUME) {
        const int saved = in ? st.k[c * n + i] : 0;
        p = load_point(st, c * n + (in ? i : n - 1));           // idle lanes: any point, done
        done = saved >= 0;
        k = __shfl_sync(0xffffffffu, done ? saved : ~saved, 0);
    } else {
        const long long g = c * stride + (in ? i : n - 1);      // idle lanes follow the last point
        p.cc = __ddiv_rn(__dsub_rn(col[g], cam.cam.col_off), cam.cam.col_scale);
        p.cr = __ddiv_rn(__dsub_rn(row[g], cam.cam.row_off), cam.cam.row_scale);
        p.ca = __ddiv_rn(__dsub_rn(alt[g], cam.cam.alt_off), cam.cam.alt_scale);
        p.lon = p.lat = -1.0;
        frames(cam, -1.0, -1.0, p.ca, 2.0, p.o);
        done = converged(p.o[0], p.o[1], p.cc, p.cr);
    }
    while (k < limit && !__all_sync(0xffffffffu, done)) {
        inverse_iteration(cam, k, p);
        ++k;
        done |= converged(p.o[0], p.o[1], p.cc, p.cr);
    }
    if (in) save_point(st, c * n + i, p, done ? k : ~k);
    if ((threadIdx.x & 31) == 0) atomicMax(ct.target + c, k);
    if (!done) {
        atomicOr(ct.state + c, kUnfinished);
        *ct.open = 1;
    }
}

// Takes the points of the cameras that go on (at first: all) and have no unfinished point towards
// iteration target[c], and counts those that do not reproject within the bound there.
__global__ void __launch_bounds__(kInvThreads, 12) inverse_advance_kernel(const VsRpcCamera *__restrict__ cams,
                                                                          long long n, InvState st, InvCounters ct,
                                                                          int first) {
    __shared__ RpcExact cam;
    const int c = blockIdx.y;
    chain_wait();
    // the same for a whole block: other blocks may set kBehind meanwhile, never kUnfinished
    if ((ct.state[c] & kUnfinished) || !(first || ct.run[c])) return;
    load_exact(cams + c, cam);
    const int to = ct.target[c];
    const long long i = blockIdx.x * static_cast<long long>(kInvThreads) + threadIdx.x;
    bool unconverged = false, behind = false;
    if (i < n) {
        const long long s = c * n + i;
        InvPoint p = load_point(st, s);
        const int from = st.k[s], end = min(to, from + kInvBurst);
        for (int k = from; k < end; ++k) inverse_iteration(cam, k, p);
        if (from < end) save_point(st, s, p, end);
        behind = end < to;
        unconverged = !behind && !converged(p.o[0], p.o[1], p.cc, p.cr);
    }
    const unsigned b = __ballot_sync(0xffffffffu, unconverged);
    const bool any_behind = __any_sync(0xffffffffu, behind);
    if ((threadIdx.x & 31) == 0 && (b || any_behind)) {
        if (b) atomicAdd(ct.count + c, __popc(b));
        if (any_behind) atomicOr(ct.state + c, kBehind);
        *ct.open = 1;
    }
}

// The results of a call whose points have all converged.
__global__ void __launch_bounds__(256) inverse_result_kernel(const VsRpcCamera *__restrict__ cams,
                                                             const double *__restrict__ alt, long long n,
                                                             long long stride, int normalized, InvState st,
                                                             InvCounters ct, double *__restrict__ lon_out,
                                                             double *__restrict__ lat_out,
                                                             double *__restrict__ alt_out) {
    chain_wait();
    const long long i = blockIdx.x * 256ll + threadIdx.x;
    if (*ct.open || i >= n) return;
    const int c = blockIdx.y;
    const VsRpcCamera &cam = cams[c];
    const long long s = c * n + i;
    const double lon = st.f[0][s], lat = st.f[1][s];
    if (normalized) {
        lon_out[s] = lon;
        lat_out[s] = lat;
        if (alt_out) alt_out[s] = st.f[10][s];
    } else {
        lon_out[s] = __dadd_rn(__dmul_rn(lon, cam.lon_scale), cam.lon_off);
        lat_out[s] = __dadd_rn(__dmul_rn(lat, cam.lat_scale), cam.lat_off);
        if (alt_out) alt_out[s] = alt[c * stride + i];
    }
}

InvState carve_inverse(Carver &cv, int n_cams, long long n, InvCounters &k) {
    InvState st;
    for (auto &f : st.f) f = cv.take<double>(static_cast<size_t>(n_cams) * n);
    st.k = cv.take<int>(static_cast<size_t>(n_cams) * n);
    const size_t m = n_cams;
    int *base = cv.take<int>(4 * m + 1);
    k = {base, base + m, base + 2 * m, base + 3 * m, base + 3 * m + 1};      // the first four: cleared together
    return st;
}

}  // namespace
}  // namespace vs

using namespace vs;

extern "C" size_t vs_rpc_inverse_project_workspace_size(int n_cams, int64_t n) {
    if (n_cams <= 0 || n < 0) return 0;
    Carver cv(nullptr);
    InvCounters k;
    carve_inverse(cv, n_cams, n, k);
    return cv.used + 256;
}

extern "C" int vs_rpc_inverse_project(const VsRpcCamera *cams, int n_cams, const double *col, const double *row,
                                      const double *alt, int64_t n, int64_t point_stride, int normalized,
                                      double *lon, double *lat, double *alt_out, int max_iter, int32_t *iterations,
                                      void *workspace, size_t workspace_bytes, void *stream) {
    VS_REQUIRE(n_cams > 0 && n_cams <= 65535 && n >= 0 && point_stride >= 0 && max_iter > 0,
               "vs_rpc_inverse_project: bad sizes");
    VS_REQUIRE(cams && workspace && (n == 0 || (col && row && alt && lon && lat)),
               "vs_rpc_inverse_project: null pointer");
    const size_t need = vs_rpc_inverse_project_workspace_size(n_cams, n);
    if (workspace_bytes < need) {
        set_error("vs_rpc_inverse_project: workspace %zu < %zu bytes", workspace_bytes, need);
        return VS_ERR_WORKSPACE;
    }
    if (n == 0) {
        if (iterations)
            for (int c = 0; c < n_cams; ++c) iterations[c] = 0;
        return VS_OK;
    }
    cudaStream_t st = as_stream(stream);
    Carver cv(workspace);
    InvCounters d;
    const InvState state = carve_inverse(cv, n_cams, n, d);
    const dim3 grid(static_cast<unsigned>(ceil_div(n, kInvThreads)), static_cast<unsigned>(n_cams));
    std::vector<int> h(3 * static_cast<size_t>(n_cams));      // targets, flags, counts
    const size_t bytes = sizeof(int) * n_cams;
    auto cuda_ok = [](cudaError_t e) {
        if (e != cudaSuccess) set_error("vs_rpc_inverse_project: %s", cudaGetErrorString(e));
        return e == cudaSuccess;
    };
    int limit = std::min(max_iter, kInvBurst);
    if (!cuda_ok(cudaMemsetAsync(d.target, 0, 3 * bytes + sizeof(int), st))) return VS_ERR_CUDA;
    inverse_first_kernel<false><<<grid, kInvThreads, 0, st>>>(cams, col, row, alt, n, point_stride, limit, state, d);
    VS_LAUNCH_CHECK("inverse_first_kernel");
    const dim3 wide(static_cast<unsigned>(ceil_div(n, 256)), static_cast<unsigned>(n_cams));
    std::vector<int> run(n_cams);
    std::vector<char> failed(n_cams, 0);
    int worst = n_cams;                       // the first camera that has failed
    for (int first = 1;; first = 0) {
        launch_chained(inverse_advance_kernel, grid, kInvThreads, 0, st, cams, n, state, d, first);
        VS_LAUNCH_CHECK("inverse_advance_kernel");
        if (worst == n_cams) {
            launch_chained(inverse_result_kernel, wide, 256, 0, st, cams, alt, n, point_stride, normalized, state, d, lon,
                           lat, alt_out);
            VS_LAUNCH_CHECK("inverse_result_kernel");
        }
        if (!cuda_ok(cudaMemcpyAsync(h.data(), d.target, 3 * bytes, cudaMemcpyDeviceToHost, st)) ||
            !cuda_ok(cudaStreamSynchronize(st)))
            return VS_ERR_CUDA;
        const int *target = h.data(), *flags = target + n_cams, *count = flags + n_cams;
        bool resume = false, any = false;
        const int reached = limit;
        for (int c = 0; c < n_cams; ++c) {
            const bool unfinished = flags[c] & kUnfinished, behind = flags[c] & kBehind;
            const bool open = unfinished || behind || count[c] > 0;
            if (open && !behind && (unfinished ? reached : target[c]) >= max_iter) {
                failed[c] = 1;
                worst = std::min(worst, c);
            }
            run[c] = !open || failed[c] ? 0 : (unfinished ? kResume : kAdvance);
            any |= run[c] != 0;
            resume |= run[c] == kResume;
            // points that left the bound again at the common iteration: their camera goes on by one
            if (run[c] == kAdvance && !behind) ++h[c];
        }
        if (!any) break;
        if (!cuda_ok(cudaMemcpyAsync(d.target, h.data(), bytes, cudaMemcpyHostToDevice, st)) ||
            !cuda_ok(cudaMemcpyAsync(d.run, run.data(), bytes, cudaMemcpyHostToDevice, st)) ||
            !cuda_ok(cudaMemsetAsync(d.state, 0, 2 * bytes + sizeof(int), st)))
            return VS_ERR_CUDA;
        if (resume) {
            limit = max_iter - limit > kInvBurst ? limit + kInvBurst : max_iter;
            inverse_first_kernel<true><<<grid, kInvThreads, 0, st>>>(cams, col, row, alt, n, point_stride, limit, state, d);
            VS_LAUNCH_CHECK("inverse_first_kernel");
        }
    }
    if (worst < n_cams) {
        set_error("vs_rpc_inverse_project: camera %d did not converge in %d iterations", worst, max_iter);
        return VS_ERR_DEGENERATE;
    }
    if (iterations)
        for (int c = 0; c < n_cams; ++c) iterations[c] = h[c];
    return VS_OK;
}
