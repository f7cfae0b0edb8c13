// (d) Fusion of per-view DSMs: the inline block of run_fuse (aggregate_2p5d.py:65-81).
//
// Per cell over the V views (float32, NaN = no measurement):
//   n = #valid; n <= 2 -> NaN                                    (aggregate_2p5d.py:69-71)
//   med = nanmedian: sorted s, ((0 + s[(n-1)/2]) + s[n/2]) / 2    (:74, numpy masked median)
//   mad = nanmedian(|x - med|)                                    (:75)
//   drop x with |x - med| > mad                                   (:76-77)
//   mean = nanmean: NaN -> 0, numpy's float32 pairwise sum over the V slots in view order
//          (8 accumulators for 8 <= V <= 128, halving above), started from 0, then the
//          float32 division by the kept count                     (:78)
// then optionally the 3x3 median blur (:81), launched from raster.cu's blur kernel.
// Cells of more than 64 views are shared by 2, 4 or 8 lanes, with the same arithmetic.
#include <algorithm>
#include <math.h>
#include <mutex>

#include "common.cuh"

namespace vs {
int launch_blur_f32(const float *in, float *out, long long h, long long w, cudaStream_t st);

namespace {

constexpr int kMaxViews = 512;
constexpr int kNaN = 0x7fffffff;

// ---- fusion for V <= 64 -------------------------------------------------------------------
// One thread fuses one cell:
//   * its V values as float32 with NaN replaced by +inf: the valid values are the n
//     smallest slots (ties with a valid +inf are the same value), so no key conversion is
//     needed, and the sign of a zero cannot change ((0 + lo) + hi) / 2, |x - med| or the
//     mask;
//   * Batcher's odd-even merge sort on N = V rounded up to 4 slots, derived from the
//     64-slot network by dropping the comparators that touch a slot >= N (those slots hold
//     +inf and every comparator puts its maximum on the higher slot, so they never change);
//   * the sorted values go to a per-thread column of shared memory, from which the
//     median's two middle order statistics are read;
//   * with a finite median m, the deviations of the sorted values split into two sorted
//     runs: fl(med - s) for the values left of the middle (ascending from the middle out)
//     and fl(s - med) for those right of it (fl(x - med) is monotone in x).  The MAD's
//     order statistics are the k-th and (k+1)-th smallest of the two runs: a binary search
//     over how many come from the left run (merge path), reading the column;
//   * the keep mask and numpy's pairwise mean read the values again in view order.
// The main kernel stages each tile of 128 cells (its V view rows, or its 128 x V block in
// the [H][W][V] layout) in shared memory with cp.async (the hardware tracks completion:
// no spin waits); each thread sorts its cell into its column of a view-major scratch
// block beside the tile (conflict-free) and reads the originals for the mean from the
// tile.  Stacks whose view rows are not 16-byte aligned are staged with 4-byte copies.
constexpr int kTileCells = 128;

__device__ __forceinline__ void cp_async16(float *smem_dst, const float *gmem_src) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async4(float *smem_dst, const float *gmem_src) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

template <int N>
__device__ __forceinline__ void cmpx(float (&a)[N], int i, int l) {
    const float lo = fminf(a[i], a[l]);
    a[l] = fmaxf(a[i], a[l]);
    a[i] = lo;
}

constexpr int pow2_ceil(int n) { return n <= 1 ? 1 : 2 * pow2_ceil((n + 1) / 2); }

// Batcher's odd-even merge sort network for N slots as a compile-time comparator list: the
// power-of-two network without the comparators that touch a slot >= N.
template <int N>
struct OemsNet {
    static constexpr int kP2 = pow2_ceil(N);
    static constexpr int kMax = 544;          // comparators of the 64-slot network
    int n = 0;
    unsigned char i[kMax] = {}, l[kMax] = {};
    constexpr OemsNet() {
        for (int p = 1; p < kP2; p <<= 1)
            for (int k = p; k >= 1; k >>= 1)
                for (int j = k % p; j + k <= kP2 - 1; j += 2 * k)
                    for (int q = 0; q < k; ++q)
                        if (q + j + k < N && (q + j) / (2 * p) == (q + j + k) / (2 * p)) {
                            i[n] = static_cast<unsigned char>(q + j);
                            l[n] = static_cast<unsigned char>(q + j + k);
                            ++n;
                        }
    }
};

// Sorts a[0..N) ascending (slots beyond the valid count hold +inf).
template <int N>
__device__ __forceinline__ void oems_sort(float (&a)[N]) {
    constexpr OemsNet<N> net{};
    constexpr int kCount = net.n;
#pragma unroll
    for (int c = 0; c < kCount; ++c) cmpx(a, net.i[c], net.l[c]);
}

__device__ __forceinline__ float median_pair(float lo, float hi) {
    return __fdiv_rn(__fadd_rn(__fadd_rn(0.0f, lo), hi), 2.0f);
}

// The median of the deviations |s(q) - med| of n sorted values with a finite median.
template <class S>
__device__ __forceinline__ float mad_of_sorted(const S &s, int n, float med) {
    const float inf = __int_as_float(0x7f800000);
    // left run A_j = med - s[m-1-j] (j < m), right run B_j = s[m+j] - med (j < n-m)
    const int m = (n & 1) ? (n - 1) >> 1 : n >> 1, nb = n - m;
    const int k = (n - 1) >> 1;
    int lo = max(0, k + 1 - nb), hi = min(k + 1, m);
    while (lo < hi) {
        const int i = (lo + hi) >> 1, j = k + 1 - i;
        if (__fsub_rn(med, s(m - 1 - i)) < __fsub_rn(s(m + j - 1), med)) lo = i + 1;
        else hi = i;
    }
    const int i = lo, j = k + 1 - i;
    const float a_last = i > 0 ? __fsub_rn(med, s(m - i)) : -inf;
    const float b_last = j > 0 ? __fsub_rn(s(m + j - 1), med) : -inf;
    const float kth = fmaxf(a_last, b_last);
    float nxt = kth;
    if (!(n & 1)) {
        const float a_next = i < m ? __fsub_rn(med, s(m - 1 - i)) : inf;
        const float b_next = j < nb ? __fsub_rn(s(m + j), med) : inf;
        nxt = fminf(a_next, b_next);
    }
    return median_pair(kth, nxt);
}

// The cell's values: value i at xs[i * si] (shared memory or global); sorted values are
// written to srt[i * ss] (shared memory); the values are read again, in view order, at
// xg[i * sg].
template <int N>
__device__ __forceinline__ float fuse_cell_v64(const float *xs, long long si, int V, float *srt, int ss,
                                               const float *__restrict__ xg, long long sg) {
    const float inf = __int_as_float(0x7f800000);
    float a[N];
    int n = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        float v = inf;
        if (i < V) {
            const float x = xs[i * si];
            const bool ok = !isnan(x);
            n += ok;
            v = ok ? x : inf;
        }
        a[i] = v;
    }
    if (n <= 2) return __int_as_float(0x7fffffff);
    oems_sort(a);
#pragma unroll
    for (int i = 0; i < N; ++i)
        if (i < V) srt[i * ss] = a[i];
    const float med = median_pair(srt[((n - 1) >> 1) * ss], srt[(n >> 1) * ss]);
    float mad = __int_as_float(0x7fffffff);
    if (isfinite(med)) {
        mad = mad_of_sorted([&](int q) -> const float & { return srt[q * ss]; }, n, med);
    } else {
        // deviations of the original values (inf - inf is NaN: missing)
        int nd = 0;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            float v = inf;
            if (i < V) {
                const float d = fabsf(__fsub_rn(xg[i * sg], med));
                const bool ok = !isnan(d);
                nd += ok;
                v = ok ? d : inf;
            }
            a[i] = v;
        }
        if (nd > 0) {
            oems_sort(a);
#pragma unroll
            for (int i = 0; i < N; ++i)
                if (i < V) srt[i * ss] = a[i];
            mad = median_pair(srt[((nd - 1) >> 1) * ss], srt[(nd >> 1) * ss]);
        }
    }
    // keep |x - med| <= mad (NaN compares false), then numpy's float32 pairwise sum of the
    // kept values (others 0) over the V slots in view order, from 0, / kept count
    int cnt = 0;
    auto kept = [&](int i, float &acc) {
        const float x = xg[i * sg];
        const bool keep = !isnan(x) && !(fabsf(__fsub_rn(x, med)) > mad);
        cnt += keep;
        acc = __fadd_rn(acc, keep ? x : 0.0f);
    };
    float res;
    if (V < 8) {
        res = 0.0f;
#pragma unroll
        for (int i = 0; i < (N < 8 ? N : 8); ++i)
            if (i < V) kept(i, res);
    } else {
        float r[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            r[j] = -0.0f;          // -0 + x == x for every x: the first kept value seeds r[j]
            kept(j, r[j]);
        }
        const int full = V - (V % 8);
#pragma unroll
        for (int b = 8; b < N; b += 8)
            if (b < full)
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (b + j < N) kept(b + j, r[j]);
        res = __fadd_rn(__fadd_rn(__fadd_rn(r[0], r[1]), __fadd_rn(r[2], r[3])),
                        __fadd_rn(__fadd_rn(r[4], r[5]), __fadd_rn(r[6], r[7])));
#pragma unroll
        for (int i = 8; i < N; ++i)
            if (i >= full && i < V) kept(i, res);
    }
    return __fdiv_rn(__fadd_rn(0.0f, res), static_cast<float>(cnt));   // cnt == 0 -> 0/0 = NaN
}

template <int N>
__global__ void __launch_bounds__(kTileCells) fuse_tile_kernel(const float *__restrict__ dsm, int layout, int V,
                                                               long long cells, float *__restrict__ out,
                                                               long long n_tiles, int aligned) {
    chain_wait();
    extern __shared__ __align__(16) float fsm[];           // the tile: V x 128 (VHW) or 128 x V (HWV)
    float *scratch = fsm + V * kTileCells;                 // sorted columns: N x 128
    const int t = threadIdx.x;
    const bool vhw = layout == VS_LAYOUT_VHW;
    for (long long tl = blockIdx.x; tl < n_tiles; tl += gridDim.x) {
        const long long c0 = tl * kTileCells;
        const int len = static_cast<int>(min(static_cast<long long>(kTileCells), cells - c0));   // multiple of 4
        if (aligned) {               // 16-byte copies: rows (VHW) or blocks (HWV) start 16-byte aligned
            if (vhw) {
                const int chunks = len >> 2;
                for (int q = t; q < V * (kTileCells / 4); q += kTileCells) {
                    const int v = q / (kTileCells / 4), ch = q - v * (kTileCells / 4);
                    if (ch < chunks) cp_async16(fsm + v * kTileCells + 4 * ch, dsm + v * cells + c0 + 4 * ch);
                }
            } else {
                const int chunks = (len * V) >> 2;
                for (int q = t; q < chunks; q += kTileCells) cp_async16(fsm + 4 * q, dsm + c0 * V + 4 * q);
            }
        } else if (vhw) {            // 4-byte copies otherwise (a thread per cell, so t < len)
            if (t < len)
                for (int v = 0; v < V; ++v) cp_async4(fsm + v * kTileCells + t, dsm + v * cells + c0 + t);
        } else {
            for (int q = t; q < len * V; q += kTileCells) cp_async4(fsm + q, dsm + c0 * V + q);
        }
        cp_async_commit();
        cp_async_wait_all();
        __syncthreads();
        const long long c = c0 + t;
        if (c < cells) {
            const float *col = vhw ? fsm + t : fsm + t * V;
            const int si = vhw ? kTileCells : 1;
            out[c] = fuse_cell_v64<N>(col, si, V, scratch + t, kTileCells, col, si);
        }
        __syncthreads();                           // the tile is refilled next
    }
}

// ---- fusion for 64 < V <= 512 -----------------------------------------------------------------
// L lanes of a warp fuse one cell: lane l holds values l, l + L, ... (at most 64, sorted by the
// network above for N slots), the lanes' runs are merged by bitonic exchanges (shuffles
// between lanes, registers within), and the sorted cell goes to shared memory, where the MAD
// is searched as above.  The pairwise mean's 8 accumulators are shared out the same way
// (accumulator j on lane j mod L), its sums formed as numpy forms them.
//
// Bound by the comparators (ALU pipe, two per clock and lane), like the kernel above.  One thread per
// cell would need up to 512 values in registers or local memory: the local-memory
// insertion sort this replaces took 1.98 ms for 97 views of 409 x 451 cells, this 0.094 ms.
// The layouts keep both the staging copies and the lanes' reads free of bank conflicts.
template <int L>
struct WideTile {
    static constexpr int CS = kTileCells / L;               // cells of a tile
    static constexpr int TS = CS + 32 / L;                  // view stride of a staged [V][cells] tile
    static constexpr int RS = 64 * CS + 32 / L;             // run stride of the sorted cells
    static constexpr int kSorted = L * RS;
    // cell pitch of a staged [cells][V] tile: congruent to L, so that 32 lanes meet 32 banks
    static __host__ __device__ int pitch(int V) { return V + ((L - V % 32 + 32) % 32); }
    static __host__ __device__ size_t floats(int layout, int V) {
        return layout == VS_LAYOUT_VHW ? static_cast<size_t>(V) * TS : static_cast<size_t>(CS) * pitch(V);
    }
};

// Sorts the cell's 64 L values (64 per lane, each lane's first N unsorted, the others +inf)
// across its lanes: rank 64 l + i ends in a[i] of lane l.
template <int N, int L>
__device__ __forceinline__ void wide_sort(float (&v)[N], float (&a)[64], int l) {
    oems_sort(v);
#pragma unroll
    for (int i = 0; i < 64; ++i) a[i] = i < N ? v[i < N ? i : 0] : __int_as_float(0x7f800000);
#pragma unroll
    for (int w = 1; w < L; w <<= 1) {
        // the halves of a group of 2w lanes are sorted: first against the other's reverse
        bool up = (l & w) != 0;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            const float t = __shfl_xor_sync(0xffffffffu, a[63 - i], 2 * w - 1);
            const float u = __shfl_xor_sync(0xffffffffu, a[i], 2 * w - 1);
            a[i] = up ? fmaxf(a[i], t) : fminf(a[i], t);
            a[63 - i] = up ? fmaxf(a[63 - i], u) : fminf(a[63 - i], u);
        }
#pragma unroll
        for (int d = w >> 1; d >= 1; d >>= 1) {
            up = (l & d) != 0;
#pragma unroll
            for (int i = 0; i < 64; ++i) {
                const float t = __shfl_xor_sync(0xffffffffu, a[i], d);
                a[i] = up ? fmaxf(a[i], t) : fminf(a[i], t);
            }
        }
#pragma unroll
        for (int d = 32; d >= 1; d >>= 1)
#pragma unroll
            for (int i = 0; i < 64; ++i)
                if (!(i & d)) cmpx(a, i, i + d);
    }
}

// Sum over the lanes of a cell.
template <int L>
__device__ __forceinline__ int lane_sum(int n) {
#pragma unroll
    for (int d = 1; d < L; d <<= 1) n += __shfl_xor_sync(0xffffffffu, n, d);
    return n;
}

// numpy's pairwise sum of x(0..n-1), n <= 128, on the cell's lanes (x(i) is asked of lane i mod
// L, and of every lane in the tail).
template <int L, class X>
__device__ __forceinline__ float wide_pairwise_block(const X &x, int first, int n, int l) {
    if (n < 8) {
        float res = 0.0f;
        for (int i = 0; i < n; ++i) res = __fadd_rn(res, x(first + i));
        return res;
    }
    constexpr int K = 8 / L;
    const int full = n - n % 8;
    float r[K];
#pragma unroll
    for (int k = 0; k < K; ++k) r[k] = x(first + k * L + l);
    for (int b = 8; b < full; b += 8)
#pragma unroll
        for (int k = 0; k < K; ++k) r[k] = __fadd_rn(r[k], x(first + b + k * L + l));
    // ((r0 + r1) + (r2 + r3)) + ((r4 + r5) + (r6 + r7)): neighbours first between the lanes, then
    // within one (a sum of two is the same on both)
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
        for (int d = 1; d < L; d <<= 1) r[k] = __fadd_rn(r[k], __shfl_xor_sync(0xffffffffu, r[k], d));
#pragma unroll
    for (int h = 1; h < K; h <<= 1)
#pragma unroll
        for (int k = 0; k + h < K; k += 2 * h) r[k] = __fadd_rn(r[k], r[k + h]);
    float res = r[0];
    for (int i = full; i < n; ++i) res = __fadd_rn(res, x(first + i));
    return res;
}

// numpy's halving recursion above 128 values, unrolled at compile time (no call stack): D levels
// cover n <= 512.
template <int L, int D, class X>
__device__ __forceinline__ float wide_pairwise(const X &x, int first, int n, int l) {
    if constexpr (D == 0) {
        return wide_pairwise_block<L>(x, first, n, l);
    } else {
        if (n <= 128) return wide_pairwise_block<L>(x, first, n, l);
        int n2 = n / 2;
        n2 -= n2 % 8;
        const float lo = wide_pairwise<L, D - 1>(x, first, n2, l);
        return __fadd_rn(lo, wide_pairwise<L, D - 1>(x, first + n2, n - n2, l));
    }
}

template <int N, int L>
__global__ void __launch_bounds__(kTileCells, 3) fuse_wide_kernel(const float *__restrict__ dsm, int layout, int V,
                                                               long long cells, float *__restrict__ out,
                                                               long long n_tiles, int aligned) {
    chain_wait();
    using T = WideTile<L>;
    extern __shared__ __align__(16) float fsm[];            // the sorted cells, then the tile
    float *tile = fsm + ((T::kSorted + 3) & ~3);
    const int tid = threadIdx.x, cell = tid / L, l = tid % L;
    const bool vhw = layout == VS_LAYOUT_VHW;
    const int pitch = T::pitch(V);
    const int sc = vhw ? 1 : pitch, sv = vhw ? T::TS : 1;
    const float inf = __int_as_float(0x7f800000);
    const float *mine = tile + cell * sc;                   // value v of the cell at mine[v * sv]
    auto sorted = [&](int q) -> float & { return fsm[(q & 63) * T::CS + (q >> 6) * T::RS + cell]; };
    for (long long tl = blockIdx.x; tl < n_tiles; tl += gridDim.x) {
        const long long c0 = tl * T::CS;
        const int len = static_cast<int>(min(static_cast<long long>(T::CS), cells - c0));
        if (vhw && aligned) {
            for (int q = tid; q < V * (T::CS / 4); q += kTileCells) {
                const int v = q / (T::CS / 4), ch = q - v * (T::CS / 4);
                if (4 * ch < len) cp_async16(tile + v * T::TS + 4 * ch, dsm + v * cells + c0 + 4 * ch);
            }
        } else if (vhw) {
            for (int q = tid; q < V * T::CS; q += kTileCells) {
                const int v = q / T::CS, c = q - v * T::CS;
                if (c < len) cp_async4(tile + v * T::TS + c, dsm + v * cells + c0 + c);
            }
        } else {                     // the tile is one run of len * V values
            int c = tid / V, v = tid - c * V;
            for (int q = tid; q < len * V; q += kTileCells) {
                cp_async4(tile + c * pitch + v, dsm + c0 * V + q);
                v += kTileCells;
                while (v >= V) {
                    v -= V;
                    ++c;
                }
            }
        }
        cp_async_commit();
        cp_async_wait_all();
        __syncthreads();
        const bool in = cell < len;
        // pass 0 sorts the values; a second pass, over the deviations, is only taken for a median
        // that is not finite
        int n = 0;
        float med = 0.0f, mad = __int_as_float(kNaN);
        bool again = false;
#pragma unroll 1
        for (int pass = 0; pass < 2; ++pass) {
            float v[N], a[64];
            int valid = 0;
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const int k = i * L + l;
                float x = inf;
                if (in && k < V) {
                    x = mine[k * sv];
                    if (pass) x = fabsf(__fsub_rn(x, med));
                    const bool ok = !isnan(x);
                    valid += ok;
                    x = ok ? x : inf;
                }
                v[i] = x;
            }
            valid = lane_sum<L>(valid);
            wide_sort<N, L>(v, a, l);
#pragma unroll
            for (int i = 0; i < 64; ++i) sorted(64 * l + i) = a[i];
            __syncwarp();
            if (pass == 0) {
                n = valid;
                if (n > 2) {
                    med = median_pair(sorted((n - 1) >> 1), sorted(n >> 1));
                    if (isfinite(med)) mad = mad_of_sorted(sorted, n, med);
                    else again = true;
                }
                __syncwarp();
                if (!__any_sync(0xffffffffu, again)) break;
            } else if (again && valid > 0) {
                mad = median_pair(sorted((valid - 1) >> 1), sorted(valid >> 1));
            }
        }
        // keep |x - med| <= mad, numpy's float32 pairwise sum of the kept values (others 0)
        int cnt = 0;
        auto kept = [&](int i) {
            const float x = in ? mine[i * sv] : 0.0f;
            const bool keep = !isnan(x) && !(fabsf(__fsub_rn(x, med)) > mad);
            cnt += keep && i % L == l;
            return keep ? x : 0.0f;
        };
        const float res = wide_pairwise<L, 4>(kept, 0, V, l);
        cnt = lane_sum<L>(cnt);
        if (in && l == 0)
            out[c0 + cell] = n <= 2 ? __int_as_float(kNaN) : __fdiv_rn(__fadd_rn(0.0f, res), static_cast<float>(cnt));
        __syncthreads();                           // the tile is refilled next
    }
}

// Lets a kernel take `bytes` of dynamic shared memory on the current device.  Asked for by every launch:
// the grant is the device's, so a flag kept per process left the second device without it.  The same
// value for every caller of a kernel, so that threads do not undo one another's.
template <typename Kernel>
bool allow_smem(Kernel kernel, size_t bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)) == cudaSuccess;
}

size_t fuse_tile_smem(int V, int N) { return sizeof(float) * static_cast<size_t>(V + N) * kTileCells; }

template <int N>
bool launch_fuse_v64(const float *dsm, int layout, int V, long long cells, float *out, bool aligned, cudaStream_t st) {
    const size_t sh = fuse_tile_smem(V, N);
    if (!allow_smem(fuse_tile_kernel<N>, fuse_tile_smem(N, N))) return false;     // the largest tile: V = N
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fuse_tile_kernel<N>, kTileCells, sh) != cudaSuccess ||
        per_sm <= 0)
        return false;
    const long long n_tiles = ceil_div(cells, static_cast<long long>(kTileCells));
    const unsigned g = static_cast<unsigned>(std::min<long long>(n_tiles, 1LL * sm_count() * per_sm));
    launch_chained(fuse_tile_kernel<N>, g, kTileCells, sh, st, dsm, layout, V, cells, out, n_tiles, aligned ? 1 : 0);
    return true;
}

template <int N, int L>
bool launch_fuse_wide_n(const float *dsm, int layout, int V, long long cells, float *out, bool aligned,
                        cudaStream_t st) {
    using T = WideTile<L>;
    const size_t base = (static_cast<size_t>(T::kSorted) + 3) & ~size_t(3);
    const size_t sh = sizeof(float) * (base + T::floats(layout, V));
    const size_t most = sizeof(float) * (base + std::max<size_t>(64 * L * T::TS, T::CS * (64 * L + 32)));    // V = 64 L
    if (!allow_smem(fuse_wide_kernel<N, L>, most)) return false;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fuse_wide_kernel<N, L>, kTileCells, sh) != cudaSuccess ||
        per_sm <= 0)
        return false;
    const long long n_tiles = ceil_div(cells, static_cast<long long>(T::CS));
    const unsigned g = static_cast<unsigned>(std::min<long long>(n_tiles, 1LL * sm_count() * per_sm));
    launch_chained(fuse_wide_kernel<N, L>, g, kTileCells, sh, st, dsm, layout, V, cells, out, n_tiles, aligned ? 1 : 0);
    return true;
}

// The fewest lanes that hold the views, each with the smallest of three networks that takes its share.  40 million
// values in all, networks of 44, 52 and 64: 72 views (2 lanes, 36 values each) 187, 202 and 232 us, 97 views (49) 151 us with 52,
// 175 with 64; 140 views (4 lanes, 35) 255, 288 and 320 us, 177 views (45) 219 and 247 us; 300 views (8 lanes, 38)
// 335, 346 and 383 us, 353 views (45) 299 and 327 us.  Each further network is three more kernels to compile.
template <int L>
bool launch_fuse_wide_l(const float *dsm, int layout, int V, long long cells, float *out, bool aligned,
                        cudaStream_t st) {
    const int share = (V + L - 1) / L;
    if (share <= 44) return launch_fuse_wide_n<44, L>(dsm, layout, V, cells, out, aligned, st);
    if (share <= 52) return launch_fuse_wide_n<52, L>(dsm, layout, V, cells, out, aligned, st);
    return launch_fuse_wide_n<64, L>(dsm, layout, V, cells, out, aligned, st);
}

// 16-byte copies need 16-byte aligned view rows (VHW) or cell blocks (HWV).
bool fuse_tile_aligned(const float *dsm, int layout, int V, long long cells) {
    (void)layout;
    (void)V;
    return (reinterpret_cast<uintptr_t>(dsm) & 15) == 0 && cells % 4 == 0;
}

int launch_fuse(const float *dsm, int layout, int V, long long cells, float *out, cudaStream_t st) {
    const bool aligned = fuse_tile_aligned(dsm, layout, V, cells);
    bool ok = false;
    if (V > 64) {
        ok = V <= 128   ? launch_fuse_wide_l<2>(dsm, layout, V, cells, out, aligned, st)
             : V <= 256 ? launch_fuse_wide_l<4>(dsm, layout, V, cells, out, aligned, st)
                        : launch_fuse_wide_l<8>(dsm, layout, V, cells, out, aligned, st);
    } else switch ((V + 3) / 4) {
        case 0: case 1: ok = launch_fuse_v64<4>(dsm, layout, V, cells, out, aligned, st); break;
        case 2: ok = launch_fuse_v64<8>(dsm, layout, V, cells, out, aligned, st); break;
        case 3: ok = launch_fuse_v64<12>(dsm, layout, V, cells, out, aligned, st); break;
        case 4: ok = launch_fuse_v64<16>(dsm, layout, V, cells, out, aligned, st); break;
        case 5: ok = launch_fuse_v64<20>(dsm, layout, V, cells, out, aligned, st); break;
        case 6: ok = launch_fuse_v64<24>(dsm, layout, V, cells, out, aligned, st); break;
        case 7: ok = launch_fuse_v64<28>(dsm, layout, V, cells, out, aligned, st); break;
        case 8: ok = launch_fuse_v64<32>(dsm, layout, V, cells, out, aligned, st); break;
        case 9: ok = launch_fuse_v64<36>(dsm, layout, V, cells, out, aligned, st); break;
        case 10: ok = launch_fuse_v64<40>(dsm, layout, V, cells, out, aligned, st); break;
        case 11: ok = launch_fuse_v64<44>(dsm, layout, V, cells, out, aligned, st); break;
        case 12: ok = launch_fuse_v64<48>(dsm, layout, V, cells, out, aligned, st); break;
        case 13: ok = launch_fuse_v64<52>(dsm, layout, V, cells, out, aligned, st); break;
        case 14: ok = launch_fuse_v64<56>(dsm, layout, V, cells, out, aligned, st); break;
        case 15: ok = launch_fuse_v64<60>(dsm, layout, V, cells, out, aligned, st); break;
        default: ok = launch_fuse_v64<64>(dsm, layout, V, cells, out, aligned, st); break;
    }
    if (!ok) {
        set_error("fuse_tile_kernel: launch configuration refused");
        return VS_ERR_CUDA;
    }
    return VS_OK;
}


}  // namespace
}  // namespace vs

using namespace vs;

// Largest grid (cells) the fusion accepts: the float32 grid plus its slack must stay well
// inside int64 (and size_t) arithmetic.
constexpr long long kMaxFuseCells = (1LL << 60) / static_cast<long long>(sizeof(float));

// h * w without overflow: 0 when either side is not positive or the product exceeds `limit`.
static long long checked_cells(int64_t h, int64_t w, long long limit) {
    if (h <= 0 || w <= 0 || h > limit || w > limit / h) return 0;
    return static_cast<long long>(h) * w;
}

extern "C" size_t vs_fuse_dsms_workspace_size(int64_t h, int64_t w) {
    const long long cells = checked_cells(h, w, kMaxFuseCells);
    if (!cells) return 0;
    return sizeof(float) * static_cast<size_t>(cells) + 256;
}

extern "C" int vs_fuse_dsms(const float *dsm, int layout, int64_t n_views, int64_t h, int64_t w, float *out,
                            int median_blur, void *workspace, size_t workspace_bytes, void *stream) {
    VS_REQUIRE(checked_cells(h, w, kMaxFuseCells) > 0 && n_views > 0 && n_views <= kMaxViews,
               "vs_fuse_dsms: bad sizes views=%lld grid=%lldx%lld", (long long)n_views, (long long)h,
               (long long)w);
    VS_REQUIRE(layout == VS_LAYOUT_HWV || layout == VS_LAYOUT_VHW, "vs_fuse_dsms: bad layout %d", layout);
    VS_REQUIRE(dsm && out, "vs_fuse_dsms: null pointer");
    cudaStream_t st = as_stream(stream);
    const long long cells = h * w;
    float *dst = out;
    if (median_blur) {
        const size_t need = vs_fuse_dsms_workspace_size(h, w);
        VS_REQUIRE(workspace, "vs_fuse_dsms: median_blur needs a workspace");
        if (workspace_bytes < need) {
            set_error("vs_fuse_dsms: workspace %zu < %zu bytes", workspace_bytes, need);
            return VS_ERR_WORKSPACE;
        }
        dst = static_cast<float *>(workspace);
    }
    const int V = static_cast<int>(n_views);
    const int s = launch_fuse(dsm, layout, V, cells, dst, st);
    if (s != VS_OK) return s;
    VS_LAUNCH_CHECK("fuse_kernel");
    if (median_blur) return launch_blur_f32(dst, out, h, w, st);
    return VS_OK;
}

// ---- fusion without any device allocation -------------------------------------------------
// Some callers cannot allocate device memory where they call the fusion: code running in a
// stream-ordered pipeline that forbids allocation after start-up, or a foreign host with no
// device allocator of its own.  vs_fuse_dsms_static keeps the blur's intermediate grid in
// this file-scope array instead of a caller workspace.  Every GPU that loads the library
// holds the array (16 MiB) until the process exits.
static __device__ __align__(256) float g_fuse_scratch[VS_FUSE_STATIC_MAX_CELLS + 64];   // + vs_fuse_dsms' 256 B slack

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_scratch_mutex;
float *g_scratch_ptr[kMaxDevices] = {};
}  // namespace

extern "C" int vs_fuse_dsms_static(const float *dsm, int layout, int64_t n_views, int64_t h, int64_t w, float *out,
                                   int median_blur, void *stream) {
    VS_REQUIRE(h > 0 && w > 0, "vs_fuse_dsms_static: bad grid %lldx%lld", (long long)h, (long long)w);
    // h and w are bounded before they are multiplied, so no product can wrap
    VS_REQUIRE(checked_cells(h, w, VS_FUSE_STATIC_MAX_CELLS) > 0,
               "vs_fuse_dsms_static: grid %lldx%lld exceeds the static scratch of %d cells", (long long)h,
               (long long)w, VS_FUSE_STATIC_MAX_CELLS);
    if (!median_blur) return vs_fuse_dsms(dsm, layout, n_views, h, w, out, 0, nullptr, 0, stream);
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
        set_error("vs_fuse_dsms_static: no usable current device");
        return VS_ERR_CUDA;
    }
    float *scratch = nullptr;
    {
        // device address of the array on the current device, looked up once per device
        // (the array's name in host code is only a host-side stand-in)
        std::lock_guard<std::mutex> lock(g_scratch_mutex);
        if (!g_scratch_ptr[dev]) {
            const cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void **>(&g_scratch_ptr[dev]), g_fuse_scratch);
            if (e != cudaSuccess) {
                g_scratch_ptr[dev] = nullptr;
                set_error("vs_fuse_dsms_static: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
                return VS_ERR_CUDA;
            }
        }
        scratch = g_scratch_ptr[dev];
    }
    // the fusion kernel writes every cell of the scratch grid before the blur reads it, so
    // nothing has to be cleared between calls
    return vs_fuse_dsms(dsm, layout, n_views, h, w, out, 1, scratch,
                        sizeof(float) * static_cast<size_t>(VS_FUSE_STATIC_MAX_CELLS + 64), stream);
}
