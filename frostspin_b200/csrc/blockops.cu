// Elementwise and reduction kernels over block lists (bandwidth-trivial ops of
// the SymmetricTensor API, kept on the device so that tensors stay resident).
#include <math.h>

#include "common.cuh"

namespace fsb {

constexpr int kOpThreads = 256;
// partial sums of the weighted reductions: a fixed count (two CTAs per SM of a
// 148-SM B200) so that the caller-owned scratch size does not depend on the GPU
constexpr int kReducePartials = 296;

__global__ void k_scale(double* __restrict__ x, int64_t n, double alpha) {
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        x[i] *= alpha;
}

__global__ void k_scale_by(double* __restrict__ x, int64_t n, const double* __restrict__ s,
                           int invert) {
    const double a = invert ? 1.0 / s[0] : s[0];
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        x[i] *= a;
}

__global__ void k_axpby(const double* __restrict__ x, double* __restrict__ y, int64_t n,
                        double a, double b) {
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        y[i] = (b == 0.0) ? a * x[i] : fma(a, x[i], b * y[i]);
}

__global__ void k_pow(const double* __restrict__ x, double* __restrict__ y, int64_t n,
                      double p) {
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const double v = x[i];
        double r;
        if (p == -1.0)
            r = 1.0 / v;
        else if (p == 2.0)
            r = v * v;
        else if (p == 0.5)
            r = sqrt(v);
        else if (p == -0.5)
            r = 1.0 / sqrt(v);
        else if (p == 1.0)
            r = v;
        else
            r = pow(v, p);
        y[i] = r;
    }
}

// Block-wide sum over T threads; result valid in thread 0.
template <int T>
__device__ __forceinline__ double block_sum(double v) {
    __shared__ double warp_part[T / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x % 32, wid = threadIdx.x / 32;
    __syncthreads();
    if (lane == 0) warp_part[wid] = v;
    __syncthreads();
    double r = 0.0;
    if (wid == 0) {
        r = (lane < T / 32) ? warp_part[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
    }
    return r;
}

// Block-wide sum of an integer, valid in every thread (sizes of a block list).
template <int T>
__device__ __forceinline__ int64_t block_total(int64_t v) {
    __shared__ int64_t part[T / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if (threadIdx.x % 32 == 0) part[threadIdx.x / 32] = v;
    __syncthreads();
    int64_t r = 0;
#pragma unroll
    for (int w = 0; w < T / 32; ++w) r += part[w];
    return r;
}

__device__ __forceinline__ int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// Where the share of a CTA that begins at unit `begin` of a list of n sizes starts:
// an entry at or before it, and the units before that entry.  kScan: by a scan of
// the list, for long ones: walking up to the share, a diagonal product of 96 blocks of
// 40 x 40 took 31 us and one of 256 blocks of 20 x 20 74 us, 10 and 27 us now.  Short
// lists are walked from their first entry (list_scanned).
template <bool kScan, int T, class Size>
__device__ __forceinline__ void list_start(int64_t n, int64_t begin, Size size, int64_t& first,
                                           int64_t& pos) {
    first = pos = 0;
    if (!kScan) return;
    __shared__ int64_t warp_sum[T / 32], found[2];
    const int lane = threadIdx.x % 32, wid = threadIdx.x / 32;
    if (threadIdx.x == 0) found[0] = n;
    int64_t done = 0;
    for (int64_t base = 0; base < n && done <= begin; base += T) {
        const int64_t q = base + threadIdx.x;
        const int64_t mine = q < n ? size(q) : 0;
        int64_t upto = mine;
#pragma unroll
        for (int o = 1; o < 32; o *= 2) {
            const int64_t v = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += v;
        }
        __syncthreads();   // the sums of the previous entries have been read
        if (lane == 31) warp_sum[wid] = upto;
        __syncthreads();
        upto += done;
#pragma unroll
        for (int w = 0; w < T / 32; ++w) {
            if (w < wid) upto += warp_sum[w];
            done += warp_sum[w];
        }
        if (upto - mine <= begin && begin < upto) {
            found[0] = q;
            found[1] = upto - mine;
        }
    }
    __syncthreads();
    // one value for the warp, so that the entries stay in uniform registers
    first = __shfl_sync(0xffffffffu, found[0], 0);
    pos = __shfl_sync(0xffffffffu, found[1], 0);
}

// mode 0: sum of squares, mode 1: plain sum.  Bound by HBM (8 bytes read per
// coefficient).  The concatenated segments are cut into one contiguous share
// per CTA, so that a CTA meets one or two segments whatever their number (200
// segments of 1 to 4 elements 20 us; 97 us in shares of at least 512 elements, all in
// one CTA), and each thread keeps eight 16-byte loads in flight (64 KB per CTA, two CTAs per
// SM; the copy bandwidth needs about 40 KB per SM).  The share of CTA b is a
// fixed function of the list, so the two-pass sum is deterministic.  12.2 M
// coefficients in 9 segments: 76 us before (every CTA strode over every
// segment, one 8-byte load per thread at a time), 17 us now.
constexpr int kReduceThreads = 512;
constexpr int kReduceUnroll = 8;

template <int MODE, bool kScan, class Table>
__global__ void __launch_bounds__(kReduceThreads, 2)
    k_weighted_reduce(const double* __restrict__ x, const __grid_constant__ Table segs,
                      int64_t n_segs, double* __restrict__ partial) {
    int64_t mine = 0;
    for (int64_t s = threadIdx.x; s < n_segs; s += kReduceThreads) mine += segs[s].length;
    const int64_t total = block_total<kReduceThreads>(mine);
    const int64_t share = ceil_div(total, gridDim.x);
    const int64_t begin = share * blockIdx.x;
    const int64_t end = begin + share < total ? begin + share : total;
    double acc = 0.0;
    int64_t s, pos;
    list_start<kScan, kReduceThreads>(n_segs, begin,
                                      [&](int64_t i) { return segs[i].length; }, s, pos);
    for (; s < n_segs && pos < end; ++s) {
        const FsSegment sg = segs[s];
        const int64_t lo = begin > pos ? begin - pos : 0;
        const int64_t hi = end - pos < sg.length ? end - pos : sg.length;
        pos += sg.length;
        if (hi <= lo) continue;
        const double* p = x + sg.offset + lo;
        int64_t n = hi - lo;
        double part = 0.0;
        // blocks start at any element: one leading element brings p to 16 bytes
        if (reinterpret_cast<uintptr_t>(p) & 8) {
            if (threadIdx.x == 0) part = (MODE == 0) ? p[0] * p[0] : p[0];
            ++p;
            --n;
        }
        const double2* p2 = reinterpret_cast<const double2*>(p);
        const int64_t n2 = n / 2;
        double sum[2] = {0.0, 0.0};
        for (int64_t i = threadIdx.x; i < n2; i += kReduceThreads * kReduceUnroll) {
            double2 v[kReduceUnroll];
#pragma unroll
            for (int u = 0; u < kReduceUnroll; ++u) {
                const int64_t k = i + u * kReduceThreads;
                v[u] = k < n2 ? __ldg(p2 + k) : make_double2(0.0, 0.0);
            }
#pragma unroll
            for (int u = 0; u < kReduceUnroll; ++u) {
                if (MODE == 0) {
                    sum[0] = fma(v[u].x, v[u].x, sum[0]);
                    sum[1] = fma(v[u].y, v[u].y, sum[1]);
                } else {
                    sum[0] += v[u].x;
                    sum[1] += v[u].y;
                }
            }
        }
        if ((n & 1) && threadIdx.x == 1) {
            const double v = __ldg(p + n - 1);
            part += (MODE == 0) ? v * v : v;
        }
        part += sum[0] + sum[1];
        acc = fma(sg.weight, part, acc);
    }
    const double r = block_sum<kReduceThreads>(acc);
    if (threadIdx.x == 0) partial[blockIdx.x] = r;
}

__global__ void __launch_bounds__(kOpThreads)
    k_final_sum(const double* __restrict__ partial, int64_t n, double* __restrict__ out) {
    double acc = 0.0;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) acc += partial[i];
    const double r = block_sum<kOpThreads>(acc);
    if (threadIdx.x == 0) out[0] = r;
}

// Units of the block-list kernels below: kUnit consecutive elements where both
// sides run in the same storage order, a kTile x kTile tile where they do not
// (one side goes through shared memory, so that both are read or written in
// rows of kTile consecutive doubles).  Units of all blocks are numbered block
// by block; a CTA takes one contiguous range of them.  Rows of kTile + 1
// doubles keep the transposed shared accesses free of bank conflicts.
constexpr int kTile = 64;
constexpr int kUnit = kTile * kTile;
constexpr int kPerThread = kUnit / kOpThreads;   // 16
constexpr int kRowStep = kOpThreads / 32;        // tile rows a pass covers

// Long blocks whose two sides run in different orders and whose shorter side is
// below kThin leave most of their tiles empty: they go element by element along the
// buffer whose rows are short (Turned), the other buffer in a few interleaved runs.
// Contractions of 9 M coefficients, tiles against this: side 1 664-724 / 42 us, 4
// 181-198 / 43 us, 8 101-108 / 44 us, 16 65 / 46 us; of 0.3 M: 8 15.3 / 13.3 us, 12
// 15.4 / 15.3 us, 16 13.3 / 15.3 us.  Diagonal products of 9 M: side 1 745-845 / 36-46
// us, 4 198-222 / 36-38 us, 8 103-120 / 36-38 us; of 0.3 M: 8 11.1 / 11.2 us.
constexpr int kThin = 16;
constexpr int kThinDiag = 10;

// A side of up to kUnit wastes no more than kTile tiles, less than a launch.
__device__ __host__ __forceinline__ bool is_thin(int64_t m, int64_t n, int limit) {
    return (m < limit || n < limit) && (m > kUnit || n > kUnit);
}

// Element f of a buffer with rows of `width` is element (f % width) * length + f / width
// of the buffer of the other order.  Rows of a run of kUnit elements come from
// one 32-bit multiply-high with constants computed once per block.
struct Turned {
    uint32_t width, mul, shift;
    int64_t length;
};

__device__ __forceinline__ Turned turned(int64_t width, int64_t length) {
    const uint32_t w = static_cast<uint32_t>(width), s = w > 1 ? 32 - __clz(w - 1) : 0;
    return {w, static_cast<uint32_t>((((1ull << s) - w) << 32) / w + 1), s, length};
}

// Pair: 0 trace, 1 same storage order (a plain dot product), 2 crossed, 3 crossed
// and thin.
__device__ __forceinline__ int pair_kind(const FsPairBlock& p) {
    if (p.b_off < 0) return 0;
    if ((p.a_trans != 0) != (p.b_trans != 0)) return 1;
    return is_thin(p.m, p.n, kThin) ? 3 : 2;
}

__device__ __forceinline__ int64_t pair_units(const FsPairBlock& p) {
    const int64_t m = p.m, n = p.n;
    switch (pair_kind(p)) {
        case 0: return ceil_div(m < n ? m : n, kUnit);
        case 2: return ceil_div(m, kTile) * ceil_div(n, kTile);
        default: return ceil_div(m * n, kUnit);
    }
}

// Bound by HBM (16 bytes read per coefficient pair).  The crossed form is the
// usual one (two C-order blocks: A by rows, B by columns); with one element per
// thread at a time B came in 8 useful bytes per 32-byte sector, after two
// 64-bit divisions.  Here a thread issues its 32 loads of a tile pair before
// the first use.  Two SU(2) corners of 13.1 M coefficients: 118 us before,
// 37 us now.
template <bool kScan, class Table>
__global__ void __launch_bounds__(kOpThreads, 2)
    k_pair_contract(const double* __restrict__ a, const double* __restrict__ b,
                    const __grid_constant__ Table pairs, int64_t n_pairs,
                    double* __restrict__ partial) {
    __shared__ double tile[kTile][kTile + 1];
    int64_t mine = 0;
    for (int64_t q = threadIdx.x; q < n_pairs; q += kOpThreads) mine += pair_units(pairs[q]);
    const int64_t total = block_total<kOpThreads>(mine);
    const int64_t begin = total * blockIdx.x / gridDim.x;
    const int64_t end = total * (blockIdx.x + 1) / gridDim.x;
    const int lane = threadIdx.x % 32, wid = threadIdx.x / 32;
    double acc = 0.0;
    int64_t q, pos;
    list_start<kScan, kOpThreads>(n_pairs, begin,
                                  [&](int64_t i) { return pair_units(pairs[i]); }, q, pos);
    for (; q < n_pairs && pos < end; ++q) {
        const FsPairBlock pb = pairs[q];
        const int64_t units = pair_units(pb);
        const int64_t lo = begin > pos ? begin - pos : 0;
        const int64_t hi = end - pos < units ? end - pos : units;
        pos += units;
        const int kind = pair_kind(pb);
        double part = 0.0;
        const double* pa = a + pb.a_off;
        const double* pbm = b + pb.b_off;
        // storage of A: R rows of C (B then holds C rows of R)
        const int64_t R = pb.a_trans ? pb.n : pb.m, C = pb.a_trans ? pb.m : pb.n;
        for (int64_t u = lo; u < hi; ++u) {
            if (kind == 0) {
                const int64_t d = R < C ? R : C;
#pragma unroll 4
                for (int k = 0; k < kPerThread; ++k) {
                    const int64_t i = u * kUnit + k * kOpThreads + threadIdx.x;
                    if (i < d) part += __ldg(pa + i * C + i);
                }
            } else if (kind == 1) {
                double va[kPerThread], vb[kPerThread];
#pragma unroll
                for (int k = 0; k < kPerThread; ++k) {
                    const int64_t f = u * kUnit + k * kOpThreads + threadIdx.x;
                    va[k] = f < R * C ? __ldg(pa + f) : 0.0;
                    vb[k] = f < R * C ? __ldg(pbm + f) : 0.0;
                }
#pragma unroll
                for (int k = 0; k < kPerThread; ++k) part = fma(va[k], vb[k], part);
            } else if (kind == 3) {
                // A has R rows of C, B has C rows of R
                const Turned t = turned(C <= R ? C : R, C <= R ? R : C);
                const double* walked = C <= R ? pa : pbm;
                const double* other = C <= R ? pbm : pa;
                const int64_t f0 = u * kUnit, i0 = f0 / t.width;
                const uint32_t j0 = static_cast<uint32_t>(f0 - i0 * t.width);
                double va[kPerThread], vb[kPerThread];
#pragma unroll
                for (int k = 0; k < kPerThread; ++k) {
                    const uint32_t e = k * kOpThreads + threadIdx.x;
                    va[k] = vb[k] = 0.0;
                    if (f0 + e < R * C) {
                        const uint32_t l = j0 + e, r = fast_div(l, t.mul, t.shift);
                        va[k] = __ldg(walked + f0 + e);
                        vb[k] = __ldg(other + (l - r * t.width) * t.length + i0 + r);
                    }
                }
#pragma unroll
                for (int k = 0; k < kPerThread; ++k) part = fma(va[k], vb[k], part);
            } else {
                const int64_t ct = ceil_div(C, kTile);
                const int64_t r0 = (u / ct) * kTile, c0 = (u % ct) * kTile;
                double va[kPerThread], vb[kPerThread];
#pragma unroll
                for (int k = 0; k < kPerThread; ++k) {
                    const int i = wid + (k / 2) * kRowStep, j = lane + (k % 2) * 32;
                    va[k] = (r0 + i < R && c0 + j < C) ? __ldg(pa + (r0 + i) * C + c0 + j) : 0.0;
                    vb[k] = (c0 + i < C && r0 + j < R) ? __ldg(pbm + (c0 + i) * R + r0 + j) : 0.0;
                }
                __syncthreads();  // the previous tile has been read
#pragma unroll
                for (int k = 0; k < kPerThread; ++k)
                    tile[wid + (k / 2) * kRowStep][lane + (k % 2) * 32] = vb[k];
                __syncthreads();
                // entries outside the block are zero in va and in the tile, so a
                // special value of either side meets only its own partner
#pragma unroll
                for (int k = 0; k < kPerThread; ++k)
                    part = fma(va[k], tile[lane + (k % 2) * 32][wid + (k / 2) * kRowStep], part);
            }
        }
        acc = fma(pb.weight, part, acc);
    }
    const double r = block_sum<kOpThreads>(acc);
    if (threadIdx.x == 0) partial[blockIdx.x] = r;
}

__host__ __device__ __forceinline__ bool diag_thin(const FsDiagBlock& d) {
    return d.x_trans && is_thin(d.m, d.n, kThinDiag);
}

// units of a block in k_diag_mul, and in k_diag_thin
__device__ __forceinline__ int64_t diag_units(const FsDiagBlock& d) {
    const int64_t m = d.m, n = d.n;
    if (diag_thin(d)) return 0;
    return d.x_trans ? ceil_div(m, kTile) * ceil_div(n, kTile) : ceil_div(m * n, kUnit);
}

__device__ __forceinline__ int64_t diag_thin_units(const FsDiagBlock& d) {
    return diag_thin(d) ? ceil_div(static_cast<int64_t>(d.m) * d.n, kUnit) : 0;
}

// Bound by HBM (16 bytes per coefficient).  The row of an element comes from
// one 32-bit multiply-high with the constants of the block's column count,
// computed once per block, and a thread issues eight loads before its stores;
// F-order inputs go through a shared tile.  12.2 M coefficients in 9 blocks:
// 63 us before (a 64-bit division per element, one load at a time),
// 36 us now.
template <bool kScan, class Table>
__global__ void __launch_bounds__(kOpThreads, 4)
    k_diag_mul(const double* __restrict__ x, const double* __restrict__ diag,
               double* __restrict__ out, const __grid_constant__ Table blocks,
               int64_t n_blocks) {
    __shared__ double tile[kTile][kTile + 1];
    int64_t mine = 0;
    for (int64_t q = threadIdx.x; q < n_blocks; q += kOpThreads) mine += diag_units(blocks[q]);
    const int64_t total = block_total<kOpThreads>(mine);
    const int64_t begin = total * blockIdx.x / gridDim.x;
    const int64_t end = total * (blockIdx.x + 1) / gridDim.x;
    const int lane = threadIdx.x % 32, wid = threadIdx.x / 32;
    constexpr int kBatch = 8;
    int64_t q, pos;
    list_start<kScan, kOpThreads>(n_blocks, begin,
                                  [&](int64_t i) { return diag_units(blocks[i]); }, q, pos);
    for (; q < n_blocks && pos < end; ++q) {
        const FsDiagBlock db = blocks[q];
        const int64_t units = diag_units(db);
        const int64_t lo = begin > pos ? begin - pos : 0;
        const int64_t hi = end - pos < units ? end - pos : units;
        pos += units;
        if (hi <= lo) continue;
        const int64_t m = db.m, n = db.n;
        const double* px = x + db.x_off;
        const double* pd = diag + db.d_off;
        double* po = out + db.out_off;
        if (!db.x_trans) {
            const uint32_t d = static_cast<uint32_t>(db.n);
            const uint32_t sh = d > 1 ? 32 - __clz(d - 1) : 0;
            const uint32_t mul = static_cast<uint32_t>(((((1ull << sh) - d) << 32) / d) + 1);
            for (int64_t u = lo; u < hi; ++u) {
                const int64_t f0 = u * kUnit;
                const int64_t i0 = f0 / n;
                const uint32_t j0 = static_cast<uint32_t>(f0 - i0 * n);
                const int64_t left = m * n - f0;
                const int cnt = left < kUnit ? static_cast<int>(left) : kUnit;
#pragma unroll
                for (int h = 0; h < kPerThread; h += kBatch) {
                    double v[kBatch], w[kBatch];
#pragma unroll
                    for (int k = 0; k < kBatch; ++k) {
                        const int t = (h + k) * kOpThreads + threadIdx.x;
                        v[k] = w[k] = 0.0;
                        if (t < cnt) {
                            v[k] = __ldg(px + f0 + t);
                            const uint32_t l = j0 + t;
                            const uint32_t r = fast_div(l, mul, sh);
                            w[k] = __ldg(pd + (db.left ? i0 + r : static_cast<int64_t>(l - r * d)));
                        }
                    }
#pragma unroll
                    for (int k = 0; k < kBatch; ++k) {
                        const int t = (h + k) * kOpThreads + threadIdx.x;
                        if (t < cnt) po[f0 + t] = v[k] * w[k];
                    }
                }
            }
        } else {
            const int64_t jt = ceil_div(n, kTile);
            for (int64_t u = lo; u < hi; ++u) {
                const int64_t i0 = (u / jt) * kTile, j0 = (u % jt) * kTile;
                __syncthreads();  // the previous tile has been read
#pragma unroll
                for (int h = 0; h < kPerThread; h += kBatch) {
                    double v[kBatch];
#pragma unroll
                    for (int k = 0; k < kBatch; ++k) {
                        const int j = wid + ((h + k) / 2) * kRowStep, i = lane + (k % 2) * 32;
                        v[k] = (j0 + j < n && i0 + i < m) ? __ldg(px + (j0 + j) * m + i0 + i) : 0.0;
                    }
#pragma unroll
                    for (int k = 0; k < kBatch; ++k)
                        tile[wid + ((h + k) / 2) * kRowStep][lane + (k % 2) * 32] = v[k];
                }
                __syncthreads();
#pragma unroll
                for (int k = 0; k < kPerThread; ++k) {
                    const int i = wid + (k / 2) * kRowStep, j = lane + (k % 2) * 32;
                    if (i0 + i < m && j0 + j < n)
                        po[(i0 + i) * n + j0 + j] =
                            tile[j][i] * __ldg(pd + (db.left ? i0 + i : j0 + j));
                }
            }
        }
    }
}

// The thin transposed blocks of a list (x has n rows of m, the output m rows of n).
// Apart, since this form took the registers that the others keep their loads in (9
// blocks of 1200 x 1200 42 us, 46 us with all forms in one kernel).
template <bool kScan, class Table>
__global__ void __launch_bounds__(kOpThreads, 4)
    k_diag_thin(const double* __restrict__ x, const double* __restrict__ diag,
                double* __restrict__ out, const __grid_constant__ Table blocks,
                int64_t n_blocks) {
    int64_t mine = 0;
    for (int64_t q = threadIdx.x; q < n_blocks; q += kOpThreads) mine += diag_thin_units(blocks[q]);
    const int64_t total = block_total<kOpThreads>(mine);
    const int64_t begin = total * blockIdx.x / gridDim.x;
    const int64_t end = total * (blockIdx.x + 1) / gridDim.x;
    constexpr int kBatch = 8;
    int64_t q, pos;
    list_start<kScan, kOpThreads>(n_blocks, begin,
                                  [&](int64_t i) { return diag_thin_units(blocks[i]); }, q, pos);
    for (; q < n_blocks && pos < end; ++q) {
        const FsDiagBlock db = blocks[q];
        const int64_t units = diag_thin_units(db);
        const int64_t lo = begin > pos ? begin - pos : 0;
        const int64_t hi = end - pos < units ? end - pos : units;
        pos += units;
        if (hi <= lo) continue;
        const int64_t m = db.m, n = db.n;
        const double* px = x + db.x_off;
        const double* pd = diag + db.d_off;
        double* po = out + db.out_off;
        const bool by_out = n <= m;   // the output's rows are the short ones
        const Turned t = turned(by_out ? n : m, by_out ? m : n);
        const bool major = by_out == (db.left != 0);   // the weight goes with f / width
        for (int64_t u = lo; u < hi; ++u) {
            const int64_t f0 = u * kUnit, i0 = f0 / t.width;
            const uint32_t j0 = static_cast<uint32_t>(f0 - i0 * t.width);
            const int64_t left = m * n - f0;
            const int cnt = left < kUnit ? static_cast<int>(left) : kUnit;
#pragma unroll
            for (int h = 0; h < kPerThread; h += kBatch) {
                double v[kBatch], w[kBatch];
                int64_t at[kBatch];
#pragma unroll
                for (int k = 0; k < kBatch; ++k) {
                    const int e = (h + k) * kOpThreads + threadIdx.x;
                    v[k] = w[k] = 0.0;
                    if (e < cnt) {
                        const uint32_t l = j0 + e, r = fast_div(l, t.mul, t.shift);
                        const uint32_t c = l - r * t.width;
                        const int64_t turn = c * t.length + i0 + r;
                        v[k] = __ldg(px + (by_out ? turn : f0 + e));
                        w[k] = __ldg(pd + (major ? i0 + r : static_cast<int64_t>(c)));
                        at[k] = by_out ? f0 + e : turn;
                    }
                }
#pragma unroll
                for (int k = 0; k < kBatch; ++k)
                    if ((h + k) * kOpThreads + static_cast<int>(threadIdx.x) < cnt)
                        po[at[k]] = v[k] * w[k];
            }
        }
    }
}

inline int elementwise_grid(int64_t n) {
    int64_t g = (n + kOpThreads - 1) / kOpThreads;
    const int64_t cap = static_cast<int64_t>(num_sms()) * 16;
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    return static_cast<int>(g);
}

}  // namespace fsb

extern "C" int fs_reduce_partials(void) { return fsb::kReducePartials; }

extern "C" int fs_scale(double* d_x, int64_t n, double alpha, void* stream) {
    if (n < 0) return FS_ERR_INVALID_ARG;
    if (n == 0) return FS_OK;
    if (d_x == nullptr) return FS_ERR_INVALID_ARG;
    fsb::k_scale<<<fsb::elementwise_grid(n), fsb::kOpThreads, 0, fsb::as_stream(stream)>>>(
        d_x, n, alpha);
    return fsb::launch_status();
}

extern "C" int fs_scale_by(double* d_x, int64_t n, const double* d_scalar, int32_t invert,
                           void* stream) {
    if (n < 0) return FS_ERR_INVALID_ARG;
    if (n == 0) return FS_OK;
    if (d_x == nullptr || d_scalar == nullptr) return FS_ERR_INVALID_ARG;
    fsb::k_scale_by<<<fsb::elementwise_grid(n), fsb::kOpThreads, 0, fsb::as_stream(stream)>>>(
        d_x, n, d_scalar, invert);
    return fsb::launch_status();
}

extern "C" int fs_axpby(const double* d_x, double* d_y, int64_t n, double a, double b,
                        void* stream) {
    if (n < 0) return FS_ERR_INVALID_ARG;
    if (n == 0) return FS_OK;
    if (d_x == nullptr || d_y == nullptr) return FS_ERR_INVALID_ARG;
    fsb::k_axpby<<<fsb::elementwise_grid(n), fsb::kOpThreads, 0, fsb::as_stream(stream)>>>(
        d_x, d_y, n, a, b);
    return fsb::launch_status();
}

extern "C" int fs_pow(const double* d_x, double* d_y, int64_t n, double p, void* stream) {
    if (n < 0) return FS_ERR_INVALID_ARG;
    if (n == 0) return FS_OK;
    if (d_x == nullptr || d_y == nullptr) return FS_ERR_INVALID_ARG;
    fsb::k_pow<<<fsb::elementwise_grid(n), fsb::kOpThreads, 0, fsb::as_stream(stream)>>>(
        d_x, d_y, n, p);
    return fsb::launch_status();
}

namespace {

// Lists of more entries than these are scanned.  Walked against scanned: contraction
// of 40 blocks of 40 x 40 16.6 / 11.6 us and of 4000 x 130 68.0 / 64.5 us, sum of
// squares 16.5 / 9.8 and 35.4 / 35.0 us, diagonal product of 17 blocks of 40 x 40 8.4 /
// 6.4 us, but of 9 of 1200 x 1200 37.5 / 39.1 us; 17 large blocks gain the sums nothing.
constexpr int64_t kReduceWalk = 24, kPairWalk = 24, kDiagWalk = 12;

// A table in device memory is longer, and scanned whatever its length.
template <class Table>
constexpr bool kInDevice = false;
template <class T>
constexpr bool kInDevice<fsb::DeviceTable<T>> = true;

template <class Table>
bool list_scanned(int64_t n, int64_t walk) {
    return kInDevice<Table> || n > walk;
}

template <int MODE, class Table>
int weighted_reduce(const double* d_x, const Table& segs, int64_t n_segs, double* d_partial,
                    int64_t n_partial, double* d_out, void* stream) {
    if (n_partial < fsb::kReducePartials) return FS_ERR_INVALID_ARG;
    if (d_partial == nullptr || d_out == nullptr) return FS_ERR_INVALID_ARG;
    if (n_segs > 0 && d_x == nullptr) return FS_ERR_INVALID_ARG;
    cudaStream_t s = fsb::as_stream(stream);
    const auto kernel = list_scanned<Table>(n_segs, kReduceWalk)
                            ? fsb::k_weighted_reduce<MODE, true, Table>
                            : fsb::k_weighted_reduce<MODE, kInDevice<Table>, Table>;
    kernel<<<fsb::kReducePartials, fsb::kReduceThreads, 0, s>>>(d_x, segs, n_segs, d_partial);
    int st = fsb::launch_status();
    if (st != FS_OK) return st;
    fsb::k_final_sum<<<1, fsb::kOpThreads, 0, s>>>(d_partial, fsb::kReducePartials, d_out);
    return fsb::launch_status();
}

template <class Table>
int pair_contract(const double* d_a, const double* d_b, const Table& pairs, int64_t n_pairs,
                  double* d_partial, int64_t n_partial, double* d_out, void* stream) {
    if (n_partial < fsb::kReducePartials) return FS_ERR_INVALID_ARG;
    if (d_partial == nullptr || d_out == nullptr) return FS_ERR_INVALID_ARG;
    if (n_pairs > 0 && d_a == nullptr) return FS_ERR_INVALID_ARG;
    cudaStream_t s = fsb::as_stream(stream);
    const auto kernel = list_scanned<Table>(n_pairs, kPairWalk)
                            ? fsb::k_pair_contract<true, Table>
                            : fsb::k_pair_contract<kInDevice<Table>, Table>;
    kernel<<<fsb::kReducePartials, fsb::kOpThreads, 0, s>>>(d_a, d_b, pairs, n_pairs, d_partial);
    int st = fsb::launch_status();
    if (st != FS_OK) return st;
    fsb::k_final_sum<<<1, fsb::kOpThreads, 0, s>>>(d_partial, fsb::kReducePartials, d_out);
    return fsb::launch_status();
}

// some, all: whether the list has thin blocks, and no others
template <class Table>
int diag_mul(const double* d_x, const double* d_diag, double* d_out, const Table& blocks,
             int64_t n_blocks, bool some, bool all, void* stream) {
    if (d_x == nullptr || d_diag == nullptr || d_out == nullptr) return FS_ERR_INVALID_ARG;
    // one wave of resident CTAs; CTAs without a unit return at once
    const int grid = 4 * fsb::num_sms();
    const bool scan = list_scanned<Table>(n_blocks, kDiagWalk);
    cudaStream_t s = fsb::as_stream(stream);
    if (!all) {
        const auto kernel = scan ? fsb::k_diag_mul<true, Table>
                                 : fsb::k_diag_mul<kInDevice<Table>, Table>;
        kernel<<<grid, fsb::kOpThreads, 0, s>>>(d_x, d_diag, d_out, blocks, n_blocks);
        const int st = fsb::launch_status();
        if (st != FS_OK) return st;
    }
    if (!some) return FS_OK;
    const auto kernel = scan ? fsb::k_diag_thin<true, Table>
                             : fsb::k_diag_thin<kInDevice<Table>, Table>;
    kernel<<<grid, fsb::kOpThreads, 0, s>>>(d_x, d_diag, d_out, blocks, n_blocks);
    return fsb::launch_status();
}

using SegmentList = fsb::InlineTable<FsSegment, FS_LIST_MAX>;
using PairList = fsb::InlineTable<FsPairBlock, FS_LIST_MAX>;
using DiagList = fsb::InlineTable<FsDiagBlock, FS_LIST_MAX>;
static_assert(sizeof(SegmentList) < 4000 && sizeof(PairList) < 4000 && sizeof(DiagList) < 4000,
              "lists share the 4 KB of kernel parameters");

// status of a host list of n entries
int list_status(const void* h, int64_t n) {
    if (n < 0 || (n > 0 && h == nullptr)) return FS_ERR_INVALID_ARG;
    return n > FS_LIST_MAX ? FS_ERR_TOO_LARGE : FS_OK;
}

}  // namespace

extern "C" int fs_weighted_sumsq(const double* d_x, const FsSegment* d_segs, int64_t n_segs,
                                 double* d_partial, int64_t n_partial, double* d_out,
                                 void* stream) {
    if (n_segs < 0 || (n_segs > 0 && d_segs == nullptr)) return FS_ERR_INVALID_ARG;
    return weighted_reduce<0>(d_x, fsb::DeviceTable<FsSegment>{d_segs}, n_segs, d_partial,
                              n_partial, d_out, stream);
}

extern "C" int fs_weighted_sum(const double* d_x, const FsSegment* d_segs, int64_t n_segs,
                               double* d_partial, int64_t n_partial, double* d_out,
                               void* stream) {
    if (n_segs < 0 || (n_segs > 0 && d_segs == nullptr)) return FS_ERR_INVALID_ARG;
    return weighted_reduce<1>(d_x, fsb::DeviceTable<FsSegment>{d_segs}, n_segs, d_partial,
                              n_partial, d_out, stream);
}

extern "C" int fs_weighted_sum_list(const double* d_x, const FsSegment* h_segs, int64_t n_segs,
                                    int32_t squares, double* d_partial, int64_t n_partial,
                                    double* d_out, void* stream) {
    const int st = list_status(h_segs, n_segs);
    if (st != FS_OK) return st;
    const SegmentList t = fsb::inline_table<FsSegment, FS_LIST_MAX>(h_segs, n_segs);
    return squares ? weighted_reduce<0>(d_x, t, n_segs, d_partial, n_partial, d_out, stream)
                   : weighted_reduce<1>(d_x, t, n_segs, d_partial, n_partial, d_out, stream);
}

extern "C" int fs_pair_contract(const double* d_a, const double* d_b,
                                const FsPairBlock* d_pairs, int64_t n_pairs,
                                double* d_partial, int64_t n_partial, double* d_out,
                                void* stream) {
    if (n_pairs < 0 || (n_pairs > 0 && d_pairs == nullptr)) return FS_ERR_INVALID_ARG;
    return pair_contract(d_a, d_b, fsb::DeviceTable<FsPairBlock>{d_pairs}, n_pairs, d_partial,
                         n_partial, d_out, stream);
}

extern "C" int fs_pair_contract_list(const double* d_a, const double* d_b,
                                     const FsPairBlock* h_pairs, int64_t n_pairs,
                                     double* d_partial, int64_t n_partial, double* d_out,
                                     void* stream) {
    const int st = list_status(h_pairs, n_pairs);
    if (st != FS_OK) return st;
    return pair_contract(d_a, d_b, fsb::inline_table<FsPairBlock, FS_LIST_MAX>(h_pairs, n_pairs),
                         n_pairs, d_partial, n_partial, d_out, stream);
}

extern "C" int fs_diag_mul(const double* d_x, const double* d_diag, double* d_out,
                           const FsDiagBlock* d_blocks, int64_t n_blocks, void* stream) {
    if (n_blocks < 0) return FS_ERR_INVALID_ARG;
    if (n_blocks == 0) return FS_OK;
    if (d_blocks == nullptr) return FS_ERR_INVALID_ARG;
    // the host cannot see the blocks: each kernel passes over the other's
    return diag_mul(d_x, d_diag, d_out, fsb::DeviceTable<FsDiagBlock>{d_blocks}, n_blocks, true,
                    false, stream);
}

extern "C" int fs_diag_mul_list(const double* d_x, const double* d_diag, double* d_out,
                                const FsDiagBlock* h_blocks, int64_t n_blocks, void* stream) {
    const int st = list_status(h_blocks, n_blocks);
    if (st != FS_OK || n_blocks == 0) return st;
    int64_t thin = 0;
    for (int64_t i = 0; i < n_blocks; ++i) thin += fsb::diag_thin(h_blocks[i]);
    return diag_mul(d_x, d_diag, d_out,
                    fsb::inline_table<FsDiagBlock, FS_LIST_MAX>(h_blocks, n_blocks), n_blocks,
                    thin > 0, thin == n_blocks, stream);
}
