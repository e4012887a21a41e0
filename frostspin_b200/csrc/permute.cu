// Abelian (U(1) / Z2) block-sparse permute as a batch of strided copies.
//
// Reference behaviour: frostspin/symmetric_tensor/abelian_symmetric_tensor.py
// :103-250 (_numba_abelian_transpose) scatters every entry of every old block to
// its new (block, row, col) with per-element divmod arithmetic.  Here the host
// plan splits the tensor into elementary blocks (one irrep segment per leg), in
// which both the source and destination offsets are affine in the leg indices.
// Legs are ordered by output stride, so the last leg is the output-innermost
// one; positions are decoded with Granlund-Montgomery division by the leg
// sizes (host-computed constants).  Absent source blocks produce zeros, as the
// reference's zero-initialised output blocks do.
#include "common.cuh"

namespace fsb {

constexpr int kPermThreads = 256;
// 8 loads of 8 bytes in flight per thread, 4 CTAs per SM: 64 KB per SM.  455 M
// coefficients in rows of ~40: 1253 us = 5.8 TB/s (1446 us with 4 loads, 1370
// us with 8 loads and 3 CTAs, 1470 us with 16 loads and 2 CTAs).
constexpr int kPermUnroll = 8;
// Tasks of few entries, whose other loads would all be masked off: rank-6 tensors
// of 0.14 and 0.75 M coefficients in small blocks 40.0 and 40.3 us (44.0 and 46.1
// us with 8 loads, 38.0 and 40.1 us when every task had 4).
constexpr int kPermUnrollShort = 2;
constexpr int kPermMaxRows = 1024;   // rows per task (shared-memory row table)

// One task = a range of rows of one elementary block, a row being one run along
// the output-innermost leg (length L).  Phase 1 decodes the outer multi-index
// of every row of the task once (Granlund-Montgomery division by the leg sizes)
// into a shared-memory table of source/destination row offsets, checking both
// ends of each row against the buffers.  Phase 2 walks the task's entries flat:
// entry idx -> (row, i) by one division by L, offsets from the table plus i
// times the innermost strides.  Consecutive threads write consecutive outputs
// (coalesced stores) and read consecutive inputs whenever the source keeps the
// same innermost leg; each thread keeps kPermUnroll loads in flight.
//
// kMulti: the EBs of several independent permutes in one launch; EB e reads
// and writes the buffer pair bufs[e.pad] (the permutes of many CTMRG runs
// advanced in lock step share one launch).
//
// perm_walk: phase 2 with U loads in flight.
template <int U>
__device__ __forceinline__ void perm_walk(const double* __restrict__ in, double* __restrict__ out,
                                          const int64_t* row_src, const int64_t* row_dst,
                                          uint32_t total, uint32_t L, uint32_t mL, uint32_t sL,
                                          int64_t osL, int64_t nsL, bool zero_fill) {
    for (uint32_t i0 = threadIdx.x; i0 < total; i0 += kPermThreads * U) {
        double v[U];
        int64_t dst[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t idx = i0 + u * kPermThreads;
            dst[u] = -1;
            v[u] = 0.0;
            if (idx < total) {
                const uint32_t row = fast_div(idx, mL, sL);
                const uint32_t i = idx - row * L;
                const int64_t rd = row_dst[row];
                if (rd >= 0) {
                    dst[u] = rd + static_cast<int64_t>(i) * nsL;
                    if (!zero_fill) v[u] = __ldg(in + row_src[row] + static_cast<int64_t>(i) * osL);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (dst[u] >= 0) out[dst[u]] = v[u];
        }
    }
}

template <bool kMulti>
__global__ void __launch_bounds__(kPermThreads, 4)
    k_perm_gather_t(const double* __restrict__ in0, int64_t in_len0, double* __restrict__ out0,
                    int64_t out_len0, const FsPermBuffers* __restrict__ bufs, int64_t n_bufs,
                    const FsPermEB* __restrict__ ebs, int64_t n_ebs,
                    const FsPermTask* __restrict__ tasks, int64_t n_tasks, int32_t* flag) {
    __shared__ FsPermEB e;
    __shared__ int64_t row_src[kPermMaxRows];
    __shared__ int64_t row_dst[kPermMaxRows];
    static_assert(sizeof(FsPermEB) % 8 == 0, "descriptor must be 8-byte granular");
    constexpr int kWords = sizeof(FsPermEB) / 8;
    for (int64_t t = blockIdx.x; t < n_tasks; t += gridDim.x) {
        const FsPermTask task = tasks[t];
        __syncthreads();  // previous task done with the shared tables
        if (task.eb < 0 || task.eb >= n_ebs || task.count > kPermMaxRows) {
            if (threadIdx.x == 0) raise_flag(flag, FS_ERR_BOUNDS);
            continue;
        }
        if (threadIdx.x < kWords) {
            reinterpret_cast<int64_t*>(&e)[threadIdx.x] =
                reinterpret_cast<const int64_t*>(ebs + task.eb)[threadIdx.x];
        }
        __syncthreads();
        const int nd = e.ndim;
        if (nd < 1 || nd > FS_PERM_MAXR) {
            if (threadIdx.x == 0) raise_flag(flag, FS_ERR_UNSUPPORTED);
            continue;
        }
        const double* in = in0;
        double* out = out0;
        int64_t in_len = in_len0, out_len = out_len0;
        if (kMulti) {
            if (e.pad < 0 || e.pad >= n_bufs) {
                if (threadIdx.x == 0) raise_flag(flag, FS_ERR_BOUNDS);
                continue;
            }
            const FsPermBuffers b = bufs[e.pad];
            in = b.in;
            out = b.out;
            in_len = b.in_len;
            out_len = b.out_len;
        }
        const uint32_t L = e.dims[nd - 1];
        const int64_t osL = e.ostride[nd - 1];
        const int64_t nsL = e.nstride[nd - 1];
        const bool zero_fill = e.obase < 0;
        const int nrows = static_cast<int>(task.count);
        for (int j = threadIdx.x; j < nrows; j += kPermThreads) {
            uint32_t q = task.start + static_cast<uint32_t>(j);
            int64_t so = e.obase, dof = e.nbase;
            for (int k = nd - 2; k >= 0; --k) {
                const uint32_t qq = fast_div(q, e.divm[k], e.divs[k]);
                const uint32_t i = q - qq * e.dims[k];
                q = qq;
                so += static_cast<int64_t>(i) * e.ostride[k];
                dof += static_cast<int64_t>(i) * e.nstride[k];
            }
            const int64_t dlast = dof + static_cast<int64_t>(L - 1) * nsL;
            const int64_t slast = so + static_cast<int64_t>(L - 1) * osL;
            bool ok = dof >= 0 && dlast < out_len;
            if (!zero_fill) ok = ok && so >= 0 && slast < in_len;
            if (!ok) {
                raise_flag(flag, FS_ERR_BOUNDS);
                dof = -1;
            }
            row_src[j] = so;
            row_dst[j] = dof;
        }
        __syncthreads();
        const uint32_t total = static_cast<uint32_t>(nrows) * L;
        const uint32_t mL = e.divm[nd - 1], sL = e.divs[nd - 1];
        if (total <= kPermUnrollShort * kPermThreads)
            perm_walk<kPermUnrollShort>(in, out, row_src, row_dst, total, L, mL, sL, osL, nsL,
                                        zero_fill);
        else
            perm_walk<kPermUnroll>(in, out, row_src, row_dst, total, L, mL, sL, osL, nsL, zero_fill);
    }
}

// ------------------------------------------------------- transposed EBs
// EBs whose unit-stride input leg (tile_leg) is not the output-innermost one:
// walked by rows they read 8 bytes of every 32-byte sector they touch.  Here a
// warp moves tiles of 32 entries of tile_leg by 32 of the last leg: every load
// of a tile is a run along tile_leg, every store a run along the last leg, the
// turn goes through shared memory.  Warps are independent (no CTA barrier) and
// have the loads of tile t + 1 in flight to registers while tile t is stored:
// 16 warps of 8 KB per SM, with a pointer step instead of index arithmetic per
// run.  Bound by HBM (16 bytes per coefficient).  Edge tensor (601 | 15, 15,
// 601), last leg moved first, 10.1 M coefficients: 65 us by rows, 36 us here; a
// 3200 x 3200 transpose 30 us = 5.5 TB/s, as a device copy.  The same with
// 8-byte cp.async into a double-buffered tile took 48 us, with 64 x 64 CTA
// tiles 42 us.
constexpr int kTileEdge = 32;
constexpr int kTileWarps = 4;
constexpr int kTileCtas = 4;                    // per SM: 128 registers, 34 KB of tiles each
constexpr int kTileLd = kTileEdge + 1;          // column reads touch distinct banks
constexpr int kTileDoubles = kTileEdge * kTileLd;
constexpr size_t kTileSmem = sizeof(double) * kTileDoubles * kTileWarps;
constexpr int kTileTaskMax = 32;                // tiles of a task: one lane decodes each

__device__ __forceinline__ void tile_fetch(double (&v)[kTileEdge], const double* __restrict__ in,
                                           int64_t so, int wa, int wb, int64_t ob) {
    const int lane = threadIdx.x % 32;
    if (lane >= wa) wb = 0;
    const double* p = in + so + lane;
#pragma unroll
    for (int j = 0; j < kTileEdge; ++j) {
        if (j < wb) v[j] = __ldg(p);
        p += ob;
    }
}

template <bool kMulti>
__global__ void __launch_bounds__(kTileWarps * 32, kTileCtas)
    k_perm_tiles(const double* __restrict__ in0, int64_t in_len0, double* __restrict__ out0,
                 int64_t out_len0, const FsPermBuffers* __restrict__ bufs, int64_t n_bufs,
                 const FsPermEB* __restrict__ ebs, int64_t n_ebs,
                 const FsPermTask* __restrict__ tasks, int64_t n_tasks, int32_t* flag) {
    extern __shared__ __align__(16) double tile_smem[];
    const int lane = threadIdx.x % 32, wid = threadIdx.x / 32;
    double* buf = tile_smem + wid * kTileDoubles;
    for (int64_t t = static_cast<int64_t>(blockIdx.x) * kTileWarps + wid; t < n_tasks;
         t += static_cast<int64_t>(gridDim.x) * kTileWarps) {
        const FsPermTask task = tasks[t];
        if (task.eb < 0 || task.eb >= n_ebs || task.count > kTileTaskMax) {
            if (lane == 0) raise_flag(flag, FS_ERR_BOUNDS);
            continue;
        }
        const FsPermEB& e = ebs[task.eb];
        const int nd = e.ndim, a = e.tile_leg;
        if (nd < 2 || nd > FS_PERM_MAXR || a < 0 || a >= nd - 1 || e.obase < 0 ||
            e.ostride[a] != 1 || e.nstride[nd - 1] != 1) {
            if (lane == 0) raise_flag(flag, FS_ERR_UNSUPPORTED);
            continue;
        }
        const double* in = in0;
        double* out = out0;
        int64_t in_len = in_len0, out_len = out_len0;
        if (kMulti) {
            if (e.pad < 0 || e.pad >= n_bufs) {
                if (lane == 0) raise_flag(flag, FS_ERR_BOUNDS);
                continue;
            }
            const FsPermBuffers b = bufs[e.pad];
            in = b.in;
            out = b.out;
            in_len = b.in_len;
            out_len = b.out_len;
        }
        const int64_t ob = e.ostride[nd - 1], na = e.nstride[a];
        const uint32_t L = e.dims[nd - 1], A = e.dims[a];
        // lane u decodes the task's tile u: outer legs, then tiles along the
        // last leg, then along tile_leg (fastest: neighbours read one run)
        int64_t so = 0, dof = 0;
        int wa = 0, wb = 0;
        if (lane < static_cast<int>(task.count)) {
            const uint32_t ta = (A + kTileEdge - 1) / kTileEdge;
            const uint32_t tb = (L + kTileEdge - 1) / kTileEdge;
            const uint32_t u = task.start + lane;
            uint32_t q = u / (ta * tb);
            const uint32_t r = u - q * (ta * tb), ib = r / ta, ia = r - ib * ta;
            const int64_t a0 = static_cast<int64_t>(ia) * kTileEdge;
            const int64_t b0 = static_cast<int64_t>(ib) * kTileEdge;
            so = e.obase + a0 + b0 * ob;
            dof = e.nbase + a0 * na + b0;
            for (int k = nd - 2; k >= 0; --k) {
                if (k == a) continue;
                const uint32_t qq = fast_div(q, e.divm[k], e.divs[k]);
                const uint32_t i = q - qq * e.dims[k];
                q = qq;
                so += static_cast<int64_t>(i) * e.ostride[k];
                dof += static_cast<int64_t>(i) * e.nstride[k];
            }
            wa = static_cast<int>(min(static_cast<int64_t>(kTileEdge), A - a0));
            wb = static_cast<int>(min(static_cast<int64_t>(kTileEdge), L - b0));
            // offsets are affine: the corners of the tile bound them
            const int64_t none = 0, za = (wa - 1) * na, zs = (wb - 1) * ob;
            if (q != 0 || dof + min(za, none) < 0 || dof + max(za, none) + wb > out_len ||
                so + min(zs, none) < 0 || so + max(zs, none) + wa > in_len) {
                raise_flag(flag, FS_ERR_BOUNDS);
                wa = wb = 0;
            }
        }
        const int n = static_cast<int>(task.count);
        double v[kTileEdge] = {};
        tile_fetch(v, in, __shfl_sync(~0u, so, 0), __shfl_sync(~0u, wa, 0),
                   __shfl_sync(~0u, wb, 0), ob);
        for (int u = 0; u < n; ++u) {
            __syncwarp();  // the previous tile has been read
#pragma unroll
            for (int j = 0; j < kTileEdge; ++j) buf[j * kTileLd + lane] = v[j];
            __syncwarp();
            if (u + 1 < n)
                tile_fetch(v, in, __shfl_sync(~0u, so, u + 1), __shfl_sync(~0u, wa, u + 1),
                           __shfl_sync(~0u, wb, u + 1), ob);
            const int ua = __shfl_sync(~0u, wa, u), ub = __shfl_sync(~0u, wb, u);
            double* q = out + __shfl_sync(~0u, dof, u) + lane;
            const double* s = buf + lane * kTileLd;
            if (lane < ub) {
#pragma unroll 8
                for (int i = 0; i < ua; ++i) {
                    *q = s[i];
                    q += na;
                }
            }
        }
        __syncwarp();
    }
}

template <bool kMulti>
int launch_tiles(const double* d_in, int64_t in_len, double* d_out, int64_t out_len,
                 const FsPermBuffers* d_bufs, int64_t n_bufs, const FsPermEB* d_ebs, int64_t n_ebs,
                 const FsPermTask* d_tasks, int64_t n_tasks, int32_t* d_flag, void* stream) {
    const int st = configure_smem(reinterpret_cast<const void*>(k_perm_tiles<kMulti>),
                                  static_cast<int>(kTileSmem));
    if (st != FS_OK) return st;
    const int64_t max_grid = static_cast<int64_t>(num_sms()) * kTileCtas;
    const int64_t want = (n_tasks + kTileWarps - 1) / kTileWarps;
    const int grid = static_cast<int>(want < max_grid ? want : max_grid);
    k_perm_tiles<kMulti><<<grid, kTileWarps * 32, kTileSmem, as_stream(stream)>>>(
        d_in, in_len, d_out, out_len, d_bufs, n_bufs, d_ebs, n_ebs, d_tasks, n_tasks, d_flag);
    return launch_status();
}

}  // namespace fsb

extern "C" int fs_abelian_permute(const double* d_in, int64_t in_len, double* d_out,
                                  int64_t out_len, const FsPermEB* d_ebs, int64_t n_ebs,
                                  const FsPermTask* d_tasks, int64_t n_tasks,
                                  int32_t* d_flag, void* stream) {
    if (n_tasks < 0 || n_ebs < 0 || in_len < 0 || out_len < 0) return FS_ERR_INVALID_ARG;
    if (n_tasks == 0) return FS_OK;
    if (d_out == nullptr || d_ebs == nullptr || d_tasks == nullptr) return FS_ERR_INVALID_ARG;
    if (d_in == nullptr && in_len > 0) return FS_ERR_INVALID_ARG;
    // one wave of resident CTAs (4 per SM at the kernel's register budget)
    const int64_t max_grid = static_cast<int64_t>(fsb::num_sms()) * 4;
    const int grid = static_cast<int>(n_tasks < max_grid ? n_tasks : max_grid);
    fsb::k_perm_gather_t<false><<<grid, fsb::kPermThreads, 0, fsb::as_stream(stream)>>>(
        d_in, in_len, d_out, out_len, nullptr, 0, d_ebs, n_ebs, d_tasks, n_tasks, d_flag);
    return fsb::launch_status();
}

extern "C" int fs_abelian_permute_multi(const FsPermBuffers* d_bufs, int64_t n_bufs,
                                        const FsPermEB* d_ebs, int64_t n_ebs,
                                        const FsPermTask* d_tasks, int64_t n_tasks,
                                        int32_t* d_flag, void* stream) {
    if (n_tasks < 0 || n_ebs < 0 || n_bufs < 0) return FS_ERR_INVALID_ARG;
    if (n_tasks == 0) return FS_OK;
    if (d_bufs == nullptr || d_ebs == nullptr || d_tasks == nullptr) return FS_ERR_INVALID_ARG;
    const int64_t max_grid = static_cast<int64_t>(fsb::num_sms()) * 4;
    const int grid = static_cast<int>(n_tasks < max_grid ? n_tasks : max_grid);
    fsb::k_perm_gather_t<true><<<grid, fsb::kPermThreads, 0, fsb::as_stream(stream)>>>(
        nullptr, 0, nullptr, 0, d_bufs, n_bufs, d_ebs, n_ebs, d_tasks, n_tasks, d_flag);
    return fsb::launch_status();
}

extern "C" int fs_permute_tiles(const double* d_in, int64_t in_len, double* d_out,
                                int64_t out_len, const FsPermEB* d_ebs, int64_t n_ebs,
                                const FsPermTask* d_tasks, int64_t n_tasks, int32_t* d_flag,
                                void* stream) {
    if (n_tasks < 0 || n_ebs < 0 || in_len < 0 || out_len < 0) return FS_ERR_INVALID_ARG;
    if (n_tasks == 0) return FS_OK;
    if (d_in == nullptr || d_out == nullptr || d_ebs == nullptr || d_tasks == nullptr)
        return FS_ERR_INVALID_ARG;
    return fsb::launch_tiles<false>(d_in, in_len, d_out, out_len, nullptr, 0, d_ebs, n_ebs,
                                    d_tasks, n_tasks, d_flag, stream);
}

extern "C" int fs_permute_tiles_multi(const FsPermBuffers* d_bufs, int64_t n_bufs,
                                      const FsPermEB* d_ebs, int64_t n_ebs,
                                      const FsPermTask* d_tasks, int64_t n_tasks,
                                      int32_t* d_flag, void* stream) {
    if (n_tasks < 0 || n_ebs < 0 || n_bufs < 0) return FS_ERR_INVALID_ARG;
    if (n_tasks == 0) return FS_OK;
    if (d_bufs == nullptr || d_ebs == nullptr || d_tasks == nullptr) return FS_ERR_INVALID_ARG;
    return fsb::launch_tiles<true>(nullptr, 0, nullptr, 0, d_bufs, n_bufs, d_ebs, n_ebs, d_tasks,
                                   n_tasks, d_flag, stream);
}
