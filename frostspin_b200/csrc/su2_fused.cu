// Fused SU(2) permute for the thin simple blocks: gather, recoupling product and
// scatter in one pass over the data.
//
// Reference behaviour: LieGroupSymmetricTensor._lie_permute_data ->
// fill_blocks_out -> permute_simple_block (frostspin/symmetric_tensor/
// lie_group_symmetric_tensor.py:96-265, :735-835): for every simple block, the
// sub-blocks of every input sector are gathered (strided view with the
// external legs permuted), multiplied by the block's recoupling isometry
// (new += U_sector @ old) and scattered into the output sectors.
//
// Here a simple block is a group with K input rows (input sectors x
// structural multiplicities), M = K output rows and E columns (the external
// multi-index, output leg order).  The CTA stages the group's recoupling
// matrix U (M x K <= 32 x 32) in shared memory and applies it column by column:
// the K inputs of a column are gathered from the input pieces, multiplied by U
// (broadcast reads) and the M results scattered to the output pieces.  Every
// row of a task is checked against its buffer (skipped and flagged,
// FS_ERR_BOUNDS); the host validates the tables before the call.
// Traffic: 8 bytes read and 8 written per coefficient (the three-launch form
// moves three times that).
//
// Work split: a task is a range of columns of one group.  A plane is one value of
// the external legs outside the two innermost output legs (L2 x L1 columns).
// Phase 1 writes, per piece and plane of the task, the element offset of the
// plane's first column into a shared table, after checking the extremes of the
// piece over the plane against the buffer; the group rows of a piece differ
// only by a constant (Su2Row.add).  Phase 2 streams the columns, 32 consecutive
// ones per warp and load, so the stores are coalesced and so are the loads
// wherever the source keeps the innermost output leg innermost.  A lane issues
// up to 32 loads before the first is used.  Groups with K <= 6 multiply column
// by column on the FP64 pipe with U in shared memory; wider ones turn the loaded
// columns in a shared buffer of the warp and multiply on the FP64 tensor cores,
// since a thread that carries one column of 24 rows reads U from shared memory
// for every second product.  Table entries are 32 bits, relative to the piece's
// base; a group whose pieces reach further runs column by column with whole
// offsets (su2_stream_wide).  The next task and its group are fetched while the
// current task streams.
//
// Bound by latency: about 9 us from a task's first load to its last store, with
// four tasks at a time per SM, against an HBM floor of 16 bytes per coefficient.
// Enlarged corner (22, 22 | 22, 22, 96, 96), 14.1 M coefficients in 1147 groups
// with L1 = 3 to 15 and K = 1 to 25: 249 us when every row of the innermost leg
// was decoded (48 per task, 400 columns for 256 threads), 140 us with longer
// tasks but every product on the FP64 pipe, 116 us with tensor cores and planes,
// 93 us now with 32-bit offsets, the early fetch and one task per resident CTA.
#include "common.cuh"

namespace fsb {

constexpr int kSu2Threads = 128;
constexpr int kSu2Warps = kSu2Threads / 32;
constexpr int kSu2Ctas = 4;         // per SM: 128 registers, 52 KB of shared tables
constexpr int kSu2MaxRows = 32;     // M, K of a fused group
constexpr int kSu2MaxPieces = 16;   // input and output pieces of a fused group
constexpr int kSu2Table = FS_SU2_TASK_TABLE;    // (piece, plane) entries of one task
constexpr int kSu2LdU = kSu2MaxRows + 4;        // 4 mod 16: fragment reads touch distinct banks
constexpr int kSu2Buf = kSu2Warps * 24 * (32 + 4);  // KB rows of 32 S + 4 doubles a warp
constexpr uint32_t kSu2None = 0xffffffffu;      // table entry: absent, skipped or past the task

// One group row: element base + table[tab + plane] + e2 ext2 + e1 ext1 of its
// buffer; base < 0: absent (input: zeros, output: not written).
struct Su2Row {
    int64_t base;
    uint32_t tab, ext2, ext1, pad;
};

struct Su2Smem {
    double buf[kSu2Buf];               // columns of the tensor-core form
    double u[kSu2MaxRows * kSu2LdU];   // zero padded
    Su2Row in[kSu2MaxRows], out[kSu2MaxRows];
    FsSu2Piece pc[2 * kSu2MaxPieces];
    FsSu2Group g;
    uint32_t table[kSu2Table + 2 * kSu2MaxPieces];   // [piece][plane], then one None
};

extern __shared__ __align__(16) uint8_t su2_raw[];
__device__ __forceinline__ Su2Smem& su2_smem() { return *reinterpret_cast<Su2Smem*>(su2_raw); }

// The columns of one pass of a warp: S runs of 32, lane l holding column l of
// each.
template <int S>
struct Su2Columns {
    uint32_t plane[S], e1[S], e2[S];

    __device__ __forceinline__ void decode(const FsSu2Group& g, int nd, uint32_t p0, uint32_t npl,
                                           int64_t c0, int64_t c_end) {
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const int64_t c = c0 + 32 * s + threadIdx.x % 32;
            uint32_t q = static_cast<uint32_t>(c);
            e1[s] = e2[s] = 0;
            if (nd > 0) {
                const uint32_t qq = fast_div(q, g.divm[nd - 1], g.divs[nd - 1]);
                e1[s] = q - qq * g.dims[nd - 1];
                q = qq;
            }
            if (nd > 1) {
                const uint32_t qq = fast_div(q, g.divm[nd - 2], g.divs[nd - 2]);
                e2[s] = q - qq * g.dims[nd - 2];
                q = qq;
            }
            plane[s] = c < c_end ? q - p0 : npl;
        }
    }

};

// x = the elements of group row w in the pass's columns
template <int S>
__device__ __forceinline__ void su2_load(double (&x)[S], const Su2Smem& sm, const Su2Row& w,
                                         const Su2Columns<S>& col, const double* __restrict__ src) {
#pragma unroll
    for (int s = 0; s < S; ++s) x[s] = 0.0;
    if (w.base < 0) return;
    const double* p = src + w.base;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const uint32_t t = sm.table[w.tab + col.plane[s]];
        if (t != kSu2None) x[s] = __ldg(p + (t + col.e2[s] * w.ext2 + col.e1[s] * w.ext1));
    }
}

template <int S>
__device__ __forceinline__ void su2_store(const double (&y)[S], const Su2Smem& sm, const Su2Row& w,
                                          const Su2Columns<S>& col, double* __restrict__ out) {
    if (w.base < 0) return;
    double* p = out + w.base;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const uint32_t t = sm.table[w.tab + col.plane[s]];
        if (t != kSu2None) p[t + col.e2[s] * w.ext2 + col.e1[s] * w.ext1] = y[s];
    }
}

// Phase 2 on the FP64 pipe, K <= KB.
template <int KB, int S>
__device__ __forceinline__ void su2_stream_fma(const Su2Smem& sm, const double* __restrict__ src,
                                               double* __restrict__ out, int M, int nd,
                                               uint32_t p0, uint32_t npl, int64_t c_begin,
                                               int64_t c_end) {
    for (int64_t c0 = c_begin + (threadIdx.x / 32) * (32 * S); c0 < c_end;
         c0 += kSu2Threads * S) {
        Su2Columns<S> col;
        col.decode(sm.g, nd, p0, npl, c0, c_end);
        double x[KB][S];
#pragma unroll
        for (int k = 0; k < KB; ++k) su2_load(x[k], sm, sm.in[k], col, src);  // past K: absent
#pragma unroll 1
        for (int m = 0; m < M; ++m) {
            double acc[S];
#pragma unroll
            for (int s = 0; s < S; ++s) acc[s] = 0.0;
#pragma unroll
            for (int k = 0; k < KB; ++k) {
                const double u = sm.u[m * kSu2LdU + k];
#pragma unroll
                for (int s = 0; s < S; ++s) acc[s] = fma(u, x[k][s], acc[s]);
            }
            su2_store(acc, sm, sm.out[m], col, out);
        }
    }
}

__device__ __forceinline__ void su2_dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// Phase 2 on the FP64 tensor cores, M, K <= KB (a multiple of 4): the warp parks
// its 32 S columns as KB rows in its buffer, multiplies two 8-column tiles at a
// time, writes the products over their columns and stores them.  W warps work
// (the widest groups need larger buffers than a quarter of the shared space).
// Loading the next columns during the products spilled and took twice the time.
template <int KB, int S, int W>
__device__ __forceinline__ void su2_stream_mma(Su2Smem& sm, const double* __restrict__ src,
                                               double* __restrict__ out, int M, int nd,
                                               uint32_t p0, uint32_t npl, int64_t c_begin,
                                               int64_t c_end) {
    constexpr int kLd = 32 * S + 4;      // 4 mod 16: fragment reads touch distinct banks
    constexpr int kMt = (KB + 7) / 8;
    static_assert(W <= kSu2Warps && W * KB * kLd <= kSu2Buf, "column buffers too small");
    const int lane = threadIdx.x % 32, wid = threadIdx.x / 32;
    if (wid >= W) return;
    const int fr = lane >> 2, fk = lane & 3;
    double* buf = sm.buf + wid * (KB * kLd);
    for (int64_t c0 = c_begin + wid * (32 * S); c0 < c_end; c0 += W * 32 * S) {
        Su2Columns<S> col;
        col.decode(sm.g, nd, p0, npl, c0, c_end);
        {
            double x[KB][S];
#pragma unroll
            for (int k = 0; k < KB; ++k) su2_load(x[k], sm, sm.in[k], col, src);  // past K: absent
            __syncwarp();   // the previous pass has been stored
#pragma unroll
            for (int k = 0; k < KB; ++k)
#pragma unroll
                for (int s = 0; s < S; ++s) buf[k * kLd + 32 * s + lane] = x[k][s];
            __syncwarp();
        }
#pragma unroll 1
        for (int nt = 0; nt < 4 * S; nt += 2) {
            double acc[kMt][2][2];
#pragma unroll
            for (int i = 0; i < kMt; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
            const double* pb = buf + fk * kLd + nt * 8 + fr;
            const double* pu = sm.u + fr * kSu2LdU + fk;
#pragma unroll
            for (int ks = 0; ks < KB / 4; ++ks) {
                const double b0 = pb[ks * 4 * kLd], b1 = pb[ks * 4 * kLd + 8];
#pragma unroll
                for (int i = 0; i < kMt; ++i) {
                    const double u = pu[i * 8 * kSu2LdU + ks * 4];
                    su2_dmma(acc[i][0], u, b0);
                    su2_dmma(acc[i][1], u, b1);
                }
            }
            __syncwarp();   // every lane has read these columns
#pragma unroll
            for (int i = 0; i < kMt; ++i) {
                if (i * 8 + fr < KB) {
                    double* d = buf + (i * 8 + fr) * kLd + nt * 8 + 2 * fk;
                    *reinterpret_cast<double2*>(d) = make_double2(acc[i][0][0], acc[i][0][1]);
                    *reinterpret_cast<double2*>(d + 8) = make_double2(acc[i][1][0], acc[i][1][1]);
                }
            }
        }
        __syncwarp();
#pragma unroll 2
        for (int m = 0; m < M; ++m) {
            double y[S];
#pragma unroll
            for (int s = 0; s < S; ++s) y[s] = buf[m * kLd + 32 * s + lane];
            su2_store(y, sm, sm.out[m], col, out);
        }
    }
}

// Phase 2 for pieces that reach 2^32 elements or more from their base (or have
// negative strides): whole offsets, one column and one output row at a time.
__device__ __noinline__ void su2_stream_wide(const double* __restrict__ src, int64_t src_len,
                                             double* __restrict__ out, int64_t out_len,
                                             int64_t c_begin, int64_t c_end, int32_t* flag) {
    const Su2Smem& sm = su2_smem();
    const FsSu2Group& g = sm.g;
    for (int64_t c = c_begin + threadIdx.x; c < c_end; c += kSu2Threads) {
        uint32_t e[FS_SU2_MAXD];
        uint32_t rem = static_cast<uint32_t>(c);
        for (int l = g.ndim - 1; l >= 0; --l) {
            const uint32_t q = fast_div(rem, g.divm[l], g.divs[l]);
            e[l] = rem - q * g.dims[l];
            rem = q;
        }
        // group row r of the pieces [first, last): its element, -1 if absent
        auto element = [&](int first, int last, int r, int64_t len) {
            for (int p = first; p < last; ++p) {
                const FsSu2Piece& pc = sm.pc[p];
                const int d = r - pc.row0;
                if (d < 0 || d >= pc.sr * pc.sc || pc.base < 0) continue;
                int64_t o = pc.base + (d / pc.sc) * pc.sr_stride + (d % pc.sc) * pc.sc_stride;
                for (int l = 0; l < g.ndim; ++l) o += static_cast<int64_t>(e[l]) * pc.ext[l];
                if (o >= 0 && o < len) return o;
                raise_flag(flag, FS_ERR_BOUNDS);
            }
            return static_cast<int64_t>(-1);
        };
        for (int m = 0; m < g.M; ++m) {
            const int64_t o = element(g.in_count, g.in_count + g.out_count, m, out_len);
            if (o < 0) continue;
            double acc = 0.0;
            for (int k = 0; k < g.K; ++k) {
                const int64_t i = element(0, g.in_count, k, src_len);
                acc = fma(sm.u[m * kSu2LdU + k], i >= 0 ? __ldg(src + i) : 0.0, acc);
            }
            out[o] = acc;
        }
    }
}

__global__ void __launch_bounds__(kSu2Threads, kSu2Ctas)
    k_su2_fused(const double* __restrict__ src, int64_t src_len, double* __restrict__ out,
                int64_t out_len, const FsSu2Group* __restrict__ groups, int64_t n_groups,
                const FsSu2Piece* __restrict__ pieces, int64_t n_pieces,
                const double* __restrict__ U, int64_t u_len, const FsPermTask* __restrict__ tasks,
                int64_t n_tasks, int32_t* flag) {
    Su2Smem& sm = su2_smem();
    const int tid = threadIdx.x;
    static_assert(sizeof(FsSu2Group) % 8 == 0 && sizeof(FsSu2Piece) % 8 == 0, "8-byte words");
    constexpr int kGroupWords = sizeof(FsSu2Group) / 8, kPieceWords = sizeof(FsSu2Piece) / 8;
    // the next task and its group are fetched while the current one streams
    FsPermTask next = {-1, 0, 0, 0};
    int64_t next_word = 0;
    auto fetch = [&](int64_t t) {
        next.eb = -1;
        if (t < n_tasks) next = tasks[t];
    };
    auto fetch_group = [&]() {
        if (next.eb >= 0 && next.eb < n_groups && tid < kGroupWords)
            next_word = reinterpret_cast<const int64_t*>(groups + next.eb)[tid];
    };
    fetch(blockIdx.x);
    fetch_group();
    for (int64_t t = blockIdx.x; t < n_tasks; t += gridDim.x) {
        const FsPermTask tk = next;
        __syncthreads();  // the previous task is done with the shared tables
        if (tid < kGroupWords) reinterpret_cast<int64_t*>(&sm.g)[tid] = next_word;
        fetch(t + gridDim.x);
        if (tk.eb < 0 || tk.eb >= n_groups) {
            if (tid == 0) raise_flag(flag, FS_ERR_BOUNDS);
            fetch_group();
            continue;
        }
        __syncthreads();
        const FsSu2Group& g = sm.g;
        const int nd = g.ndim, M = g.M, K = g.K;
        const bool ok = M >= 0 && M <= kSu2MaxRows && K >= 0 && K <= kSu2MaxRows &&
                        nd >= 0 && nd <= FS_SU2_MAXD && g.in_count >= 0 &&
                        g.in_count <= kSu2MaxPieces && g.out_count >= 0 &&
                        g.out_count <= kSu2MaxPieces && g.in_first >= 0 &&
                        g.in_first + g.in_count <= n_pieces && g.out_first >= 0 &&
                        g.out_first + g.out_count <= n_pieces && g.u_off >= 0 &&
                        g.u_off + static_cast<int64_t>(M) * K <= u_len;
        if (!ok) {
            if (tid == 0) raise_flag(flag, FS_ERR_BOUNDS);
            fetch_group();
            continue;
        }
        const uint32_t L1 = nd > 0 ? g.dims[nd - 1] : 1u, L2 = nd > 1 ? g.dims[nd - 2] : 1u;
        const int64_t c_begin = tk.start;
        const int64_t c_end = min(static_cast<int64_t>(tk.start) + tk.count, g.ncols);
        if (c_end <= c_begin || L1 == 0 || L2 == 0) {
            fetch_group();
            continue;
        }
        // the task's planes
        auto plane_of = [&](int64_t c) {
            uint32_t q = static_cast<uint32_t>(c);
            if (nd > 0) q = fast_div(q, g.divm[nd - 1], g.divs[nd - 1]);
            if (nd > 1) q = fast_div(q, g.divm[nd - 2], g.divs[nd - 2]);
            return q;
        };
        const uint32_t p0 = plane_of(c_begin);
        const int64_t npl64 = static_cast<int64_t>(plane_of(c_end - 1)) - p0 + 1;
        const int npc = g.in_count + g.out_count;
        if (npl64 * npc > kSu2Table) {
            if (tid == 0) raise_flag(flag, FS_ERR_BOUNDS);
            fetch_group();
            continue;
        }
        const uint32_t npl = static_cast<uint32_t>(npl64);
        for (int i = tid; i < kSu2MaxRows * kSu2MaxRows; i += kSu2Threads) {
            const int m = i / kSu2MaxRows, k = i % kSu2MaxRows;
            sm.u[m * kSu2LdU + k] = m < M && k < K ? __ldg(U + g.u_off + m * K + k) : 0.0;
        }
        for (int i = tid; i < npc * kPieceWords; i += kSu2Threads) {
            const int p = i / kPieceWords, w = i - p * kPieceWords;
            const int64_t at = p < g.in_count ? g.in_first + p : g.out_first + (p - g.in_count);
            reinterpret_cast<int64_t*>(&sm.pc[p])[w] =
                reinterpret_cast<const int64_t*>(pieces + at)[w];
        }
        __syncthreads();
        fetch_group();
        // the piece of every group row
        if (tid < 2 * kSu2MaxRows) {
            const bool is_in = tid < kSu2MaxRows;
            const int k = is_in ? tid : tid - kSu2MaxRows;
            Su2Row row = {-1, 0, 0, 0, 0};
            const int first = is_in ? 0 : g.in_count, last = is_in ? g.in_count : npc;
            for (int p = first; p < last; ++p) {
                const FsSu2Piece& pc = sm.pc[p];
                const int d = k - pc.row0, rows = pc.sr * pc.sc;
                if (k == 0 && (pc.row0 < 0 || pc.row0 + rows > (is_in ? K : M)))
                    raise_flag(flag, FS_ERR_BOUNDS);
                if (d < 0 || d >= rows || k >= (is_in ? K : M) || pc.base < 0) continue;
                row.base = pc.base + (d / pc.sc) * pc.sr_stride + (d % pc.sc) * pc.sc_stride;
                row.tab = static_cast<uint32_t>(p) * (npl + 1);
                row.ext1 = nd > 0 ? static_cast<uint32_t>(pc.ext[nd - 1]) : 0;
                row.ext2 = nd > 1 ? static_cast<uint32_t>(pc.ext[nd - 2]) : 0;
            }
            (is_in ? sm.in : sm.out)[k] = row;
        }
        // the first column of every plane relative to the piece's base
        bool wide = false;
        for (int j = tid; j < npc * (static_cast<int>(npl) + 1); j += kSu2Threads) {
            const uint32_t p = static_cast<uint32_t>(j) / (npl + 1), pl = j - p * (npl + 1);
            const FsSu2Piece& pc = sm.pc[p];
            const bool is_in = static_cast<int>(p) < g.in_count;
            uint32_t entry = kSu2None;
            if (pl < npl && pc.base >= 0) {
                uint32_t rem = p0 + pl;
                int64_t off = 0;
                for (int l = nd - 3; l >= 0; --l) {
                    const uint32_t q = fast_div(rem, g.divm[l], g.divs[l]);
                    off += static_cast<int64_t>(rem - q * g.dims[l]) * pc.ext[l];
                    rem = q;
                }
                // offsets are affine in (structural row, column): extremes
                const int64_t none = 0;
                const int64_t za = (pc.sr - 1) * pc.sr_stride, zb = (pc.sc - 1) * pc.sc_stride;
                const int64_t z1 = nd > 0 ? static_cast<int64_t>(L1 - 1) * pc.ext[nd - 1] : 0;
                const int64_t z2 = nd > 1 ? static_cast<int64_t>(L2 - 1) * pc.ext[nd - 2] : 0;
                const int64_t lo = min(z1, none) + min(z2, none);
                const int64_t hi = off + max(z1, none) + max(z2, none);
                if (pc.base + off + lo + min(za, none) + min(zb, none) < 0 ||
                    pc.base + hi + max(za, none) + max(zb, none) >= (is_in ? src_len : out_len)) {
                    raise_flag(flag, FS_ERR_BOUNDS);
                } else if (lo < 0 || off < 0 || hi >= static_cast<int64_t>(kSu2None)) {
                    wide = true;
                } else {
                    entry = static_cast<uint32_t>(off);
                }
            }
            sm.table[j] = entry;
        }
        if (__syncthreads_or(wide)) {
            su2_stream_wide(src, src_len, out, out_len, c_begin, c_end, flag);
            continue;
        }
#define FSB_FMA(kb, s) su2_stream_fma<kb, s>(sm, src, out, M, nd, p0, npl, c_begin, c_end)
#define FSB_MMA(kb, s, w) su2_stream_mma<kb, s, w>(sm, src, out, M, nd, p0, npl, c_begin, c_end)
        const int w = K > M ? K : M;
        if (w <= 1)
            FSB_FMA(1, 8);
        else if (w <= 2)
            FSB_FMA(2, 6);
        else if (w <= 3)
            FSB_FMA(3, 5);
        else if (w <= 4)
            FSB_FMA(4, 4);
        else if (w <= 6)
            FSB_FMA(6, 3);
        else if (w <= 8)
            FSB_MMA(8, 3, 4);
        else if (w <= 12)
            FSB_MMA(12, 2, 4);
        else if (w <= 16)
            FSB_MMA(16, 1, 4);
        else if (w <= 20)
            FSB_MMA(20, 1, 4);
        else if (w <= 24)
            FSB_MMA(24, 1, 4);
        else
            FSB_MMA(32, 1, 3);
#undef FSB_FMA
#undef FSB_MMA
    }
}

}  // namespace fsb

extern "C" int fs_su2_fused_limits(int32_t* max_rows, int32_t* max_pieces, int32_t* threads) {
    if (max_rows == nullptr || max_pieces == nullptr || threads == nullptr)
        return FS_ERR_INVALID_ARG;
    *max_rows = fsb::kSu2MaxRows;
    *max_pieces = fsb::kSu2MaxPieces;
    *threads = fsb::kSu2Threads;
    return FS_OK;
}

extern "C" int fs_su2_permute_fused(const double* d_src, int64_t src_len, double* d_out,
                                    int64_t out_len, const FsSu2Group* d_groups,
                                    int64_t n_groups, const FsSu2Piece* d_pieces,
                                    int64_t n_pieces, const double* d_u, int64_t u_len,
                                    const FsPermTask* d_tasks, int64_t n_tasks, int32_t* d_flag,
                                    void* stream) {
    if (src_len < 0 || out_len < 0 || n_groups < 0 || n_pieces < 0 || u_len < 0 || n_tasks < 0)
        return FS_ERR_INVALID_ARG;
    if (n_tasks == 0) return FS_OK;
    if (d_out == nullptr || d_groups == nullptr || d_pieces == nullptr || d_tasks == nullptr ||
        (d_u == nullptr && u_len > 0) || (d_src == nullptr && src_len > 0))
        return FS_ERR_INVALID_ARG;
    constexpr int smem = static_cast<int>(sizeof(fsb::Su2Smem));
    const int st = fsb::configure_smem(reinterpret_cast<const void*>(fsb::k_su2_fused), smem);
    if (st != FS_OK) return st;
    const int64_t max_grid = static_cast<int64_t>(fsb::num_sms()) * fsb::kSu2Ctas;
    const int grid = static_cast<int>(n_tasks < max_grid ? n_tasks : max_grid);
    fsb::k_su2_fused<<<grid, fsb::kSu2Threads, smem, fsb::as_stream(stream)>>>(
        d_src, src_len, d_out, out_len, d_groups, n_groups, d_pieces, n_pieces, d_u, u_len,
        d_tasks, n_tasks, d_flag);
    return fsb::launch_status();
}
