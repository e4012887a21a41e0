// Grouped FP64 GEMM over irrep sectors: the plain double-precision path, on the
// FP64 tensor cores (DMMA, mma.sync m8n8k4 f64 -- Blackwell has no tcgen05 kind
// for f64, so this is the FP64 tensor path of sm_100a).
//
// Reference behaviour: SymmetricTensor.__matmul__ (frostspin/symmetric_tensor/
// symmetric_tensor.py:453-489) calls numpy's dgemm once per shared irrep block.
// Here every sector product of one contraction is a problem in one launch, and
// CTAs stride over the output tiles of all problems (a static persistent
// schedule), so sectors of very uneven sizes share the machine.  Problems travel
// with the kernel's parameters, and the CTAs enumerate the tiles themselves
// (TileList); long lists and the longest launches read problems and tiles from
// device memory (TileTable).
//
// 64x64 output tile per CTA, 4 warps of 32x32 (4x4 m8n8 fragments), k staged
// 16 deep through a 3-stage cp.async pipeline, 3 CTAs per SM.  Sector blocks
// start at any element offset, so copies are 8-byte cp.async with zero fill at
// the edges.  Shared layouts follow the global layout of each operand (row- or
// column-major, per problem; the tile body is instantiated for the four
// combinations) with padding chosen so that every fragment load of a half warp
// touches 32 distinct banks.
#include "common.cuh"

namespace fsb {

constexpr int kTM = 64;
constexpr int kTN = 64;
constexpr int kTK = 16;
constexpr int kStages = 3;
constexpr int kGemmThreads = 128;
constexpr int kLdK = kTK + 4;   // stride of a [row][k] tile (20 doubles, 4 mod 16)
constexpr int kLdR = kTM + 4;   // stride of a [k][row] tile (68 doubles, 4 mod 16)
constexpr int kOpTile = kTM * kLdK;  // >= kTK * kLdR
static_assert(kTM == kTN, "square tiles: one stage size for A and B");
static_assert(kOpTile >= kTK * kLdR, "stage too small for the k-major layout");
constexpr int kStageDoubles = 2 * kOpTile;
constexpr size_t kGemmSmem = sizeof(double) * kStageDoubles * kStages;

__device__ __forceinline__ void cp_async8(double* dst, const double* src, bool valid) {
    const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
    const int n = valid ? 8 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(n));
}

__device__ __forceinline__ void cp_async_commit() {
    asm volatile("cp.async.commit_group;\n" ::);
}

template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// One k slice of op(A) (rows m0.., k0..) and op(B) (k0.., cols n0..) into a stage.
// A stage holds A in [m][k] (TA == 0) or [k][m] (TA == 1) and B in [k][n]
// (TB == 0) or [n][k] (TB == 1): always the global contiguous direction
// innermost, so the copies are coalesced.
template <bool TA, bool TB>
__device__ __forceinline__ void load_stage(const FsGemmProblem& p, int m0, int n0, int k0,
                                           double* stage) {
    double* sa = stage;
    double* sb = stage + kOpTile;
#pragma unroll
    for (int u = 0; u < (kTM * kTK) / kGemmThreads; ++u) {
        const int e = threadIdx.x + u * kGemmThreads;
        const int k = TA ? e / kTM : e % kTK;
        const int m = TA ? e % kTM : e / kTK;
        const bool ok = (m0 + m < p.M) && (k0 + k < p.K);
        const int64_t off = TA ? static_cast<int64_t>(k0 + k) * p.lda + (m0 + m)
                               : static_cast<int64_t>(m0 + m) * p.lda + (k0 + k);
        cp_async8(sa + (TA ? k * kLdR + m : m * kLdK + k), ok ? p.A + off : p.A, ok);
    }
#pragma unroll
    for (int u = 0; u < (kTN * kTK) / kGemmThreads; ++u) {
        const int e = threadIdx.x + u * kGemmThreads;
        const int k = TB ? e % kTK : e / kTN;
        const int n = TB ? e / kTK : e % kTN;
        const bool ok = (n0 + n < p.N) && (k0 + k < p.K);
        const int64_t off = TB ? static_cast<int64_t>(n0 + n) * p.ldb + (k0 + k)
                               : static_cast<int64_t>(k0 + k) * p.ldb + (n0 + n);
        cp_async8(sb + (TB ? n * kLdK + k : k * kLdR + n), ok ? p.B + off : p.B, ok);
    }
}

// The DMMAs of one staged k slice for one warp's 32x32 block: k steps at or
// beyond k_left, fragment rows at or beyond rows_left and fragment columns at
// or beyond cols_left (all warp-uniform) are skipped.
template <bool TA, bool TB>
__device__ __forceinline__ void mma_slice(double (&acc)[4][4][2], const double* sa,
                                          const double* sb, int k_left, int rows_left,
                                          int cols_left) {
    constexpr int a_step_i = TA ? 8 : 8 * kLdK;   // next fragment row block
    constexpr int a_step_k = TA ? 4 * kLdR : 4;   // next k-step
    constexpr int b_step_j = TB ? 8 * kLdK : 8;
    constexpr int b_step_k = TB ? 4 : 4 * kLdR;
#pragma unroll
    for (int ks = 0; ks < kTK / 4; ++ks) {
        if (ks * 4 >= k_left) break;
        double a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = sa[ks * a_step_k + i * a_step_i];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = sb[ks * b_step_k + j * b_step_j];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (i * 8 >= rows_left) break;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (j * 8 >= cols_left) break;
                dmma(acc[i][j], a[i], b[j]);
            }
        }
    }
}

// One 64x64 output tile: the cp.async pipeline over k and the DMMA fragments.
template <bool TA, bool TB>
__device__ __forceinline__ void dgemm_tile(const FsGemmProblem& p, int m0, int n0,
                                           double* smem) {
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int wm = (warp & 1) * 32;
    const int wn = (warp >> 1) * 32;
    const int fr = lane >> 2;  // fragment row (A, C) / column (B)
    const int fk = lane & 3;   // fragment k (A, B) / column pair (C)

    double acc[4][4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

    // per-thread fragment offsets inside a stage (k = 0)
    const int a_off = TA ? fk * kLdR + wm + fr : (wm + fr) * kLdK + fk;
    const int b_off = TB ? (wn + fr) * kLdK + fk : fk * kLdR + wn + fr;

    const int nk = (p.K + kTK - 1) / kTK;
    __syncthreads();  // every warp is done with the previous tile's stages
#pragma unroll
    for (int s = 0; s < kStages - 1; ++s) {
        if (s < nk) load_stage<TA, TB>(p, m0, n0, s * kTK, smem + s * kStageDoubles);
        cp_async_commit();
    }
    for (int kt = 0; kt < nk; ++kt) {
        cp_async_wait<kStages - 2>();
        __syncthreads();
        {
            const int nxt = kt + kStages - 1;
            if (nxt < nk)
                load_stage<TA, TB>(p, m0, n0, nxt * kTK, smem + (nxt % kStages) * kStageDoubles);
            cp_async_commit();
        }
        const double* sa = smem + (kt % kStages) * kStageDoubles + a_off;
        const double* sb = smem + (kt % kStages) * kStageDoubles + kOpTile + b_off;
        // the full padded slice: at 168 registers this kernel has no room for
        // the edge tests (the streaming kernel skips padded fragments)
        mma_slice<TA, TB>(acc, sa, sb, kTK, kTM, kTN);
    }
    cp_async_wait<0>();

#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int gi = m0 + wm + i * 8 + fr;
        if (gi >= p.M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int gj = n0 + wn + j * 8 + fk * 2 + h;
                if (gj >= p.N) continue;
                double* c = p.C + static_cast<int64_t>(gi) * p.ldc + gj;
                const double v = p.alpha * acc[i][j][h];
                *c = (p.beta == 0.0) ? v : fma(p.beta, *c, v);
            }
        }
    }
}

// Where a launch finds its problems and output tiles (TM x TN): a device table of
// both, or problems passed with the kernel's parameters, whose tiles are
// enumerated here -- problem by problem, column-major when a problem has more
// tile columns than rows (its few row tiles then share each B column block in
// L2).  `find` takes non-decreasing t for one cursor; false: an invalid entry.
struct TileTable {
    const FsGemmProblem* problems;
    int64_t n_problems;
    const FsGemmTile* tiles;
    int64_t n_tiles;

    struct Cursor {};
    template <int TM, int TN>
    __device__ __forceinline__ bool find(Cursor&, int64_t t, FsGemmProblem& p, int& m0,
                                         int& n0) const {
        const FsGemmTile tile = tiles[t];
        if (tile.problem < 0 || tile.problem >= n_problems) return false;
        p = problems[tile.problem];
        m0 = tile.tm * TM;
        n0 = tile.tn * TN;
        return m0 < p.M && n0 < p.N;
    }
};

template <int N>
struct TileList {
    FsGemmProblem v[N];
    int64_t n_problems;
    int64_t n_tiles;

    struct Cursor {
        int problem = 0;
        int64_t first = 0;   // the problem's first tile
    };
    template <int TM, int TN>
    __host__ __device__ __forceinline__ static int64_t count(const FsGemmProblem& p) {
        return (static_cast<int64_t>(p.M) + TM - 1) / TM * ((static_cast<int64_t>(p.N) + TN - 1) / TN);
    }
    template <int TM, int TN>
    __device__ __forceinline__ bool find(Cursor& c, int64_t t, FsGemmProblem& p, int& m0,
                                         int& n0) const {
        int64_t n = count<TM, TN>(v[c.problem]);
        while (t >= c.first + n) {
            c.first += n;
            n = count<TM, TN>(v[++c.problem]);
        }
        p = v[c.problem];
        // keep the fields in registers: the compiler would read them from the
        // parameters again for every k slice
        asm volatile("" : "+l"(p.A), "+l"(p.B), "+l"(p.lda), "+l"(p.ldb), "+r"(p.M), "+r"(p.N), "+r"(p.K));
        // a problem has fewer than 2^31 tiles (host)
        const uint32_t k = static_cast<uint32_t>(t - c.first);
        const uint32_t nr = (static_cast<uint32_t>(p.M) + TM - 1) / TM;
        const uint32_t nc = (static_cast<uint32_t>(p.N) + TN - 1) / TN;
        const uint32_t q = k / (nc > nr ? nr : nc), r = k - q * (nc > nr ? nr : nc);
        m0 = static_cast<int>(nc > nr ? r : q) * TM;
        n0 = static_cast<int>(nc > nr ? q : r) * TN;
        return true;
    }
};

template <class Tiles>
__global__ void __launch_bounds__(kGemmThreads, 3)
    k_grouped_dgemm(const __grid_constant__ Tiles tiles) {
    extern __shared__ __align__(16) double smem[];
    typename Tiles::Cursor cursor;
    for (int64_t t = blockIdx.x; t < tiles.n_tiles; t += gridDim.x) {
        FsGemmProblem p;
        int m0, n0;
        if (!tiles.template find<kTM, kTN>(cursor, t, p, m0, n0)) continue;
        switch ((p.transA ? 2 : 0) | (p.transB ? 1 : 0)) {
            case 0: dgemm_tile<false, false>(p, m0, n0, smem); break;
            case 1: dgemm_tile<false, true>(p, m0, n0, smem); break;
            case 2: dgemm_tile<true, false>(p, m0, n0, smem); break;
            default: dgemm_tile<true, true>(p, m0, n0, smem); break;
        }
    }
}

// Streaming variant for launches whose problems share both transpose flags,
// used for short-K sector products (wide recouplings and projector
// applications with K of a few tens): one cp.async ring runs continuously
// across the CTA's tiles, so the first k slices of the next tile load while
// the current tile finishes and writes its outputs, and fragments or k steps
// wholly outside the problem (M, N, K padding of the 64x64x16 tiling) issue no
// DMMA.  Tiles of problems with K = 0 consume no stage (their output is
// beta * C).
template <class Tiles>
struct TileCursor {
    typename Tiles::Cursor at;
    int64_t t;
    FsGemmProblem p;
    int m0, n0, nk;
};

template <class Tiles>
__device__ __forceinline__ bool cursor_seek(TileCursor<Tiles>& c, int64_t t, const Tiles& tiles,
                                            bool need_k) {
    for (; t < tiles.n_tiles; t += gridDim.x) {
        if (!tiles.template find<kTM, kTN>(c.at, t, c.p, c.m0, c.n0)) continue;
        c.nk = (c.p.K + kTK - 1) / kTK;
        if (need_k && c.nk == 0) continue;
        c.t = t;
        return true;
    }
    c.t = tiles.n_tiles;
    return false;
}

template <bool TA, bool TB, class Tiles>
__global__ void __launch_bounds__(kGemmThreads, 3)
    k_grouped_dgemm_stream(const __grid_constant__ Tiles tiles) {
    extern __shared__ __align__(16) double smem[];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int wm = (warp & 1) * 32;
    const int wn = (warp >> 1) * 32;
    const int fr = lane >> 2;
    const int fk = lane & 3;
    const int a_off = TA ? fk * kLdR + wm + fr : (wm + fr) * kLdK + fk;
    const int b_off = TB ? (wn + fr) * kLdK + fk : fk * kLdR + wn + fr;

    // loader: the next (tile, k slice) to fetch; tiles without k slices skipped
    TileCursor<Tiles> ld;
    bool ld_ok = cursor_seek(ld, blockIdx.x, tiles, true);
    int ld_k = 0;
    int64_t issued = 0;
    auto issue = [&]() {
        if (ld_ok) {
            load_stage<TA, TB>(ld.p, ld.m0, ld.n0, ld_k * kTK,
                               smem + (issued % kStages) * kStageDoubles);
            ++issued;
            if (++ld_k == ld.nk) {
                ld_k = 0;
                ld_ok = cursor_seek(ld, ld.t + gridDim.x, tiles, true);
            }
        }
        cp_async_commit();
    };

    // consumer: every tile of this CTA in order (K = 0 tiles included)
    TileCursor<Tiles> cs;
    bool cs_ok = cursor_seek(cs, blockIdx.x, tiles, false);
    int cs_k = 0;
    int64_t consumed = 0;
    double acc[4][4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

#pragma unroll
    for (int s = 0; s < kStages - 1; ++s) issue();

    while (cs_ok) {
        if (cs_k < cs.nk) {
            // stage `consumed` is the consumed-th issued one: its group is
            // complete once at most kStages - 2 newer groups are pending
            cp_async_wait<kStages - 2>();
            __syncthreads();  // and every warp is done with the slot refilled next
            issue();
            const double* sa = smem + (consumed % kStages) * kStageDoubles + a_off;
            const double* sb = smem + (consumed % kStages) * kStageDoubles + kOpTile + b_off;
            mma_slice<TA, TB>(acc, sa, sb, cs.p.K - cs_k * kTK, cs.p.M - (cs.m0 + wm),
                              cs.p.N - (cs.n0 + wn));
            ++consumed;
            ++cs_k;
        }
        if (cs_k < cs.nk) continue;
        // tile done: write it while the next tile's first slices load
        const FsGemmProblem& p = cs.p;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int gi = cs.m0 + wm + i * 8 + fr;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int gj = cs.n0 + wn + j * 8 + fk * 2 + h;
                    if (gi < p.M && gj < p.N) {
                        double* c = p.C + static_cast<int64_t>(gi) * p.ldc + gj;
                        const double v = p.alpha * acc[i][j][h];
                        *c = (p.beta == 0.0) ? v : fma(p.beta, *c, v);
                    }
                    acc[i][j][h] = 0.0;
                }
            }
        }
        cs_k = 0;
        cs_ok = cursor_seek(cs, cs.t + gridDim.x, tiles, false);
    }
    cp_async_wait<0>();
}

}  // namespace fsb

extern "C" int fs_dgemm_tile_shape(int32_t* tile_m, int32_t* tile_n) {
    if (tile_m == nullptr || tile_n == nullptr) return FS_ERR_INVALID_ARG;
    *tile_m = fsb::kTM;
    *tile_n = fsb::kTN;
    return FS_OK;
}

namespace {

inline int persistent_grid(int64_t n_tiles, int ctas) {
    const int64_t max_grid = static_cast<int64_t>(fsb::num_sms()) * ctas;
    return static_cast<int>(n_tiles < max_grid ? n_tiles : max_grid);
}

template <class Tiles>
int launch_tiles(const Tiles& tiles, cudaStream_t s) {
    const int cfg = fsb::configure_smem(reinterpret_cast<const void*>(fsb::k_grouped_dgemm<Tiles>),
                                        static_cast<int>(fsb::kGemmSmem));
    if (cfg != FS_OK) return cfg;
    fsb::k_grouped_dgemm<<<persistent_grid(tiles.n_tiles, 3), fsb::kGemmThreads, fsb::kGemmSmem,
                           s>>>(tiles);
    return fsb::launch_status();
}

template <bool TA, bool TB, class Tiles>
int launch_stream_t(const Tiles& tiles, cudaStream_t s) {
    const int cfg = fsb::configure_smem(
        reinterpret_cast<const void*>(fsb::k_grouped_dgemm_stream<TA, TB, Tiles>),
        static_cast<int>(fsb::kGemmSmem));
    if (cfg != FS_OK) return cfg;
    fsb::k_grouped_dgemm_stream<TA, TB><<<persistent_grid(tiles.n_tiles, 3), fsb::kGemmThreads,
                                          fsb::kGemmSmem, s>>>(tiles);
    return fsb::launch_status();
}

template <class Tiles>
int launch_stream(const Tiles& tiles, bool ta, bool tb, cudaStream_t s) {
    if (ta) return tb ? launch_stream_t<true, true>(tiles, s) : launch_stream_t<true, false>(tiles, s);
    return tb ? launch_stream_t<false, true>(tiles, s) : launch_stream_t<false, false>(tiles, s);
}

}  // namespace

extern "C" int fs_grouped_dgemm(const FsGemmProblem* d_problems, int64_t n_problems,
                                const FsGemmTile* d_tiles, int64_t n_tiles, void* stream) {
    if (n_tiles < 0 || n_problems < 0) return FS_ERR_INVALID_ARG;
    if (n_tiles == 0) return FS_OK;
    if (d_problems == nullptr || d_tiles == nullptr) return FS_ERR_INVALID_ARG;
    return launch_tiles(fsb::TileTable{d_problems, n_problems, d_tiles, n_tiles},
                        fsb::as_stream(stream));
}

extern "C" int fs_grouped_dgemm_uniform(const FsGemmProblem* d_problems, int64_t n_problems,
                                        const FsGemmTile* d_tiles, int64_t n_tiles,
                                        int32_t trans_a, int32_t trans_b, void* stream) {
    if (n_tiles < 0 || n_problems < 0) return FS_ERR_INVALID_ARG;
    if (n_tiles == 0) return FS_OK;
    if (d_problems == nullptr || d_tiles == nullptr) return FS_ERR_INVALID_ARG;
    return launch_stream(fsb::TileTable{d_problems, n_problems, d_tiles, n_tiles}, trans_a != 0,
                         trans_b != 0, fsb::as_stream(stream));
}

// ---------------------------------------------------------------- wide GEMMs
// Products of a small matrix with many columns (a corner on a wide half network,
// projector applications: M and K of a few tens, N of 1e5 and more).  Both the
// FP64 tensor pipe (2 M K per column) and HBM (8 (M + K) bytes per column) bound
// them, so neither may wait for the other: op(A) of a problem stays in shared
// memory for all its columns, and the 16 warps of the SM work on their own strips
// of 8 NT columns without a CTA barrier.  A warp loads its strip straight into
// DMMA B fragments (all K rows in flight, four rows of 64 bytes per load),
// multiplies it by every 8-row block of A, and turns each 8 x 8 NT block of C
// through a small buffer into whole 64 NT-byte runs.  The 64 x 64 tiles of the
// streaming kernel reload A for every tile by 8-byte cp.async and write C in
// halves of sectors.  9 sectors with M = K = 7 to 51 and N = 0.1 to 0.2 M: 313 us
// there (L2 write sectors 4 times the ideal), 201 us here.  The 16 warps take 128
// registers a thread; over all forms ptxas stores 132 and loads 508 spilled bytes.
//
// CTA b takes an equal share of the estimated time of all strips, problem by
// problem, so it loads one or two A.  The host adds up the times: with every CTA
// counting the strips of every problem, 30 sectors of 8 x 8 on 0.1 M columns took
// 42 us, 17 us now.
namespace fsb {

constexpr int kWideWarps = 16;
constexpr int kWideThreads = 32 * kWideWarps;
constexpr int kWideMaxProblems = 40;
constexpr int kWideBufC = 16 * (16 + 2);   // a warp's block of C
// doubles of the largest op(A) beside the C buffers, in 227 KB
constexpr int kWideMaxA = 227 * 1024 / 8 - kWideWarps * kWideBufC;

struct WideList {
    FsGemmProblem v[kWideMaxProblems];
    int64_t pos[kWideMaxProblems + 1];   // time of all strips before each problem
    int32_t n_problems;
    int32_t a_doubles;   // shared doubles of the largest op(A)
};

// padded rows, k and leading dimension of A in shared memory: 4 mod 8 doubles,
// so that the 8 x 4 fragment reads of a half warp touch distinct banks
__host__ __device__ __forceinline__ int wide_rows(int M) { return (M + 7) / 8 * 8; }
// k steps of 4, rounded up to an instantiated number
__host__ __device__ __forceinline__ int wide_steps(int K) {
    const int n = K > 4 ? (K + 3) / 4 : 1;
    return n <= 2 ? n : (n + 1) / 2 * 2;
}
__host__ __device__ __forceinline__ int wide_k(int K) { return 4 * wide_steps(K); }
__host__ __device__ __forceinline__ int wide_ld(int K) {
    const int k4 = wide_k(K);
    return k4 % 8 == 0 ? k4 + 4 : k4;
}
// columns of a strip: its fragments take up to 64 registers, and longer runs of B
// and C rows serve short K (M = K = 8 on 2 M columns 50 us in strips of 32, 64 us
// in strips of 16; M = K = 32 on 0.6 M columns 87 and 72 us)
__host__ __device__ __forceinline__ int wide_cols(int K) {
    return wide_steps(K) <= 4 ? 32 : wide_steps(K) <= 16 ? 16 : 8;
}
__host__ __device__ __forceinline__ int64_t wide_strip_count(int N, int K) {
    return (static_cast<int64_t>(N) + wide_cols(K) - 1) / wide_cols(K);
}
// relative time of a strip, in 1 / 2944 cycles of an SM: FP64 FMAs at 64 per cycle,
// bytes at 23, the shorter of the two about half hidden, and what a strip takes
// whatever its size (64 cycles; 0 and 16 left the CTAs of the smallest sectors
// late: 40 ragged sectors of M <= 150 on 0.3 M columns 9 % and 6 % slower).
// Rounded to whole cycles of a column, a strip of 1 x 1 had counted 1 / 129 of one
// of 4 x 3: 9 sectors of up to 4 x 3 on 0.3 M columns 93 us, 15 us now.
constexpr int64_t kWideStrip = 2944 * 64;
__host__ __device__ __forceinline__ int64_t wide_cost(int M, int K) {
    const int64_t math = static_cast<int64_t>(wide_rows(M)) * wide_k(K) * 23;
    const int64_t mem = (static_cast<int64_t>(M) + K) * 8 * 64;
    return (math > mem ? 2 * math + mem : 2 * mem + math) * wide_cols(K) + kWideStrip;
}

// The columns n0 .. n0 + 8 NT - 1 of op(B) as DMMA fragments, one k step at a
// time; columns past `left` and rows past K are zero.
struct WideSource {
    const double* p;   // this lane's row of step 0, column 0
    int64_t sk, sn;
    int K, left;       // columns left, 0: nothing to load
    template <int NT>
    __device__ __forceinline__ void load(double (&b)[NT], int ks) {
        const int lane = threadIdx.x % 32;
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            const bool ok = 4 * ks + (lane & 3) < K && 8 * j + (lane >> 2) < left;
            b[j] = ok ? __ldg(p + 8 * j * sn) : 0.0;
        }
        p += 4 * sk;
    }
};

// H blocks of 8 rows of C = A b for one strip: A at pa (this lane's fragment
// row and k), through the warp's buffer sc to d, `rows` rows left.  kNext: the
// strip's last rows; each fragment of b is replaced by the next strip's once its
// products are issued, so that the loads run behind the products and the stores.
template <int H, bool kNext, int NT, int KS>
__device__ __forceinline__ void wide_rows_of(double (&b)[KS][NT], const double* pa, int ld,
                                             double* sc, double* d, int64_t ldc, int rows,
                                             bool col_ok, double alpha, double beta,
                                             WideSource next) {
    constexpr int kCols = 8 * NT;
    constexpr int kLdC = kCols + 2;
    const int lane = threadIdx.x % 32;
    const int fr = lane >> 2, fk = lane & 3;
    double acc[H][NT][2];
#pragma unroll
    for (int h = 0; h < H; ++h)
#pragma unroll
        for (int j = 0; j < NT; ++j) acc[h][j][0] = acc[h][j][1] = 0.0;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
#pragma unroll
        for (int h = 0; h < H; ++h) {
            const double a = pa[h * 8 * ld + 4 * ks];
#pragma unroll
            for (int j = 0; j < NT; ++j) dmma(acc[h][j], a, b[ks][j]);
        }
        if (kNext) next.load(b[ks], ks);
    }
    __syncwarp();   // the previous block has been stored
#pragma unroll
    for (int h = 0; h < H; ++h)
#pragma unroll
        for (int j = 0; j < NT; ++j)
            *reinterpret_cast<double2*>(sc + (8 * h + fr) * kLdC + 8 * j + 2 * fk) =
                make_double2(alpha * acc[h][j][0], alpha * acc[h][j][1]);
    __syncwarp();
    const int r0 = lane / kCols;
    const double* c = sc + r0 * kLdC + lane % kCols;
    if (!col_ok) return;
    if (beta == 0.0) {
#pragma unroll
        for (int r = 0; r < 8 * H; r += 32 / kCols) {
            if (r + r0 < rows) *d = c[r * kLdC];
            d += (32 / kCols) * ldc;
        }
    } else {
#pragma unroll
        for (int r = 0; r < 8 * H; r += 32 / kCols) {
            if (r + r0 < rows) *d = fma(beta, *d, c[r * kLdC]);
            d += (32 / kCols) * ldc;
        }
    }
}

// The strips [first, last) of one problem, k steps padded to KS with zeros, H
// blocks of 8 rows at a time.
template <int H, int NT, int KS>
__device__ __forceinline__ void wide_strips(const FsGemmProblem& p, const double* sa, int ld,
                                            double* sc, int64_t first, int64_t last) {
    constexpr int kCols = 8 * NT;
    const int lane = threadIdx.x % 32, wid = threadIdx.x / 32;
    const int fr = lane >> 2, fk = lane & 3;
    const int M = p.M, N = p.N, K = p.K;
    const int64_t sk = p.transB ? 1 : p.ldb, sn = p.transB ? p.ldb : 1;
    const int64_t ldc = p.ldc;
    const double alpha = p.alpha, beta = p.beta;
    const double* pa = sa + fr * ld + fk;
    auto source = [&](int64_t strip) {
        const int64_t n0 = strip * kCols;
        return WideSource{p.B + fk * sk + (n0 + fr) * sn, sk, sn, K,
                          strip < last ? static_cast<int>(min(N - n0, static_cast<int64_t>(kCols)))
                                       : 0};
    };
    int64_t s = first + wid;
    double b[KS][NT];
    WideSource now = source(s);
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) now.load(b[ks], ks);
#pragma unroll 1
    for (; s < last; s += kWideWarps) {
        const int64_t n0 = s * kCols;
        const WideSource next = source(s + kWideWarps);
        const bool col_ok = n0 + lane % kCols < N;
        double* d = p.C + (lane / kCols) * ldc + n0 + lane % kCols;
        int m0 = 0;
#pragma unroll 1
        for (; m0 + 8 * H < M; m0 += 8 * H) {
            wide_rows_of<H, false>(b, pa + m0 * ld, ld, sc, d, ldc, 8 * H, col_ok, alpha, beta,
                                   next);
            d += 8 * H * ldc;
        }
        if (H > 1 && m0 + 8 < M)
            wide_rows_of<H, true>(b, pa + m0 * ld, ld, sc, d, ldc, M - m0, col_ok, alpha, beta,
                                  next);
        else
            wide_rows_of<1, true>(b, pa + m0 * ld, ld, sc, d, ldc, M - m0, col_ok, alpha, beta,
                                  next);
    }
}

__global__ void __launch_bounds__(kWideThreads, 1)
    k_dgemm_wide(const __grid_constant__ WideList list) {
    extern __shared__ __align__(16) double wide_smem[];
    double* sa = wide_smem;
    double* sc = wide_smem + list.a_doubles + threadIdx.x / 32 * kWideBufC;

    const int64_t total = list.pos[list.n_problems];
    const int64_t lo = total / gridDim.x * blockIdx.x +
                       total % gridDim.x * blockIdx.x / gridDim.x;
    const int64_t hi = total / gridDim.x * (blockIdx.x + 1) +
                       total % gridDim.x * (blockIdx.x + 1) / gridDim.x;
#pragma unroll 1
    for (int i = 0; i < list.n_problems && list.pos[i] < hi; ++i) {
        if (list.pos[i + 1] <= lo) continue;   // its divisions would cost as much as a strip
        const FsGemmProblem& p = list.v[i];
        const int64_t cost = wide_cost(p.M, p.K), pos = list.pos[i];
        const int64_t first = lo > pos ? (lo - pos + cost - 1) / cost : 0;
        const int64_t last = min((hi - pos + cost - 1) / cost, wide_strip_count(p.N, p.K));
        if (first >= last || p.M <= 0) continue;
        const int m8 = wide_rows(p.M), k4 = wide_k(p.K), ld = wide_ld(p.K);
        __syncthreads();   // the previous problem's A has been read
        for (int e = threadIdx.x; e < m8 * k4; e += kWideThreads) {
            // consecutive threads along the contiguous direction of A
            const int m = p.transA ? e % m8 : e / k4, k = p.transA ? e / m8 : e % k4;
            double v = 0.0;
            if (m < p.M && k < p.K)
                v = p.A[p.transA ? static_cast<int64_t>(k) * p.lda + m
                                 : static_cast<int64_t>(m) * p.lda + k];
            sa[m * ld + k] = v;
        }
        __syncthreads();
        switch (k4 / 4) {
#define FSB_WIDE(h, nt, ks) \
    case ks: wide_strips<h, nt, ks>(p, sa, ld, sc, first, last); break;
            FSB_WIDE(1, 4, 1)
            FSB_WIDE(1, 4, 2)
            FSB_WIDE(1, 4, 4)
            FSB_WIDE(2, 2, 6)
            FSB_WIDE(2, 2, 8)
            FSB_WIDE(2, 2, 10)
            FSB_WIDE(2, 2, 12)
            FSB_WIDE(2, 2, 14)
            FSB_WIDE(2, 2, 16)
            FSB_WIDE(2, 1, 18)
            FSB_WIDE(2, 1, 20)
            FSB_WIDE(2, 1, 22)
            FSB_WIDE(2, 1, 24)
            FSB_WIDE(2, 1, 26)
            FSB_WIDE(2, 1, 28)
            FSB_WIDE(2, 1, 30)
            FSB_WIDE(2, 1, 32)
#undef FSB_WIDE
        }
    }
}

}  // namespace fsb

extern "C" int fs_dgemm_wide_limits(int32_t* max_problems, int32_t* max_k, int32_t* max_a) {
    if (max_problems == nullptr || max_k == nullptr || max_a == nullptr) return FS_ERR_INVALID_ARG;
    *max_problems = fsb::kWideMaxProblems;
    *max_k = 128;
    *max_a = fsb::kWideMaxA;
    return FS_OK;
}

extern "C" int fs_grouped_dgemm_wide(const FsGemmProblem* h_problems, int64_t n_problems,
                                     void* stream) {
    if (n_problems < 0) return FS_ERR_INVALID_ARG;
    if (n_problems == 0) return FS_OK;
    if (h_problems == nullptr) return FS_ERR_INVALID_ARG;
    if (n_problems > fsb::kWideMaxProblems) return FS_ERR_TOO_LARGE;
    fsb::WideList list;
    memcpy(list.v, h_problems, sizeof(FsGemmProblem) * static_cast<size_t>(n_problems));
    list.n_problems = static_cast<int32_t>(n_problems);
    list.a_doubles = 0;
    list.pos[0] = 0;
    for (int64_t i = 0; i < n_problems; ++i) {
        const FsGemmProblem& p = h_problems[i];
        if (p.M < 0 || p.N < 0 || p.K < 0) return FS_ERR_INVALID_ARG;
        if (p.K > 128 || p.M > fsb::kWideMaxA) return FS_ERR_TOO_LARGE;
        const int64_t a = static_cast<int64_t>(fsb::wide_rows(p.M)) * fsb::wide_ld(p.K);
        if (a > fsb::kWideMaxA) return FS_ERR_TOO_LARGE;
        if (a > list.a_doubles) list.a_doubles = static_cast<int32_t>(a);
        list.pos[i + 1] = list.pos[i] + fsb::wide_strip_count(p.N, p.K) * fsb::wide_cost(p.M, p.K);
    }
    const int bytes = static_cast<int>(sizeof(double)) *
                      (list.a_doubles + fsb::kWideWarps * fsb::kWideBufC);
    // one limit for every size: one CTA runs per SM whatever it asks for
    const int st = fsb::configure_smem(reinterpret_cast<const void*>(fsb::k_dgemm_wide),
                                       static_cast<int>(sizeof(double)) *
                                           (fsb::kWideMaxA + fsb::kWideWarps * fsb::kWideBufC));
    if (st != FS_OK) return st;
    fsb::k_dgemm_wide<<<fsb::num_sms(), fsb::kWideThreads, bytes, fsb::as_stream(stream)>>>(list);
    return fsb::launch_status();
}

// ---------------------------------------------------------------- thin GEMMs
// C[MxN] = alpha A[MxK] B[KxN] + beta C for M, K <= 32 and N large: the
// recoupling products of a non-abelian permute (one small isometry applied to
// many external-degeneracy columns).  Bandwidth bound: each thread owns output
// columns, A is staged once per tile in shared memory and read as broadcasts,
// the accumulators live in registers (M rounded up to 4, 8, 16 or 32).  Both
// operands row-major (transA == transB == 0; the host checks).
namespace fsb {

constexpr int kThinMax = 32;
constexpr int kThinThreads = 128;
constexpr int kThinColsPerThread = 4;

// MB, KB: M and K rounded up to 4, 8, 16 or 32; NC: columns a thread carries
// at once (KB * NC <= 32 doubles of operands in registers).  Every load of a
// pass (KB per column, predicated on k < K) is issued before its FMAs, so each
// thread keeps up to 32 loads in flight: with the k loop rolled, one load per
// column at a time left the kernel latency bound at a third of the HBM
// bandwidth.
template <int MB, int KB, int NC>
__device__ __forceinline__ void thin_tile(const FsGemmProblem& p, const double* su, int n0) {
#pragma unroll
    for (int c0 = 0; c0 < kThinColsPerThread; c0 += NC) {
        int cols[NC];
        bool ok[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            cols[c] = n0 + threadIdx.x + (c0 + c) * kThinThreads;
            ok[c] = cols[c] < p.N;
        }
        double x[KB][NC];
#pragma unroll
        for (int k = 0; k < KB; ++k)
#pragma unroll
            for (int c = 0; c < NC; ++c)
                x[k][c] = (ok[c] && k < p.K)
                              ? __ldg(p.B + static_cast<int64_t>(k) * p.ldb + cols[c])
                              : 0.0;
#pragma unroll
        for (int m = 0; m < MB; ++m) {
            if (m >= p.M) break;
            double acc[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) acc[c] = 0.0;
#pragma unroll
            for (int k = 0; k < KB; ++k) {
                // su holds zeros for k >= K (the staging pads the rows)
                const double u = su[m * kThinMax + k];
#pragma unroll
                for (int c = 0; c < NC; ++c) acc[c] = fma(u, x[k][c], acc[c]);
            }
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                if (!ok[c]) continue;
                double* dst = p.C + static_cast<int64_t>(m) * p.ldc + cols[c];
                const double v = p.alpha * acc[c];
                *dst = (p.beta == 0.0) ? v : fma(p.beta, *dst, v);
            }
        }
    }
}

template <int MB>
__device__ __forceinline__ void thin_tile_k(const FsGemmProblem& p, const double* su, int n0) {
    if (p.K <= 4)
        thin_tile<MB, 4, 4>(p, su, n0);
    else if (p.K <= 8)
        thin_tile<MB, 8, 4>(p, su, n0);
    else if (p.K <= 16)
        thin_tile<MB, 16, 2>(p, su, n0);
    else
        thin_tile<MB, 32, 1>(p, su, n0);
}

template <class Tiles>
__global__ void __launch_bounds__(kThinThreads, 4)
    k_grouped_dgemm_thin(const __grid_constant__ Tiles tiles) {
    __shared__ double su[kThinMax * kThinMax];
    constexpr int kCols = kThinThreads * kThinColsPerThread;
    __shared__ FsGemmProblem p;   // in registers beside the operands it spills
    typename Tiles::Cursor cursor;
    for (int64_t t = blockIdx.x; t < tiles.n_tiles; t += gridDim.x) {
        FsGemmProblem found;
        int m0, n0;   // every row is in one tile; tables leave tm at 0
        if (!tiles.template find<kThinMax, kCols>(cursor, t, found, m0, n0)) continue;
        if (found.M > kThinMax || found.K > kThinMax || found.transA || found.transB) continue;
        __syncthreads();  // previous tile's reads of su and p are done
        if (threadIdx.x == 0) p = found;
        __syncthreads();
        // rows m < M of U, zero-padded to kThinMax columns (the unrolled k
        // loop reads up to K rounded up)
        const int mk = p.M * kThinMax;
        for (int i = threadIdx.x; i < mk; i += kThinThreads) {
            const int m = i / kThinMax, k = i - m * kThinMax;
            su[i] = (k < p.K) ? p.A[static_cast<int64_t>(m) * p.lda + k] : 0.0;
        }
        __syncthreads();
        if (p.M <= 4)
            thin_tile_k<4>(p, su, n0);
        else if (p.M <= 8)
            thin_tile_k<8>(p, su, n0);
        else if (p.M <= 16)
            thin_tile_k<16>(p, su, n0);
        else
            thin_tile_k<32>(p, su, n0);
    }
}

}  // namespace fsb

extern "C" int fs_thin_dgemm_shape(int32_t* max_m, int32_t* max_k, int32_t* tile_n) {
    if (max_m == nullptr || max_k == nullptr || tile_n == nullptr) return FS_ERR_INVALID_ARG;
    *max_m = fsb::kThinMax;
    *max_k = fsb::kThinMax;
    *tile_n = fsb::kThinThreads * fsb::kThinColsPerThread;
    return FS_OK;
}

namespace {

template <class Tiles>
int launch_thin(const Tiles& tiles, cudaStream_t s) {
    fsb::k_grouped_dgemm_thin<<<persistent_grid(tiles.n_tiles, 8), fsb::kThinThreads, 0, s>>>(
        tiles);
    return fsb::launch_status();
}

}  // namespace

extern "C" int fs_grouped_dgemm_thin(const FsGemmProblem* d_problems, int64_t n_problems,
                                     const FsGemmTile* d_tiles, int64_t n_tiles, void* stream) {
    if (n_tiles < 0 || n_problems < 0) return FS_ERR_INVALID_ARG;
    if (n_tiles == 0) return FS_OK;
    if (d_problems == nullptr || d_tiles == nullptr) return FS_ERR_INVALID_ARG;
    return launch_thin(fsb::TileTable{d_problems, n_problems, d_tiles, n_tiles},
                       fsb::as_stream(stream));
}

namespace {

// Problems by value: 3.5 KB of parameters, or 31 KB for longer lists.
template <int N>
int launch_list(const FsGemmProblem* h, int64_t n, int kind, cudaStream_t s) {
    fsb::TileList<N> t;
    memcpy(t.v, h, sizeof(FsGemmProblem) * static_cast<size_t>(n));
    t.n_problems = n;
    t.n_tiles = 0;
    constexpr int kThinCols = fsb::kThinThreads * fsb::kThinColsPerThread;
    for (int64_t i = 0; i < n; ++i) {
        const FsGemmProblem& p = h[i];
        if (p.M < 0 || p.N < 0 || p.K < 0) return FS_ERR_INVALID_ARG;
        const int64_t tiles =
            kind == FS_DGEMM_THIN
                ? fsb::TileList<N>::template count<fsb::kThinMax, kThinCols>(p)
                : fsb::TileList<N>::template count<fsb::kTM, fsb::kTN>(p);
        if (tiles >= (1ll << 31)) return FS_ERR_TOO_LARGE;
        t.n_tiles += tiles;
        if (kind == FS_DGEMM_UNIFORM && ((p.transA != 0) != (h[0].transA != 0) ||
                                         (p.transB != 0) != (h[0].transB != 0)))
            return FS_ERR_INVALID_ARG;
        if (kind == FS_DGEMM_THIN &&
            (p.M > fsb::kThinMax || p.K > fsb::kThinMax || p.transA || p.transB))
            return FS_ERR_INVALID_ARG;
    }
    if (t.n_tiles == 0) return FS_OK;
    if (kind == FS_DGEMM_TILES) return launch_tiles(t, s);
    if (kind == FS_DGEMM_UNIFORM) return launch_stream(t, h[0].transA != 0, h[0].transB != 0, s);
    return launch_thin(t, s);
}

}  // namespace

extern "C" int fs_grouped_dgemm_list(const FsGemmProblem* h_problems, int64_t n_problems,
                                     int32_t kind, void* stream) {
    constexpr int kShort = 40;
    static_assert(sizeof(fsb::TileList<kShort>) < 4000, "short lists fit 4 KB of parameters");
    static_assert(sizeof(fsb::TileList<FS_DGEMM_LIST_MAX>) <= 32764, "kernel parameter limit");
    if (n_problems < 0 || kind < FS_DGEMM_TILES || kind > FS_DGEMM_THIN) return FS_ERR_INVALID_ARG;
    if (n_problems == 0) return FS_OK;
    if (h_problems == nullptr) return FS_ERR_INVALID_ARG;
    if (n_problems > FS_DGEMM_LIST_MAX) return FS_ERR_TOO_LARGE;
    cudaStream_t s = fsb::as_stream(stream);
    return n_problems <= kShort ? launch_list<kShort>(h_problems, n_problems, kind, s)
                                : launch_list<FS_DGEMM_LIST_MAX>(h_problems, n_problems, kind, s);
}

// ------------------------------------------------------------ split-K reduce
// When a contraction has too few output tiles to fill the GPU, the host cuts
// long-K sector problems into K chunks whose partial products go to a
// workspace (slice j of an item at W + j * slice); this kernel sums the slices
// in order (deterministic, no atomics) and applies alpha / beta into C.
namespace fsb {

template <class Table>
__global__ void __launch_bounds__(256)
    k_splitk_reduce(const __grid_constant__ Table items, int64_t n_items) {
    const int64_t it = blockIdx.y;
    if (it >= n_items) return;
    const FsSplitReduce r = items[it];
    const int64_t n = static_cast<int64_t>(r.M) * r.N;
    for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < n;
         e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        double v = 0.0;
        for (int j = 0; j < r.nslices; ++j) v += __ldg(r.W + j * r.slice + e);
        const int64_t i = e / r.N, c = e - i * r.N;
        double* dst = r.C + i * r.ldc + c;
        *dst = (r.beta == 0.0) ? r.alpha * v : fma(r.beta, *dst, r.alpha * v);
    }
}

}  // namespace fsb

namespace {

template <class Table>
int splitk_reduce(const Table& items, int64_t n_items, int64_t max_elems, void* stream) {
    const int64_t blocks = (max_elems + 255) / 256;
    const int gx = static_cast<int>(blocks < 4 * fsb::num_sms() ? blocks : 4 * fsb::num_sms());
    fsb::k_splitk_reduce<<<dim3(gx, static_cast<unsigned>(n_items)), 256, 0,
                           fsb::as_stream(stream)>>>(items, n_items);
    return fsb::launch_status();
}

}  // namespace

extern "C" int fs_splitk_reduce(const FsSplitReduce* d_items, int64_t n_items,
                                int64_t max_elems, void* stream) {
    if (n_items < 0 || max_elems < 0) return FS_ERR_INVALID_ARG;
    if (n_items == 0 || max_elems == 0) return FS_OK;
    if (d_items == nullptr) return FS_ERR_INVALID_ARG;
    if (n_items > 65535) return FS_ERR_TOO_LARGE;
    return splitk_reduce(fsb::DeviceTable<FsSplitReduce>{d_items}, n_items, max_elems, stream);
}

extern "C" int fs_splitk_reduce_list(const FsSplitReduce* h_items, int64_t n_items,
                                     int64_t max_elems, void* stream) {
    if (n_items < 0 || max_elems < 0) return FS_ERR_INVALID_ARG;
    if (n_items == 0 || max_elems == 0) return FS_OK;
    if (h_items == nullptr) return FS_ERR_INVALID_ARG;
    if (n_items > FS_SPLIT_LIST_MAX) return FS_ERR_TOO_LARGE;
    return splitk_reduce(fsb::inline_table<FsSplitReduce, FS_SPLIT_LIST_MAX>(h_items, n_items),
                         n_items, max_elems, stream);
}

// Tile table from runs (see FsTileRun): one thread per tile, binary search of
// its run over the sorted run starts.
namespace fsb {

__global__ void __launch_bounds__(256)
    k_expand_tiles(const FsTileRun* __restrict__ runs, int64_t n_runs, int64_t total,
                   FsGemmTile* __restrict__ tiles) {
    for (int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < total;
         t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        int64_t lo = 0, hi = n_runs - 1;   // last run with start <= t
        while (lo < hi) {
            const int64_t mid = (lo + hi + 1) / 2;
            if (__ldg(&runs[mid].start) <= t)
                lo = mid;
            else
                hi = mid - 1;
        }
        const FsTileRun r = runs[lo];
        const int64_t k = t - r.start;
        if (r.col_major) {
            const int32_t nr = r.nrow > 0 ? r.nrow : 1;
            tiles[t] = FsGemmTile{r.problem, static_cast<int32_t>(k % nr),
                                  static_cast<int32_t>(k / nr), 0};
        } else {
            const int32_t nc = r.ncol > 0 ? r.ncol : 1;
            tiles[t] = FsGemmTile{r.problem, static_cast<int32_t>(k / nc),
                                  static_cast<int32_t>(k % nc), 0};
        }
    }
}

}  // namespace fsb

extern "C" int fs_expand_tiles(const FsTileRun* d_runs, int64_t n_runs, int64_t total,
                               FsGemmTile* d_tiles, void* stream) {
    if (n_runs < 0 || total < 0) return FS_ERR_INVALID_ARG;
    if (total == 0) return FS_OK;
    if (n_runs == 0 || d_runs == nullptr || d_tiles == nullptr) return FS_ERR_INVALID_ARG;
    const int64_t blocks = (total + 255) / 256;
    const int grid = static_cast<int>(blocks < 8 * fsb::num_sms() ? blocks : 8 * fsb::num_sms());
    fsb::k_expand_tiles<<<grid, 256, 0, fsb::as_stream(stream)>>>(d_runs, n_runs, total,
                                                                  d_tiles);
    return fsb::launch_status();
}
