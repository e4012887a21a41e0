// O(2) <-> U(1) change of basis of symmetric-tensor blocks.
//
// Reference behaviour (frostspin/symmetric_tensor/o2_symmetric_tensor.py): an
// O(2) tensor stores its 0odd and 0even blocks and the U(1) blocks of charge
// n > 0.  Its U(1) form adds the charge -n blocks, obtained from the charge n
// ones by the Sz reflection with a sign per row and per column
// (_generate_neg_sz_blocks :798-851, _numba_generate_refl_block :327-354),
// and the charge-0 block, an orthogonal mix of the 0odd and 0even blocks
// (_numba_merge_b0oe :269-288); back from U(1), the charge-0 block is split
// into 0odd and 0even again (_numba_split_b0 :291-310).
//
// Every one of these is a separable gather: output element (i, j) of a block is
// a sum over at most four terms t of rcoef_t[i] * src_t[ridx_t[i], cidx_t[j]] *
// ccoef_t[j].  The host builds the per-row and per-column tables; one launch
// covers every block of a cast.  A CTA walks output rows (grid-stride), loads
// the row's index and coefficient of each term once, and its threads stride
// over the columns, so output stores are coalesced.  Products are rounded
// step by step in the reference's order ((rcoef * x) * ccoef, terms summed in
// order, no fused multiply-add), so the results equal the reference's loops.
//
// Bound by latency: every source load waits for its column's index, so what
// counts is warps in flight (40 per SM) rather than loads per warp.  The term
// counts that occur (1 for reflections and copies, 2 for the merge, 4 for the
// split) are separate forms with two columns per thread; the general loop over
// up to four terms took 64 us for each cast of 5.6 M coefficients, this 55 us,
// with 80 bytes spilled at the 48 registers that ten CTAs per SM leave.
// Tiles of 8 rows x 256 columns (100 registers) took 90 us; 32 x 32 tiles per
// warp 48 us, but 17 us instead of 4.5 us at 70 000 coefficients.
#include "common.cuh"

namespace fsb {

constexpr int kO2Threads = 128;
constexpr int kO2Cols = 2;     // columns of a thread at a time
constexpr int kO2Ctas = 10;    // per SM

// Row i of a block, NT terms, kO2Cols columns of a thread at a time.
template <int NT>
__device__ __forceinline__ bool o2_row(const FsO2Block& blk, int nt,
                                       const double* __restrict__ src, int64_t src_len,
                                       double* __restrict__ out, int64_t out_len,
                                       const int64_t* __restrict__ index,
                                       const double* __restrict__ coef, int64_t i) {
    int64_t rbase[NT];
    double rc[NT];
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        const FsO2Term& tm = blk.terms[t < nt ? t : 0];
        rbase[t] = tm.src_off + __ldg(index + tm.ridx_off + i) * tm.rs;
        rc[t] = __ldg(coef + tm.rcoef_off + i);
    }
    const int64_t ncols = blk.ncols, orow = blk.out_off + i * ncols;
    bool fine = true;
    for (int64_t j0 = threadIdx.x; j0 < ncols; j0 += kO2Threads * kO2Cols) {
        double x[NT][kO2Cols], cc[NT][kO2Cols];
        bool ok[NT][kO2Cols];
        int64_t pos[NT][kO2Cols];
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const FsO2Term& tm = blk.terms[t < nt ? t : 0];
#pragma unroll
            for (int c = 0; c < kO2Cols; ++c) {
                const int64_t j = j0 + c * kO2Threads;
                const bool here = j < ncols && t < nt;
                pos[t][c] = here ? rbase[t] + __ldg(index + tm.cidx_off + j) * tm.cs : 0;
                cc[t][c] = here ? __ldg(coef + tm.ccoef_off + j) : 0.0;
                ok[t][c] = here && static_cast<uint64_t>(pos[t][c]) < static_cast<uint64_t>(src_len);
                fine = fine && (ok[t][c] || !here);
            }
        }
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int c = 0; c < kO2Cols; ++c) x[t][c] = ok[t][c] ? __ldg(src + pos[t][c]) : 0.0;
#pragma unroll
        for (int c = 0; c < kO2Cols; ++c) {
            double acc = 0.0;
#pragma unroll
            for (int t = 0; t < NT; ++t)
                if (ok[t][c])
                    acc = __dadd_rn(acc, __dmul_rn(__dmul_rn(rc[t], x[t][c]), cc[t][c]));
            const int64_t j = j0 + c * kO2Threads;
            if (j < ncols) {
                if (static_cast<uint64_t>(orow + j) < static_cast<uint64_t>(out_len))
                    out[orow + j] = acc;
                else
                    fine = false;
            }
        }
    }
    return fine;
}

__global__ void __launch_bounds__(kO2Threads, kO2Ctas)
    k_o2_recombine(const double* __restrict__ src, int64_t src_len, double* __restrict__ out,
                   int64_t out_len, const FsO2Block* __restrict__ blocks,
                   const int64_t* __restrict__ index, const double* __restrict__ coef,
                   int32_t* flag) {
    const FsO2Block& blk = blocks[blockIdx.y];
    const int nt = blk.nterms < FS_O2_MAXTERMS ? blk.nterms : FS_O2_MAXTERMS;
    bool fine = true;
    for (int64_t i = blockIdx.x; i < blk.nrows; i += gridDim.x) {
        bool f = true;
        if (nt == 1) {
            f = o2_row<1>(blk, nt, src, src_len, out, out_len, index, coef, i);
        } else if (nt == 2) {
            f = o2_row<2>(blk, nt, src, src_len, out, out_len, index, coef, i);
        } else if (nt > 2) {
            f = o2_row<4>(blk, nt, src, src_len, out, out_len, index, coef, i);
        } else {   // an empty sum
            for (int64_t j = threadIdx.x; j < blk.ncols; j += kO2Threads) {
                const int64_t o = blk.out_off + i * blk.ncols + j;
                if (static_cast<uint64_t>(o) < static_cast<uint64_t>(out_len))
                    out[o] = 0.0;
                else
                    f = false;
            }
        }
        fine = fine && f;
    }
    if (!fine) raise_flag(flag, FS_ERR_BOUNDS);
}

}  // namespace fsb

extern "C" int fs_o2_recombine(const double* d_src, int64_t src_len, double* d_out,
                               int64_t out_len, const FsO2Block* d_blocks, int64_t n_blocks,
                               const int64_t* d_index, const double* d_coef, int64_t max_rows,
                               int32_t* d_flag, void* stream) {
    if (n_blocks < 0 || max_rows < 0 || src_len < 0 || out_len < 0) return FS_ERR_INVALID_ARG;
    if (n_blocks == 0 || max_rows == 0) return FS_OK;
    if (d_blocks == nullptr || d_index == nullptr || d_coef == nullptr || d_out == nullptr)
        return FS_ERR_INVALID_ARG;
    if (d_src == nullptr && src_len > 0) return FS_ERR_INVALID_ARG;
    if (n_blocks > 65535) return FS_ERR_TOO_LARGE;
    const int64_t cap = static_cast<int64_t>(fsb::num_sms()) * 8;
    const int gx = static_cast<int>(max_rows < cap ? max_rows : cap);
    fsb::k_o2_recombine<<<dim3(gx, static_cast<unsigned>(n_blocks)), fsb::kO2Threads, 0,
                          fsb::as_stream(stream)>>>(d_src, src_len, d_out, out_len, d_blocks,
                                                    d_index, d_coef, d_flag);
    return fsb::launch_status();
}
