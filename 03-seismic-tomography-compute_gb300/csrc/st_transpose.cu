// CSR transpose by a stable counting sort of the entries on their column.
//
// The entries of A are in (row, column) order, so a stable sort on the column
// alone lists every column's entries by ascending row: A^T. Least significant
// digit first with digits of up to ten bits (1024 bins): a matrix of up to 2^20
// columns takes two passes over 12 bytes per entry (column, row, value).
//
// Bound by memory. Each CTA owns one contiguous range of the entries, all CTAs
// resident at once: a histogram pass counts the range's digits, a scan over
// [digit][CTA] gives every CTA its first place per digit, and the scatter pass
// walks the range in tiles of 4096, sorts each tile in shared memory (ranks by
// warp match, so equal digits keep their order) and writes it out in runs of
// equal digit. Against the general triplet sort (64-bit keys, 8-bit digits, a
// scattered write per entry; six passes for 10^6 columns x 2*10^6 rows) it
// moves a third of the bytes in long runs. Measured: 45M entries, 125,000 columns
// (two passes of 523 us) 1.3 ms against 5.1 ms of kernels; the first tomography
// solve on a new 361M-entry matrix, transpose included, 74.4 -> 35.5 ms.
//
// The columns lie in arrays that callers may write (st_csr_device_arrays). The last
// pass looks for columns outside the matrix and for entries that repeat one; a
// matrix with either is transposed by the triplet sort, which drops the former and
// sums the latter.
#include "st_sort.cuh"
#include "st_sparse.cuh"

#include <algorithm>

namespace stg {
namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int TR_THREADS = 256;
constexpr int TR_WARPS = TR_THREADS / 32;
constexpr int TR_ITEMS = 16;
constexpr int TR_TILE = TR_THREADS * TR_ITEMS;
constexpr int TR_BITS = 10;
constexpr int TR_BINS = 1 << TR_BITS;
constexpr int TR_CTAS_PER_SM = 3;  // 72 KB of shared memory each

struct TrSmem {
    unsigned short cnt[TR_WARPS][TR_BINS];  // a warp's count, then its first place, per digit
    unsigned start[TR_BINS];                // the tile's first place per digit
    unsigned run[TR_BINS];                  // the range's next output place per digit
    unsigned wsum[TR_WARPS];
    unsigned key[TR_TILE];
    int row[TR_TILE];
    float val[TR_TILE];
};

__global__ void __launch_bounds__(TR_THREADS) tr_hist_kernel(const int* __restrict__ key, long long n, long long range,
                                                             int shift, int bins, long long* __restrict__ hist) {
    __shared__ unsigned h[TR_BINS];
    for (int b = threadIdx.x; b < bins; b += TR_THREADS) h[b] = 0;
    __syncthreads();
    const long long e0 = (long long)blockIdx.x * range, e1 = min(e0 + range, n);  // e0 is a multiple of the tile
    const unsigned mask = (unsigned)bins - 1;
    const long long v1 = e0 + ((e1 - e0) & ~3ll);
    for (long long e = e0 + 4 * (long long)threadIdx.x; e < v1; e += 4 * TR_THREADS) {
        const int4 k = __ldg(reinterpret_cast<const int4*>(key + e));
        atomicAdd(&h[((unsigned)k.x >> shift) & mask], 1u);
        atomicAdd(&h[((unsigned)k.y >> shift) & mask], 1u);
        atomicAdd(&h[((unsigned)k.z >> shift) & mask], 1u);
        atomicAdd(&h[((unsigned)k.w >> shift) & mask], 1u);
    }
    const long long e = v1 + threadIdx.x;
    if (e < e1) atomicAdd(&h[((unsigned)key[e] >> shift) & mask], 1u);
    __syncthreads();
    for (int b = threadIdx.x; b < bins; b += TR_THREADS) hist[(long long)b * gridDim.x + blockIdx.x] = h[b];
}

__global__ void __launch_bounds__(TR_THREADS, TR_CTAS_PER_SM)
    tr_scatter_kernel(const int* __restrict__ key, const int* __restrict__ row, const float* __restrict__ val,
                      long long n, long long range, int shift, int bins, const long long* __restrict__ offs,
                      int* __restrict__ okey, int* __restrict__ orow, float* __restrict__ oval) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TrSmem& S = *reinterpret_cast<TrSmem*>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned mask = (unsigned)bins - 1, lt = (1u << lane) - 1;
    for (int b = tid; b < bins; b += TR_THREADS) S.run[b] = (unsigned)offs[(long long)b * gridDim.x + blockIdx.x];
    const long long r0 = (long long)blockIdx.x * range, r1 = min(r0 + range, n);
    for (long long t0 = r0; t0 < r1; t0 += TR_TILE) {
        const int m = (int)min((long long)TR_TILE, r1 - t0);
        for (int b = tid; b < TR_WARPS * bins; b += TR_THREADS) S.cnt[b / bins][b & (bins - 1)] = 0;
        __syncthreads();
        // rank every entry among its warp's earlier entries of the same digit
        unsigned k[TR_ITEMS];
        unsigned short rank[TR_ITEMS];
        const int first = warp * (32 * TR_ITEMS) + lane;
#pragma unroll
        for (int j = 0; j < TR_ITEMS; ++j) {
            const int i = first + 32 * j;
            k[j] = i < m ? (unsigned)key[t0 + i] : 0u;
        }
#pragma unroll
        for (int j = 0; j < TR_ITEMS; ++j) {
            const bool valid = first + 32 * j < m;
            const unsigned d = valid ? (k[j] >> shift) & mask : 0xffffffffu;
            const unsigned peers = __match_any_sync(FULL, d);
            unsigned old = 0;
            if (valid) old = S.cnt[warp][d];
            __syncwarp();
            if (valid && (peers & lt) == 0) S.cnt[warp][d] = (unsigned short)(old + __popc(peers));
            __syncwarp();
            rank[j] = (unsigned short)(old + __popc(peers & lt));
        }
        __syncthreads();
        // per digit: the warps' first places and the tile's count; then an
        // exclusive scan over the digits (bins / 256 consecutive ones a thread)
        constexpr int PER = TR_BINS / TR_THREADS;
        unsigned c[PER], mine = 0;
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            const int b = tid * PER + q;
            unsigned s = 0;
            if (b < bins) {
                for (int w = 0; w < TR_WARPS; ++w) {
                    const unsigned x = S.cnt[w][b];
                    S.cnt[w][b] = (unsigned short)s;
                    s += x;
                }
            }
            c[q] = s;
            mine += s;
        }
        unsigned incl = mine;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) S.wsum[warp] = incl;
        __syncthreads();
        unsigned base = incl - mine;
        for (int w = 0; w < warp; ++w) base += S.wsum[w];
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            const int b = tid * PER + q;
            if (b < bins) S.start[b] = base;
            base += c[q];
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < TR_ITEMS; ++j) {
            const int i = first + 32 * j;
            if (i < m) {
                const unsigned d = (k[j] >> shift) & mask;
                const unsigned p = S.start[d] + S.cnt[warp][d] + rank[j];
                S.key[p] = k[j];
                S.row[p] = __ldg(row + t0 + i);
                S.val[p] = __ldg(val + t0 + i);
            }
        }
        __syncthreads();
        for (int i = tid; i < m; i += TR_THREADS) {
            const unsigned kk = S.key[i], d = (kk >> shift) & mask;
            const unsigned dst = S.run[d] + ((unsigned)i - S.start[d]);
            okey[dst] = (int)kk;
            orow[dst] = S.row[i];
            oval[dst] = S.val[i];
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            const int b = tid * PER + q;
            if (b < bins) S.run[b] += c[q];
        }
        // the next tile's first barrier comes before run, start or the staged entries are used again
    }
}

// Row of every entry, G lanes per row.
template <int G>
__global__ void tr_rows_kernel(const long long* __restrict__ rp, long long rows, int* __restrict__ out) {
    const int lane = threadIdx.x % G;
    for (long long i = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / G; i < rows;
         i += (long long)gridDim.x * blockDim.x / G)
        for (long long p = rp[i] + lane; p < rp[i + 1]; p += G) out[p] = (int)i;
}

// Row pointers from the sorted keys: entry u is the first of every row in (key[u-1], key[u]].
// *irregular: a key outside the rows (such keys are passed over) or a repeated entry.
// Four entries a thread (the arrays are 16-byte aligned): a transpose of 361M entries
// takes 18.15 ms, 18.9 with one at a time.
__global__ void tr_rowptr_kernel(const int* __restrict__ key, const int* __restrict__ col, long long n, long long rows,
                                 long long* __restrict__ rp, int* __restrict__ irregular) {
    bool bad = false;
    for (long long u0 = 4 * (blockIdx.x * (long long)blockDim.x + threadIdx.x); u0 < n;
         u0 += 4 * (long long)gridDim.x * blockDim.x) {
        int k[5], c[5];
        k[0] = u0 == 0 ? -1 : __ldg(key + u0 - 1);
        c[0] = u0 == 0 ? -1 : __ldg(col + u0 - 1);
        if (u0 + 4 <= n) {
            const int4 k4 = __ldg(reinterpret_cast<const int4*>(key + u0)), c4 = __ldg(reinterpret_cast<const int4*>(col + u0));
            k[1] = k4.x, k[2] = k4.y, k[3] = k4.z, k[4] = k4.w;
            c[1] = c4.x, c[2] = c4.y, c[3] = c4.z, c[4] = c4.w;
        } else {
            for (int i = 1; i <= 4; ++i) {
                k[i] = u0 + i - 1 < n ? key[u0 + i - 1] : -1;
                c[i] = u0 + i - 1 < n ? col[u0 + i - 1] : -1;
            }
        }
#pragma unroll
        for (int i = 1; i <= 4; ++i) {
            const long long u = u0 + i - 1, r = k[i], prev = k[i - 1];
            if (u >= n) break;
            if (r < 0 || r >= rows || prev >= rows || (u > 0 && (prev < 0 || (prev == r && c[i - 1] == c[i])))) {
                bad = true;
                continue;
            }
            for (long long q = prev + 1; q <= r; ++q) rp[q] = u;
            if (u == n - 1)
                for (long long q = r + 1; q <= rows; ++q) rp[q] = n;
        }
    }
    if (bad) *irregular = 1;
}

unsigned tr_blocks(long long work) {
    return (unsigned)std::max<long long>(1, std::min<long long>((work + 255) / 256, 152LL * 16));
}

}  // namespace

int build_transpose(const DevCsr& A, DevCsr* T, cudaStream_t st) {
    ST_CHECK(A.rows < (1ll << 31), ST_ERR_ARG, "rows must fit int32 to transpose");
    ST_CHECK(A.cols >= 0 && A.cols < (1ll << 31), ST_ERR_ARG, "columns must fit int32 indices");
    ST_CHECK(A.nnz < (1ll << 32), ST_ERR_ARG, "at most 2^32-1 entries per transpose");
    // the entries the row pointers cover (a handle made with a count of zero entries has none)
    long long n = 0;
    ST_CUDA(cudaMemcpyAsync(&n, A.row_ptr + A.rows, sizeof(n), cudaMemcpyDeviceToHost, st));
    ST_CUDA(cudaStreamSynchronize(st));
    n = std::max<long long>(0, std::min(n, A.nnz));
    DevCsr out;
    out.rows = A.cols;
    out.cols = A.rows;
    out.nnz = n;
    struct Checks {
        int irregular = 0;
        UnevenRows rows;
    };
    int irregular = 0;
    auto expand = [&](int* rowidx) -> int {
        if (n >= 12 * A.rows) tr_rows_kernel<32><<<tr_blocks(A.rows * 32), 256, 0, st>>>(A.row_ptr, A.rows, rowidx);
        else tr_rows_kernel<4><<<tr_blocks(A.rows * 4), 256, 0, st>>>(A.row_ptr, A.rows, rowidx);
        count_launch();
        ST_CUDA(cudaGetLastError());
        return ST_OK;
    };
    auto build = [&]() -> int {
        ST_CUDA(cudaMalloc(&out.row_ptr, (size_t)(A.cols + 1) * sizeof(long long)));
        if (n == 0) {
            ST_CUDA(cudaMemsetAsync(out.row_ptr, 0, (size_t)(A.cols + 1) * sizeof(long long), st));
            return ST_OK;
        }
        ST_CUDA(cudaMalloc(&out.col, (size_t)n * sizeof(int)));
        ST_CUDA(cudaMalloc(&out.val, (size_t)n * sizeof(float)));
        int bits = 1;
        while (bits < 31 && (1ll << bits) < A.cols) ++bits;
        const int passes = (bits + TR_BITS - 1) / TR_BITS;
        const int digit = (bits + passes - 1) / passes;
        const int bins = 1 << digit;
        int dev = 0, nsm = 0;
        ST_CUDA(cudaGetDevice(&dev));
        ST_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
        const long long tiles = (n + TR_TILE - 1) / TR_TILE;
        const long long ctas = std::min<long long>(tiles, (long long)std::max(nsm, 1) * TR_CTAS_PER_SM);
        const long long range = (tiles + ctas - 1) / ctas * TR_TILE;
        const unsigned grid = (unsigned)((n + range - 1) / range);
        const long long hn = (long long)bins * grid;
        DeviceBuffers bufs;
        auto* rowidx = static_cast<int*>(bufs.get((size_t)n * 4));  // the rows, then the last pass's keys
        auto* hist = static_cast<long long*>(bufs.get((size_t)hn * 8 + sizeof(Checks)));  // the checks behind it
        auto* offs = static_cast<long long*>(bufs.get((size_t)hn * 8));
        void* stmp = bufs.get(scan_tmp_bytes(hn));
        if (!rowidx || !hist || !offs || !stmp) return bufs.fail();
        auto* found = reinterpret_cast<Checks*>(hist + hn);
        ST_CUDA(cudaMemsetAsync(found, 0, sizeof(Checks), st));
        int* bk[2] = {nullptr, nullptr};
        int* br[2] = {nullptr, nullptr};
        float* bv[2] = {nullptr, nullptr};
        for (int p = 0; p < std::min(passes - 1, 2); ++p) {
            bk[p] = static_cast<int*>(bufs.get((size_t)n * 4));
            br[p] = static_cast<int*>(bufs.get((size_t)n * 4));
            bv[p] = static_cast<float*>(bufs.get((size_t)n * 4));
            if (!bk[p] || !br[p] || !bv[p]) return bufs.fail();
        }
        ST_TRY(expand(rowidx));
        ST_CUDA(cudaFuncSetAttribute(tr_scatter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(TrSmem)));
        const int* ik = A.col;
        const int* ir = rowidx;
        const float* iv = A.val;
        // the last pass's keys go over the rows once those have been read (two passes or more)
        int* keys = passes > 1 ? rowidx : static_cast<int*>(bufs.get((size_t)n * 4));
        if (!keys) return bufs.fail();
        for (int p = 0; p < passes; ++p) {
            const bool last = p == passes - 1;
            tr_hist_kernel<<<grid, TR_THREADS, 0, st>>>(ik, n, range, p * digit, bins, hist);
            count_launch();
            ST_CUDA(cudaGetLastError());
            ST_TRY(exclusive_scan_i64(hist, offs, hn, nullptr, stmp, st));
            int* ok = last ? keys : bk[p & 1];
            int* orw = last ? out.col : br[p & 1];
            float* ov = last ? out.val : bv[p & 1];
            tr_scatter_kernel<<<grid, TR_THREADS, sizeof(TrSmem), st>>>(ik, ir, iv, n, range, p * digit, bins, offs, ok,
                                                                        orw, ov);
            count_launch();
            ST_CUDA(cudaGetLastError());
            ik = ok;
            ir = orw;
            iv = ov;
        }
        tr_rowptr_kernel<<<tr_blocks(n), 256, 0, st>>>(keys, out.col, n, A.cols, out.row_ptr, &found->irregular);
        count_launch();
        ST_CUDA(cudaGetLastError());
        ST_TRY(measure_rows(out, &found->rows, nullptr, st));
        Checks h;
        ST_CUDA(cudaMemcpyAsync(&h, found, sizeof(h), cudaMemcpyDeviceToHost, st));
        ST_CUDA(cudaStreamSynchronize(st));
        irregular = h.irregular;
        out.lanes = lanes_of(out, h.rows);
        return ST_OK;
    };
    auto build_sorted = [&]() -> int {
        DeviceBuffers bufs;
        auto* rowidx = static_cast<int*>(bufs.get((size_t)n * 4));
        if (!rowidx) return bufs.fail();
        ST_TRY(expand(rowidx));
        ST_TRY((build_csr<int, float>(A.cols, A.rows, n, A.col, rowidx, A.val, false, &out, st)));
        ST_CUDA(cudaStreamSynchronize(st));
        return ST_OK;
    };
    int rc = build();
    if (rc == ST_OK && irregular) {
        out.release();
        rc = build_sorted();
    }
    if (rc < 0) {
        cudaStreamSynchronize(st);
        out.release();
        return rc;
    }
    *T = out;
    return ST_OK;
}

}  // namespace stg
