// CSR sparse path on the GPU: the triplet -> CSR builder of
// CSRMatrix::build_from_triplets (sparse/csr_matrix.cpp:25-72), the 7-point
// FD stencil matrix (:74-116), SpMV / SpMV^T (:118-166), scale,
// add_diagonal, Frobenius norm (:168-193), and the Krylov solvers of
// SparseOps (sparse/sparse_ops.cpp:8-113) -- plain CG, Jacobi-PCG and the
// damped normal-equation solve of the tomography system -- with FP32
// vectors and matrix values, int32 column indices, int64 row pointers, and
// every inner product, residual norm and step scalar on the device in FP64 or,
// with no fewer bits, in triples of FP32 values folded into FP64 (TripleSum).
#include "st_sort.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <initializer_list>
#include <memory>
#include <vector>

#include "st_sparse.cuh"
#include "st_update.cuh"

#include <cstdlib>

namespace stg {
namespace {

constexpr unsigned FULL = 0xffffffffu;

int bits_for(long long v) {
    int b = 0;
    while (b < 63 && (1ll << b) <= v) ++b;
    return std::max(b, 1);
}

int grid_cap() {
    static int n = 0;
    if (!n) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        n = std::max(n, 1);
    }
    return n * 16;
}

unsigned blocks_for(long long work, int threads = 256) {
    long long b = (work + threads - 1) / threads;
    return (unsigned)std::max<long long>(1, std::min<long long>(b, grid_cap()));
}

// The CG vector kernels: four CTAs per SM (each thread a few elements), so
// that their per-thread FP64 partial sums and block reductions stay small.
unsigned cg_blocks(long long work) {
    long long b = (work + 255) / 256;
    return (unsigned)std::max<long long>(1, std::min<long long>(b, grid_cap() / 4));
}

// ---------------------------------------------------------------- builder kernels
template <class TI>
__global__ void keys_kernel(const TI* __restrict__ r, const TI* __restrict__ c, long long n, long long R, long long Cc,
                            int cb, unsigned long long* __restrict__ keys, unsigned* __restrict__ pay) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const long long rr = (long long)r[i], cc = (long long)c[i];
        const bool ok = rr >= 0 && rr < R && cc >= 0 && cc < Cc;
        keys[i] = ok ? (((unsigned long long)rr << cb) | (unsigned long long)cc) : ((unsigned long long)R << cb);
        pay[i] = (unsigned)i;
    }
}

__global__ void heads_kernel(const unsigned long long* __restrict__ keys, long long n, long long R, int cb,
                             long long* __restrict__ flag) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const unsigned long long k = keys[i];
        const bool valid = (long long)(k >> cb) < R;
        flag[i] = (valid && (i == 0 || keys[i - 1] != k)) ? 1 : 0;
    }
}

// One thread per run of equal keys: sums the duplicates in input order (FP64).
template <class TV>
__global__ void merge_kernel(const unsigned long long* __restrict__ keys, const unsigned* __restrict__ pay, long long n,
                             int cb, const long long* __restrict__ flag, const long long* __restrict__ uidx,
                             const TV* __restrict__ v_in, int* __restrict__ col_out, float* __restrict__ val_out,
                             long long* __restrict__ urow) {
    const unsigned long long cmask = (1ull << cb) - 1;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        if (!flag[i]) continue;
        const unsigned long long k = keys[i];
        long long j = i + 1;
        while (j < n && keys[j] == k) ++j;
        double sum = 0.0;
        if (j - i == 1) {
            sum = (double)v_in[pay[i]];
        } else {
            // visit the run's input positions in increasing order
            unsigned last = 0;
            bool first = true;
            for (long long m = i; m < j; ++m) {
                unsigned best = 0xffffffffu;
                for (long long q = i; q < j; ++q) {
                    const unsigned p = pay[q];
                    if ((first || p > last) && p < best) best = p;
                }
                sum += (double)v_in[best];
                last = best;
                first = false;
            }
        }
        const long long u = uidx[i];
        col_out[u] = (int)(k & cmask);
        val_out[u] = (float)sum;
        urow[u] = (long long)(k >> cb);
    }
}

__global__ void rowptr_kernel(const long long* __restrict__ urow, long long nnz, long long R,
                              long long* __restrict__ rp) {
    for (long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x; u < nnz; u += (long long)gridDim.x * blockDim.x) {
        const long long r = urow[u];
        const long long prev = u == 0 ? -1 : urow[u - 1];
        for (long long q = prev + 1; q <= r; ++q) rp[q] = u;
        if (u == nnz - 1)
            for (long long q = r + 1; q <= R; ++q) rp[q] = nnz;
    }
}

// pad_to_alignment trigger (csr_matrix.cpp:223-264): a row i with
// roundup8(row_ptr[i]) > row_ptr[i+1].
__global__ void pad_trigger_kernel(const long long* __restrict__ rp, long long R, int* __restrict__ trig) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < R; i += (long long)gridDim.x * blockDim.x)
        if (((rp[i] + 7) / 8) * 8 > rp[i + 1]) atomicOr(trig, 1);
}

__global__ void pad_len_kernel(const long long* __restrict__ rp, long long R, long long* __restrict__ plen) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < R; i += (long long)gridDim.x * blockDim.x)
        plen[i] = ((rp[i + 1] - rp[i] + 7) / 8) * 8;
}

__global__ void pad_scatter_kernel(const long long* __restrict__ rp, const int* __restrict__ col,
                                   const float* __restrict__ val, long long R, const long long* __restrict__ nrp,
                                   int* __restrict__ ncol, float* __restrict__ nval) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < R; i += (long long)gridDim.x * blockDim.x) {
        const long long a = rp[i], len = rp[i + 1] - a, o = nrp[i], plen = nrp[i + 1] - o;
        for (long long k = 0; k < len; ++k) {
            ncol[o + k] = col[a + k];
            nval[o + k] = val[a + k];
        }
        for (long long k = len; k < plen; ++k) {
            ncol[o + k] = (int)i;
            nval[o + k] = 0.0f;
        }
    }
}

__global__ void fill_last_kernel(long long* rp, long long R, const long long* total) { rp[R] = *total; }

// A sum of products held as an unevaluated triple of FP32 values (the three-fold
// sum of Ogita, Rump and Oishi, "Accurate sum and dot product", 2005): the products
// are split exactly by FMA, the rounding errors of the leading sum and of the sum
// of those errors are kept, and only the third part is rounded. n products lose at
// most about (n 2^-24)^3 of the sum of their magnitudes, a chain of FP64 additions
// n 2^-53, so up to TRIPLE_MAX products (2^-48) the triple is no less precise than
// FP64. The FP64 pipe takes a warp's operation in 16 cycles here (conversions
// too), the FP32 one in a quarter of a cycle. Only for factors that triple_safe
// admits: zero or 2^-50 .. 2^50, so that no error term underflows and 2^27
// products stay below 2^128; the callers take FP64 sums otherwise (tiny values,
// infinities, NaN).
constexpr int TRIPLE_MAX = 256;
__device__ __forceinline__ bool triple_safe(float a) {
    const unsigned m = __float_as_uint(a) & 0x7fffffffu;
    return (m - 0x26800000u <= 0x58800000u - 0x26800000u) | (m == 0u);
}
// a + b = s + returned error, exactly.
__device__ __forceinline__ float two_sum(float a, float b, float& s) {
    s = __fadd_rn(a, b);
    const float z = __fsub_rn(s, a);
    return __fadd_rn(__fsub_rn(a, __fsub_rn(s, z)), __fsub_rn(b, z));
}
struct TripleSum {
    float h = 0.0f, m = 0.0f, l = 0.0f;
    __device__ __forceinline__ void add(float a, float b) {
        const float p = __fmul_rn(a, b);
        const float e = two_sum(h, p, h), f = two_sum(m, __fmaf_rn(a, b, -p), m), g = two_sum(m, e, m);
        l = __fadd_rn(l, __fadd_rn(f, g));
    }
    __device__ __forceinline__ void merge(const TripleSum& t) {
        const float e = two_sum(h, t.h, h), f = two_sum(m, t.m, m), g = two_sum(m, e, m);
        l = __fadd_rn(__fadd_rn(l, t.l), __fadd_rn(f, g));
    }
    __device__ __forceinline__ double value() const { return (double)h + ((double)m + (double)l); }
};
// Two of them, an instruction for both.
__device__ __forceinline__ F2 two_sum(F2 a, F2 b, F2& s) {
    const F2 n1 = pack(-1.0f, -1.0f), t = add2(a, b), z = fma2(n1, a, t);
    s = t;
    return add2(fma2(n1, fma2(n1, z, t), a), fma2(n1, z, b));
}
struct TripleSum2 {
    F2 h{0}, m{0}, l{0};
    __device__ __forceinline__ void add_squares(F2 a) {
        const F2 p = mul2(a, a), e = two_sum(h, p, h), f = two_sum(m, fma2(a, a, fma2(p, pack(-1.0f, -1.0f), F2{0})), m),
                 g = two_sum(m, e, m);
        l = add2(l, add2(f, g));
    }
    __device__ __forceinline__ TripleSum half(int k) const {
        TripleSum a, b;
        unpack(h, a.h, b.h);
        unpack(m, a.m, b.m);
        unpack(l, a.l, b.l);
        return k ? b : a;
    }
};

// ---------------------------------------------------------------- SpMV
// y[row] = sum val*x[col] with G threads per row (FP32 accumulation, a
// G-way strided partial sum per row reduced by shuffles), optional
// y += add_scale * add and FP64 accumulation of dot(pdot, y).
// Each lane loads the column and value of up to K of its row's entries at a
// time (coalesced), then issues all K gathers of x before it sums: the gathers,
// which wait on L2, are all in flight at once. The rest of a longer row follows
// in more such turns (TURNS: rows of 256 entries and more on average, some of
// thousands) or one entry at a time (shorter rows: a second turn, mostly empty,
// measured 0.655 ms against 0.561 with 16 lanes on rows of 180). PF: the group pulls the columns and values of the row
// it takes two rows on into L2. Resident CTAs per SM are pinned (six at 40
// registers, five at 48 for the 10-entry variant): the gathers need the warps.
template <int G, int K, bool PF, bool TURNS>
__global__ void __launch_bounds__(256, K >= 10 ? 5 : 6) spmv_kernel(const long long* __restrict__ rp, const int* __restrict__ col,
                                                   const float* __restrict__ val, const float* __restrict__ x,
                                                   float* __restrict__ y, long long rows, const float* __restrict__ add,
                                                   float add_scale, const float* __restrict__ pdot,
                                                   double* __restrict__ dot_acc, const int* __restrict__ done) {
    if (done && *done) return;
    __shared__ double red[8];
    const int lane = threadIdx.x % G;
    const long long gid = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / G;
    const long long stride = ((long long)gridDim.x * blockDim.x) / G;
    // the warp's first group: every lane of a warp runs the same number of
    // iterations (groups past the last row idle through them), so the
    // full-warp shuffles below always see all 32 lanes
    const long long gfirst = (blockIdx.x * (long long)blockDim.x + (threadIdx.x & ~31u)) / G;
    double local = 0.0;
    constexpr long long PFR = 2;  // rows ahead
    for (long long it = 0; gfirst + it * stride < rows; ++it) {
        const long long row = gid + it * stride;
        const bool active = row < rows;
        const long long a = active ? rp[row] : 0, b = active ? rp[row + 1] : 0;
        if (PF && active && row + PFR * stride < rows) {
            const long long na = rp[row + PFR * stride], nb = rp[row + PFR * stride + 1];
            const long long l0 = na >> 5, l1 = (nb + 31) >> 5;  // 32 four-byte entries per line
            for (long long l = l0 + lane; l < l1; l += G) {
                const long long e = l << 5;
                asm volatile("prefetch.global.L2 [%0];" ::"l"(col + e));
                asm volatile("prefetch.global.L2 [%0];" ::"l"(val + e));
            }
        }
        float s0 = 0.0f, s1 = 0.0f;
        auto turn = [&](long long q) {
            int cs[K];
            float vs[K], xs[K];
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const long long e = q + lane + (long long)k * G;
                cs[k] = e < b ? __ldg(col + e) : 0;
                vs[k] = e < b ? __ldg(val + e) : 0.0f;
            }
#pragma unroll
            for (int k = 0; k < K; ++k) xs[k] = (q + lane + (long long)k * G < b) ? __ldg(x + cs[k]) : 0.0f;
#pragma unroll
            for (int k = 0; k < K; k += 2) {
                s0 = fmaf(vs[k], xs[k], s0);
                if (k + 1 < K) s1 = fmaf(vs[k + 1], xs[k + 1], s1);
            }
        };
        if (TURNS) {
            for (long long q = a; q < b; q += (long long)K * G) turn(q);
        } else {
            turn(a);
            for (long long p = a + lane + (long long)K * G; p < b; p += G)
                s0 = fmaf(__ldg(val + p), __ldg(x + __ldg(col + p)), s0);
        }
        float sum = s0 + s1;
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(FULL, sum, o, G);
        if (lane == 0 && active) {
            if (add) sum = fmaf(add_scale, add[row], sum);
            y[row] = sum;
            if (pdot) local += (double)pdot[row] * (double)sum;
        }
    }
    if (dot_acc) {
        // only the groups' first lanes hold row products: fold those of the
        // warp (none to fold for one group per warp), then the block's warps,
        // into one of the accumulator's CG_SLOTS addresses
        for (int o = 16; o >= G; o >>= 1) local += __shfl_xor_sync(FULL, local, o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = local;
        __syncthreads();
        if (threadIdx.x == 0) {
            double t = 0.0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
            atomicAdd(dot_acc + blockIdx.x % CG_SLOTS, t);
        }
    }
}

__device__ __forceinline__ void copy16_async(void* dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}

// Short rows (fewer than ten entries on average): a CTA takes 128 consecutive
// rows at a time, copies their columns and values to shared memory as a stream of
// 16-byte pieces (whatever row they belong to), and every thread then works
// through its own row there. Neighbouring rows gather neighbouring x, so a warp's
// gather is a line or two; multiplied along the stream a gather met all the offsets
// of a row, seven lines, and the L1 set the pace. A group of lanes per row spends
// most of its instructions on predicates and waits for the row pointers, the
// columns and the gathers one after another for 28 bytes of values. A tile with
// more entries than fit in shared memory is summed a warp per row; matrices with much
// of their entries in such tiles, or in tiles with a long row that one thread works
// through, go to a group of lanes per row (lanes_of).
// 7 entries per row on a 256^3 grid, 72 bytes per row: 192 us a product (a copy of
// the bytes takes 178); products along the stream 244, four lanes per row 600. 40
// CG iterations there with tiles of 256 / 128 / 64 rows 24.3 / 23.5 / 23.3 ms
// (smaller tiles overflow more easily), a tile per warp 25.9 (spills), two tiles in
// turn at fewer warps per SM 28.0.
constexpr int SR_ROWS = 128;
constexpr int SR_CAP = 1408;  // entries of a tile (11 per row): 11 KB, sixteen CTAs per SM
constexpr int SR_LONG = 32;   // a longer row makes its tile wait for the thread that has it
constexpr long long SHORT_ROWS = 10;
template <bool SPLIT>
__global__ void __launch_bounds__(SR_ROWS, 16) spmv_rows_kernel(const long long* __restrict__ rp, const int* __restrict__ col,
                                                              const float* __restrict__ val,
                                                              const float* __restrict__ x, float* __restrict__ y,
                                                              long long rows,
                                                              const float* __restrict__ add, float add_scale,
                                                              const float* __restrict__ pdot,
                                                              double* __restrict__ dot_acc,
                                                              const int* __restrict__ done) {
    if (done && *done) return;
    __shared__ __align__(16) int scol[SR_CAP + 8];
    __shared__ __align__(16) float sval[SR_CAP + 8];
    __shared__ double red[SR_ROWS / 32];
    const int tid = threadIdx.x;
    double local = 0.0;
    for (long long r0 = (long long)blockIdx.x * SR_ROWS; r0 < rows; r0 += (long long)gridDim.x * SR_ROWS) {
        const long long row = r0 + tid;
        const bool active = row < rows;
        const long long rlast = min(r0 + SR_ROWS, rows);
        const long long e0 = rp[r0], e1 = rp[rlast];
        const long long base = e0 & ~3ll;  // 16-byte aligned start of the tile's entries
        const long long a = active ? rp[row] : 0, b = active ? rp[row + 1] : 0;
        float sum = 0.0f;
        if (e1 - base <= SR_CAP) {
            const int m = (int)(e1 - base);
            for (int k = 4 * tid; k < m; k += 4 * SR_ROWS) {
                const int bytes = min(16, 4 * (m - k));
                copy16_async(scol + k, col + base + k, bytes);
                copy16_async(sval + k, val + base + k, bytes);
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            // four strided partial sums; SPLIT: each in two parts, its second and fourth
            // entry in the other one (the shorter chains of four lanes per row)
            float t[4] = {0.0f, 0.0f, 0.0f, 0.0f}, u[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            const int kb = (int)(b - base);
            int k = (int)(a - base);
            // eight gathers in flight (the rows of a 7-point stencil): 256^3 192 us, four at a time 195
            float xs[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) xs[i] = k + i < kb ? __ldg(x + scol[k + i]) : 0.0f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (k + i < kb) t[i] = fmaf(sval[k + i], xs[i], 0.0f);
                if (SPLIT && k + 4 + i < kb) u[i] = fmaf(sval[k + 4 + i], xs[4 + i], 0.0f);
                if (!SPLIT && k + 4 + i < kb) t[i] = fmaf(sval[k + 4 + i], xs[4 + i], t[i]);
            }
            k += 8;
            for (int j = 2; k < kb; k += 4, ++j) {
#pragma unroll
                for (int i = 0; i < 4; ++i) xs[i] = k + i < kb ? __ldg(x + scol[k + i]) : 0.0f;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float& part = SPLIT && j == 3 ? u[i] : t[i];
                    if (k + i < kb) part = fmaf(sval[k + i], xs[i], part);
                }
            }
            sum = ((t[0] + u[0]) + (t[2] + u[2])) + ((t[1] + u[1]) + (t[3] + u[3]));
            __syncthreads();
        } else {
            const int lane = tid & 31;
            for (int w = 0; w < 32; ++w) {  // the warp's 32 rows, one after another
                const long long ra = __shfl_sync(FULL, a, w), rb = __shfl_sync(FULL, b, w);
                float s = 0.0f;
                for (long long e = ra + lane; e < rb; e += 32) s = fmaf(__ldg(val + e), __ldg(x + __ldg(col + e)), s);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
                if (lane == w) sum = s;
            }
        }
        if (active) {
            if (add) sum = fmaf(add_scale, add[row], sum);
            y[row] = sum;
            if (pdot) local += (double)pdot[row] * (double)sum;
        }
    }
    if (dot_acc) {
        for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(FULL, local, o);
        if ((tid & 31) == 0) red[tid >> 5] = local;
        __syncthreads();
        if (tid == 0) {
            double t = 0.0;
            for (int w = 0; w < SR_ROWS / 32; ++w) t += red[w];
            atomicAdd(dot_acc + blockIdx.x % CG_SLOTS, t);
        }
    }
}

int launch_spmv_rows(const DevCsr& A, const float* x, float* y, const float* add, float add_scale, const float* pdot,
                     double* dot_acc, const int* done, cudaStream_t st) {
    const long long tiles = (A.rows + SR_ROWS - 1) / SR_ROWS;
    const unsigned blocks = (unsigned)std::max<long long>(1, std::min<long long>(tiles, grid_cap()));  // 16 per SM
    const auto kernel = A.nnz >= 5 * A.rows ? spmv_rows_kernel<true> : spmv_rows_kernel<false>;
    kernel<<<blocks, SR_ROWS, 0, st>>>(A.row_ptr, A.col, A.val, x, y, A.rows, add, add_scale, pdot, dot_acc, done);
    count_launch();
    ST_CUDA(cudaGetLastError());
    return ST_OK;
}

template <int G, int K, bool PF, bool TURNS>
int launch_spmv_g(const DevCsr& A, const float* x, float* y, const float* add, float add_scale, const float* pdot,
                  double* dot_acc, const int* done, cudaStream_t st) {
    // up to 64 CTAs of 256 threads per SM, the rest by the grid-stride loop
    // (measured on the 2M-ray matrix: 16 per SM 0.58 ms, 32 0.56, 64 0.54 for A x)
    const long long b = (A.rows * G + 255) / 256;
    const unsigned blocks = (unsigned)std::max<long long>(1, std::min<long long>(b, (long long)grid_cap() * 4));
    spmv_kernel<G, K, PF, TURNS><<<blocks, 256, 0, st>>>(A.row_ptr, A.col, A.val, x, y, A.rows, add, add_scale, pdot, dot_acc,
                                                  done);
    count_launch();
    ST_CUDA(cudaGetLastError());
    return ST_OK;
}

// ---------------------------------------------------------------- vectors / CG
__global__ void f64_to_f32_kernel(const double* a, float* b, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        b[i] = (float)a[i];
}
__global__ void f32_to_f64_kernel(const float* a, double* b, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        b[i] = (double)a[i];
}

// Block sums of a and b added to acc_a / acc_b; slots > 1: into slot
// blockIdx % slots of each (the CG accumulators).
__device__ __forceinline__ void block_add2(double a, double b, double* acc_a, double* acc_b, int slots = 1) {
    __shared__ double ra[8], rb[8];
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(FULL, a, o);
        b += __shfl_xor_sync(FULL, b, o);
    }
    if ((threadIdx.x & 31) == 0) {
        ra[threadIdx.x >> 5] = a;
        rb[threadIdx.x >> 5] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double ta = 0.0, tb = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            ta += ra[w];
            tb += rb[w];
        }
        if (acc_a) atomicAdd(acc_a + blockIdx.x % slots, ta);
        if (acc_b) atomicAdd(acc_b + blockIdx.x % slots, tb);
    }
}

// r = b, z = M r, p = z, x = 0; acc rz = <r,z>, bb = <b,b>.
__global__ void cg_init_kernel(const float* __restrict__ b, const float* __restrict__ dinv, long long n,
                               float* __restrict__ x, float* __restrict__ r, float* __restrict__ z,
                               float* __restrict__ p, double* rz, double* bb) {
    double a = 0.0, c = 0.0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float bi = b[i];
        const float zi = dinv ? dinv[i] * bi : bi;
        x[i] = 0.0f;
        r[i] = bi;
        if (z) z[i] = zi;
        p[i] = zi;
        a += (double)bi * (double)zi;
        c += (double)bi * (double)bi;
    }
    block_add2(a, c, rz, bb, CG_SLOTS);
}

// Whether every given pointer (null ones aside) may be read as 16-byte quads.
inline bool quads_ok(std::initializer_list<const void*> ps) {
    for (const void* p : ps)
        if (reinterpret_cast<uintptr_t>(p) & 15) return false;
    return true;
}

// x += alpha p, r -= alpha q, z = M r; acc rz_new = <r,z>, rr = <r,r>.
// Bound by memory (8 words per unknown): read and written
// four unknowns at a time where the caller's x allows it (quads), so that a
// thread has five 16-byte loads in flight, with the inner products carried in
// triples of FP32 values over the thread's quads. 16.8M unknowns: 83 us (a copy of
// the bytes takes 79), 146 with FP64 products, 169 with single words as well.
// alpha = rz_old / pq; |pq| < 1e-30 stops the solve (sparse_ops.cpp:37,88).
// The scalars are formed once per block (FP64 is a slow pipe on this GPU).
// skip_rz: <r, z> comes from the stencil preconditioner's kernel instead.
__global__ void cg_update_kernel(long long n, float* __restrict__ x, float* __restrict__ r, float* __restrict__ z,
                                 const float* __restrict__ p, const float* __restrict__ q,
                                 const float* __restrict__ dinv, CgScalars* sc, int k, int skip_rz, int quads) {
    __shared__ float s_alpha;
    __shared__ int s_stop;
    if (threadIdx.x == 0) {
        int stop = sc->done;
        float alpha = 0.0f;
        if (!stop) {
            const double pq = cg_slot_sum(sc->acc[k % 3].pq);
            if (fabs(pq) < 1e-30) {
                stop = 1;
                if (blockIdx.x == 0) {
                    sc->done = 1;
                    sc->breakdown = 1;
                }
            } else {
                alpha = (float)(cg_slot_sum(sc->acc[(k + 2) % 3].rzn) / pq);
            }
        }
        s_alpha = alpha;
        s_stop = stop;
    }
    __syncthreads();
    if (s_stop) return;
    const float alpha = s_alpha;
    double a = 0.0, c = 0.0;
    TripleSum rz, rr;
    int held = 0;  // products in each triple
    const long long n4 = quads ? n >> 2 : 0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
        const float4 p4 = reinterpret_cast<const float4*>(p)[i], q4 = reinterpret_cast<const float4*>(q)[i];
        float4 x4 = reinterpret_cast<float4*>(x)[i], r4 = reinterpret_cast<float4*>(r)[i];
        float4 d4 = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
        if (dinv) d4 = reinterpret_cast<const float4*>(dinv)[i];
        x4 = make_float4(fmaf(alpha, p4.x, x4.x), fmaf(alpha, p4.y, x4.y), fmaf(alpha, p4.z, x4.z), fmaf(alpha, p4.w, x4.w));
        r4 = make_float4(fmaf(-alpha, q4.x, r4.x), fmaf(-alpha, q4.y, r4.y), fmaf(-alpha, q4.z, r4.z),
                         fmaf(-alpha, q4.w, r4.w));
        const float4 z4 = make_float4(d4.x * r4.x, d4.y * r4.y, d4.z * r4.z, d4.w * r4.w);
        reinterpret_cast<float4*>(x)[i] = x4;
        reinterpret_cast<float4*>(r)[i] = r4;
        if (z) reinterpret_cast<float4*>(z)[i] = z4;
        const bool safe = triple_safe(r4.x) & triple_safe(r4.y) & triple_safe(r4.z) & triple_safe(r4.w) &
                          triple_safe(z4.x) & triple_safe(z4.y) & triple_safe(z4.z) & triple_safe(z4.w);
        if (!safe) {
            const double r0 = r4.x, r1 = r4.y, r2 = r4.z, r3 = r4.w;
            a += (r0 * (double)z4.x + r1 * (double)z4.y) + (r2 * (double)z4.z + r3 * (double)z4.w);
            c += (r0 * r0 + r1 * r1) + (r2 * r2 + r3 * r3);
            continue;
        }
        rz.add(r4.x, z4.x);
        rz.add(r4.y, z4.y);
        rz.add(r4.z, z4.z);
        rz.add(r4.w, z4.w);
        rr.add(r4.x, r4.x);
        rr.add(r4.y, r4.y);
        rr.add(r4.z, r4.z);
        rr.add(r4.w, r4.w);
        if ((held += 4) == TRIPLE_MAX) {
            a += rz.value();
            c += rr.value();
            rz = rr = TripleSum();
            held = 0;
        }
    }
    a += rz.value();
    c += rr.value();
    for (long long i = 4 * n4 + blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        x[i] = fmaf(alpha, p[i], x[i]);
        const float ri = fmaf(-alpha, q[i], r[i]);
        r[i] = ri;
        const float zi = dinv ? dinv[i] * ri : ri;
        if (z) z[i] = zi;
        a += (double)ri * (double)zi;
        c += (double)ri * (double)ri;
    }
    block_add2(a, c, skip_rz ? nullptr : sc->acc[k % 3].rzn, sc->acc[k % 3].rr, CG_SLOTS);
}

// z = dinv r + S sum_a w_a (2 v - v(-e_a) - v(+e_a)), v = S r and 0 outside
// the grid (the weighted Dirichlet Laplacian between the two diagonal
// scalings: symmetric positive definite with dinv); acc += <r, z>; p = z when
// p is set (the first iteration).
__global__ void stencil_prec_kernel(long long n, const float* __restrict__ r, const float* __restrict__ dinv,
                                    const float* __restrict__ sq, int gx, int gy, int gz, float wx, float wy,
                                    float wz, float* __restrict__ z, float* __restrict__ p, double* acc,
                                    const int* done) {
    if (done && *done) return;
    const long long sy = gz, sx = (long long)gy * gz;
    double a = 0.0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int iz = (int)(i % gz);
        const long long t = i / gz;
        const int iy = (int)(t % gy), ix = (int)(t / gy);
        const float si = sq[i], ri = r[i], vi = si * ri;
        auto v = [&](long long j) { return sq[j] * r[j]; };
        const float lz = 2.0f * vi - (iz > 0 ? v(i - 1) : 0.0f) - (iz < gz - 1 ? v(i + 1) : 0.0f);
        const float ly = 2.0f * vi - (iy > 0 ? v(i - sy) : 0.0f) - (iy < gy - 1 ? v(i + sy) : 0.0f);
        const float lx = 2.0f * vi - (ix > 0 ? v(i - sx) : 0.0f) - (ix < gx - 1 ? v(i + sx) : 0.0f);
        const float zi = fmaf(dinv[i], ri, si * fmaf(wx, lx, fmaf(wy, ly, wz * lz)));
        z[i] = zi;
        if (p) p[i] = zi;
        a += (double)ri * (double)zi;
    }
    block_add2(a, 0.0, acc, nullptr, CG_SLOTS);
}

// Convergence test after the update (sqrt(rr)/||b|| < tol) and
// p = z + beta p with beta = rz_new / rz_old; clears the accumulators of
// iteration k+1.
__global__ void cg_pupdate_kernel(long long n, float* __restrict__ p, const float* __restrict__ z, CgScalars* sc,
                                  int k, double tol) {
    __shared__ float s_beta;
    __shared__ int s_stop;
    if (threadIdx.x == 0) {
        int stop = sc->done;
        float beta = 0.0f;
        if (!stop) {
            const double rel = sqrt(cg_slot_sum(sc->acc[k % 3].rr)) / sqrt(cg_slot_sum(sc->bb));
            if (blockIdx.x == 0) {
                sc->iters = k + 1;
                sc->rel = rel;
                CgAcc& nxt = sc->acc[(k + 1) % 3];
                for (int i = 0; i < CG_SLOTS; ++i) nxt.pq[i] = nxt.rr[i] = nxt.rzn[i] = 0.0;
            }
            if (rel < tol) {
                stop = 1;
                if (blockIdx.x == 0) sc->done = 1;
            } else {
                beta = (float)(cg_slot_sum(sc->acc[k % 3].rzn) / cg_slot_sum(sc->acc[(k + 2) % 3].rzn));
            }
        }
        s_beta = beta;
        s_stop = stop;
    }
    __syncthreads();
    if (s_stop) return;
    const float beta = s_beta;
    const long long n4 = n >> 2;  // p, z and r are the solver's own vectors: 16-byte aligned
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
        const float4 z4 = reinterpret_cast<const float4*>(z)[i];
        const float4 p4 = reinterpret_cast<float4*>(p)[i];
        reinterpret_cast<float4*>(p)[i] = make_float4(fmaf(beta, p4.x, z4.x), fmaf(beta, p4.y, z4.y),
                                                      fmaf(beta, p4.z, z4.z), fmaf(beta, p4.w, z4.w));
    }
    const long long i = 4 * n4 + blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i < n) p[i] = fmaf(beta, p[i], z[i]);
}

// Jacobi diagonal of sparse_ops.cpp:60-73: 1/A_ii from the first entry with
// col == row when |A_ii| > 1e-30, otherwise 1.
__global__ void jacobi_kernel(const long long* __restrict__ rp, const int* __restrict__ col,
                              const float* __restrict__ val, long long rows, float* __restrict__ dinv) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < rows; i += (long long)gridDim.x * blockDim.x) {
        float d = 1.0f;
        for (long long p = rp[i]; p < rp[i + 1]; ++p)
            if (col[p] == i) {
                if (fabsf(val[p]) > 1e-30f) d = 1.0f / val[p];
                break;
            }
        dinv[i] = d;
    }
}

// diag of A^T A + lam I from the rows of A^T: 1 / (sum_k AT[j,k]^2 + lam). G lanes
// per row, over its entries (coalesced); a group's rows lie a grid apart (neighbouring
// cells are heavy together: where rays meet, a row holds thousands of entries), and
// lane w keeps the sum of its w-th row, so that the FP64 division runs on full warps.
// Triples of FP32 values carry the squares, two to an instruction, and rows whose sum
// they cannot hold are summed again in FP64. Bound by the FP32 instructions and, where
// lengths differ, by the rows that take longest: groups of 8 and 16 join a row's sums in
// few steps for four or two rows at once, and four times the blocks that fit even the
// lengths out. 8 / 16 / 32 lanes, us: 262,144 rows of 40 entries 33 / 56 / 87 (47 a
// thread per row in FP64), of 202 68 / 88 / 128 (214); the cells of rays, mean 211 on
// 54^3 84 / 72 / 80, mean 361 on 100^3 482 / 465 / 511, with as many blocks as fit 108 /
// 84 / 80 and 487 / 466 / 565; means of 3000 from 2 to 20,000 45 / - / 17.
// Short rows (less than 24 entries on average) are staged through shared memory
// instead, a thread per row: 2M rows of 7 entries 58 us (85 in FP64).
// Rows beyond this many entries go to the whole warp.
__host__ __device__ constexpr int nj_far(int G) { return G == 8 ? 1024 : 4096; }

// This lane's squares among p[0 .. n), G lanes over them; full triples go to far. Two
// sums per instruction, joined at the end.
template <int G>
__device__ __forceinline__ void add_squares(const float* __restrict__ p, long long n, int lane, TripleSum& s,
                                            double& far) {
    int held = 0;
    TripleSum2 t;
    p += lane;
    for (; n - lane > 7 * G; n -= 8 * G, p += 8 * G) {
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = __ldg(p + G * k);
#pragma unroll
        for (int k = 0; k < 8; k += 2) t.add_squares(pack(v[k], v[k + 1]));
        if ((held += 4) == TRIPLE_MAX) {
            far += t.half(0).value() + t.half(1).value();
            t = TripleSum2();
            held = 0;
        }
    }
    const int m = (int)n - lane;
    float v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = G * k < m ? __ldg(p + G * k) : 0.0f;
#pragma unroll
    for (int k = 0; k < 8; k += 2)
        if (G * k < m) t.add_squares(pack(v[k], v[k + 1]));
    s = t.half(0);
    s.merge(t.half(1));
}

// Whether a sum of squares needs FP64: out of range on the way (infinite or NaN then),
// or so small that what the triples lose to underflow, 2^-149 a product, may count.
__device__ __forceinline__ bool squares_odd(float h, double far) {
    return !(h <= 0x1p120f) || (far == 0.0 ? !(h >= 0x1p-40f) : !(far >= 0x1p-40 && far <= 0x1p200));
}

template <int G>
__device__ __forceinline__ void merge_lanes(TripleSum& s, double& far) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
        TripleSum t;
        t.h = __shfl_xor_sync(FULL, s.h, o);
        t.m = __shfl_xor_sync(FULL, s.m, o);
        t.l = __shfl_xor_sync(FULL, s.l, o);
        s.merge(t);
    }
    if (__any_sync(FULL, far != 0.0)) {
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) far += __shfl_xor_sync(FULL, far, o);
    }
}

// The same sum in FP64.
template <int G>
__device__ __noinline__ double squares64(const float* __restrict__ val, long long a, long long b, int lane) {
    double t = 0.0;
    for (long long e = a + lane; e < b; e += G) t += (double)val[e] * (double)val[e];
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) t += __shfl_xor_sync(FULL, t, o);
    return t;
}

template <int G>
__global__ void __launch_bounds__(256, 4) normal_jacobi_kernel(const long long* __restrict__ rp,
                                                               const float* __restrict__ val, long long rows, double lam,
                                                               float* __restrict__ dinv) {
    const int lane = threadIdx.x % G, wl = threadIdx.x & 31;
    const long long groups = (long long)gridDim.x * (blockDim.x / G);
    const long long first = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / G;
    const int ahead = (wl - lane) / G;  // groups of the warp before this one
    for (long long r0 = first; r0 - ahead < rows; r0 += G * groups) {
        TripleSum mine;
        double mfar = 0.0;
        for (int w = 0; w < G && r0 - ahead + w * groups < rows; ++w) {
            const long long r = r0 + w * groups;
            const long long a = r < rows ? rp[r] : 0, b = r < rows ? rp[r + 1] : 0;
            const bool rest = G < 32 && b - a > nj_far(G);
            TripleSum s;
            double far = 0.0;
            add_squares<G>(val + a, rest ? 0 : b - a, lane, s, far);
            merge_lanes<G>(s, far);
            unsigned odd = __ballot_sync(FULL, b > a && !rest && squares_odd(s.h, far));
            if (odd) {
                const double t = squares64<G>(val, a, rest ? a : b, lane);
                if ((odd >> (wl - lane)) & (FULL >> (32 - G))) {
                    s = TripleSum();
                    far = t;
                }
            }
            if (lane == w) {
                mine = s;
                mfar = far;
            }
            if constexpr (G < 32) {
                for (unsigned m = __ballot_sync(FULL, rest && lane == 0); m; m &= m - 1) {
                    const int src = __ffs((int)m) - 1;
                    const long long fa = __shfl_sync(FULL, a, src), fb = __shfl_sync(FULL, b, src);
                    far = 0.0;
                    add_squares<32>(val + fa, fb - fa, wl, s, far);
                    merge_lanes<32>(s, far);
                    odd = __ballot_sync(FULL, squares_odd(s.h, far));
                    if (odd) {
                        s = TripleSum();
                        far = squares64<32>(val, fa, fb, wl);
                    }
                    if (wl == src + w) {
                        mine = s;
                        mfar = far;
                    }
                }
            }
        }
        const long long i = r0 + lane * groups;
        if (i < rows) dinv[i] = (float)(1.0 / (mfar + mine.value() + lam));
    }
}

constexpr int NJ_ROWS = 256;
__global__ void __launch_bounds__(NJ_ROWS) normal_jacobi_rows_kernel(const long long* __restrict__ rp,
                                                                     const float* __restrict__ val, long long rows,
                                                                     double lam, float* __restrict__ dinv) {
    constexpr int CAP = 24 * NJ_ROWS;
    __shared__ float v[CAP];
    for (long long r0 = (long long)blockIdx.x * NJ_ROWS; r0 < rows; r0 += (long long)gridDim.x * NJ_ROWS) {
        const long long i = r0 + threadIdx.x;
        const long long e0 = rp[r0], e1 = rp[min(r0 + NJ_ROWS, rows)];
        const long long a = i < rows ? rp[i] : 0, b = i < rows ? rp[i + 1] : 0;
        const bool staged = e1 - e0 <= CAP;
        if (staged)
            for (long long e = e0 + threadIdx.x; e < e1; e += NJ_ROWS) v[e - e0] = __ldg(val + e);
        __syncthreads();
        TripleSum2 s;
        double t = 0.0;
        bool safe = staged;
        if (staged) {
            const int kb = (int)(b - e0);
            int held = 0;
            for (int k = (int)(a - e0); k < kb; k += 2) {
                const float v0 = v[k], v1 = k + 1 < kb ? v[k + 1] : 0.0f;
                safe = safe & triple_safe(v0) & triple_safe(v1);
                s.add_squares(pack(v0, v1));
                if (++held == TRIPLE_MAX) {
                    t += s.half(0).value() + s.half(1).value();
                    s = TripleSum2();
                    held = 0;
                }
            }
            TripleSum both = s.half(0);
            both.merge(s.half(1));
            t += both.value();
        }
        if (!safe) {
            t = 0.0;
            for (long long e = a; e < b; ++e) t += (double)val[e] * (double)val[e];
        }
        if (i < rows) dinv[i] = (float)(1.0 / (t + lam));
        __syncthreads();
    }
}

__global__ void scale_kernel(float* v, long long n, float a) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        v[i] *= a;
}

__global__ void add_diag_kernel(const long long* __restrict__ rp, const int* __restrict__ col, float* __restrict__ val,
                                long long rows, float a) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < rows; i += (long long)gridDim.x * blockDim.x)
        for (long long p = rp[i]; p < rp[i + 1]; ++p)
            if (col[p] == i) {
                val[p] += a;
                break;
            }
}

__global__ void sumsq_kernel(const float* __restrict__ v, long long n, double* acc) {
    double a = 0.0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        a += (double)v[i] * (double)v[i];
    block_add2(a, 0.0, acc, nullptr);
}

__global__ void dot64_kernel(const double* __restrict__ a, const double* __restrict__ b, long long n, double* acc) {
    double s = 0.0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        s += a[i] * b[i];
    block_add2(s, 0.0, acc, nullptr);
}

__global__ void axpby_kernel(float* __restrict__ out, const float* __restrict__ a, const float* __restrict__ b,
                             float beta, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = a[i] - beta * b[i];
}

// 7-point stencil triplets of build_fd_stencil_7point (csr_matrix.cpp:74-116),
// emitted in the reference's per-row order, 7 slots per row (unused slots get
// an out-of-range row and are dropped by the builder).
__global__ void fd_triplets_kernel(const double* __restrict__ vel, long long nx, long long ny, long long nz, double idx2,
                                   double idy2, double idz2, double dt2, long long* __restrict__ tr,
                                   long long* __restrict__ tc, double* __restrict__ tv) {
    const long long n = nx * ny * nz;
    for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < n; r += (long long)gridDim.x * blockDim.x) {
        const long long ix = r / (ny * nz), rem = r % (ny * nz), iy = rem / nz, iz = rem % nz;
        const double v = vel[r];
        const double v2dt2 = v * v * dt2;
        const double diag = -2.0 * v2dt2 * (idx2 + idy2 + idz2) + 2.0;
        long long* rr = tr + 7 * r;
        long long* cc = tc + 7 * r;
        double* vv = tv + 7 * r;
        int k = 0;
        auto put = [&](bool ok, long long c, double val) {
            rr[k] = ok ? r : -1;
            cc[k] = ok ? c : 0;
            vv[k] = ok ? val : 0.0;
            ++k;
        };
        put(true, r, diag);
        put(ix > 0, r - ny * nz, v2dt2 * idx2);
        put(ix < nx - 1, r + ny * nz, v2dt2 * idx2);
        put(iy > 0, r - nz, v2dt2 * idy2);
        put(iy < ny - 1, r + nz, v2dt2 * idy2);
        put(iz > 0, r - 1, v2dt2 * idz2);
        put(iz < nz - 1, r + 1, v2dt2 * idz2);
    }
}

}  // namespace

// ---------------------------------------------------------------- builder (host side)

template <class TI, class TV>
int build_csr(long long rows, long long cols, long long n, const TI* r, const TI* c, const TV* v, bool pad,
              DevCsr* out, cudaStream_t st) {
    ST_CHECK(rows >= 0 && cols >= 0 && n >= 0, ST_ERR_ARG, "negative CSR extents");
    ST_CHECK(cols < (1ll << 31), ST_ERR_ARG, "columns must fit int32 indices");
    ST_CHECK(n < (1ll << 32), ST_ERR_ARG, "at most 2^32-1 triplets per build");
    const int cb = bits_for(cols);
    const int rb = bits_for(rows);  // rows itself (the drop marker) must be representable
    ST_CHECK(cb + rb <= 64, ST_ERR_ARG, "row/column index range too large");
    DeviceBuffers bufs;
    auto alloc = [&](size_t bytes) -> void* { return bufs.get(bytes); };
    ST_CUDA(cudaMalloc(&out->row_ptr, (size_t)(rows + 1) * sizeof(long long)));
    out->rows = rows;
    out->cols = cols;
    if (n == 0) {
        ST_CUDA(cudaMemsetAsync(out->row_ptr, 0, (size_t)(rows + 1) * sizeof(long long), st));
        out->nnz = 0;
        return ST_OK;
    }
    auto* keys = static_cast<unsigned long long*>(alloc((size_t)n * 8));
    auto* pay = static_cast<unsigned*>(alloc((size_t)n * 4));
    auto* keys2 = static_cast<unsigned long long*>(alloc((size_t)n * 8));
    auto* pay2 = static_cast<unsigned*>(alloc((size_t)n * 4));
    void* rtmp = alloc(radix_tmp_bytes(n));
    if (!keys || !pay || !keys2 || !pay2 || !rtmp) return bufs.fail();
    keys_kernel<TI><<<blocks_for(n), 256, 0, st>>>(r, c, n, rows, cols, cb, keys, pay);
    count_launch();
    ST_CUDA(cudaGetLastError());
    ST_TRY(radix_sort_u64(keys, pay, keys2, pay2, n, cb + rb, rtmp, st));
    // reuse keys2 / pay2 storage for the head flags and unique indices
    auto* flag = reinterpret_cast<long long*>(keys2);
    auto* uidx = static_cast<long long*>(alloc((size_t)n * 8));
    auto* total = static_cast<long long*>(alloc(64));
    void* stmp = alloc(scan_tmp_bytes(n));
    if (!uidx || !total || !stmp) return bufs.fail();
    heads_kernel<<<blocks_for(n), 256, 0, st>>>(keys, n, rows, cb, flag);
    count_launch();
    ST_CUDA(cudaGetLastError());
    ST_TRY(exclusive_scan_i64(flag, uidx, n, total, stmp, st));
    long long nnz = 0;
    ST_CUDA(cudaMemcpyAsync(&nnz, total, sizeof(long long), cudaMemcpyDeviceToHost, st));
    ST_CUDA(cudaStreamSynchronize(st));
    out->nnz = nnz;
    ST_CUDA(cudaMalloc(&out->col, (size_t)std::max<long long>(nnz, 1) * sizeof(int)));
    ST_CUDA(cudaMalloc(&out->val, (size_t)std::max<long long>(nnz, 1) * sizeof(float)));
    auto* urow = static_cast<long long*>(alloc((size_t)std::max<long long>(nnz, 1) * 8));
    if (!urow) return bufs.fail();
    merge_kernel<TV><<<blocks_for(n), 256, 0, st>>>(keys, pay, n, cb, flag, uidx, v, out->col, out->val, urow);
    count_launch();
    ST_CUDA(cudaGetLastError());
    if (nnz == 0) {
        ST_CUDA(cudaMemsetAsync(out->row_ptr, 0, (size_t)(rows + 1) * sizeof(long long), st));
    } else {
        rowptr_kernel<<<blocks_for(nnz), 256, 0, st>>>(urow, nnz, rows, out->row_ptr);
        count_launch();
        ST_CUDA(cudaGetLastError());
    }
    if (pad && rows > 0) {
        int* trig = static_cast<int*>(alloc(64));
        if (!trig) return bufs.fail();
        ST_CUDA(cudaMemsetAsync(trig, 0, sizeof(int), st));
        pad_trigger_kernel<<<blocks_for(rows), 256, 0, st>>>(out->row_ptr, rows, trig);
        count_launch();
        int h = 0;
        ST_CUDA(cudaMemcpyAsync(&h, trig, sizeof(int), cudaMemcpyDeviceToHost, st));
        ST_CUDA(cudaStreamSynchronize(st));
        if (h) {
            ST_CHECK(rows <= cols, ST_ERR_ARG,
                     "pad-to-8 entries use col = row, out of range for %lld rows x %lld cols", rows, cols);
            auto* plen = static_cast<long long*>(alloc((size_t)(rows + 1) * 8));
            long long* nrp = nullptr;
            ST_CUDA(cudaMalloc(&nrp, (size_t)(rows + 1) * sizeof(long long)));
            if (!plen) return bufs.fail();
            pad_len_kernel<<<blocks_for(rows), 256, 0, st>>>(out->row_ptr, rows, plen);
            count_launch();
            ST_TRY(exclusive_scan_i64(plen, nrp, rows, total, stmp, st));
            fill_last_kernel<<<1, 1, 0, st>>>(nrp, rows, total);
            count_launch();
            long long pn = 0;
            ST_CUDA(cudaMemcpyAsync(&pn, total, sizeof(long long), cudaMemcpyDeviceToHost, st));
            ST_CUDA(cudaStreamSynchronize(st));
            int* ncol = nullptr;
            float* nval = nullptr;
            ST_CUDA(cudaMalloc(&ncol, (size_t)std::max<long long>(pn, 1) * sizeof(int)));
            ST_CUDA(cudaMalloc(&nval, (size_t)std::max<long long>(pn, 1) * sizeof(float)));
            pad_scatter_kernel<<<blocks_for(rows), 256, 0, st>>>(out->row_ptr, out->col, out->val, rows, nrp, ncol,
                                                                 nval);
            count_launch();
            ST_CUDA(cudaGetLastError());
            ST_CUDA(cudaStreamSynchronize(st));
            cudaFree(out->row_ptr);
            cudaFree(out->col);
            cudaFree(out->val);
            out->row_ptr = nrp;
            out->col = ncol;
            out->val = nval;
            out->nnz = pn;
        }
    }
    UnevenRows u;
    ST_TRY(measure_rows(*out, total, &u, st));
    ST_CUDA(cudaStreamSynchronize(st));
    out->lanes = lanes_of(*out, u);
    return ST_OK;
}

template int build_csr<long long, double>(long long, long long, long long, const long long*, const long long*,
                                          const double*, bool, DevCsr*, cudaStream_t);
template int build_csr<int, float>(long long, long long, long long, const int*, const int*, const float*, bool,
                                   DevCsr*, cudaStream_t);

// What spmv_rows_kernel is slow on (UnevenRows), a warp per tile.
__global__ void uneven_tiles_kernel(const long long* __restrict__ rp, long long rows, unsigned long long* out) {
    const int lane = threadIdx.x & 31;
    unsigned long long entries = 0, longest = 0, heaviest = 0;
    for (long long r0 = ((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5) * SR_ROWS; r0 < rows;
         r0 += (((long long)gridDim.x * blockDim.x) >> 5) * SR_ROWS) {
        const long long total = rp[min(r0 + SR_ROWS, rows)] - rp[r0];
        long long most = 0;
        for (long long r = r0 + lane; r < min(r0 + SR_ROWS, rows); r += 32) most = max(most, rp[r + 1] - rp[r]);
        for (int o = 16; o > 0; o >>= 1) most = max(most, __shfl_xor_sync(FULL, most, o));
        if (most > SR_LONG || total > SR_CAP - 3) entries += (unsigned long long)total;
        longest = max(longest, (unsigned long long)most);
        heaviest = max(heaviest, (unsigned long long)total);
    }
    if (lane == 0 && entries) {
        atomicAdd(out, entries);
        atomicMax(out + 1, longest);
        atomicMax(out + 2, heaviest);
    }
}

// Where an eighth of the entries or more lie in such tiles, the rows go to groups
// of lanes: two lanes (fewer than five entries a row) or four, and eight where single
// rows set the pace (beyond 1024 entries); those keep a warp to themselves in the row
// tiles unless they share a tile or hardly a tile is without one. 1M rows, row tiles / lanes, us: a half of 18 entries
// and a half of none 56 / 33; 1 row of 128 at 600, the others 3, 149 / 82; a power law
// of mean 6.2 up to 2000 sorted by length 552 / 57, in random order 106 / 82; 1 row of
// 1000 at 4000 101 / 120 (four lanes 149); 1000 rows, one of 5000, 61 / 53.
int measure_rows(const DevCsr& A, void* scratch, UnevenRows* u, cudaStream_t st) {
    if (u) *u = UnevenRows();
    // a small matrix is built in less time than a few products save (the measure takes 16 us)
    if (A.nnz < 4096 || A.nnz >= SHORT_ROWS * A.rows) return ST_OK;
    auto* acc = static_cast<unsigned long long*>(scratch);
    if (u) ST_CUDA(cudaMemsetAsync(acc, 0, sizeof(UnevenRows), st));
    uneven_tiles_kernel<<<blocks_for((A.rows + SR_ROWS - 1) / SR_ROWS * 32), 256, 0, st>>>(A.row_ptr, A.rows, acc);
    count_launch();
    ST_CUDA(cudaGetLastError());
    if (u) ST_CUDA(cudaMemcpyAsync(u, acc, sizeof(UnevenRows), cudaMemcpyDeviceToHost, st));
    return ST_OK;
}

int lanes_of(const DevCsr& A, const UnevenRows& u) {
    if (8 * u.entries <= (unsigned long long)A.nnz) return 0;
    if (u.longest <= 1024) return A.nnz >= 5 * A.rows ? 4 : 2;
    return u.heaviest > 8192 || 16 * u.entries > 15 * (unsigned long long)A.nnz ? 8 : 0;
}

int launch_spmv(const DevCsr& A, const float* x, float* y, const float* add, float add_scale, const float* pdot,
                double* dot_acc, const int* done, cudaStream_t st) {
    const double avg = A.rows > 0 ? (double)A.nnz / (double)A.rows : 0.0;
    // tuning override: SEISMIC_GB300_SPMV_G=<1|2|4|8|16|32> threads per row
    static const int forced = [] {
        const char* e = std::getenv("SEISMIC_GB300_SPMV_G");
        return e ? std::atoi(e) : 0;
    }();
    switch (forced) {
        case 32: return launch_spmv_g<32, 6, false, true>(A, x, y, add, add_scale, pdot, dot_acc, done, st);
        case 16: return launch_spmv_g<16, 10, true, false>(A, x, y, add, add_scale, pdot, dot_acc, done, st);
        case 8: return launch_spmv_g<8, 4, true, false>(A, x, y, add, add_scale, pdot, dot_acc, done, st);
        case 4: return launch_spmv_g<4, 4, false, false>(A, x, y, add, add_scale, pdot, dot_acc, done, st);
        case 2: return launch_spmv_g<2, 4, false, false>(A, x, y, add, add_scale, pdot, dot_acc, done, st);
        case 1: return launch_spmv_rows(A, x, y, add, add_scale, pdot, dot_acc, done, st);
        default: break;
    }
    // measured on the 2M-ray matrix (180 entries per row) and its transpose (360): 16 threads per
    // row with 10 entries held per lane and the L2 prefetch 0.545 ms; the transpose with 32
    // threads, 6 entries per lane, no prefetch and the rest in turns 0.570 ms (0.640 with the rest one by one)
    if (avg >= 256) return launch_spmv_g<32, 6, false, true>(A, x, y, add, add_scale, pdot, dot_acc, done, st);
    if (avg >= 24) return launch_spmv_g<16, 10, true, false>(A, x, y, add, add_scale, pdot, dot_acc, done, st);
    if (avg >= SHORT_ROWS) return launch_spmv_g<8, 4, true, false>(A, x, y, add, add_scale, pdot, dot_acc, done, st);
    if (A.lanes == 8) return launch_spmv_g<8, 4, true, false>(A, x, y, add, add_scale, pdot, dot_acc, done, st);
    if (A.lanes == 4) return launch_spmv_g<4, 4, false, false>(A, x, y, add, add_scale, pdot, dot_acc, done, st);
    if (A.lanes == 2) return launch_spmv_g<2, 4, false, false>(A, x, y, add, add_scale, pdot, dot_acc, done, st);
    return launch_spmv_rows(A, x, y, add, add_scale, pdot, dot_acc, done, st);
}

int launch_f64_to_f32(const double* a, float* b, long long n, cudaStream_t st) {
    f64_to_f32_kernel<<<blocks_for(n), 256, 0, st>>>(a, b, n);
    count_launch();
    ST_CUDA(cudaGetLastError());
    return ST_OK;
}
int launch_f32_to_f64(const float* a, double* b, long long n, cudaStream_t st) {
    f32_to_f64_kernel<<<blocks_for(n), 256, 0, st>>>(a, b, n);
    count_launch();
    ST_CUDA(cudaGetLastError());
    return ST_OK;
}
int launch_jacobi(const DevCsr& A, float* dinv, cudaStream_t st) {
    jacobi_kernel<<<blocks_for(A.rows), 256, 0, st>>>(A.row_ptr, A.col, A.val, A.rows, dinv);
    count_launch();
    ST_CUDA(cudaGetLastError());
    return ST_OK;
}
int launch_normal_jacobi(const DevCsr& AT, double lam, float* dinv, cudaStream_t st) {
    if (AT.nnz >= 480 * AT.rows)
        normal_jacobi_kernel<32><<<blocks_for(AT.rows * 32), 256, 0, st>>>(AT.row_ptr, AT.val, AT.rows, lam, dinv);
    else if (AT.nnz >= 160 * AT.rows)
        normal_jacobi_kernel<16><<<blocks_for(AT.rows * 16), 256, 0, st>>>(AT.row_ptr, AT.val, AT.rows, lam, dinv);
    else if (AT.nnz >= 24 * AT.rows)
        normal_jacobi_kernel<8><<<blocks_for(AT.rows * 8), 256, 0, st>>>(AT.row_ptr, AT.val, AT.rows, lam, dinv);
    else
        normal_jacobi_rows_kernel<<<blocks_for(AT.rows), NJ_ROWS, 0, st>>>(AT.row_ptr, AT.val, AT.rows, lam, dinv);
    count_launch();
    ST_CUDA(cudaGetLastError());
    return ST_OK;
}
int launch_scale(float* v, long long n, float a, cudaStream_t st) {
    scale_kernel<<<blocks_for(n), 256, 0, st>>>(v, n, a);
    count_launch();
    ST_CUDA(cudaGetLastError());
    return ST_OK;
}
int launch_add_diag(DevCsr& A, float a, cudaStream_t st) {
    add_diag_kernel<<<blocks_for(A.rows), 256, 0, st>>>(A.row_ptr, A.col, A.val, A.rows, a);
    count_launch();
    ST_CUDA(cudaGetLastError());
    return ST_OK;
}
int launch_sumsq(const float* v, long long n, double* acc, cudaStream_t st) {
    ST_CUDA(cudaMemsetAsync(acc, 0, sizeof(double), st));
    sumsq_kernel<<<blocks_for(n), 256, 0, st>>>(v, n, acc);
    count_launch();
    ST_CUDA(cudaGetLastError());
    return ST_OK;
}
int launch_dot64(const double* a, const double* b, long long n, double* acc, cudaStream_t st) {
    ST_CUDA(cudaMemsetAsync(acc, 0, sizeof(double), st));
    dot64_kernel<<<blocks_for(n), 256, 0, st>>>(a, b, n, acc);
    count_launch();
    ST_CUDA(cudaGetLastError());
    return ST_OK;
}

__global__ void sqrt_kernel(const float* __restrict__ a, float* __restrict__ out, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = sqrtf(a[i]);
}

int launch_sqrt(const float* a, float* out, long long n, cudaStream_t st) {
    sqrt_kernel<<<blocks_for(n), 256, 0, st>>>(a, out, n);
    count_launch();
    ST_CUDA(cudaGetLastError());
    return ST_OK;
}

int launch_residual(float* out, const float* b, const float* Ax, long long n, cudaStream_t st) {
    axpby_kernel<<<blocks_for(n), 256, 0, st>>>(out, b, Ax, 1.0f, n);
    count_launch();
    ST_CUDA(cudaGetLastError());
    return ST_OK;
}
int launch_fd_triplets(const double* vel, long long nx, long long ny, long long nz, double idx2, double idy2,
                       double idz2, double dt2, long long* tr, long long* tc, double* tv, cudaStream_t st) {
    fd_triplets_kernel<<<blocks_for(nx * ny * nz), 256, 0, st>>>(vel, nx, ny, nz, idx2, idy2, idz2, dt2, tr, tc, tv);
    count_launch();
    ST_CUDA(cudaGetLastError());
    return ST_OK;
}

// ---------------------------------------------------------------- CG driver
int cg_loop(const CgProblem& P, CgWork& W, int k0, int max_iter, double tol, int check_every, CgResult* res,
            cudaStream_t st);

int run_cg(const CgProblem& P, CgWork& W, int max_iter, double tol, int check_every, CgResult* res,
           cudaStream_t st) {
    const long long n = P.n;
    ST_CUDA(cudaMemsetAsync(W.sc, 0, sizeof(CgScalars), st));
    // iteration -1 stores rz in acc[2].rzn
    // (stencil: p and <r, z> from the preconditioner kernel below)
    cg_init_kernel<<<cg_blocks(n), 256, 0, st>>>(P.b, P.sq ? nullptr : P.dinv, n, P.x, W.r,
                                                   P.dinv && !P.sq ? W.z : nullptr, W.p,
                                                   P.sq ? nullptr : W.sc->acc[2].rzn, W.sc->bb);
    count_launch();
    ST_CUDA(cudaGetLastError());
    if (P.sq) {
        stencil_prec_kernel<<<cg_blocks(n), 256, 0, st>>>(n, W.r, P.dinv, P.sq, P.gx, P.gy, P.gz, P.w[0], P.w[1],
                                                           P.w[2], W.z, W.p, W.sc->acc[2].rzn, nullptr);
        count_launch();
        ST_CUDA(cudaGetLastError());
    }
    CgScalars h{};
    ST_CUDA(cudaMemcpyAsync(&h, W.sc, sizeof(h), cudaMemcpyDeviceToHost, st));
    ST_CUDA(cudaStreamSynchronize(st));
    res->iters = 0;
    res->rel = 0.0;
    res->breakdown = 0;
    if (std::sqrt(cg_slot_sum(h.bb)) < 1e-30) return ST_OK;  // sparse_ops.cpp:22,83
    return cg_loop(P, W, 0, max_iter, tol, check_every, res, st);
}

int resume_cg(const CgProblem& P, CgWork& W, int max_iter, double tol, int check_every, CgResult* res,
              cudaStream_t st) {
    if (res->breakdown || res->iters == 0 || res->iters >= max_iter) return ST_OK;
    // the last iteration stopped before p = z + beta p: clear the stop and
    // run that update (a zero tolerance never stops it)
    const int k = res->iters;
    ST_CUDA(cudaMemsetAsync(&W.sc->done, 0, sizeof(int), st));
    cg_pupdate_kernel<<<cg_blocks(P.n), 256, 0, st>>>(P.n, W.p, P.dinv || P.sq ? W.z : W.r, W.sc, k - 1, 0.0);
    count_launch();
    ST_CUDA(cudaGetLastError());
    return cg_loop(P, W, k, max_iter, tol, check_every, res, st);
}

// Iterations k0 .. of a solve whose state is in W (check_every iterations
// between host reads of the scalars).
int cg_loop(const CgProblem& P, CgWork& W, int k0, int max_iter, double tol, int check_every, CgResult* res,
            cudaStream_t st) {
    const long long n = P.n;
    CgScalars h{};
    const float* zp = P.dinv ? W.z : W.r;
    const int quads = quads_ok({P.x, W.r, W.z, W.p, W.q, P.dinv});
    int k = k0;
    while (k < max_iter) {
        const int batch = std::min(check_every, max_iter - k);
        for (int j = 0; j < batch; ++j, ++k) {
            if (P.AT) {
                ST_TRY(launch_spmv(*P.A, W.p, W.t, nullptr, 0.0f, nullptr, nullptr, &W.sc->done, st));
                ST_TRY(launch_spmv(*P.AT, W.t, W.q, W.p, (float)P.lam, W.p, W.sc->acc[k % 3].pq, &W.sc->done, st));
            } else {
                ST_TRY(launch_spmv(*P.A, W.p, W.q, nullptr, 0.0f, W.p, W.sc->acc[k % 3].pq, &W.sc->done, st));
            }
            cg_update_kernel<<<cg_blocks(n), 256, 0, st>>>(n, P.x, W.r, P.dinv && !P.sq ? W.z : nullptr, W.p,
                                                             W.q, P.sq ? nullptr : P.dinv, W.sc, k, P.sq != nullptr,
                                                             quads);
            count_launch();
            if (P.sq) {
                stencil_prec_kernel<<<cg_blocks(n), 256, 0, st>>>(n, W.r, P.dinv, P.sq, P.gx, P.gy, P.gz, P.w[0],
                                                                   P.w[1], P.w[2], W.z, nullptr,
                                                                   W.sc->acc[k % 3].rzn, &W.sc->done);
                count_launch();
            }
            cg_pupdate_kernel<<<cg_blocks(n), 256, 0, st>>>(n, W.p, zp, W.sc, k, tol);
            count_launch();
            ST_CUDA(cudaGetLastError());
        }
        ST_CUDA(cudaMemcpyAsync(&h, W.sc, sizeof(h), cudaMemcpyDeviceToHost, st));
        ST_CUDA(cudaStreamSynchronize(st));
        if (h.done) break;
    }
    res->iters = h.iters;
    res->rel = h.rel;
    res->breakdown = h.breakdown;
    return ST_OK;
}

}  // namespace stg
