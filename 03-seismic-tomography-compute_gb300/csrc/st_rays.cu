// Straight-ray path-length matrix for traveltime tomography.
//
// Row i of A holds, for every cell j that ray i crosses, the length of the
// ray inside that cell (times the cell size), so A s = traveltimes for the
// slowness model s. The traversal is the exact voxel walk of Amanatides and
// Woo ("A fast voxel traversal algorithm for ray tracing", Eurographics
// 1987): the ray p(t) = p0 + t (p1 - p0), t in [0, 1], is cut at every
// cell face it crosses, in order of t; ties go to x, then y, then z. All
// arithmetic is FP64 with explicit rounding (no contractions) so the host
// restatement in the oracle produces the same lengths bit for bit; values
// are rounded to FP32 once, when the CSR is built.
//
// The result has the CSRMatrix::build_from_triplets semantics
// (sparse/csr_matrix.cpp:25-72): per-row columns ascending, no padding, columns
// j = (ix*ny + iy)*nz + iz. No sort is needed for it: a ray crosses the cells
// monotonically along each axis, so its columns are ascending up to the
// reversal of whole runs.
//   1. ray_bound_kernel: from the end points alone, the most steps a ray can
//      take; a tile of 32 rays gets that many rows of 32 scratch entries.
//   2. ray_walk_kernel: one walk per ray, a thread each; entry j of lane l goes
//      to row j of its tile, so a warp's stores are whole lines.
//   3. a scan of the counts gives the row pointers.
//   4. ray_place_kernel: a warp per ray. Entry i lies in the run [xs, xe) of its
//      x plane and the run [ys, ye) of its (x, y) column; with the ray's
//      direction along each axis its ascending place is
//        (x up ? xs : m - xe) + (y up ? ys - xs : xe - ye) + (z up ? i - ys : ye - 1 - i).
// The walk is bound by the FP64 pipe (a warp's operation takes 16 cycles): times
// are compared as integers, and the correctly rounded quotient is formed with
// the axis's reciprocal. Rays that this form cannot take (end points that are
// not finite, extreme ranges) walk with plain FP64 operations; a ray that
// outruns its bound, or scratch that cannot be had, sends the call to the triplet
// builder. 500k rays on 50^3 cells
// (45M entries): build, transpose and two products 6.3 ms, 16.8 with two plain
// walks and the sort of the triplets.
#include "st_fp64.cuh"
#include "st_sort.cuh"
#include "st_sparse.cuh"

#include <algorithm>
#include <cmath>

namespace stg {
namespace {

struct RayGrid {
    int nx, ny, nz;
    double h;
};

__host__ __device__ inline double dadd(double a, double b) {
#ifdef __CUDA_ARCH__
    return __dadd_rn(a, b);
#else
    return a + b;
#endif
}
__host__ __device__ inline double dsub(double a, double b) {
#ifdef __CUDA_ARCH__
    return __dsub_rn(a, b);
#else
    return a - b;
#endif
}
__host__ __device__ inline double dmul(double a, double b) {
#ifdef __CUDA_ARCH__
    return __dmul_rn(a, b);
#else
    return a * b;
#endif
}
__host__ __device__ inline double ddiv(double a, double b) {
#ifdef __CUDA_ARCH__
    return __ddiv_rn(a, b);
#else
    return a / b;
#endif
}

__host__ __device__ inline int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// Parameter t at which the ray leaves cell index c along one axis.
__device__ inline double t_exit(int c, int step, double p0, double d) {
    if (step == 0) return 1e300;
    const double face = (double)(step > 0 ? c + 1 : c);
    return ddiv(dsub(face, p0), d);
}

// Walks ray e; emit(col, length) for every crossed cell, in traversal order.
template <class F>
__device__ void walk(const double* e, const RayGrid& G, F emit) {
    const double p0[3] = {e[0], e[1], e[2]};
    const double d[3] = {dsub(e[3], e[0]), dsub(e[4], e[1]), dsub(e[5], e[2])};
    const double len = sqrt(dadd(dadd(dmul(d[0], d[0]), dmul(d[1], d[1])), dmul(d[2], d[2])));
    const int n[3] = {G.nx, G.ny, G.nz};
    int c[3], step[3];
    double tm[3];
    for (int a = 0; a < 3; ++a) {
        c[a] = clampi((int)floor(p0[a]), 0, n[a] - 1);
        step[a] = d[a] > 0.0 ? 1 : (d[a] < 0.0 ? -1 : 0);
        tm[a] = t_exit(c[a], step[a], p0[a], d[a]);
    }
    double t = 0.0;
    const int max_iter = G.nx + G.ny + G.nz + 3;
    for (int it = 0; it < max_iter; ++it) {
        const int ax = (tm[0] <= tm[1] && tm[0] <= tm[2]) ? 0 : (tm[1] <= tm[2] ? 1 : 2);
        const double tn = tm[ax];
        const double te = tn < 1.0 ? tn : 1.0;
        const double seg = dmul(dmul(dsub(te, t), len), G.h);
        if (seg > 0.0) emit(((long long)c[0] * G.ny + c[1]) * G.nz + c[2], seg);
        if (tn >= 1.0) break;
        t = tn;
        c[ax] += step[ax];
        if (c[ax] < 0 || c[ax] >= n[ax]) break;
        tm[ax] = t_exit(c[ax], step[ax], p0[ax], d[ax]);
    }
}

// FP64 order as integer order (-0 and +0 alike; no NaN).
__device__ __forceinline__ long long time_key(double t) {
    const long long b = __double_as_longlong(t);
    return b < 0 ? (long long)0x8000000000000000ull - b : b;
}

// x / d through the axis's reciprocal y; an x below 2^-400 goes to the division.
__device__ __forceinline__ double quotient(double x, double d, double y) {
    const unsigned hx = (unsigned)__double2hiint(x) & 0x7fffffffu;
    if (hx < (623u << 20) && (hx | (unsigned)__double2loint(x))) return __ddiv_rn(x, d);
    return quotient_of(x, d, y);
}

// Whether the fast walk takes an axis: finite, and d zero or of moderate size.
__device__ __forceinline__ bool fast_axis(double p, double d) {
    const unsigned hp = (unsigned)__double2hiint(p) & 0x7fffffffu;
    return hp < (1323u << 20) && (moderate(d) || d == 0.0);
}

// The most iterations of walk(): one and, per axis, the faces between the start
// cell and the end point (one more for rounding).
__device__ __forceinline__ int step_bound(const double* e, const RayGrid& G) {
    const int n[3] = {G.nx, G.ny, G.nz};
    long long b = 1;
    for (int a = 0; a < 3; ++a) {
        const long long c = clampi((int)floor(e[a]), 0, n[a] - 1), f = (long long)(int)floor(e[3 + a]);
        const long long span = (f > c ? f - c : c - f) + 1;
        b += span < n[a] ? span : n[a];
    }
    return (int)min(b, (long long)G.nx + G.ny + G.nz + 3);
}

__global__ void ray_bound_kernel(const double* __restrict__ ends, long long nrays, RayGrid G,
                                 long long* __restrict__ height, int* __restrict__ tallest) {
    const long long tiles = (nrays + 31) / 32;
    const int lane = threadIdx.x & 31;
    for (long long t = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; t < tiles;
         t += ((long long)gridDim.x * blockDim.x) >> 5) {
        const long long i = 32 * t + lane;
        int b = i < nrays ? step_bound(ends + 6 * i, G) : 0;
        for (int o = 16; o > 0; o >>= 1) b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
        if (lane == 0) {
            height[t] = b;
            atomicMax(tallest, b);
        }
    }
}

// Directions of a ray's axes: bits 0-2 set where x / y / z descends.
__global__ void __launch_bounds__(128)
    ray_walk_kernel(const double* __restrict__ ends, long long nrays, RayGrid G, const long long* __restrict__ height,
                    const long long* __restrict__ off, int* __restrict__ scol, float* __restrict__ sval,
                    long long* __restrict__ count, unsigned char* __restrict__ down, int* __restrict__ overrun) {
    const int lane = threadIdx.x & 31;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nrays;
         i += (long long)gridDim.x * blockDim.x) {
        const long long base = 32 * off[i >> 5] + lane;
        const int rows = (int)height[i >> 5];
        const double* e = ends + 6 * i;
        const double px = e[0], py = e[1], pz = e[2];
        const double dx = dsub(e[3], px), dy = dsub(e[4], py), dz = dsub(e[5], pz);
        int k = 0;
        bool over = false;
        auto emit = [&](int col, float v) {
            if (k < rows) {
                scol[base + 32ll * k] = col;
                sval[base + 32ll * k] = v;
            } else {
                over = true;
            }
            ++k;
        };
        if (fast_axis(px, dx) && fast_axis(py, dy) && fast_axis(pz, dz)) {
            const double len = sqrt(dadd(dadd(dmul(dx, dx), dmul(dy, dy)), dmul(dz, dz)));
            int cx = clampi((int)floor(px), 0, G.nx - 1), cy = clampi((int)floor(py), 0, G.ny - 1),
                cz = clampi((int)floor(pz), 0, G.nz - 1);
            const double one = 1.0;
            const double ux = dx > 0.0 ? one : -one, uy = dy > 0.0 ? one : -one, uz = dz > 0.0 ? one : -one;
            const double yx = dx != 0.0 ? __drcp_rn(dx) : 0.0, yy = dy != 0.0 ? __drcp_rn(dy) : 0.0,
                         yz = dz != 0.0 ? __drcp_rn(dz) : 0.0;
            double fx = (double)(dx > 0.0 ? cx + 1 : cx), fy = (double)(dy > 0.0 ? cy + 1 : cy),
                   fz = (double)(dz > 0.0 ? cz + 1 : cz);
            double tx = dx != 0.0 ? quotient(dsub(fx, px), dx, yx) : 1e300;
            double ty = dy != 0.0 ? quotient(dsub(fy, py), dy, yy) : 1e300;
            double tz = dz != 0.0 ? quotient(dsub(fz, pz), dz, yz) : 1e300;
            const long long kone = time_key(1.0);
            double t = 0.0;
            // cells left along each axis before the ray leaves the grid, and the column's step
            int lx = dx > 0.0 ? G.nx - 1 - cx : cx, ly = dy > 0.0 ? G.ny - 1 - cy : cy,
                lz = dz > 0.0 ? G.nz - 1 - cz : cz;
            const int sx = dx > 0.0 ? G.ny * G.nz : -G.ny * G.nz, sy = dy > 0.0 ? G.nz : -G.nz,
                      sz = dz > 0.0 ? 1 : -1;
            int col = (cx * G.ny + cy) * G.nz + cz;
            for (;;) {
                const long long kx = time_key(tx), ky = time_key(ty), kz = time_key(tz);
                const int ax = (kx <= ky && kx <= kz) ? 0 : (ky <= kz ? 1 : 2);
                const double tn = ax == 0 ? tx : (ax == 1 ? ty : tz);
                const bool last = (ax == 0 ? kx : (ax == 1 ? ky : kz)) >= kone;
                const double seg = dmul(dmul(dsub(last ? one : tn, t), len), G.h);
                if (__double_as_longlong(seg) > 0) emit(col, (float)seg);
                int& left = ax == 0 ? lx : (ax == 1 ? ly : lz);
                if (last || left == 0) break;
                --left;
                t = tn;
                col += ax == 0 ? sx : (ax == 1 ? sy : sz);
                const double f = dadd(ax == 0 ? fx : (ax == 1 ? fy : fz), ax == 0 ? ux : (ax == 1 ? uy : uz));
                const double q = quotient(dsub(f, ax == 0 ? px : (ax == 1 ? py : pz)),
                                          ax == 0 ? dx : (ax == 1 ? dy : dz), ax == 0 ? yx : (ax == 1 ? yy : yz));
                if (ax == 0) {
                    fx = f;
                    tx = q;
                } else if (ax == 1) {
                    fy = f;
                    ty = q;
                } else {
                    fz = f;
                    tz = q;
                }
            }
        } else {
            walk(e, G, [&](long long col, double v) { emit((int)col, (float)v); });
        }
        count[i] = k;
        down[i] = (unsigned char)((dx < 0.0 ? 1 : 0) | (dy < 0.0 ? 2 : 0) | (dz < 0.0 ? 4 : 0));
        if (over) *overrun = 1;
    }
}

constexpr int PLACE_WARPS = 8;

// Shared memory per warp: the ray's columns and values, and a bit per entry that
// starts an x plane / an (x, y) column.
__host__ __device__ inline size_t place_bytes(int tallest) {
    const int chunks = (tallest + 31) / 32;
    return (size_t)chunks * 32 * 8 + (size_t)chunks * 8;
}

__global__ void __launch_bounds__(PLACE_WARPS * 32)
    ray_place_kernel(long long nrays, RayGrid G, int tallest, const long long* __restrict__ off,
                     const int* __restrict__ scol, const float* __restrict__ sval,
                     const unsigned char* __restrict__ down, const long long* __restrict__ rp,
                     int* __restrict__ col_out, float* __restrict__ val_out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int chunks = (tallest + 31) / 32;
    int* cols = reinterpret_cast<int*>(smem_raw + warp * place_bytes(tallest));
    float* vals = reinterpret_cast<float*>(cols + 32 * chunks);
    unsigned* hx = reinterpret_cast<unsigned*>(vals + 32 * chunks);
    unsigned* hy = hx + chunks;
    const unsigned le = lane == 31 ? 0xffffffffu : (2u << lane) - 1, gt = ~le;
    const int nyz = G.ny * G.nz;
    const long long tiles = (nrays + 31) / 32;
    for (long long t = blockIdx.x; t < tiles; t += gridDim.x) {
        for (int r = warp; r < 32; r += warps) {
            const long long i = 32 * t + r;
            if (i >= nrays) break;
            const long long o = rp[i];
            const int m = (int)(rp[i + 1] - o);
            const long long base = 32 * off[t] + r;
            int px = -1, py = -1;  // plane and column of the entry before the chunk
            for (int q = 0; 32 * q < m; ++q) {
                const int j = 32 * q + lane;
                const int c = j < m ? scol[base + 32ll * j] : 0;
                const float v = j < m ? sval[base + 32ll * j] : 0.0f;
                cols[j] = c;
                vals[j] = v;
                const int X = c / nyz, Y = c / G.nz;
                const int xp = __shfl_up_sync(0xffffffffu, X, 1), yp = __shfl_up_sync(0xffffffffu, Y, 1);
                const unsigned bx = __ballot_sync(0xffffffffu, j < m && X != (lane ? xp : px));
                const unsigned by = __ballot_sync(0xffffffffu, j < m && Y != (lane ? yp : py));
                if (lane == 0) {
                    hx[q] = bx;
                    hy[q] = by;
                }
                px = __shfl_sync(0xffffffffu, X, 31);
                py = __shfl_sync(0xffffffffu, Y, 31);
            }
            __syncwarp();
            const unsigned dn = down[i];
            const int last = (m - 1) / 32;
            auto first_of = [&](const unsigned* h, int q) {
                unsigned b = h[q] & le;
                while (!b) b = h[--q];  // entry 0 starts a run
                return 32 * q + 31 - __clz((int)b);
            };
            auto end_of = [&](const unsigned* h, int q) {
                unsigned b = h[q] & gt;
                while (!b && q < last) b = h[++q];
                return b ? 32 * q + __ffs((int)b) - 1 : m;
            };
            for (int q = 0; q <= last && m > 0; ++q) {
                const int j = 32 * q + lane;
                if (j < m) {
                    const int xs = first_of(hx, q), xe = end_of(hx, q), ys = first_of(hy, q), ye = end_of(hy, q);
                    const int pos = (dn & 1 ? m - xe : xs) + (dn & 2 ? xe - ye : ys - xs) +
                                    (dn & 4 ? ye - 1 - j : j - ys);
                    col_out[o + pos] = cols[j];
                    val_out[o + pos] = vals[j];
                }
            }
            __syncwarp();
        }
    }
}

__global__ void ray_count_kernel(const double* __restrict__ ends, long long nrays, RayGrid G, long long* count) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nrays;
         i += (long long)gridDim.x * blockDim.x) {
        long long k = 0;
        walk(ends + 6 * i, G, [&](long long, double) { ++k; });
        count[i] = k;
    }
}

__global__ void ray_write_kernel(const double* __restrict__ ends, long long nrays, RayGrid G,
                                 const long long* __restrict__ off, long long* rows, long long* cols, double* vals) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nrays;
         i += (long long)gridDim.x * blockDim.x) {
        long long k = off[i];
        walk(ends + 6 * i, G, [&](long long col, double v) {
            rows[k] = i;
            cols[k] = col;
            vals[k] = v;
            ++k;
        });
    }
}

unsigned grid_for(long long n) {
    return (unsigned)std::max<long long>(1, std::min<long long>((n + 255) / 256, 152LL * 32));
}

}  // namespace

// The walk-once builder; *done = false (and nothing built) where a ray outran its
// bound, the rows do not fit in shared memory, or an allocation fails: a tile's
// scratch is 32 times its longest ray's bound, so rays of mixed lengths can ask for
// many times what the triplets of their entries take.
static int build_walk_once(long long nrays, const double* d_ends, const RayGrid& G, DevCsr* out, bool* done,
                           cudaStream_t st) {
    *done = false;
    const long long tiles = (nrays + 31) / 32;
    DeviceBuffers bufs;
    auto* height = static_cast<long long*>(bufs.get((size_t)tiles * 8));
    auto* off = static_cast<long long*>(bufs.get((size_t)(tiles + 1) * 8));
    auto* count = static_cast<long long*>(bufs.get((size_t)nrays * 8));
    auto* down = static_cast<unsigned char*>(bufs.get((size_t)nrays));
    auto* info = static_cast<int*>(bufs.get(64));  // tallest, overrun; from 16 bytes on the rows' measure
    void* stmp = bufs.get(scan_tmp_bytes(nrays));
    if (!height || !off || !count || !down || !info || !stmp) return ST_OK;
    auto allocate = [&](auto** p, size_t n) {
        if (cudaMalloc(p, n * sizeof(**p)) == cudaSuccess) return true;
        cudaGetLastError();
        *p = nullptr;
        out->release();
        return false;
    };
    ST_CUDA(cudaMemsetAsync(info, 0, 2 * sizeof(int), st));
    ray_bound_kernel<<<grid_for(tiles * 32), 256, 0, st>>>(d_ends, nrays, G, height, info);
    count_launch();
    ST_CUDA(cudaGetLastError());
    ST_TRY(exclusive_scan_i64(height, off, tiles, off + tiles, stmp, st));
    long long rows = 0;
    int h[2] = {0, 0};
    ST_CUDA(cudaMemcpyAsync(&rows, off + tiles, sizeof(rows), cudaMemcpyDeviceToHost, st));
    ST_CUDA(cudaMemcpyAsync(h, info, sizeof(int), cudaMemcpyDeviceToHost, st));
    ST_CUDA(cudaStreamSynchronize(st));
    const int tallest = h[0];
    int warps = PLACE_WARPS;
    while (warps > 1 && warps * place_bytes(tallest) > 200 * 1024) warps /= 2;
    const size_t smem = warps * place_bytes(tallest);
    if (smem > 200 * 1024) return ST_OK;
    auto* scol = static_cast<int*>(bufs.get((size_t)rows * 32 * 4));
    auto* sval = static_cast<float*>(bufs.get((size_t)rows * 32 * 4));
    if (!scol || !sval) return ST_OK;
    ray_walk_kernel<<<(unsigned)std::min<long long>((nrays + 127) / 128, 1 << 20), 128, 0, st>>>(
        d_ends, nrays, G, height, off, scol, sval, count, down, info + 1);
    count_launch();
    ST_CUDA(cudaGetLastError());
    if (!allocate(&out->row_ptr, (size_t)(nrays + 1))) return ST_OK;
    ST_TRY(exclusive_scan_i64(count, out->row_ptr, nrays, out->row_ptr + nrays, stmp, st));
    long long nnz = 0;
    ST_CUDA(cudaMemcpyAsync(&nnz, out->row_ptr + nrays, sizeof(nnz), cudaMemcpyDeviceToHost, st));
    ST_CUDA(cudaMemcpyAsync(h, info, 2 * sizeof(int), cudaMemcpyDeviceToHost, st));
    ST_CUDA(cudaStreamSynchronize(st));
    if (h[1]) {
        out->release();
        return ST_OK;
    }
    ST_CHECK(nnz < (1ll << 32), ST_ERR_ARG, "at most 2^32-1 triplets per build");
    if (!allocate(&out->col, (size_t)std::max<long long>(nnz, 1))) return ST_OK;
    if (!allocate(&out->val, (size_t)std::max<long long>(nnz, 1))) return ST_OK;
    out->rows = nrays;
    out->cols = (long long)G.nx * G.ny * G.nz;
    out->nnz = nnz;
    ST_CUDA(cudaFuncSetAttribute(ray_place_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    ray_place_kernel<<<(unsigned)std::min<long long>(tiles, 152LL * 16), warps * 32, smem, st>>>(
        nrays, G, tallest, off, scol, sval, down, out->row_ptr, out->col, out->val);
    count_launch();
    ST_CUDA(cudaGetLastError());
    UnevenRows u;
    ST_TRY(measure_rows(*out, info + 4, &u, st));
    ST_CUDA(cudaStreamSynchronize(st));
    out->lanes = lanes_of(*out, u);
    *done = true;
    return ST_OK;
}

// Builds the ray matrix of nrays rays (device endpoints [nrays][6] =
// x0 y0 z0 x1 y1 z1 in cell units) over an nx*ny*nz grid of cells of size h.
int build_ray_csr(long long nrays, const double* d_ends, int nx, int ny, int nz, double h, DevCsr* out,
                  long long* total_nnz, cudaStream_t st) {
    ST_CHECK(nrays >= 0 && nx > 0 && ny > 0 && nz > 0, ST_ERR_ARG, "bad ray-matrix extents");
    ST_CHECK((long long)nx * ny * nz < (1ll << 31), ST_ERR_ARG, "cell count must fit int32 columns");
    ST_CHECK(h > 0.0 && std::isfinite(h), ST_ERR_ARG, "cell size must be positive");
    const RayGrid G{nx, ny, nz, h};
    if (nrays > 0) {
        bool done = false;
        ST_TRY(build_walk_once(nrays, d_ends, G, out, &done, st));
        if (done) {
            if (total_nnz) *total_nnz = out->nnz;
            return ST_OK;
        }
    }
    DeviceBuffers bufs;
    auto* count = static_cast<long long*>(bufs.get((size_t)(nrays + 1) * 8));
    auto* off = static_cast<long long*>(bufs.get((size_t)(nrays + 1) * 8));
    auto* tot = static_cast<long long*>(bufs.get(64));
    void* stmp = bufs.get(scan_tmp_bytes(std::max<long long>(nrays, 1)));
    if (!count || !off || !tot || !stmp) return bufs.fail();
    long long n = 0;
    if (nrays > 0) {
        ray_count_kernel<<<grid_for(nrays), 256, 0, st>>>(d_ends, nrays, G, count);
        count_launch();
        ST_CUDA(cudaGetLastError());
        ST_TRY(exclusive_scan_i64(count, off, nrays, tot, stmp, st));
        ST_CUDA(cudaMemcpyAsync(&n, tot, sizeof(long long), cudaMemcpyDeviceToHost, st));
        ST_CUDA(cudaStreamSynchronize(st));
    }
    if (total_nnz) *total_nnz = n;
    auto* r = static_cast<long long*>(bufs.get((size_t)std::max<long long>(n, 1) * 8));
    auto* c = static_cast<long long*>(bufs.get((size_t)std::max<long long>(n, 1) * 8));
    auto* v = static_cast<double*>(bufs.get((size_t)std::max<long long>(n, 1) * 8));
    if (!r || !c || !v) return bufs.fail();
    if (n > 0) {
        ray_write_kernel<<<grid_for(nrays), 256, 0, st>>>(d_ends, nrays, G, off, r, c, v);
        count_launch();
        ST_CUDA(cudaGetLastError());
    }
    return build_csr<long long, double>(nrays, (long long)nx * ny * nz, n, r, c, v, false, out, st);
}

}  // namespace stg
