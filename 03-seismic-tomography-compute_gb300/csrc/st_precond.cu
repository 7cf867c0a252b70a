// CUDA-core layers of the learned CG preconditioner (the 32 -> 32 channel
// layers run on the tensor cores, st_conv.cu).
//
// The network maps a residual r of the damped tomography normal equations
// on an nx x ny x nz cell grid (compact, x slowest) to a correction
//     z = dinv * r + s_out * N(s_in * r, s_in * dinv * r),
//     N = C_out o (relu(conv_K(h) + h))^K o relu(C_in),
// with dinv the Jacobi diagonal, s_in = 1 / rms(r) and s_out = rms(r) *
// mean(dinv); N has no biases, so z scales with r. C_in: 2 -> 32 channels,
// C_out: 32 -> 1, both 3x3x3 with zero padding. Activations h are padded
// channels-last BF16 volumes ([(nx+2)(ny+2)(nz+2)][32], zero border).
//
// Weight layouts (FP32 masters): C_in [32][2][27], C_out [32][27], conv_k
// [32][32][27] (out, in, tap = (kd*3 + kh)*3 + kw).
#include "st_common.cuh"

#include <algorithm>

namespace stg {
namespace {

constexpr int CH = 32;
constexpr int NTAP = 27;

struct Vol {
    int nx, ny, nz;
    __host__ __device__ long long pad_row(int x, int y, int z) const {  // padded row of interior (x, y, z)
        return ((long long)(x + 1) * (ny + 2) + (y + 1)) * (nz + 2) + (z + 1);
    }
    __host__ __device__ long long n() const { return (long long)nx * ny * nz; }
};

__device__ __forceinline__ void decode(long long i, const Vol& v, int& x, int& y, int& z) {
    z = (int)(i % v.nz);
    const long long t = i / v.nz;
    y = (int)(t % v.ny);
    x = (int)(t / v.ny);
}

__device__ __forceinline__ void load_row32(const __nv_bfloat16* p, float f[CH]) {
    const uint4* q = reinterpret_cast<const uint4*>(p);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint4 u = q[j];
        const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 t = __bfloat1622float2(b[e]);
            f[8 * j + 2 * e] = t.x;
            f[8 * j + 2 * e + 1] = t.y;
        }
    }
}

__device__ __forceinline__ void store_row32(__nv_bfloat16* p, const float f[CH]) {
    uint4* q = reinterpret_cast<uint4*>(p);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        uint4 u;
        __nv_bfloat162* b = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
        for (int e = 0; e < 4; ++e) b[e] = __floats2bfloat162_rn(f[8 * j + 2 * e], f[8 * j + 2 * e + 1]);
        q[j] = u;
    }
}

// h0 = relu(C_in([s r, s dinv r])) into the padded layout (interior rows only;
// the border stays as allocated, zero).
__global__ void in_conv_kernel(const float* __restrict__ r, const float* __restrict__ dinv, const float* scale,
                               const float* __restrict__ w, Vol v, __nv_bfloat16* __restrict__ h) {
    __shared__ float ws[CH * 2 * NTAP];
    for (int i = threadIdx.x; i < CH * 2 * NTAP; i += blockDim.x) ws[i] = w[i];
    __syncthreads();
    const float s = *scale;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < v.n(); i += (long long)gridDim.x * blockDim.x) {
        int x, y, z;
        decode(i, v, x, y, z);
        float acc[CH];
#pragma unroll
        for (int c = 0; c < CH; ++c) acc[c] = 0.0f;
        for (int tap = 0; tap < NTAP; ++tap) {
            const int xx = x + tap / 9 - 1, yy = y + (tap / 3) % 3 - 1, zz = z + tap % 3 - 1;
            if (xx < 0 || xx >= v.nx || yy < 0 || yy >= v.ny || zz < 0 || zz >= v.nz) continue;
            const long long j = ((long long)xx * v.ny + yy) * v.nz + zz;
            const float a = s * r[j], b = a * dinv[j];
#pragma unroll
            for (int c = 0; c < CH; ++c) acc[c] = fmaf(ws[(c * 2) * NTAP + tap], a, fmaf(ws[(c * 2 + 1) * NTAP + tap], b, acc[c]));
        }
#pragma unroll
        for (int c = 0; c < CH; ++c) acc[c] = fmaxf(acc[c], 0.0f);
        store_row32(h + v.pad_row(x, y, z) * CH, acc);
    }
}

// dW_in[c][k][tap] += sum_v g[v][c] * in_k[v + s_tap]; one block per tap and
// slab of voxels, block-reduced, one atomic per weight per block.
__global__ void in_conv_wgrad_kernel(const float* __restrict__ r, const float* __restrict__ dinv, const float* scale,
                                     const __nv_bfloat16* __restrict__ g, Vol v, float* __restrict__ dw) {
    const int tap = blockIdx.y;
    const int dx = tap / 9 - 1, dy = (tap / 3) % 3 - 1, dz = tap % 3 - 1;
    const float s = *scale;
    float acc[2 * CH];
#pragma unroll
    for (int c = 0; c < 2 * CH; ++c) acc[c] = 0.0f;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < v.n(); i += (long long)gridDim.x * blockDim.x) {
        int x, y, z;
        decode(i, v, x, y, z);
        const int xx = x + dx, yy = y + dy, zz = z + dz;
        if (xx < 0 || xx >= v.nx || yy < 0 || yy >= v.ny || zz < 0 || zz >= v.nz) continue;
        const long long j = ((long long)xx * v.ny + yy) * v.nz + zz;
        const float a = s * r[j], b = a * dinv[j];
        float gg[CH];
        load_row32(g + v.pad_row(x, y, z) * CH, gg);
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            acc[2 * c] = fmaf(gg[c], a, acc[2 * c]);
            acc[2 * c + 1] = fmaf(gg[c], b, acc[2 * c + 1]);
        }
    }
    __shared__ float red[2 * CH][8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int c = 0; c < 2 * CH; ++c) {
        float t = acc[c];
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) red[c][warp] = t;
    }
    __syncthreads();
    if (threadIdx.x < 2 * CH) {
        float t = 0.0f;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[threadIdx.x][w];
        atomicAdd(&dw[threadIdx.x * NTAP + tap], t);  // [c][k] flattened as c*2+k, times NTAP, plus tap
    }
}

// Two FP32 fused multiply-adds in one instruction.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    return (f32x2)__float_as_uint(lo) | ((f32x2)__float_as_uint(hi) << 32);
}
__device__ __forceinline__ float sum2(f32x2 v) {
    return __uint_as_float((unsigned)v) + __uint_as_float((unsigned)(v >> 32));
}
// Two BF16 values (low half first) as FP32.
__device__ __forceinline__ f32x2 unpack2(unsigned u) {
    return (f32x2)(u << 16) | ((f32x2)(u & 0xffff0000u) << 32);
}

// A warp's eight z positions x four groups of eight channels: lane = 4 z + group,
// so that a row access of the warp is 512 contiguous bytes.
//
// zhat = C_out(h); z = dinv * r + s_out * zhat (zhat kept for training). Each lane
// forms the partial sums of its channels for 4 x 2 outputs (x, y): a row that is
// loaded and unpacked serves up to six of them, and a weight two. Bound by
// instructions and their latency: 0.86 G products at 100^3 in 75 us; one output per
// thread unpacked every row 27 times and read a weight per product (275 us).
constexpr int OC_X = 4, OC_Y = 2;
__global__ void __launch_bounds__(128, 3) out_conv_kernel(const __nv_bfloat16* __restrict__ h, const float* __restrict__ w,
                                                       Vol v, const float* __restrict__ r,
                                                       const float* __restrict__ dinv, const float* s_out,
                                                       float* __restrict__ zhat, float* __restrict__ z) {
    __shared__ __align__(16) float ws[NTAP * CH];  // [tap][channel]
    for (int i = threadIdx.x; i < CH * NTAP; i += blockDim.x) ws[i] = w[(i % CH) * NTAP + i / CH];
    __syncthreads();
    const float so = s_out ? *s_out : 0.0f;
    const int lane = threadIdx.x & 31, cg = lane & 3;
    const int W2 = v.nz + 2;
    const long long P2 = (long long)(v.ny + 2) * W2;
    const unsigned ZT = (v.nz + 7) / 8, YT = (v.ny + OC_Y - 1) / OC_Y, XT = (v.nx + OC_X - 1) / OC_X;
    for (unsigned g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < ZT * YT * XT; g += gridDim.x * blockDim.x >> 5) {
        const unsigned col = g / ZT;
        const int zt = (int)(g - col * ZT), xt = (int)(col / YT), yt = (int)(col - xt * YT);
        const int x0 = xt * OC_X, y0 = yt * OC_Y, z0 = zt * 8 + (lane >> 2), zc = min(z0, v.nz - 1);
        f32x2 acc[OC_X][OC_Y] = {};
#pragma unroll 1
        for (int kz = 0; kz < 3; ++kz) {
            const float* wz = ws + kz * CH + cg * 8;
#pragma unroll
            for (int xi = 0; xi < OC_X + 2; ++xi) {
                const __nv_bfloat16* hp = h + (min(x0 + xi, v.nx + 1) * P2 + zc + kz) * CH + cg * 8;
                f32x2 row[OC_Y + 2][4];
#pragma unroll
                for (int yj = 0; yj < OC_Y + 2; ++yj) {
                    const uint4 u = *reinterpret_cast<const uint4*>(hp + (long long)min(y0 + yj, v.ny + 1) * W2 * CH);
                    row[yj][0] = unpack2(u.x);
                    row[yj][1] = unpack2(u.y);
                    row[yj][2] = unpack2(u.z);
                    row[yj][3] = unpack2(u.w);
                }
#pragma unroll
                for (int kx = 0; kx < 3; ++kx) {
                    const int i = xi - kx;
                    if (i < 0 || i >= OC_X) continue;
#pragma unroll
                    for (int ky = 0; ky < 3; ++ky) {
                        const float4 wa = *reinterpret_cast<const float4*>(wz + (kx * 9 + ky * 3) * CH);
                        const float4 wb = *reinterpret_cast<const float4*>(wz + (kx * 9 + ky * 3) * CH + 4);
                        const f32x2 w4[4] = {pack2(wa.x, wa.y), pack2(wa.z, wa.w), pack2(wb.x, wb.y),
                                             pack2(wb.z, wb.w)};
#pragma unroll
                        for (int j = 0; j < OC_Y; ++j)
#pragma unroll
                            for (int c = 0; c < 4; ++c) acc[i][j] = fma2(w4[c], row[j + ky][c], acc[i][j]);
                    }
                }
            }
        }
#pragma unroll
        for (int i = 0; i < OC_X; ++i)
#pragma unroll
            for (int j = 0; j < OC_Y; ++j) {
                float s = sum2(acc[i][j]);
                s += __shfl_xor_sync(0xffffffffu, s, 1);
                s += __shfl_xor_sync(0xffffffffu, s, 2);
                const int x = x0 + i, y = y0 + j;
                if (cg == i && x < v.nx && y < v.ny && z0 < v.nz) {  // lane group i stores column x0 + i
                    const long long e = ((long long)x * v.ny + y) * v.nz + z0;
                    if (zhat) zhat[e] = s;
                    if (z) z[e] = fmaf(so, s, dinv[e] * r[e]);
                }
            }
    }
}

// Backward of C_out (and C^T itself): dh[v][c] = sum_tap w[c][tap] * dzhat[v - s_tap]
// (BF16, interior rows). Each lane forms its eight channels of 2 x 2 voxels, so a
// weight that is read serves four of them and the rows leave as 16-byte stores:
// 61 us at 100^3, bound by instruction issue (71%); a thread per voxel read a
// weight per product (113 us).
constexpr int OD_X = 2, OD_Y = 2;
__global__ void __launch_bounds__(128, 5) out_conv_dgrad_kernel(const float* __restrict__ dz, const float* __restrict__ w,
                                                             Vol v, __nv_bfloat16* __restrict__ dh) {
    __shared__ __align__(16) float ws[NTAP * CH];  // [tap][channel]
    for (int i = threadIdx.x; i < CH * NTAP; i += blockDim.x) ws[i] = w[(i % CH) * NTAP + i / CH];
    __syncthreads();
    const int lane = threadIdx.x & 31, cg = lane & 3;
    const unsigned ZT = (v.nz + 7) / 8, YT = (v.ny + OD_Y - 1) / OD_Y, XT = (v.nx + OD_X - 1) / OD_X;
    for (unsigned g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < ZT * YT * XT; g += gridDim.x * blockDim.x >> 5) {
        const unsigned col = g / ZT;
        const int zt = (int)(g - col * ZT), xt = (int)(col / YT), yt = (int)(col - xt * YT);
        const int x0 = xt * OD_X, y0 = yt * OD_Y, z0 = zt * 8 + (lane >> 2);
        float acc[OD_X][OD_Y][8] = {};
        unsigned inside = 0;  // bit 4 xi + yj: column (x0 + xi - 1, y0 + yj - 1) is in the volume
#pragma unroll
        for (int xi = 0; xi < OD_X + 2; ++xi)
#pragma unroll
            for (int yj = 0; yj < OD_Y + 2; ++yj) {
                const int xx = x0 + xi - 1, yy = y0 + yj - 1;
                inside |= (xx >= 0 && xx < v.nx && yy >= 0 && yy < v.ny ? 1u : 0u) << (4 * xi + yj);
            }
        const float* corner = dz + ((long long)(x0 - 1) * v.ny + (y0 - 1)) * v.nz;  // read only where inside
        float in[OD_X + 2][OD_Y + 2][3];  // [..][..][kz]
#pragma unroll
        for (int kz = 0; kz < 3; ++kz) {
            const int zz = z0 + 1 - kz;
            const unsigned ok = zz >= 0 && zz < v.nz ? inside : 0u;
#pragma unroll
            for (int xi = 0; xi < OD_X + 2; ++xi)
#pragma unroll
                for (int yj = 0; yj < OD_Y + 2; ++yj)
                    in[xi][yj][kz] = (ok >> (4 * xi + yj)) & 1u ? __ldg(corner + (xi * v.ny + yj) * v.nz + zz) : 0.0f;
        }
        // in the order of the taps: the sums are rounded to BF16, and another order
        // would round some of them the other way
#pragma unroll
        for (int kx = 0; kx < 3; ++kx)
#pragma unroll
            for (int ky = 0; ky < 3; ++ky)
#pragma unroll
                for (int kz = 0; kz < 3; ++kz) {
                    const float* wt = ws + (kx * 9 + ky * 3 + kz) * CH + cg * 8;
                    const float4 wa = *reinterpret_cast<const float4*>(wt);
                    const float4 wb = *reinterpret_cast<const float4*>(wt + 4);
                    const float w8[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
#pragma unroll
                    for (int i = 0; i < OD_X; ++i)
#pragma unroll
                        for (int j = 0; j < OD_Y; ++j)
#pragma unroll
                            for (int c = 0; c < 8; ++c)
                                acc[i][j][c] = fmaf(w8[c], in[i + 2 - kx][j + 2 - ky][kz], acc[i][j][c]);
                }
#pragma unroll
        for (int i = 0; i < OD_X; ++i)
#pragma unroll
            for (int j = 0; j < OD_Y; ++j) {
                const int x = x0 + i, y = y0 + j;
                if (x >= v.nx || y >= v.ny || z0 >= v.nz) continue;
                uint4 u;
                __nv_bfloat162* b = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
                for (int c = 0; c < 4; ++c) b[c] = __floats2bfloat162_rn(acc[i][j][2 * c], acc[i][j][2 * c + 1]);
                *reinterpret_cast<uint4*>(dh + v.pad_row(x, y, z0) * CH + cg * 8) = u;
            }
    }
}

// dw[c][tap] += sum over voxels v of dz[v] h[v + s_tap][c]. Gathered by rows of h (its
// border is zero): each lane holds a row's eight channels once for the nine taps
// of its block's kd, and the nine values of dz slide along y, three new ones a row.
// The 72 sums of a lane are reduced over the warp's z positions every OW_FLUSH
// units, then over the block, and added with one atomic per weight and block: the
// blocks are large and the sums short so that the chains of FP32 additions stay
// no longer than before (error against 64 bits 2.0e-7 at 32^3, 1.4e-7 at 100^3;
// 2.3e-7, 1.7e-7 before). 32^3: 10.7 us, 100^3: 84 us, bound by latency and the
// shuffles; one tap per block unpacked every row 27 times (21.0 and 220 us).
constexpr int OW_Y = 8, OW_FLUSH = 6, OW_WARPS = 16;
__global__ void __launch_bounds__(OW_WARPS * 32, 1) out_conv_wgrad_kernel(const float* __restrict__ dz,
                                                                const __nv_bfloat16* __restrict__ h, Vol v,
                                                                float* __restrict__ dw) {
    const int kd = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int zl = lane >> 2, cg = lane & 3;
    const long long nzg = (v.nz + 7) / 8, nyc = (v.ny + OW_Y - 1) / OW_Y;
    __shared__ float red[OW_WARPS][4][72];
    for (int i = lane; i < 4 * 72; i += 32) red[warp][i / 72][i % 72] = 0.0f;
    __syncwarp();
    f32x2 acc[9][4];
    auto clear = [&]() {
#pragma unroll
        for (int t = 0; t < 9; ++t)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[t][c] = 0;
    };
    auto flush = [&]() {
#pragma unroll
        for (int t = 0; t < 9; ++t)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                float lo = __uint_as_float((unsigned)acc[t][c]), hi = __uint_as_float((unsigned)(acc[t][c] >> 32));
#pragma unroll
                for (int o = 4; o < 32; o <<= 1) {
                    lo += __shfl_xor_sync(0xffffffffu, lo, o);
                    hi += __shfl_xor_sync(0xffffffffu, hi, o);
                }
                if (zl == 0) {
                    red[warp][cg][t * 8 + 2 * c] += lo;
                    red[warp][cg][t * 8 + 2 * c + 1] += hi;
                }
            }
        clear();
    };
    clear();
    int n = 0;  // units since the last flush
    for (long long u = (long long)blockIdx.x * OW_WARPS + warp; u < nzg * nyc * v.nx; u += (long long)gridDim.x * OW_WARPS) {
        const int x = (int)(u / (nzg * nyc)), m = (int)(u - x * (nzg * nyc));
        const int z = (m % (int)nzg) * 8 + zl, y0 = (m / (int)nzg) * OW_Y, y1 = min(v.ny, y0 + OW_Y);
        const int vx = x - (kd - 1);
        if (vx < 0 || vx >= v.nx) continue;
        const float* plane = dz + (long long)vx * v.ny * v.nz + z;
        // dz at (vx, y, z + 1), z, z - 1: the taps kw = 0, 1, 2
        auto dz_row = [&](int y, float g[3]) {
            const bool in = y >= 0 && y < v.ny;
            const float* p = plane + (long long)y * v.nz;
            g[0] = in && z + 1 < v.nz ? p[1] : 0.0f;
            g[1] = in && z < v.nz ? p[0] : 0.0f;
            g[2] = in && z >= 1 && z <= v.nz ? p[-1] : 0.0f;
        };
        const uint4* rows = reinterpret_cast<const uint4*>(h + v.pad_row(x, y0, z < v.nz ? z : 0) * CH + cg * 8);
        const long long pitch = (long long)(v.nz + 2) * (CH / 8);
        auto h_row = [&](int y) {
            return y < y1 && z < v.nz ? rows[(y - y0) * pitch] : make_uint4(0u, 0u, 0u, 0u);
        };
        float ga[3], gb[3], gc[3], gn[3];
        dz_row(y0 - 1, ga);
        dz_row(y0, gb);
        dz_row(y0 + 1, gc);
        uint4 row = h_row(y0);
        for (int y = y0; y < y1; ++y) {
            const uint4 next = h_row(y + 1);
            dz_row(y + 2, gn);
            const f32x2 f[4] = {unpack2(row.x), unpack2(row.y), unpack2(row.z), unpack2(row.w)};
#pragma unroll
            for (int kw = 0; kw < 3; ++kw) {
                const f32x2 c2 = pack2(gc[kw], gc[kw]), b2 = pack2(gb[kw], gb[kw]), a2 = pack2(ga[kw], ga[kw]);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    acc[kw][c] = fma2(f[c], c2, acc[kw][c]);
                    acc[3 + kw][c] = fma2(f[c], b2, acc[3 + kw][c]);
                    acc[6 + kw][c] = fma2(f[c], a2, acc[6 + kw][c]);
                }
            }
            row = next;
#pragma unroll
            for (int kw = 0; kw < 3; ++kw) {
                ga[kw] = gb[kw];
                gb[kw] = gc[kw];
                gc[kw] = gn[kw];
            }
        }
        if (++n == OW_FLUSH) {
            flush();
            n = 0;
        }
    }
    if (n) flush();
    __syncthreads();
    for (int i = threadIdx.x; i < 4 * 72; i += blockDim.x) {
        const int g = i / 72, e = i % 72, t = e / 8, c = g * 8 + e % 8;
        float p[OW_WARPS];
#pragma unroll
        for (int w = 0; w < OW_WARPS; ++w) p[w] = red[w][g][e];
#pragma unroll
        for (int o = OW_WARPS / 2; o > 0; o /= 2)
#pragma unroll
            for (int w = 0; w < o; ++w) p[w] += p[w + o];
        atomicAdd(&dw[c * NTAP + kd * 9 + t], p[0]);
    }
}

// g = dh * [h > 0] over interior rows (BF16, padded layout).
__global__ void relu_mask_kernel(const __nv_bfloat16* __restrict__ dh, const __nv_bfloat16* __restrict__ h, Vol v,
                                 __nv_bfloat16* __restrict__ g) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < v.n(); i += (long long)gridDim.x * blockDim.x) {
        int x, y, z;
        decode(i, v, x, y, z);
        const long long q = v.pad_row(x, y, z) * CH;
        float a[CH], b[CH];
        load_row32(dh + q, a);
        load_row32(h + q, b);
#pragma unroll
        for (int c = 0; c < CH; ++c) a[c] = b[c] > 0.0f ? a[c] : 0.0f;
        store_row32(g + q, a);
    }
}

// acc[0] += sum r^2, acc[1] += sum dinv (multi-block, FP64 atomics).
__global__ void pc_sums_kernel(const float* __restrict__ r, const float* __restrict__ dinv, long long n, double* acc) {
    double a = 0.0, b = 0.0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        a += (double)r[i] * (double)r[i];
        b += (double)dinv[i];
    }
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    __shared__ double ra[8], rb[8];
    if ((threadIdx.x & 31) == 0) {
        ra[threadIdx.x >> 5] = a;
        rb[threadIdx.x >> 5] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        a = b = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            a += ra[w];
            b += rb[w];
        }
        atomicAdd(acc, a);
        atomicAdd(acc + 1, b);
    }
}

// s[0] = 1 / rms(r), s[1] = rms(r) * mean(dinv)
__global__ void pc_finalize_kernel(const double* acc, long long n, float* s) {
    const double rms = sqrt(acc[0] / (double)n);
    s[0] = rms > 0.0 ? (float)(1.0 / rms) : 0.0f;
    s[1] = (float)(rms * (acc[1] / (double)n));
}

// a = s_in * sqrt(dinv) * r
__global__ void pc_scale_in_kernel(const float* __restrict__ r, const float* __restrict__ dinv, const float* s,
                                   long long n, float* __restrict__ a) {
    const float si = s[0];
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        a[i] = si * sqrtf(dinv[i]) * r[i];
}

// z = dinv * r + (1 / s_in) * sqrt(dinv) * y
__global__ void pc_combine_kernel(const float* __restrict__ y, const float* __restrict__ r,
                                  const float* __restrict__ dinv, const float* s, long long n, float* __restrict__ z) {
    const float si = s[0];
    const float inv = si > 0.0f ? 1.0f / si : 0.0f;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        z[i] = fmaf(inv * sqrtf(dinv[i]), y[i], dinv[i] * r[i]);
}

// The same with a block of one tap: every row is unpacked 27 times, but 27 times the
// blocks share a small volume. 8^3 4.1 us (6.2 by rows), 16^3 6.2 (10.2).
__global__ void out_conv_wgrad_tap_kernel(const float* __restrict__ dz, const __nv_bfloat16* __restrict__ h, Vol v,
                                      float* __restrict__ dw) {
    const int tap = blockIdx.y;
    const int W2 = v.nz + 2, P2 = (v.ny + 2) * W2;
    const long long shift = (long long)(tap / 9 - 1) * P2 + ((tap / 3) % 3 - 1) * W2 + (tap % 3 - 1);
    float acc[CH];
#pragma unroll
    for (int c = 0; c < CH; ++c) acc[c] = 0.0f;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < v.n(); i += (long long)gridDim.x * blockDim.x) {
        int x, y, z;
        decode(i, v, x, y, z);
        const float g = dz[i];
        float f[CH];
        load_row32(h + (v.pad_row(x, y, z) + shift) * CH, f);
#pragma unroll
        for (int c = 0; c < CH; ++c) acc[c] = fmaf(g, f[c], acc[c]);
    }
    __shared__ float red[CH][8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int c = 0; c < CH; ++c) {
        float t = acc[c];
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) red[c][warp] = t;
    }
    __syncthreads();
    if (threadIdx.x < CH) {
        float t = 0.0f;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[threadIdx.x][w];
        atomicAdd(&dw[threadIdx.x * NTAP + tap], t);
    }
}

// CTAs of four warps, a warp per group of bx x by x 8 voxels, all at once up to 16 per SM.
unsigned grid_groups(const Vol& v, int bx, int by) {
    const long long g = (long long)((v.nz + 7) / 8) * ((v.ny + by - 1) / by) * ((v.nx + bx - 1) / bx);
    return (unsigned)std::max<long long>(1, std::min<long long>((g + 3) / 4, 152 * 16));
}

// Blocks of out_conv_wgrad_kernel: a warp per 8 x OW_Y rows, three kd, one wave of one per SM.
dim3 wgrad_grid(const Vol& v) {
    const long long units = (long long)((v.nz + 7) / 8) * ((v.ny + OW_Y - 1) / OW_Y) * v.nx;
    return dim3((unsigned)std::max<long long>(1, std::min<long long>((units + OW_WARPS - 1) / OW_WARPS, 152 / 3)), 3);
}

unsigned grid_for(long long n, int cap = 152 * 16) {
    return (unsigned)std::max<long long>(1, std::min<long long>((n + 255) / 256, cap));
}

int launch_out_wgrad(const float* dz, const void* h, const Vol& v, float* dw, cudaStream_t st) {
    const auto* hb = static_cast<const __nv_bfloat16*>(h);
    // 16^3 6.2 us by taps, 10.2 by rows; 18^3 8.2 both; 22^3 12.3, 10.2
    if (v.n() <= 5000) out_conv_wgrad_tap_kernel<<<dim3(grid_for(v.n(), 64), NTAP), 256, 0, st>>>(dz, hb, v, dw);
    else out_conv_wgrad_kernel<<<wgrad_grid(v), OW_WARPS * 32, 0, st>>>(dz, hb, v, dw);
    count_launch();
    ST_CUDA(cudaGetLastError());
    return ST_OK;
}

}  // namespace
}  // namespace stg

using namespace stg;

extern "C" {

int st_pc_in_conv(const float* r, const float* dinv, const float* scale, const float* w, void* h, int64_t nx,
                  int64_t ny, int64_t nz, void* stream) {
    ST_CHECK(r && dinv && scale && w && h, ST_ERR_ARG, "null argument");
    const Vol v{(int)nx, (int)ny, (int)nz};
    in_conv_kernel<<<grid_for(v.n()), 256, 0, (cudaStream_t)stream>>>(r, dinv, scale, w, v,
                                                                      static_cast<__nv_bfloat16*>(h));
    count_launch();
    ST_CUDA(cudaGetLastError());
    return ST_OK;
}

int st_pc_in_conv_wgrad(const float* r, const float* dinv, const float* scale, const void* g, float* dw, int64_t nx,
                        int64_t ny, int64_t nz, void* stream) {
    ST_CHECK(r && dinv && scale && g && dw, ST_ERR_ARG, "null argument");
    const Vol v{(int)nx, (int)ny, (int)nz};
    in_conv_wgrad_kernel<<<dim3(grid_for(v.n(), 64), NTAP), 256, 0, (cudaStream_t)stream>>>(
        r, dinv, scale, static_cast<const __nv_bfloat16*>(g), v, dw);
    count_launch();
    ST_CUDA(cudaGetLastError());
    return ST_OK;
}

int st_pc_out_conv(const void* h, const float* w, const float* r, const float* dinv, const float* s_out, float* zhat,
                   float* z, int64_t nx, int64_t ny, int64_t nz, void* stream) {
    ST_CHECK(h && w && (!z || (r && dinv && s_out)), ST_ERR_ARG, "null argument");
    const Vol v{(int)nx, (int)ny, (int)nz};
    out_conv_kernel<<<grid_groups(v, OC_X, OC_Y), 128, 0, (cudaStream_t)stream>>>(static_cast<const __nv_bfloat16*>(h), w,
                                                                                  v, r, dinv, s_out, zhat, z);
    count_launch();
    ST_CUDA(cudaGetLastError());
    return ST_OK;
}

int st_pc_out_conv_bwd(const float* dzhat, const void* h, const float* w, void* dh, float* dw, int64_t nx, int64_t ny,
                       int64_t nz, void* stream) {
    ST_CHECK(dzhat && h && w && dh && dw, ST_ERR_ARG, "null argument");
    const Vol v{(int)nx, (int)ny, (int)nz};
    cudaStream_t st = (cudaStream_t)stream;
    out_conv_dgrad_kernel<<<grid_groups(v, OD_X, OD_Y), 128, 0, st>>>(dzhat, w, v, static_cast<__nv_bfloat16*>(dh));
    count_launch();
    ST_CUDA(cudaGetLastError());
    return launch_out_wgrad(dzhat, h, v, dw, st);
}

int st_pc_relu_mask(const void* dh, const void* h, void* g, int64_t nx, int64_t ny, int64_t nz, void* stream) {
    ST_CHECK(dh && h && g, ST_ERR_ARG, "null argument");
    const Vol v{(int)nx, (int)ny, (int)nz};
    relu_mask_kernel<<<grid_for(v.n()), 256, 0, (cudaStream_t)stream>>>(static_cast<const __nv_bfloat16*>(dh),
                                                                        static_cast<const __nv_bfloat16*>(h), v,
                                                                        static_cast<__nv_bfloat16*>(g));
    count_launch();
    ST_CUDA(cudaGetLastError());
    return ST_OK;
}

int st_pc_scales(const float* r, const float* dinv, double* acc, float* scales, int64_t n, void* stream) {
    ST_CHECK(r && dinv && acc && scales, ST_ERR_ARG, "null argument");
    cudaStream_t st = (cudaStream_t)stream;
    ST_CUDA(cudaMemsetAsync(acc, 0, 2 * sizeof(double), st));
    pc_sums_kernel<<<grid_for(n, 152 * 4), 256, 0, st>>>(r, dinv, n, acc);
    count_launch();
    pc_finalize_kernel<<<1, 1, 0, st>>>(acc, n, scales);
    count_launch();
    ST_CUDA(cudaGetLastError());
    return ST_OK;
}

int st_pc_scale_in(const float* r, const float* dinv, const float* scales, float* a, int64_t n, void* stream) {
    ST_CHECK(r && dinv && scales && a, ST_ERR_ARG, "null argument");
    pc_scale_in_kernel<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(r, dinv, scales, n, a);
    count_launch();
    ST_CUDA(cudaGetLastError());
    return ST_OK;
}

int st_pc_combine(const float* y, const float* r, const float* dinv, const float* scales, float* z, int64_t n,
                  void* stream) {
    ST_CHECK(y && r && dinv && scales && z, ST_ERR_ARG, "null argument");
    pc_combine_kernel<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(y, r, dinv, scales, n, z);
    count_launch();
    ST_CUDA(cudaGetLastError());
    return ST_OK;
}

int st_pc_tconv1(const float* a, const float* w, void* h, int64_t nx, int64_t ny, int64_t nz, void* stream) {
    ST_CHECK(a && w && h, ST_ERR_ARG, "null argument");
    const Vol v{(int)nx, (int)ny, (int)nz};
    out_conv_dgrad_kernel<<<grid_groups(v, OD_X, OD_Y), 128, 0, (cudaStream_t)stream>>>(a, w, v,
                                                                                       static_cast<__nv_bfloat16*>(h));
    count_launch();
    ST_CUDA(cudaGetLastError());
    return ST_OK;
}

int st_pc_conv1_wgrad(const float* dz, const void* h, float* dw, int64_t nx, int64_t ny, int64_t nz, void* stream) {
    ST_CHECK(dz && h && dw, ST_ERR_ARG, "null argument");
    const Vol v{(int)nx, (int)ny, (int)nz};
    return launch_out_wgrad(dz, h, v, dw, (cudaStream_t)stream);
}

}  // extern "C"

// ---------------------------------------------------------------- network handle
// The trained preconditioner as one native object (weights packed once,
// activations allocated once), applied by st_pcnet_apply inside the native
// flexible CG. It is the symmetric positive (semi)definite form
//     z = D r + S G^T G S r,   D = diag(dinv), S = sqrt(D),
//     G = (I + conv_K) ... (I + conv_1) C^T,   C^T: 1 -> 32 channels,
// so G^T = C (I + conv_1^T) ... (I + conv_K^T): the tensor-core kernel with
// the transposed packing and the residual added. The input is scaled by
// 1 / rms(r) and the output back, which keeps z linear in r.

struct st_pcnet {
    int device = 0;
    int nx = 0, ny = 0, nz = 0, layers = 0;
    float* w_c = nullptr;      // C: [32][27]
    void* packed = nullptr;    // layers x 55,296 bytes (conv_k)
    void* packed_t = nullptr;  // layers x 55,296 bytes (conv_k^T)
    void* u = nullptr;         // two padded BF16 volumes (ping-pong)
    float* a = nullptr;        // scaled input / output, n floats
    double* acc = nullptr;
    float* scales = nullptr;
    size_t vol_bytes = 0;
};

namespace stg {
long long pcnet_points(const st_pcnet* p) { return (long long)p->nx * p->ny * p->nz; }
}  // namespace stg

extern "C" {

int st_pcnet_create(int64_t nx, int64_t ny, int64_t nz, int layers, int device, st_pcnet** out) {
    ST_CHECK(out && nx > 0 && ny > 0 && nz > 0 && layers >= 0 && layers <= 64, ST_ERR_ARG, "bad network shape");
    ST_CUDA(cudaSetDevice(device));
    st_pcnet* p = new st_pcnet();
    p->device = device;
    p->nx = (int)nx;
    p->ny = (int)ny;
    p->nz = (int)nz;
    p->layers = layers;
    p->vol_bytes = (size_t)(nx + 2) * (size_t)(ny + 2) * (size_t)(nz + 2) * CH * 2;
    const size_t wb = (size_t)std::max(layers, 1) * NTAP * CH * CH * 2;
    const size_t n = (size_t)(nx * ny * nz);
    const bool ok = cudaMalloc(&p->w_c, CH * NTAP * 4) == cudaSuccess && cudaMalloc(&p->packed, wb) == cudaSuccess &&
                    cudaMalloc(&p->packed_t, wb) == cudaSuccess &&
                    cudaMalloc(&p->u, 2 * p->vol_bytes) == cudaSuccess &&
                    cudaMalloc(&p->a, n * sizeof(float)) == cudaSuccess &&
                    cudaMalloc(&p->acc, 2 * sizeof(double)) == cudaSuccess &&
                    cudaMalloc(&p->scales, 2 * sizeof(float)) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        cudaFree(p->w_c);
        cudaFree(p->packed);
        cudaFree(p->packed_t);
        cudaFree(p->u);
        cudaFree(p->a);
        cudaFree(p->acc);
        cudaFree(p->scales);
        delete p;
        set_error("device allocation for the preconditioner network failed");
        return ST_ERR_ALLOC;
    }
    ST_CUDA(cudaMemset(p->u, 0, 2 * p->vol_bytes));
    ST_CUDA(cudaMemset(p->w_c, 0, CH * NTAP * 4));
    ST_CUDA(cudaMemset(p->packed, 0, wb));
    ST_CUDA(cudaMemset(p->packed_t, 0, wb));
    *out = p;
    return ST_OK;
}

int st_pcnet_destroy(st_pcnet* p) {
    if (!p) return ST_OK;
    cudaSetDevice(p->device);
    cudaDeviceSynchronize();
    cudaFree(p->w_c);
    cudaFree(p->packed);
    cudaFree(p->packed_t);
    cudaFree(p->u);
    cudaFree(p->a);
    cudaFree(p->acc);
    cudaFree(p->scales);
    delete p;
    return ST_OK;
}

// w_c: device FP32 [32][27]; w_k: `layers` consecutive [32][32][27] FP32 blocks.
int st_pcnet_set_weights(st_pcnet* p, const float* w_c, const float* w_k) {
    ST_CHECK(p && w_c && (p->layers == 0 || w_k), ST_ERR_ARG, "null argument");
    ST_CUDA(cudaSetDevice(p->device));
    ST_CUDA(cudaMemcpy(p->w_c, w_c, CH * NTAP * 4, cudaMemcpyDeviceToDevice));
    for (int k = 0; k < p->layers; ++k) {
        const float* w = w_k + (size_t)k * CH * CH * NTAP;
        const size_t off = (size_t)k * NTAP * CH * CH * 2;
        ST_TRY(st_conv3d_pack_weights(w, static_cast<char*>(p->packed) + off, 0, nullptr));
        ST_TRY(st_conv3d_pack_weights(w, static_cast<char*>(p->packed_t) + off, 1, nullptr));
    }
    ST_CUDA(cudaDeviceSynchronize());
    return ST_OK;
}

int st_pcnet_apply(st_pcnet* p, const float* r, const float* dinv, float* z, void* stream) {
    ST_CHECK(p && r && dinv && z, ST_ERR_ARG, "null argument");
    const long long n = (long long)p->nx * p->ny * p->nz;
    char* u0 = static_cast<char*>(p->u);
    char* u1 = u0 + p->vol_bytes;
    ST_TRY(st_pc_scales(r, dinv, p->acc, p->scales, n, stream));
    ST_TRY(st_pc_scale_in(r, dinv, p->scales, p->a, n, stream));
    ST_TRY(st_pc_tconv1(p->a, p->w_c, u0, p->nx, p->ny, p->nz, stream));
    const size_t wsz = (size_t)NTAP * CH * CH * 2;
    for (int k = 0; k < p->layers; ++k) {  // u <- (I + conv_k) u
        ST_TRY(st_conv3d_bf16(u0, static_cast<char*>(p->packed) + k * wsz, nullptr, u0, u1, 0, p->nx, p->ny, p->nz, 0,
                              stream));
        std::swap(u0, u1);
    }
    for (int k = p->layers - 1; k >= 0; --k) {  // u <- (I + conv_k^T) u
        ST_TRY(st_conv3d_bf16(u0, static_cast<char*>(p->packed_t) + k * wsz, nullptr, u0, u1, 0, p->nx, p->ny,
                              p->nz, 0, stream));
        std::swap(u0, u1);
    }
    ST_TRY(st_pc_out_conv(u0, p->w_c, nullptr, nullptr, nullptr, p->a, nullptr, p->nx, p->ny, p->nz, stream));
    return st_pc_combine(p->a, r, dinv, p->scales, z, n, stream);
}

}  // extern "C"
