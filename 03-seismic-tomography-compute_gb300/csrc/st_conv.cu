// 3x3x3 convolution of a 32-channel volume on the 5th-generation tensor
// cores (tcgen05), the building block of the learned CG preconditioner.
//
// Layout. A volume of D x H x W voxels is stored padded and channels-last:
// [(D+2) (H+2) (W+2)][32] BF16 (64 bytes per voxel), zero on the one-voxel
// border. Flattening the padded volume to rows q = (d*(H+2) + h)*(W+2) + w
// turns every tap (kd, kh, kw) of the stencil into a constant row shift
// s = (kd-1) PL + (kh-1)(W+2) + (kw-1), PL = (H+2)(W+2), and the zero border
// supplies the convolution's zero padding. So for a tile of 128 consecutive
// rows of one plane, out[128 x 32] = sum over 27 taps of
// in[rows + s][128 x 32] . W_tap[32 x 32]^T: an implicit GEMM with M = 128
// voxels, N = 32 output channels and K = 27 x 32.
//
// Layout of the contraction. With the voxels as the matrix unit's 128 rows and
// the 32 output channels as its columns, every instruction reads 4 KB of voxels
// from shared memory for 32 columns: the operand feed, not the multiply, set the
// pace (0.129 ms on a 100^3 volume, the multiply unit busy 18.5%). So the weights
// are the M operand and the voxels the N operand, and the three depth taps are
// stacked along M: one instruction multiplies N voxels of input plane p (shifted
// by one in-plane tap) by the 32 x 32 weights of kd = 2, 1, 0 for the output planes
// p - 1, p, p + 1. Output plane q lives in TMEM lanes 32 (q mod 4) .. + 31 (lane =
// channel, column = voxel), so a plane's three contributions meet in its block as
// the CTA marches along depth, and each input plane is read once. 100^3: 0.069 ms,
// 802 TFLOP/s (40% of BF16; a quarter of the M rows is disabled, and at 256 voxels
// the instruction's operands take three quarters of the shared-memory bandwidth
// that the epilogue needs as well); 32^3: 13 us, mostly start and end. The M rows are a
// window of four 32-row blocks into [kd2 kd1 kd0 - kd2 kd1 kd0], started at the
// block that puts kd2 on plane p - 1; the lanes of the fourth block, and of
// planes outside the CTA's range, are disabled for the instruction.
//
// Data path per CTA (persistent, one per SM, 18 warps). The work is cut into
// units: one in-plane tile position (N voxels) for a run of consecutive planes
// d0..d1-1, marched over the input planes d0-1..d1:
//   warp 0  loads per input plane the N + 2(W+3)-row
//           window ([row][32 channels], 64-byte swizzled: one copy of whole rows,
//           where 16-byte channel-block columns made the copy engine the bound at
//           four requests a row) into a ring of window slots;
//   warp 1  allocates N TMEM columns and issues 18 tcgen05.mma.kind::f16 (9
//           in-plane taps x 2 K steps; BF16 x BF16 -> FP32, M = 128, K = 16) per
//           input plane: every tap is a start row inside the window (the swizzle
//           goes by the address, and eight rows follow eight rows at 512 bytes);
//           the weights lie in the canonical no-swizzle K-major layout (8-row x
//           16-byte core matrices);
//   warps 2-17 epilogue, four warps per lane quarter (= block): when an output
//           plane is complete they read its block (tcgen05.ld), write zeros
//           back for the plane that takes the block next, and then, while the
//           matrix unit goes on, turn four voxels at a time through shared memory
//           (lane = channel in, four channels of a voxel out): + optional residual
//           input, + bias, optional ReLU, BF16 (or FP32) store of 8-byte pieces, zero
//           on border rows so the output keeps the padded convention. (Pairs of
//           channels exchanged by shuffles took four times the instructions and set
//           the pace: 82 us at 100^3.)
// Every mbarrier wait is bounded by a %globaltimer deadline: on expiry the
// kernel records CONV_FLAG_TIMEOUT, drains its own copies and MMAs (bounded
// too), frees TMEM and returns.
#include "st_common.cuh"

#include <algorithm>
#include <mutex>

namespace stg {
namespace {

constexpr int CH = 32;
constexpr int TM = 128;
constexpr int NTAP = 27;
constexpr int WB_BLOCK = CH * 16;                // 512 B: 32 output channels x 8 input channels
constexpr int WB_CB = 7 * WB_BLOCK;              // one channel block: kd2 kd1 kd0 - kd2 kd1 kd0
constexpr int WB_TAP = 4 * WB_CB;                // one in-plane tap
constexpr int W_BYTES = 9 * WB_TAP;              // 129,024
constexpr int MAX_SLOT = 3;
constexpr int MAX_WIDTH = 269;
constexpr int STAGE_FLOATS = 4 * CH;             // four voxels per epilogue warp (small: the windows want the room)
constexpr int EPI_WARPS = 16;                    // four per lane quarter
constexpr int CONV_THREADS = 64 + 32 * EPI_WARPS;
constexpr int SMEM_LIMIT = 232448;
constexpr unsigned CONV_FLAG_TIMEOUT = 1u;

struct ConvArgs {
    const void* w;          // packed weights (global, 16-byte aligned)
    const float* bias;      // [32] or null
    const __nv_bfloat16* add;  // residual input, padded layout, or null
    void* out;              // padded layout, BF16 or FP32
    int out_f32;
    int D, H, W;
    int relu;
    int rows_box, nload;    // TMA box rows and boxes per window column
    int nslot;              // window slots
    int tiles_per_plane;    // in-plane tile positions (units' columns)
    int dchunk, units;      // planes per unit, units = tiles_per_plane * ceil(D / dchunk)
    unsigned* flags;
    unsigned long long timeout_ns;
};

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ int read_abort(const int* p) { return *reinterpret_cast<const volatile int*>(p); }

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(smem_u32(bar))
        : "memory");
}

// Shared-memory matrix descriptor, canonical K-major layout without swizzle:
// start address, leading (K-direction) and stride (M/N-direction) byte
// offsets between 8-row x 16-byte core matrices, descriptor version 1.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// The same for K-major rows of 64 bytes, 64-byte swizzled, eight rows every 512
// bytes.
__device__ __forceinline__ uint64_t smem_desc_sw64(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(512u >> 4) << 32) | (1ull << 46) | (4ull << 61);
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, M = 128.
constexpr uint32_t idesc_n(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);
}
// Accumulating form that leaves the TMEM lanes set in off[] as they are; the
// descriptors as low and high words.
__device__ __forceinline__ void mma_bf16_lanes(uint32_t tmem_d, uint32_t alo, uint32_t ahi, uint32_t blo, uint32_t bhi,
                                               uint32_t idesc, const uint32_t off[4]) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, 1, 0;\n\tmov.b64 da, {%1, %2};\n\t"
        "mov.b64 db, {%3, %4};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, {%6, %7, %8, %9}, p;\n\t}" ::"r"(tmem_d),
        "r"(alo), "r"(ahi), "r"(blo), "r"(bhi), "r"(idesc), "r"(off[0]), "r"(off[1]), "r"(off[2]), "r"(off[3])
        : "memory");
}

// True in one lane of a converged warp.
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r != 0;
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 32 consecutive FP32 accumulator columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float v[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// Zeros into 32 consecutive columns of this warp's TMEM lanes.
__device__ __forceinline__ void tmem_zero32(uint32_t taddr) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, "
        "%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1};" ::"r"(taddr),
        "r"(0)
        : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

struct __align__(16) ConvSmem {
    uint64_t full[MAX_SLOT], empty[MAX_SLOT], tfull[4], tempty[4], done;
    uint32_t tmem_base;
    int abort;
};

// Unit u: in-plane tile column u % tiles_per_plane, planes [d0, d1).
struct ConvUnit {
    int col, d0, d1;
};
__device__ __forceinline__ ConvUnit unit_of(const ConvArgs& a, int u) {
    ConvUnit r;
    r.col = u % a.tiles_per_plane;
    r.d0 = (u / a.tiles_per_plane) * a.dchunk;
    r.d1 = min(a.D, r.d0 + a.dchunk);
    return r;
}

template <int N>
__global__ void __launch_bounds__(CONV_THREADS, 1)
    conv3d_tc_kernel(const __grid_constant__ CUtensorMap map, const ConvArgs a) {
    constexpr uint32_t ID = idesc_n(N);
    constexpr int HC = N / 4;  // columns of one epilogue warp
    extern __shared__ __align__(128) unsigned char smem_raw[];
    // the swizzle pattern repeats every 512 bytes: slots and boxes start on one
    unsigned char* smem = smem_raw + ((512u - (smem_u32(smem_raw) & 511u)) & 511u);
    const int W2 = a.W + 2;
    const int PL = (a.H + 2) * W2;
    const uint32_t box_bytes = (uint32_t)a.rows_box * (CH * 2);
    const uint32_t slot_bytes = box_bytes * (uint32_t)a.nload;  // one plane window
    unsigned char* wsm = smem;                                   // weights
    unsigned char* slots = smem + W_BYTES;                       // 512-byte aligned
    ConvSmem* cs = reinterpret_cast<ConvSmem*>(slots + a.nslot * slot_bytes);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint64_t lim = a.timeout_ns;
    const uint64_t dlim = lim > WAIT_DRAIN_NS ? lim : WAIT_DRAIN_NS;

    if (threadIdx.x == 0) {
        for (int s = 0; s < a.nslot; ++s) {
            mbar_init(&cs->full[s], 1);
            mbar_init(&cs->empty[s], 1);
        }
        for (int s = 0; s < 4; ++s) {
            mbar_init(&cs->tfull[s], 1);
            mbar_init(&cs->tempty[s], 128);
        }
        mbar_init(&cs->done, 1);
        cs->abort = 0;
        fence_mbar_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&cs->tmem_base)),
                     "r"(N)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = cs->tmem_base;
    // The weights, 16 bytes a thread and both of a block's places (512-byte bulk
    // copies, 216 of them, kept the copy engine busy for 10 us).
    {
        const uint4* src = static_cast<const uint4*>(a.w);  // [tap][channel block][32 rows] of 16 bytes
        for (int c = threadIdx.x; c < NTAP * CH * 4; c += CONV_THREADS) {
            const int tap = c >> 7, cb = (c >> 5) & 3, row = c & 31, kd = tap / 9, t = tap - 9 * kd;
            unsigned char* dst = wsm + t * WB_TAP + cb * WB_CB + (2 - kd) * WB_BLOCK + row * 16;
            const uint4 w = __ldg(src + c);
            *reinterpret_cast<uint4*>(dst) = w;
            *reinterpret_cast<uint4*>(dst + 4 * WB_BLOCK) = w;
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    // the epilogue warps' lane quarter and columns; the accumulators start at zero
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const uint32_t tlane = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * HC);
    if (warp >= 2) {
#pragma unroll
        for (int c = 0; c < HC; c += 32) tmem_zero32(tlane + (uint32_t)c);
        tmem_wait_st();
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();

    // Windows are numbered g = 0, 1, ... in the CTA's unit order; window g goes
    // to slot g % nslot. A unit of planes [d0, d1) takes d1 - d0 + 2 of them.
    if (warp == 0) {
        if (lane == 0) {
            int g = 0;
            bool stop = false;
            for (int u = blockIdx.x; u < a.units && !stop; u += gridDim.x) {
                const ConvUnit U = unit_of(a, u);
                const int p0 = U.col * N;
                const int nfill = U.d1 - U.d0 + 2;
                for (int j = 0; j < nfill; ++j, ++g) {
                    const int slot = g % a.nslot;
                    if (g >= a.nslot && !mbar_wait_bounded(&cs->empty[slot], ((g / a.nslot) - 1) & 1, lim)) {
                        atomicOr(a.flags, CONV_FLAG_TIMEOUT);
                        cs->abort = 1;
                        stop = true;
                        break;
                    }
                    if (read_abort(&cs->abort)) {
                        stop = true;
                        break;
                    }
                    unsigned char* sb = slots + slot * slot_bytes;
                    const int q0 = (U.d0 + j) * PL + p0 - (W2 + 1);
                    mbar_arrive_expect_tx(&cs->full[slot], slot_bytes);
                    for (int l = 0; l < a.nload; ++l)
                        tma_load_2d(sb + l * box_bytes, &map, &cs->full[slot], 0, q0 + l * a.rows_box);
                }
            }
            // drain: every issued window has landed before the CTA may exit
            for (int f = (g > a.nslot ? g - a.nslot : 0); f < g; ++f)
                if (!mbar_wait_bounded(&cs->full[f % a.nslot], (f / a.nslot) & 1, dlim))
                    atomicOr(a.flags, CONV_FLAG_TIMEOUT);
        }
    } else if (warp == 1) {
        // The whole warp runs the loop and one elected lane issues: addresses and
        // descriptors stay in uniform registers. Issued from a branch on the lane
        // number every instruction moved its nine operands there first (290
        // cycles each, whatever its size).
        bool ok = true;
        unsigned used = 0;  // four byte counts modulo 256: planes that have taken each block
        int g = 0;
        const uint32_t wb = smem_u32(wsm) >> 4, slots4 = smem_u32(slots) >> 4;
        const uint64_t adesc = smem_desc(0, WB_CB, 128u), bdesc = smem_desc_sw64(0);
        const uint32_t alo0 = (uint32_t)adesc, ahi = (uint32_t)(adesc >> 32), blo0 = (uint32_t)bdesc,
                       bhi = (uint32_t)(bdesc >> 32);
        const uint32_t rowstep = (uint32_t)W2 * (CH * 2u / 16u);
        for (int u = blockIdx.x; ok && u < a.units; u += gridDim.x) {
            const ConvUnit U = unit_of(a, u);
            for (int p = U.d0 - 1; p <= U.d1; ++p, ++g) {
                // a plane that starts here takes its block once that has been read and zeroed
                if (p + 1 < U.d1) {
                    const int sh = ((p + 1) & 3) * 8;
                    const unsigned n = (used >> sh) & 255u;
                    if (n > 0 && !__all_sync(0xffffffffu, mbar_wait_bounded(&cs->tempty[(p + 1) & 3], (n - 1) & 1, lim))) {
                        ok = false;
                        break;
                    }
                    // 255 wraps to 2, not to 0: the same parity, and a block once taken stays so
                    used = (used & ~(255u << sh)) | ((n == 255u ? 2u : n + 1) << sh);
                }
                const int slot = g % a.nslot;
                if (!__all_sync(0xffffffffu,
                                mbar_wait_bounded(&cs->full[slot], (g / a.nslot) & 1, lim) && !read_abort(&cs->abort))) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                uint32_t off[4];
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    // the output plane among p - 1 .. p + 2 that lives in block b
                    const int q = p - 1 + ((b - (p - 1)) & 3);
                    off[b] = (q <= p + 1 && q >= U.d0 && q < U.d1) ? 0u : 0xffffffffu;
                }
                const uint32_t alo = alo0 + wb + (uint32_t)((1 - p) & 3) * (WB_BLOCK / 16);
                const uint32_t blo = blo0 + slots4 + (uint32_t)slot * (slot_bytes >> 4);
                if (elect_one()) {
#pragma unroll
                    for (int t = 0; t < 9; ++t)
#pragma unroll
                        for (int ks = 0; ks < 2; ++ks)
                            mma_bf16_lanes(tmem, alo + (uint32_t)(t * (WB_TAP / 16) + ks * (2 * WB_CB / 16)), ahi,
                                           blo + (uint32_t)(t / 3) * rowstep + (uint32_t)((t % 3) * 4 + ks * 2), bhi, ID,
                                           off);
                    mma_commit(&cs->empty[slot]);
                    if (p - 1 >= U.d0) mma_commit(&cs->tfull[(p - 1) & 3]);
                }
                __syncwarp();
            }
        }
        if (!ok && lane == 0) {
            atomicOr(a.flags, CONV_FLAG_TIMEOUT);
            cs->abort = 1;
        }
        // drain: no MMA runs when TMEM is freed (commits of the lane that issued them)
        if (elect_one()) {
            mma_commit(&cs->done);
            if (!mbar_wait_bounded(&cs->done, 0, dlim)) atomicOr(a.flags, CONV_FLAG_TIMEOUT);
        }
        __syncwarp();
    } else {
        const int vl = lane >> 3, cg = lane & 7;  // the voxel of four and the four channels this lane stores
        float* stage = reinterpret_cast<float*>(cs + 1) + (warp - 2) * STAGE_FLOATS;
        float bias[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) bias[c] = a.bias ? a.bias[4 * cg + c] : 0.0f;
        int cnt = 0;
        bool stop = false;
        for (int u = blockIdx.x; u < a.units && !stop; u += gridDim.x) {
            const ConvUnit U = unit_of(a, u);
            const int pc = U.col * N + half * HC;  // in-plane position of this warp's first column
            unsigned inside[HC / 32], valid[HC / 32];
#pragma unroll
            for (int w = 0; w < HC / 32; ++w) {
                const int p = pc + 32 * w + lane, h = p / W2, x = p - h * W2;
                inside[w] = __ballot_sync(0xffffffffu, h >= 1 && h <= a.H && x >= 1 && x <= a.W) >> vl;
                valid[w] = __ballot_sync(0xffffffffu, p < PL) >> vl;
            }
            for (int d = U.d0 + ((quarter - U.d0) & 3); d < U.d1; d += 4, ++cnt) {
                // warp-uniform outcome: the TMEM accesses below are warp-collective
                const bool ok = __all_sync(0xffffffffu, mbar_wait_bounded(&cs->tfull[quarter], cnt & 1, lim));
                if (!ok) {
                    if (lane == 0) atomicOr(a.flags, CONV_FLAG_TIMEOUT);
                    cs->abort = 1;
                    stop = true;
                    break;
                }
                tc_fence_after();
                const long long q0 = ((long long)(d + 1) * PL + pc + vl) * CH + 4 * cg;
                float v[HC];
#pragma unroll
                for (int c = 0; c < HC; c += 32) tmem_ld32(tlane + (uint32_t)c, v + c);
#pragma unroll
                for (int c = 0; c < HC; c += 32) tmem_zero32(tlane + (uint32_t)c);
                tmem_wait_st();
                tc_fence_before();
                mbar_arrive(&cs->tempty[quarter]);  // the block is free for the plane after next
#pragma unroll
                for (int h = 0; h < HC / 4; h += 8) {  // eight groups' residual inputs in flight
                    uint2 add[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const int i = 4 * (h + k);
                        add[k] = make_uint2(0u, 0u);
                        if (a.add && ((inside[i / 32] >> (i % 32)) & 1u))
                            add[k] = *reinterpret_cast<const uint2*>(a.add + q0 + (long long)i * CH);
                    }
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const int i = 4 * (h + k);
                        __syncwarp();
#pragma unroll
                        for (int e = 0; e < 4; ++e) stage[e * CH + lane] = v[i + e];
                        __syncwarp();
                        float x[4];
                        *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(stage + vl * CH + 4 * cg);
                        const __nv_bfloat162* ab = reinterpret_cast<const __nv_bfloat162*>(&add[k]);
                        const bool ins = (inside[i / 32] >> (i % 32)) & 1u;
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const float2 f = __bfloat1622float2(ab[e]);
                            x[2 * e] = (x[2 * e] + f.x) + bias[2 * e];
                            x[2 * e + 1] = (x[2 * e + 1] + f.y) + bias[2 * e + 1];
                        }
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            if (a.relu) x[e] = fmaxf(x[e], 0.0f);
                            if (!ins) x[e] = 0.0f;
                        }
                        if ((valid[i / 32] >> (i % 32)) & 1u) {
                            const long long q = q0 + (long long)i * CH;
                            if (a.out_f32) {
                                *reinterpret_cast<float4*>(static_cast<float*>(a.out) + q) =
                                    make_float4(x[0], x[1], x[2], x[3]);
                            } else {
                                uint2 u;
                                __nv_bfloat162* b2 = reinterpret_cast<__nv_bfloat162*>(&u);
                                b2[0] = __floats2bfloat162_rn(x[0], x[1]);
                                b2[1] = __floats2bfloat162_rn(x[2], x[3]);
                                *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(a.out) + q) = u;
                            }
                        }
                    }
                }
            }
        }
    }
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(N) : "memory");
    }
}

// [co][ci][kd][kh][kw] FP32 (the usual conv weight order) -> packed BF16
// [tap][cb][co][8 ci]. transpose: the weights of the input gradient, i.e. the
// taps mirrored and in/out channels swapped.
__global__ void pack_weights_kernel(const float* __restrict__ w, __nv_bfloat16* __restrict__ out, int transpose) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= NTAP * CH * CH) return;
    const int tap = i / (CH * CH), r = i % (CH * CH), cb = r / (8 * CH), r2 = r % (8 * CH), co = r2 / 8,
              ci = cb * 8 + r2 % 8;
    float v;
    if (transpose) v = w[((size_t)ci * CH + co) * NTAP + (NTAP - 1 - tap)];
    else v = w[((size_t)co * CH + ci) * NTAP + tap];
    out[i] = __float2bfloat16_rn(v);
}

int num_sms_conv() {
    static int n = 0;
    if (n == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 1;
    }
    return n;
}

// The padded volume viewed as [rows][32 channels], box {32 channels, box_rows},
// 64-byte swizzled in shared memory.
int make_rows_map(CUtensorMap* map, const __nv_bfloat16* base, long long rows, int box_rows) {
    EncodeTiledFn enc = nullptr;
    ST_TRY(get_encode_tiled(&enc));
    cuuint64_t dims[2] = {CH, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)CH * 2};
    cuuint32_t box[2] = {CH, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<__nv_bfloat16*>(base), dims, strides, box,
                     estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    ST_CHECK(r == CUDA_SUCCESS, ST_ERR_CUDA, "cuTensorMapEncodeTiled (conv) failed (%d)", (int)r);
    return ST_OK;
}

// ---------------------------------------------------------------- weight gradient
// dW[co][ci][tap] += sum over interior voxels v of g[v][co] x[v + s_tap][ci]
// for a 32 -> 32 layer, on the tensor cores: an implicit GEMM with
// M = (kw, ci), N = co and K = the padded volume's rows q, cut into 9 tiles
// (kd, kh) and split over CTAs along K. g's border rows are zeroed on the way
// in, so a K step may run over them; x's border is zero by the padded
// convention, and rows past the volume arrive as zeros from the TMA bounds fill.
//
// Both operands are contiguous along their channels (M and N) in memory, and the
// matrix unit takes them so: a 64-byte swizzled tile of rows is its M-major
// layout, 32 channels wide, eight rows (K) every 512 bytes. The three kw taps are
// the same rows of x one row apart, so one window of x serves them: the M
// blocks of an instruction lie 64 bytes, one row, apart (the fourth, kw = 2, is
// not used). Per K step of 128 rows the TMA brings that window and g's rows into
// a ring of slots, warps 2-5 zero g's border rows, and warp 1 issues eight
// tcgen05.mma (M = 128, N = 32, K = 16), in turn into four accumulators so that
// no sum runs longer than a quarter of the K range. The epilogue adds the four,
// turns them through shared memory and adds them to dW (FP32 atomics, three
// neighbouring taps each). Every wait is bounded as in the forward conv.
//
// 32^3: 13.3 us, 100^3: 176 us (316 TFLOP/s of the products counted, bound by the
// 32-column instructions, a quarter of whose rows is not used). Transposing both
// operands through registers (ldmatrix / stmatrix) to K-major tiles of four taps
// took 37.5 and 606 us, bound by the transposes and by the atomics of 44 partial
// sums per weight. Error against 64 bits 4.4e-7 and 1.7e-5 (7.7e-7 and 2.7e-5).
constexpr int WG_KSTEP = 128;
constexpr int WG_TILES = 9;
constexpr int WG_SLOTS = 6;
constexpr int WG_X_ROWS = WG_KSTEP + 8;              // kw = -1 .. 2, in whole groups of eight rows
constexpr int WG_X_BYTES = WG_X_ROWS * CH * 2;
constexpr int WG_SLOT_BYTES = WG_X_BYTES + WG_KSTEP * CH * 2;
constexpr int WG_ACC = 4;
constexpr int WG_THREADS = 192;
constexpr int WG_TMEM_COLS = WG_ACC * CH;
static_assert(WG_X_BYTES % 512 == 0 && WG_SLOT_BYTES % 512 == 0, "swizzle blocks");

struct WgradArgs {
    float* dw;
    int D, H, W;
    int ksteps;      // ceil((D+2)(H+2)(W+2) / WG_KSTEP)
    int splits;      // CTAs per tile
    unsigned* flags;
    unsigned long long timeout_ns;
};

struct WgradSmem {
    uint64_t full[WG_SLOTS], ready[WG_SLOTS], empty[WG_SLOTS], done;
    uint32_t tmem_base;
    int abort;
};

// Descriptor of an M-major (N-major) operand, 64-byte swizzled: blocks of 32
// channels every lbo bytes, groups of eight rows every 512 bytes.
__device__ __forceinline__ uint64_t smem_desc_mn64(uint32_t addr, uint32_t lbo) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(512u >> 4) << 32) |
           (1ull << 46) | (4ull << 61);
}
constexpr uint32_t WG_IDESC = idesc_n(CH) | (1u << 15) | (1u << 16);  // A and B M- / N-major

__device__ __forceinline__ void mma_bf16_words(uint32_t tmem_d, uint32_t alo, uint32_t ahi, uint32_t blo, uint32_t bhi,
                                               uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %6, 0;\n\tmov.b64 da, {%1, %2};\n\t"
        "mov.b64 db, {%3, %4};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t}" ::"r"(tmem_d),
        "r"(alo), "r"(ahi), "r"(blo), "r"(bhi), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void named_sync_128() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

__global__ void __launch_bounds__(WG_THREADS, 1)
    conv32_wgrad_tc_kernel(const __grid_constant__ CUtensorMap mx, const __grid_constant__ CUtensorMap mg,
                           const WgradArgs a) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char* slots = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    WgradSmem* cs = reinterpret_cast<WgradSmem*>(slots + WG_SLOTS * WG_SLOT_BYTES);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x % WG_TILES, split = blockIdx.x / WG_TILES;
    const int k0 = (int)((long long)a.ksteps * split / a.splits);
    const int nk = (int)((long long)a.ksteps * (split + 1) / a.splits) - k0;
    const int W2 = a.W + 2;
    const int PL = (a.H + 2) * W2;
    const uint64_t lim = a.timeout_ns;
    const uint64_t dlim = lim > WAIT_DRAIN_NS ? lim : WAIT_DRAIN_NS;

    if (threadIdx.x == 0) {
        for (int s = 0; s < WG_SLOTS; ++s) {
            mbar_init(&cs->full[s], 1);
            mbar_init(&cs->ready[s], 128);
            mbar_init(&cs->empty[s], 1);
        }
        mbar_init(&cs->done, 1);
        cs->abort = 0;
        fence_mbar_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&cs->tmem_base)),
                     "r"(WG_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = cs->tmem_base;

    if (warp == 0) {
        if (lane == 0) {
            const int shift = (tile / 3 - 1) * PL + (tile % 3 - 1) * W2 - 1;
            int k = 0;
            for (; k < nk; ++k) {
                const int s = k % WG_SLOTS;
                if (k >= WG_SLOTS && !mbar_wait_bounded(&cs->empty[s], ((k / WG_SLOTS) - 1) & 1, lim)) {
                    atomicOr(a.flags, CONV_FLAG_TIMEOUT);
                    cs->abort = 1;
                    break;
                }
                if (read_abort(&cs->abort)) break;
                const int q0 = (k0 + k) * WG_KSTEP;
                unsigned char* sb = slots + s * WG_SLOT_BYTES;
                mbar_arrive_expect_tx(&cs->full[s], WG_SLOT_BYTES);
                tma_load_2d(sb, &mx, &cs->full[s], 0, q0 + shift);
                tma_load_2d(sb + WG_X_BYTES, &mg, &cs->full[s], 0, q0);
            }
            // drain: every issued slot has landed before the CTA may exit
            for (int f = (k > WG_SLOTS ? k - WG_SLOTS : 0); f < k; ++f)
                if (!mbar_wait_bounded(&cs->full[f % WG_SLOTS], (f / WG_SLOTS) & 1, dlim))
                    atomicOr(a.flags, CONV_FLAG_TIMEOUT);
        }
    } else if (warp == 1) {
        // the whole warp runs the loop and one elected lane issues (as in the forward conv)
        bool ok = true;
        const uint32_t slots4 = smem_u32(slots) >> 4;
        const uint64_t ad = smem_desc_mn64(0, CH * 2), bd = smem_desc_mn64(WG_X_BYTES, 512);
        const uint32_t alo0 = (uint32_t)ad + slots4, ahi = (uint32_t)(ad >> 32), blo0 = (uint32_t)bd + slots4,
                       bhi = (uint32_t)(bd >> 32);
        for (int k = 0; k < nk; ++k) {
            const int s = k % WG_SLOTS;
            if (!__all_sync(0xffffffffu,
                            mbar_wait_bounded(&cs->ready[s], (k / WG_SLOTS) & 1, lim) && !read_abort(&cs->abort))) {
                ok = false;
                break;
            }
            tc_fence_after();
            const uint32_t off = (uint32_t)s * (WG_SLOT_BYTES / 16);
            if (elect_one()) {
#pragma unroll
                for (int j = 0; j < WG_KSTEP / 16; ++j)  // 16 rows of 64 bytes each
                    mma_bf16_words(tmem + (uint32_t)(j % WG_ACC) * CH, alo0 + off + j * 64u, ahi, blo0 + off + j * 64u, bhi,
                                   WG_IDESC, j >= WG_ACC || k > 0);
                mma_commit(&cs->empty[s]);
            }
            __syncwarp();
        }
        if (!ok && lane == 0) {
            atomicOr(a.flags, CONV_FLAG_TIMEOUT);
            cs->abort = 1;
        }
        // the last commit tracks every MMA issued: the accumulators are final
        // (and, after an abort, no MMA is left running when TMEM is freed)
        if (elect_one()) {
            mma_commit(&cs->done);
            if (!mbar_wait_bounded(&cs->done, 0, dlim)) atomicOr(a.flags, CONV_FLAG_TIMEOUT);
        }
        __syncwarp();
    } else {
        const int tt = threadIdx.x - 64;
        bool ok = true;
        for (int k = 0; k < nk; ++k) {
            const int s = k % WG_SLOTS;
            if (!mbar_wait_bounded(&cs->full[s], (k / WG_SLOTS) & 1, lim) || read_abort(&cs->abort)) {
                atomicOr(a.flags, CONV_FLAG_TIMEOUT);
                cs->abort = 1;
                ok = false;
                break;
            }
            // g rows outside the interior contribute nothing (rows past the volume are zero already)
            const unsigned q = (unsigned)(k0 + k) * WG_KSTEP + tt;
            const unsigned d = q / (unsigned)PL, rem = q - d * PL, h = rem / (unsigned)W2, w = rem - h * W2;
            if (d - 1u >= (unsigned)a.D || h - 1u >= (unsigned)a.H || w - 1u >= (unsigned)a.W) {
                uint4* row = reinterpret_cast<uint4*>(slots + s * WG_SLOT_BYTES + WG_X_BYTES + tt * (CH * 2));
#pragma unroll
                for (int j = 0; j < 4; ++j) row[j] = make_uint4(0u, 0u, 0u, 0u);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic writes read by the tensor cores
            mbar_arrive(&cs->ready[s]);
        }
        if (ok) ok = mbar_wait_bounded(&cs->done, 0, dlim) && !read_abort(&cs->abort);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok && lane == 0) {
            atomicOr(a.flags, CONV_FLAG_TIMEOUT);
            cs->abort = 1;
        }
        // every slot has been read: the sums go through the first one, [co][ci][kw]
        float* out = reinterpret_cast<float*>(slots);
        const int kw = warp & 3;  // TMEM lanes 32 kw .. : lane = ci
        if (ok && kw < 3) {
            tc_fence_after();
            float v[CH];
            tmem_ld32(tmem + ((uint32_t)(kw * 32) << 16), v);
#pragma unroll
            for (int i = 1; i < WG_ACC; ++i) {
                float t[CH];
                tmem_ld32(tmem + ((uint32_t)(kw * 32) << 16) + (uint32_t)i * CH, t);
#pragma unroll
                for (int co = 0; co < CH; ++co) v[co] += t[co];
            }
            tc_fence_before();
#pragma unroll
            for (int co = 0; co < CH; ++co) out[(co * CH + lane) * 3 + kw] = v[co];
        }
        named_sync_128();
        if (!read_abort(&cs->abort))
            for (int i = tt; i < CH * CH * 3; i += 128) {
                const int cc = i / 3;
                atomicAdd(&a.dw[(size_t)cc * NTAP + tile * 3 + (i - cc * 3)], out[i]);
            }
    }
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(WG_TMEM_COLS)
                     : "memory");
    }
}

__device__ unsigned g_conv_flags;

}  // namespace

}  // namespace stg

using namespace stg;

extern "C" {

int st_conv3d_pack_weights(const float* w, void* packed, int transpose, void* stream) {
    ST_CHECK(w && packed, ST_ERR_ARG, "null argument");
    ST_CHECK((reinterpret_cast<uintptr_t>(packed) & 15) == 0, ST_ERR_ARG, "packed weights not 16-byte aligned");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    pack_weights_kernel<<<(NTAP * CH * CH + 255) / 256, 256, 0, st>>>(w, static_cast<__nv_bfloat16*>(packed),
                                                                      transpose);
    count_launch();
    ST_CUDA(cudaGetLastError());
    return ST_OK;
}

int st_conv3d_bf16(const void* in, const void* packed_w, const float* bias, const void* add, void* out, int out_fp32,
                   int64_t D, int64_t H, int64_t W, int relu, void* stream) {
    ST_CHECK(in && packed_w && out, ST_ERR_ARG, "null argument");
    ST_CHECK(D > 0 && H > 0 && W > 0, ST_ERR_ARG, "bad volume extents");
    ST_CHECK(in != out && (!add || add != out), ST_ERR_ARG, "output must not alias the inputs");
    auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    ST_CHECK(al16(in) && al16(packed_w) && al16(out) && (!add || al16(add)), ST_ERR_ARG,
             "conv buffers must be 16-byte aligned");
    const long long W2 = W + 2, PL = (H + 2) * W2, rows = (D + 2) * PL;
    ST_CHECK(rows < (1ll << 31), ST_ERR_ARG, "volume too large");
    ST_CHECK(W <= MAX_WIDTH, ST_ERR_UNSUPPORTED, "volume width %lld too large for the conv tiles", (long long)W);
    // Voxels per instruction (256 or 128) and planes per unit: the fewest cycles
    // over the rounds of units on the SMs. A unit of dc planes takes dc + 2 input
    // planes of 18 instructions; one of 256 voxels measured 128 cycles, of 128 64
    // (of 64 49); a round's first window and last epilogue are not hidden. 100^3:
    // 256 voxels; volumes whose planes fill few tiles (32^3) take 128 so that more
    // SMs have work.
    const long long nsm = num_sms_conv();
    auto window = [&](int n, int* nl, int* rb) {
        // one plane's window: win rows, loaded as nl boxes of rb rows (<= 256, a
        // multiple of 8 so that every TMA destination stays 512-byte aligned)
        const long long win = n + 2 * (W2 + 1);
        *nl = (int)((win + 255) / 256);
        *rb = (int)((((win + *nl - 1) / *nl) + 7) / 8 * 8);
        while (*rb > 256) {
            ++*nl;
            *rb = (int)((((win + *nl - 1) / *nl) + 7) / 8 * 8);
        }
    };
    auto smem_of = [&](int n, int slots) {
        int nl, rb;
        window(n, &nl, &rb);
        return (size_t)W_BYTES + (size_t)slots * (CH * 2) * nl * rb + sizeof(ConvSmem) + EPI_WARPS * STAGE_FLOATS * 4 + 512;
    };
    int N = 0;
    long long best_cost = -1, best_dc = 1;
    for (int n = 256; n >= 128; n /= 2) {
        if (smem_of(n, n == 256 ? 2 : 1) > (size_t)SMEM_LIMIT) continue;  // 256: widths up to 197
        const long long tiles = (PL + n - 1) / n, mma = n / 2;
        for (long long dc = 1; dc <= D; ++dc) {
            const long long units = tiles * ((D + dc - 1) / dc);
            const long long cost = (units + nsm - 1) / nsm * ((dc + 2) * 18 * mma + 3000);
            if (best_cost < 0 || cost < best_cost) {
                best_cost = cost;
                best_dc = dc;
                N = n;
            }
        }
    }
    ST_CHECK(N > 0, ST_ERR_UNSUPPORTED, "volume width %lld too large for the conv tiles", (long long)W);
    int nload, rows_box;
    window(N, &nload, &rows_box);
    int nslot = MAX_SLOT;  // two from widths of 102 (256 voxels) and 165 (128), one from 263
    while (smem_of(N, nslot) > (size_t)SMEM_LIMIT) --nslot;
    const size_t smem = smem_of(N, nslot);
    const __nv_bfloat16* src = static_cast<const __nv_bfloat16*>(in);
    CUtensorMap map;
    ST_TRY(make_rows_map(&map, src, rows, rows_box));
    unsigned* flags = nullptr;
    ST_CUDA(cudaGetSymbolAddress(reinterpret_cast<void**>(&flags), g_conv_flags));
    ConvArgs a{};
    a.w = packed_w;
    a.bias = bias;
    a.add = static_cast<const __nv_bfloat16*>(add);
    a.out = out;
    a.out_f32 = out_fp32;
    a.D = (int)D;
    a.H = (int)H;
    a.W = (int)W;
    a.relu = relu;
    a.rows_box = rows_box;
    a.nload = nload;
    a.nslot = nslot;
    a.tiles_per_plane = (int)((PL + N - 1) / N);
    a.dchunk = (int)best_dc;
    a.units = (int)((long long)a.tiles_per_plane * ((D + a.dchunk - 1) / a.dchunk));
    a.flags = flags;
    a.timeout_ns = 2000000000ull;
    auto kern = N == 256 ? conv3d_tc_kernel<256> : conv3d_tc_kernel<128>;
    static std::mutex mu;
    static size_t configured[2] = {0, 0};
    {
        std::lock_guard<std::mutex> lk(mu);
        size_t& c = configured[N == 256 ? 1 : 0];
        if (c < smem) {
            ST_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            c = smem;
        }
    }
    const int grid = std::min(a.units, num_sms_conv());
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    kern<<<grid, CONV_THREADS, smem, st>>>(map, a);
    count_launch();
    ST_CUDA(cudaGetLastError());
    return ST_OK;
}

int st_conv3d_wgrad(const void* x, const void* g, float* dw, int64_t nx, int64_t ny, int64_t nz, void* stream) {
    ST_CHECK(x && g && dw, ST_ERR_ARG, "null argument");
    ST_CHECK(nx > 0 && ny > 0 && nz > 0, ST_ERR_ARG, "bad volume extents");
    auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    ST_CHECK(al16(x) && al16(g), ST_ERR_ARG, "conv buffers must be 16-byte aligned");
    const long long rows = (nx + 2) * (ny + 2) * (nz + 2);
    ST_CHECK(rows + (ny + 2) * (nz + 2) + nz + 3 < (1ll << 31), ST_ERR_ARG, "volume too large");
    CUtensorMap mx, mg;
    ST_TRY(make_rows_map(&mx, static_cast<const __nv_bfloat16*>(x), rows, WG_X_ROWS));
    ST_TRY(make_rows_map(&mg, static_cast<const __nv_bfloat16*>(g), rows, WG_KSTEP));
    unsigned* flags = nullptr;
    ST_CUDA(cudaGetSymbolAddress(reinterpret_cast<void**>(&flags), g_conv_flags));
    WgradArgs a{};
    a.dw = dw;
    a.D = (int)nx;
    a.H = (int)ny;
    a.W = (int)nz;
    a.ksteps = (int)((rows + WG_KSTEP - 1) / WG_KSTEP);
    // one CTA per SM over the 9 tiles, at least one K step each
    a.splits = std::max(1, std::min(a.ksteps, num_sms_conv() / WG_TILES));
    a.flags = flags;
    a.timeout_ns = 2000000000ull;
    const size_t smem = (size_t)WG_SLOTS * WG_SLOT_BYTES + sizeof(WgradSmem) + 1024;
    static std::once_flag once;
    static cudaError_t attr = cudaSuccess;
    std::call_once(once, [&] {
        attr = cudaFuncSetAttribute(conv32_wgrad_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    });
    ST_CUDA(attr);
    conv32_wgrad_tc_kernel<<<WG_TILES * a.splits, WG_THREADS, smem, static_cast<cudaStream_t>(stream)>>>(mx, mg, a);
    count_launch();
    ST_CUDA(cudaGetLastError());
    return ST_OK;
}

int st_conv3d_check(void* stream) {
    unsigned h = 0;
    ST_CUDA(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)));
    ST_CUDA(cudaMemcpyFromSymbol(&h, g_conv_flags, sizeof(h)));
    const unsigned zero = 0;
    ST_CUDA(cudaMemcpyToSymbol(g_conv_flags, &zero, sizeof(zero)));
    ST_CHECK(!(h & CONV_FLAG_TIMEOUT), ST_ERR_TIMEOUT, "a conv3d wait timed out");
    return ST_OK;
}

}  // extern "C"
