// Forward shot on a small grid as one launch: every block keeps a brick of the
// grid on its SM for all nt steps (u_t in registers, u_t and u_{t-1} in shared
// memory, the coefficient in either) and exchanges only the faces of its brick
// with the four neighbouring blocks.
//
// Such a grid is bound by latency: one launch per two steps costs 2.6 us per step
// at 48 x 40 x 56 and 6.9 us at 128^3, where the 24 MB it moves take 3.5 us from
// HBM and less from L2. Here a step costs its arithmetic plus one exchange
// through L2: 1.4 us and 4.2 us (0.4 and 2.9 us of it arithmetic, about 1 us from
// a block's send to its neighbour's receipt). Each exchanged value travels in
// one 8-byte word with the number of its step, so a word is read with its tag in
// one access and the exchange needs no fence, no flag and no grid barrier.
// Packed two-value arithmetic (24 fewer instructions per group) gained nothing:
// its constants cost the registers that keep the eight-plane variant from spilling.
#include "st_solver_impl.cuh"
#include "st_update.cuh"

#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

namespace stg {
namespace {

constexpr int RES_THREADS = 512;     // most threads of a block: 128 registers each
constexpr int RES_SMEM = 232448;     // shared memory a block can have
__host__ __device__ constexpr bool res_c_reg(int K) { return K <= 4; }  // c in registers
constexpr size_t RES_HEAD = 256;     // bytes ahead of the exchange words: arrival count, abort word
constexpr uint64_t RES_START_NS = 60000000000ull;  // all blocks resident (another kernel may hold SMs)
constexpr uint64_t RES_WAIT_NS = 2000000000ull;    // a neighbour's step

// The split of the grid: PX x PY blocks of K x rows columns each.
struct ResPlan {
    int K = 0;              // x planes of a block (registers: 2 x 4K values per thread)
    int px = 0, py = 0;     // blocks
    int rows = 0;           // y rows of a block
    int nz4 = 0;            // groups of four z per column
    int threads = 0;        // rows * nz4 rounded up to whole warps
    size_t smem = 0;
    size_t bytes = 0;       // head and exchange words
};

struct ResArgs {
    StepArgs a;             // coefficients, sponge, limits, source position, receivers
    const float* c;         // device layout
    float* cur;             // u_nt, u_{nt-1}: interior written at the end
    float* prev;
    float* next;            // u_{next_step}, as launches of two steps leave the third field
    int next_step;
    const float* wav;       // nt + 1 values, NaN: no injection
    unsigned char* xch;     // head | per block and parity: xlo | xhi | ylo | yhi
    float* seis;
    int nt, nrec;
    int px, py, rows, nz4;
    unsigned base;          // tag of u_0
};

struct alignas(16) Word2 {
    unsigned long long a, b;
};

__device__ __forceinline__ void send2(unsigned char* p, float v0, float v1, unsigned tag) {
    const unsigned long long t = (unsigned long long)tag << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(t | __float_as_uint(v0)),
                 "l"(t | __float_as_uint(v1))
                 : "memory");
}
__device__ __forceinline__ Word2 recv2(const unsigned char* p) {
    Word2 w;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(w.a), "=l"(w.b) : "l"(p) : "memory");
    return w;
}
__device__ __forceinline__ unsigned load_relaxed(const unsigned* p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint64_t now_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// v = *p where cond, without a branch.
__device__ __forceinline__ void load_shared_if(bool cond, const float* p, float& v) {
    asm volatile("{\n\t.reg .pred c;\n\tsetp.ne.u32 c, %2, 0;\n\t@c ld.shared.f32 %0, [%1];\n\t}"
                 : "+f"(v)
                 : "r"(smem_u32(p)), "r"((unsigned)cond));
}

// A group of four values is two 16-byte words, the second `half` bytes after
// the first, so that a warp's accesses are contiguous.
__device__ __forceinline__ void send_group(unsigned char* p, unsigned half, const float v[4], unsigned tag) {
    send2(p, v[0], v[1], tag);
    send2(p + half, v[2], v[3], tag);
}

// A group to be received; p null: none.
struct Pending {
    const unsigned char* p;
    unsigned half;
    Word2 w0, w1;
    __device__ __forceinline__ void issue() {
        w0 = recv2(p);
        w1 = recv2(p + half);
    }
    __device__ __forceinline__ bool ready(unsigned tag) const {
        return (unsigned)(w0.a >> 32) == tag && (unsigned)(w0.b >> 32) == tag && (unsigned)(w1.a >> 32) == tag &&
               (unsigned)(w1.b >> 32) == tag;
    }
    // Waits for the group of tag; false when the limit ran out or another block
    // gave up.
    __device__ __forceinline__ bool wait(unsigned tag, const unsigned* abort_word, uint64_t limit) {
        uint64_t t0 = 0;
        for (int i = 0; !ready(tag); ++i) {
            if (i == 256) {
                const uint64_t now = now_ns();
                if (t0 == 0) t0 = now;
                if (now - t0 > limit || load_relaxed(abort_word)) return false;
                i = 0;
            }
            issue();
        }
        return true;
    }
    __device__ __forceinline__ void get(float v[4]) const {
        v[0] = __uint_as_float((unsigned)w0.a);
        v[1] = __uint_as_float((unsigned)w0.b);
        v[2] = __uint_as_float((unsigned)w1.a);
        v[3] = __uint_as_float((unsigned)w1.b);
    }
};

// The guarded update of a group (a result beyond the amplitude limit or not
// finite), out of line: everything is still in shared memory (own: u_t of the
// group, pv: u_{t-1}, um / up: its x neighbours).
__device__ __noinline__ float4 guarded_group(const float* own, const float* pvp, const float* ump, const float* upp,
                                             int srow, bool first_z, bool last_z, float4 cv4, float Dx, float4 Dyz4,
                                             const ResArgs& r) {
    const StepArgs& a = r.a;
    float u[4], pv[4], um[4], up[4], ym[4], yp[4], cv[4], Dyz[4], D[4], res[4];
    ld4(own, u);
    ld4(pvp, pv);
    ld4(ump, um);
    ld4(upp, up);
    ld4(own - srow, ym);
    ld4(own + srow, yp);
    const float zm0 = first_z ? 0.0f : own[-1], zp3 = last_z ? 0.0f : own[4];
    f4_to(cv4, cv);
    f4_to(Dyz4, Dyz);
    sponge4f(Dx, Dyz, D);
    int fired = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float zm = k == 0 ? zm0 : u[k - 1], zp = k == 3 ? zp3 : u[k + 1], upd = D[k] * pv[k];
        res[k] = update_fast(u[k], upd, um[k], up[k], ym[k], yp[k], zm, zp, cv[k], a.ax, a.ay, a.az);
        if (!(fabsf(res[k]) <= a.amp))
            res[k] = guarded_body(u[k], upd, um[k], up[k], ym[k], yp[k], zm, zp, cv[k], a.ax, a.ay, a.az, a.amp, &fired);
    }
    if (a.stable_sponge) damp4(D, res);
    if (fired) atomicOr(a.flags, FLAG_GUARD);
    return make_float4(res[0], res[1], res[2], res[3]);
}

// Block (bx, by) owns planes [bx K, bx K + xcnt) and rows [by rows, by rows +
// ycnt); a thread owns the group of four z at (row, z4) of all K planes.
// Shared memory: the field of the brick with one halo row on either y side, two
// buffers: a step reads u_t from one and u_{t-1}, at the thread's own groups,
// from the other, and then writes u_{t+1} there (one barrier per step). u_t of
// the own groups and, up to four planes, c are in registers too. The x
// neighbours of a point are in the thread's own registers, or (first and last
// plane) received; the z neighbours across groups come by shuffle.
// What bounds a step is its instructions and the latency of the exchange, so the
// groups of a phase are independent of one another up to one common test for
// the guarded update. Registers must not spill: with this much shared memory
// the L1 that would hold them is a few KB.
// STABLE: the stable sponge rule (StepArgs::stable_sponge).
template <int K, bool STABLE>
__global__ void __launch_bounds__(RES_THREADS, 1) resident_shot_kernel(const __grid_constant__ ResArgs r) {
    extern __shared__ __align__(128) float smem[];
    constexpr bool C_REG = res_c_reg(K);
    const StepArgs& a = r.a;
    const int tid = threadIdx.x, T = blockDim.x, lane = tid & 31;
    const int bx = blockIdx.x % r.px, by = blockIdx.x / r.px;
    const int x0 = bx * K, y0 = by * r.rows;
    const int xcnt = min(K, a.nx - x0), ycnt = min(r.rows, a.ny - y0);
    const int srow = r.nz4 * 4, pitch = (r.rows + 2) * srow;
    float* const S0 = smem;
    float* const S1 = smem + K * pitch;
    float* const Xlo = smem + 2 * K * pitch + tid * 4;  // [T][4], [T][4]: the thread's own x halo groups
    float* const Xhi = Xlo + T * 4;
    float* const Cs = Xhi + T * 4;                          // [K][T][4] unless c is in registers
    float* const Dx = smem + 2 * K * pitch + (C_REG ? 2 : K + 2) * T * 4;  // [K]

    const int row = tid / r.nz4, z4 = tid - row * r.nz4;
    const bool act = row < ycnt;
    const int y = y0 + row, zc = z4 * 4;
    const int zvalid = min(4, a.nz - zc);
    const int own = (act ? row + 1 : 1) * srow + zc;  // of the thread's group in a plane of S
    const long long at0 = (x0 + 1) * a.plane + (long long)(y + 1) * a.NZP + zc + Layout::ZOFF;

    // where this block's faces arrive and where it sends its own
    const unsigned xhalf = T * 16, yhalf = K * r.nz4 * 16;
    const unsigned xbytes = 2 * xhalf, ybytes = 2 * yhalf;  // one face of one parity
    const unsigned par = 2 * (xbytes + ybytes);             // one parity of one block
    unsigned char* const words = r.xch + RES_HEAD;
    unsigned* const arrived = reinterpret_cast<unsigned*>(r.xch);
    unsigned* const abort_word = arrived + 1;
    const unsigned mine = blockIdx.x * 2 * par;  // offset of the block's xlo | xhi | ylo | yhi
    const bool has_xlo = bx > 0, has_xhi = bx + 1 < r.px, has_ylo = by > 0, has_yhi = by + 1 < r.py;
    const unsigned to_xlo = mine - 2 * par + xbytes + tid * 16;  // the left block's xhi
    const unsigned to_xhi = mine + 2 * par + tid * 16;           // the right block's xlo
    const unsigned to_ylo = mine - r.px * 2 * par + 2 * xbytes + ybytes + z4 * 16;
    const unsigned to_yhi = mine + r.px * 2 * par + 2 * xbytes + z4 * 16;
    const bool send_xlo = act && has_xlo, send_xhi = act && has_xhi;
    const bool send_ylo = act && has_ylo && row == 0, send_yhi = act && has_yhi && row == ycnt - 1;
    const bool warp_y = __any_sync(0xffffffffu, send_ylo || send_yhi);

    // the halo rows: nface groups per side, shared out over the threads; the
    // first group of each thread is set up here (dst: its place in a buffer of S)
    const int nface = xcnt * r.nz4;
    const int nyg = ((has_ylo ? 1 : 0) + (has_yhi ? 1 : 0)) * nface;
    auto y_group = [&](int j, unsigned& src, int& dst) {
        const bool hi = !has_ylo || j >= nface;
        const int i = hi && has_ylo ? j - nface : j;
        const int k = i / r.nz4, z = i - k * r.nz4;
        src = 2 * xbytes + (hi ? ybytes : 0) + i * 16;
        dst = k * pitch + (hi ? (ycnt + 1) * srow : 0) + z * 4;
    };
    unsigned ysrc = 0;
    int ydst = 0;
    if (tid < nyg) y_group(tid, ysrc, ydst);

    // sponge: D(min distance) as the smaller of the x and the y/z factor
    float Dyz[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int d = min(min(y, a.ny - 1 - y), min(zc + j, a.nz - 1 - zc - j));
        Dyz[j] = d >= 0 && d < a.sw ? a.dtab[d] : 1.0f;
        if (!act) Dyz[j] = 0.0f;  // keeps a thread without points at 0
    }
    if (tid < K) {
        const int d = min(x0 + tid, a.nx - 1 - x0 - tid);
        Dx[tid] = d >= 0 && d < a.sw ? a.dtab[d] : 1.0f;
    }

    // receivers of the group: planes rmask, numbered from ir0 on; and the source
    unsigned rmask = 0;
    int ir0 = 0, iry = 0;
    const int rk = a.rz - zc;
    if (act && r.seis && rk >= 0 && rk < 4) {
        const int dy = y - a.ry0;
        if (dy >= 0 && dy % a.rsy == 0 && dy / a.rsy < a.rny) {
            iry = dy / a.rsy;
            for (int k = xcnt - 1; k >= 0; --k) {
                const int dx = x0 + k - a.rx0;
                if (dx >= 0 && dx % a.rsx == 0 && dx / a.rsx < a.rnx) {
                    rmask |= 1u << k;
                    ir0 = dx / a.rsx;
                }
            }
        }
    }
    const int inj_j = a.inj_z - zc;
    const bool src_here = act && y == a.inj_y && inj_j >= 0 && inj_j < 4 && a.inj_x >= x0 && a.inj_x < x0 + xcnt;
    const int inj_k = src_here ? a.inj_x - x0 : -1;
    const bool warp_src = __any_sync(0xffffffffu, src_here), warp_rec = __any_sync(0xffffffffu, rmask != 0);

    // z neighbours in another warp
    const bool first_z = z4 == 0, last_z = z4 + 1 == r.nz4;
    const bool load_zm = act && lane == 0 && z4 > 0, load_zp = act && lane == 31 && z4 + 1 < r.nz4;

    float u[K][4], C[C_REG ? K : 1][4];  // u_t, c
    for (int i = tid; i < 2 * K * pitch; i += T) smem[i] = 0.0f;
    const float none[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    st4(Xlo, none);
    st4(Xhi, none);
#pragma unroll
    for (int k = 0; k < K; ++k) {
        float cv[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (act && k < xcnt) ld4(r.c + at0 + k * a.plane, cv);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (j >= zvalid) cv[j] = 0.0f;  // with u = 0 these points stay 0 by themselves
            if constexpr (C_REG) C[k][j] = cv[j];
            u[k][j] = 0.0f;
        }
        if constexpr (!C_REG) st4(Cs + k * T * 4, cv);
    }
    __syncthreads();
    if (src_here) {
        const float w = r.wav[0];
        if (!isnan(w)) {
#pragma unroll
            for (int k = 0; k < K; ++k)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (k == inj_k && j == inj_j) u[k][j] += w;
            S0[inj_k * pitch + own + inj_j] += w;
        }
    }

    // all blocks run from here on
    bool ok = true;
    const bool lost = a.withhold < 0 && blockIdx.x == 0;  // the wait test: this block leaves after u_0
    if (tid == 0) {
        atomicAdd(arrived, 1u);
        const uint64_t t0 = now_ns();
        while (load_relaxed(arrived) < gridDim.x) {
            if (now_ns() - t0 > RES_START_NS) {
                ok = false;
                break;
            }
        }
        if (lost) ok = false;
    }

    // the faces of u_t, t the parity of the buffers
    auto receive = [&](int t, unsigned tag, float* S) {
        const unsigned char* in = words + mine + (t & 1) * par;
        Pending l{in + tid * 16, xhalf}, h{in + xbytes + tid * 16, xhalf}, g{in + ysrc, yhalf};
        if (send_xlo) l.issue();
        if (send_xhi) h.issue();
        if (tid < nyg) g.issue();
        float v[4];
        if (send_xlo) {
            ok = l.wait(tag, abort_word, a.timeout_ns) && ok;
            l.get(v);
            st4(Xlo, v);
        }
        if (send_xhi) {
            ok = h.wait(tag, abort_word, a.timeout_ns) && ok;
            h.get(v);
            st4(Xhi, v);
        }
        for (int j = tid; j < nyg; j += T) {
            int dst = ydst;
            if (j != tid) {
                unsigned src;
                y_group(j, src, dst);
                g.p = in + src;
                g.issue();
            }
            ok = g.wait(tag, abort_word, a.timeout_ns) && ok;
            g.get(v);
            st4(S + dst, v);
        }
    };

    // u_{t+1} of the group of plane k. Threads without points and planes beyond
    // the grid run it on zeros with a zero coefficient, so they stay 0 without a
    // mask; such threads store nothing.
    auto point = [&](int k, const float v[4], const float um[4], const float up[4], const float* Sc, const float* Sn,
                     float res[4], bool& bad) {
        const float* Sk = Sc + k * pitch + own;
        float zm0 = __shfl_up_sync(0xffffffffu, v[3], 1);
        float zp3 = __shfl_down_sync(0xffffffffu, v[0], 1);
        load_shared_if(load_zm, Sk - 1, zm0);
        load_shared_if(load_zp, Sk + 4, zp3);
        zm0 = first_z ? 0.0f : zm0;
        zp3 = last_z ? 0.0f : zp3;
        float pv[4], ym[4], yp[4], cv[4], D[4];
        ld4(Sn + k * pitch + own, pv);
        ld4(Sk - srow, ym);
        ld4(Sk + srow, yp);
        if constexpr (!C_REG) ld4(Cs + k * T * 4, cv);
        sponge4f(Dx[k], Dyz, D);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if constexpr (C_REG) cv[j] = C[k][j];
            res[j] = update_fast(v[j], D[j] * pv[j], um[j], up[j], ym[j], yp[j], j == 0 ? zm0 : v[j - 1],
                                 j == 3 ? zp3 : v[j + 1], cv[j], a.ax, a.ay, a.az);
            bad = bad || !(fabsf(res[j]) <= a.amp);
        }
        if constexpr (STABLE) {
#pragma unroll
            for (int j = 0; j < 4; ++j) res[j] *= D[j];
        }
    };
    auto guarded = [&](int k, const float* Sc, const float* Sn) {
        float cv[4] = {0.0f, 0.0f, 0.0f, 0.0f}, res[4];
        if constexpr (C_REG) {
#pragma unroll
            for (int j = 0; j < 4; ++j) cv[j] = C[k][j];
        } else {
            ld4(Cs + k * T * 4, cv);
        }
        if (act) {
            const float* Sk = Sc + k * pitch + own;
            f4_to(guarded_group(Sk, Sn + k * pitch + own, k == 0 ? Xlo : Sk - pitch, k == K - 1 ? Xhi : Sk + pitch, srow,
                                first_z, last_z, make_float4(cv[0], cv[1], cv[2], cv[3]), Dx[k],
                                make_float4(Dyz[0], Dyz[1], Dyz[2], Dyz[3]), r),
                  res);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) u[k][j] = act ? res[j] : 0.0f;
    };
    // receivers of u_{t+1}, all planes
    float* seis_t = r.seis + (size_t)ir0 * a.rny + iry;
    auto sample = [&]() {
        float* q = seis_t;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const float v01 = rk & 1 ? u[k][1] : u[k][0], v23 = rk & 1 ? u[k][3] : u[k][2];
            if (rmask >> k & 1u) {
                *q = rk & 2 ? v23 : v01;
                q += a.rny;
            }
        }
    };
    // receivers, then the source, of plane k (the source's warp)
    auto sample_inject = [&](int k, int t) {
        if (rmask >> k & 1u)
            seis_t[__popc(rmask & ((1u << k) - 1u)) * a.rny] =
                rk & 2 ? (rk & 1 ? u[k][3] : u[k][2]) : (rk & 1 ? u[k][1] : u[k][0]);
        if (k == inj_k) {
            const float w = r.wav[t + 1];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (j == inj_j && !isnan(w)) u[k][j] += w;
        }
    };
    // One step: the first and the last plane go first, so that their faces
    // travel while the others are updated.
    auto step = [&](int t, const float* Sc, float* Sn) {
        const unsigned tag = r.base + (unsigned)t + 1u;
        unsigned char* const out = words + ((t + 1) & 1) * par;
        float old0[4], oldL[4];  // u_t of the first and the last plane
        {
            float um[4], up[4], res0[4], resL[4];
            bool bad = false;
            ld4(Xlo, um);
            ld4(Xhi, up);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                old0[j] = u[0][j];
                oldL[j] = u[K - 1][j];
            }
            if constexpr (K == 1) {
                point(0, old0, um, up, Sc, Sn, resL, bad);
            } else {
                point(0, old0, um, u[1], Sc, Sn, res0, bad);
                point(K - 1, oldL, u[K - 2], up, Sc, Sn, resL, bad);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if constexpr (K > 1) u[0][j] = res0[j];
                u[K - 1][j] = resL[j];
            }
            if (bad) {
                guarded(0, Sc, Sn);
                if (K > 1) guarded(K - 1, Sc, Sn);
            }
        }
        if (warp_src) {
            sample_inject(0, t);
            if (K > 1) sample_inject(K - 1, t);
        }
        if (send_xlo) send_group(out + to_xlo, xhalf, u[0], tag);
        if (send_xhi) send_group(out + to_xhi, xhalf, u[K - 1], tag);
        if constexpr (K > 2) {
            bool bad = false;
            float um[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) um[j] = old0[j];
#pragma unroll
            for (int k = 1; k < K - 1; ++k) {
                float v[4], res[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] = u[k][j];
                point(k, v, um, k + 1 == K - 1 ? oldL : u[k + 1], Sc, Sn, res, bad);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    um[j] = v[j];
                    u[k][j] = res[j];
                }
            }
            if (bad) {
#pragma unroll
                for (int k = 1; k < K - 1; ++k) guarded(k, Sc, Sn);
            }
            if (warp_src) {
#pragma unroll
                for (int k = 1; k < K - 1; ++k) sample_inject(k, t);
            }
        }
        if (warp_y) {
            if (send_ylo) {
                unsigned char* p = out + to_ylo;
#pragma unroll
                for (int k = 0; k < K; ++k, p += r.nz4 * 16) send_group(p, yhalf, u[k], tag);
            }
            if (send_yhi) {
                unsigned char* p = out + to_yhi;
#pragma unroll
                for (int k = 0; k < K; ++k, p += r.nz4 * 16) send_group(p, yhalf, u[k], tag);
            }
        }
        if (act) {
#pragma unroll
            for (int k = 0; k < K; ++k) st4(Sn + k * pitch + own, u[k]);
        }
        if (warp_rec && !warp_src) sample();
        seis_t += r.nrec;
        if (t + 1 == r.next_step && act) {
#pragma unroll
            for (int k = 0; k < K; ++k)
                if (k < xcnt) st4(r.next + at0 + k * a.plane, u[k]);
        }
        if (t + 1 < r.nt) receive(t + 1, tag, Sn);
        return __syncthreads_or(!ok) != 0;
    };

    // u_0
    if (send_xlo) send_group(words + to_xlo, xhalf, u[0], r.base);
    if (send_xhi) send_group(words + to_xhi, xhalf, u[K - 1], r.base);
#pragma unroll
    for (int k = 0; k < K; ++k) {
        if (send_ylo) send_group(words + to_ylo + k * r.nz4 * 16, yhalf, u[k], r.base);
        if (send_yhi) send_group(words + to_yhi + k * r.nz4 * 16, yhalf, u[k], r.base);
    }
    bool dead = __syncthreads_or(!ok) != 0;
    if (!dead) {
        receive(0, r.base, S0);
        dead = __syncthreads_or(!ok) != 0;
    }
    for (int t = 0; t < r.nt && !dead; ++t) dead = step(t, t & 1 ? S1 : S0, t & 1 ? S0 : S1);
    if (dead) {
        if (tid == 0 && !lost) {
            atomicExch(abort_word, 1u);
            atomicOr(a.flags, FLAG_TIMEOUT);
        }
        return;
    }
    if (act) {
        const float* prev = r.nt & 1 ? S0 : S1;  // u_{nt-1}
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (k < xcnt) {
                float pv[4];
                ld4(prev + k * pitch + own, pv);
                st4(r.cur + at0 + k * a.plane, u[k]);
                st4(r.prev + at0 + k * a.plane, pv);
            }
        }
    }
}

// The split of an nx x ny x nz grid over at most nsm blocks, K = 0 when it does
// not fit: K planes and as few rows as the blocks allow, at most RES_THREADS
// groups of four z per plane and the brick in shared memory. Of the K that
// fit, the one whose step is shortest by the count of the instructions issued
// for the points, of the exchanged groups, and of the rounds in which a block
// receives its halo rows. Measured per step, K = 1 / 2 / 4 / 8 (x: does not fit):
// 24^3 1.43 / 1.53 / 2.11 / 3.45 us, 48 x 40 x 56 1.61 / 1.62 / 2.14 / 5.07,
// 64^3 2.05 / 1.73 / 1.80 / 3.63, 100^3 x / x / 2.52 / 3.54, 112^3 x / x / x / 3.88
// (5.97 by launches of two steps). Where even that K receives its halo rows in four
// rounds or more, launches of two steps are the faster ones: us per step resident / by
// launches, three rounds 40 x 40 x 500 3.9 / 4.2, 36 x 36 x 500 3.9 / 4.1; four 25 x 25 x
// 700 4.2 / 3.5, 16 x 16 x 1500 4.2 / 3.4, 60 x 60 x 400 5.9 / 5.8, 70 x 70 x 250 5.3 / 5.5;
// six 50 x 50 x 500 6.9 / 6.0; eight 20 x 20 x 1300 6.3 / 4.0.
ResPlan plan_resident(const Layout& L, int nsm) {
    ResPlan best;
    double best_cost = 0.0;
    long long best_rounds = 0;
    const long long nz4 = (L.nz + 3) / 4;
    for (int K : {1, 2, 4, 8}) {
        const long long px = (L.nx + K - 1) / K;
        if (px > nsm) continue;
        const long long py_max = std::min<long long>(nsm / px, L.ny);
        const long long rows = (L.ny + py_max - 1) / py_max, py = (L.ny + rows - 1) / rows;
        if (rows * nz4 > RES_THREADS) continue;
        const long long T = (rows * nz4 + 31) / 32 * 32;
        const long long smem = (2 * K * (rows + 2) * nz4 + (res_c_reg(K) ? 2 : K + 2) * T) * 16 + K * 4;
        if (smem > RES_SMEM) continue;
        const long long rounds = (2 * K * nz4 + T - 1) / T;
        const double cost = 0.8 * (double)(K * T) + 4.0 * (double)(T + K * nz4) + 600.0 * (double)(rounds - 1);
        if (best.K && cost >= best_cost) continue;
        best_cost = cost;
        best_rounds = rounds;
        best.K = K;
        best.px = (int)px;
        best.py = (int)py;
        best.rows = (int)rows;
        best.nz4 = (int)nz4;
        best.threads = (int)T;
        best.smem = (size_t)smem;
        best.bytes = RES_HEAD + (size_t)(px * py) * 2 * 64 * (size_t)(T + K * nz4);
    }
    if (best_rounds > 3) best.K = 0;
    return best;
}

using ResKernel = void (*)(const ResArgs);
template <bool STABLE>
ResKernel resident_kernel(int K) {
    return K == 1   ? resident_shot_kernel<1, STABLE>
           : K == 2 ? resident_shot_kernel<2, STABLE>
           : K == 4 ? resident_shot_kernel<4, STABLE>
                    : resident_shot_kernel<8, STABLE>;
}

}  // namespace

// Runs all nt steps of a shot without snapshots in one launch. *done = false:
// the grid does not fit, or the device cannot hold all its blocks at once, and
// nothing has been launched. The fields have been zeroed and cur = f[ic], prev = f[ip].
int resident_shot(st_solver* s, const StepArgs& a, const st_shot* shot, float* seis, bool* done) {
    *done = false;
    const Layout& L = s->L;
    int nsm = 0;
    ST_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, s->device));
    const ResPlan P = plan_resident(L, nsm);
    if (!P.K) return ST_OK;
    const ResKernel kernel = a.stable_sponge ? resident_kernel<true>(P.K) : resident_kernel<false>(P.K);
    // the exchange words (their tags rise from launch to launch) and the wavelet
    const int nt = shot->nt;
    const size_t wav_at = (P.bytes + 255) / 256 * 256, need = wav_at + sizeof(float) * ((size_t)nt + 1);
    const size_t had = s->res_cap;
    if (ensure_buffer(s, &s->res_buf, &s->res_cap, need) < 0) {
        cudaGetLastError();  // no room: the launches of two steps need none
        return ST_OK;
    }
    unsigned char* xch = static_cast<unsigned char*>(s->res_buf);
    if (s->res_cap != had || s->res_tag > 0xffffffffu - (unsigned)nt - 2u) {
        ST_CUDA(cudaMemsetAsync(xch, 0, P.bytes, s->stream));
        s->res_tag = 1;
    } else {
        ST_CUDA(cudaMemsetAsync(xch, 0, RES_HEAD, s->stream));
    }
    std::vector<float> wav((size_t)nt + 1, std::nanf(""));
    for (int t = 0; t < nt; ++t) {
        float w;
        if (finite_sample(shot->wavelet, shot->wavelet_len, t, &w)) wav[(size_t)t] = w;
    }
    ST_CUDA(cudaMemcpyAsync(xch + wav_at, wav.data(), sizeof(float) * wav.size(), cudaMemcpyHostToDevice, s->stream));

    ResArgs r{};
    r.a = a;
    r.a.nx = (int)L.nx;
    r.a.ny = (int)L.ny;
    r.a.nz = (int)L.nz;
    r.a.NZP = (int)L.NZP;
    r.a.plane = L.plane;
    if (r.a.timeout_ns == 0) r.a.timeout_ns = RES_WAIT_NS;
    r.c = s->c;
    r.cur = s->f[s->ic];
    r.prev = s->f[s->ip];
    r.next = s->f[s->in];
    r.next_step = nt % 2 ? nt - 2 : nt - 3;
    r.wav = reinterpret_cast<const float*>(xch + wav_at);
    r.xch = xch;
    r.seis = seis;
    r.nt = nt;
    r.nrec = (int)(shot->rec.nx * shot->rec.ny);
    r.px = P.px;
    r.py = P.py;
    r.rows = P.rows;
    r.nz4 = P.nz4;
    r.base = s->res_tag;

    ST_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, RES_SMEM));
    // One such launch at a time per device: each holds its SMs until its last step.
    constexpr int MAX_DEVICES = 64;
    static std::mutex mutex;
    static cudaEvent_t last[MAX_DEVICES] = {};
    if (s->device >= MAX_DEVICES) return ST_OK;
    std::lock_guard<std::mutex> lock(mutex);
    cudaEvent_t& ev = last[s->device];
    if (!ev) ST_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    ST_CUDA(cudaStreamWaitEvent(s->stream, ev, 0));
    void* args[] = {&r};
    const cudaError_t e = cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kernel), dim3(P.px * P.py),
                                                      dim3(P.threads), args, P.smem, s->stream);
    if (e == cudaErrorCooperativeLaunchTooLarge) {
        cudaGetLastError();
        return ST_OK;
    }
    ST_CUDA(e);
    ::stg::count_launch();
    s->res_tag += (unsigned)nt + 1u;
    ST_CUDA(cudaEventRecord(ev, s->stream));
    *done = true;
    return ST_OK;
}

}  // namespace stg
