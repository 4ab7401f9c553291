// nn_kernels.cu -- kernels of the learned warm start: a 3-D U-Net mapping the
// initial field B0 to a grid displacement x(X) - X.  Activations are BF16,
// channels-last ([voxel][channel], voxel = x + nx (y + ny z)), viewed with a
// channel stride so that a concatenation is two views into one buffer.  The
// 3x3x3 convolutions (forward, input gradient, weight gradient) are implicit
// GEMMs on the 5th-generation tensor cores with FP32 accumulation in tensor
// memory (nn_tc.cuh); padding is periodic in x and y and zero in z, as the
// relaxation's boundaries are.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "glemur.h"
#include "gm_internal.h"
#include "nn_tc.cuh"

namespace gmnn {

// ---- tensor-core GEMM check -------------------------------------------------

// D[128 x N] = A[128 x K] . B[N x K]^T with BF16 operands (row-major in global
// memory) and FP32 accumulation in tensor memory; one CTA of 128 threads.
// status[0] is set to 1 when the completion wait gives up.
__global__ void __launch_bounds__(128) k_tc_gemm(const __nv_bfloat16* __restrict__ A,
                                                 const __nv_bfloat16* __restrict__ B, float* __restrict__ D, int N,
                                                 int K, int* status) {
    extern __shared__ __align__(128) unsigned char sm[];
    unsigned char* sA = sm;                               // 128 x K
    unsigned char* sB = sm + 128 * K * 2;                 // N x K
    uint64_t* bar = reinterpret_cast<uint64_t*>(sB + N * K * 2);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int e = tid; e < 128 * K; e += 128) {
        const int r = e / K, k = e % K;
        *reinterpret_cast<__nv_bfloat16*>(sA + kmajor_off(r, k, K)) = A[e];
    }
    for (int e = tid; e < N * K; e += 128) {
        const int r = e / K, k = e % K;
        *reinterpret_cast<__nv_bfloat16*>(sB + kmajor_off(r, k, K)) = B[e];
    }
    if (tid == 0) mbar_init_tc(bar);
    fence_async_smem();
    uint32_t ncols = 32;
    while ((int)ncols < N) ncols <<= 1;
    if (warp == 0) tmem_alloc(tslot, ncols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = *tslot;
    if (tid == 0) {
        const uint32_t id = idesc_bf16(128, N);
        for (int kk = 0; kk < K / 16; kk++) {
            const uint64_t ad = smem_desc(sm_addr(sA) + kk * 256, 128, (uint32_t)K * 16);
            const uint64_t bd = smem_desc(sm_addr(sB) + kk * 256, 128, (uint32_t)K * 16);
            mma_bf16(tbase, ad, bd, id, kk > 0);
        }
        mma_commit(bar);
    }
    const bool ok = mbar_wait_tc(bar, 0);
    tc_fence_after();
    if (ok) {
        for (int c = 0; c < N; c += 16) {
            float v[16];
            tmem_ld16(tbase + ((uint32_t)(32 * warp) << 16) + (uint32_t)c, v);
#pragma unroll
            for (int q = 0; q < 16; q++) D[(32 * warp + lane) * N + c + q] = v[q];
        }
    } else if (lane == 0) {
        atomicExch(status, 1);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_free(tbase, ncols);
}

// ---- convolution: forward and input gradient --------------------------------

struct ConvArgs {
    const __nv_bfloat16* in1; int ld1, c1;   // first input view (channels 0 .. c1-1)
    const __nv_bfloat16* in2; int ld2, c2;   // optional second view (channels c1 .. c1+c2-1)
    const __nv_bfloat16* W;                  // [27][Np][Kc] BF16: rows = output channels, K = input channels
    const float* bias;                       // [Np] or null
    __nv_bfloat16* out; int ldo, co;         // output view (co channels written)
    const __nv_bfloat16* mask; int ldm;      // optional: out *= (mask > 0), mask has co channels
    int relu;
    int nx, ny, nz, xper, yper;
    int Kc, Np;                              // padded input channels (multiple of 16), padded outputs
    int Nt;                                  // output channels per CTA (multiple of 16; blockIdx.y picks the slice)
    int vec;                                 // out and mask rows start on 16 bytes: 8 channels an access
    int* status;
    int stall;                               // failure-detection test: wait on an mbarrier nothing arrives on
};

__device__ __forceinline__ int wrap(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }

// 16-byte asynchronous copy global -> shared (cp.async, L2 only), or 16 zero
// bytes when !valid (source size 0: nothing is read from src).
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Sixteen accumulators of voxel v, output channels c .. c + 15: bias, ReLU,
// mask, BF16; 8 channels a store (and mask load) where the views allow it.
__device__ __forceinline__ void conv_store16(const ConvArgs& a, long long v, int c, const float acc[16]) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int c8 = c + 8 * h;
        if (c8 >= a.co) break;
        if (a.vec && c8 + 8 <= a.co) {
            uint4 m = make_uint4(0, 0, 0, 0);
            if (a.mask) m = *reinterpret_cast<const uint4*>(a.mask + v * a.ldm + c8);
            const __nv_bfloat16* mb = reinterpret_cast<const __nv_bfloat16*>(&m);
            __nv_bfloat16 o[8];
#pragma unroll
            for (int q = 0; q < 8; q++) {
                float y = acc[8 * h + q] + (a.bias ? __ldg(a.bias + c8 + q) : 0.f);
                if (a.relu) y = fmaxf(y, 0.f);
                if (a.mask && !(__bfloat162float(mb[q]) > 0.f)) y = 0.f;
                o[q] = __float2bfloat16_rn(y);
            }
            *reinterpret_cast<uint4*>(a.out + v * a.ldo + c8) = *reinterpret_cast<const uint4*>(o);
        } else {
#pragma unroll
            for (int q = 0; q < 8; q++) {
                if (c8 + q >= a.co) break;
                float y = acc[8 * h + q] + (a.bias ? a.bias[c8 + q] : 0.f);
                if (a.relu) y = fmaxf(y, 0.f);
                if (a.mask && !(__bfloat162float(a.mask[v * a.ldm + c8 + q]) > 0.f)) y = 0.f;
                a.out[v * a.ldo + c8 + q] = __float2bfloat16_rn(y);
            }
        }
    }
}

// ---- convolution on resident input planes ---------------------------------------

// Every input plane is copied once, the weights are resident and each MMA serves three
// taps.  (Copying a tap's 128 voxels x K channels for every tap, 27 times the input,
// took 375 us for 24 -> 24 channels at 64x64x128, with 3 % tensor activity; this takes
// 38.)  A CTA takes items of 8 x 16 voxels and kz
// output planes and marches along z; an input plane of the tile with its halo
// (10 x 18 voxels) is copied into shared memory and all taps read it there.  In
// the K-major no-swizzle layout a row of a core matrix is the 16 bytes of 8
// channels of one voxel; with a plane stored as [8-channel group][y][x][16
// bytes], 8 rows along x are 128 contiguous bytes, 8-row groups (the next y) are
// one halo row apart (the descriptor's stride-dimension offset, 160 bytes) and
// the two core matrices of a K = 16 step one group apart (its leading-dimension
// offset), so an in-plane tap is nothing but another start address.  The three
// taps along z of an in-plane tap use the same 128 x 16 operand for the output
// planes p - 2, p - 1 and p: their weights are stacked along N and the
// accumulators of consecutive output planes lie in consecutive columns.  (An MMA
// takes 46 clocks up to N = 48, 57 at N = 96, N / 2 from N = 128 on.)
//
// Warps 0-3 read finished accumulators and store, warps 4-7 copy planes, warps 0-3 and
// 8-11 the weights of the CTA's output channels (all 27 taps, once), one thread of warp
// 12 issues the MMAs; they meet in mbarriers only.  With the copies, MMAs and stores of
// a step in one program order every step was a chain of about 9000 clocks around 2000
// clocks of MMAs.
constexpr int kTileX = 8, kTileY = 16, kHaloX = kTileX + 2, kSlots = kHaloX * (kTileY + 2);
constexpr int kMaxPlanes = 3, kMaxKz = 32;
constexpr int kPlaneThreads = 416, kCopyThreads = 128;

// Copies.  The layout scatters the 16-byte groups of a voxel or weight row over shared
// memory.  Asynchronous copies (cp.async) do that at 16 bytes a clock and SM whatever
// the order of lanes, but need few warps and no registers: the planes go that way, a
// warp taking 16 slots x 2 groups (32 bytes of a voxel) an instruction.  Loads into
// registers and stores are faster if many warps share the latency and neither side
// has conflicts: the weights go that way, the groups of a row in gl neighbouring
// lanes and the groups' stride in shared memory padded so that 8 such lanes write all
// 32 banks.
constexpr int kGroupBytes = kSlots * 16;       // one plane of 8 channels

struct ConvLanes {
    int ng, gl, sl;            // groups; lanes per row; rows per load of a warp
    __host__ __device__ explicit ConvLanes(int channels)
        : ng(channels >> 3), gl(ng >= 6 ? 8 : ng), sl(32 / gl) {}
    __host__ __device__ int row_stride(int rows) const { return rows * 16 + 128 / gl; }      // of a group (rows a multiple of 8)
};

struct ConvPlace { int x0, y0, z0, kz; };

__device__ __forceinline__ ConvPlace conv_place(int item, int tx, int ty, int kz, int nz) {
    ConvPlace q;
    q.x0 = item % tx * kTileX;
    q.y0 = item / tx % ty * kTileY;
    q.z0 = item / (tx * ty) * kz;
    q.kz = min(kz, nz - q.z0);
    return q;
}

// rows x L.ng groups of weights to shared memory at dst (group stride gs) by four
// warps, eight 16-byte loads of a thread in flight; src(r) is row r, or null for
// zeros.
template <class Src>
__device__ __forceinline__ void conv_copy_rows(const ConvLanes& L, int rows, uint32_t dst, int gs, int wq, int lane, Src src) {
    const int g0 = lane & (L.gl - 1), dr = 4 * L.sl;
    int r = wq * L.sl + lane / L.gl, g = g0;
    do {
        uint4 v[8];
        uint32_t d[8];
#pragma unroll
        for (int q = 0; q < 8; q++) {
            v[q] = make_uint4(0, 0, 0, 0);
            d[q] = 0;
            if (r < rows) {
                if (g < L.ng) {
                    d[q] = dst + g * gs + r * 16;
                    const __nv_bfloat16* p = src(r);
                    if (p) v[q] = __ldg(reinterpret_cast<const uint4*>(p + 8 * g));
                }
                g += L.gl;
                if (g - g0 >= L.ng) { g = g0; r += dr; }
            }
        }
#pragma unroll
        for (int q = 0; q < 8; q++)
            if (d[q])
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(d[q]), "r"(v[q].x), "r"(v[q].y), "r"(v[q].z),
                             "r"(v[q].w)
                             : "memory");
    } while (r < rows);
    fence_async_smem();
}

// The four warps that copy the planes of a CTA's items, in turn into NA buffers.  A
// plane's full barrier is arrived on once its copies have landed, when the next plane
// has been issued or before a wait (others may need the plane before that wait can
// end).  False when a wait ran out.
__device__ __forceinline__ bool conv_copy_planes(const ConvArgs& a, int tx, int ty, int items, int kz, int NA,
                                                 uint32_t stA, uint64_t* full, uint64_t* empty, int wq, int lane) {
    const int ng = a.Kc >> 3, gh = lane >> 4, planeBytes = ng * kGroupBytes;
    uint64_t* pending = nullptr;
    uint32_t n = 0;                                    // planes so far
    int buf = 0;
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
        const ConvPlace w = conv_place(item, tx, ty, kz, a.nz);
        // the voxels within a plane of this thread's slots 16 (wq + 4 q) + lane % 16:
        // halo points wrap, -1 for what is zero (beyond the domain)
        int vx[3];
#pragma unroll
        for (int q = 0; q < 3; q++) {
            const int s = 16 * (wq + 4 * q) + (lane & 15), sy = s / kHaloX;
            const int i = w.x0 + s - sy * kHaloX - 1, j = w.y0 + sy - 1;
            const bool in = s < kSlots && (i >= 0 || a.xper) && (j >= 0 || a.yper) && (i < a.nx || (a.xper && i == a.nx)) &&
                            (j < a.ny || (a.yper && j == a.ny));
            vx[q] = in ? wrap(i, a.nx) + a.nx * wrap(j, a.ny) : -1;
        }
        for (int p = 0; p < w.kz + 2; p++, n++) {
            if (n >= (uint32_t)NA && !mbar_test_tc(&empty[buf], n / NA - 1 & 1)) {
                if (pending) {
                    cp_async_wait<0>();
                    fence_async_smem();
                    mbar_arrive_tc(pending);
                    pending = nullptr;
                }
                if (!mbar_wait_tc(&empty[buf], n / NA - 1 & 1)) return false;
            }
            const int k = w.z0 + p - 1;
            const bool zin = k >= 0 && k < a.nz;
            const long long plane = (long long)a.nx * a.ny * (zin ? k : 0);
            const __nv_bfloat16* src = a.in1 + plane * a.ld1 + 8 * gh;
            const uint32_t dst = stA + buf * planeBytes + gh * kGroupBytes;
#pragma unroll
            for (int q = 0; q < 3; q++) {
                const int s = 16 * (wq + 4 * q) + (lane & 15);
                if (s >= kSlots) continue;
                const bool in = zin && vx[q] >= 0;
                const __nv_bfloat16* v = src + (long long)max(vx[q], 0) * a.ld1;
                const uint32_t d = dst + s * 16;
                if (a.c2 == 0) {
                    for (int g = 0; g < ng; g += 2) {
                        const bool on = in && 8 * (g + gh) < a.c1;
                        cp_async16(d + g * kGroupBytes, on ? v + 8 * g : a.in1, on);
                    }
                } else {
                    for (int g = 0; g < ng; g += 2) {
                        const int c = 8 * (g + gh) - a.c1;
                        const bool on = in && c < a.c2;
                        cp_async16(d + g * kGroupBytes, !on ? a.in1 : c < 0 ? v + 8 * g : a.in2 + (plane + vx[q]) * a.ld2 + c, on);
                    }
                }
            }
            cp_async_commit();
            if (pending) {
                cp_async_wait<1>();
                fence_async_smem();
                mbar_arrive_tc(pending);
            }
            pending = &full[buf];
            buf = buf + 1 == NA ? 0 : buf + 1;
        }
    }
    cp_async_wait<0>();
    if (pending) {
        fence_async_smem();
        mbar_arrive_tc(pending);
    }
    return true;
}

struct ConvPlaneArgs {
    ConvArgs a;                                // a.Nt: output channels per CTA
    int kz;                                    // output planes per item
    int tx, ty, items;                         // tiles along x, y; items (tiles x chunks along z)
    int ncols;                                 // tensor-memory columns, at least kz Nt
    int planes;                                // input planes in shared memory (2 .. kMaxPlanes)
};

// The mbarriers and shared scalars of a CTA, in front of its operands.
struct ConvPlaneShared {
    uint64_t full[kMaxPlanes], empty[kMaxPlanes];      // input planes: copied; read by the MMAs
    uint64_t wfull[9];                                 // the weights of an in-plane tap
    uint64_t afull[kMaxKz], aempty[kMaxKz];            // accumulators: complete; read
    uint64_t done, never;                              // all MMAs; nothing arrives on the last
    uint32_t tslot;
};
constexpr int kPlaneShared = (sizeof(ConvPlaneShared) + 127) / 128 * 128;

__global__ void __launch_bounds__(kPlaneThreads) k_conv_planes(const ConvPlaneArgs b) {
    extern __shared__ __align__(128) unsigned char sm[];
    ConvPlaneShared& sh = *reinterpret_cast<ConvPlaneShared*>(sm);
    const ConvArgs& a = b.a;
    const int Nt = a.Nt, n0 = blockIdx.y * Nt, Kc = a.Kc, NA = b.planes;
    const ConvLanes L(Kc);
    const int gs = kGroupBytes, rs = L.row_stride(3 * Nt), planeBytes = L.ng * gs, tapBytes = L.ng * rs;
    unsigned char* stB = sm + kPlaneShared;                    // 9 in-plane taps
    unsigned char* stA = stB + 9 * tapBytes;                   // NA planes
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int q = 0; q < NA; q++) { mbar_init_tc(&sh.full[q], kCopyThreads); mbar_init_tc(&sh.empty[q]); }
        for (int q = 0; q < 9; q++) mbar_init_tc(&sh.wfull[q], kCopyThreads);
        for (int q = 0; q < b.kz; q++) { mbar_init_tc(&sh.afull[q]); mbar_init_tc(&sh.aempty[q], 4); }
        mbar_init_tc(&sh.done);
        mbar_init_tc(&sh.never);
    }
    if (warp == 0) tmem_alloc(&sh.tslot, b.ncols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = sh.tslot;

    auto place = [&](int item) { return conv_place(item, b.tx, b.ty, b.kz, a.nz); };
    // failure-detection test: a bounded wait that runs out before any copy or MMA
    bool ok = a.stall ? mbar_wait_tc(&sh.never, 0, 1u << 10) : true;
    if (__syncthreads_and(ok)) {
        // the weights, before they have else to do, by warps 0-3 and 8-11: in-plane tap
        // u = 3 dj + di as rows [dk = +1 | 0 | -1] x Nt; rows beyond the channels are zero
        if (warp < 4 || (warp >= 8 && warp < 12))
            for (int u = warp >> 3; u < 9; u += 2) {
                conv_copy_rows(L, 3 * Nt, sm_addr(stB + u * tapBytes), rs, warp & 3, lane, [&](int r) {
                    const int dk = r >= 2 * Nt ? 2 : r >= Nt ? 1 : 0, o = n0 + r - dk * Nt;
                    return o < a.Np ? a.W + ((size_t)((2 - dk) * 9 + u) * a.Np + o) * Kc : nullptr;
                });
                mbar_arrive_tc(&sh.wfull[u]);
            }
        if (warp < 4) {
            // epilogue: output o of the item is the accumulator in columns o Nt ..
            uint32_t use = 0;
            for (int item = blockIdx.x; item < b.items && ok; item += gridDim.x, use ^= 1) {
                const ConvPlace w = place(item);
                const int i = w.x0 + (lane & 7), j = w.y0 + 4 * warp + (lane >> 3);
                const bool valid = i < a.nx && j < a.ny;
                const long long v = (long long)i + (long long)a.nx * (j + (long long)a.ny * w.z0);
                for (int o = 0; o < w.kz; o++) {
                    ok = __all_sync(~0u, mbar_wait_tc(&sh.afull[o], use));
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t col = tbase + ((uint32_t)(32 * warp) << 16) + (uint32_t)(o * Nt);
                    for (int c0 = 0; c0 < Nt; c0 += 16) {
                        float acc[16];
                        tmem_ld16(col + c0, acc);
                        if (c0 + 16 >= Nt) {
                            // the last read: the columns are free
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive_tc(&sh.aempty[o]);
                        }
                        if (valid) conv_store16(a, v + (long long)a.nx * a.ny * o, n0 + c0, acc);
                    }
                }
            }
        } else if (warp < 8) {
            ok = conv_copy_planes(a, b.tx, b.ty, b.items, b.kz, NA, sm_addr(stA), sh.full, sh.empty, warp & 3, lane);
        } else if (warp == 12 && elect_one()) {
            // MMAs.  The per-MMA arithmetic is adding to the low words of the
            // descriptors: what this thread does between two MMAs, the tensor core waits for
            uint32_t n = 0, use = 0;
            int buf = 0;
            const int ks = Kc / 16;
            const uint32_t ak = 2 * gs >> 4, bk = 2 * rs >> 4;
            const uint64_t bd0 = smem_desc(sm_addr(stB), rs, 128);
            for (int item = blockIdx.x; item < b.items && ok; item += gridDim.x, use ^= 1) {
                const ConvPlace w = place(item);
                for (int p = 0; p < w.kz + 2; p++, n++) {
                    const int lo = max(p - 2, 0), hi = min(p, w.kz - 1);
                    const bool fresh = p < w.kz;               // output p is new
                    if (fresh && item != (int)blockIdx.x) ok = mbar_wait_tc(&sh.aempty[p], use ^ 1);
                    ok = ok && mbar_wait_tc(&sh.full[buf], n / NA & 1);
                    const uint32_t d = tbase + lo * Nt, id = idesc_bf16(128, (hi - lo + 1) * Nt);
                    const uint64_t ad0 = smem_desc(sm_addr(stA + buf * planeBytes), gs, kHaloX * 16);
                    const uint64_t bdp = bd0 + (lo - p + 2) * Nt;
#pragma unroll
                    for (int u = 0; u < 9; u++) {
                        if (n == 0) ok = ok && mbar_wait_tc(&sh.wfull[u], 0);
                        if (!ok) break;
                        if (u == 0 || n == 0) tc_fence_after();
                        uint64_t ad = ad0 + u / 3 * kHaloX + u % 3, bd = bdp + (uint32_t)(u * (tapBytes >> 4));
                        int kk = 0;
                        if (fresh && u == 0) {
                            // the first product of output p does not accumulate
                            if (p > lo) mma_bf16(d, ad, bd, idesc_bf16(128, (p - lo) * Nt), true);
                            mma_bf16(tbase + p * Nt, ad, bd + (p - lo) * Nt, idesc_bf16(128, Nt), false);
                            ad += ak;
                            bd += bk;
                            kk = 1;
                        }
                        for (; kk < ks; kk++) {
                            mma_bf16(d, ad, bd, id, true);
                            ad += ak;
                            bd += bk;
                        }
                    }
                    if (!ok) break;
                    mma_commit(&sh.empty[buf]);
                    if (p >= 2) mma_commit(&sh.afull[p - 2]);
                    buf = buf + 1 == NA ? 0 : buf + 1;
                }
            }
            // every MMA has completed before the tensor memory is freed
            mma_commit(&sh.done);
            if (!mbar_wait_tc(&sh.done, 0)) ok = false;
        }
    }
    tc_fence_before();
    ok = __syncthreads_and(ok);
    if (!ok && tid == 0) atomicExch(a.status, 1);
    if (warp == 0) tmem_free(tbase, b.ncols);
}

// ---- convolution with many input channels -------------------------------------------

// The same with the weights streamed, for layers whose weights do not fit the
// shared memory: for each tap (along z first) and chunk of
// input channels a stage of Nt x kch weights, used for the kz output planes of
// the item; the planes in a ring of at least kz + 1 buffers with all channels.
// Warps 0-3 store, 4-7 copy planes, the next copy weights (the latency of
// their loads is what bounds a group), one thread of the last issues the MMAs.
constexpr int kWideGroups = 4, kWideThreads = 32 * (4 + 4 + 4 * kWideGroups + 1), kWideStages = 8, kWideKz = 4;

struct ConvWideArgs {
    ConvArgs a;                                // a.Nt: output channels per CTA
    int kz;                                    // output planes per item, at most kWideKz
    int tx, ty, items;
    int ncols, sets;                           // tensor-memory columns; accumulator sets (1 or 2) of kz Nt
    int planes;                                // plane buffers (kz + 1 ..)
    int kch, stages;                           // input channels per stage (divides Kc), stages
};

struct ConvWideShared {
    uint64_t full[kWideKz + 2], empty[kWideKz + 2];
    uint64_t wfull[kWideStages], wempty[kWideStages];
    uint64_t afull[2], aempty[2];
    uint64_t done, never;
    uint32_t tslot;
};
constexpr int kWideShared = (sizeof(ConvWideShared) + 127) / 128 * 128;

__global__ void __launch_bounds__(kWideThreads) k_conv_wide(const ConvWideArgs b) {
    extern __shared__ __align__(128) unsigned char sm[];
    ConvWideShared& sh = *reinterpret_cast<ConvWideShared*>(sm);
    const ConvArgs& a = b.a;
    const int Nt = a.Nt, n0 = blockIdx.y * Nt, Kc = a.Kc, NA = b.planes, S = b.stages, KCH = b.kch, nch = Kc / KCH;
    const ConvLanes L(Kc), LW(KCH);
    const int gs = kGroupBytes, rs = LW.row_stride(Nt), planeBytes = L.ng * gs, stepBytes = LW.ng * rs;
    unsigned char* stB = sm + kWideShared;
    unsigned char* stA = stB + S * stepBytes;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int q = 0; q < NA; q++) { mbar_init_tc(&sh.full[q], kCopyThreads); mbar_init_tc(&sh.empty[q]); }
        for (int q = 0; q < S; q++) { mbar_init_tc(&sh.wfull[q], kCopyThreads); mbar_init_tc(&sh.wempty[q]); }
        for (int q = 0; q < 2; q++) { mbar_init_tc(&sh.afull[q]); mbar_init_tc(&sh.aempty[q], 4); }
        mbar_init_tc(&sh.done);
        mbar_init_tc(&sh.never);
    }
    if (warp == 0) tmem_alloc(&sh.tslot, b.ncols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = sh.tslot;
    auto place = [&](int item) { return conv_place(item, b.tx, b.ty, b.kz, a.nz); };
    bool ok = a.stall ? mbar_wait_tc(&sh.never, 0, 1u << 10) : true;
    if (__syncthreads_and(ok)) {
        if (warp < 4) {
            uint32_t m = 0;                            // items so far
            for (int item = blockIdx.x; item < b.items; item += gridDim.x, m++) {
                const ConvPlace w = place(item);
                const int set = m % b.sets;
                ok = __all_sync(~0u, mbar_wait_tc(&sh.afull[set], m / b.sets & 1));
                if (!ok) break;
                tc_fence_after();
                const int i = w.x0 + (lane & 7), j = w.y0 + 4 * warp + (lane >> 3);
                const bool valid = i < a.nx && j < a.ny;
                const long long v = (long long)i + (long long)a.nx * (j + (long long)a.ny * w.z0);
                const uint32_t col = tbase + ((uint32_t)(32 * warp) << 16) + (uint32_t)(set * b.kz * Nt);
                for (int o = 0; o < w.kz; o++)
                    for (int c0 = 0; c0 < Nt; c0 += 16) {
                        float acc[16];
                        tmem_ld16(col + o * Nt + c0, acc);
                        if (o == w.kz - 1 && c0 + 16 >= Nt) {
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive_tc(&sh.aempty[set]);
                        }
                        if (valid) conv_store16(a, v + (long long)a.nx * a.ny * o, n0 + c0, acc);
                    }
            }
        } else if (warp < 8) {
            ok = conv_copy_planes(a, b.tx, b.ty, b.items, b.kz, NA, sm_addr(stA), sh.full, sh.empty, warp & 3, lane);
        } else if (warp < 8 + 4 * kWideGroups) {
            // weights: groups of four warps, a stage in turn.  All stages have one shape, so
            // a thread's at most eight 16-byte groups are worked out once (by the general
            // row copy the instructions of the copies were the kernel's bound: 240 -> 48
            // channels at 32x32x64 160 us, now 122)
            const int grp = (warp >> 2) - 2, t = tid & 127;
            uint32_t from[8], to[8];                   // ~0: none; rows beyond the channels are zero
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const int e = t + 128 * q, r = e / LW.ng, g = e - r * LW.ng;
                to[q] = r < Nt ? (uint32_t)(g * rs + r * 16) : ~0u;
                from[q] = r < Nt && n0 + r < a.Np ? (uint32_t)(r * Kc + 8 * g) : ~0u;
            }
            const uint32_t st0 = sm_addr(stB);
            int tap = 0, c = 0, st = 0;
            uint32_t turn = 0, round = 0;              // stages so far, rounds of the ring
            for (int item = blockIdx.x; item < b.items && ok; item += gridDim.x)
                for (int q = 0; q < 27 * nch && ok; q++, turn++) {
                    if (turn % kWideGroups == (uint32_t)grp) {
                        const __nv_bfloat16* W = a.W + ((size_t)tap * a.Np + n0) * Kc + c * KCH;
                        uint4 v[8];
#pragma unroll
                        for (int e = 0; e < 8; e++) {
                            v[e] = make_uint4(0, 0, 0, 0);
                            if (from[e] != ~0u) v[e] = __ldg(reinterpret_cast<const uint4*>(W + from[e]));
                        }
                        // (the loads are out before the wait)
                        ok = round == 0 || mbar_wait_tc(&sh.wempty[st], round - 1 & 1);
                        if (!ok) break;
#pragma unroll
                        for (int e = 0; e < 8; e++)
                            if (to[e] != ~0u)
                                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(st0 + st * stepBytes + to[e]),
                                             "r"(v[e].x), "r"(v[e].y), "r"(v[e].z), "r"(v[e].w)
                                             : "memory");
                        fence_async_smem();
                        mbar_arrive_tc(&sh.wfull[st]);
                    }
                    if (++st == S) { st = 0; round++; }
                    if (++c == nch) { c = 0; if (++tap == 27) tap = 0; }
                }
        } else if (elect_one()) {
            uint32_t n = 0, m = 0;                     // planes, items so far
            uint32_t wq = 0;                           // parity of the current round of stages
            int sq = 0;                                // stage
            const int ks = KCH / 16;
            const uint32_t id = idesc_bf16(128, Nt);
            const uint64_t ad00 = smem_desc(sm_addr(stA), gs, kHaloX * 16), bd00 = smem_desc(sm_addr(stB), rs, 128);
            const uint32_t ak = 2 * gs >> 4, bk = 2 * rs >> 4;
            for (int item = blockIdx.x; item < b.items && ok; item += gridDim.x, m++) {
                const ConvPlace w = place(item);
                const int set = m % b.sets;
                if (m >= (uint32_t)b.sets) ok = mbar_wait_tc(&sh.aempty[set], m / b.sets - 1 & 1);
                const uint32_t d0 = tbase + set * b.kz * Nt;
                int b0 = n % NA;                       // buffer of plane dk
                for (int dk = 0; dk < 3 && ok; dk++) {
                    // planes dk .. dk + kz - 1; those not yet waited for
                    for (int p = dk == 0 ? 0 : w.kz - 1 + dk; p < w.kz + dk; p++)
                        ok = ok && mbar_wait_tc(&sh.full[(n + p) % NA], (n + p) / NA & 1);
                    const uint32_t pstep = planeBytes >> 4;
                    for (int u = 0; u < 9 && ok; u++) {
                        const uint32_t tapoff = u / 3 * kHaloX + u % 3;
                        for (int c = 0; c < nch; c++) {
                            ok = mbar_wait_tc(&sh.wfull[sq], wq);
                            if (!ok) break;
                            tc_fence_after();
                            const uint64_t bdc = bd00 + (uint32_t)(sq * (stepBytes >> 4));
                            const uint32_t aoff = tapoff + c * (KCH / 8) * (gs >> 4);
                            const bool first = dk == 0 && u == 0 && c == 0;
                            uint32_t aplane = b0 * pstep;
                            for (int z = 0; z < w.kz; z++) {
                                uint64_t ad = ad00 + aplane + aoff, bd = bdc;
                                const uint32_t d = d0 + z * Nt;
                                for (int kk = 0; kk < ks; kk++) {
                                    mma_bf16(d, ad, bd, id, !first || kk > 0);
                                    ad += ak;
                                    bd += bk;
                                }
                                aplane = aplane == (NA - 1) * pstep ? 0 : aplane + pstep;
                            }
                            mma_commit(&sh.wempty[sq]);
                            if (++sq == S) { sq = 0; wq ^= 1; }
                        }
                    }
                    if (!ok) break;
                    b0 = b0 + 1 == NA ? 0 : b0 + 1;
                    for (int p = dk; p < (dk == 2 ? w.kz + 2 : dk + 1); p++) mma_commit(&sh.empty[(n + p) % NA]);
                }
                if (!ok) break;
                mma_commit(&sh.afull[set]);
                n += w.kz + 2;
            }
            mma_commit(&sh.done);
            if (!mbar_wait_tc(&sh.done, 0)) ok = false;
        }
    }
    tc_fence_before();
    ok = __syncthreads_and(ok);
    if (!ok && tid == 0) atomicExch(a.status, 1);
    if (warp == 0) tmem_free(tbase, b.ncols);
}

// ---- convolution: weight gradient --------------------------------------------

// dW[t][o][i] = sum_v dout[v][o] in[v + off(t)][i]: a GEMM over the voxels (K) with
// both operands MN-major, read as they lie: 16 bytes are 8 channels of one voxel,
// one row of a core matrix, and 8 voxels along x are a core matrix.  A CTA takes
// blocks of 8 x 16 voxels and kb planes, a slice of at most 3 groups of 8 input
// channels and a slice of at most 48 output channels.  The kb + 2 input planes of a
// block with their halo lie in shared memory one after the other as [8-channel
// group][y][x][16 bytes], so the groups of three consecutive planes are one run of
// equal strides: the three taps along z are stacked along M (3 planes x 3 groups x 8 = 72
// of 128 rows; the rows beyond read what follows and are dropped), and the nine
// in-plane taps are nine start addresses with an accumulator each (9 x 48 columns).
// An MMA takes 16 voxels (two rows along x: the K-direction offset is a halo row, 160
// bytes) against as many of the upstream gradient, [8-channel group][voxel][16 bytes].
// Accumulators stay in tensor memory over a chain of blocks and are then added to dW.
// (The tensor core's sums are truncated: the error grows with the products in a
// chain, 3e-6 of the gradient at 3500 voxels; kWgChain bounds it.)  Slices of 5 groups (120 rows) take
// fewer MMAs, but the copies bound them, as their planes leave room for two a block
// (72 -> 24 channels at 64x64x128: 195 us).
//
// With the 27 taps' rows copied one by one (27 times the input through cp.async, 16
// bytes a clock) this took 2700 of the 4200 us of a training step.
//
// Warps 0-3 add the accumulators of a finished chain to dW, warps 4-7 copy planes,
// 8-11 the upstream gradient, one thread of warp 12 issues the MMAs; an accumulator's
// next chain starts when it has been read.
constexpr int kWgKb = 6, kWgGroups = 3, kWgN = 48, kWgThreads = 416;
constexpr long long kWgChain = 22528;
constexpr int kDoutGroup = 128 * 16;           // one plane of 8 output channels

struct WgradArgs {
    const __nv_bfloat16* dout; int ldd, co;  // upstream gradient (channels up to co rounded to 8 readable)
    const __nv_bfloat16* in1; int ld1, c1;   // forward input views (channels up to ci rounded to 8 read)
    const __nv_bfloat16* in2; int ld2;
    float* dW;                               // [27][co][ci] FP32, accumulated with atomics
    int ci;
    int nx, ny, nz, xper, yper;
    int tx, ty, kb, blocks;                  // tiles along x, y; planes per block; blocks (tiles x chunks along z)
    int cs, cslices, N;                      // input groups per slice, slices; output channels per slice (MMA columns)
    int ncols;                               // tensor-memory columns, at least 9 N
    int chain;                               // blocks per chain
    int* status;
    int stall;                               // failure-detection test: wait on an mbarrier nothing arrives on
};

struct WgradShared {
    uint64_t full[2], empty[2];              // the two block buffers: copied; read by the MMAs
    uint64_t afull, aempty[9];               // the chain's MMAs; an in-plane tap's accumulator read
    uint64_t done, never;
    uint32_t tslot;
};
constexpr int kWgShared = 256;
static_assert(sizeof(WgradShared) <= kWgShared);

// Bytes of a block buffer: the planes, and the upstream gradient's.  (The MMAs read 16
// groups from the last three planes' start; what is beyond them lies in the rest of
// the shared memory, which wgrad_smem leaves room for.)
__host__ __device__ inline int wg_block_bytes(int cs, int kb, int N) {
    return (kb + 2) * cs * kGroupBytes + kb * (N / 8) * kDoutGroup;
}
inline size_t wgrad_smem(int cs, int kb, int N) {
    const size_t past = (size_t)(kb - 1) * cs * kGroupBytes + 16 * kGroupBytes;      // end of the last MMA's rows
    const size_t one = wg_block_bytes(cs, kb, N);
    return kWgShared + one + std::max(one, past);
}

__global__ void __launch_bounds__(kWgThreads) k_conv_wgrad(const WgradArgs a) {
    extern __shared__ __align__(128) unsigned char sm[];
    WgradShared& sh = *reinterpret_cast<WgradShared*>(sm);
    const int cs = a.cs, N = a.N, kb = a.kb, blockBytes = wg_block_bytes(cs, kb, N), planeBytes = cs * kGroupBytes;
    const int slice = blockIdx.y % a.cslices, o0 = blockIdx.y / a.cslices * N;
    const int c0 = slice * cs * 8;                             // first input channel of the slice
    const uint32_t st = sm_addr(sm) + kWgShared;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int q = 0; q < 2; q++) { mbar_init_tc(&sh.full[q], 256); mbar_init_tc(&sh.empty[q]); }
        mbar_init_tc(&sh.afull);
        for (int u = 0; u < 9; u++) mbar_init_tc(&sh.aempty[u], 4);
        mbar_init_tc(&sh.done);
        mbar_init_tc(&sh.never);
    }
    if (warp == 0) tmem_alloc(&sh.tslot, a.ncols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = sh.tslot;
    // failure-detection test: a bounded wait that runs out before any copy or MMA
    bool ok = a.stall ? mbar_wait_tc(&sh.never, 0, 1u << 10) : true;
    if (__syncthreads_and(ok)) {
        if (warp < 4) {
            // row 32 warp + lane: stacked group row / 8 = dk cs + group, channel row % 8
            const int row = 32 * warp + lane, sg = row >> 3, dk = sg / cs, ich = c0 + (sg - dk * cs) * 8 + (row & 7);
            const bool mine = dk < 3 && ich < a.ci;
            const int mine_blocks = (a.blocks - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
            for (int c = 0; c * a.chain < mine_blocks; c++) {
                ok = __all_sync(~0u, mbar_wait_tc(&sh.afull, c & 1));
                if (!ok) break;
                tc_fence_after();
                for (int u = 0; u < 9; u++) {
                    for (int n0 = 0; n0 < N; n0 += 16) {
                        float acc[16];
                        tmem_ld16(tbase + ((uint32_t)(32 * warp) << 16) + (uint32_t)(u * N + n0), acc);
                        if (n0 + 16 >= N) {
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive_tc(&sh.aempty[u]);
                        }
                        if (!mine) continue;
                        float* w = a.dW + ((size_t)(dk * 9 + u) * a.co + o0 + n0) * a.ci + ich;
#pragma unroll
                        for (int q = 0; q < 16; q++)
                            if (o0 + n0 + q < a.co) atomicAdd(w + (size_t)q * a.ci, acc[q]);
                    }
                    __syncwarp();
                }
            }
        } else if (warp < 12) {
            const int wq = warp & 3, gh = lane >> 4;
            uint64_t* pending = nullptr;
            auto flush = [&]() {
                if (!pending) return;
                cp_async_wait<0>();
                fence_async_smem();
                mbar_arrive_tc(pending);
                pending = nullptr;
            };
            uint32_t n = 0;
            for (int blk = blockIdx.x; blk < a.blocks && ok; blk += gridDim.x, n++) {
                const ConvPlace w = conv_place(blk, a.tx, a.ty, kb, a.nz);
                const int buf = n & 1;
                if (n >= 2 && !mbar_test_tc(&sh.empty[buf], (n >> 1) - 1 & 1)) {
                    flush();
                    ok = mbar_wait_tc(&sh.empty[buf], (n >> 1) - 1 & 1);
                    if (!ok) break;
                }
                const uint32_t dst = st + buf * blockBytes;
                if (warp < 8) {
                    // the planes z0 - 1 .. z0 + kz: slots 16 (wq + 4 q) + lane % 16, two groups a copy
#pragma unroll
                    for (int q = 0; q < 3; q++) {
                        const int s = 16 * (wq + 4 * q) + (lane & 15), sy = s / kHaloX;
                        if (s >= kSlots) continue;
                        int i = w.x0 + s - sy * kHaloX - 1, j = w.y0 + sy - 1;
                        const bool in = (i >= 0 || a.xper) && (j >= 0 || a.yper) && (i < a.nx || (a.xper && i == a.nx)) &&
                                        (j < a.ny || (a.yper && j == a.ny));
                        i = wrap(i, a.nx);
                        j = wrap(j, a.ny);
                        for (int p = 0; p < w.kz + 2; p++) {
                            const int k = w.z0 + p - 1;
                            const bool on = in && k >= 0 && k < a.nz;
                            const long long v = on ? (long long)i + (long long)a.nx * (j + (long long)a.ny * k) : 0;
                            for (int g = gh; g < cs; g += 2) {
                                const int c = c0 + 8 * g;
                                const __nv_bfloat16* src = c < a.c1 ? a.in1 + v * a.ld1 + c : a.in2 + v * a.ld2 + (c - a.c1);
                                cp_async16(dst + p * planeBytes + g * kGroupBytes + s * 16, on && c < a.ci ? src : a.in1, on && c < a.ci);
                            }
                        }
                    }
                } else {
                    // the upstream gradient: voxels 16 (wq + 4 q) + lane % 16
                    const uint32_t dd = dst + (kb + 2) * planeBytes;
#pragma unroll
                    for (int q = 0; q < 2; q++) {
                        const int s = 16 * (wq + 4 * q) + (lane & 15), i = w.x0 + (s & 7), j = w.y0 + (s >> 3);
                        const bool in = i < a.nx && j < a.ny;
                        for (int p = 0; p < w.kz; p++) {
                            const long long v = in ? (long long)i + (long long)a.nx * (j + (long long)a.ny * (w.z0 + p)) : 0;
                            for (int g = gh; g < N / 8; g += 2) {
                                const bool on = in && o0 + 8 * g < a.co;
                                cp_async16(dd + (p * (N / 8) + g) * kDoutGroup + s * 16, on ? a.dout + v * a.ldd + o0 + 8 * g : a.dout, on);
                            }
                        }
                    }
                }
                cp_async_commit();
                if (pending) {
                    cp_async_wait<1>();
                    fence_async_smem();
                    mbar_arrive_tc(pending);
                }
                pending = &sh.full[buf];
            }
            flush();
            cp_async_wait_all();
        } else if (elect_one()) {
            // A and B both MN-major (transpose bits 15 and 16)
            const uint32_t id = idesc_bf16(128, N) | (1u << 15) | (1u << 16);
            const uint64_t ad00 = smem_desc(st, kHaloX * 16, kGroupBytes);
            const uint64_t bd00 = smem_desc(st + (kb + 2) * planeBytes, 128, kDoutGroup);
            const uint32_t bplane = (N / 8) * (kDoutGroup >> 4);
            uint32_t n = 0, chains = 0;                // blocks, finished chains so far
            int link = 0;                              // blocks of the current chain
            for (int blk = blockIdx.x; blk < a.blocks && ok; blk += gridDim.x, n++) {
                const int buf = n & 1, kz = min(kb, a.nz - blk / (a.tx * a.ty) * kb);
                ok = mbar_wait_tc(&sh.full[buf], n >> 1 & 1);
                if (!ok) break;
                tc_fence_after();
                uint64_t ad0 = ad00 + (uint32_t)(buf * (blockBytes >> 4)), bd0 = bd00 + (uint32_t)(buf * (blockBytes >> 4));
                const bool head = link == 0;                   // the chain's first products do not accumulate
                for (int p = 0; p < kz && ok; p++) {
                    const bool more = !head || p > 0;
#pragma unroll
                    for (int u = 0; u < 9; u++) {
                        if (!more && n > 0) {
                            ok = ok && mbar_wait_tc(&sh.aempty[u], chains - 1 & 1);
                            if (!ok) break;
                            tc_fence_after();
                        }
                        uint64_t ad = ad0 + u / 3 * kHaloX + u % 3, bd = bd0;
#pragma unroll
                        for (int kk = 0; kk < 8; kk++) {
                            mma_bf16(tbase + u * N, ad, bd, id, more || kk > 0);
                            ad += 2 * kHaloX;
                            bd += 16;
                        }
                    }
                    ad0 += planeBytes >> 4;
                    bd0 += bplane;
                }
                if (!ok) break;
                mma_commit(&sh.empty[buf]);
                if (++link == a.chain || blk + (int)gridDim.x >= a.blocks) {
                    mma_commit(&sh.afull);
                    link = 0;
                    chains++;
                }
            }
            // every MMA has completed before the accumulators are read or freed
            mma_commit(&sh.done);
            if (!mbar_wait_tc(&sh.done, 0)) ok = false;
        }
    }
    tc_fence_before();
    ok = __syncthreads_and(ok);
    if (!ok && tid == 0) atomicExch(a.status, 1);
    if (warp == 0) tmem_free(tbase, a.ncols);
}

// The passes below move each value once: they take W channels of a voxel at a time,
// 8 (16 bytes) where the views start on 16 bytes with strides and channel counts that
// are multiples of 8, else 1.  One channel a thread, with a division for each, they
// took 480 us of a training step at 64x64x128, 8 take 260.
template <int W>
struct Chan;
template <>
struct Chan<1> {
    __nv_bfloat16 v[1];
    __device__ static Chan load(const __nv_bfloat16* p) { return Chan{{*p}}; }
    __device__ void store(__nv_bfloat16* p) const { *p = v[0]; }
};
template <>
struct alignas(16) Chan<8> {
    __nv_bfloat16 v[8];
    __device__ static Chan load(const __nv_bfloat16* p) {
        Chan r;
        *reinterpret_cast<uint4*>(r.v) = *reinterpret_cast<const uint4*>(p);
        return r;
    }
    __device__ void store(__nv_bfloat16* p) const { *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(v); }
};
static bool by8(const void* p, int ld, int c) { return !(reinterpret_cast<uintptr_t>(p) & 15) && ld % 8 == 0 && c % 8 == 0; }

// Sum over voxels of an upstream gradient per channel (bias gradient).  A thread
// keeps its W channels (n = kBiasThreads W / c voxels a block at a time); blockIdx.y
// picks the channels where c / W exceeds a block.  Few large blocks: what 300 blocks of
// 256 threads took (16 us) were additions to the same addresses.
constexpr int kBiasThreads = 1024;
template <int W>
__global__ void __launch_bounds__(kBiasThreads) k_bias_grad(const __nv_bfloat16* __restrict__ d, int ld, int c, long long V, float* __restrict__ db) {
    __shared__ float red[kBiasThreads][W + 1];
    const int groups = min(c / W - kBiasThreads * (int)blockIdx.y, kBiasThreads), n = kBiasThreads / groups;
    const int r = (int)threadIdx.x / groups, c0 = (kBiasThreads * blockIdx.y + threadIdx.x % groups) * W;
    float s[W] = {};
    if (r < n)
#pragma unroll 4
        for (long long v = (long long)blockIdx.x * n + r; v < V; v += (long long)gridDim.x * n) {
            const Chan<W> x = Chan<W>::load(d + v * ld + c0);
#pragma unroll
            for (int q = 0; q < W; q++) s[q] += __bfloat162float(x.v[q]);
        }
#pragma unroll
    for (int q = 0; q < W; q++) red[threadIdx.x][q] = s[q];
    __syncthreads();
    for (int m = n; m > 1;) {
        const int h = (m + 1) / 2;
        if (r + h < m)
#pragma unroll
            for (int q = 0; q < W; q++) red[threadIdx.x][q] += red[threadIdx.x + h * groups][q];
        m = h;
        __syncthreads();
    }
    if (r == 0)
#pragma unroll
        for (int q = 0; q < W; q++) atomicAdd(&db[c0 + q], red[threadIdx.x][q]);
}

// The 8 children of the coarse voxel of index q / groups, and its W channels
// (q % groups) W.  Ix is unsigned where the indexes fit 31 bits.
template <class Ix>
struct Children {
    int ch;
    long long vc, vf[8];
    __device__ Children(Ix q, int groups, int W, int nx, int ny) {
        const Ix v = q / (Ix)groups, cx = nx / 2, cy = ny / 2;
        ch = (int)(q - v * groups) * W;
        vc = v;
        const Ix t = v / cx, i = v - t * cx, k = t / cy, j = t - k * cy;
#pragma unroll
        for (int d = 0; d < 8; d++)
            vf[d] = (long long)(2 * i + (d & 1)) + (long long)nx * ((long long)(2 * j + ((d >> 1) & 1)) + (long long)ny * (long long)(2 * k + (d >> 2)));
    }
};

// 2x2x2 average pooling (forward) and its adjoint (backward: each child gets
// 1/8 of the parent's gradient).  Fine grid (nx, ny, nz), coarse (nx/2, ...).
template <int W, class Ix>
__global__ void k_pool(const __nv_bfloat16* __restrict__ in, int ldi, __nv_bfloat16* __restrict__ out, int ldo, int c,
                       int nx, int ny, int nz, int backward, int accumulate) {
    const Ix n = (Ix)((long long)(nx / 2) * (ny / 2) * (nz / 2) * (c / W));
    for (Ix q = (Ix)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (Ix)gridDim.x * blockDim.x) {
        const Children<Ix> f(q, c / W, W, nx, ny);
        if (!backward) {
            float s[W] = {};
#pragma unroll
            for (int d = 0; d < 8; d++) {
                const Chan<W> x = Chan<W>::load(in + f.vf[d] * ldi + f.ch);
#pragma unroll
                for (int w = 0; w < W; w++) s[w] += __bfloat162float(x.v[w]);
            }
            Chan<W> y;
#pragma unroll
            for (int w = 0; w < W; w++) y.v[w] = __float2bfloat16_rn(0.125f * s[w]);
            y.store(out + f.vc * ldo + f.ch);
        } else {
            // in = coarse gradient, out = fine gradient
            const Chan<W> g = Chan<W>::load(in + f.vc * ldi + f.ch);
#pragma unroll
            for (int d = 0; d < 8; d++) {
                __nv_bfloat16* o = out + f.vf[d] * ldo + f.ch;
                Chan<W> y{};
                if (accumulate) y = Chan<W>::load(o);
#pragma unroll
                for (int w = 0; w < W; w++)
                    y.v[w] = __float2bfloat16_rn((accumulate ? __bfloat162float(y.v[w]) : 0.f) + 0.125f * __bfloat162float(g.v[w]));
                y.store(o);
            }
        }
    }
}

// Nearest-neighbour 2x upsampling (forward) and its adjoint (backward: the sum
// of the 8 children).  Coarse grid (nx/2, ...), fine (nx, ny, nz).
template <int W, class Ix>
__global__ void k_upsample(const __nv_bfloat16* __restrict__ in, int ldi, __nv_bfloat16* __restrict__ out, int ldo,
                           int c, int nx, int ny, int nz, int backward) {
    const Ix n = (Ix)((long long)(nx / 2) * (ny / 2) * (nz / 2) * (c / W));
    for (Ix q = (Ix)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (Ix)gridDim.x * blockDim.x) {
        const Children<Ix> f(q, c / W, W, nx, ny);
        if (!backward) {
            const Chan<W> x = Chan<W>::load(in + f.vc * ldi + f.ch);
#pragma unroll
            for (int d = 0; d < 8; d++) x.store(out + f.vf[d] * ldo + f.ch);
        } else {
            // in = fine gradient, out = coarse gradient
            float s[W] = {};
#pragma unroll
            for (int d = 0; d < 8; d++) {
                const Chan<W> x = Chan<W>::load(in + f.vf[d] * ldi + f.ch);
#pragma unroll
                for (int w = 0; w < W; w++) s[w] += __bfloat162float(x.v[w]);
            }
            Chan<W> y;
#pragma unroll
            for (int w = 0; w < W; w++) y.v[w] = __float2bfloat16_rn(s[w]);
            y.store(out + f.vc * ldo + f.ch);
        }
    }
}

// d *= (y > 0): the gradient through a ReLU from its output.
template <int W, class Ix>
__global__ void k_relu_bwd(__nv_bfloat16* __restrict__ d, int ldd, const __nv_bfloat16* __restrict__ y, int ldy, int c,
                           long long V) {
    const Ix groups = c / W, n = (Ix)(V * (c / W));
    for (Ix q = (Ix)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (Ix)gridDim.x * blockDim.x) {
        const Ix v = q / groups, ch = (q - v * groups) * W;
        const Chan<W> x = Chan<W>::load(y + (long long)v * ldy + ch);
        Chan<W> g = Chan<W>::load(d + (long long)v * ldd + ch);
#pragma unroll
        for (int w = 0; w < W; w++)
            if (!(__bfloat162float(x.v[w]) > 0.f)) g.v[w] = __float2bfloat16_rn(0.f);
        g.store(d + (long long)v * ldd + ch);
    }
}

// Masked mean-square error of the 3 output channels against the target
// (FP32, [V][3]); planes k = 0 and nz-1 are excluded (their displacement is
// imposed to be zero).  Writes the gradient (BF16) and adds the loss sum.
// A training sample moved by a symmetry of the periodic cross-section: the
// value at cell (i, j) is read at the source cell u = (i + sx) mod nx,
// v = (j + sy) mod ny, then (sym & 4) u <-> v, (sym & 2) v -> ny - 1 - v,
// (sym & 1) u -> nx - 1 - u; a vector's x, y components are transformed as the
// positions (x negated for bit 1, y for bit 2, then swapped for bit 4), so
// the field and the displacement stay a solution pair of the relaxation (the
// force J x B transforms as a polar vector under reflections).
__device__ __forceinline__ void sym_source(int i, int j, int nx, int ny, int sx, int sy, int sym, int* is, int* js) {
    int u = (i + sx) % nx, v = (j + sy) % ny;
    if (sym & 4) { const int w = u; u = v; v = w; }
    if (sym & 2) v = ny - 1 - v;
    if (sym & 1) u = nx - 1 - u;
    *is = u;
    *js = v;
}
__device__ __forceinline__ void sym_vector(int sym, float* vx, float* vy) {
    if (sym & 1) *vx = -*vx;
    if (sym & 2) *vy = -*vy;
    if (sym & 4) { const float w = *vx; *vx = *vy; *vy = w; }
}

__global__ void k_mse(const __nv_bfloat16* __restrict__ y, int ldy, const float* __restrict__ tgt,
                      __nv_bfloat16* __restrict__ dy, int lddy, int nx, int ny, int nz, float scale,
                      float* __restrict__ loss, int sx, int sy, int sym) {
    __shared__ float red[256];
    const long long V = (long long)nx * ny * nz;
    float s = 0.f;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < V; v += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(v % nx), j = (int)((v / nx) % ny), k = (int)(v / ((long long)nx * ny));
        const bool in = k > 0 && k < nz - 1;
        int is, js;
        sym_source(i, j, nx, ny, sx, sy, sym, &is, &js);
        const long long vt = (long long)is + (long long)nx * (js + (long long)ny * k);
        float t[3] = {tgt[3 * vt], tgt[3 * vt + 1], tgt[3 * vt + 2]};
        sym_vector(sym, &t[0], &t[1]);
        for (int c = 0; c < 3; c++) {
            const float e = in ? __bfloat162float(y[v * ldy + c]) - t[c] : 0.f;
            s += e * e;
            dy[v * lddy + c] = __float2bfloat16_rn(2.f * scale * e);
        }
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) atomicAdd(loss, red[0] * scale);
}

// Adam on FP32 master weights W[27][co][ci] and b[co]; then the BF16 operand
// layouts: Wf[27][Npo][Kci] (forward: rows = outputs) and Wb[27][Npi][Kco]
// (input gradient: taps flipped, rows = inputs).
__global__ void k_adam(float* __restrict__ W, float* __restrict__ mW, float* __restrict__ vW,
                       const float* __restrict__ gW, float* __restrict__ b, float* __restrict__ mb,
                       float* __restrict__ vb, const float* __restrict__ gb, int co, int ci, float lr, float b1,
                       float b2, float c1, float c2, float eps, __nv_bfloat16* __restrict__ Wf, int Npo, int Kci,
                       __nv_bfloat16* __restrict__ Wb, int Npi, int Kco, float* __restrict__ bpad, int step) {
    const long long n = 27LL * co * ci;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n + co; q += (long long)gridDim.x * blockDim.x) {
        if (q < n) {
            float w = W[q];
            if (step) {
                const float g = gW[q];
                const float m = b1 * mW[q] + (1 - b1) * g, v = b2 * vW[q] + (1 - b2) * g * g;
                mW[q] = m;
                vW[q] = v;
                w -= lr * (m / c1) / (sqrtf(v / c2) + eps);
                W[q] = w;
            }
            const int t = (int)(q / ((long long)co * ci)), o = (int)((q / ci) % co), i = (int)(q % ci);
            const __nv_bfloat16 wb = __float2bfloat16_rn(w);
            Wf[((size_t)t * Npo + o) * Kci + i] = wb;
            Wb[((size_t)(26 - t) * Npi + i) * Kco + o] = wb;
        } else {
            const int o = (int)(q - n);
            float x = b[o];
            if (step) {
                const float g = gb[o];
                const float m = b1 * mb[o] + (1 - b1) * g, v = b2 * vb[o] + (1 - b2) * g * g;
                mb[o] = m;
                vb[o] = v;
                x -= lr * (m / c1) / (sqrtf(v / c2) + eps);
                b[o] = x;
            }
            bpad[o] = x;
        }
    }
}

// Input channels (B0x, B0y, B0z - 1) of the inner points, from the ghosted
// AoS B0 of the reference layout (REAL T); ld channels, the rest zero.
// The sample is moved by a symmetry of the periodic cross-section (sym_source,
// sym_vector): whole-cell translations, mirrors and the x <-> y swap, used to
// augment training data.
template <typename T>
__global__ void k_input(const T* __restrict__ B0, int nx, int ny, int nz, __nv_bfloat16* __restrict__ x, int ld,
                        int sx, int sy, int sym) {
    const long long V = (long long)nx * ny * nz;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < V; v += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(v % nx), j = (int)((v / nx) % ny), k = (int)(v / ((long long)nx * ny));
        int is, js;
        sym_source(i, j, nx, ny, sx, sy, sym, &is, &js);
        const long long g = (long long)(is + 1) + (long long)(nx + 2) * ((js + 1) + (long long)(ny + 2) * (k + 1));
        float b[3] = {(float)B0[3 * g], (float)B0[3 * g + 1], (float)B0[3 * g + 2] - 1.f};
        sym_vector(sym, &b[0], &b[1]);
        for (int c = 0; c < ld; c++) x[v * ld + c] = __float2bfloat16_rn(c < 3 ? b[c] : 0.f);
    }
}

// ---- the warm-start grid: displacement -> smoothed -> positions ------------

// Displacement channels 0..2 of a network output (BF16, [V][ld]) computed on
// the input translated by (sx, sy) (gm_nn_input), moved back to the grid's
// own cells and weighted: d(i, j, k) = w y((i - sx) mod nx, (j - sy) mod ny, k),
// added to d unless `first`.
__global__ void k_wg_acc(const __nv_bfloat16* __restrict__ y, int ld, int nx, int ny, int nz, int sx, int sy, float w,
                         int first, float* __restrict__ d) {
    const long long V = (long long)nx * ny * nz;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < V; v += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(v % nx), j = (int)((v / nx) % ny);
        const long long k = v / ((long long)nx * ny);
        const int is = (i - sx + nx) % nx, js = (j - sy + ny) % ny;
        const long long u = is + (long long)nx * (js + (long long)ny * k);
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const float val = w * __bfloat162float(y[u * ld + c]);
            d[3 * v + c] = first ? val : d[3 * v + c] + val;
        }
    }
}

// One 3x3x3 box-filter pass, periodic in x / y as selected, zero beyond the
// z range: out(i, j, k) = (1/27) sum of the 27 neighbours.
__global__ void k_wg_box(const float* __restrict__ in, float* __restrict__ out, int nx, int ny, int nz, int xper,
                         int yper) {
    const long long V = (long long)nx * ny * nz;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < V; v += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(v % nx), j = (int)((v / nx) % ny), k = (int)(v / ((long long)nx * ny));
        float acc[3] = {0.f, 0.f, 0.f};
        for (int dk = -1; dk <= 1; dk++) {
            const int kk = k + dk;
            if (kk < 0 || kk >= nz) continue;
            for (int dj = -1; dj <= 1; dj++) {
                int jj = j + dj;
                if (jj < 0 || jj >= ny) {
                    if (!yper) continue;
                    jj = (jj + ny) % ny;
                }
                for (int di = -1; di <= 1; di++) {
                    int ii = i + di;
                    if (ii < 0 || ii >= nx) {
                        if (!xper) continue;
                        ii = (ii + nx) % nx;
                    }
                    const float* q = in + 3 * (ii + (long long)nx * (jj + (long long)ny * kk));
                    acc[0] += q[0]; acc[1] += q[1]; acc[2] += q[2];
                }
            }
        }
#pragma unroll
        for (int c = 0; c < 3; c++) out[3 * v + c] = acc[c] * (1.f / 27.f);
    }
}

// Positions of the warm grid in the reference layout (ghosted AoS): the
// identity grid xid plus the displacement (in grid spacings) at the inner
// points, the first and last inner z-planes held; periodic x / y ghosts are
// the images of the opposite inner points shifted by -/+ (L + d) (x first,
// then y, so corners carry both shifts); other ghosts keep xid.
template <typename T>
__global__ void k_wg_grid(const float* __restrict__ d, const T* __restrict__ xid, T* __restrict__ xb, int nx, int ny,
                          int nz, int xper, int yper, double dx, double dy, double dz, double Lx, double Ly) {
    const long long G = (long long)(nx + 2) * (ny + 2) * (nz + 2);
    for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < G; g += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(g % (nx + 2)), j = (int)((g / (nx + 2)) % (ny + 2));
        const int k = (int)(g / ((long long)(nx + 2) * (ny + 2)));
        int is = i, js = j;
        double sx = 0, sy = 0;
        if (xper && i == 0) { is = nx; sx = -(Lx + dx); }
        if (xper && i == nx + 1) { is = 1; sx = Lx + dx; }
        if (yper && j == 0) { js = ny; sy = -(Ly + dy); }
        if (yper && j == ny + 1) { js = 1; sy = Ly + dy; }
        const long long gs = is + (long long)(nx + 2) * (js + (long long)(ny + 2) * k);
        double x[3] = {(double)xid[3 * gs], (double)xid[3 * gs + 1], (double)xid[3 * gs + 2]};
        if (is >= 1 && is <= nx && js >= 1 && js <= ny && k >= 2 && k <= nz - 1) {
            const float* q = d + 3 * ((is - 1) + (long long)nx * ((js - 1) + (long long)ny * (k - 1)));
            x[0] += (double)q[0] * dx;
            x[1] += (double)q[1] * dy;
            x[2] += (double)q[2] * dz;
        }
        x[0] += sx;
        x[1] += sy;
        xb[3 * g] = (T)x[0];
        xb[3 * g + 1] = (T)x[1];
        xb[3 * g + 2] = (T)x[2];
    }
}

// The launch of a convolution: k_conv_planes with resident weights or
// k_conv_wide with streamed ones, the candidates (output slices, planes per item)
// compared by an estimate in clocks.  An MMA with N columns takes
// max(46, 32 + N / 4, N / 2) clocks; CTAs on an SM share the tensor core; resident
// weights arrive at about 40 bytes a clock and SM, a stage of streamed ones takes 600
// clocks more, and an item of k_conv_wide starts 4000 clocks late; a plane's barriers take about 700 clocks of one CTA that another
// hides; starting and draining a CTA takes 5000.  Against all shapes that fit, the
// choice was the fastest or within 10 % of it (64x64x128: 24 -> 24 channels 38 us,
// 72 -> 24 75 us, 24 -> 72 81 us; 32x32x64: 240 -> 48 122 us with streamed weights,
// the only form that fits; 16x16x32: 48 -> 192 19 us, 24 streamed).
struct ConvPlan {
    bool wide;
    int Nt, kz, occ, planes, ncols, sets, kch, stages;
    long long items;
    dim3 grid;
    size_t smem;
};

static bool choose_conv(const ConvArgs& a, ConvPlan* best) {
    int dev = 0, nsm = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const long long cols = (long long)((a.nx + kTileX - 1) / kTileX) * ((a.ny + kTileY - 1) / kTileY);
    const ConvLanes L(a.Kc);
    const size_t limit = 227 * 1024, plane = (size_t)L.ng * kGroupBytes;
    double tbest = 0;
    auto mma = [](double N) { return std::max(46.0, std::max(32 + N / 4, N / 2)); };
    int last = 0;
    for (int Nt = 16; Nt <= 256 && Nt <= a.Np; Nt += 16) {
        const int slices = (a.Np + Nt - 1) / Nt;
        if (slices == last) continue;          // no fewer slices than the width before
        last = slices;
        const double ksteps = a.Kc / 16;
        ConvPlan c;
        c.Nt = Nt;
        if (Nt <= 80) {
            c.wide = false;
            c.planes = 3;
            c.smem = kPlaneShared + (size_t)9 * L.ng * L.row_stride(3 * Nt) + 3 * plane;
            if (c.smem > limit) { c.planes = 2; c.smem -= plane; }
            for (int kz = 1; c.smem <= limit && kz <= kMaxKz && kz <= a.nz && kz * Nt <= 512; kz++) {
                c.kz = kz;
                c.ncols = 32;
                while (c.ncols < kz * Nt) c.ncols <<= 1;
                c.occ = std::min((int)(228 * 1024 / (c.smem + 1024)), std::min(512 / c.ncols, 4));
                c.items = cols * ((a.nz + kz - 1) / kz);
                const long long gx = std::max(1ll, std::min(c.items, (long long)nsm * c.occ / slices));
                c.grid = dim3((unsigned)gx, (unsigned)slices);
                const double on = (double)((gx * slices + nsm - 1) / nsm);        // CTAs on an SM
                const double per = 9 * ksteps * mma(3.0 * Nt * kz / (kz + 2));
                const double t = (double)((c.items + gx - 1) / gx) * (kz + 2) * std::max(on * per, per + (c.planes > 2 ? 700 : 1500)) +
                                 27.0 * Nt * a.Kc * 2 / 40 * on + 5000;
                if (c.items < (1ll << 31) && (tbest == 0 || t < tbest)) { tbest = t; *best = c; }
            }
        }
        c.wide = true;
        c.occ = 1;
        for (int kz = 1; kz <= kWideKz && kz <= a.nz && kz * Nt <= 512; kz++) {
            c.kz = kz;
            c.planes = kz + 1;
            c.kch = a.Kc;
            auto step = [&]() { return (size_t)(c.kch / 8) * ConvLanes(c.kch).row_stride(Nt); };
            auto room = [&](int stages) { return kWideShared + c.planes * plane + stages * step() <= limit; };
            // the widest chunk of at most 16 KB of which six stages fit
            int nch = 1;
            for (; nch <= a.Kc / 16; nch++) {
                if (a.Kc / 16 % nch) continue;
                c.kch = a.Kc / nch;
                if (Nt * c.kch * 2 <= 16384 && room(6)) break;
            }
            if (nch > a.Kc / 16) continue;
            c.stages = room(8) ? 8 : 6;
            c.sets = 2 * kz * Nt <= 512 ? 2 : 1;
            c.ncols = 32;
            while (c.ncols < c.sets * kz * Nt) c.ncols <<= 1;
            c.items = cols * ((a.nz + kz - 1) / kz);
            const long long gx = std::max(1ll, std::min(c.items, (long long)nsm / slices));
            c.grid = dim3((unsigned)gx, (unsigned)slices);
            c.smem = kWideShared + c.planes * plane + c.stages * step();
            const double item = 27.0 * nch * std::max(ksteps / nch * kz * mma(Nt), 600 + Nt * c.kch * 2 / 40.0);
            const double t = (double)((c.items + gx - 1) / gx) * (item + 4000) + 8000;
            if (c.items < (1ll << 31) && (tbest == 0 || t < tbest)) { tbest = t; *best = c; }
        }
    }
    return tbest > 0;
}

static unsigned nb(long long n) {
    long long b = (n + 255) / 256;
    return (unsigned)(b < 1 ? 1 : (b > 152 * 16 ? 152 * 16 : b));
}

}  // namespace gmnn

using gmnn::ConvArgs;
using gmnn::WgradArgs;

extern "C" {

int gm_nn_tc_gemm_check(const void* A, const void* B, float* D, int N, int K, int* status) {
    if (!A || !B || !D || !status) return gm::fail(GM_EPARAM, "gm_nn_tc_gemm_check: null argument");
    if (N < 16 || N > 256 || N % 16 || K < 16 || K > 256 || K % 16)
        return gm::fail(GM_EPARAM, "gm_nn_tc_gemm_check: N and K must be multiples of 16 in [16, 256]");
    const size_t smem = (size_t)(128 + N) * K * 2 + 16;
    cudaError_t e = cudaFuncSetAttribute(gmnn::k_tc_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return gm::fail(GM_ECUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
    gmnn::k_tc_gemm<<<1, 128, smem>>>((const __nv_bfloat16*)A, (const __nv_bfloat16*)B, D, N, K, status);
    e = cudaDeviceSynchronize();
    if (e != cudaSuccess) return gm::fail(GM_ECUDA, std::string("k_tc_gemm: ") + cudaGetErrorString(e));
    return GM_OK;
}

static int check_view_align(const void* p, int ld, const char* what) {
    if (p && ((reinterpret_cast<uintptr_t>(p) & 15) || (ld % 8)))
        return gm::fail(GM_EPARAM, std::string(what) + ": views must start on 16 bytes with a channel stride that is a multiple of 8");
    return GM_OK;
}

namespace {
// failure-detection test hook (gm_nn_debug_stall): read when a convolution is launched
int g_nn_stall = 0;
}  // namespace

int gm_nn_debug_stall(int on) {
    g_nn_stall = on ? 1 : 0;
    return GM_OK;
}

int gm_nn_conv(const void* in1, int ld1, int c1, const void* in2, int ld2, int c2, const void* W, const float* bias,
               void* out, int ldo, int co, const void* mask, int ldm, int relu, int nx, int ny, int nz, int xper,
               int yper, int Kc, int Np, int* status, void* stream) {
    if (!in1 || !W || !out || !status) return gm::fail(GM_EPARAM, "gm_nn_conv: null argument");
    if (Kc % 16 || Kc < 16 || Kc > 256 || Np % 16 || Np < 16 || Np > 256 || c1 + (in2 ? c2 : 0) > Kc || co > Np ||
        c1 % 8)
        return gm::fail(GM_EPARAM, "gm_nn_conv: channel counts out of range");
    if (nx < 1 || ny < 1 || nz < 1) return gm::fail(GM_EPARAM, "gm_nn_conv: grid out of range");
    int rc;
    if ((rc = check_view_align(in1, ld1, "gm_nn_conv in1")) || (rc = check_view_align(in2, ld2, "gm_nn_conv in2")))
        return rc;
    ConvArgs a;
    a.in1 = (const __nv_bfloat16*)in1; a.ld1 = ld1; a.c1 = c1;
    a.in2 = (const __nv_bfloat16*)in2; a.ld2 = ld2; a.c2 = in2 ? c2 : 0;
    a.W = (const __nv_bfloat16*)W; a.bias = bias;
    a.out = (__nv_bfloat16*)out; a.ldo = ldo; a.co = co;
    a.mask = (const __nv_bfloat16*)mask; a.ldm = ldm; a.relu = relu;
    a.nx = nx; a.ny = ny; a.nz = nz; a.xper = xper; a.yper = yper; a.Kc = Kc; a.Np = Np; a.status = status;
    a.stall = g_nn_stall;
    auto aligned = [](const void* q, int ld) { return q == nullptr || (!(reinterpret_cast<uintptr_t>(q) & 15) && ld % 8 == 0); };
    a.vec = aligned(out, ldo) && aligned(mask, ldm);
    gmnn::ConvPlan c;
    if (!gmnn::choose_conv(a, &c)) return gm::fail(GM_EPARAM, "gm_nn_conv: grid out of range");
    a.Nt = c.Nt;
    const int tx = (nx + gmnn::kTileX - 1) / gmnn::kTileX, ty = (ny + gmnn::kTileY - 1) / gmnn::kTileY;
    cudaError_t e = c.wide ? cudaFuncSetAttribute(gmnn::k_conv_wide, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024)
                           : cudaFuncSetAttribute(gmnn::k_conv_planes, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return gm::fail(GM_ECUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
    if (c.wide)
        gmnn::k_conv_wide<<<c.grid, gmnn::kWideThreads, c.smem, (cudaStream_t)stream>>>(
            gmnn::ConvWideArgs{a, c.kz, tx, ty, (int)c.items, c.ncols, c.sets, c.planes, c.kch, c.stages});
    else
        gmnn::k_conv_planes<<<c.grid, gmnn::kPlaneThreads, c.smem, (cudaStream_t)stream>>>(
            gmnn::ConvPlaneArgs{a, c.kz, tx, ty, (int)c.items, c.ncols, c.planes});
    e = cudaGetLastError();
    return e == cudaSuccess ? GM_OK : gm::fail(GM_ECUDA, std::string("convolution launch: ") + cudaGetErrorString(e));
}

int gm_nn_conv_wgrad(const void* dout, int ldd, int co, const void* in1, int ld1, int c1, const void* in2, int ld2,
                     int c2, float* dW, int ci, int nx, int ny, int nz, int xper, int yper, int vchunk, int* status,
                     void* stream) {
    if (!dout || !in1 || !dW || !status) return gm::fail(GM_EPARAM, "gm_nn_conv_wgrad: null argument");
    const long long V = (long long)nx * ny * nz;
    if (ci > c1 + (in2 ? c2 : 0) || ci < 1 || co > 256 || co < 1 || vchunk < 0 || vchunk % 64 || c1 % 8 ||
        nx < 1 || ny < 1 || nz < 1 || V >= (1ll << 31))
        return gm::fail(GM_EPARAM, "gm_nn_conv_wgrad: channel counts, grid or chunk out of range");
    int rc;
    if ((rc = check_view_align(dout, ldd, "gm_nn_conv_wgrad dout")) ||
        (rc = check_view_align(in1, ld1, "gm_nn_conv_wgrad in1")) || (rc = check_view_align(in2, ld2, "gm_nn_conv_wgrad in2")))
        return rc;
    WgradArgs a;
    a.dout = (const __nv_bfloat16*)dout; a.ldd = ldd; a.co = co;
    a.in1 = (const __nv_bfloat16*)in1; a.ld1 = ld1; a.c1 = in2 ? c1 : (ci + 7) / 8 * 8;
    a.in2 = (const __nv_bfloat16*)(in2 ? in2 : in1); a.ld2 = in2 ? ld2 : ld1;
    a.dW = dW; a.ci = ci;
    a.nx = nx; a.ny = ny; a.nz = nz; a.xper = xper; a.yper = yper;
    a.tx = (nx + gmnn::kTileX - 1) / gmnn::kTileX;
    a.ty = (ny + gmnn::kTileY - 1) / gmnn::kTileY;
    a.status = status;
    a.stall = g_nn_stall;
    // even slices of at most kWgGroups input groups and kWgN output channels
    const int ng = (ci + 7) / 8, nslices = (co + gmnn::kWgN - 1) / gmnn::kWgN;
    a.cslices = (ng + gmnn::kWgGroups - 1) / gmnn::kWgGroups;
    a.cs = (ng + a.cslices - 1) / a.cslices;
    a.N = ((co + nslices - 1) / nslices + 15) / 16 * 16;
    a.ncols = 32;
    while (a.ncols < 9 * a.N) a.ncols <<= 1;
    int dev = 0, nsm = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    // planes per block and CTAs along the blocks: one wave; a plane's MMAs take 3300
    // clocks, a block about 1000 more, its copies 1 clock per 7.5 bytes; vchunk asks for at least that many voxels a CTA.
    // Chains of lim voxels are those of 608 CTAs (four on each of 152 SMs) with 128 of the
    // stacked (tap, channel) rows each; a chain is no longer (the truncation error no
    // larger), and where the voxels are many no more than 3000 voxels (1500 of chains
    // beyond 8000) shorter, so that the error is the same to 1e-5 of the gradient.  No chain
    // is longer than kWgChain, so that on larger grids the error stops growing with them
    // (72 -> 24 channels at 128x128x256: 110,080 voxels, 1.5e-4 of the gradient and 1355 us
    // without it, 2.6e-5 and 1167 with it).
    const long long lim = std::min(gmnn::kWgChain, std::max(512ll, V * ((27 * ng * 8 + 127) / 128) / 608));
    const long long shorter = lim > 8000 ? 1500 : 3000;
    const long long slices = (long long)a.cslices * nslices;
    double tbest = 0;
    long long gx = 1;
    for (int kb = 1; kb <= gmnn::kWgKb && kb <= nz; kb++) {
        if (gmnn::wgrad_smem(a.cs, kb, a.N) > 227 * 1024) break;
        const long long blocks = (long long)a.tx * a.ty * ((nz + kb - 1) / kb);
        long long g = std::max(1ll, std::min(blocks, nsm / slices));
        if (lim > 3512) g = std::min(g, (V + lim - shorter - 1) / (lim - shorter));
        if (vchunk > 0) g = std::min(g, (V + vchunk - 1) / vchunk);
        const double load = gmnn::wg_block_bytes(a.cs, kb, a.N) / 7.5;
        const double t = load + (double)((blocks + g - 1) / g) * (std::max(3300.0 * kb, load) + 1000);
        if (tbest == 0 || t < tbest) {
            tbest = t;
            gx = g;
            a.kb = kb;
            a.blocks = (int)blocks;
        }
    }
    a.chain = (int)std::max(1ll, lim / (128 * a.kb));
    const size_t smem = gmnn::wgrad_smem(a.cs, a.kb, a.N);
    cudaError_t e = cudaFuncSetAttribute(gmnn::k_conv_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return gm::fail(GM_ECUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
    gmnn::k_conv_wgrad<<<dim3((unsigned)gx, (unsigned)slices), gmnn::kWgThreads, smem, (cudaStream_t)stream>>>(a);
    e = cudaGetLastError();
    return e == cudaSuccess ? GM_OK : gm::fail(GM_ECUDA, std::string("k_conv_wgrad: ") + cudaGetErrorString(e));
}

int gm_nn_bias_grad(const void* d, int ld, int c, long long V, float* db, void* stream) {
    const bool w8 = gmnn::by8(d, ld, c);
    const int groups = w8 ? c / 8 : c, n = gmnn::kBiasThreads / std::max(1, std::min(groups, gmnn::kBiasThreads));
    const dim3 grid((unsigned)std::max(1ll, std::min((V + 4 * n - 1) / (4 * n), 152ll)), (unsigned)((groups + gmnn::kBiasThreads - 1) / gmnn::kBiasThreads));
    auto kern = w8 ? gmnn::k_bias_grad<8> : gmnn::k_bias_grad<1>;
    kern<<<grid, gmnn::kBiasThreads, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)d, ld, c, V, db);
    return cudaGetLastError() == cudaSuccess ? GM_OK : gm::fail(GM_ECUDA, "k_bias_grad");
}

int gm_nn_pool(const void* in, int ldi, void* out, int ldo, int c, int nx, int ny, int nz, int backward,
               int accumulate, void* stream) {
    if (nx % 2 || ny % 2 || nz % 2) return gm::fail(GM_EPARAM, "gm_nn_pool: grid sizes must be even");
    const long long n = (long long)(nx / 2) * (ny / 2) * (nz / 2) * c;
    const bool w8 = gmnn::by8(in, ldi, c) && gmnn::by8(out, ldo, c) && n / 8 < (1ll << 31);
    auto kern = w8 ? gmnn::k_pool<8, unsigned> : n < (1ll << 31) ? gmnn::k_pool<1, unsigned> : gmnn::k_pool<1, long long>;
    kern<<<gmnn::nb(w8 ? n / 8 : n), 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)in, ldi, (__nv_bfloat16*)out, ldo, c,
                                                                     nx, ny, nz, backward, accumulate);
    return cudaGetLastError() == cudaSuccess ? GM_OK : gm::fail(GM_ECUDA, "k_pool");
}

int gm_nn_upsample(const void* in, int ldi, void* out, int ldo, int c, int nx, int ny, int nz, int backward,
                   void* stream) {
    if (nx % 2 || ny % 2 || nz % 2) return gm::fail(GM_EPARAM, "gm_nn_upsample: grid sizes must be even");
    const long long n = (long long)(nx / 2) * (ny / 2) * (nz / 2) * c;
    const bool w8 = gmnn::by8(in, ldi, c) && gmnn::by8(out, ldo, c) && n / 8 < (1ll << 31);
    auto kern = w8 ? gmnn::k_upsample<8, unsigned> : n < (1ll << 31) ? gmnn::k_upsample<1, unsigned> : gmnn::k_upsample<1, long long>;
    kern<<<gmnn::nb(w8 ? n / 8 : n), 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)in, ldi, (__nv_bfloat16*)out, ldo, c,
                                                                     nx, ny, nz, backward);
    return cudaGetLastError() == cudaSuccess ? GM_OK : gm::fail(GM_ECUDA, "k_upsample");
}

int gm_nn_input(const void* B0, int precision, int nx, int ny, int nz, void* x, int ld, int sx, int sy, int sym,
                void* stream) {
    if (sx < 0 || sx >= nx || sy < 0 || sy >= ny) return gm::fail(GM_EPARAM, "gm_nn_input: shift out of range");
    if (sym < 0 || sym > 7 || ((sym & 4) && nx != ny))
        return gm::fail(GM_EPARAM, "gm_nn_input: sym is 0..7, and the x <-> y swap needs nx == ny");
    const long long V = (long long)nx * ny * nz;
    if (precision == 32)
        gmnn::k_input<float><<<gmnn::nb(V), 256, 0, (cudaStream_t)stream>>>((const float*)B0, nx, ny, nz,
                                                                              (__nv_bfloat16*)x, ld, sx, sy, sym);
    else
        gmnn::k_input<double><<<gmnn::nb(V), 256, 0, (cudaStream_t)stream>>>((const double*)B0, nx, ny, nz,
                                                                               (__nv_bfloat16*)x, ld, sx, sy, sym);
    return cudaGetLastError() == cudaSuccess ? GM_OK : gm::fail(GM_ECUDA, "k_input");
}

int gm_nn_disp_accumulate(const void* y, int ldy, int nx, int ny, int nz, int sx, int sy, float w, int first,
                          float* d, void* stream) {
    if (!y || !d || ldy < 3 || sx < 0 || sx >= nx || sy < 0 || sy >= ny)
        return gm::fail(GM_EPARAM, "gm_nn_disp_accumulate: bad argument");
    const long long V = (long long)nx * ny * nz;
    gmnn::k_wg_acc<<<gmnn::nb(V), 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)y, ldy, nx, ny, nz, sx, sy, w,
                                                                   first, d);
    return cudaGetLastError() == cudaSuccess ? GM_OK : gm::fail(GM_ECUDA, "gm_nn_disp_accumulate");
}

int gm_nn_warm_grid(const float* d, const gm_params* p, int passes, const void* xid, float* scratch, void* xb,
                    void* stream) {
    if (!d || !p || !xid || !scratch || !xb || passes < 0)
        return gm::fail(GM_EPARAM, "gm_nn_warm_grid: bad argument");
    const int nx = p->nx, ny = p->ny, nz = p->nz;
    const long long V = (long long)nx * ny * nz, G = (long long)(nx + 2) * (ny + 2) * (nz + 2);
    cudaStream_t s = (cudaStream_t)stream;
    float* a = scratch;
    float* b = scratch + 3 * V;
    if (cudaMemcpyAsync(a, d, 3 * V * sizeof(float), cudaMemcpyDeviceToDevice, s) != cudaSuccess)
        return gm::fail(GM_ECUDA, "gm_nn_warm_grid: copy of the displacement failed");
    for (int q = 0; q < passes; q++) {
        gmnn::k_wg_box<<<gmnn::nb(V), 256, 0, s>>>(a, b, nx, ny, nz, p->xPeri, p->yPeri);
        float* t = a; a = b; b = t;
    }
    if (p->precision == 32)
        gmnn::k_wg_grid<float><<<gmnn::nb(G), 256, 0, s>>>(a, (const float*)xid, (float*)xb, nx, ny, nz, p->xPeri,
                                                            p->yPeri, p->dx, p->dy, p->dz, p->Lx, p->Ly);
    else
        gmnn::k_wg_grid<double><<<gmnn::nb(G), 256, 0, s>>>(a, (const double*)xid, (double*)xb, nx, ny, nz, p->xPeri,
                                                             p->yPeri, p->dx, p->dy, p->dz, p->Lx, p->Ly);
    return cudaGetLastError() == cudaSuccess ? GM_OK : gm::fail(GM_ECUDA, "gm_nn_warm_grid");
}

int gm_nn_zero(void* p, size_t bytes, void* stream) {
    const cudaError_t e = cudaMemsetAsync(p, 0, bytes, (cudaStream_t)stream);
    return e == cudaSuccess ? GM_OK : gm::fail(GM_ECUDA, std::string("cudaMemsetAsync: ") + cudaGetErrorString(e));
}

int gm_nn_relu_bwd(void* d, int ldd, const void* y, int ldy, int c, long long V, void* stream) {
    const bool w8 = gmnn::by8(d, ldd, c) && gmnn::by8(y, ldy, c) && V * (c / 8) < (1ll << 31);
    auto kern = w8 ? gmnn::k_relu_bwd<8, unsigned> : V * c < (1ll << 31) ? gmnn::k_relu_bwd<1, unsigned> : gmnn::k_relu_bwd<1, long long>;
    kern<<<gmnn::nb(w8 ? V * (c / 8) : V * c), 256, 0, (cudaStream_t)stream>>>((__nv_bfloat16*)d, ldd, (const __nv_bfloat16*)y, ldy, c, V);
    return cudaGetLastError() == cudaSuccess ? GM_OK : gm::fail(GM_ECUDA, "k_relu_bwd");
}

int gm_nn_mse(const void* y, int ldy, const float* tgt, void* dy, int lddy, int nx, int ny, int nz, float scale,
              float* loss, int sx, int sy, int sym, void* stream) {
    if (sx < 0 || sx >= nx || sy < 0 || sy >= ny) return gm::fail(GM_EPARAM, "gm_nn_mse: shift out of range");
    if (sym < 0 || sym > 7 || ((sym & 4) && nx != ny))
        return gm::fail(GM_EPARAM, "gm_nn_mse: sym is 0..7, and the x <-> y swap needs nx == ny");
    const long long V = (long long)nx * ny * nz;
    gmnn::k_mse<<<gmnn::nb(V) > 256 ? 256 : gmnn::nb(V), 256, 0, (cudaStream_t)stream>>>(
        (const __nv_bfloat16*)y, ldy, tgt, (__nv_bfloat16*)dy, lddy, nx, ny, nz, scale, loss, sx, sy, sym);
    return cudaGetLastError() == cudaSuccess ? GM_OK : gm::fail(GM_ECUDA, "k_mse");
}

int gm_nn_adam(float* W, float* mW, float* vW, const float* gW, float* b, float* mb, float* vb, const float* gb, int co,
               int ci, float lr, float b1, float b2, int t, float eps, void* Wf, int Npo, int Kci, void* Wb, int Npi,
               int Kco, float* bpad, void* stream) {
    const float c1 = t > 0 ? 1.f - powf(b1, (float)t) : 1.f, c2 = t > 0 ? 1.f - powf(b2, (float)t) : 1.f;
    gmnn::k_adam<<<gmnn::nb(27LL * co * ci + co), 256, 0, (cudaStream_t)stream>>>(
        W, mW, vW, gW, b, mb, vb, gb, co, ci, lr, b1, b2, c1, c2, eps, (__nv_bfloat16*)Wf, Npo, Kci,
        (__nv_bfloat16*)Wb, Npi, Kco, bpad, t > 0 ? 1 : 0);
    return cudaGetLastError() == cudaSuccess ? GM_OK : gm::fail(GM_ECUDA, "k_adam");
}

}  // extern "C"
