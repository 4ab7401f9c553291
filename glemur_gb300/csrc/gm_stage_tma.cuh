// gm_stage_tma.cuh -- the RK stage kernel: TMA-fed plane rings, two points per
// thread.
//
//   * A tile is 32 x 2 NW columns (NW warps); a warp covers two rows of 16
//     x-neighbouring pairs, and a thread's arithmetic runs on its pair
//     (gm_vec2.cuh: packed FP32 instructions, 64-bit shared-memory accesses).
//   * One thread streams, plane by plane, every operand of the stage with
//     cp.async.bulk.tensor into shared-memory rings: the grid positions
//     (tile + 2-point halo, all three components as one 4-D box), the scaled
//     field B0s (same box) and the increments k_0..k_{n-1} over the tile;
//     completion is tracked by one mbarrier per ring slot.
//   * J for plane k is formed in the same iteration as B of plane k+1, so an
//     iteration needs a single __syncthreads; the march is unrolled by two, so
//     that the diagonals a, b, c of two planes alternate between two register
//     sets instead of being copied.
// Waits on the mbarriers are bounded: after kWaitLimit polls the CTA records
// GM_ST_TIMEOUT, drains the copies it has in flight (again bounded) and
// returns.
//
// What bounds it.  FP32: the algorithmic traffic of a stage is 12 + 3 n reals
// per point (21 + 3 in stage 5).  The form with one point per thread and
// scalar instructions took 450 to 650 thread instructions per point at 57 %
// issue activity: issue-bound, 0.44 of the measured HBM bandwidth.  FP64: the
// FP64 pipe (one warp instruction per 15 clocks and SM on a GB300), so what
// counts there is the number of FP64 operations per point.
#pragma once

#include <cuda.h>

#include <type_traits>

#include "gm_kernels_impl.cuh"
#include "gm_point.cuh"

namespace gmk {

constexpr int HX2 = TX + 4;              // row pitch of position, B0s and B planes: the tile + 2-point halo
constexpr unsigned kWaitLimit = 1u << 20;      // polls: about 1.3 s

// Tile of NW warps: 32 x 2 NW columns.
template <int NW>
struct TileShape {
    static constexpr int TYR = 2 * NW;                   // tile rows
    static constexpr int HYR = TYR + 4, BYR = TYR + 2;   // position / B plane rows
    static constexpr int PLANE_C = HYR * HX2;            // elements of one component of a position plane
    static constexpr int PLANE_X = 3 * PLANE_C;
    static constexpr int BPLANE_C = BYR * HX2;           // of a B plane
};

// elements rounded up so that a slot (a TMA destination) starts on 128 bytes
template <typename T>
constexpr int slot_round(int elems) {
    return (int)(((elems * sizeof(T) + 127) / 128) * 128 / sizeof(T));
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// bounded wait; returns false when the limit ran out
static __device__ __noinline__ bool mbar_wait_loop(uint64_t* bar, uint32_t parity) {
    for (unsigned it = 0; it < kWaitLimit; it++)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity) {
    return mbar_try_wait(bar, parity) || mbar_wait_loop(bar, parity);
}

__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2,
                                            int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
        : "memory");
}

// The columns of A at a pair / a point whose shared-memory addresses in the
// planes k-1, k, k+1 are xm, x0, xp; C is the component stride in bytes.
template <typename T, int C>
__device__ __forceinline__ void diffs(uint32_t xm, uint32_t x0, uint32_t xp, typename PairOf<T>::type A[3][3]) {
    constexpr int E = sizeof(T), R = HX2 * E;
#pragma unroll
    for (int l = 0; l < 3; l++) {
        const int q = l * C;
        const auto c = Sh<T>::ld2(x0 + q);
        A[l][0] = mk2(vsub(hi(c), Sh<T>::ld(x0 + q - E)), vsub(Sh<T>::ld(x0 + q + 2 * E), lo(c)));
        A[l][1] = vsub(Sh<T>::ld2(x0 + q + R), Sh<T>::ld2(x0 + q - R));
        A[l][2] = vsub(Sh<T>::ld2(xp + q), Sh<T>::ld2(xm + q));
    }
}
template <typename T, int C>
__device__ __forceinline__ void diffs1(uint32_t xm, uint32_t x0, uint32_t xp, T A[3][3]) {
    constexpr int E = sizeof(T), R = HX2 * E;
#pragma unroll
    for (int l = 0; l < 3; l++) {
        const int q = l * C;
        A[l][0] = vsub(Sh<T>::ld(x0 + q + E), Sh<T>::ld(x0 + q - E));
        A[l][1] = vsub(Sh<T>::ld(x0 + q + R), Sh<T>::ld(x0 + q - R));
        A[l][2] = vsub(Sh<T>::ld(xp + q), Sh<T>::ld(xm + q));
    }
}

// Positions around a point by its shared-memory addresses in the planes k-1, k,
// k+1 and in the B0s plane.  The face formula reads nothing else: the form that
// read B0 from global memory stalled every plane of a line-tied run (110 us a
// stage on 97x75x133, 35 % issue).
template <typename T, int C>
struct SharedX {
    uint32_t xm, x0, xp, b0;
    __device__ __forceinline__ T operator()(int l, int di, int dj, int dk) const {
        return Sh<T>::ld((dk < 0 ? xm : dk > 0 ? xp : x0) + (uint32_t)(l * C + (dj * HX2 + di) * (int)sizeof(T)));
    }
    __device__ __forceinline__ T s(int l) const { return Sh<T>::ld(b0 + l * C); }
};
template <int AX, int C, typename T>
__device__ __forceinline__ Vec3<T> b_face_s(const KP<T>& p, uint32_t xm, uint32_t x0, uint32_t xp, uint32_t b0, int i,
                                            int j, int k) {
    T r, d;
    return b_face_v<AX>(p, SharedX<T, C>{xm, x0, xp, b0}, i, j, k, &r, &d);
}
// the line-tied z ghost planes, two of a run (out of line, as det_sheared2)
template <int C, typename T>
__device__ __noinline__ Vec3<T> b_face_z(const KP<T>& p, uint32_t xm, uint32_t x0, uint32_t xp, uint32_t b0, int i,
                                         int j, int k) {
    return b_face_s<2, C>(p, xm, x0, xp, b0, i, j, k);
}

// Shared memory of the stage kernels, all in the dynamic buffer (the base is
// rounded up to 128 bytes at run time; the launch asks for 128 bytes of
// slack):
//   XR position-plane slots (the tile + 2-point halo, three components),
//   BR slots of B0s planes (same box),
//   KS slots of k-planes (the n arrays k_0..k_{n-1} over the tile),
//   3 B planes (the tile + face halo, in the pitch of the position planes),
//   the mbarriers, warp maxima, the abort flags and the work-item slot.
// Every slot is a multiple of 128 bytes, the alignment TMA destinations need.
// CTAs per SM the kernel is built for, of NW + 2 warps: FP32 16 warps an SM (up
// to 128 registers a thread; from 17 warps on the limit is 96), FP64 8; the
// shared memory follows.
constexpr int STAGE_HALO_WARPS = 2;
template <int NW>
constexpr int stage_threads() { return 32 * (NW + STAGE_HALO_WARPS); }
template <typename T, int NW>
constexpr int stage_ctas() { return (sizeof(T) == 4 ? 16 : 8) / (NW + STAGE_HALO_WARPS); }

template <typename T, bool PRESS, int NS, int NW>
struct StageSmem {
    using S = TileShape<NW>;
    static constexpr int SLOT = slot_round<T>(S::PLANE_X);
    static constexpr int BSLOT = slot_round<T>(3 * S::BPLANE_C);
    static constexpr int NK = NS;                                 // k arrays read by stage NS
    static constexpr int KBOX = 3 * S::TYR * TX;                  // elements of one k-array plane
    static constexpr int KSLOT = NK * KBOX;
    static constexpr int XMIN = PRESS ? 4 : 3;                    // position planes an iteration reads
    static constexpr size_t bytes(int xr, int br, int ks) {
        return sizeof(T) * ((size_t)(xr + br) * SLOT + 3 * (size_t)BSLOT + (size_t)ks * KSLOT) + 128 + 8 * (xr + br + ks) +
               8 * NW + 64;
    }
    static constexpr bool fits(int xr, int br, int ks) {
        return (bytes(xr, br, ks) + 1024) * stage_ctas<T, NW>() <= 228 * 1024;
    }
    // Position and B0s planes are loaded XR - XMIN and BR - 1 iterations ahead, two
    // where the CTAs per SM the kernel is built for still fit (an iteration is about
    // the latency of a copy: one ahead left 2.8 to 3.7 of 9.5 cycles per instruction
    // in waiting for it), else one.  k planes have two slots, or one where two would
    // not fit (the plane is then loaded during the B phase of its own iteration).
    static constexpr int KS = fits(XMIN + 1, 2, 2) ? 2 : 1;
    static constexpr int XR = fits(XMIN + 2, 2, KS) ? XMIN + 2 : XMIN + 1;
    static constexpr int BR = fits(XR, 3, KS) ? 3 : 2;
    static constexpr size_t OFF_B0 = sizeof(T) * (size_t)XR * SLOT;
    static constexpr size_t OFF_K = OFF_B0 + sizeof(T) * (size_t)BR * SLOT;
    static constexpr size_t OFF_B = OFF_K + sizeof(T) * KS * (size_t)KSLOT;
    static constexpr size_t OFF_BAR = OFF_B + sizeof(T) * 3 * (size_t)BSLOT;
    static constexpr int NBAR = XR + BR + KS;                    // x slots, B0s slots, k slots
    static constexpr size_t OFF_WMAX = OFF_BAR + 8 * NBAR;
    static constexpr size_t OFF_CTL = OFF_WMAX + 8 * NW;
    static constexpr size_t BYTES = bytes(XR, BR, KS);
    static_assert(BYTES <= 227 * 1024, "stage tile does not fit the shared memory");
};

// What a CTA keeps in shared memory besides the planes.
struct StageCtl {
    uint32_t ph;                 // completion parity of each mbarrier, carried from tile to tile
    // A bounded wait ran out: set in iteration kk's entry (kk & 1), which every
    // warp reads behind the next barrier, so that all leave in the same iteration.
    int abort[2];
    int work;                    // batched launch: the current work item
    int skip;                    // batched launch: the item's run is stopped (stage_stopped)
};

// Whether a tile has nothing to compute: a stopped run, or an earlier stage of this
// step that gave up a wait or failed its alignment check.  Another CTA of the same
// launch may set the status bits at any time, so one thread decides for its CTA, in
// front of a barrier: warps that each read the word could part, and those that went
// on would wait at the march's barrier (a fixed thread count) for the others forever.
__device__ __forceinline__ int stage_stopped(const DevState* st) {
    return st->done | (int)(st->status & (GM_ST_TIMEOUT | GM_ST_ALIGN));
}

// The start grid's own images, refreshed by stage 5 of the first attempted step
// (a retry reads them; until then they are those the caller supplied).
template <typename T>
__device__ __noinline__ void refresh_images(const KP<T>& p, T* X0, int i, int j, int k, bool pairs, bool two, int ix,
                                            int iy, int iz) {
    using V = typename PairOf<T>::type;
    T* q = X0 + gidx(p.px, p.py, i, j, k);
    if (pairs) {
        const V v[3] = {ldv2(q), ldv2(q + p.cs), ldv2(q + 2 * p.cs)};
        if (ix) st_xyz(q + ix, p.cs, image_shift<T>(v[0], ix, p.Lx, p.dx), v[1], v[2]);
        store_images_yz<T, V>(p, q, v, ix, iy, iz);
        return;
    }
    for (int h = 0; h < (two ? 2 : 1); h++) {
        const T u[3] = {q[h], q[h + p.cs], q[h + 2 * p.cs]};
        store_pos<T>(p, X0, i + h, j, k, u);
    }
}

// The pressure gradient at a pair on plane k from the planes k-1, k, k+1 (grad_p's
// formula): with the columns of A and r = 1/det A, jac^-1 = 2 d A^-1 and the
// second differences over d d, every spacing but that of p0's derivative
// cancels: grad(1/Delta) Delta = -4 sum_l S_l (A^-1)_l with S_l = sum_{a,b}
// delta_b delta_l x_a (A^-1)_{ba}.  The second differences are differences of
// differences of neighbours, which are exact or nearly so.
template <typename T, int C>
__device__ __forceinline__ void grad_p2(const KP<T>& p, uint32_t xm, uint32_t x0, uint32_t xp,
                                        const typename PairOf<T>::type A[3][3], typename PairOf<T>::type r,
                                        const typename PairOf<T>::type pe[3], typename PairOf<T>::type g[3]) {
    using V = typename PairOf<T>::type;
    using M = Sh<T>;
    constexpr int E = sizeof(T), R = HX2 * E;
    const V quarter = splat<V>((T)0.25);
    const V a[3] = {A[0][0], A[1][0], A[2][0]}, b[3] = {A[0][1], A[1][1], A[2][1]}, c[3] = {A[0][2], A[1][2], A[2][2]};
    V Ai[3][3];   // rows of A^-1
    vcross(b, c, Ai[0]);
    vcross(c, a, Ai[1]);
    vcross(a, b, Ai[2]);
#pragma unroll
    for (int e = 0; e < 9; e++) Ai[e / 3][e % 3] = vmul(Ai[e / 3][e % 3], r);
    V S[3];
#pragma unroll
    for (int l = 0; l < 3; l++) {
        const int q = l * C;
        const V xc = M::ld2(x0 + q);
        const V ex = mk2(M::ld(x0 + q - E), lo(xc)), fx = mk2(hi(xc), M::ld(x0 + q + 2 * E));
        const V yp = M::ld2(x0 + q + R), ym = M::ld2(x0 + q - R), zp = M::ld2(xp + q), zm = M::ld2(xm + q);
        const V dxx = vsub(vsub(fx, xc), vsub(xc, ex));
        const V dyy = vsub(vsub(yp, xc), vsub(xc, ym));
        const V dzz = vsub(vsub(zp, xc), vsub(xc, zm));
        // differences along y and z at x - 1 .. x + 2, then along x
        const V dy = vsub(yp, ym), dz = vsub(zp, zm);
        const T dyl = vsub(M::ld(x0 + q + R - E), M::ld(x0 + q - R - E));
        const T dyr = vsub(M::ld(x0 + q + R + 2 * E), M::ld(x0 + q - R + 2 * E));
        const T dzl = vsub(M::ld(xp + q - E), M::ld(xm + q - E)), dzr = vsub(M::ld(xp + q + 2 * E), M::ld(xm + q + 2 * E));
        const V dxy = vmul(mk2(vsub(hi(dy), dyl), vsub(dyr, lo(dy))), quarter);
        const V dxz = vmul(mk2(vsub(hi(dz), dzl), vsub(dzr, lo(dz))), quarter);
        const V dyz = vmul(vsub(vsub(M::ld2(xp + q + R), M::ld2(xm + q + R)), vsub(M::ld2(xp + q - R), M::ld2(xm + q - R))),
                           quarter);
        const V i0 = Ai[0][l], i1 = Ai[1][l], i2 = Ai[2][l];
        if (l == 0) {
            S[0] = vfma(dxx, i0, vfma(dxy, i1, vmul(dxz, i2)));
            S[1] = vfma(dxy, i0, vfma(dyy, i1, vmul(dyz, i2)));
            S[2] = vfma(dxz, i0, vfma(dyz, i1, vmul(dzz, i2)));
        } else {
            S[0] = vfma(dxx, i0, vfma(dxy, i1, vfma(dxz, i2, S[0])));
            S[1] = vfma(dxy, i0, vfma(dyy, i1, vfma(dyz, i2, S[1])));
            S[2] = vfma(dxz, i0, vfma(dyz, i1, vfma(dzz, i2, S[2])));
        }
    }
    // 1/Delta = r 8 dx dy dz
    const V det1 = vmul(r, splat<V>(p.vol8));
    const V w = vmul(pe[0], splat<V>((T)-4));
#pragma unroll
    for (int l = 0; l < 3; l++) {
        V t = vmul(w, vfma(S[0], Ai[0][l], vfma(S[1], Ai[1][l], vmul(S[2], Ai[2][l]))));
        t = vfma(pe[1], Ai[0][l], vfma(pe[2], Ai[1][l], t));
        g[l] = vmul(t, det1);
    }
}

// One RK stage over the 32 x 2 NW x TZ block (bx, by, bz) of one case.
// Iteration kk of the z march computes B on plane kb = kk - 1 (the tile and
// its face halo) and then J, k_n and the stage position on plane kc = kk - 2.
// NW warps own the tile's pairs: the diagonals a, b, c and 1/det of plane kc
// stay in their registers from the iteration that computed its B, and B of the
// planes kc - 1 and kc is read back from shared memory (three planes), written
// in the two previous iterations.  Two more warps compute B on the face halo,
// one of them issues and awaits the copies; as some of the NW warps' extra work
// it held up every iteration's barrier (3.2 of 10.6 cycles per instruction).  Halo
// points stand where the domain ends in a partial tile, so a pair is always
// inner points.  Operands arrive by TMA one iteration ahead: position plane
// kk + 1 (into the slot of plane kk + 1 - XR: the B phase last read it in the
// previous iteration, and so did the pressure gradient, which reads planes
// kc - 1 .. kc + 1, with its fifth slot), the B0s plane of the next B phase
// and the k planes of the next J phase.  `base` is the 128-byte aligned shared
// buffer with initialised mbarriers; the mbarrier parities in its StageCtl
// carry over to the next tile.  Returns false after a bounded wait ran out or
// an alignment check failed (the status word says which).  Every thread of the
// CTA is here: whether the tile is computed at all has been settled for all of
// them (stage_stopped).
//
// Stage 5 does not store x_6 = x_5 - sum b_5m k_m, the start of a rejected
// step's retry (rungeKutta.cu:216-227): it is x_0 up to rounding, and X[cur]
// still holds x_0.  With the cancellation-free error norm x_6 is not formed
// either: x_new = x_5 + sum_m (c_m - b_5m) k_m.
template <typename T, bool PRESS, int NS, int NW>
__device__ __forceinline__ bool stage_tile(const StageArgsTMA<T>& A, int bx, int by, int bz, unsigned char* base) {
    using V = typename PairOf<T>::type;
    using L = StageSmem<T, PRESS, NS, NW>;
    using S = TileShape<NW>;
    using M = Sh<T>;
    constexpr bool LAST = NS == 5;
    constexpr int n = NS;
    constexpr int XR = L::XR, BR = L::BR, KS = L::KS;
    constexpr int XD = XR - L::XMIN, BD = BR - 1;        // iterations the copies run ahead
    constexpr int TYR = S::TYR;
    // strides in bytes: element, row, components of the planes, slots
    constexpr int E = sizeof(T), R = HX2 * E, C = S::PLANE_C * E, BC = S::BPLANE_C * E, KC = TX * TYR * E;
    constexpr int XSLOT = L::SLOT * E, BSLOT = L::BSLOT * E, KSLOT = L::KSLOT * E;

    const StageArgs<T>& a = A.a;
    const KP<T>& p = a.p;
    DevState* st = a.st;

    uint64_t* bars = reinterpret_cast<uint64_t*>(base + L::OFF_BAR);       // x | B0s | k
    T* s_wmax = reinterpret_cast<T*>(base + L::OFF_WMAX);
    StageCtl* ctl = reinterpret_cast<StageCtl*>(base + L::OFF_CTL);
    volatile int* s_abort = ctl->abort;
    auto barrier = [] { asm volatile("bar.sync 1, %0;" ::"n"(stage_threads<NW>()) : "memory"); };
    uint32_t sb, tid;      // (volatile: kept, not recomputed)
    asm volatile("mov.u32 %0, %1;" : "=r"(sb) : "r"(smem_u32(base)));
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));
    const int lane = tid & 31, warp = tid >> 5;
    const int i0 = bx * TX, j0 = by * TYR, k0 = bz * a.TZ;
    const int nx = p.nx, ny = p.ny, nz = p.nz;
    const int kend = min(k0 + a.TZ, nz);
    const int cur = st->cur;
    const bool zPeri = p.zPeri != 0;

    // self-check of the alignment TMA needs: destination slots on 128 bytes,
    // mbarriers on 8 bytes, tensor maps on 64 bytes, box start on 16 bytes; on
    // failure record a status bit and issue no copy
    if ((sb & 127u) || ((XSLOT | KSLOT | (int)L::OFF_B0 | (int)L::OFF_K) & 127) || (smem_u32(bars) & 7u) ||
        (reinterpret_cast<uintptr_t>(&A.tm[0]) & 63u) || ((i0 * E) & 15)) {
        if (tid == 0) atomicOr(&st->status, (unsigned)GM_ST_ALIGN);
        return false;
    }
    const uint32_t ph0 = ctl->ph;      // rewritten at the end, behind a barrier
    // ring slot of a position plane
    auto xslot = [&](int plane) { return (plane + 20) % XR; };
    auto bslot = [&](int plane) { return (plane + 6) % BR; };
    auto kbar = [&](int q) { return XR + BR + (KS == 2 ? (q & 1) : 0); };
    T dmax = 0;
    bool bad = false;
    int kstop = kend + 2;              // the iteration that was left early

    if (warp >= NW) {
        // ---- the halo warps: NW the rows, NW + 1 the columns and the copies -------
        const bool producer = tid == 32 * (NW + 1), rows = warp == NW;
        const CUtensorMap* tmap = &A.tm[(n == 0) ? cur : 2 + ((n - 1) & 1)];
        uint32_t ph = ph0;
        auto wait_bar = [&](int b) {
            const bool ok = mbar_wait_bounded(&bars[b], (ph >> b) & 1u);
            ph ^= 1u << b;
            return ok;
        };
        auto issue_x = [&](int q) {
            uint64_t* b = &bars[xslot(q)];
            mbar_expect_tx(b, S::PLANE_X * E);
            tma_load_4d(base + xslot(q) * XSLOT, tmap, b, i0, j0, q + 2, 0);
        };
        auto issue_b0 = [&](int q) {
            uint64_t* b = &bars[XR + bslot(q)];
            mbar_expect_tx(b, S::PLANE_X * E);
            tma_load_4d(base + L::OFF_B0 + bslot(q) * XSLOT, &A.tm[4], b, i0, j0, q + 2, 0);
        };
        auto issue_k = [&](int q) {
            uint64_t* b = &bars[kbar(q)];
            mbar_expect_tx(b, KSLOT);
#pragma unroll
            for (int m = 0; m < n; m++)
                tma_load_4d(base + L::OFF_K + (KS == 2 ? (q & 1) : 0) * KSLOT + m * (L::KBOX * E), &A.tm[5 + m], b, i0, j0,
                            q, 0);
        };
        // rows: lanes 0-15 the row below the tile, 16-31 the row above it, one
        // pair each; columns: one point per lane, left then right
        const int ic = i0 + 2 * (lane & 15);
        const int iend = min(i0 + TX, nx), jend = min(j0 + TYR, ny);
        const bool hup = lane >= 16, hright = lane >= TYR;
        const int jR = hup ? jend : j0 - 1;
        const bool doR = rows && ic < nx, faceR = !p.yPeri && (hup ? jend == ny : j0 == 0);
        const int iC = hright ? iend : i0 - 1, jC = j0 + (lane % TYR);
        const bool doC = !rows && jC < ny && lane < 2 * TYR, faceC = !p.xPeri && (hright ? iend == nx : i0 == 0);
        const uint32_t aR = sb + ((jR - j0 + 2) * HX2 + (ic - i0 + 2)) * E;
        const uint32_t aC = sb + ((jC - j0 + 2) * HX2 + (iC - i0 + 2)) * E;
        // failure-detection test (a.stall): the first position planes are
        // withheld, so the bounded waits for them run out
        if (producer) {
            if (!a.stall)
                for (int q = k0 - 2; q <= min(k0 + XD, kend + 1); q++) issue_x(q);
            for (int q = k0 - 1; q <= min(k0 - 2 + BD, kend); q++) issue_b0(q);
        }
        uint32_t o2 = xslot(k0 - 2) * XSLOT, o1 = xslot(k0 - 1) * XSLOT, o0 = xslot(k0) * XSLOT;
        uint32_t q2 = 0, q1 = BSLOT, q0 = 2 * BSLOT;
        for (int kk = k0; kk <= kend + 1; kk++) {
            // position plane kk and the B0s plane of kb = kk-1 have arrived
            if (producer) {
                bool ok = true;
                for (int q = kk == k0 ? k0 - 2 : kk; q <= kk; q++) ok = wait_bar(xslot(q)) && ok;
                ok = wait_bar(XR + bslot(kk - 1)) && ok;
                if (!ok) {
                    s_abort[(kk - 1) & 1] = 1;
                    atomicOr(&st->status, (unsigned)GM_ST_TIMEOUT);
                }
            }
            barrier();
            if (s_abort[(kk - 1) & 1]) {
                kstop = kk;
                break;
            }
            // refills, into slots whose last reader was the previous iteration
            // (every thread is past this iteration's barrier)
            if (producer) {
                if (kk > k0 && kk + XD <= kend + 1) issue_x(kk + XD);
                if (kk - 1 + BD <= kend) issue_b0(kk - 1 + BD);
                // k planes: the next J phase's (two slots), or this one's (one slot:
                // the previous J phase, its last reader, is behind the barrier)
                const int qk = KS == 2 ? kk - 1 : kk - 2;
                if (n > 0 && qk >= k0 && qk < kend) issue_k(qk);
            }
            const int kb = kk - 1;
            if (kb >= k0 && kb < kend) {
                __syncwarp();
                const uint32_t ob0 = L::OFF_B0 + bslot(kb) * XSLOT, obd = L::OFF_B + q0 - R;
                if (doR) {
                    const uint32_t s0 = aR + ob0, d0 = aR + obd;
                    V Bh[3];
                    if (!faceR) {
                        V Ah[3][3], rh;
                        diffs<T, C>(aR + o2, aR + o1, aR + o0, Ah);
                        const V s[3] = {M::ld2(s0), M::ld2(s0 + C), M::ld2(s0 + 2 * C)};
                        b_from<T>(Ah, s, Bh, &rh, true);
                    } else {
                        const Vec3<T> u = b_face_s<1, C>(p, aR + o2, aR + o1, aR + o0, s0, ic, jR, kb);
                        const Vec3<T> v = b_face_s<1, C>(p, aR + o2 + E, aR + o1 + E, aR + o0 + E, s0 + E, ic + 1, jR, kb);
                        Bh[0] = mk2(u.x, v.x); Bh[1] = mk2(u.y, v.y); Bh[2] = mk2(u.z, v.z);
                    }
#pragma unroll
                    for (int l = 0; l < 3; l++) M::st2(d0 + l * BC, Bh[l]);
                }
                if (doC) {
                    const uint32_t s0 = aC + ob0, d0 = aC + obd;
                    T Bh[3];
                    if (!faceC) {
                        T Ah[3][3], rh;
                        diffs1<T, C>(aC + o2, aC + o1, aC + o0, Ah);
                        const T s[3] = {M::ld(s0), M::ld(s0 + C), M::ld(s0 + 2 * C)};
                        b_from<T>(Ah, s, Bh, &rh, true);
                    } else {
                        const Vec3<T> u = b_face_s<0, C>(p, aC + o2, aC + o1, aC + o0, s0, iC, jC, kb);
                        Bh[0] = u.x; Bh[1] = u.y; Bh[2] = u.z;
                    }
#pragma unroll
                    for (int l = 0; l < 3; l++) M::st(d0 + l * BC, Bh[l]);
                }
                __syncwarp();
            }
            o2 = o1; o1 = o0;
            o0 = o0 == (XR - 1) * XSLOT ? 0 : o0 + XSLOT;
            const uint32_t qt = q2;
            q2 = q1; q1 = q0; q0 = qt;
        }
        // the k planes are awaited by the warps that read them; their parities
        // follow from the tile's planes
        if (producer) {
            if (n > 0)
                for (int q = k0; q < kend; q++) ph ^= 1u << kbar(q);
            ctl->ph = ph;
        }
    } else {
        // ---- a pair of the tile: columns ic, ic + 1 of row jc -------------------
        const int ic = i0 + 2 * (lane & 15), jr = 2 * warp + (lane >> 4), jc = j0 + jr;
        const bool own = ic < nx && jc < ny, own2 = own && ic + 1 < nx;
        const uint32_t ax = sb + ((jr + 2) * HX2 + (ic - i0 + 2)) * E;          // in a position / B0s plane
        const uint32_t ab = ax + (uint32_t)L::OFF_B - R;                        // in a B plane (one halo row fewer)
        const uint32_t ak = sb + (uint32_t)L::OFF_K + (jr * TX + (ic - i0)) * E;
        const T dtT = (T)st->dt;
        V exy = splat<V>((T)0);
        if (own) exy = mk2(vmul(vmul(p.ex[ic], p.ey[jc]), dtT), own2 ? vmul(vmul(p.ex[ic + 1], p.ey[jc]), dtT) : (T)0);
        const int iy = image_step(p.yPeri, jc, ny), ix = image_step(p.xPeri, ic, nx);
        // both points of a pair have the same images when nx is even; an odd nx,
        // or a direction of three points (two images), takes the general store
        const bool pairs = !(nx & 1) && !(p.xPeri && nx < 4) && !(p.yPeri && ny < 4) && !(zPeri && nz < 4);
        const bool xyimage = (iy | ix | image_step(p.xPeri, ic + 1, nx)) != 0;
        const bool first = LAST && st->nAttempted == 0;
        V pe[3];
        if (PRESS) {
            T e[2][3];
#pragma unroll
            for (int h = 0; h < 2; h++) p0_at(p, ic + h, jc, e[h]);
#pragma unroll
            for (int q = 0; q < 3; q++) pe[q] = mk2(e[0][q], e[1][q]);
        }
        // addresses of the pair in the position planes kk - 3 .. kk and in the B
        // planes kb - 2 .. kb, stepped with kk
        uint32_t x3 = ax + xslot(k0 - 3) * XSLOT, x2 = ax + xslot(k0 - 2) * XSLOT, x1 = ax + xslot(k0 - 1) * XSLOT,
                 x0 = ax + xslot(k0) * XSLOT;
        uint32_t b2 = ab, b1 = ab + BSLOT, b0 = ab + 2 * BSLOT;
        uint32_t kph = ph0 >> (XR + BR);         // parity of the k slots
        uint32_t s0 = ax + (uint32_t)L::OFF_B0 + bslot(k0 - 1) * XSLOT;      // in the B0s plane kb
        // the outputs: the plane's base (the same for all threads) and the pair's
        // offset in the plane, in bytes
        T* const Xb = LAST ? a.X[cur ^ 1] : a.XS[n & 1];
        char* xo = reinterpret_cast<char*>(Xb + (long long)p.px * p.py * (k0 + 2));
        char* ko = LAST ? nullptr : reinterpret_cast<char*>(a.K[n] + (long long)p.kpx * ny * k0);
        const uint32_t gx = (uint32_t)(ic + 2 + p.px * (jc + 2)) * E, gk = (uint32_t)(ic + p.kpx * jc) * E;
        const long long cs = p.cs * E, kcs = p.kcs * E;

        // One iteration; Ac, Rc: the diagonals of plane kc, An, Rn: those of plane kb.
        auto iteration = [&](int kk, const V (&Ac)[3][3], const V& Rc, V (&An)[3][3], V& Rn) -> bool {
            const int kb = kk - 1, kc = kk - 2;
            const T ezk = __ldg(&p.ez[max(kc, 0)]);
            barrier();
            if (s_abort[(kk - 1) & 1]) return false;
            // B on plane kb
            V Bp[3];
            {
                if (!zPeri && (unsigned)kb >= (unsigned)nz) {
                    // line-tied ghost plane
                    Vec3<T> u = {0, 0, 0}, v = {0, 0, 0};
                    if (own) u = b_face_z<C, T>(p, x2, x1, x0, s0, ic, jc, kb);
                    if (own2) v = b_face_z<C, T>(p, x2 + E, x1 + E, x0 + E, s0 + E, ic + 1, jc, kb);
                    Bp[0] = mk2(u.x, v.x); Bp[1] = mk2(u.y, v.y); Bp[2] = mk2(u.z, v.z);
                } else {
                    diffs<T, C>(x2, x1, x0, An);
                    const V s[3] = {M::ld2(s0), M::ld2(s0 + C), M::ld2(s0 + 2 * C)};
                    b_from<T>(An, s, Bp, &Rn, own);
                }
#pragma unroll
                for (int l = 0; l < 3; l++) M::st2_if(own2, b0 + l * BC, Bp[l]);
                if ((nx & 1) && own && !own2) {
#pragma unroll
                    for (int l = 0; l < 3; l++) M::st(b0 + l * BC, lo(Bp[l]));
                }
            }
            // J, k_n and the stage position on plane kc
            if (kc >= k0) {
                // Stokes current (current.cu:290-406).  The circulation around a
                // quadrilateral P1..P4, sum (B_a + B_b).(x_b - x_a) over its edges,
                // regroups exactly into sum B_a.(x_{a+1} - x_{a-1}); for the quads
                // through the face neighbours (-x,-y,+x,+y), (-y,-z,+y,+z) and
                // (-z,-x,+z,+x) that is I0 = b.dxB - a.dyB, I1 = c.dyB - b.dzB and
                // I2 = a.dzB - c.dxB with the diagonals a = x(+x) - x(-x), b, c and
                // dxB = B(+x) - B(-x), ...  The quads' area vectors are
                // (1/2) a x b, (1/2) b x c, (1/2) c x a (for a quadrilateral,
                // (1/4) sum of consecutive edge cross products = (1/2) d1 x d2),
                // and the matrix with those rows has the inverse
                // 2 [a b c] P / det(a, b, c), so J = (a I1 + b I2 + c I0) / det.
                V I0, I1, I2, Bz[3];
#pragma unroll
                for (int l = 0; l < 3; l++) {
                    Bz[l] = M::ld2(b1 + l * BC);
                    const V dx = mk2(vsub(hi(Bz[l]), M::ld(b1 + l * BC - E)), vsub(M::ld(b1 + l * BC + 2 * E), lo(Bz[l])));
                    const V dy = vsub(M::ld2(b1 + l * BC + R), M::ld2(b1 + l * BC - R));
                    const V dz = vsub(Bp[l], M::ld2(b2 + l * BC));
                    if (l == 0) {
                        I0 = vfms(Ac[l][1], dx, vmul(Ac[l][0], dy));
                        I1 = vfms(Ac[l][2], dy, vmul(Ac[l][1], dz));
                        I2 = vfms(Ac[l][0], dz, vmul(Ac[l][2], dx));
                    } else {
                        I0 = vfma(Ac[l][1], dx, vfma(vneg(Ac[l][0]), dy, I0));
                        I1 = vfma(Ac[l][2], dy, vfma(vneg(Ac[l][1]), dz, I1));
                        I2 = vfma(Ac[l][0], dz, vfma(vneg(Ac[l][2]), dx, I2));
                    }
                }
                V Jv[3], kn[3];
#pragma unroll
                for (int l = 0; l < 3; l++) Jv[l] = vfma(Ac[l][0], I1, vfma(Ac[l][1], I2, vmul(Ac[l][2], I0)));
                vcross(Jv, Bz, kn);
                const V f = vmul(vmul(exy, splat<V>(ezk)), Rc);
#pragma unroll
                for (int l = 0; l < 3; l++) kn[l] = vmul(kn[l], f);
                if (PRESS) {
                    V gp[3];
                    grad_p2<T, C>(p, x3, x2, x1, Ac, Rc, pe, gp);
#pragma unroll
                    for (int l = 0; l < 3; l++) kn[l] = vfma(splat<V>(-dtT), gp[l], kn[l]);
                }
                V xa[3];
#pragma unroll
                for (int l = 0; l < 3; l++) xa[l] = M::ld2(x2 + l * C);
                uint32_t kp = ak;                    // k_m component l at kp + (3 m + l) KC
                if (n > 0) {
                    const int ks = KS == 2 ? (kc & 1) : 0;
                    kp += ks * KSLOT;
                    if (!mbar_wait_bounded(&bars[XR + BR + ks], (kph >> ks) & 1u)) {
                        s_abort[kk & 1] = 1;
                        atomicOr(&st->status, (unsigned)GM_ST_TIMEOUT);
                    }
                    kph ^= 1u << ks;
                }
                if (!LAST) {
                    // x_{n+1} = x_n + sum_{m<=n} (b[n+1][m] - b[n][m]) k_m (rungeKutta.cu:216-227)
#pragma unroll
                    for (int m = 0; m < n; m++) {
                        const V w = splat<V>(p.db[n][m]);
#pragma unroll
                        for (int l = 0; l < 3; l++) xa[l] = vfma(w, M::ld2(kp + (3 * m + l) * KC), xa[l]);
                    }
                    const V w = splat<V>(p.db[n][n]);
#pragma unroll
                    for (int l = 0; l < 3; l++) xa[l] = vfma(w, kn[l], xa[l]);
                    if (own2) {
#pragma unroll
                        for (int l = 0; l < 3; l++) stv(reinterpret_cast<T*>(ko + l * kcs + gk), kn[l]);
                    }
                    if ((nx & 1) && own && !own2) {
#pragma unroll
                        for (int l = 0; l < 3; l++) *reinterpret_cast<T*>(ko + l * kcs + gk) = lo(kn[l]);
                    }
                } else {
                    // stage 5: x_new and the error norm |x_new - x*| or |sum (c - c*) k|
                    V e[3];
                    if (p.errMode == 0) {
                        // the reference's sums in their order (x_6 and its last term, which
                        // is zero, apart; c_1 = c_4 = c*_1 = 0): a first step's error norm is
                        // rounding, and its dt follows from it
                        V xst[3];
#pragma unroll
                        for (int m = 0; m < 5; m++)
#pragma unroll
                            for (int l = 0; l < 3; l++)
                                xa[l] = vfma(splat<V>(p.db[5][m]), M::ld2(kp + (3 * m + l) * KC), xa[l]);
#pragma unroll
                        for (int l = 0; l < 3; l++) xst[l] = xa[l];
#pragma unroll
                        for (int m = 0; m < 6; m++) {
                            if (m == 1) continue;
#pragma unroll
                            for (int l = 0; l < 3; l++) {
                                if (l == 2 && !p.zUpdate) continue;
                                const V km = m < 5 ? M::ld2(kp + (3 * m + l) * KC) : kn[l];
                                if (m != 4) xa[l] = vfma(splat<V>(p.c[m]), km, xa[l]);
                                xst[l] = vfma(splat<V>(p.cst[m]), km, xst[l]);
                            }
                        }
#pragma unroll
                        for (int l = 0; l < 3; l++) e[l] = vsub(xa[l], xst[l]);
                    } else {
                        // sum (c - c*) k: no cancellation against x
                        e[0] = e[1] = e[2] = splat<V>((T)0);
#pragma unroll
                        for (int m = 0; m < 6; m++) {
                            const V wc = splat<V>(p.cb[m]), wz = splat<V>(p.cbz[m]), we = splat<V>(p.cmcT[m]);
#pragma unroll
                            for (int l = 0; l < 3; l++) {
                                const V km = m < 5 ? M::ld2(kp + (3 * m + l) * KC) : kn[l];
                                xa[l] = vfma(l == 2 ? wz : wc, km, xa[l]);
                                e[l] = vfma(we, km, e[l]);
                            }
                        }
                    }
#pragma unroll
                    for (int l = 0; l < 3; l++) {
                        const T y1 = lo(xa[l]), y2 = hi(xa[l]), e1 = lo(e[l]), e2 = hi(e[l]);
                        if (own && (l < 2 || p.zUpdate)) max_nn(dmax, e1);
                        if (own2 && (l < 2 || p.zUpdate)) max_nn(dmax, e2);
                        // NaN/Inf anywhere in k_0..k_5
                        bad |= own && (!finite_bits(y1) || !finite_bits(e1));
                        bad |= own2 && (!finite_bits(y2) || !finite_bits(e2));
                    }
                }
                const int iz = image_step(p.zPeri, kc, nz);
                if (pairs) {
                    if (own2) {
#pragma unroll
                        for (int l = 0; l < 3; l++) stv(reinterpret_cast<T*>(xo + l * cs + gx), xa[l]);
                    }
                    if (own2 && (ix | iy | iz)) {
                        T* q = reinterpret_cast<T*>(xo + gx);
                        if (ix) st_xyz(q + ix, p.cs, image_shift<T>(xa[0], ix, p.Lx, p.dx), xa[1], xa[2]);
                        if (iy | iz) store_images_call<T, V>(p, q, xa[0], xa[1], xa[2], ix, iy, iz);
                    }
                } else {
                    T* q = reinterpret_cast<T*>(xo + gx);
                    if (own) st_xyz(q, p.cs, lo(xa[0]), lo(xa[1]), lo(xa[2]));
                    if (own2) st_xyz(q + 1, p.cs, hi(xa[0]), hi(xa[1]), hi(xa[2]));
                    if (own && (xyimage || iz)) {
                        store_point_images<T>(p, Xb, ic, jc, kc, lo(xa[0]), lo(xa[1]), lo(xa[2]));
                        if (own2) store_point_images<T>(p, Xb, ic + 1, jc, kc, hi(xa[0]), hi(xa[1]), hi(xa[2]));
                    }
                }
                if (LAST && first && own && (xyimage || iz)) refresh_images<T>(p, a.X[cur], ic, jc, kc, pairs, own2, ix, iy, iz);
                xo += (long long)p.px * p.py * E;
                if (!LAST) ko += (long long)p.kpx * ny * E;
            }
            // step the rings
            x3 = x2; x2 = x1; x1 = x0;
            x0 = x0 == ax + (XR - 1) * XSLOT ? ax : x0 + XSLOT;
            const uint32_t bt = b2;
            b2 = b1; b1 = b0; b0 = bt;
            s0 = s0 == ax + (uint32_t)L::OFF_B0 + (BR - 1) * XSLOT ? ax + (uint32_t)L::OFF_B0 : s0 + XSLOT;
            return true;
        };

        const V zero = splat<V>((T)0);
        V A0[3][3], A1[3][3], R0 = zero, R1 = zero;
#pragma unroll
        for (int e = 0; e < 9; e++) { A0[e / 3][e % 3] = zero; A1[e / 3][e % 3] = zero; }
#pragma unroll 1
        for (int kk = k0; kk <= kend + 1; kk += 2) {
            if (!iteration(kk, A0, R0, A1, R1)) break;
            if (kk + 1 > kend + 1) break;
            if (!iteration(kk + 1, A1, R1, A0, R0)) break;
        }
    }
    if (bad) atomicOr(&st->status, (unsigned)GM_ST_NAN);
    if (LAST) {
        for (int o = 16; o > 0; o >>= 1) max_nn(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
        if (lane == 0 && warp < NW) s_wmax[warp] = dmax;
    }
    __syncthreads();       // the warp maxima; ctl for the next tile
    const bool left = s_abort[0] || s_abort[1];
    if (left && tid == 32 * (NW + 1)) {
        // left early: the copies that may still be in flight (bounded waits); those
        // of an iteration's start have been waited for.  A slot's parity follows
        // from the tile's earlier planes in it.
        auto drain = [&](int b, int uses) { mbar_wait_bounded(&bars[b], ((ph0 >> b) + uses) & 1u); };
        for (int q = kstop + 1; q <= min(max(kstop - 1, k0) + XD, kend + 1); q++) drain(xslot(q), (q - (k0 - 2)) / XR);
        for (int q = kstop; q <= min(kstop - 2 + BD, kend); q++) drain(XR + bslot(q), (q - (k0 - 1)) / BR);
        if (n > 0)
            for (int q = max(k0, kstop - 3); q <= min(kstop - (KS == 2 ? 2 : 3), kend - 1); q++)
                drain(kbar(q), KS == 2 ? (q - k0) / 2 : q - k0);
    }
    if (LAST && tid == 0) {
        T m = 0;
        for (int w = 0; w < NW; w++) max_nn(m, s_wmax[w]);
        if (m > 0) atomicMax(&st->maxDeltaBits, (unsigned long long)__double_as_longlong((double)m));
    }
    return !left;
}

// Shared-memory set-up common to the stage kernels: the 128-byte aligned
// base, the mbarriers and the abort flag.
template <typename T, bool PRESS, int NS, int NW>
__device__ __forceinline__ unsigned char* stage_smem_setup(unsigned char* smraw) {
    using L = StageSmem<T, PRESS, NS, NW>;
    unsigned char* base = smraw + ((128u - (smem_u32(smraw) & 127u)) & 127u);
    uint64_t* bars = reinterpret_cast<uint64_t*>(base + L::OFF_BAR);
    StageCtl* ctl = reinterpret_cast<StageCtl*>(base + L::OFF_CTL);
    if (threadIdx.x == 0) {
        ctl->ph = 0;
        ctl->abort[0] = ctl->abort[1] = 0;
        for (int s = 0; s < L::NBAR; s++) mbar_init(&bars[s], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    return base;
}

// One RK stage of one case: one CTA per 32 x 2 NW x TZ block.
template <typename T, bool PRESS, int NS, int NW>
__global__ void __launch_bounds__(stage_threads<NW>(), stage_ctas<T, NW>())
    k_stage_tma(const __grid_constant__ StageArgsTMA<T> A) {
    extern __shared__ __align__(128) unsigned char smraw[];
    if (__syncthreads_or(threadIdx.x == 0 ? stage_stopped(A.a.st) : 0)) return;
    unsigned char* base = stage_smem_setup<T, PRESS, NS, NW>(smraw);
    stage_tile<T, PRESS, NS, NW>(A, blockIdx.x, blockIdx.y, blockIdx.z, base);
}

// One RK stage of many cases: a persistent launch whose CTAs take work items
// (case, tile) from a counter until none is left; cases whose controller has
// stopped are skipped.  The counter is reset by the batched controller.
template <typename T, bool PRESS, int NS>
__global__ void __launch_bounds__(stage_threads<STAGE_BATCH_NW>(), stage_ctas<T, STAGE_BATCH_NW>())
    k_stage_tma_batch(const StageArgsTMA<T>* __restrict__ cases, const int4* __restrict__ work, int nwork,
                      int* __restrict__ counter) {
    constexpr int NW = STAGE_BATCH_NW;
    using L = StageSmem<T, PRESS, NS, NW>;
    extern __shared__ __align__(128) unsigned char smraw[];
    unsigned char* base = stage_smem_setup<T, PRESS, NS, NW>(smraw);
    StageCtl* ctl = reinterpret_cast<StageCtl*>(base + L::OFF_CTL);
    for (;;) {
        if (threadIdx.x == 0) {
            const int w = atomicAdd(counter, 1);
            ctl->work = w;
            ctl->skip = w < nwork && stage_stopped(cases[work[w].x].a.st);
        }
        __syncthreads();
        const int w = ctl->work, skip = ctl->skip;
        __syncthreads();   // both are rewritten only after every thread has read them
        if (w >= nwork) break;
        if (skip) continue;
        const int4 it = work[w];
        if (!stage_tile<T, PRESS, NS, NW>(cases[it.x], it.y, it.z, it.w, base)) break;
        __syncthreads();   // the next tile's copies overwrite slots this one read
    }
}

// f(integral constant NS) for a run-time stage index
template <typename F>
static auto stage_dispatch(int n, F f) {
    switch (n) {
        case 0: return f(std::integral_constant<int, 0>());
        case 1: return f(std::integral_constant<int, 1>());
        case 2: return f(std::integral_constant<int, 2>());
        case 3: return f(std::integral_constant<int, 3>());
        case 4: return f(std::integral_constant<int, 4>());
        default: return f(std::integral_constant<int, 5>());
    }
}

template <typename T, bool PRESS>
cudaError_t prepare_stage_tma_p() {
    const int lim = 227 * 1024;
    for (int n = 0; n < 6; n++) {
        const cudaError_t e = stage_dispatch(n, [&](auto N) {
            cudaError_t r = cudaFuncSetAttribute(k_stage_tma<T, PRESS, N.value, STAGE_NW>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
            if (r == cudaSuccess)
                r = cudaFuncSetAttribute(k_stage_tma<T, PRESS, N.value, STAGE_NW_SMALL>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
            if (r == cudaSuccess)
                r = cudaFuncSetAttribute(k_stage_tma_batch<T, PRESS, N.value>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         lim);
            return r;
        });
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

template <typename T, bool PRESS>
int stage_tma_batch_occupancy_p() {
    int nb = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &nb, k_stage_tma_batch<T, PRESS, 5>, stage_threads<STAGE_BATCH_NW>(), StageSmem<T, PRESS, 5, STAGE_BATCH_NW>::BYTES);
    return e == cudaSuccess && nb > 0 ? nb : 1;
}

template <typename T, bool PRESS>
cudaError_t launch_stage_tma_batch_p(const StageArgsTMA<T>* cases, const int4* work, int nwork, int* counter, int n,
                                     int nblocks, cudaStream_t s) {
    return stage_dispatch(n, [&](auto N) {
        constexpr size_t sm = StageSmem<T, PRESS, N.value, STAGE_BATCH_NW>::BYTES;
        k_stage_tma_batch<T, PRESS, N.value><<<nblocks, stage_threads<STAGE_BATCH_NW>(), sm, s>>>(cases, work, nwork, counter);
        return cudaGetLastError();
    });
}

template <typename T, bool PRESS>
cudaError_t launch_stage_tma_p(const StageArgsTMA<T>& A, int nw, dim3 grid, cudaStream_t s) {
    return stage_dispatch(A.a.n, [&](auto N) {
        if (nw == STAGE_NW)
            k_stage_tma<T, PRESS, N.value, STAGE_NW>
                <<<grid, stage_threads<STAGE_NW>(), StageSmem<T, PRESS, N.value, STAGE_NW>::BYTES, s>>>(A);
        else
            k_stage_tma<T, PRESS, N.value, STAGE_NW_SMALL>
                <<<grid, stage_threads<STAGE_NW_SMALL>(), StageSmem<T, PRESS, N.value, STAGE_NW_SMALL>::BYTES, s>>>(A);
        return cudaGetLastError();
    });
}

#define GMK_INSTANTIATE_TMA(T, PRESS)                                                                          \
    template cudaError_t prepare_stage_tma_p<T, PRESS>();                                                      \
    template cudaError_t launch_stage_tma_p<T, PRESS>(const StageArgsTMA<T>&, int, dim3, cudaStream_t);        \
    template int stage_tma_batch_occupancy_p<T, PRESS>();                                                      \
    template cudaError_t launch_stage_tma_batch_p<T, PRESS>(const StageArgsTMA<T>*, const int4*, int, int*, int, int, \
                                                            cudaStream_t);

}  // namespace gmk
