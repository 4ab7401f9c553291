// gm_fields.cuh -- the relaxation in two elementwise passes: B at every point
// (k_b_field), then J, the increment and the stage position from it
// (k_stage_field), or J and the reductions (k_diag_field).
//
// Which runs use it:
//   * the frictional Stokes stages in FP64 (single case).  A GB300 SM issues one
//     FP64 warp instruction in 15 clocks, so those stages cost their FP64
//     operations; the one-pass tile kernel computes B again on the halo of every
//     tile, 19 to 75 % of the points in x, y and two planes of every z chunk.
//     Here each B is formed once (34 operations) and the stage needs 57 more
//     and its sums, lanes are full for any nx, and the points spread evenly over
//     the SMs.  The second pass's reads hit L2 or hide behind the FP64 pipe.
//   * the inertial equation, the Classic current, and the currents that come from a
//     kernel of their own (Stokes4th, StokesQuint, StokesTri), in either precision:
//     their stages ran in the general tile kernel, one CTA per SM, waiting for its
//     loads.
//   * gm_refresh and the convergence checks of a batch.
//
// In FP64 a point's arithmetic is that of the tile kernel (gm_stage_tma.cuh),
// operation by operation, so results do not depend on which of the two ran (the B and
// Delta that gm_refresh exports are the general tile kernel's).  In
// FP32 B, J and the velocity's increments keep the formulas of the general tile
// kernel (`kPlain`): J is a difference quotient of B, and its rounding (1e-5 of
// |J| on 128x128x256) enters the velocity and the exported J at first order, so
// another form, though closer to the exact value, would move them by as much.
#pragma once

#include <type_traits>

#include "gm_kernels_impl.cuh"
#include "gm_point.cuh"

namespace gmk {

template <typename T>
constexpr int field_threads() { return sizeof(T) == 8 ? 64 : 128; }

// the grid a stage reads (the step start for stage 0, chosen on the device)
template <typename T>
__device__ __forceinline__ const T* stage_input(const StageArgs<T>& a) {
    return a.n == 0 ? a.X[a.st->cur] : a.XS[(a.n - 1) & 1];
}

// A load of what a kernel of the step has written (positions, B and Delta, J, the
// increments): these grids start while the one before still runs, and __ldg is for data
// that no one writes while the grid is there.  An ordinary load, in its place behind
// after_previous.  (Left to the compiler, the loads of k_b_field in FP64 came as they were
// used: 32x32x64 133 -> 148 us a step.)  B0 and its scaled copy are the upload's.

__device__ __forceinline__ float ld_step(const float* q) {
    float r;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(r) : "l"(q));
    return r;
}
__device__ __forceinline__ double ld_step(const double* q) {
    double r;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(r) : "l"(q));
    return r;
}
// Positions around the point at padded index g in global memory.
template <typename T>
struct GlobalX {
    const T* x;
    const T* b0s;
    int px, pxy;
    long long cs;
    __device__ __forceinline__ T operator()(int l, int di, int dj, int dk) const {
        return ld_step(x + l * cs + di + dj * px + dk * pxy);
    }
    __device__ __forceinline__ T s(int l) const { return __ldg(b0s + l * cs); }
};
template <typename T>
__device__ __forceinline__ GlobalX<T> at_point(const KP<T>& p, const T* X, const T* B0s, long long g) {
    return GlobalX<T>{X + g, B0s + g, p.px, p.px * p.py, p.cs};
}

template <typename T>
constexpr bool kPlain = sizeof(T) == 4;

// the padded positions as the tile accessor of b_face and grad_p
template <typename T>
struct GlobalTile {
    const KP<T>& p;
    const T* X;
    __device__ __forceinline__ T x(int k, int l, int j, int i) const {
        return ld_step(X + l * p.cs + gidx(p.px, p.py, i, j, k));
    }
};

// As the general tile kernel's tile for j_classic: the positions, and 1/Delta from RF
// (FP64: 1/det(a, b, c), so no division).
template <typename T>
struct ClassicTile {
    const KP<T>& p;
    const T *X, *RF;
    __device__ __forceinline__ T x(int k, int l, int j, int i) const {
        return ld_step(X + l * p.cs + gidx(p.px, p.py, i, j, k));
    }
};
template <typename T>
__device__ __forceinline__ T inv_delta(const ClassicTile<T>& t, int k, int j, int i) {
    const T r = ld_step(t.RF + gidx(t.p.px, t.p.py, i, j, k));
    return sizeof(T) == 4 ? rcp_rn(r) : vmul(r, t.p.vol8);
}

// B and Delta at an inner or image point: B_JacB0 (rungeKutta.cu:79-106), as
// b_interior.
template <typename T>
__device__ __forceinline__ void b_plain(const KP<T>& p, const GlobalX<T>& X, const T* __restrict__ B0, long long g,
                                        T B[3], T* D) {
    T jac[3][3];
#pragma unroll
    for (int l = 0; l < 3; l++) {
        jac[l][0] = (X(l, 1, 0, 0) - X(l, -1, 0, 0)) * p.hdx1;
        jac[l][1] = (X(l, 0, 1, 0) - X(l, 0, -1, 0)) * p.hdy1;
        jac[l][2] = (X(l, 0, 0, 1) - X(l, 0, 0, -1)) * p.hdz1;
    }
    const T detJac1 = rcp_rn(det_guarded(jac));
    const T b0 = __ldg(&B0[g]), b1 = __ldg(&B0[p.cs + g]), b2 = __ldg(&B0[2 * p.cs + g]);
#pragma unroll
    for (int l = 0; l < 3; l++) B[l] = (jac[l][0] * b0 + jac[l][1] * b1 + jac[l][2] * b2) * detJac1;
    *D = rcp_rn(detJac1);
}

// B at the inner points and on the faces next to them (line-tied: updateBbound's
// formula; periodic: at the image points).  OUT: B and Delta into the exported
// arrays; else B and 1/det(a, b, c) (FP32: Delta) into the padded fields BF, RF.  PLAIN:
// by the general tile kernel's formulas, for FP32 and for what gm_refresh exports: the
// folded constants of the other form are one more rounding each (FP64 braids: B off by
// 2.2e-16 of its norm against 1.8e-16, Delta by 2.0e-16 against 1.7e-16).
template <typename T, bool OUT, bool PLAIN>
__global__ void __launch_bounds__(field_threads<T>()) k_b_field(const __grid_constant__ StageArgs<T> a, int always) {
    const KP<T>& p = a.p;
    after_previous();
    let_next();
    if (!always && a.st->done) return;
    const int nx = p.nx, ny = p.ny, nz = p.nz;
    const unsigned q = blockIdx.x * (unsigned)field_threads<T>() + threadIdx.x, N = (unsigned)p.N;
    int i, j, k, face = -1;
    if (q < N) {
        const unsigned r = q / (unsigned)nx;
        i = (int)(q - r * (unsigned)nx);
        k = (int)(r / (unsigned)ny);
        j = (int)(r - (unsigned)k * (unsigned)ny);
    } else {
        unsigned f = q - N;
        const unsigned nyz = (unsigned)ny * nz, nxz = (unsigned)nx * nz, nxy = (unsigned)nx * ny;
        if (f < 2 * nyz) {
            face = 0;
            i = f < nyz ? -1 : nx;
            f = f < nyz ? f : f - nyz;
            j = (int)(f % ny); k = (int)(f / ny);
        } else if ((f -= 2 * nyz) < 2 * nxz) {
            face = 1;
            j = f < nxz ? -1 : ny;
            f = f < nxz ? f : f - nxz;
            i = (int)(f % nx); k = (int)(f / nx);
        } else if ((f -= 2 * nxz) < 2 * nxy) {
            face = 2;
            k = f < nxy ? -1 : nz;
            f = f < nxy ? f : f - nxy;
            i = (int)(f % nx); j = (int)(f / nx);
        } else {
            return;
        }
    }
    const long long g = gidx(p.px, p.py, i, j, k);
    const GlobalX<T> X = at_point(p, stage_input(a), a.B0s, g);
    const bool tied = (face == 0 && !p.xPeri) || (face == 1 && !p.yPeri) || (face == 2 && !p.zPeri);
    T B[3], r, D;
    if (PLAIN) {
        const GlobalTile<T> t{p, stage_input(a)};
        if (tied && face == 0) b_face<T>(p, t, a.B0, 0, i, j, k, B, &D);
        else if (tied && face == 1) b_face<T>(p, t, a.B0, 1, i, j, k, B, &D);
        else if (tied) b_face<T>(p, t, a.B0, 2, i, j, k, B, &D);
        else b_plain(p, X, a.B0, g, B, &D);
        r = D;
    } else {
        T d;
        if (tied) {
            const Vec3<T> v = face == 0   ? b_face_v<0>(p, X, i, j, k, &r, &d)
                              : face == 1 ? b_face_v<1>(p, X, i, j, k, &r, &d)
                                          : b_face_v<2>(p, X, i, j, k, &r, &d);
            B[0] = v.x; B[1] = v.y; B[2] = v.z;
        } else {
            T A[3][3];
            diffs_v<T>(X, A);
            const T s[3] = {X.s(0), X.s(1), X.s(2)};
            b_from<T, T>(A, s, B, &r, true, &d);
        }
        D = vmul(d, p.inv8);
    }
    if (!OUT) {
#pragma unroll
        for (int l = 0; l < 3; l++) a.BF[l * p.cs + g] = B[l];
        a.RF[g] = r;
    } else {
        const long long o = (long long)(i + 1) + (long long)(nx + 2) * ((long long)(j + 1) + (long long)(ny + 2) * (k + 1));
#pragma unroll
        for (int l = 0; l < 3; l++) a.outB[3 * o + l] = B[l];
        a.outD[o] = D;
    }
}

// J of the Stokes current at the point g, up to the factor 1/det(a, b, c) (see
// stage_tile): a I1 + b I2 + c I0.
template <typename T>
__device__ __forceinline__ void j_unscaled(const KP<T>& p, const T A[3][3], const T* BF, long long g, T J[3]) {
    const int px = p.px, pxy = p.px * p.py;
    T I0, I1, I2;
#pragma unroll
    for (int l = 0; l < 3; l++) {
        const T* b = BF + l * p.cs + g;
        const T dx = vsub(ld_step(b + 1), ld_step(b - 1)), dy = vsub(ld_step(b + px), ld_step(b - px)),
                dz = vsub(ld_step(b + pxy), ld_step(b - pxy));
        if (l == 0) {
            I0 = vfms(A[l][1], dx, vmul(A[l][0], dy));
            I1 = vfms(A[l][2], dy, vmul(A[l][1], dz));
            I2 = vfms(A[l][0], dz, vmul(A[l][2], dx));
        } else {
            I0 = vfma(A[l][1], dx, vfma(vneg(A[l][0]), dy, I0));
            I1 = vfma(A[l][2], dy, vfma(vneg(A[l][1]), dz, I1));
            I2 = vfma(A[l][0], dz, vfma(vneg(A[l][2]), dx, I2));
        }
    }
#pragma unroll
    for (int l = 0; l < 3; l++) J[l] = vfma(A[l][0], I1, vfma(A[l][1], I2, vmul(A[l][2], I0)));
}

// One RK stage from the B field: J, k_n and the next stage position (stage 5:
// x_new and the error norm) at every inner point, as stage_tile.  JOUT:
// 0 the Stokes current, 1 J and B come from the exported arrays (a current with a
// kernel of its own), 2 the Classic current.  INERTIA: the velocity equation
// (rungeKutta.cu:195-212).
template <typename T, bool PRESS, bool INERTIA, int JOUT, bool LAST>
__global__ void __launch_bounds__(field_threads<T>()) k_stage_field(const __grid_constant__ StageArgs<T> a) {
    const KP<T>& p = a.p;
    DevState* st = a.st;
    after_previous();
    let_next();
    if (st->done) return;
    const int nx = p.nx, ny = p.ny, n = a.n, cur = st->cur;
    const unsigned q = blockIdx.x * (unsigned)field_threads<T>() + threadIdx.x;
    double dmax = 0;
    bool bad = false;
    if (q < (unsigned)p.N) {
        const unsigned r = q / (unsigned)nx;
        const int i = (int)(q - r * (unsigned)nx), k = (int)(r / (unsigned)ny), j = (int)(r - (unsigned)k * (unsigned)ny);
        const long long g = gidx(p.px, p.py, i, j, k), kl = (long long)i + (long long)p.kpx * r;
        const long long cs = p.cs, KC = p.kcs;
        const GlobalX<T> X = at_point(p, stage_input(a), a.B0s, g);
        const T dtT = (T)st->dt;
        T A[3][3], J[3], B[3], R = 0, D = 0, kn[3];
        const bool plain = kPlain<T>;
        if (!plain && (JOUT == 0 || PRESS)) diffs_v<T>(X, A);
        if (JOUT == 2) {
            j_classic<T>(p, ClassicTile<T>{p, stage_input(a), a.RF}, a.B0, i, j, k, J);
            R = ld_step(a.RF + g);
#pragma unroll
            for (int l = 0; l < 3; l++) B[l] = ld_step(a.BF + l * cs + g);
            D = plain ? R : vmul(rcp_stage<T>(R), p.inv8);
        } else if (JOUT == 0 && plain) {
            T xn[6][3], bn[6][3];
            const int px = p.px, pxy = p.px * p.py;
#pragma unroll
            for (int l = 0; l < 3; l++) {
                const T* b = a.BF + l * cs + g;
                B[l] = ld_step(b);
                xn[0][l] = X(l, -1, 0, 0); xn[1][l] = X(l, 1, 0, 0);
                xn[2][l] = X(l, 0, -1, 0); xn[3][l] = X(l, 0, 1, 0);
                xn[4][l] = X(l, 0, 0, -1); xn[5][l] = X(l, 0, 0, 1);
                bn[0][l] = ld_step(b - 1); bn[1][l] = ld_step(b + 1);
                bn[2][l] = ld_step(b - px); bn[3][l] = ld_step(b + px);
                bn[4][l] = ld_step(b - pxy); bn[5][l] = ld_step(b + pxy);
            }
            stokes<T>(xn, bn, J);
            D = ld_step(a.RF + g);
        } else if (JOUT == 0) {
            j_unscaled(p, A, a.BF, g, J);
            R = ld_step(a.RF + g);
#pragma unroll
            for (int l = 0; l < 3; l++) B[l] = ld_step(a.BF + l * cs + g);
            if (INERTIA) D = vmul(rcp_stage<T>(R), p.inv8);
        } else {
            const long long o = (long long)(i + 1) + (long long)(nx + 2) * ((long long)(j + 1) + (long long)(ny + 2) * (k + 1));
#pragma unroll
            for (int l = 0; l < 3; l++) { J[l] = ld_step(a.outJ + 3 * (long long)q + l); B[l] = ld_step(a.outB + 3 * o + l); }
            D = ld_step(a.outD + o);
            if (PRESS && !plain) R = rcp_stage<T>(vmul(D, p.vol8));
        }
        if (plain) cross3(J, B, kn);
        else vcross(J, B, kn);
        T gp[3] = {0, 0, 0};
        if (PRESS && plain) grad_p<T>(p, GlobalTile<T>{p, stage_input(a)}, i, j, k, D, gp);
        else if (PRESS) grad_p1<T>(p, X, i, j, A, R, gp);
        T uc[3] = {0, 0, 0}, ku[3] = {0, 0, 0};
        if (!INERTIA) {
            T f = vmul(vmul(vmul(p.ex[i], p.ey[j]), dtT), p.ez[k]);
            if (JOUT == 0 && !plain) f = vmul(f, R);
#pragma unroll
            for (int l = 0; l < 3; l++) {
                kn[l] = vmul(kn[l], f);
                if (PRESS) kn[l] = vfma(-dtT, gp[l], kn[l]);
            }
        } else {
            // k_x = dt u, k_u = dt Delta (J x B) - dt nu u Delta - dt grad p
            const T* Un = n == 0 ? a.U[cur] : a.US[(n - 1) & 1];
            T f = vmul(dtT, D);
            const T w = vmul(f, p.nu);
            if (JOUT == 0 && !plain) f = vmul(f, R);
#pragma unroll
            for (int l = 0; l < 3; l++) {
                uc[l] = Un[l * KC + kl];
                if (plain) {
                    ku[l] = kn[l] * (dtT * D);
                    ku[l] -= dtT * p.nu * uc[l] * D;
                } else {
                    ku[l] = vfma(-w, uc[l], vmul(kn[l], f));
                }
                if (PRESS) ku[l] = vfma(-dtT, gp[l], ku[l]);
                kn[l] = vmul(dtT, uc[l]);
                bad |= !finite_bits(ku[l]);
            }
        }
        T xa[3];
#pragma unroll
        for (int l = 0; l < 3; l++) {
            bad |= !finite_bits(kn[l]);
            xa[l] = X(l, 0, 0, 0);
        }
        if (!LAST) {
            // x_{n+1} = x_n + sum_{m<=n} (b[n+1][m] - b[n][m]) k_m (rungeKutta.cu:216-227)
            for (int m = 0; m < n; m++) {
                const T w = p.db[n][m];
                const T* Km = a.K[m] + kl;
#pragma unroll
                for (int l = 0; l < 3; l++) xa[l] = vfma(w, ld_step(Km + l * KC), xa[l]);
            }
            // u_{n+1} = u_n + sum_{m<=n} (b[n+1][m] - b[n][m]) k_u,m
            T ua[3] = {uc[0], uc[1], uc[2]};
            if (INERTIA)
                for (int m = 0; m < n; m++) {
                    const T wm = p.db[n][m];
#pragma unroll
                    for (int l = 0; l < 3; l++) ua[l] = vfma(wm, ld_step(a.KU[m] + l * KC + kl), ua[l]);
                }
            const T w = p.db[n][n];
#pragma unroll
            for (int l = 0; l < 3; l++) {
                xa[l] = vfma(w, kn[l], xa[l]);
                a.K[n][l * KC + kl] = kn[l];
            }
            if (INERTIA) {
#pragma unroll
                for (int l = 0; l < 3; l++) {
                    a.KU[n][l * KC + kl] = ku[l];
                    a.US[n & 1][l * KC + kl] = vfma(w, ku[l], ua[l]);
                }
            }
        } else {
            // stage 5 (see stage_tile): x_new and |x_new - x*| or |sum (c - c*) k|
            T km[6][3];
            double e[3] = {0, 0, 0};
#pragma unroll
            for (int m = 0; m < 5; m++)
#pragma unroll
                for (int l = 0; l < 3; l++) km[m][l] = ld_step(a.K[m] + l * KC + kl);
#pragma unroll
            for (int l = 0; l < 3; l++) km[5][l] = kn[l];
            if (plain && p.errMode != 0) {
                // The FP64 sums matter only where they can raise the maximum of the
                // launch so far: an FP32 estimate, off by at most 7 * 2^-24 of the sum of
                // magnitudes, leaves most points out (the FP64 pipe was 41 of the 63 us
                // of this stage at 64x64x128, which now takes 47).  NaN and infinities take
                // the FP64 sums.
                const float sofar = __double2float_rd(__longlong_as_double((long long)*(volatile unsigned long long*)&st->maxDeltaBits));
                bool need = false;
#pragma unroll
                for (int l = 0; l < 3; l++) {
                    float est = 0, size = 0;
#pragma unroll
                    for (int m = 0; m < 6; m++) {
                        const float t = (float)p.cmcT[m] * (float)km[m][l];
                        est += t;
                        size += fabsf(t);
                    }
                    need |= !(fabsf(est) + (size * 0x1p-20f + 0x1p-140f) < sofar);
                }
                if (need)
#pragma unroll
                    for (int l = 0; l < 3; l++)
#pragma unroll
                        for (int m = 0; m < 6; m++) e[l] += p.cmc[m] * (double)km[m][l];
            }
            if (plain || p.errMode == 0) {
                T xst[3];
#pragma unroll
                for (int m = 0; m < 5; m++)
#pragma unroll
                    for (int l = 0; l < 3; l++) xa[l] = vfma(p.db[5][m], km[m][l], xa[l]);
#pragma unroll
                for (int l = 0; l < 3; l++) xst[l] = xa[l];
#pragma unroll
                for (int m = 0; m < 6; m++) {
                    if (m == 1) continue;
#pragma unroll
                    for (int l = 0; l < 3; l++) {
                        if (l == 2 && !p.zUpdate) continue;
                        if (m != 4) xa[l] = vfma(p.c[m], km[m][l], xa[l]);
                        if (p.errMode == 0) xst[l] = vfma(p.cst[m], km[m][l], xst[l]);
                    }
                }
                if (p.errMode == 0)
#pragma unroll
                    for (int l = 0; l < 3; l++) e[l] = (double)vsub(xa[l], xst[l]);
            } else {
#pragma unroll
                for (int m = 0; m < 6; m++)
#pragma unroll
                    for (int l = 0; l < 3; l++) {
                        xa[l] = vfma(l == 2 ? p.cbz[m] : p.cb[m], km[m][l], xa[l]);
                        e[l] = vfma((double)p.cmcT[m], (double)km[m][l], e[l]);
                    }
            }
#pragma unroll
            for (int l = 0; l < 3; l++) {
                if (l < 2 || p.zUpdate) max_nn(dmax, e[l]);
                bad |= !finite_bits(xa[l]) || !finite_bits(e[l]);
            }
            if (INERTIA) {
                // u_6 and u_new = u_6 + sum c k_u (rungeKutta.cu:311-322)
                T kum[6][3];
#pragma unroll
                for (int m = 0; m < 5; m++)
#pragma unroll
                    for (int l = 0; l < 3; l++) kum[m][l] = ld_step(a.KU[m] + l * KC + kl);
#pragma unroll
                for (int l = 0; l < 3; l++) {
                    kum[5][l] = ku[l];
                    T u6 = uc[l];
#pragma unroll
                    for (int m = 0; m < 6; m++) u6 = vfma(p.db[5][m], kum[m][l], u6);
                    T un = u6;
#pragma unroll
                    for (int m = 0; m < 6; m++) un = vfma(p.c[m], kum[m][l], un);
                    a.U[cur][l * KC + kl] = u6;
                    a.U[cur ^ 1][l * KC + kl] = un;
                }
            }
        }
        T* Xo = LAST ? a.X[cur ^ 1] : a.XS[n & 1];
        st_xyz(Xo + g, cs, xa[0], xa[1], xa[2]);
        const int ix = image_step(p.xPeri, i, nx), iy = image_step(p.yPeri, j, ny), iz = image_step(p.zPeri, k, p.nz);
        if (ix | iy | iz) {
            store_point_images<T>(p, Xo, i, j, k, xa[0], xa[1], xa[2]);
            // the start grid's own images, refreshed by the first attempted step (see refresh_images)
            if (LAST && st->nAttempted == 0) {
                T* X0 = a.X[cur] + g;
                store_point_images<T>(p, a.X[cur], i, j, k, X0[0], X0[cs], X0[2 * cs]);
            }
        }
    }
    if (bad) atomicOr(&st->status, (unsigned)GM_ST_NAN);
    if (LAST) {
        for (int o = 16; o > 0; o >>= 1) max_nn(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
        if ((threadIdx.x & 31) == 0 && dmax > 0)
            atomicMax(&st->maxDeltaBits, (unsigned long long)__double_as_longlong(dmax));
    }
}

// ---- currents with a kernel of their own -------------------------------------------

// J = sum_m I_m (n_{m+1} x n_{m+2}) / det(n_0, n_1, n_2): the solve of the three
// circulations I over the area vectors n, with one reciprocal.
template <typename T>
__device__ __forceinline__ void solve3(const T n[3][3], const T I[3], T J[3]) {
    T c[3][3];
    vcross(n[1], n[2], c[0]);
    vcross(n[2], n[0], c[1]);
    vcross(n[0], n[1], c[2]);
    const T r = rcp_stage<T>(vfma(n[0][0], c[0][0], vfma(n[0][1], c[0][1], vmul(n[0][2], c[0][2]))));
#pragma unroll
    for (int l = 0; l < 3; l++) J[l] = vmul(vfma(I[0], c[0][l], vfma(I[1], c[1][l], vmul(I[2], c[2][l]))), r);
}
// c += a x b
template <typename T>
__device__ __forceinline__ void cross_add(const T a[3], const T b[3], T c[3]) {
    c[0] = vfma(a[1], b[2], vfma(vneg(a[2]), b[1], c[0]));
    c[1] = vfma(a[2], b[0], vfma(vneg(a[0]), b[2], c[1]));
    c[2] = vfma(a[0], b[1], vfma(vneg(a[1]), b[0], c[2]));
}

// Octilateral Stokes current (JStokes4th, src/current.cu:413-736) at every
// inner point, from the positions (padded SoA) and the ghosted B of the
// reference layout (ghost edges included).  For each plane through the point,
// axes (u, v) = (x, y), (y, z), (z, x): the circulation of B around the eight
// neighbours v0..v7 = (-1,-1) (0,-1) (1,-1) (1,0) (1,1) (0,1) (-1,1) (-1,0) and
// the polygon's area vector; then the 3x3 solve.  By exact identities of closed
// polygons, sum (B_e + B_{e+1})/2 . (x_{e+1} - x_e) = 1/2 sum B_e . (x_{e+1} -
// x_{e-1}), and the area is 1/2 [sum over the corners (v2 - v1) x (v3 - v1) +
// (v3 - v7) x (v5 - v1)], the inner diamond by its diagonals.  In FP64 the
// operations are the time: 330 a point instead of 730 (48x48x96: 300 -> 150 us).
template <typename T>
__global__ void __launch_bounds__(field_threads<T>()) k_j_oct(const __grid_constant__ StageArgs<T> a, int always) {
    const KP<T>& p = a.p;
    after_previous();
    let_next();
    if (!always && a.st->done) return;
    const int nx = p.nx, ny = p.ny;
    const unsigned q = blockIdx.x * (unsigned)field_threads<T>() + threadIdx.x;
    if (q >= (unsigned)p.N) return;
    const unsigned r = q / (unsigned)nx;
    const int i = (int)(q - r * (unsigned)nx), k = (int)(r / (unsigned)ny), j = (int)(r - (unsigned)k * (unsigned)ny);
    const GlobalX<T> X = at_point(p, stage_input(a), a.B0s, gidx(p.px, p.py, i, j, k));
    const int bs[3] = {3, 3 * (nx + 2), 3 * (nx + 2) * (ny + 2)};
    const T* B = a.outB + 3 * ((i + 1) + (long long)(nx + 2) * ((j + 1) + (long long)(ny + 2) * (k + 1)));
    const int ru[8] = {-1, 0, 1, 1, 1, 0, -1, -1}, rv[8] = {-1, -1, -1, 0, 1, 1, 1, 0};
    T n[3][3], I[3];
#pragma unroll
    for (int pl = 0; pl < 3; pl++) {
        const int u = pl, v = (pl + 1) % 3;
        T x[8][3];
#pragma unroll
        for (int e = 0; e < 8; e++) {
            int o[3] = {0, 0, 0};
            o[u] = ru[e];
            o[v] = rv[e];
#pragma unroll
            for (int l = 0; l < 3; l++) x[e][l] = X(l, o[0], o[1], o[2]);
        }
        T s = 0, area[3] = {0, 0, 0};
#pragma unroll
        for (int e = 0; e < 8; e++) {
            T chord[3];
#pragma unroll
            for (int l = 0; l < 3; l++) {
                chord[l] = vsub(x[(e + 1) & 7][l], x[(e + 7) & 7][l]);
                s = vfma(ld_step(B + ru[e] * bs[u] + rv[e] * bs[v] + l), chord[l], s);
            }
            if (!(e & 1)) {      // a corner
                T edge[3];
#pragma unroll
                for (int l = 0; l < 3; l++) edge[l] = vsub(x[e][l], x[(e + 7) & 7][l]);
                cross_add(edge, chord, area);
            }
        }
        T d1[3], d2[3];
#pragma unroll
        for (int l = 0; l < 3; l++) { d1[l] = vsub(x[3][l], x[7][l]); d2[l] = vsub(x[5][l], x[1][l]); }
        cross_add(d1, d2, area);
        I[pl] = s;               // twice the circulation, and twice the area
#pragma unroll
        for (int l = 0; l < 3; l++) n[pl][l] = area[l];
    }
    T J[3];
    solve3(n, I, J);
#pragma unroll
    for (int l = 0; l < 3; l++) a.outJ[3 * (long long)q + l] = J[l];
}

// Quintilateral Stokes current (JStokesQuint, src/current.cu:737-1199) at
// every inner point, from the positions and the exported ghosted B, as
// k_j_oct.  Per plane, axes (u, v, w) = (x, y, z), (y, z, x), (z, x, y) and
// P(a, b) the neighbour at in-plane offsets (a - 1, b - 1): the diamond through
// the face neighbours, with a corner triangle's two outer edges in place of one
// diamond edge where the orientation tests pick one.  The tests are the
// reference's as written: each later test reads the edge vectors the previous
// one stored, the third compares with 4 instead of 0, the first triangle's
// edges take the B averages of the other edge, and in the (y, z, x) and
// (z, x, y) planes the fourth triangle's second edge runs from P(1, 2), not
// P(0, 2), to P(0, 1) (src/current.cu:995-996, 1104-1105).
// With p.jTri, the triangular Stokes current (JStokesTri, src/current.cu:
// 1202-1681): the same tests, but a plane where they pick a triangle takes that
// triangle alone (its two outer edges and the reversed diamond edge) as the
// contour and half the outer edges' cross product as the area vector.  The
// reference adds that to an area vector it never set (src/current.cu:1420-
// 1424), and its compiled kernel returns NaN in J wherever a plane takes a
// triangle; the unset start is NaN here too, so the stage's NaN check stops
// the step there.
template <typename T>
__device__ __forceinline__ T quiet_nan() {
    if constexpr (sizeof(T) == 8) return __longlong_as_double(0x7ff8000000000000ll);
    else return __int_as_float(0x7fc00000);
}

template <typename T>
__device__ __noinline__ void j_quint_point(const KP<T>& p, const T* X, const T* Bg, T* J, long long q, int i, int j, int k) {
    const int ax[3][3] = {{0, 1, 2}, {1, 2, 0}, {2, 0, 1}};
    const long long nx2 = p.nx + 2, ny2 = p.ny + 2;
    {
        T NA[3][3], II[3];
#pragma unroll
        for (int pl = 0; pl < 3; pl++) {
            T x[3][3][3], b[3][3][3], xwp[3], xwm[3];
#pragma unroll
            for (int aa = 0; aa < 3; aa++)
#pragma unroll
                for (int bb = 0; bb < 3; bb++) {
                    int o[3] = {0, 0, 0};
                    o[ax[pl][0]] = aa - 1; o[ax[pl][1]] = bb - 1;
                    const long long g = gidx(p.px, p.py, i + o[0], j + o[1], k + o[2]);
                    const long long gb = (i + 1 + o[0]) + nx2 * ((j + 1 + o[1]) + ny2 * (long long)(k + 1 + o[2]));
#pragma unroll
                    for (int l = 0; l < 3; l++) { x[aa][bb][l] = X[l * p.cs + g]; b[aa][bb][l] = Bg[3 * gb + l]; }
                }
            {
                int o[3] = {0, 0, 0};
                o[ax[pl][2]] = 1;
                const long long gp = gidx(p.px, p.py, i + o[0], j + o[1], k + o[2]);
                const long long gm = gidx(p.px, p.py, i - o[0], j - o[1], k - o[2]);
#pragma unroll
                for (int l = 0; l < 3; l++) { xwp[l] = X[l * p.cs + gp]; xwm[l] = X[l * p.cs + gm]; }
            }
            T dx1[3], dx2[3], dx3[3], dx4[3], dx5[3], dx6[3], c[3];
            int tri = 0;
#pragma unroll
            for (int l = 0; l < 3; l++) {
                dx1[l] = x[1][0][l] - x[1][1][l];
                dx2[l] = x[2][1][l] - x[1][1][l];
                dx3[l] = x[1][2][l] - x[1][1][l];
                dx4[l] = x[0][1][l] - x[1][1][l];
                dx5[l] = xwp[l] - x[1][1][l];
                dx6[l] = xwm[l] - x[1][1][l];
            }
            auto dot = [](const T* u, const T* v) { return u[0] * v[0] + u[1] * v[1] + u[2] * v[2]; };
            cross3(dx1, dx2, c);
            if (dot(c, dx5) < 0 || dot(c, dx6) > 0) {
#pragma unroll
                for (int l = 0; l < 3; l++) { dx5[l] = x[2][0][l] - x[1][0][l]; dx6[l] = x[2][1][l] - x[2][0][l]; }
                tri = 2;
            }
            if (tri != 0) {
                cross3(dx2, dx3, c);
                if (dot(c, dx5) < 0 || dot(c, dx6) > 0) {
#pragma unroll
                    for (int l = 0; l < 3; l++) { dx5[l] = x[2][2][l] - x[2][1][l]; dx6[l] = x[1][2][l] - x[2][2][l]; }
                    tri = 3;
                }
            }
            if (tri != 0) {
                cross3(dx3, dx4, c);
                if (dot(c, dx5) < 0 || dot(c, dx6) > 4) {
#pragma unroll
                    for (int l = 0; l < 3; l++) { dx5[l] = x[0][2][l] - x[1][2][l]; dx6[l] = x[0][1][l] - (pl == 0 ? x[0][2][l] : x[1][2][l]); }
                    tri = 4;
                }
            }
            cross3(dx4, dx1, c);
            if (tri != 0) {
                if (dot(c, dx5) < 0 || dot(c, dx6) > 0) {
#pragma unroll
                    for (int l = 0; l < 3; l++) { dx5[l] = x[1][0][l] - x[0][0][l]; dx6[l] = x[0][0][l] - x[0][1][l]; }
                    tri = 1;
                }
            }
            T I = 0;
#pragma unroll
            for (int l = 0; l < 3; l++) {
                dx1[l] = x[1][0][l] - x[0][1][l];
                dx2[l] = x[2][1][l] - x[1][0][l];
                dx3[l] = x[1][2][l] - x[2][1][l];
                dx4[l] = x[0][1][l] - x[1][2][l];
                if (p.jTri && tri != 0) {
                    // the triangle's closing edge: the diamond edge reversed
                    if (tri == 1) I -= (b[1][0][l] + b[0][1][l]) / 2 * dx1[l];
                    if (tri == 2) I -= (b[2][1][l] + b[1][0][l]) / 2 * dx2[l];
                    if (tri == 3) I -= (b[1][2][l] + b[2][1][l]) / 2 * dx3[l];
                    if (tri == 4) I -= (b[0][1][l] + b[1][2][l]) / 2 * dx4[l];
                } else {
                    if (tri != 1) I += (b[1][0][l] + b[0][1][l]) / 2 * dx1[l];
                    if (tri != 2) I += (b[2][1][l] + b[1][0][l]) / 2 * dx2[l];
                    if (tri != 3) I += (b[1][2][l] + b[2][1][l]) / 2 * dx3[l];
                    if (tri != 4) I += (b[0][1][l] + b[1][2][l]) / 2 * dx4[l];
                }
                if (tri == 1) I += (b[0][1][l] + b[0][0][l]) / 2 * dx5[l] + (b[1][0][l] + b[0][0][l]) / 2 * dx6[l];
                if (tri == 2) I += (b[1][0][l] + b[2][0][l]) / 2 * dx5[l] + (b[2][1][l] + b[2][0][l]) / 2 * dx6[l];
                if (tri == 3) I += (b[2][1][l] + b[2][2][l]) / 2 * dx5[l] + (b[1][2][l] + b[2][2][l]) / 2 * dx6[l];
                if (tri == 4) I += (b[1][2][l] + b[0][2][l]) / 2 * dx5[l] + (b[0][1][l] + b[0][2][l]) / 2 * dx6[l];
            }
            T c12[3], c23[3], c34[3], c41[3], c56[3] = {0, 0, 0};
            cross3(dx1, dx2, c12);
            cross3(dx2, dx3, c23);
            cross3(dx3, dx4, c34);
            cross3(dx4, dx1, c41);
            if (tri > 0) cross3(dx5, dx6, c56);
            II[pl] = I;
#pragma unroll
            for (int l = 0; l < 3; l++) {
                if (p.jTri && tri > 0) {
                    NA[pl][l] = quiet_nan<T>() + c56[l] / 2;
                } else {
                    NA[pl][l] = (c12[l] + c23[l] + c34[l] + c41[l]) / 4;
                    if (tri > 0) NA[pl][l] += c56[l] / 2;
                }
            }
        }
        const T det = NA[0][0] * NA[1][1] * NA[2][2] + NA[0][1] * NA[1][2] * NA[2][0] + NA[0][2] * NA[1][0] * NA[2][1] -
                      NA[0][0] * NA[1][2] * NA[2][1] - NA[0][1] * NA[1][0] * NA[2][2] - NA[0][2] * NA[1][1] * NA[2][0];
        const T det1 = (T)1 / det;
        T N1[3][3];
        N1[0][0] = (NA[1][1] * NA[2][2] - NA[1][2] * NA[2][1]) * det1;
        N1[0][1] = (NA[0][2] * NA[2][1] - NA[0][1] * NA[2][2]) * det1;
        N1[0][2] = (NA[0][1] * NA[1][2] - NA[0][2] * NA[1][1]) * det1;
        N1[1][0] = (NA[1][2] * NA[2][0] - NA[1][0] * NA[2][2]) * det1;
        N1[1][1] = (NA[0][0] * NA[2][2] - NA[0][2] * NA[2][0]) * det1;
        N1[1][2] = (NA[0][2] * NA[1][0] - NA[0][0] * NA[1][2]) * det1;
        N1[2][0] = (NA[1][0] * NA[2][1] - NA[1][1] * NA[2][0]) * det1;
        N1[2][1] = (NA[0][1] * NA[2][0] - NA[0][0] * NA[2][1]) * det1;
        N1[2][2] = (NA[0][0] * NA[1][1] - NA[0][1] * NA[1][0]) * det1;
#pragma unroll
        for (int l = 0; l < 3; l++) {
            T Jl = 0;
#pragma unroll
            for (int m = 0; m < 3; m++) Jl += N1[l][m] * II[m];
            J[3 * q + l] = Jl;
        }
    }
}

// The tests' first step alone decides whether a plane takes a triangle; where no
// plane does, the three contours are the diamonds and J is the Stokes current in
// its closed form (117 FP64 operations a point against about 700).
template <typename T>
__global__ void __launch_bounds__(field_threads<T>()) k_j_quint(const __grid_constant__ StageArgs<T> a, int always) {
    const KP<T>& p = a.p;
    after_previous();
    let_next();
    if (!always && a.st->done) return;
    const int nx = p.nx, ny = p.ny;
    const unsigned q = blockIdx.x * (unsigned)field_threads<T>() + threadIdx.x;
    if (q >= (unsigned)p.N) return;
    const unsigned r = q / (unsigned)nx;
    const int i = (int)(q - r * (unsigned)nx), k = (int)(r / (unsigned)ny), j = (int)(r - (unsigned)k * (unsigned)ny);
    const T* Xin = stage_input(a);
    const GlobalX<T> X = at_point(p, Xin, a.B0s, gidx(p.px, p.py, i, j, k));
    T m[3][3], pl[3][3], A[3][3];        // offsets to the -/+ neighbours along each axis
#pragma unroll
    for (int l = 0; l < 3; l++) {
        const T xc = X(l, 0, 0, 0);
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const T lo = X(l, -(d == 0), -(d == 1), -(d == 2)), hi = X(l, d == 0, d == 1, d == 2);
            m[d][l] = vsub(lo, xc);
            pl[d][l] = vsub(hi, xc);
            A[l][d] = vsub(hi, lo);
        }
    }
    bool tri = false;
#pragma unroll
    for (int u = 0; u < 3; u++) {
        const int v = (u + 1) % 3, w = (u + 2) % 3;
        T c[3];
        vcross(m[v], pl[u], c);
        tri |= vfma(c[0], pl[w][0], vfma(c[1], pl[w][1], vmul(c[2], pl[w][2]))) < 0 ||
               vfma(c[0], m[w][0], vfma(c[1], m[w][1], vmul(c[2], m[w][2]))) > 0;
    }
    if (tri) {
        j_quint_point<T>(p, Xin, a.outB, a.outJ, (long long)q, i, j, k);
        return;
    }
    const long long nx2 = nx + 2, o[3] = {3, 3 * nx2, 3 * nx2 * (ny + 2)};
    const T* B = a.outB + 3 * ((i + 1) + nx2 * ((j + 1) + (long long)(ny + 2) * (k + 1)));
    T I0, I1, I2;
#pragma unroll
    for (int l = 0; l < 3; l++) {
        const T dx = vsub(ld_step(B + o[0] + l), ld_step(B - o[0] + l)), dy = vsub(ld_step(B + o[1] + l), ld_step(B - o[1] + l)),
                dz = vsub(ld_step(B + o[2] + l), ld_step(B - o[2] + l));
        if (l == 0) {
            I0 = vfms(A[l][1], dx, vmul(A[l][0], dy));
            I1 = vfms(A[l][2], dy, vmul(A[l][1], dz));
            I2 = vfms(A[l][0], dz, vmul(A[l][2], dx));
        } else {
            I0 = vfma(A[l][1], dx, vfma(vneg(A[l][0]), dy, I0));
            I1 = vfma(A[l][2], dy, vfma(vneg(A[l][1]), dz, I1));
            I2 = vfma(A[l][0], dz, vfma(vneg(A[l][2]), dx, I2));
        }
    }
    T n[3];
    const T b[3] = {A[0][1], A[1][1], A[2][1]}, c[3] = {A[0][2], A[1][2], A[2][2]};
    vcross(b, c, n);
    const T det = vfma(A[0][0], n[0], vfma(A[1][0], n[1], vmul(A[2][0], n[2]))), rd = rcp_stage<T>(det);
#pragma unroll
    for (int l = 0; l < 3; l++)
        a.outJ[3 * (long long)q + l] = vmul(vfma(A[l][0], I1, vfma(A[l][1], I2, vmul(A[l][2], I0))), rd);
}

// ---- refresh: J and the reductions ---------------------------------------------

// 1 / sqrt(x) and sqrt(x) from an approximation y of the former: with t = x y and the
// residual e = 1 - t y of its square, (1 - e)^(-1/2) = 1 + e/2 + 3 e^2/8 + ... (binomial series),
// so x^(-1/2) = y (1 + w) and x^(1/2) = t (1 + w) with w = e (1/2 + 3 e/8).  The hardware's
// approximation has about 20 bits; what is left out is of the order e^3 < 2^-57.
struct InvSqrt {
    double y, t, w;
    __device__ __forceinline__ explicit InvSqrt(double x) {
        asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
        t = x * y;
        const double e = fma(-t, y, 1.0);
        w = e * fma(0.375, e, 0.5);
    }
    __device__ __forceinline__ double root() const { return fma(t, w, t); }
    __device__ __forceinline__ double inverse() const { return fma(y, w, y); }
};

// x as a double, by integer operations; `plain` is cleared where x is subnormal or not finite.
__device__ __forceinline__ double widen(float x, bool& plain) {
    const unsigned b = __float_as_uint(x), t = b << 1;
    plain &= t == 0 || t - 0x01000000u < 0xfe000000u;
    const unsigned hi = (b & 0x80000000u) | (t ? ((b & 0x7fffffffu) >> 3) + 0x38000000u : 0u);
    return __hiloint2double((int)hi, (int)(b << 29));
}
// +0, or x > 0 and neither subnormal nor infinite nor NaN
__device__ __forceinline__ bool is_zero(double x) { return (__double2hiint(x) | __double2loint(x)) == 0; }
__device__ __forceinline__ bool in_range(double x) { return (unsigned)__double2hiint(x) - 0x00100000u < 0x7fe00000u || is_zero(x); }

// The sums and maxima of one thread, in doubles.
struct DiagSums {
    double s[5] = {0, 0, 0, 0, 0};       // |J x B|, |J||B|, their ratio, B^2 Delta, |B - e_z|^2
    double m[2] = {0, 0};                // |B|, |J|
    double m2[2] = {0, 0};               // |B|^2, |J|^2 (the points of addf)
    __device__ __forceinline__ void add(const double B[3], const double J[3], double b2D) {
        const double bn = sqrt(B[0] * B[0] + B[1] * B[1] + B[2] * B[2]), jn = sqrt(J[0] * J[0] + J[1] * J[1] + J[2] * J[2]);
        const double cx = J[1] * B[2] - J[2] * B[1], cy = J[2] * B[0] - J[0] * B[2], cz = J[0] * B[1] - J[1] * B[0];
        const double cn = sqrt(cx * cx + cy * cy + cz * cz);
        s[0] += cn;
        s[1] += jn * bn;
        if (jn * bn > 0) s[2] += cn / (jn * bn);
        s[3] += b2D;
        s[4] += B[0] * B[0] + B[1] * B[1] + (B[2] - 1.0) * (B[2] - 1.0);
        m[0] = fmax(m[0], bn);
        m[1] = fmax(m[1], jn);
    }
    // B and J of an FP32 run: the squares of the components' products are far inside the
    // range of doubles, so |J||B| is one square root, the maxima are those of the squares,
    // and neither root nor quotient is an IEEE one: 34 FP64 operations a point against 85
    // (an SM issues one FP64 warp instruction in 15 clocks; conversions and comparisons of
    // doubles count too, so both are made of integer operations).  A 128x128x256 refresh
    // takes 425 us with it, about 660 with add() alone.  (Pairs of floats, 312 us, hold 46
    // bits of each term, and fewer where a square's lower half is subnormal.)  Where
    // something is subnormal or not finite, add()'s form.
    __device__ __forceinline__ void addf(const float Bf[3], const float Jf[3], float b2, float Dw) {
        bool plain = true;
        const double B0 = widen(Bf[0], plain), B1 = widen(Bf[1], plain), B2 = widen(Bf[2], plain);
        const double J0 = widen(Jf[0], plain), J1 = widen(Jf[1], plain), J2 = widen(Jf[2], plain);
        const double b2w = widen(b2, plain), Dww = widen(Dw, plain);
        const double bp = fma(B1, B1, B0 * B0), bb = fma(B2, B2, bp), z = B2 - 1.0;
        const double jj = fma(J2, J2, fma(J1, J1, J0 * J0));
        const double cx = fma(J1, B2, -(J2 * B1)), cy = fma(J2, B0, -(J0 * B2)), cz = fma(J0, B1, -(J1 * B0));
        const double cc = fma(cz, cz, fma(cy, cy, cx * cx)), xx = jj * bb;
        if (!(plain && in_range(cc) && in_range(xx))) {
            const double Bd[3] = {Bf[0], Bf[1], Bf[2]}, Jd[3] = {Jf[0], Jf[1], Jf[2]};
            add(Bd, Jd, (double)b2 * (double)Dw);
            return;
        }
        const InvSqrt c(cc), x(xx);
        const double cn = is_zero(cc) ? 0.0 : c.root();
        s[0] += cn;
        s[1] += is_zero(xx) ? 0.0 : x.root();
        s[2] = fma(cn, is_zero(xx) ? 0.0 : x.inverse(), s[2]);
        s[3] = fma(b2w, Dww, s[3]);
        s[4] += fma(z, z, bp);
        max_nn(m2[0], bb);
        max_nn(m2[1], jj);
    }
    __device__ __forceinline__ void finish() {
        for (int q = 0; q < 2; q++) m[q] = fmax(m[q], sqrt(m2[q]));
    }
};

constexpr int kDiagThreads = 128;

// J (unless a current's own kernel has written it) and the reductions at the
// current grid, from the exported B and Delta with their face ghosts as
// k_b_field leaves them (diagnostics.cu:12-134).  One partial per CTA, in a fixed order.
// Both precisions fill the FP64 pipe (FP32: 86 % active, 40 instructions a point) at 16
// warps an SM and 128 registers, in one wave of CTAs: a CTA's own reduction is another 70 of
// its threads' FP64 instructions (128x128x256 in FP32, the refresh: 425 us; two waves 447,
// 32 warps and 64 registers with some spills 462).
template <typename T, bool JOUT>
__global__ void __launch_bounds__(kDiagThreads, 4) k_diag_field(const __grid_constant__ StageArgs<T> a) {
    const KP<T>& p = a.p;
    const int nx = p.nx, ny = p.ny, nz = p.nz, cur = a.st->cur;
    const long long nx2 = nx + 2, nxy2 = (long long)(nx + 2) * (ny + 2);
    DiagSums sums;
    double e2 = 0, u2 = 0, um = 0;
    T q1m = 0, wm = (T)(sizeof(T) == 4 ? FLT_MAX : DBL_MAX), dm = wm;
    bool convex = true;
    for (unsigned q = blockIdx.x * kDiagThreads + threadIdx.x; q < (unsigned)p.N; q += gridDim.x * kDiagThreads) {
        const unsigned r = q / (unsigned)nx;
        const int i = (int)(q - r * (unsigned)nx), k = (int)(r / (unsigned)ny), j = (int)(r - (unsigned)k * (unsigned)ny);
        const GlobalX<T> X = at_point(p, a.X[cur], a.B0s, gidx(p.px, p.py, i, j, k));
        const long long o = (long long)(i + 1) + nx2 * (j + 1) + nxy2 * (k + 1);
        const T* Bo = a.outB + 3 * o;
        T xc[3], xn[6][3], Bc[3], Jv[3];
#pragma unroll
        for (int l = 0; l < 3; l++) {
            xc[l] = X(l, 0, 0, 0);
            xn[0][l] = X(l, -1, 0, 0); xn[1][l] = X(l, 1, 0, 0);
            xn[2][l] = X(l, 0, -1, 0); xn[3][l] = X(l, 0, 1, 0);
            xn[4][l] = X(l, 0, 0, -1); xn[5][l] = X(l, 0, 0, 1);
            Bc[l] = Bo[l];
        }
        const T D = a.outD[o];
        if (JOUT) {
#pragma unroll
            for (int l = 0; l < 3; l++) Jv[l] = a.outJ[3 * (long long)q + l];
        } else {
            T bn[6][3];
#pragma unroll
            for (int l = 0; l < 3; l++) {
                bn[0][l] = Bo[l - 3]; bn[1][l] = Bo[l + 3];
                bn[2][l] = Bo[l - 3 * nx2]; bn[3][l] = Bo[l + 3 * nx2];
                bn[4][l] = Bo[l - 3 * nxy2]; bn[5][l] = Bo[l + 3 * nxy2];
            }
            stokes<T>(xn, bn, Jv);
#pragma unroll
            for (int l = 0; l < 3; l++) a.outJ[3 * (long long)q + l] = Jv[l];
        }
        T jxb[3];
        cross3(Jv, Bc, jxb);
        const T b2 = Bc[0] * Bc[0] + Bc[1] * Bc[1] + Bc[2] * Bc[2];
        q1m = fmax(q1m, sqrt(jxb[0] * jxb[0] + jxb[1] * jxb[1] + jxb[2] * jxb[2]) / b2);
        const int bound = (i == 0) + (j == 0) + (k == 0) + (i == nx - 1) + (j == ny - 1) + (k == nz - 1);
        const T w = (T)1 / (T)(1 << bound);
        if constexpr (sizeof(T) == 4) sums.addf(Bc, Jv, b2, D * w);
        else sums.add(Bc, Jv, b2 * D * w);
        if (p.wantXbAn) {
            // distance to the analytically relaxed grid (maths.cu:332-377)
            const double Xi = (double)(p.dx * (T)i + p.Ox), Yi = (double)(p.dy * (T)j + p.Oy), Zi = (double)(p.dz * (T)k + p.Oz);
            const double ph = exp(-(Xi * Xi + Yi * Yi) / (p.ar * p.ar) - Zi * Zi / (p.az * p.az)) * p.phi1;
            const double sp = sin(ph), cp = cos(ph);
            const double a0 = (double)xc[0] - cp * Xi - sp * Yi, a1 = (double)xc[1] + sp * Xi - cp * Yi, a2 = (double)xc[2] - Zi;
            e2 += a0 * a0 + a1 * a1 + a2 * a2;
        }
        if (p.inertia) {
            // kinetic energy sum |u|^2 Delta with the boundary weights
            // (maths.cu:684-710) and max |u|
            const T* Uc = a.U[cur] + (long long)i + (long long)p.kpx * r;
            const double u0 = Uc[0], u1 = Uc[p.kcs], uz = Uc[2 * p.kcs];
            const T uu2 = (T)u0 * (T)u0 + (T)u1 * (T)u1 + (T)uz * (T)uz;
            u2 += (double)(uu2 * D) * (double)w;
            um = fmax(um, sqrt(u0 * u0 + u1 * u1 + uz * uz));
        }
        // Delta, also on the ghost planes of line-tied faces next to this point
        dm = fmin(dm, D);
        if (bound) {
            if (!p.xPeri && i == 0) dm = fmin(dm, a.outD[o - 1]);
            if (!p.xPeri && i == nx - 1) dm = fmin(dm, a.outD[o + 1]);
            if (!p.yPeri && j == 0) dm = fmin(dm, a.outD[o - nx2]);
            if (!p.yPeri && j == ny - 1) dm = fmin(dm, a.outD[o + nx2]);
            if (!p.zPeri && k == 0) dm = fmin(dm, a.outD[o - nxy2]);
            if (!p.zPeri && k == nz - 1) dm = fmin(dm, a.outD[o + nxy2]);
        }
        // wedge products and convexity (maths.cu:497-643)
        T wmin = 0;
#pragma unroll
        for (int u = 0; u < 2; u++)
#pragma unroll
            for (int v = 0; v < 2; v++) {
                T d1[3], d2[3], cc[3];
#pragma unroll
                for (int l = 0; l < 3; l++) { d1[l] = xn[u][l] - xc[l]; d2[l] = xn[2 + v][l] - xc[l]; }
                cross3(d1, d2, cc);
#pragma unroll
                for (int t = 0; t < 2; t++) {
                    T d3[3];
#pragma unroll
                    for (int l = 0; l < 3; l++) d3[l] = xn[4 + t][l] - xc[l];
                    T wc = cc[0] * d3[0] + cc[1] * d3[1] + cc[2] * d3[2];
                    const int sg = u + v + t;
                    if (wc < 0 && (sg & 1)) convex = false;
                    if (wc > 0 && !(sg & 1)) convex = false;
                    if (sg == 0) wmin = -wc;
                    if (!(sg & 1)) wc = -wc;
                    if (wc < wmin) wmin = wc;
                }
            }
        wm = fmin(wm, wmin);
    }
    sums.finish();
    double v[R_COUNT] = {sums.s[0], sums.s[1], sums.s[2], sums.s[3], sums.s[4], e2, u2,
                         (double)q1m, sums.m[0], sums.m[1], um, (double)dm, (double)wm, convex ? 1.0 : -1.0};
    // fixed-order reduction: within the warps, then over them
    __shared__ double red[kDiagThreads / 32][R_COUNT];
#pragma unroll
    for (int r = 0; r < R_COUNT; r++)
        for (int o = 16; o > 0; o >>= 1) {
            const double x = __shfl_xor_sync(0xffffffffu, v[r], o);
            v[r] = r <= R_LAST_SUM ? v[r] + x : r <= R_LAST_MAX ? fmax(v[r], x) : fmin(v[r], x);
        }
    if ((threadIdx.x & 31) == 0)
        for (int r = 0; r < R_COUNT; r++) red[threadIdx.x >> 5][r] = v[r];
    __syncthreads();
    if (threadIdx.x < R_COUNT) {
        const int r = threadIdx.x;
        double acc = red[0][r];
        for (int q = 1; q < kDiagThreads / 32; q++)
            acc = r <= R_LAST_SUM ? acc + red[q][r] : r <= R_LAST_MAX ? fmax(acc, red[q][r]) : fmin(acc, red[q][r]);
        a.part[(long long)blockIdx.x * R_COUNT + r] = acc;
    }
}

// CTAs (and partials) of k_diag_field: enough to fill the SMs, no more.
template <typename T>
int diag_blocks(long long N) {
    const long long b = (N + kDiagThreads - 1) / kDiagThreads;
    return (int)(b < kMaxDiagBlocks ? b : kMaxDiagBlocks);
}

template <typename T>
cudaError_t launch_diag_field(const StageArgs<T>& a, int jout, cudaStream_t s) {
    const int nb = diag_blocks<T>(a.p.N);
    if (jout) k_diag_field<T, true><<<nb, kDiagThreads, 0, s>>>(a);
    else k_diag_field<T, false><<<nb, kDiagThreads, 0, s>>>(a);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_b_field(const StageArgs<T>& a, int out, int always, cudaStream_t s) {
    const long long n = a.p.N + 2ll * ((long long)a.p.ny * a.p.nz + (long long)a.p.nx * a.p.nz + (long long)a.p.nx * a.p.ny);
    const int t = field_threads<T>();
    const unsigned nb = (unsigned)((n + t - 1) / t);
    auto kern = out == B_EXPORT ? k_b_field<T, true, true>
                : out == B_OUT  ? k_b_field<T, true, kPlain<T>>
                                : k_b_field<T, false, kPlain<T>>;
    return launch_next(kern, nb, t, 0, s, a, always);
}

template <typename T>
cudaError_t launch_j_own(const StageArgs<T>& a, int always, cudaStream_t s) {
    const int t = field_threads<T>();
    const unsigned nb = (unsigned)((a.p.N + t - 1) / t);
    return launch_next(a.p.jOct ? k_j_oct<T> : k_j_quint<T>, nb, t, 0, s, a, always);
}

template <typename T>
cudaError_t launch_stage_field(const StageArgs<T>& a, int pressure, int jout, cudaStream_t s) {
    const int t = field_threads<T>();
    const unsigned nb = (unsigned)((a.p.N + t - 1) / t);
    auto by = [](int v, auto f) { v ? f(std::true_type()) : f(std::false_type()); };
    cudaError_t rc = cudaErrorInvalidValue;
    by(pressure, [&](auto P) {
        by(a.p.inertia, [&](auto I) {
            by(a.n == 5, [&](auto L) {
                if (jout == 1) rc = launch_next(k_stage_field<T, P.value, I.value, 1, L.value>, nb, t, 0, s, a);
                else if (jout == 2) rc = launch_next(k_stage_field<T, P.value, I.value, 2, L.value>, nb, t, 0, s, a);
                // FP32 frictional Stokes stages run in the tile kernel
                else if constexpr (sizeof(T) == 8 || I.value)
                    rc = launch_next(k_stage_field<T, P.value, I.value, 0, L.value>, nb, t, 0, s, a);
            });
        });
    });
    return rc;
}

#define GMK_INSTANTIATE_FIELDS(T)                                                       \
    template cudaError_t launch_b_field<T>(const StageArgs<T>&, int, int, cudaStream_t);    \
    template cudaError_t launch_stage_field<T>(const StageArgs<T>&, int, int, cudaStream_t); \
    template cudaError_t launch_j_own<T>(const StageArgs<T>&, int, cudaStream_t);            \
    template cudaError_t launch_diag_field<T>(const StageArgs<T>&, int, cudaStream_t);       \
    template int diag_blocks<T>(long long);

}  // namespace gmk
