// gm_point.cuh -- the arithmetic of one point, or of a pair of points, of the
// relaxation: B from the grid's differences, B on line-tied faces, the pressure
// gradient, periodic images.  The tile kernel (gm_stage_tma.cuh) and the field
// kernels (gm_fields.cuh) share it.
#pragma once

#include "gm_kernels_impl.cuh"
#include "gm_vec2.cuh"

namespace gmk {

// Reciprocal for the stage kernel, by Newton's iteration r <- r + r (1 - x r)
// from the hardware's approximation: one step in FP32 (within ~1 ulp; FP32
// parity is held to 1e-5), two in FP64 (the approximation has about 20 bits;
// the last step's residual is exact to an FMA, so the result is the rounded
// reciprocal but for rare ties: with __drcp_rn in its place periodic, line-tied,
// pressure and inertial FP64 runs came out the same).
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ double rcp_approx(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return r;
}
__device__ __forceinline__ F2 rcp_approx(F2 x) { return mk2(rcp_approx(lo(x)), rcp_approx(hi(x))); }
__device__ __forceinline__ D2 rcp_approx(D2 x) { return mk2(rcp_approx(lo(x)), rcp_approx(hi(x))); }
template <typename T, typename V>
__device__ __forceinline__ V rcp_stage(V x) {
    V r = rcp_approx(x);
    const V one = splat<V>((T)1), nx = vneg(x);
#pragma unroll
    for (int it = 0; it < (sizeof(T) == 4 ? 1 : 2); it++) r = vfma(vfma(nx, r, one), r, r);
    return r;
}

// FP32: the determinant d of the columns of A, recomputed in double from the
// same entries when the cell is strongly sheared: |d| small against the bound
// |a|_1 |b|_1 |c|_1 of the six Sarrus products.
__device__ __forceinline__ float det_sheared(float d, float a0, float a1, float a2, float b0, float b1, float b2,
                                             float c0, float c1, float c2) {
    const float m = (fabsf(a0) + fabsf(a1) + fabsf(a2)) * (fabsf(b0) + fabsf(b1) + fabsf(b2)) *
                    (fabsf(c0) + fabsf(c1) + fabsf(c2));
    if (!(fabsf(d) < 0.03125f * m)) return d;
    const double jd[3][3] = {{a0, b0, c0}, {a1, b1, c1}, {a2, b2, c2}};
    return (float)det3<double>(jd);
}
// The cheap test in front of it: |v|_1 <= sqrt(3) |v|_2, so a cell with
// d^2 > (0.03125 sqrt(27))^2 |a|^2 |b|^2 |c|^2 cannot be one; everything else
// (an underflow or a NaN of the squares too) takes the test above.
constexpr float kShear2 = 0.0266f;
template <typename V>
__device__ __forceinline__ V norm2(const V A[3][3], int c) {
    return vfma(A[2][c], A[2][c], vfma(A[1][c], A[1][c], vmul(A[0][c], A[0][c])));
}
// (out of line: the double determinant would double the plane loop's code)
static __device__ __noinline__ F2 det_sheared2(F2 d, F2 a0, F2 a1, F2 a2, F2 b0, F2 b1, F2 b2, F2 c0, F2 c1, F2 c2) {
    const float x = det_sheared(lo(d), lo(a0), lo(a1), lo(a2), lo(b0), lo(b1), lo(b2), lo(c0), lo(c1), lo(c2));
    const float y = det_sheared(hi(d), hi(a0), hi(a1), hi(a2), hi(b0), hi(b1), hi(b2), hi(c0), hi(c1), hi(c2));
    return mk2(x, y);
}
__device__ __forceinline__ float det_guard(float d, const float A[3][3], bool act) {
    const float t = vmul(vmul(norm2(A, 0), norm2(A, 1)), vmul(norm2(A, 2), kShear2));
    if (!(vmul(d, d) > t) && act)
        d = det_sheared(d, A[0][0], A[1][0], A[2][0], A[0][1], A[1][1], A[2][1], A[0][2], A[1][2], A[2][2]);
    return d;
}
__device__ __forceinline__ F2 det_guard(F2 d, const F2 A[3][3], bool act) {
    const F2 t = vmul(vmul(norm2(A, 0), norm2(A, 1)), vmul(norm2(A, 2), splat<F2>(kShear2))), q = vmul(d, d);
    if (!(lo(q) > lo(t) && hi(q) > hi(t)) && act)
        d = det_sheared2(d, A[0][0], A[1][0], A[2][0], A[0][1], A[1][1], A[2][1], A[0][2], A[1][2], A[2][2]);
    return d;
}
__device__ __forceinline__ double det_guard(double d, const double[3][3], bool) { return d; }
__device__ __forceinline__ D2 det_guard(D2 d, const D2[3][3], bool) { return d; }

// B = (s_x a + s_y b + s_z c) / det(a, b, c) with the unscaled central
// differences a = x(+x) - x(-x), b, c (the columns of A) and the pre-scaled
// field s = (4 dy dz B0x, 4 dx dz B0y, 4 dx dy B0z): since jac = [a/2dx, b/2dy,
// c/2dz], this is jac.B0 / det(jac) of B_JacB0 (rungeKutta.cu:79-99) with the
// constant factors folded.  *r = 1/det(a, b, c) (Delta = 1 / (8 dx dy dz r)).
// Without `act` the result is not used (and B may come out inexact).  *det, where
// asked for: the determinant.
template <typename T, typename V>
__device__ __forceinline__ void b_from(const V A[3][3], const V s[3], V B[3], V* r, bool act, V* det = nullptr) {
    const V b[3] = {A[0][1], A[1][1], A[2][1]}, c[3] = {A[0][2], A[1][2], A[2][2]};
    V n[3];
    vcross(b, c, n);
    V d = vfma(A[0][0], n[0], vfma(A[1][0], n[1], vmul(A[2][0], n[2])));
    if (sizeof(T) == 4) d = det_guard(d, A, act);
    if (det) *det = d;
    const V q = rcp_stage<T>(d);
    const V s0 = vmul(s[0], q), s1 = vmul(s[1], q), s2 = vmul(s[2], q);
#pragma unroll
    for (int l = 0; l < 3; l++) B[l] = vfma(A[l][0], s0, vfma(A[l][1], s1, vmul(A[l][2], s2)));
    *r = q;
}

template <typename T>
struct Vec3 { T x, y, z; };

// B on the ghost plane of a line-tied face with normal axis AX, at the point
// (i, j, k): updateBbound, src/boundaries.cu:39-446.  The ghost plane continues
// by one spacing outwards, and in-plane neighbours at the edges of the
// reference's 16-wide launch blocks are the own position shifted by the spacing
// (boundaries.cu:72-109, 212-237, 340-365); the differences come out in the
// scaling of b_from, and B.n = B0.n is s.n over its scale w (one corrected
// step, so the quotient is B0.n but for rare last bits).
// X(l, di, dj, dk): component l of the position at that offset from the point;
// X.s(l): the scaled field there.  *r, *d as from b_from.
template <int AX, typename T, class XT>
__device__ __forceinline__ Vec3<T> b_face_v(const KP<T>& p, const XT& X, int i, int j, int k, T* r, T* d) {
    const int idx[3] = {i, j, k};
    const int n3[3] = {p.nx, p.ny, p.nz};
    const T d3[3] = {p.dx, p.dy, p.dz};
    const bool side = idx[AX] >= 0;
    const int in = side ? -1 : 1;
    T A[3][3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        if (a == AX) {
#pragma unroll
            for (int l = 0; l < 3; l++) {
                T xo = X(l, 0, 0, 0);
                if (l == AX) xo = side ? vadd(xo, d3[AX]) : vsub(xo, d3[AX]);
                if (AX == 2 && l < 2 && p.shear)
                    xo = p.shearTab[10 * ((long long)side * p.nx * p.ny + (long long)j * p.nx + i) + l];
                const T xn = X(l, AX == 0 ? in : 0, AX == 1 ? in : 0, AX == 2 ? in : 0);
                A[l][a] = side ? vsub(xo, xn) : vsub(xn, xo);
            }
        } else {
            const int u = idx[a];
            const bool eL = u % 16 == 0, eR = u % 16 == 15 || u == n3[a] - 1;
            const int ol = eL ? 0 : -1, orr = eR ? 0 : 1;
#pragma unroll
            for (int l = 0; l < 3; l++) {
                T vl = X(l, a == 0 ? ol : 0, a == 1 ? ol : 0, a == 2 ? ol : 0);
                T vr = X(l, a == 0 ? orr : 0, a == 1 ? orr : 0, a == 2 ? orr : 0);
                if (l == a) {
                    if (eL) vl = vsub(vl, d3[a]);
                    if (eR) vr = vadd(vr, d3[a]);
                }
                if (AX == 2 && l < 2 && p.shear) {
                    // an initially distorted grid: the neighbours extrapolated at the
                    // block edges carry the distortion (k_shear_table)
                    const T* tb = p.shearTab + 10 * ((long long)side * p.nx * p.ny + (long long)j * p.nx + i);
                    if (eL) vl = tb[2 + 4 * a + l];
                    if (eR) vr = tb[4 + 4 * a + l];
                }
                A[l][a] = vsub(vr, vl);
            }
        }
    }
    const T s[3] = {X.s(0), X.s(1), X.s(2)};
    T B[3];
    b_from<T, T>(A, s, B, r, true, d);
    const T q = vmul(s[AX], p.w4i[AX]);
    B[AX] = vfma(vfma(-q, p.w4[AX], s[AX]), p.w4i[AX], q);
    return Vec3<T>{B[0], B[1], B[2]};
}

// The columns of A at a point.
template <typename T, class XT>
__device__ __forceinline__ void diffs_v(const XT& X, T A[3][3]) {
#pragma unroll
    for (int l = 0; l < 3; l++) {
        A[l][0] = vsub(X(l, 1, 0, 0), X(l, -1, 0, 0));
        A[l][1] = vsub(X(l, 0, 1, 0), X(l, 0, -1, 0));
        A[l][2] = vsub(X(l, 0, 0, 1), X(l, 0, 0, -1));
    }
}

// p0(X) and its derivatives along x, y times 2 dx, 2 dy at the column (i, j).
template <typename T>
__device__ __forceinline__ void p0_at(const KP<T>& p, int i, int j, T pe[3]) {
    const T X = p.dx * (T)i + p.Ox, Y = p.dy * (T)j + p.Oy;
    const T ex = p.p0Amp != (T)0 ? p.p0Amp * exp(-(X * X + Y * Y) * p.inv_p0W2) : (T)0;
    const T be2 = -2 * p.beta * ex * p.inv_p0W2;
    pe[0] = p.beta * ((T)1 + ex);
    pe[1] = be2 * X * (2 * p.dx);
    pe[2] = be2 * Y * (2 * p.dy);
}

// The pressure gradient at a point, as grad_p2 (gm_stage_tma.cuh).
template <typename T, class XT>
__device__ __forceinline__ void grad_p1(const KP<T>& p, const XT& X, int i, int j, const T A[3][3], T r, T g[3]) {
    const T a[3] = {A[0][0], A[1][0], A[2][0]}, b[3] = {A[0][1], A[1][1], A[2][1]}, c[3] = {A[0][2], A[1][2], A[2][2]};
    T Ai[3][3], S[3], pe[3];
    vcross(b, c, Ai[0]);
    vcross(c, a, Ai[1]);
    vcross(a, b, Ai[2]);
#pragma unroll
    for (int e = 0; e < 9; e++) Ai[e / 3][e % 3] = vmul(Ai[e / 3][e % 3], r);
    p0_at(p, i, j, pe);
#pragma unroll
    for (int l = 0; l < 3; l++) {
        const T q = (T)0.25, xc = X(l, 0, 0, 0);
        const T dxx = vsub(vsub(X(l, 1, 0, 0), xc), vsub(xc, X(l, -1, 0, 0)));
        const T dyy = vsub(vsub(X(l, 0, 1, 0), xc), vsub(xc, X(l, 0, -1, 0)));
        const T dzz = vsub(vsub(X(l, 0, 0, 1), xc), vsub(xc, X(l, 0, 0, -1)));
        const T dxy = vmul(vsub(vsub(X(l, 1, 1, 0), X(l, 1, -1, 0)), vsub(X(l, -1, 1, 0), X(l, -1, -1, 0))), q);
        const T dxz = vmul(vsub(vsub(X(l, 1, 0, 1), X(l, 1, 0, -1)), vsub(X(l, -1, 0, 1), X(l, -1, 0, -1))), q);
        const T dyz = vmul(vsub(vsub(X(l, 0, 1, 1), X(l, 0, 1, -1)), vsub(X(l, 0, -1, 1), X(l, 0, -1, -1))), q);
        const T i0 = Ai[0][l], i1 = Ai[1][l], i2 = Ai[2][l];
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
    const T det1 = vmul(r, p.vol8), w = vmul(pe[0], (T)-4);
#pragma unroll
    for (int l = 0; l < 3; l++) {
        T t = vmul(w, vfma(S[0], Ai[0][l], vfma(S[1], Ai[1][l], vmul(S[2], Ai[2][l]))));
        t = vfma(pe[1], Ai[0][l], vfma(pe[2], Ai[1][l], t));
        g[l] = vmul(t, det1);
    }
}

// Offsets (elements) from a stored position to its periodic images along x and
// y, 0 where there is none: ghost layers 1 and 2 hold the images of the two
// inner layers of the opposite face, shifted by -/+ (L + d) as setGridPeriFace
// writes them (boundaries.cu:546-549, 561-564, 576-579).
__device__ __forceinline__ int image_step(int peri, int i, int n) { return !peri ? 0 : i < 2 ? n : i >= n - 2 ? -n : 0; }

template <typename T, typename V>
__device__ __forceinline__ V image_shift(V v, int step, T L, T d) {
    return step > 0 ? vadd(vadd(v, splat<V>(L)), splat<V>(d)) : vsub(vsub(v, splat<V>(L)), splat<V>(d));
}

template <typename T, typename V>
__device__ __forceinline__ void st_xyz(T* q, long long cs, V a, V b, V c) {
    stv(q, a);
    stv(q + cs, b);
    stv(q + 2 * cs, c);
}

// The periodic images, beyond those along x alone, of the position v stored at
// q (ix, iy, iz: image_step).
template <typename T, typename V>
__device__ __forceinline__ void store_images_yz(const KP<T>& p, T* q, const V v[3], int ix, int iy, int iz) {
    const long long cs = p.cs, oy = (long long)iy * p.px;
    const V vx = image_shift<T>(v[0], ix, p.Lx, p.dx), vy = image_shift<T>(v[1], iy, p.Ly, p.dy);
    if (iy) st_xyz(q + oy, cs, v[0], vy, v[2]);
    if (ix && iy) st_xyz(q + ix + oy, cs, vx, vy, v[2]);
    if (iz) {
        T* qz = q + (long long)iz * p.px * p.py;
        const V vz = image_shift<T>(v[2], iz, p.Lz, p.dz);
        st_xyz(qz, cs, v[0], v[1], vz);
        if (ix) st_xyz(qz + ix, cs, vx, v[1], vz);
        if (iy) st_xyz(qz + oy, cs, v[0], vy, vz);
        if (ix && iy) st_xyz(qz + ix + oy, cs, vx, vy, vz);
    }
}
template <typename T, typename V>
__device__ __noinline__ void store_images_call(const KP<T>& p, T* q, V a, V b, V c, int ix, int iy, int iz) {
    const V v[3] = {a, b, c};
    store_images_yz<T, V>(p, q, v, ix, iy, iz);
}
// Every image of one point, in any grid: a direction of three points, whose
// middle point has two images, takes the loop over all shifts (store_pos).
template <typename T>
__device__ __noinline__ void store_point_images(const KP<T>& p, T* X, int i, int j, int k, T a, T b, T c) {
    const T v[3] = {a, b, c};
    store_pos<T>(p, X, i, j, k, v);
}
__device__ __forceinline__ bool finite_bits(float x) { return (__float_as_uint(x) & 0x7f800000u) != 0x7f800000u; }
__device__ __forceinline__ bool finite_bits(double x) { return ((unsigned)__double2hiint(x) & 0x7ff00000u) != 0x7ff00000u; }

// Running maximum of non-negative values; NaN never wins (maths.cu:144-153).
// In FP64 on the bits (non-negative doubles order as integers): a comparison
// of doubles would cost a slot of the FP64 pipe.
__device__ __forceinline__ void max_nn(float& m, float x) { m = fmaxf(m, fabsf(x)); }
__device__ __forceinline__ void max_nn(double& m, double x) {
    const long long b = __double_as_longlong(x) & 0x7fffffffffffffffll;
    if (b > __double_as_longlong(m) && b <= 0x7ff0000000000000ll) m = __longlong_as_double(b);
}

}  // namespace gmk
