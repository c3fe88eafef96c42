// Per-step leapfrog kernels with the exact semantics of the reference step
// templates (one launch = one time step over the whole padded grid):
//   cda_time_scalar_1D  pysit/solvers/constant_density_acoustic/time/scalar/
//                       constant_density_acoustic_time_scalar_1D.h:44-131
//   cda_time_scalar_2D  ..._2D.h:43-180
//   cda_time_scalar_3D  ..._3D.h:46-236
// Zero-extended stencils (fd_manual.hpp:5-70), Dirichlet outer ring, right PML
// profile read at r[n_r - ((n-1) - i)] (_2D.h:143-157), psi integrated on every
// non-ring cell in 3D.  These kernels serve the per-step API (time_step) and the
// plain per-shot path; the batched pipeline lives in wave2d_tile.cuh / wave3d_tile.cuh.
//
// One thread per cell, z (the contiguous axis) on threadIdx.x.  Taps outside
// [0, n) are zero, which is the zero extension of the reference.  In FP64 the FP64 units
// bound the step (86% busy; DRAM 7%), so what counts is FP64 instructions per cell: zeros are
// tested on the integer units, first derivatives are taken only where they enter, and the PML
// update is one quotient,
//     u' = 2 u - u_{k-1} + (2 dt^2 C^2 (F - ...) + 2 dt s (u_{k-1} - u) - 2 dt^2 s2 u) / (2 + dt s),
// in place of three; only a small correction is divided, so the last sum sets the rounding.
// Measured, one time_step + compute_dWaveOp on 193 x 193 x 153 cells, order 4, FP64: 1266 -> 801 us.
#include <algorithm>

#include "common.cuh"

namespace pgb {
namespace {

template <typename T>
struct Prof {  // one axis: left / right PML profile
    const T* l; int nl;
    const T* r; int nr;
    __device__ __forceinline__ T at(int i, int n) const {
        if (nl > 0 && i < nl) return l[i];
        if (nr > 0 && i >= n - nr) return r[nr - ((n - 1) - i)];
        return T(0);
    }
};

__device__ __forceinline__ bool nonzero(float a) { return (__float_as_uint(a) << 1) != 0; }
__device__ __forceinline__ bool nonzero(double a) {  // on the integer units
    return ((unsigned)__double2hiint(a) << 1 | (unsigned)__double2loint(a)) != 0;
}

__device__ __forceinline__ bool nonfinite(float a) { return (__float_as_uint(a) & 0x7f800000u) == 0x7f800000u; }
__device__ __forceinline__ bool nonfinite(double a) {
    return ((unsigned)__double2hiint(a) & 0x7ff00000u) == 0x7ff00000u;
}

// one axis: 1 / h and 1 / h^2
template <typename T>
struct Axis {
    T id, id2;
};

// the 2R+1 values of v along one axis around position p of n, element stride s
template <typename T, int R>
struct Taps {
    T t[2 * R + 1];
    __device__ __forceinline__ Taps(const T* __restrict__ v, long long idx, long long s, int p, int n) {
#pragma unroll
        for (int m = -R; m <= R; ++m) t[m + R] = p + m < 0 || p + m >= n ? T(0) : __ldg(v + idx + m * s);
    }
    // acc + second derivative.  The taps stay unscaled and each axis cancels by itself: with 1/h^2
    // in the taps and the centre taps of all axes taken at once (709 us instead of 801) the FP64
    // rounding error of u' in plain cells was 1.4 to 2 times as large.  Fused multiply-adds by name:
    // left to the compiler, the product of u and the centre weight was taken once, rounded, for the
    // three axes (error of u' in plain cells 1.06 to 1.15 times as large).
    __device__ __forceinline__ T add_d2(T acc, const Axis<T>& x) const {
        T b = 0;
#pragma unroll
        for (int m = -R; m <= R; ++m) b = ::fma(T(d2tap(R, m)), t[m + R], b);
        return ::fma(b, x.id2, acc);
    }
    // First derivative from the differences of opposite taps, 1/h last.  1/h in the taps saves that
    // multiplication, but rounds each tap twice: error of Phi' at orders 6 and 8 1.05 to 1.3 times that
    // of the taps summed one by one (spacings 7.3 to 12.5); this form 0.90 to 0.97 times.
    __device__ __forceinline__ T sum_d1() const {
        T b = 0;
#pragma unroll
        for (int m = R; m >= 1; --m) b = ::fma(T(d1w(R, m)), t[R + m] - t[R - m], b);
        return b;
    }
    __device__ __forceinline__ T add_d1(T acc, const Axis<T>& x) const { return ::fma(sum_d1(), x.id, acc); }
    __device__ __forceinline__ T d1(const Axis<T>& x) const { return sum_d1() * x.id; }
    // a tap beside the centre is nonzero
    __device__ __forceinline__ bool any_nonzero() const {
        bool any = false;
#pragma unroll
        for (int m = -R; m <= R; ++m)
            if (m != 0) any |= nonzero(t[m + R]);
        return any;
    }
    // a tap beside the centre is Inf or NaN
    __device__ __forceinline__ bool any_nonfinite() const {
        bool any = false;
#pragma unroll
        for (int m = -R; m <= R; ++m)
            if (m != 0) any |= nonfinite(t[m + R]);
        return any;
    }
};

// u_{k+1} = dt^2 A - (u_{k-1} - 2 u_k), A = C^2 F: the product is added last, in one rounding
template <typename T>
__device__ __forceinline__ T plain_update(T A, T um, T uc, T dt2) {
    return ::fma(dt2, A, ::fma(T(2), uc, -um));
}

// u_{k+1} where a sigma is nonzero: A = C^2 (F - ...), a = dt * sum of the sigmas; w = the sum of
// their products times 2 dt^2, zero where only one is nonzero
template <typename T>
__device__ __forceinline__ T pml_update(T A, T um, T uc, T a, T w, T dt2x2) {
    T num = dt2x2 * A + (a + a) * (um - uc);
    num -= w * uc;
    return (T(2) * uc - um) + num * (T(1) / (T(2) + a));
}

template <typename T>
struct Step1DArgs {
    const T *km1_u, *k_phiz, *k_u, *C, *rhs;
    Prof<T> pz;
    Axis<T> z;
    T dt, dt2, dt2x2;
    int nz;
    T *kp1_phiz, *kp1_u;
};

template <typename T, int R>
__global__ void __launch_bounds__(256) step1d_kernel(Step1DArgs<T> a) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.nz) return;
    if (k == 0 || k == a.nz - 1) {
        a.kp1_phiz[k] = 0;
        a.kp1_u[k] = 0;
        return;
    }
    const Taps<T, R> uz(a.k_u, k, 1, k, a.nz);
    const T um = a.km1_u[k], uc = uz.t[R], ph = a.k_phiz[k];
    T F = uz.add_d2(a.rhs[k], a.z);
    const Taps<T, R> qz(a.k_phiz, k, 1, k, a.nz);
    if (qz.any_nonzero()) F = qz.add_d1(F, a.z);
    const T sz = a.pz.at(k, a.nz);
    const T A = a.C[k] * a.C[k] * F;
    if (nonzero(sz)) {
        const T az = a.dt * sz;
        a.kp1_phiz[k] = ph - az * (ph + uz.d1(a.z));
        a.kp1_u[k] = pml_update(A, um, uc, az, T(0), a.dt2x2);
    } else {
        a.kp1_phiz[k] = ph;
        a.kp1_u[k] = plain_update(A, um, uc, a.dt2);
    }
}

template <typename T>
struct Step2DArgs {
    const T *km1_u, *k_phix, *k_phiz, *k_u, *C, *rhs;
    Prof<T> px, pz;
    Axis<T> x, z;
    T dt, dt2, dt2x2;
    int nx, nz;
    T *kp1_phix, *kp1_phiz, *kp1_u;
};

template <typename T, int R>
__global__ void __launch_bounds__(256) step2d_kernel(Step2DArgs<T> a) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    int i = blockIdx.y * blockDim.y + threadIdx.y;
    if (k >= a.nz || i >= a.nx) return;
    long long idx = (long long)i * a.nz + k;
    if (i == 0 || i == a.nx - 1 || k == 0 || k == a.nz - 1) {
        a.kp1_phix[idx] = 0;
        a.kp1_phiz[idx] = 0;
        a.kp1_u[idx] = 0;
        return;
    }
    const Taps<T, R> ux(a.k_u, idx, a.nz, i, a.nx), uz(a.k_u, idx, 1, k, a.nz);
    const T um = a.km1_u[idx], uc = uz.t[R];
    const T phx = a.k_phix[idx], phz = a.k_phiz[idx];
    T F = uz.add_d2(ux.add_d2(a.rhs[idx], a.x), a.z);
    const Taps<T, R> qx(a.k_phix, idx, a.nz, i, a.nx), qz(a.k_phiz, idx, 1, k, a.nz);
    if (qx.any_nonzero() || qz.any_nonzero()) F = qz.add_d1(qx.add_d1(F, a.x), a.z);
    const T sx = a.px.at(i, a.nx), sz = a.pz.at(k, a.nz);
    const T A = a.C[idx] * a.C[idx] * F;
    if (nonzero(sz) || nonzero(sx)) {
        const T ax = a.dt * sx, az = a.dt * sz;
        a.kp1_phix[idx] = (phx - ax * phx) + (az - ax) * ux.d1(a.x);
        a.kp1_phiz[idx] = (phz - az * phz) + (ax - az) * uz.d1(a.z);
        a.kp1_u[idx] = pml_update(A, um, uc, ax + az, nonzero(sx) && nonzero(sz) ? a.dt2x2 * (sx * sz) : T(0), a.dt2x2);
    } else {
        a.kp1_phix[idx] = phx;
        a.kp1_phiz[idx] = phz;
        a.kp1_u[idx] = plain_update(A, um, uc, a.dt2);
    }
}

template <typename T>
struct Step3DArgs {
    const T *km1_u, *k_phix, *k_phiy, *k_phiz, *k_psi, *k_u, *C, *rhs;
    Prof<T> px, py, pz;
    Axis<T> x, y, z;
    T dt, dt2, dt2x2;
    int nx, ny, nz;
    unsigned zblocks;  // blocks along z; grid x runs over (y, z) blocks, for any ny the interface takes
    T *kp1_phix, *kp1_phiy, *kp1_phiz, *kp1_psi, *kp1_u;
};

// blocks of 128 threads an SM for the registers that each radius needs without spills
__host__ __device__ constexpr int step3d_blocks(int R) { return R == 1 ? 8 : R == 2 ? 6 : R == 3 ? 4 : 3; }

template <typename T, int R>
__global__ void __launch_bounds__(128, step3d_blocks(R)) step3d_kernel(Step3DArgs<T> a) {
    int k = (blockIdx.x % a.zblocks) * blockDim.x + threadIdx.x;
    int j = (blockIdx.x / a.zblocks) * blockDim.y + threadIdx.y;
    int i = blockIdx.y;
    if (k >= a.nz || j >= a.ny) return;
    long long ys = a.nz, xs = (long long)a.ny * a.nz;
    long long idx = (long long)i * xs + (long long)j * ys + k;
    if (i == 0 || i == a.nx - 1 || j == 0 || j == a.ny - 1 || k == 0 || k == a.nz - 1) {
        a.kp1_u[idx] = 0;
        a.kp1_phix[idx] = 0;
        a.kp1_phiy[idx] = 0;
        a.kp1_phiz[idx] = 0;
        a.kp1_psi[idx] = 0;
        return;
    }
    const Taps<T, R> ux(a.k_u, idx, xs, i, a.nx), uy(a.k_u, idx, ys, j, a.ny), uz(a.k_u, idx, 1, k, a.nz);
    const T um = a.km1_u[idx], uc = uz.t[R], ps = a.k_psi[idx];
    T F = ux.add_d2(a.rhs[idx], a.x);
    F = uz.add_d2(uy.add_d2(F, a.y), a.z);
    {   // one test for the three axes: a body this long stays a branch
        const Taps<T, R> qx(a.k_phix, idx, xs, i, a.nx), qy(a.k_phiy, idx, ys, j, a.ny), qz(a.k_phiz, idx, 1, k, a.nz);
        if (qx.any_nonzero() || qy.any_nonzero() || qz.any_nonzero())
            F = qz.add_d1(qy.add_d1(qx.add_d1(F, a.x), a.y), a.z);
    }
    const T sx = a.px.at(i, a.nx), sy = a.py.at(j, a.ny), sz = a.pz.at(k, a.nz);
    const T c2 = a.C[idx] * a.C[idx];
    a.kp1_psi[idx] = ps + a.dt * uc;
    const bool bx = nonzero(sx), by = nonzero(sy), bz = nonzero(sz);
    if (bx || by || bz) {
        const T ax = a.dt * sx, ay = a.dt * sy, az = a.dt * sz, s = ax + ay + az;
        const T phx = a.k_phix[idx], phy = a.k_phiy[idx], phz = a.k_phiz[idx];
        T qx = (phx - ax * phx) + (s - T(2) * ax) * ux.d1(a.x);
        T qy = (phy - ay * phy) + (s - T(2) * ay) * uy.d1(a.y);
        T qz = (phz - az * phz) + (s - T(2) * az) * uz.d1(a.z);
        // products of sigmas: where two are nonzero; an Inf or NaN in psi counts everywhere
        const Taps<T, R> px(a.k_psi, idx, xs, i, a.nx), py(a.k_psi, idx, ys, j, a.ny), pz(a.k_psi, idx, 1, k, a.nz);
        T w = 0;
        if ((bx && by) || (bx && bz) || (by && bz) || nonfinite(ps) || px.any_nonfinite() || py.any_nonfinite() ||
            pz.any_nonfinite()) {
            const T syz = sy * sz, szx = sz * sx, sxy = sx * sy;
            qx += a.dt * (syz * px.d1(a.x));
            qy += a.dt * (szx * py.d1(a.y));
            qz += a.dt * (sxy * pz.d1(a.z));
            F -= (sx * syz) * ps;
            w = a.dt2x2 * (sxy + syz + szx);
        }
        a.kp1_phix[idx] = qx;
        a.kp1_phiy[idx] = qy;
        a.kp1_phiz[idx] = qz;
        a.kp1_u[idx] = pml_update(c2 * F, um, uc, s, w, a.dt2x2);
    } else {
        a.kp1_phix[idx] = a.k_phix[idx];
        a.kp1_phiy[idx] = a.k_phiy[idx];
        a.kp1_phiz[idx] = a.k_phiz[idx];
        a.kp1_u[idx] = plain_update(c2 * F, um, uc, a.dt2);
    }
}

// dWaveOp = (u+ - 2u + u-)/dt^2 + S1 (u+ - u-)/(2dt) + S2 u + S3 psi; threads along z, rows (i, j) on the
// block's second axis: no 64-bit division per cell.
// 78% of the FP64 units' rate, DRAM 24%: cells without a sigma skip the sigma terms
template <typename T>
__global__ void __launch_bounds__(256) dwaveop_kernel(int dim, const T* __restrict__ um,
                                                      const T* __restrict__ uc,
                                                      const T* __restrict__ up,
                                                      const T* __restrict__ psi,
                                                      const T* __restrict__ sgx,
                                                      const T* __restrict__ sgy,
                                                      const T* __restrict__ sgz, int nx, int ny,
                                                      int nz, T idt2, T i2dt, T* __restrict__ out) {
    const long long rows = (long long)nx * ny;
    for (long long r = blockIdx.x * (long long)blockDim.y + threadIdx.y; r < rows; r += (long long)gridDim.x * blockDim.y) {
        const int i = (int)(r >> 31 ? r / ny : (unsigned)r / (unsigned)ny), j = (int)(r - (long long)i * ny);
        const T sx = sgx ? sgx[i] : T(0), sy = sgy ? sgy[j] : T(0);
        const bool brow = nonzero(sx) || nonzero(sy);
        for (long long k = blockIdx.y * blockDim.x + threadIdx.x; k < nz; k += gridDim.y * blockDim.x) {
            const long long c = r * nz + k;
            const T sz = sgz ? sgz[k] : T(0);
            const T a = um[c], b = uc[c], d = up[c], p = dim == 3 && psi ? psi[c] : T(0);
            T v = ((d - T(2) * b) + a) * idt2;
            // one branch for all sigma terms; Inf and NaN take it everywhere
            if (brow || nonzero(sz) || nonfinite(v) || nonfinite(p)) {
                const T srow = sx + sy, sxy = sx * sy;
                v += ((srow + sz) * i2dt) * (d - a);
                v += (sxy + srow * sz) * b;
                v += (sxy * sz) * p;
            }
            out[c] = v;
        }
    }
}

template <typename T>
Prof<T> prof(const void* l, int nl, const void* r, int nr) {
    return Prof<T>{static_cast<const T*>(l), nl, static_cast<const T*>(r), nr};
}

template <typename T>
Axis<T> axis(double h) {
    return Axis<T>{T(1.0 / h), T(1.0 / (T(h) * T(h)))};
}

template <typename T>
int launch1d(int order, const void* km1_u, const void* k_phiz, const void* k_u, const void* C,
             const void* rhs, const void* zl, int nzl, const void* zr, int nzr, double dt,
             double dz, int nz, void* kp1_phiz, void* kp1_u, cudaStream_t s) {
    const Axis<T> z = axis<T>(dz);
    Step1DArgs<T> a{(const T*)km1_u, (const T*)k_phiz, (const T*)k_u, (const T*)C, (const T*)rhs,
                    prof<T>(zl, nzl, zr, nzr), z, T(dt), T(T(dt) * T(dt)), T(2) * T(T(dt) * T(dt)),
 nz, (T*)kp1_phiz, (T*)kp1_u};
    dim3 blk(256), grd(ceil_div(nz, 256));
    switch (order) {
        case 2: step1d_kernel<T, 1><<<grd, blk, 0, s>>>(a); break;
        case 4: step1d_kernel<T, 2><<<grd, blk, 0, s>>>(a); break;
        case 6: step1d_kernel<T, 3><<<grd, blk, 0, s>>>(a); break;
        case 8: step1d_kernel<T, 4><<<grd, blk, 0, s>>>(a); break;
    }
    PGB_CHECK_CUDA(cudaGetLastError());
    return PYSIT_OK;
}

template <typename T>
int launch2d(int order, const void* km1_u, const void* k_phix, const void* k_phiz,
             const void* k_u, const void* C, const void* rhs, const void* xl, int nxl,
             const void* xr, int nxr, const void* zl, int nzl, const void* zr, int nzr,
             double dt, double dx, double dz, int nx, int nz, void* kp1_phix, void* kp1_phiz,
             void* kp1_u, cudaStream_t s) {
    const Axis<T> x = axis<T>(dx), z = axis<T>(dz);
    Step2DArgs<T> a{(const T*)km1_u, (const T*)k_phix, (const T*)k_phiz, (const T*)k_u,
                    (const T*)C, (const T*)rhs, prof<T>(xl, nxl, xr, nxr), prof<T>(zl, nzl, zr, nzr),
                    x, z, T(dt), T(T(dt) * T(dt)), T(2) * T(T(dt) * T(dt)), nx, nz, (T*)kp1_phix, (T*)kp1_phiz, (T*)kp1_u};
    dim3 blk(32, 8), grd(ceil_div(nz, 32), ceil_div(nx, 8));
    switch (order) {
        case 2: step2d_kernel<T, 1><<<grd, blk, 0, s>>>(a); break;
        case 4: step2d_kernel<T, 2><<<grd, blk, 0, s>>>(a); break;
        case 6: step2d_kernel<T, 3><<<grd, blk, 0, s>>>(a); break;
        case 8: step2d_kernel<T, 4><<<grd, blk, 0, s>>>(a); break;
    }
    PGB_CHECK_CUDA(cudaGetLastError());
    return PYSIT_OK;
}

template <typename T>
int launch3d(int order, const void* km1_u, const void* k_phix, const void* k_phiy,
             const void* k_phiz, const void* k_psi, const void* k_u, const void* C,
             const void* rhs, const void* xl, int nxl, const void* xr, int nxr, const void* yl,
             int nyl, const void* yr, int nyr, const void* zl, int nzl, const void* zr, int nzr,
             double dt, double dx, double dy, double dz, int nx, int ny, int nz, void* kp1_phix,
             void* kp1_phiy, void* kp1_phiz, void* kp1_psi, void* kp1_u, cudaStream_t s) {
    const Axis<T> x = axis<T>(dx), y = axis<T>(dy), z = axis<T>(dz);
    Step3DArgs<T> a{(const T*)km1_u, (const T*)k_phix, (const T*)k_phiy, (const T*)k_phiz,
                    (const T*)k_psi, (const T*)k_u, (const T*)C, (const T*)rhs,
                    prof<T>(xl, nxl, xr, nxr), prof<T>(yl, nyl, yr, nyr), prof<T>(zl, nzl, zr, nzr),
                    x, y, z, T(dt), T(T(dt) * T(dt)), T(2) * T(T(dt) * T(dt)), nx, ny, nz, (unsigned)ceil_div(nz, 32),
                    (T*)kp1_phix, (T*)kp1_phiy, (T*)kp1_phiz, (T*)kp1_psi, (T*)kp1_u};
    const long long yz = (long long)ceil_div(nz, 32) * ceil_div(ny, 4);
    PGB_REQUIRE(yz < (1LL << 31), "grid too large for the per-step 3D kernel");
    dim3 blk(32, 4), grd((unsigned)yz, nx);
    switch (order) {
        case 2: step3d_kernel<T, 1><<<grd, blk, 0, s>>>(a); break;
        case 4: step3d_kernel<T, 2><<<grd, blk, 0, s>>>(a); break;
        case 6: step3d_kernel<T, 3><<<grd, blk, 0, s>>>(a); break;
        case 8: step3d_kernel<T, 4><<<grd, blk, 0, s>>>(a); break;
    }
    PGB_CHECK_CUDA(cudaGetLastError());
    return PYSIT_OK;
}

int check_common(int dtype, int order) {
    PGB_REQUIRE(dtype == PYSIT_F32 || dtype == PYSIT_F64, "dtype must be PYSIT_F32 or PYSIT_F64 (got %d)", dtype);
    PGB_REQUIRE(order == 2 || order == 4 || order == 6 || order == 8,
                "spatial_accuracy_order must be one of 2, 4, 6, 8 (got %d)", order);
    return PYSIT_OK;
}

int check_sigma(const void* l, int nl, const void* r, int nr, int n, const char* ax) {
    PGB_REQUIRE(nl >= 0 && nr >= 0, "negative PML profile length on axis %s", ax);
    PGB_REQUIRE(nl == 0 || l, "NULL left PML profile on axis %s", ax);
    PGB_REQUIRE(nr == 0 || r, "NULL right PML profile on axis %s", ax);
    PGB_REQUIRE(nl <= n && nr <= n, "PML profile longer than the axis %s (n=%d)", ax, n);
    return PYSIT_OK;
}

}  // namespace
}  // namespace pgb

using namespace pgb;

extern "C" int pysit_cda_step_1d(int dtype, int order, const void* km1_u, const void* k_phiz,
                                 const void* k_u, const void* C, const void* rhs,
                                 const void* zlpml, int n_zlpml, const void* zrpml, int n_zrpml,
                                 double dt, double dz, int nz, void* kp1_phiz, void* kp1_u,
                                 void* stream) {
    int rc = check_common(dtype, order);
    if (rc) return rc;
    PGB_REQUIRE(nz >= 3, "nz must be >= 3 (got %d)", nz);
    PGB_REQUIRE(km1_u && k_phiz && k_u && C && rhs && kp1_phiz && kp1_u, "NULL array argument");
    rc = check_sigma(zlpml, n_zlpml, zrpml, n_zrpml, nz, "z");
    if (rc) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == PYSIT_F64)
        return launch1d<double>(order, km1_u, k_phiz, k_u, C, rhs, zlpml, n_zlpml, zrpml, n_zrpml,
                                dt, dz, nz, kp1_phiz, kp1_u, s);
    return launch1d<float>(order, km1_u, k_phiz, k_u, C, rhs, zlpml, n_zlpml, zrpml, n_zrpml, dt,
                           dz, nz, kp1_phiz, kp1_u, s);
}

extern "C" int pysit_cda_step_2d(int dtype, int order, const void* km1_u, const void* k_phix,
                                 const void* k_phiz, const void* k_u, const void* C,
                                 const void* rhs, const void* xlpml, int n_xlpml,
                                 const void* xrpml, int n_xrpml, const void* zlpml, int n_zlpml,
                                 const void* zrpml, int n_zrpml, double dt, double dx, double dz,
                                 int nx, int nz, void* kp1_phix, void* kp1_phiz, void* kp1_u,
                                 void* stream) {
    int rc = check_common(dtype, order);
    if (rc) return rc;
    PGB_REQUIRE(nx >= 3 && nz >= 3, "grid must be at least 3x3 (got %dx%d)", nx, nz);
    PGB_REQUIRE(km1_u && k_phix && k_phiz && k_u && C && rhs && kp1_phix && kp1_phiz && kp1_u,
                "NULL array argument");
    if ((rc = check_sigma(xlpml, n_xlpml, xrpml, n_xrpml, nx, "x"))) return rc;
    if ((rc = check_sigma(zlpml, n_zlpml, zrpml, n_zrpml, nz, "z"))) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == PYSIT_F64)
        return launch2d<double>(order, km1_u, k_phix, k_phiz, k_u, C, rhs, xlpml, n_xlpml, xrpml,
                                n_xrpml, zlpml, n_zlpml, zrpml, n_zrpml, dt, dx, dz, nx, nz,
                                kp1_phix, kp1_phiz, kp1_u, s);
    return launch2d<float>(order, km1_u, k_phix, k_phiz, k_u, C, rhs, xlpml, n_xlpml, xrpml,
                           n_xrpml, zlpml, n_zlpml, zrpml, n_zrpml, dt, dx, dz, nx, nz, kp1_phix,
                           kp1_phiz, kp1_u, s);
}

extern "C" int pysit_cda_step_3d(int dtype, int order, const void* km1_u, const void* k_phix,
                                 const void* k_phiy, const void* k_phiz, const void* k_psi,
                                 const void* k_u, const void* C, const void* rhs,
                                 const void* xlpml, int n_xlpml, const void* xrpml, int n_xrpml,
                                 const void* ylpml, int n_ylpml, const void* yrpml, int n_yrpml,
                                 const void* zlpml, int n_zlpml, const void* zrpml, int n_zrpml,
                                 double dt, double dx, double dy, double dz, int nx, int ny,
                                 int nz, void* kp1_phix, void* kp1_phiy, void* kp1_phiz,
                                 void* kp1_psi, void* kp1_u, void* stream) {
    int rc = check_common(dtype, order);
    if (rc) return rc;
    PGB_REQUIRE(nx >= 3 && ny >= 3 && nz >= 3, "grid must be at least 3x3x3 (got %dx%dx%d)", nx, ny, nz);
    PGB_REQUIRE(ny <= 65535 * 8 && nx <= 65535, "grid too large for the per-step 3D kernel");
    PGB_REQUIRE(km1_u && k_phix && k_phiy && k_phiz && k_psi && k_u && C && rhs && kp1_phix &&
                    kp1_phiy && kp1_phiz && kp1_psi && kp1_u,
                "NULL array argument");
    if ((rc = check_sigma(xlpml, n_xlpml, xrpml, n_xrpml, nx, "x"))) return rc;
    if ((rc = check_sigma(ylpml, n_ylpml, yrpml, n_yrpml, ny, "y"))) return rc;
    if ((rc = check_sigma(zlpml, n_zlpml, zrpml, n_zrpml, nz, "z"))) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == PYSIT_F64)
        return launch3d<double>(order, km1_u, k_phix, k_phiy, k_phiz, k_psi, k_u, C, rhs, xlpml,
                                n_xlpml, xrpml, n_xrpml, ylpml, n_ylpml, yrpml, n_yrpml, zlpml,
                                n_zlpml, zrpml, n_zrpml, dt, dx, dy, dz, nx, ny, nz, kp1_phix,
                                kp1_phiy, kp1_phiz, kp1_psi, kp1_u, s);
    return launch3d<float>(order, km1_u, k_phix, k_phiy, k_phiz, k_psi, k_u, C, rhs, xlpml,
                           n_xlpml, xrpml, n_xrpml, ylpml, n_ylpml, yrpml, n_yrpml, zlpml, n_zlpml,
                           zrpml, n_zrpml, dt, dx, dy, dz, nx, ny, nz, kp1_phix, kp1_phiy,
                           kp1_phiz, kp1_psi, kp1_u, s);
}

extern "C" int pysit_cda_dwaveop(int dtype, int dim, const void* km1_u, const void* k_u,
                                 const void* kp1_u, const void* psi_k, const void* sig_x,
                                 const void* sig_y, const void* sig_z, int nx, int ny, int nz,
                                 double dt, void* out, void* stream) {
    PGB_REQUIRE(dtype == PYSIT_F32 || dtype == PYSIT_F64, "bad dtype %d", dtype);
    PGB_REQUIRE(dim >= 1 && dim <= 3, "dim must be 1, 2 or 3 (got %d)", dim);
    PGB_REQUIRE(nx >= 1 && ny >= 1 && nz >= 1, "bad grid size");
    PGB_REQUIRE(km1_u && k_u && kp1_u && out, "NULL array argument");
    PGB_REQUIRE(dim < 3 || psi_k, "3D dWaveOp needs psi_k");
    const long long rows = (long long)nx * ny;
    const dim3 blk = rows < 8 ? dim3(256) : dim3(32, 8);  // few rows (1D): the whole block along z
    const dim3 blocks((unsigned)std::min((rows + blk.y - 1) / blk.y, 1LL << 20),
                      (unsigned)std::min(((long long)nz + blk.x - 1) / blk.x, 65535LL));
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == PYSIT_F64) {
        dwaveop_kernel<double><<<blocks, blk, 0, s>>>(
            dim, (const double*)km1_u, (const double*)k_u, (const double*)kp1_u,
            (const double*)psi_k, (const double*)sig_x, (const double*)sig_y, (const double*)sig_z,
            nx, ny, nz, 1.0 / (dt * dt), 1.0 / (2.0 * dt), (double*)out);
    } else {
        dwaveop_kernel<float><<<blocks, blk, 0, s>>>(
            dim, (const float*)km1_u, (const float*)k_u, (const float*)kp1_u, (const float*)psi_k,
            (const float*)sig_x, (const float*)sig_y, (const float*)sig_z, nx, ny, nz,
            (float)(1.0 / (dt * dt)), (float)(1.0 / (2.0 * dt)), (float*)out);
    }
    PGB_CHECK_CUDA(cudaGetLastError());
    return PYSIT_OK;
}
