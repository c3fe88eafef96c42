// Batched 3D leapfrog step: one block per tile of a shot's grid (forward, recompute, adjoint).
//
// Same maths as the reference step cda_time_scalar_3D (pysit/solvers/
// constant_density_acoustic/time/scalar/constant_density_acoustic_time_scalar_3D.h:107-235)
// with the fusions of the batched pipeline (traces of u_k, dWaveOp_k, ic += q_k dWaveOp_k).
//
// A tile is x0..x1-1 by the y-rows of a block by a z-range of at most 32 vectors; a thread owns
// one y-row and one 16-byte vector along z and walks x in chunks of RX planes: the RX + 2R
// planes of its column are loaded at once and serve the RX planes' x-derivatives, then each
// plane's y- and z-neighbours follow.  The rows and planes that threads and chunks share come
// from L1.  A warp takes 32 / nzv rows of a z-range of nzv vectors, so narrow ranges fill warps.
// Tile kinds (block-uniform):
//   0     interior: R cells clear of the padding, off the outer ring: no PML state, no masks;
//   2-4   faces across x, y, z: at most that axis in the padding (with its rim), so that every
//         product of two sigmas vanishes and psi plays no part;
//   1     the rest of the PML shell (edges, corners): the general update.
// 3D auxiliary state: Phi_x/y/z is non-zero only inside the padding; psi
// (integrated on every cell by the reference, _3D.h:216,230) only influences
// the outputs through products of two or three sigmas, so the batched path
// integrates it only where at least two axes are inside the padding.
//
// What bounds it: latency (two thirds of a warp's cycles wait on loads with four 4-warp blocks per SM at
// 128 registers; issue slots 28-31 %, DRAM 43-55 %, L1 43-47 % busy; the four-plane kernels of order
// 8 spill 12 to 60 bytes in FP32).  Four planes per round need 13 vector loads of u_k per output vector
// instead of 21, the faces' update 135-180 thread instructions per cell instead of the general update's
// 276.  Measured against the kernels this one replaces, which walked 64 planes one at a time in two
// kernels (us per step, before -> now): 440 x 440 x 340, order 8, FP32 forward / recompute / adjoint
// 593 / 595 / 707 -> 483 / 530 / 632; 121 x 107 x 95, order 4, FP32, 4 shots 200 -> 80; 180 x 170 x 150,
// order 8, FP32 201 -> 55; 53 x 49 x 45, order 4, FP64, 2 shots 708 -> 49.  Three blocks per SM (80
// registers, spills) were 12 % slower.
#pragma once
#include "pairs.cuh"
#include "tma.cuh"

namespace pgb {
namespace {

template <typename T> struct Vec3;
template <> struct Vec3<float> { using type = float4; static constexpr int N = 4; };
template <> struct Vec3<double> { using type = double2; static constexpr int N = 2; };

template <typename T>
__device__ __forceinline__ typename Vec3<T>::type ldv(const T* q) {
    return *reinterpret_cast<const typename Vec3<T>::type*>(q);
}

// a lane's V cells as an array (the components of a vector load)
template <typename T>
__device__ __forceinline__ T vc(const typename Vec3<T>::type& a, int v) {
    return reinterpret_cast<const T*>(&a)[v];
}

// store the first n of a lane's V cells: one vector store when all belong to the task
template <typename T, bool STREAM>
__device__ __forceinline__ void st_lane(T* q, const T* a, int n) {
    using VT = typename Vec3<T>::type;
    constexpr int V = Vec3<T>::N;
    if (n == V) {
        if constexpr (STREAM) __stcs(reinterpret_cast<VT*>(q), *reinterpret_cast<const VT*>(a));
        else *reinterpret_cast<VT*>(q) = *reinterpret_cast<const VT*>(a);
    } else {
#pragma unroll
        for (int v = 0; v < V; ++v)
            if (v < n) {
                if constexpr (STREAM) __stcs(q + v, a[v]);
                else q[v] = a[v];
            }
    }
}

// first derivative sum_m a_m (v_+m - v_-m) of each of a lane's cells along x or y
// from the 2R tap vectors t (t[R - m] at -m, t[R + m - 1] at +m), scaled by h
template <typename T, int R>
__device__ __forceinline__ void dd1_taps(const typename Vec3<T>::type (&t)[2 * R], T h, T* out) {
#pragma unroll
    for (int v = 0; v < Vec3<T>::N; ++v) {
        T a = T(0);
#pragma unroll
        for (int m = 1; m <= R; ++m) a += T(d1w(R, m)) * (vc<T>(t[R + m - 1], v) - vc<T>(t[R - m], v));
        out[v] = a * h;
    }
}
template <typename T, int R>
__device__ __forceinline__ void load_taps(const T* q, int s, typename Vec3<T>::type (&t)[2 * R]) {
#pragma unroll
    for (int m = 1; m <= R; ++m) {
        t[R - m] = ldv(q - m * s);
        t[R + m - 1] = ldv(q + m * s);
    }
}
// the centre window along z: the lane's V cells with HZ cells on either side
template <typename T, int NB>
__device__ __forceinline__ void load_window(const T* q, T* w) {
    constexpr int V = Vec3<T>::N;
#pragma unroll
    for (int b = 0; b <= 2 * NB; ++b) {
        const typename Vec3<T>::type a = ldv(q + (b - NB) * V);
#pragma unroll
        for (int v = 0; v < V; ++v) w[b * V + v] = vc<T>(a, v);
    }
}


// a tile's part of its shot's injection box; the cells' values in shared memory
struct InjBox {
    int x0, x1, y0, y1, z0, z1;
    __device__ __forceinline__ bool meets(int j, int zl, int V) const {
        return x1 > x0 && j >= y0 && j < y1 && zl < z1 && zl + V > z0;
    }
    template <typename T>
    __device__ __forceinline__ T at(const T* rhs, int x, int y, int z) const {
        return z < z0 || z >= z1 ? T(0) : rhs[((x - x0) * (y1 - y0) + (y - y0)) * (z1 - z0) + z - z0];
    }
};

// factor of the adjoint source added after the step: fac = dt^2, or 2 dt^2 / (2 + dt (sx + sy + sz))
// where a sigma is nonzero, the factor the reference's update applies to C^2 (rhs + ...)
// (_3D.h:220-226); the update is linear in rhs, so adding it afterwards equals injecting it
template <typename T>
__device__ __forceinline__ T inject_fac(const WaveParams<T>& p, T sx, T sy, T sz) {
    return (sx != T(0) || sy != T(0) || sz != T(0)) ? T(2) * p.dt2 / (T(2) + p.dt * (sx + sy + sz)) : p.dt2;
}

// General update of edges and corners: V cells per thread along z, plane by plane.  Operand
// groups no cell of the vector needs are skipped: Phi taps that can only meet zero state, psi
// away from the bands where two axes are in the padding, the PML terms where no sigma is set.
// Cells of the outer ring get zero.
template <typename T, int R, int MODE>
__device__ __forceinline__ void general_update(const WaveParams<T>& p, const T* rhs, const InjBox ib, const int shot,
                                               const int x0, const int x1, const int j, const int zl, const int ze,
                                               FiniteCheck<T>& chk) {
    using VT = typename Vec3<T>::type;
    constexpr int V = Vec3<T>::N;
    constexpr int AL = 16 / (int)sizeof(T);
    constexpr int HZ = (R + AL - 1) / AL * AL;
    constexpr int NB = HZ / V;
    constexpr int NW = (2 * NB + 1) * V;
    constexpr int C0 = NB * V;
    const int nv = min(V, ze - zl);  // cells of the lane's vector inside the task
    const long long sh = (long long)shot * p.fstride;
    const int ys = p.ldz, xs = p.rows_y * p.ldz;  // a field of one shot has fewer than 2^31 elements
    // what the x sweep does not change: y and z sigmas and masks
    const T sy = __ldg(p.sgy + j);
    const T my = MODE == kRecomp ? __ldg(p.mgy + j) : T(0);
    const bool py = j < p.pyl || j >= p.ny - p.pyr;
    const bool neary = j - R < p.pyl || j + R >= p.ny - p.pyr;
    T sz[V], mz[V];
    bool okz[V], pz[V];
    bool any_sz = false, any_pz = false, any_nearz = false;
#pragma unroll
    for (int v = 0; v < V; ++v) {
        const int k = zl + v;
        const bool in = v < nv;
        sz[v] = in ? __ldg(p.sgz + k) : T(0);
        mz[v] = in && MODE == kRecomp ? __ldg(p.mgz + k) : T(0);
        okz[v] = in && j > 0 && j < p.ny - 1 && k > 0 && k < p.nz - 1;
        pz[v] = in && (k < p.pzl || k >= p.nz - p.pzr);
        any_sz |= sz[v] != T(0);
        any_pz |= pz[v];
        any_nearz |= in && (k - R < p.pzl || k + R >= p.nz - p.pzr);
    }
    const bool inj_col = ib.meets(j, zl, V);
    long long o = ((long long)(x0 + p.hx) * p.rows_y + (j + p.hy)) * p.ldz + kOZ + zl;
    for (int i = x0; i < x1; ++i, o += xs) {
        const T sx = __ldg(p.sgx + i);
        const bool px = i < p.pxl || i >= p.nx - p.pxr;
        const bool nearx = i - R < p.pxl || i + R >= p.nx - p.pxr;
        const bool okx = i > 0 && i < p.nx - 1;
        const T* u = p.u_cur + sh + o;
        // u: Laplacian in difference form per axis and the first derivatives
        T w[NW];
        load_window<T, NB>(u, w);
        T uc[V], F[V], dux[V], duy[V], duz[V];
        {
            VT t[2 * R];
            load_taps<T, R>(u, xs, t);
#pragma unroll
            for (int v = 0; v < V; ++v) {
                uc[v] = w[C0 + v];
                T a2 = T(0), a1 = T(0);
#pragma unroll
                for (int m = 1; m <= R; ++m) {
                    const T up = vc<T>(t[R + m - 1], v), um = vc<T>(t[R - m], v);
                    a2 += T(d2w(R, m)) * ((up - uc[v]) + (um - uc[v]));
                    a1 += T(d1w(R, m)) * (up - um);
                }
                F[v] = a2 * p.idx2;
                dux[v] = a1 * p.idx;
            }
            load_taps<T, R>(u, ys, t);
#pragma unroll
            for (int v = 0; v < V; ++v) {
                T a2 = T(0), a1 = T(0);
#pragma unroll
                for (int m = 1; m <= R; ++m) {
                    const T up = vc<T>(t[R + m - 1], v), um = vc<T>(t[R - m], v);
                    a2 += T(d2w(R, m)) * ((up - uc[v]) + (um - uc[v]));
                    a1 += T(d1w(R, m)) * (up - um);
                }
                F[v] += a2 * p.idy2;
                duy[v] = a1 * p.idy;
            }
        }
#pragma unroll
        for (int v = 0; v < V; ++v) {
            T a2 = T(0), a1 = T(0);
#pragma unroll
            for (int m = 1; m <= R; ++m) {
                const T up = w[C0 + v + m], um = w[C0 + v - m];
                a2 += T(d2w(R, m)) * ((up - uc[v]) + (um - uc[v]));
                a1 += T(d1w(R, m)) * (up - um);
            }
            F[v] += a2 * p.idz2;
            duz[v] = a1 * p.idz;
        }
        // Phi derivatives: the state is zero outside the padding; a tap group no cell can
        // see non-zero is skipped (one that some cells need adds exact zeros to the others)
        if (nearx || py || any_pz) {
            VT t[2 * R];
            T d[V];
            load_taps<T, R>(p.phx_in + sh + o, xs, t);
            dd1_taps<T, R>(t, p.idx, d);
#pragma unroll
            for (int v = 0; v < V; ++v) F[v] += d[v];
        }
        if (neary || px || any_pz) {
            VT t[2 * R];
            T d[V];
            load_taps<T, R>(p.phy_in + sh + o, ys, t);
            dd1_taps<T, R>(t, p.idy, d);
#pragma unroll
            for (int v = 0; v < V; ++v) F[v] += d[v];
        }
        if (any_nearz || px || py) {
            load_window<T, NB>(p.phz_in + sh + o, w);
#pragma unroll
            for (int v = 0; v < V; ++v) {
                T a = T(0);
#pragma unroll
                for (int m = 1; m <= R; ++m) a += T(d1w(R, m)) * (w[C0 + v + m] - w[C0 + v - m]);
                F[v] += a * p.idz;
            }
        }
        T rh[V];
        const bool inj_row = inj_col && i >= ib.x0 && i < ib.x1;
        if (inj_row) {
#pragma unroll
            for (int v = 0; v < V; ++v) {
                rh[v] = ib.at(rhs, i, j, zl + v);
                if (MODE != kAdj) F[v] += rh[v];
            }
        }
        bool psireg[V];
        bool any_ps = false;
#pragma unroll
        for (int v = 0; v < V; ++v) {
            psireg[v] = (int)px + (int)py + (int)pz[v] >= 2;
            any_ps |= psireg[v];
        }
        T ps[V];
        if (any_ps) {
            const VT a = ldv(p.psi_in + sh + o);
#pragma unroll
            for (int v = 0; v < V; ++v) ps[v] = psireg[v] ? vc<T>(a, v) : T(0);
        } else {
#pragma unroll
            for (int v = 0; v < V; ++v) ps[v] = T(0);
        }
        const VT uo_v = ldv(p.u_prev + sh + o);
        const VT c2_v = __ldg(reinterpret_cast<const VT*>(p.c2 + o));
        alignas(16) T un[V];
        if (sx != T(0) || sy != T(0) || any_sz) {
            // psi derivatives where two sigmas meet (zero elsewhere, as the products they enter)
            T dpx[V], dpy[V], dpz[V];
#pragma unroll
            for (int v = 0; v < V; ++v) dpx[v] = dpy[v] = dpz[v] = T(0);
            if (sy != T(0) && any_sz) {
                VT t[2 * R];
                load_taps<T, R>(p.psi_in + sh + o, xs, t);
                dd1_taps<T, R>(t, p.idx, dpx);
            }
            if (sx != T(0) && any_sz) {
                VT t[2 * R];
                load_taps<T, R>(p.psi_in + sh + o, ys, t);
                dd1_taps<T, R>(t, p.idy, dpy);
            }
            if (sx != T(0) && sy != T(0)) {
                load_window<T, NB>(p.psi_in + sh + o, w);
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    T a = T(0);
#pragma unroll
                    for (int m = 1; m <= R; ++m) a += T(d1w(R, m)) * (w[C0 + v + m] - w[C0 + v - m]);
                    dpz[v] = a * p.idz;
                }
            }
            const VT phx_v = ldv(p.phx_in + sh + o), phy_v = ldv(p.phy_in + sh + o), phz_v = ldv(p.phz_in + sh + o);
            alignas(16) T nxo[V], nyo[V], nzo[V];
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const T szv = sz[v], uo = vc<T>(uo_v, v), c2 = vc<T>(c2_v, v);
                const T phx = vc<T>(phx_v, v), phy = vc<T>(phy_v, v), phz = vc<T>(phz_v, v);
                const bool pml = sx != T(0) || sy != T(0) || szv != T(0);
                const bool ok = okx && okz[v];
                const T psx = sy != T(0) && szv != T(0) ? dpx[v] : T(0);
                const T psy = szv != T(0) && sx != T(0) ? dpy[v] : T(0);
                const T psz = sx != T(0) && sy != T(0) ? dpz[v] : T(0);
                const T nx_ = phx - p.dt * sx * phx + p.dt * (sy + szv - sx) * dux[v] + p.dt * (sy * szv * psx);
                const T ny_ = phy - p.dt * sy * phy + p.dt * (szv + sx - sy) * duy[v] + p.dt * (szv * sx * psy);
                const T nz_ = phz - p.dt * szv * phz + p.dt * (sx + sy - szv) * duz[v] + p.dt * (sx * sy * psz);
                // (a division only where two sigmas meet: FP64 takes a dozen instructions for it)
                T fac1;
                if (sx == T(0) && sy == T(0)) fac1 = __ldg(p.fcz + min(zl + v, p.nz - 1));
                else if (szv != T(0) || (sx != T(0) && sy != T(0))) fac1 = T(2) * p.dt2 / (T(2) + p.dt * (sx + sy + szv));
                else fac1 = sx != T(0) ? __ldg(p.fcx + i) : __ldg(p.fcy + j);
                // the reference multiplies sigma_x sigma_y sigma_z psi by C^2 (_3D.h:219); the
                // consistent form (psi_c2 = 0) leaves it out, as the matrix operator does
                const T src = p.psi_c2 ? c2 * (F[v] - (sx * sy * szv) * ps[v]) : c2 * F[v] - (sx * sy * szv) * ps[v];
                const T fac2 = src - (uo - T(2) * uc[v]) * p.idt2 + (sx + sy + szv) * uo * p.i2dt -
                               (sx * sy + sy * szv + szv * sx) * uc[v];
                const T upml = fac1 * fac2, uplain = p.dt2 * c2 * F[v] - (uo - T(2) * uc[v]);
                un[v] = ok ? (pml ? upml : uplain) : T(0);
                // cells outside the padding keep their zero state
                nxo[v] = ok && pml ? nx_ : T(0);
                nyo[v] = ok && pml ? ny_ : T(0);
                nzo[v] = ok && pml ? nz_ : T(0);
            }
            st_lane<T, false>(p.phx_out + sh + o, nxo, nv);
            st_lane<T, false>(p.phy_out + sh + o, nyo, nv);
            st_lane<T, false>(p.phz_out + sh + o, nzo, nv);
        } else {
#pragma unroll
            for (int v = 0; v < V; ++v)
                un[v] = okx && okz[v] ? p.dt2 * vc<T>(c2_v, v) * F[v] - (vc<T>(uo_v, v) - T(2) * uc[v]) : T(0);
        }
        if (MODE == kAdj && inj_row) {
            // the adjoint source after the step: u' += fac C^2 rhs (see inject_fac)
#pragma unroll
            for (int v = 0; v < V; ++v)
                if (okx && okz[v]) un[v] = ::fma(inject_fac(p, sx, sy, sz[v]) * vc<T>(c2_v, v), rh[v], un[v]);
        }
        if (any_ps) {
            alignas(16) T pso[V];
#pragma unroll
            for (int v = 0; v < V; ++v) pso[v] = psireg[v] && okx && okz[v] ? ps[v] + p.dt * uc[v] : T(0);
            st_lane<T, false>(p.psi_out + sh + o, pso, nv);
        }
        st_lane<T, false>(p.u_prev + sh + o, un, nv);
        if (MODE == kRecomp && p.dw_out) {
            const T mx = __ldg(p.mgx + i);
            alignas(16) T dwo[V];
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const T szv = sz[v], mzv = mz[v], c2 = vc<T>(c2_v, v), sxyz = sx * sy * szv;
                T d = p.psi_c2 ? c2 * (F[v] - sxyz * ps[v]) : c2 * F[v] - sxyz * ps[v];
                d += ((mx + my + mzv) - (sx + sy + szv)) * (un[v] - vc<T>(uo_v, v)) * p.i2dt +
                     ((mx * my + my * mzv + mzv * mx) - (sx * sy + sy * szv + szv * sx)) * uc[v] + (mx * my * mzv) * ps[v];
                dwo[v] = okx && okz[v] ? d : T(0);
            }
            st_lane<T, true>(p.dw_out + sh + o, dwo, nv);
        }
        if (MODE == kAdj && p.image) {
            const VT dw_v = __ldcs(reinterpret_cast<const VT*>(p.dw_in + sh + o));
            const VT ic_v = ldv(p.ic + sh + o);
            alignas(16) T ico[V];
#pragma unroll
            for (int v = 0; v < V; ++v) ico[v] = vc<T>(ic_v, v) + uc[v] * vc<T>(dw_v, v);
            st_lane<T, false>(p.ic + sh + o, ico, nv);
        }
        if (MODE == kFwd || (MODE == kRecomp && p.nan_check)) {
#pragma unroll
            for (int v = 0; v < V; v += 2)
                chk.see(PairOps<T>::mk(v < nv ? un[v] : T(0), v + 1 < nv ? un[v + 1] : T(0)));
        }
    }
}


// sums of one axis: second derivative (difference form; FP64: over first differences) and first
// derivative of a pair from the 2R + 1 values t(-R) .. t(R), unscaled
template <typename T, int R, bool D1, typename F>
__device__ __forceinline__ void axis_sums(const F& t, typename PairOps<T>::P& a2, typename PairOps<T>::P& a1) {
    using O = PairOps<T>;
    using P = typename O::P;
    const P uc = t(0);
    a2 = O::dup(T(0));
    a1 = a2;
#pragma unroll
    for (int m = 1; m <= R; ++m) {
        const P up = t(m), um = t(-m);
        if (sizeof(T) == 8)
            a2 = O::fma(O::dup(T(c2sum(R, m - 1))), O::sub(O::sub(up, t(m - 1)), O::sub(t(1 - m), um)), a2);
        else
            a2 = O::fma(O::dup(T(d2w(R, m))), O::add(O::sub(up, uc), O::sub(um, uc)), a2);
        if (D1) a1 = O::fma(O::dup(T(d1w(R, m))), O::sub(up, um), a1);
    }
}

__device__ __forceinline__ void pf(const void* q) { asm volatile("prefetch.global.L1 [%0];" ::"l"(q)); }

// the operands of planes x .. x+n-1 of a thread's row that no earlier chunk has read
template <typename T, int R, int MODE, bool PML, int RX>
__device__ __forceinline__ void prefetch_planes(const WaveParams<T>& p, const long long sh, const long long o, const int n) {
    const long long xs = (long long)p.rows_y * p.ldz;
#pragma unroll
    for (int r = 0; r < RX; ++r) {
        if (r >= n) break;
        const long long q = o + (long long)r * xs;
        pf(p.u_cur + sh + q + R * xs);
        pf(p.u_prev + sh + q);
        pf(p.c2 + q);
        if (MODE == kAdj && p.image) {
            pf(p.dw_in + sh + q);
            pf(p.ic + sh + q);
        }
        if (PML) {
            pf(p.phx_in + sh + q + R * xs);
            pf(p.phy_in + sh + q);
            pf(p.phz_in + sh + q);
        }
    }
}

// Interior: RX planes from x on
template <typename T, int R, int MODE, int RX>
__device__ __forceinline__ void interior_planes(const WaveParams<T>& p, const T* rhs, const InjBox& ib, const bool inj_col,
                                                const long long sh, const long long o0, const int x, const int n,
                                                const int j, const int zl, FiniteCheck<T>& chk) {
    using O = PairOps<T>;
    using P = typename O::P;
    constexpr int V = V16<T>::N, NP = V / 2, HZ = (R + V - 1) / V * V, NB = HZ / V, C0 = NB * V;
    constexpr bool DIFF = sizeof(T) == 8;
    const long long ys = p.ldz, xs = (long long)p.rows_y * p.ldz;
    const T* u = p.u_cur + sh + o0;
    P Fx[RX][NP];
    {
        Pairs<T, NP> cv[RX + 2 * R];
        // planes past the tile's last one are read too (the next planes or the halo) and not used
#pragma unroll
        for (int q = 0; q < RX + 2 * R; ++q) ldp(cv[q], u + (long long)(min(q, n - 1 + 2 * R) - R) * xs);
#pragma unroll
        for (int r = 0; r < RX; ++r)
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                const P uc = cv[R + r].p[k];
                P F = O::dup(T(0));
#pragma unroll
                for (int m = 1; m <= R; ++m) {
                    const P up = cv[R + r + m].p[k], um = cv[R + r - m].p[k];
                    if (DIFF)
                        F = O::fma(O::dup(T(c2sum(R, m - 1)) * p.idx2),
                                   O::sub(O::sub(up, cv[R + r + m - 1].p[k]), O::sub(cv[R + r + 1 - m].p[k], um)), F);
                    else
                        F = O::fma(O::dup(T(d2w(R, m)) * p.idx2), O::add(O::sub(up, uc), O::sub(um, uc)), F);
                }
                Fx[r][k] = F;
            }
    }
    // The other operands of plane r.  The adjoint step reads them before plane r - 1 is stored (440 x
    // 440 x 340, order 8, FP32: 3 % faster than after its stores); the other modes, which hold fewer
    // operands a plane, after (forward 1.5 % faster than before).
    constexpr bool AHEAD = MODE == kAdj;
    Window<T, NP, NB> w;
    Pairs<T, NP> ya[2 * R], cc, um, dwi, ici;
    auto fetch = [&](int r) {
        const long long o = o0 + (long long)r * xs;
        const T* ur = u + (long long)r * xs;
        w.load(ur - HZ, nullptr);
#pragma unroll
        for (int m = 1; m <= R; ++m) {
            ldp(ya[R - m], ur - m * ys);
            ldp(ya[R + m - 1], ur + m * ys);
        }
        ldr(cc, p.c2 + o);
        ldp(um, p.u_prev + sh + o);
        if (MODE == kAdj && p.image) {
            ldp(dwi, p.dw_in + sh + o);
            ldp(ici, p.ic + sh + o);
        }
    };
    if (AHEAD) fetch(0);
#pragma unroll
    for (int r = 0; r < RX; ++r) {
        if (r >= n) break;
        const long long o = o0 + (long long)r * xs;
        if (!AHEAD) fetch(r);
        Pairs<T, NP> un, dwo, ico;
        const bool inj_row = inj_col && x + r >= ib.x0 && x + r < ib.x1;
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            const int c = C0 + 2 * k;
            const P uc = w.at(c);
            P Fy = O::dup(T(0)), Fz = Fy;
#pragma unroll
            for (int m = 1; m <= R; ++m) {
                const P up = ya[R + m - 1].p[k], dn = ya[R - m].p[k];
                if (DIFF) {
                    const P up1 = m == 1 ? uc : ya[R + m - 2].p[k], dn1 = m == 1 ? uc : ya[R - m + 1].p[k];
                    Fy = O::fma(O::dup(T(c2sum(R, m - 1)) * p.idy2), O::sub(O::sub(up, up1), O::sub(dn1, dn)), Fy);
                    Fz = O::fma(O::dup(T(c2sum(R, m - 1)) * p.idz2),
                                O::sub(O::sub(w.at(c + m), w.at(c + m - 1)), O::sub(w.at(c - m + 1), w.at(c - m))), Fz);
                } else {
                    Fy = O::fma(O::dup(T(d2w(R, m)) * p.idy2), O::add(O::sub(up, uc), O::sub(dn, uc)), Fy);
                    Fz = w.d2(Fz, O::dup(T(d2w(R, m)) * p.idz2), c, m);
                }
            }
            P F = O::add(O::add(Fx[r][k], Fy), Fz);
            T rh[2];
            if (inj_row) {
                rh[0] = ib.at(rhs, x + r, j, zl + 2 * k);
                rh[1] = ib.at(rhs, x + r, j, zl + 2 * k + 1);
                if (MODE != kAdj) F = O::add(F, O::mk(rh[0], rh[1]));
            }
            const P uo = um.p[k], c2 = cc.p[k];
            // u_{k+1} = dt^2 C^2 F - (u_{k-1} - 2 u_k)
            const P q = O::fma(O::dup(T(-2)), uc, uo);
            un.p[k] = O::fma(O::mul(O::dup(p.dt2), c2), F, O::mul(q, O::dup(T(-1))));
            if (MODE == kRecomp) dwo.p[k] = O::mul(c2, F);
            if (MODE == kAdj && inj_row)
                un.p[k] = O::mk(::fma(p.dt2 * O::lo(c2), rh[0], O::lo(un.p[k])), ::fma(p.dt2 * O::hi(c2), rh[1], O::hi(un.p[k])));
            if (MODE == kAdj) ico.p[k] = O::fma(uc, dwi.p[k], ici.p[k]);
            if (MODE == kFwd || (MODE == kRecomp && p.nan_check)) chk.see(un.p[k]);
        }
        if (AHEAD && r + 1 < RX && r + 1 < n) fetch(r + 1);
        stp(p.u_prev + sh + o, un);
        if (MODE == kRecomp && p.dw_out) stp_cs(p.dw_out + sh + o, dwo);
        if (MODE == kAdj && p.image) stp(p.ic + sh + o, ico);
    }
}

// per-thread constants of a face tile's columns (what the x walk does not change)
template <typename T, int NP>
struct FaceCol {
    T sy, my;
    T sz[2 * NP], mz[2 * NP];
    typename PairOps<T>::P fz[NP];  // z faces: 2 dt^2 / (2 + dt sz)
    bool zall, any_sz;              // no cell on the ring along y or z; a cell with sigma_z
    bool need_xz, need_yz, need_z;  // Phi taps along x / y / z that this column needs whatever x is
};

// Faces: RX planes from x on.  AX (0 x, 1 y, 2 z): the axis that may be in the padding.  With one
// sigma s nonzero at most, the split-field update (_3D.h:196-230) is
//     Phi_AX' = Phi_AX - dt s Phi_AX - dt s du/dAX,   Phi_o' = Phi_o + dt s du/do  (the others),
//     u' = 2 dt^2 / (2 + dt s) (C^2 F - (u_{k-1} - 2u)/dt^2 + s u_{k-1}/(2dt)),
// the general update with its zero terms left out.
template <typename T, int R, int MODE, int RX, int AX>
__device__ __forceinline__ void face_planes(const WaveParams<T>& p, const T* rhs, const InjBox& ib, const bool inj_col,
                                            const FaceCol<T, V16<T>::N / 2>& col, const long long sh, const long long o0,
                                            const int x, const int n, const int j, const int zl,
                                            FiniteCheck<T>& chk) {
    using O = PairOps<T>;
    using P = typename O::P;
    constexpr int V = V16<T>::N, NP = V / 2, HZ = (R + V - 1) / V * V, NB = HZ / V, C0 = NB * V;
    const long long ys = p.ldz, xs = (long long)p.rows_y * p.ldz;
    const T* u = p.u_cur + sh + o0;
    P Fx[RX][NP], dux[RX][NP], dpx[RX][NP];
    {
        Pairs<T, NP> cv[RX + 2 * R];
#pragma unroll
        for (int q = 0; q < RX + 2 * R; ++q) ldp(cv[q], u + (long long)(min(q, n - 1 + 2 * R) - R) * xs);
#pragma unroll
        for (int r = 0; r < RX; ++r)
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                P a2, a1;
                axis_sums<T, R, true>([&](int m) { return cv[R + r + m].p[k]; }, a2, a1);
                Fx[r][k] = a2;
                dux[r][k] = O::mul(a1, O::dup(p.idx));
            }
    }
    // Phi_x is zero outside the padding: taps that can only meet zeros are not read
    const bool needx = AX != 0 ? col.need_xz : (x - R < p.pxl || x + n - 1 + R >= p.nx - p.pxr);
    if (needx) {
        Pairs<T, NP> px[RX + 2 * R];
#pragma unroll
        for (int q = 0; q < RX + 2 * R; ++q) ldp(px[q], p.phx_in + sh + o0 + (long long)(min(q, n - 1 + 2 * R) - R) * xs);
#pragma unroll
        for (int r = 0; r < RX; ++r)
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                P a = O::dup(T(0));
#pragma unroll
                for (int m = 1; m <= R; ++m) a = O::fma(O::dup(T(d1w(R, m))), O::sub(px[R + r + m].p[k], px[R + r - m].p[k]), a);
                dpx[r][k] = a;
            }
    }
#pragma unroll
    for (int r = 0; r < RX; ++r) {
        if (r >= n) break;
        const int i = x + r;
        const long long o = o0 + (long long)r * xs;
        const T sx = AX == 0 ? __ldg(p.sgx + i) : T(0);
        const bool pxin = AX == 0 && (i < p.pxl || i >= p.nx - p.pxr);
        const T* ur = u + (long long)r * xs;
        Window<T, NP, NB> w;
        w.load(ur - HZ, nullptr);
        Pairs<T, NP> ya[2 * R], cc, um;
#pragma unroll
        for (int m = 1; m <= R; ++m) {
            ldp(ya[R - m], ur - m * ys);
            ldp(ya[R + m - 1], ur + m * ys);
        }
        ldr(cc, p.c2 + o);
        ldp(um, p.u_prev + sh + o);
        Pairs<T, NP> dwi, ici;
        if (MODE == kAdj && p.image) {
            ldp(dwi, p.dw_in + sh + o);
            ldp(ici, p.ic + sh + o);
        }
        P F[NP], duy[NP], duz[NP], uc[NP];
        {
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                const int c = C0 + 2 * k;
                uc[k] = w.at(c);
                P a2, a1;
                axis_sums<T, R, true>([&](int m) { return m == 0 ? uc[k] : m > 0 ? ya[R + m - 1].p[k] : ya[R + m].p[k]; }, a2, a1);
                F[k] = O::fma(Fx[r][k], O::dup(p.idx2), O::mul(a2, O::dup(p.idy2)));
                duy[k] = O::mul(a1, O::dup(p.idy));
                P z2 = O::dup(T(0)), z1 = z2;
#pragma unroll
                for (int m = 1; m <= R; ++m) {
                    if (sizeof(T) == 8)
                        z2 = O::fma(O::dup(T(c2sum(R, m - 1))),
                                    O::sub(O::sub(w.at(c + m), w.at(c + m - 1)), O::sub(w.at(c - m + 1), w.at(c - m))), z2);
                    else
                        z2 = w.d2(z2, O::dup(T(d2w(R, m))), c, m);
                    z1 = w.d1(z1, O::dup(T(d1w(R, m))), c, m);
                }
                F[k] = O::fma(z2, O::dup(p.idz2), F[k]);
                duz[k] = O::mul(z1, O::dup(p.idz));
            }
        }
        if (needx)
#pragma unroll
            for (int k = 0; k < NP; ++k) F[k] = O::fma(dpx[r][k], O::dup(p.idx), F[k]);
        if (col.need_yz || pxin) {
            Pairs<T, NP> t[2 * R];
#pragma unroll
            for (int m = 1; m <= R; ++m) {
                ldp(t[R - m], p.phy_in + sh + o - m * ys);
                ldp(t[R + m - 1], p.phy_in + sh + o + m * ys);
            }
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                P a = O::dup(T(0));
#pragma unroll
                for (int m = 1; m <= R; ++m) a = O::fma(O::dup(T(d1w(R, m))), O::sub(t[R + m - 1].p[k], t[R - m].p[k]), a);
                F[k] = O::fma(a, O::dup(p.idy), F[k]);
            }
        }
        Window<T, NP, NB> wz;
        if (col.need_z || pxin) {
            wz.load(p.phz_in + sh + o - HZ, nullptr);
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                P a = O::dup(T(0));
#pragma unroll
                for (int m = 1; m <= R; ++m) a = wz.d1(a, O::dup(T(d1w(R, m))), C0 + 2 * k, m);
                F[k] = O::fma(a, O::dup(p.idz), F[k]);
            }
        }
        const bool inj_row = inj_col && i >= ib.x0 && i < ib.x1;
        T rh[V];
        if (inj_row) {
#pragma unroll
            for (int v = 0; v < V; ++v) rh[v] = ib.at(rhs, i, j, zl + v);
            if (MODE != kAdj)
#pragma unroll
                for (int k = 0; k < NP; ++k) F[k] = O::add(F[k], O::mk(rh[2 * k], rh[2 * k + 1]));
        }
        Pairs<T, NP> un, dwo;
        const T s1 = AX == 0 ? sx : col.sy;  // the face's sigma where it is the same for the vector
        const bool pml = AX == 2 ? col.any_sz : s1 != T(0);
        const bool ring = !(col.zall && i > 0 && i < p.nx - 1);
        const bool xok = i > 0 && i < p.nx - 1 && j > 0 && j < p.ny - 1;
        auto mask = [&](P a, int k) {  // cells of the outer ring (or past the grid's end) get zero
            const int z = zl + 2 * k;
            return O::mk(xok && z > 0 && z < p.nz - 1 ? O::lo(a) : T(0), xok && z + 1 < p.nz - 1 ? O::hi(a) : T(0));
        };
        P plain[NP];
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            const P q = O::fma(O::dup(T(-2)), uc[k], um.p[k]);
            plain[k] = O::fma(O::mul(O::dup(p.dt2), cc.p[k]), F[k], O::mul(q, O::dup(T(-1))));
            un.p[k] = plain[k];
        }
        if (pml) {
            Pairs<T, NP> phx, phy, phz, nx_, ny_, nz_;
            ldp(phx, p.phx_in + sh + o);
            ldp(phy, p.phy_in + sh + o);
            const T f1 = AX == 0 ? __ldg(p.fcx + i) : AX == 1 ? __ldg(p.fcy + j) : T(0);
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                phz.p[k] = wz.at(C0 + 2 * k);
                const P S = AX == 2 ? O::mk(col.sz[2 * k], col.sz[2 * k + 1]) : O::dup(s1);
                const P a = O::mul(O::dup(p.dt), S), na = O::mul(a, O::dup(T(-1)));
                auto own = [&](P phi, P du) { return O::fma(na, du, O::fma(na, phi, phi)); };
                auto other = [&](P phi, P du) { return O::fma(a, du, phi); };
                nx_.p[k] = AX == 0 ? own(phx.p[k], dux[r][k]) : other(phx.p[k], dux[r][k]);
                ny_.p[k] = AX == 1 ? own(phy.p[k], duy[k]) : other(phy.p[k], duy[k]);
                nz_.p[k] = AX == 2 ? own(phz.p[k], duz[k]) : other(phz.p[k], duz[k]);
                const P fac1 = AX == 2 ? col.fz[k] : O::dup(f1);
                const P q = O::fma(O::dup(T(-2)), uc[k], um.p[k]);
                P fac2 = O::fma(q, O::dup(-p.idt2), O::mul(cc.p[k], F[k]));
                fac2 = O::fma(O::mul(S, um.p[k]), O::dup(p.i2dt), fac2);
                un.p[k] = O::mul(fac1, fac2);
                if (AX == 2) {  // cells of the vector outside the padding: the plain update, zero state
                    const bool p0 = col.sz[2 * k] != T(0), p1 = col.sz[2 * k + 1] != T(0);
                    auto sel = [&](P b, P c) { return O::mk(p0 ? O::lo(b) : O::lo(c), p1 ? O::hi(b) : O::hi(c)); };
                    un.p[k] = sel(un.p[k], plain[k]);
                    nx_.p[k] = sel(nx_.p[k], O::dup(T(0)));
                    ny_.p[k] = sel(ny_.p[k], O::dup(T(0)));
                    nz_.p[k] = sel(nz_.p[k], O::dup(T(0)));
                }
                if (ring) {
                    nx_.p[k] = mask(nx_.p[k], k);
                    ny_.p[k] = mask(ny_.p[k], k);
                    nz_.p[k] = mask(nz_.p[k], k);
                }
            }
            stp(p.phx_out + sh + o, nx_);
            stp(p.phy_out + sh + o, ny_);
            stp(p.phz_out + sh + o, nz_);
        }
        if (ring)
#pragma unroll
            for (int k = 0; k < NP; ++k) un.p[k] = mask(un.p[k], k);
        if (MODE == kAdj && inj_row) {
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                T t[2] = {O::lo(un.p[k]), O::hi(un.p[k])};
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    const int z = zl + 2 * k + v;
                    if (xok && z > 0 && z < p.nz - 1)
                        t[v] = ::fma(inject_fac(p, sx, AX == 1 ? col.sy : T(0), AX == 2 ? col.sz[2 * k + v] : T(0)) *
                                         (v ? O::hi(cc.p[k]) : O::lo(cc.p[k])), rh[2 * k + v], t[v]);
                }
                un.p[k] = O::mk(t[0], t[1]);
            }
        }
        stp(p.u_prev + sh + o, un);
        if (MODE == kRecomp && p.dw_out) {
            // dWaveOp = C^2 F + (sm - s)(u' - u_{k-1})/(2dt)
            const T m1 = AX == 0 ? __ldg(p.mgx + i) : col.my;
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                const P S = AX == 2 ? O::mk(col.sz[2 * k], col.sz[2 * k + 1]) : O::dup(s1);
                const P M = AX == 2 ? O::mk(col.mz[2 * k], col.mz[2 * k + 1]) : O::dup(m1);
                const P d = O::add(O::mul(cc.p[k], F[k]),
                                   O::mul(O::mul(O::sub(M, S), O::sub(un.p[k], um.p[k])), O::dup(p.i2dt)));
                dwo.p[k] = ring ? mask(d, k) : d;
            }
        }
        if (MODE == kAdj && p.image) {
#pragma unroll
            for (int k = 0; k < NP; ++k) ici.p[k] = O::fma(uc[k], dwi.p[k], ici.p[k]);
            stp(p.ic + sh + o, ici);
        }
        if (MODE == kRecomp && p.dw_out) stp_cs(p.dw_out + sh + o, dwo);
        if (MODE == kFwd || (MODE == kRecomp && p.nan_check))
#pragma unroll
            for (int k = 0; k < NP; ++k) chk.see(un.p[k]);
    }
}

#ifndef PGB_T3_MINB
#define PGB_T3_MINB 4  // resident 4-warp blocks per SM the FP32 register budget aims at (128 registers)
#endif
template <typename T, int R, int MODE, int RX>
__global__ void __launch_bounds__(kT3, (sizeof(T) == 4 ? PGB_T3_MINB : 1))
    wave3d_tile_kernel(const __grid_constant__ WaveParams<T> p, const Tile3d* __restrict__ tiles, int nint, int nshell,
                       int rec) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int V = V16<T>::N, NP = V / 2;
    using O = PairOps<T>;
    using P = typename O::P;
    const int shot = blockIdx.y + blockIdx.z * gridDim.y;
    int t = (int)blockIdx.x - rec;
    if (t < 0) {  // leading blocks record the traces of u_k, one pass per warp
        const long long nb = (long long)gridDim.y * gridDim.z;
        const long long pass = ((long long)blockIdx.x * nb + shot) * (blockDim.x / 32) + (threadIdx.x >> 5);
        pdl_handover();
        if (MODE != kAdj && pass < record_passes(p)) record_pass(p, pass);
        return;
    }
    if (shot >= p.nshot) return;
    t = t < nshell ? nint + t : t - nshell;  // the table holds the interior tiles first
    const int4 t0 = __ldg(reinterpret_cast<const int4*>(tiles + t)), t1 = __ldg(reinterpret_cast<const int4*>(tiles + t) + 1);
    const int x0 = t0.x, x1 = t0.y, y0 = t0.z, y1 = t0.w, zs = t1.x, ze = t1.y, kind = t1.z, inv = t1.w;
    const int nzv = (ze - zs + V - 1) / V, lane = threadIdx.x & 31;
    const int lr = (lane * inv) >> 16, rpw = (32 * inv) >> 16;  // the lane's row of the warp, rows per warp
    const int j = y0 + (threadIdx.x >> 5) * rpw + lr, zl = zs + (lane - lr * nzv) * V;
    InjBox ib{0, 0, 0, 0, 0, 0};
    T* rhs = reinterpret_cast<T*>(smem_raw);
    if (p.inj.on) {
        const int* bx = p.inj.box + shot * 6;
        const InjBox b{max(__ldg(bx), x0), min(__ldg(bx + 1), x1), max(__ldg(bx + 2), y0),
                       min(__ldg(bx + 3), y1), max(__ldg(bx + 4), zs), min(__ldg(bx + 5), ze)};
        if (b.x0 < b.x1 && b.y0 < b.y1 && b.z0 < b.z1) {
            ib = b;
            const int w = b.z1 - b.z0, h = (b.y1 - b.y0) * w, n = (b.x1 - b.x0) * h;
            for (int c = threadIdx.x; c < n; c += blockDim.x) {
                const int dx = c / h, e = c - dx * h, dy = e / w;
                rhs[c] = inject_rhs3(p.inj, bx, shot, b.x0 + dx, b.y0 + dy, b.z0 + e - dy * w);
            }
            __syncthreads();
        }
    }
    pdl_handover();
    if (lr >= rpw || j >= y1) return;
    const bool inj_col = ib.meets(j, zl, V);
    const long long sh = (long long)shot * p.fstride;
    const long long xs = (long long)p.rows_y * p.ldz;
    const long long oc = ((long long)(x0 + p.hx) * p.rows_y + (j + p.hy)) * p.ldz + kOZ + zl;
    FiniteCheck<T> chk;
    if (kind == 0) {
#pragma unroll 1
        for (int x = x0; x < x1; x += RX) {
            prefetch_planes<T, R, MODE, false, RX>(p, sh, oc + (long long)(x + RX - x0) * xs, x1 - x - RX);
            interior_planes<T, R, MODE, RX>(p, rhs, ib, inj_col, sh, oc + (long long)(x - x0) * xs, x, min(RX, x1 - x), j,
                                            zl, chk);
        }
    } else if (kind == 1) {
        general_update<T, R, MODE>(p, rhs, ib, shot, x0, x1, j, zl, ze, chk);
    } else {
        constexpr int RF = RX > 2 ? 2 : RX;
        FaceCol<T, NP> col;
        col.sy = __ldg(p.sgy + j);
        col.my = MODE == kRecomp ? __ldg(p.mgy + j) : T(0);
        col.zall = j > 0 && j < p.ny - 1;
        col.any_sz = false;
        bool any_pz = false, any_nearz = false;
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const int k = zl + v;
            const bool in = k < ze;
            col.sz[v] = in ? __ldg(p.sgz + k) : T(0);
            col.mz[v] = in && MODE == kRecomp ? __ldg(p.mgz + k) : T(0);
            col.zall &= k > 0 && k < p.nz - 1;
            col.any_sz |= col.sz[v] != T(0);
            any_pz |= in && (k < p.pzl || k >= p.nz - p.pzr);
            any_nearz |= in && (k - R < p.pzl || k + R >= p.nz - p.pzr);
        }
        const bool py = j < p.pyl || j >= p.ny - p.pyr, neary = j - R < p.pyl || j + R >= p.ny - p.pyr;
        col.need_xz = py || any_pz;
        col.need_yz = neary || any_pz;
        col.need_z = any_nearz || py;
#pragma unroll
        for (int k = 0; k < NP; ++k)
            col.fz[k] = O::mk(__ldg(p.fcz + min(zl + 2 * k, p.nz - 1)), __ldg(p.fcz + min(zl + 2 * k + 1, p.nz - 1)));
#define PGB_F(AX)                                                                                                       \
    _Pragma("unroll 1") for (int x = x0; x < x1; x += RF) {                                                             \
        prefetch_planes<T, R, MODE, true, RF>(p, sh, oc + (long long)(x + RF - x0) * xs, x1 - x - RF);                  \
        face_planes<T, R, MODE, RF, AX>(p, rhs, ib, inj_col, col, sh, oc + (long long)(x - x0) * xs, x,                 \
                                        min(RF, x1 - x), j, zl, chk);                                                   \
    }
        if (kind == 2) { PGB_F(0); }
        else if (kind == 3) { PGB_F(1); }
        else { PGB_F(2); }
#undef PGB_F
    }
    if (MODE != kAdj && p.err && chk.bad()) atomicOr(p.err, PGB_ERR_NONFINITE);
}

template <typename T, int R, int MODE, int RX>
void prep3_one() {
    cudaFuncSetAttribute(wave3d_tile_kernel<T, R, MODE, RX>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxInj3d);
}

}  // namespace

template <typename T, int R>
void wave3d_tile_prepare() {
    prep3_one<T, R, kFwd, 1>(); prep3_one<T, R, kRecomp, 1>(); prep3_one<T, R, kAdj, 1>();
    prep3_one<T, R, kFwd, 4>(); prep3_one<T, R, kRecomp, 4>(); prep3_one<T, R, kAdj, 4>();
}

template <typename T, int R, int MODE>
void launch_wave3d_tiles(const WaveParams<T>& p, const Tile3d* tiles, int nint, int nshell, int planes, int threads,
                         int inj_cap, cudaStream_t s) {
    const int gz = ceil_div(p.nshot, 65535), gy = ceil_div(p.nshot, gz);
    // recorder blocks: one pass per warp, the same number for every shot
    const long long passes = MODE != kAdj && p.rec.traces ? ((long long)p.nshot * p.rec.nrec * p.rec.lanes + 31) / 32 : 0;
    const int rec = ceil_div(passes, (long long)gy * gz * (threads / 32));
    const dim3 grid(rec + nint + nshell, gy, gz);
    const size_t smem = inj_cap * sizeof(T);
    if (planes == 1)
        launch_step(wave3d_tile_kernel<T, R, MODE, 1>, grid, dim3(threads), smem, s, p, tiles, nint, nshell, rec);
    else
        launch_step(wave3d_tile_kernel<T, R, MODE, 4>, grid, dim3(threads), smem, s, p, tiles, nint, nshell, rec);
}

#define PGB_INST3D(T, R, M) \
    template void launch_wave3d_tiles<T, R, M>(const WaveParams<T>&, const Tile3d*, int, int, int, int, int, cudaStream_t);
#define PGB_INSTANTIATE_3D(T, R)                                         \
    PGB_INST3D(T, R, kFwd) PGB_INST3D(T, R, kRecomp) PGB_INST3D(T, R, kAdj) \
    template void wave3d_tile_prepare<T, R>();

}  // namespace pgb
