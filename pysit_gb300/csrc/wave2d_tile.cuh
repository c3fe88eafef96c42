// Batched 2D leapfrog step: one block per tile of a shot's grid, one strip of rows per thread
// (forward, recompute, adjoint, Born scattered field).
//
// Same maths as the reference step cda_time_scalar_2D (pysit/solvers/
// constant_density_acoustic/time/scalar/constant_density_acoustic_time_scalar_2D.h:88-179)
// with the fusions of the batched pipeline:
//   kFwd    (with kRecomp and kBorn: leading blocks of the launch record the traces of u_k);
//   kRecomp the imaging operand dWaveOp_k (constant_density_acoustic_base.py:24-40)
//           from the stencil's own bracket F: C^2 F where the step and mesh
//           sigmas agree, plus the sigma differences elsewhere (the right PML,
//           whose step profile is read one node further out, _2D.h:143-157);
//   kAdj    the time-reversed adjoint step with ic += q_k * dWaveOp_k fused
//           (temporal_modeling.py:312-365);
//   kBorn   the scattered field u1 of linearised modelling, its source -m1 dWaveOp0_k
//           added inside the bracket (linear_forward_model, temporal_modeling.py:520-535).
//
// Work decomposition: a table of tiles (x0, rows, zs, cells, kind) covers the padded grid of one
// shot once; blockIdx.x is the tile (the PML-shell tiles, the longer ones, first), blockIdx.y/z
// the shot.  A thread updates RS consecutive x-rows of one vector along z; the 2R + RS rows of
// its column are loaded up front and serve all RS rows, the z-neighbours come as whole vectors
// per row.  Everything is read straight from global memory: the threads of a block share rows
// and vectors through L1, and a thread's loads are all independent, so four 4-warp blocks per SM
// (128 registers) keep the memory busy without shared-memory staging, barriers or waits.  What
// bounds a full launch is latency (16 warps per SM, long-scoreboard stalls first, issue slots 38-43 %,
// DRAM 41-53 %, L1 38-44 % busy); a block fetches the same tile of the next shot into L2, whose block
// starts about when it ends.
// The injection of a tile's cells (source taps; adjoint source at the receivers) is worked out
// by the whole block into shared memory before the update, in tiles that meet the shot's box.
// Tile kinds (block-uniform):
//   kind 0  interior: at least R cells away from the padding and off the outer
//           (Dirichlet) ring, no PML state, no masks;
//   kind 1  PML shell: the padding and its R-wide rim, Phi_x / Phi_z carried where both
//           sigmas vanish as in the reference;
//   kind 2  PML shell tiles without sigma_x (the z-bands): the update's sigma terms are
//           per-column constants.
// The arithmetic runs on cell pairs (packed f32x2 instructions in FP32).
// Measured against the persistent warps with shared-memory row rings this kernel replaces
// (us per step, before -> now): 1232 x 464 cells, order 8, FP32, 1 shot 33.9 -> 4.4, 16 shots
// 61 -> 43, 64 shots forward / recompute / adjoint 181 / 185 / 224 -> 157 / 166 / 222;
// 461 x 203, order 8, FP64, 6 shots 247 -> 60; 141 x 81, order 4, FP64, 1 shot 154 -> 5.5.
// Staging the tiles in shared memory with bulk copies was slower or equal at every size (64
// shots forward 159-178 us with four single-stage blocks per SM, 255-350 us with persistent
// blocks, two stages and a copying warp).
#pragma once
#include "pairs.cuh"
#include "tma.cuh"

namespace pgb {
namespace {

// One thread's strip of a tile: RS consecutive x-rows of one vector along z, operands read
// straight from global memory (L1 serves the rows and vectors that neighbouring threads share).
template <typename T, int R, int MODE, int RS, int KIND, bool INJ>
__device__ __forceinline__ void tile_update(const WaveParams<T>& p, const T* rhs, const int shot, const int x0,
                                            const int rows, const int zs, const int r0, const int q, const int4 ib,
                                            FiniteCheck<T>& chk) {
    using O = PairOps<T>;
    using P = typename O::P;
    constexpr bool PML = KIND != 0;
    constexpr int V = wave2d_cells(PML);
    constexpr int AL = V > V16<T>::N ? V : V16<T>::N, HZ = (R + AL - 1) / AL * AL, NB = HZ / V;
    constexpr int NP = V / 2, C0 = NB * V;
    constexpr bool DIFF = sizeof(T) == 8;  // FP64: derivatives over first differences (fewest FP64 instructions)
    const int zl = zs + q * V;
    const long long sh = (long long)shot * p.fstride;
    const bool img = MODE == kAdj && p.image;
    T sgz[V], mgz[V];
    bool zall = true;  // no cell of the thread on the outer ring or past the grid's end along z
#pragma unroll
    for (int v = 0; v < V; ++v) {
        const int z = zl + v;
        zall &= z > 0 && z < p.nz - 1;
        sgz[v] = (PML && z < p.nz) ? __ldg(p.sgz + z) : T(0);
        mgz[v] = (PML && MODE == kRecomp && z < p.nz) ? __ldg(p.mgz + z) : T(0);
    }
    P wx[R + 1], wz[R + 1], a1[R + 1];
#pragma unroll
    for (int k = 1; k <= R; ++k) {
        wx[k] = O::dup((DIFF ? T(c2sum(R, k - 1)) : T(d2w(R, k))) * p.idx2);
        wz[k] = O::dup((DIFF ? T(c2sum(R, k - 1)) : T(d2w(R, k))) * p.idz2);
        a1[k] = O::dup(T(d1w(R, k)));
    }
    const bool injz = INJ && zl < ib.w && zl + V > ib.z;  // the thread's cells meet the injection box along z
    const int ldz = p.ldz;
    const long long o0 = (long long)(x0 + r0 + kHalo) * ldz + kOZ + zl;  // the strip's first cell in a field
    const T* u = p.u_cur + sh + o0;
    // what the update of a column needs of sigma_z where sigma_x is zero
    P zdt[NP], zkx[NP], zkz[NP], zfac[NP], zsi[NP], zds[NP];
    if (KIND == 2) {
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            const P S = O::mk(sgz[2 * k], sgz[2 * k + 1]);
            zdt[k] = O::mul(O::dup(p.dt), S);
            zkx[k] = O::mul(zdt[k], O::dup(p.idx));
            zkz[k] = O::mul(O::sub(O::dup(T(0)), zdt[k]), O::dup(p.idz));
            zfac[k] = O::mk(__ldg(p.fcz + min(zl + 2 * k, p.nz - 1)), __ldg(p.fcz + min(zl + 2 * k + 1, p.nz - 1)));
            zsi[k] = O::mul(S, O::dup(p.i2dt));
            zds[k] = O::mul(O::sub(O::mk(mgz[2 * k], mgz[2 * k + 1]), S), O::dup(p.i2dt));
        }
    }
    T sxr[RS], mxr[RS];
    if (KIND == 1) {
#pragma unroll
        for (int r = 0; r < RS; ++r) {
            const int x = min(x0 + r0 + r, p.nx - 1);
            sxr[r] = __ldg(p.sgx + x);
            mxr[r] = MODE == kRecomp ? __ldg(p.mgx + x) : T(0);
        }
    }
    Pairs<T, NP> cv[RS + 2 * R], px[PML ? RS + 2 * R : 1], um[RS], cc[RS];
    // rows past the tile's last one are read too (the next rows of the field, or its halo:
    // clamped to the strip's last row that exists) and not used
#pragma unroll
    for (int j = 0; j < RS + 2 * R; ++j) ldp(cv[j], u + (long long)(min(j, rows - r0 + 2 * R - 1) - R) * ldz);
#pragma unroll
    for (int r = 0; r < RS; ++r) {
        const long long d = (long long)min(r, rows - r0 - 1) * ldz;
        ldp(um[r], p.u_prev + sh + o0 + d);
        ldr(cc[r], p.c2 + o0 + d);
    }
    if (PML) {
#pragma unroll
        for (int j = 0; j < RS + 2 * R; ++j)
            ldp(px[j], p.phx_in + sh + o0 + (long long)(min(j, rows - r0 + 2 * R - 1) - R) * ldz);
    }
    // Row r's neighbours along z and imaging operands.  A thread of one or two rows reads them all before
    // it stores the first (1232 x 464, FP32, one shot: 4.4 us a step, 4.7 row by row); one of four rows
    // reads them row by row (64 shots: 157 us, 161 with the next row's ahead of the stores), and so does
    // the FP64 adjoint step (461 x 203 x 40 shots: 369 us, 372 up front).
    constexpr bool FRONT = RS < 4 && !(sizeof(T) == 8 && MODE == kAdj);
    constexpr int NF = FRONT ? RS : 1;
    Window<T, NP, NB> wf[NF], wpf[NF];
    Pairs<T, NP> dwf[NF], icf[NF];
    auto fetch = [&](int r) {
        const int f = FRONT ? r : 0;
        const long long o = o0 + (long long)r * ldz;
        wf[f].load(u + (long long)r * ldz - HZ, &cv[R + r]);
        if ((MODE == kAdj && img) || MODE == kBorn) {  // for kBorn: dWaveOp0 and m1
            ldp(dwf[f], p.dw_in + sh + o);
            if (MODE == kBorn) ldr(icf[f], p.m1 + o);
            else ldp(icf[f], p.ic + sh + o);
        }
        if (PML) wpf[f].load(p.phz_in + sh + o - HZ, nullptr);
    };
    if (FRONT) {
#pragma unroll
        for (int r = 0; r < RS; ++r)
            if (r0 + r < rows) fetch(r);
    }
    {
#pragma unroll
        for (int r = 0; r < RS; ++r) {
            if (r0 + r >= rows) break;
            const int xr = x0 + r0 + r;
            const long long o = o0 + (long long)r * ldz;
            if (!FRONT) fetch(r);
            const auto &w = wf[FRONT ? r : 0], &wp = wpf[FRONT ? r : 0];
            const auto &dwi = dwf[FRONT ? r : 0], &ici = icf[FRONT ? r : 0];
            T sx = T(0), mgx = T(0);
            if (KIND == 1) {
                sx = sxr[r];
                mgx = mxr[r];
            }
            T rh[V];
            const bool inj_row = injz && xr >= ib.x && xr < ib.y;
            if (inj_row) {
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    const int z = zl + v;
                    rh[v] = z < ib.z || z >= ib.w ? T(0) : rhs[(xr - ib.x) * (ib.w - ib.z) + z - ib.z];
                }
            }
            // interior tiles never touch the outer (Dirichlet) ring: no masks there
            const bool ring = PML && !(zall && xr > 0 && xr < p.nx - 1);
            Pairs<T, NP> un, dwo, pxo, pzo, ico;
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                const int c = C0 + 2 * k;  // the pair's first cell in the window
                // first difference j of the column / of the window (FP64 path)
                auto ex = [&](int j) { return O::sub(cv[R + r + j + 1].p[k], cv[R + r + j].p[k]); };
                auto ez = [&](int j) { return O::sub(w.at(c + j + 1), w.at(c + j)); };
                const P uc = w.at(c);
                // Laplacian in difference form: sum_m w_m ((u_+m - u_0) + (u_-m - u_0)),
                // equal to the central stencil because the weights sum to zero, and free
                // of the large cancellation of w_0 u_0 (the FP32 path depends on this)
                // (x and z accumulate separately: two short dependency chains)
                P Fx = O::dup(T(0)), Fz = Fx;
                if (DIFF) {  // one chain: an FP64 addition less
#pragma unroll
                    for (int d = R; d >= 1; --d) Fz = O::fma(wx[d], O::sub(ex(d - 1), ex(-d)), Fz);
#pragma unroll
                    for (int d = R; d >= 1; --d) Fz = O::fma(wz[d], O::sub(ez(d - 1), ez(-d)), Fz);
                } else {
#pragma unroll
                    for (int d = 1; d <= R; ++d) {
                        Fx = O::fma(wx[d], O::add(O::sub(cv[R + r + d].p[k], uc), O::sub(cv[R + r - d].p[k], uc)), Fx);
                        Fz = w.d2(Fz, wz[d], c, d);
                    }
                }
                P F = DIFF ? Fz : O::add(Fx, Fz);
                if (MODE != kAdj && inj_row) F = O::add(F, O::mk(rh[2 * k], rh[2 * k + 1]));
                if (MODE == kBorn) F = O::sub(F, O::mul(ici.p[k], dwi.p[k]));  // rhs = -m1 dWaveOp0
                const P uo = um[r].p[k], c2 = cc[r].p[k];
                P unew, d;
                if (PML) {
                    P dpx = O::dup(T(0)), dpz = dpx, dx1 = dpx, dz1 = dpx;
#pragma unroll
                    for (int e = 1; e <= R; ++e) {
                        const P a = a1[e];
                        dpx = O::fma(a, O::sub(px[R + r + e].p[k], px[R + r - e].p[k]), dpx);
                        dpz = wp.d1(dpz, a, c, e);
                        dx1 = O::fma(a, O::sub(cv[R + r + e].p[k], cv[R + r - e].p[k]), dx1);
                        dz1 = w.d1(dz1, a, c, e);
                    }
                    F = O::add(F, O::fma(dpx, O::dup(p.idx), O::mul(dpz, O::dup(p.idz))));
                    // split-field PML update (_2D.h:157-170), branch-free: with both sigmas
                    // zero it reduces to the plain leapfrog update and carries Phi unchanged
                    const P phx = px[R + r].p[k], phz = wp.at(c), c2F = O::mul(c2, F);
                    if (KIND == 2) {  // the same with sigma_x zero, its terms left out
                        pxo.p[k] = O::fma(zkx[k], dx1, phx);
                        pzo.p[k] = O::fma(zkz[k], dz1, O::fma(zdt[k], O::mul(phz, O::dup(T(-1))), phz));
                        P fac2 = O::fma(O::fma(O::dup(T(-2)), uc, uo), O::dup(-p.idt2), c2F);
                        fac2 = O::fma(zsi[k], uo, fac2);
                        unew = O::mul(zfac[k], fac2);
                        if (MODE == kRecomp) d = O::fma(zds[k], O::sub(unew, uo), c2F);
                    } else {
                    const P szp = O::mk(sgz[2 * k], sgz[2 * k + 1]);
                    const P dsx = O::dup(p.dt * sx), dsz = O::mul(O::dup(p.dt), szp);
                    const P S = O::add(O::dup(sx), szp);  // sx + sz
                    // Phi' = Phi - dt s Phi + dt (s_other - s) du/dn
                    pxo.p[k] = O::fma(O::mul(O::sub(dsz, dsx), O::dup(p.idx)), dx1, O::fma(dsx, O::mul(phx, O::dup(T(-1))), phx));
                    pzo.p[k] = O::fma(O::mul(O::sub(dsx, dsz), O::dup(p.idz)), dz1, O::fma(dsz, O::mul(phz, O::dup(T(-1))), phz));
                    // u' = 2 dt^2 / (2 + dt S) * (C^2 F - (u_{k-1} - 2u)/dt^2 + S u_{k-1}/(2dt) - sx sz u)
                    const P den = O::fma(O::dup(p.dt), S, O::dup(T(2)));
                    const P fac1 = O::mul(O::dup(T(2) * p.dt2), O::mk(rcp_(O::lo(den)), rcp_(O::hi(den))));
                    P fac2 = O::fma(O::fma(O::dup(T(-2)), uc, uo), O::dup(-p.idt2), c2F);
                    fac2 = O::fma(O::mul(S, O::dup(p.i2dt)), uo, fac2);
                    fac2 = O::fma(O::mul(O::dup(-sx), szp), uc, fac2);
                    unew = O::mul(fac1, fac2);
                    if (MODE == kRecomp) {
                        // dWaveOp = C^2 F + (sm - s)(u' - u_{k-1})/(2dt) + (smx smz - sx sz) u
                        const P mzp = O::mk(mgz[2 * k], mgz[2 * k + 1]);
                        const P dS = O::sub(O::add(O::dup(mgx), mzp), S);
                        const P dP = O::sub(O::mul(O::dup(mgx), mzp), O::mul(O::dup(sx), szp));
                        d = O::fma(O::mul(dS, O::dup(p.i2dt)), O::sub(unew, uo), c2F);
                        d = O::fma(dP, uc, d);
                    }
                    }
                } else {
                    // u_{k+1} = dt^2 C^2 F - (u_{k-1} - 2 u_k)
                    const P qq = O::fma(O::dup(T(-2)), uc, uo);
                    unew = O::fma(O::mul(O::dup(p.dt2), c2), F, O::mul(qq, O::dup(T(-1))));
                    if (MODE == kRecomp) d = O::mul(c2, F);
                }
                if (MODE == kAdj && inj_row) {
                    // the adjoint source after the step: u' += fac C^2 rhs, fac = dt^2 or
                    // 2 dt^2 / (2 + dt (sx + sz)) where a sigma is nonzero (_2D.h:157-179, linear in rhs)
                    T t[2] = {O::lo(unew), O::hi(unew)};
#pragma unroll
                    for (int v = 0; v < 2; ++v) {
                        const T sz = sgz[2 * k + v];
                        const T fac = (sx != T(0) || sz != T(0)) ? T(2) * p.dt2 / (T(2) + p.dt * (sx + sz)) : p.dt2;
                        t[v] = ::fma(fac * (v ? O::hi(c2) : O::lo(c2)), rh[2 * k + v], t[v]);
                    }
                    unew = O::mk(t[0], t[1]);
                }
                un.p[k] = unew;
                if (MODE == kRecomp) dwo.p[k] = d;
                if (MODE == kAdj) ico.p[k] = O::fma(uc, dwi.p[k], ici.p[k]);
            }
            if (ring) {  // cells of the outer ring (or past the grid's end) get zero
                const bool xok = xr > 0 && xr < p.nx - 1;
#pragma unroll
                for (int k = 0; k < NP; ++k) {
                    const int z = zl + 2 * k;
                    const bool ok0 = xok && z > 0 && z < p.nz - 1, ok1 = xok && z + 1 < p.nz - 1;
                    auto mask = [&](P a) { return O::mk(ok0 ? O::lo(a) : T(0), ok1 ? O::hi(a) : T(0)); };
                    un.p[k] = mask(un.p[k]);
                    pxo.p[k] = mask(pxo.p[k]);
                    pzo.p[k] = mask(pzo.p[k]);
                    if (MODE == kRecomp) dwo.p[k] = mask(dwo.p[k]);
                }
            }
            if (MODE == kFwd || MODE == kBorn || (MODE == kRecomp && p.nan_check)) {
#pragma unroll
                for (int k = 0; k < NP; ++k) chk.see(un.p[k]);
            }
            stp(p.u_prev + sh + o, un);
            if (PML) {
                stp(p.phx_out + sh + o, pxo);
                stp(p.phz_out + sh + o, pzo);
            }
            if (MODE == kRecomp && p.dw_out) stp_cs(p.dw_out + sh + o, dwo);
            if (MODE == kAdj && img) stp(p.ic + sh + o, ico);
        }
    }
}

// test aid (WaveParams::wait_fault): a bounded wait on an mbarrier on which nothing ever arrives
// runs out; the block sets the plan's error word and leaves its tile undone
template <typename T>
__device__ __noinline__ bool waits_in_vain(const WaveParams<T>& p) {
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);  // one arrival expected, none ever made
    }
    __syncthreads();
    const bool ok = mbar_test_bounded(&bar, 0u, p.polls ? p.polls : 64u);
    if (!ok && threadIdx.x == 0 && p.err) atomicOr(p.err, PGB_ERR_TIMEOUT);
    return !ok;
}

#ifndef PGB_T2_MINB
#define PGB_T2_MINB 4  // resident blocks per SM the FP32 register budget aims at (128 registers)
#endif
template <typename T, int R, int MODE, int RS>
__global__ void __launch_bounds__(kT2, (sizeof(T) == 4 ? PGB_T2_MINB : 2))
    wave2d_tile_kernel(const __grid_constant__ WaveParams<T> p, const Tile2d* __restrict__ tiles, int nint, int nshell,
                       int rec) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    if (p.wait_fault && waits_in_vain(p)) return;
    const int shot = blockIdx.y + blockIdx.z * gridDim.y;
    int t = (int)blockIdx.x - rec;
    if (t < 0) {  // leading blocks record the traces of u_k, one pass per warp
        const long long n = (long long)gridDim.y * gridDim.z;
        const long long pass = ((long long)blockIdx.x * n + shot) * (blockDim.x / 32) + (threadIdx.x >> 5);
        pdl_handover();
        if (MODE != kAdj && pass < record_passes(p)) record_pass(p, pass);
        return;
    }
    if (shot >= p.nshot) return;
    t = t < nshell ? nint + t : t - nshell;  // the table holds the interior tiles first
    const int4 t0 = __ldg(reinterpret_cast<const int4*>(tiles + t)), t1 = __ldg(reinterpret_cast<const int4*>(tiles + t) + 1);
    const int x0 = t0.x, rows = t0.y, zs = t0.z, ncell = t0.w, nzv = t1.x, inv = t1.y;
    const int kind = t1.z;
    const bool pml = kind != 0;
    const int s0 = (threadIdx.x * inv) >> 16, q = threadIdx.x - s0 * nzv, r0 = s0 * RS;
    // the injection of the tile's cells
    int4 ib = make_int4(0, 0, 0, 0);
    T* rhs = reinterpret_cast<T*>(smem_raw);
    if (MODE != kBorn && p.inj.on) {
        const int* bx = p.inj.box + shot * 6;
        const int bx0 = max(__ldg(bx), x0), bx1 = min(__ldg(bx + 1), x0 + rows);
        const int bz0 = max(__ldg(bx + 4), zs), bz1 = min(__ldg(bx + 5), zs + ncell);
        if (bx0 < bx1 && bz0 < bz1) {
            ib = make_int4(bx0, bx1, bz0, bz1);
            const int w = bz1 - bz0, n = (bx1 - bx0) * w;
            for (int c = threadIdx.x; c < n; c += blockDim.x) {
                const int dx = c / w;
                rhs[c] = inject_rhs(p.inj, bx, shot, bx0 + dx, bz0 + c - dx * w);
            }
            __syncthreads();
        }
    }
    pdl_handover();
    // fetch the same tile of the next shot into L2: its block starts about when this one ends
    if (p.pf_next && shot + 1 < p.nshot) {
        const long long org = (long long)(shot + 1) * p.fstride + (long long)(x0 + kHalo) * p.ldz + kOZ + zs;
        const uint32_t bytes = (uint32_t)((ncell * (int)sizeof(T) + 15) / 16 * 16);
        auto rows_of = [&](const T* b) {
            for (int r = threadIdx.x & 31; r < rows; r += 32) prefetch_l2(b + org + (long long)r * p.ldz, bytes);
        };
        const int w = threadIdx.x >> 5;
        if (w == 0) rows_of(p.u_prev);
        if (w == 1) rows_of(p.u_cur);
        if (pml && w == 2) rows_of(p.phx_in);
        if (pml && w == 3) rows_of(p.phz_in);
        if ((MODE == kAdj && p.image) || MODE == kBorn) {
            if (w == 2) rows_of(p.dw_in);
            if (MODE == kAdj && w == 3) rows_of(p.ic);
        }
    }
    if (r0 >= rows || s0 >= ((int)(blockDim.x * inv) >> 16)) return;
    FiniteCheck<T> chk;
    // (the injection is looked at row by row only in tiles that meet the box)
    const bool inj = ib.y > ib.x;
#define PGB_U(KIND)                                                                                     \
    if (MODE != kBorn && inj)                                                                           \
        tile_update<T, R, MODE, RS, KIND, MODE != kBorn>(p, rhs, shot, x0, rows, zs, r0, q, ib, chk);   \
    else                                                                                                \
        tile_update<T, R, MODE, RS, KIND, false>(p, rhs, shot, x0, rows, zs, r0, q, ib, chk);
    if (kind == 0) { PGB_U(0) }
    else if (kind == 2) { PGB_U(2) }
    else { PGB_U(1) }
#undef PGB_U
    if (MODE != kAdj && p.err && chk.bad()) atomicOr(p.err, PGB_ERR_NONFINITE);
}

}  // namespace

template <typename T, int R, int MODE>
void launch_wave2d_tiles(const WaveParams<T>& p, const Tile2d* tiles, int nint, int nshell, int strip, int threads,
                         int inj_cap, cudaStream_t s) {
    const int gz = ceil_div(p.nshot, 65535), gy = ceil_div(p.nshot, gz);
    // recorder blocks: one pass per warp, the same number for every shot
    const long long passes = MODE != kAdj && p.rec.traces ? ((long long)p.nshot * p.rec.nrec * p.rec.lanes + 31) / 32 : 0;
    const int rec = ceil_div(passes, (long long)gy * gz * (threads / 32));
    const dim3 grid(rec + nint + nshell, gy, gz);
    const size_t smem = inj_cap * sizeof(T);
#define PGB_G(RS) launch_step(wave2d_tile_kernel<T, R, MODE, RS>, grid, dim3(threads), smem, s, p, tiles, nint, nshell, rec)
    switch (strip) {
        case 1: PGB_G(1); break;
        case 2: PGB_G(2); break;
        default: PGB_G(sizeof(T) == 4 ? 4 : 2); break;
    }
#undef PGB_G
}

#define PGB_INST2D(T, R, M) \
    template void launch_wave2d_tiles<T, R, M>(const WaveParams<T>&, const Tile2d*, int, int, int, int, int, cudaStream_t);
#define PGB_INSTANTIATE_2D(T, R) PGB_INST2D(T, R, kFwd) PGB_INST2D(T, R, kRecomp) PGB_INST2D(T, R, kAdj) PGB_INST2D(T, R, kBorn)

}  // namespace pgb
