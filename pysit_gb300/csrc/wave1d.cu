// Batched 1D leapfrog step (forward, recompute, adjoint modes) on the internal zero-halo layout
// of wave.cuh, for cda_time_scalar_1D (pysit/solvers/constant_density_acoustic/time/scalar/
// constant_density_acoustic_time_scalar_1D.h:78-130).
//
// A whole run of steps is one launch: a cluster of up to sixteen blocks per shot holds the shot's
// wavefields in shared memory, a block's cells one thread each (or a few), and meets once per step
// at the cluster barrier after writing the cells its neighbours' stencils reach into their halos.
// Checkpoints, traces, dWaveOp and the image go to and come from global memory as the steps pass.
// What bounds a step: in FP64 the few FP64 units of the cluster's SMs, then the barrier.  Measured
// against one launch per step of one thread per cell (800 steps of 799 cells, order 4, FP64, whole
// gradient call): 6.4 -> 4.0 ms.  Grids too long for a cluster and launches that fill the GPU
// (wave1d_sweeps) step as before, one launch each.
#include <cooperative_groups.h>

#include <algorithm>

#include "wave.cuh"

namespace pgb {
namespace {

template <typename T>
__device__ __forceinline__ void record3(const WaveParams<T>& p, long long id) {
    long long total = (long long)p.nshot * p.rec.nrec;
    if (id >= total) return;
    int shot = (int)(id / p.rec.nrec), r = (int)(id - (long long)shot * p.rec.nrec);
    int e0 = __ldg(p.rec.rowptr + id), e1 = __ldg(p.rec.rowptr + id + 1);
    const T* u = p.u_cur + (long long)shot * p.fstride;
    T acc = T(0);
    for (int e = e0; e < e1; ++e) acc += __ldg(p.rec.w + e) * u[__ldg(p.rec.off + e)];
    p.rec.traces[shot * p.rec.tr_sstride + r] = acc;
}

// derivative taps around v (a cell's address) along a 32-bit stride s (a field of one
// shot has fewer than 2^31 elements): first derivative sum_m a_m (v_+m - v_-m) ...
template <typename T, int R>
__device__ __forceinline__ T dd1(const T* __restrict__ v, int s) {
    T a = T(0);
#pragma unroll
    for (int m = 1; m <= R; ++m) a += T(d1w(R, m)) * (v[m * s] - v[-m * s]);
    return a;
}
// ... and second derivative in difference form: sum_m w_m ((v_+m - v_0) + (v_-m - v_0)),
// equal to the central stencil (the weights sum to zero) with far less FP32
// cancellation than w_0 v_0 + sum_m w_m (v_+m + v_-m)
template <typename T, int R>
__device__ __forceinline__ T dd2(const T* __restrict__ v, int s) {
    const T c = v[0];
    T a = T(0);
#pragma unroll
    for (int m = 1; m <= R; ++m) a += T(d2w(R, m)) * ((v[m * s] - c) + (v[-m * s] - c));
    return a;
}

// 1D: one axis (z), Phi_z only (_1D.h:117-129).
template <typename T, int R, int MODE>
__global__ void __launch_bounds__(256) wave1d_kernel(const WaveParams<T> p, int ntile) {
    const int b = blockIdx.x;
    if (b >= ntile * p.nshot) {
        if (MODE != kAdj) record3(p, (long long)(b - ntile * p.nshot) * blockDim.x + threadIdx.x);
        return;
    }
    const int shot = b / ntile;
    const int k = (b - shot * ntile) * blockDim.x + threadIdx.x;
    if (k >= p.nz) return;
    const long long sh = (long long)shot * p.fstride;
    const long long o = kOZ + k;
    const T* __restrict__ u = p.u_cur + sh;
    const bool ok = k > 0 && k < p.nz - 1;
    const T sz = __ldg(p.sgz + k);
    const T uc = u[o], uo = p.u_prev[sh + o], c2 = __ldg(p.c2 + o);
    T F = dd2<T, R>(u + o, 1) * p.idz2 + dd1<T, R>(p.phz_in + sh + o, 1) * p.idz;
    const int* bx = p.inj.box + shot * 6;
    if (p.inj.on) F += inject_rhs3(p.inj, bx, shot, 0, 0, k);
    T unew;
    if (sz != T(0)) {
        const T dudz = dd1<T, R>(u + o, 1) * p.idz;
        const T phz = p.phz_in[sh + o];
        T nz_ = phz - p.dt * sz * (phz + dudz);
        const T fac1 = T(2) * p.dt2 / (T(2) + p.dt * sz);
        const T fac2 = c2 * F - (uo - T(2) * uc) * p.idt2 + sz * uo * p.i2dt;
        unew = fac1 * fac2;
        if (!ok) { unew = T(0); nz_ = T(0); }
        p.phz_out[sh + o] = nz_;
    } else {
        unew = p.dt2 * c2 * F - (uo - T(2) * uc);
        if (!ok) unew = T(0);
    }
    p.u_prev[sh + o] = unew;
    if (MODE == kRecomp && p.dw_out) {
        const T mz = __ldg(p.mgz + k);
        T d = c2 * F + (mz - sz) * (unew - uo) * p.i2dt;
        __stcs(p.dw_out + sh + o, ok ? d : T(0));
    }
    if (MODE == kAdj && p.image) p.ic[sh + o] += uc * __ldcs(p.dw_in + sh + o);
}

// ---- many steps in one launch ---------------------------------------------------------
namespace cg = cooperative_groups;
constexpr int kH1 = 4;       // halo cells on either side of a block's cells
constexpr int kThreads1 = 512;  // threads of a block at most
constexpr int kAmpSteps = 16;  // steps whose injection amplitudes are staged at once

// shared memory of a block: u x 2, Phi_z x 2 (with halos); C^2, sigmas, factor, image; amplitudes;
// the injection entries of its cells
template <typename T>
size_t sweep1d_smem(int cells, int npts) {
    return sizeof(T) * (4 * (size_t)(cells + 2 * kH1) + 5 * (size_t)cells + (size_t)kAmpSteps * npts) + 2 * sizeof(int) * (size_t)cells;
}

template <typename T, int R, int MODE>
__global__ void __launch_bounds__(kThreads1) wave1d_sweep_kernel(const WaveParams<T> p, const Sweep1d<T> q) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cg::cluster_group cl = cg::this_cluster();
    const int rank = cl.block_rank(), nc = cl.num_blocks();
    const int shot = blockIdx.x / nc;
    const int a = rank * q.cells, n = min(q.cells, p.nz - a);  // the block's cells a .. a+n-1
    const int w = q.cells + 2 * kH1, tid = threadIdx.x, nt = q.threads;  // nt threads step cells, the warps after them record
    const int rw = (tid - nt) >> 5, nrw = (blockDim.x - nt) >> 5;
    // u and Phi_z, each twice, w apart: `cur` (0 or w) is the offset of u_k and Phi_k, w - cur that of
    // u_{k-1} -> u_{k+1} and Phi_{k+1}
    T* const us = reinterpret_cast<T*>(smem_raw) + kH1;
    T* const ps = us + 2 * w;
    T* c2 = us + 4 * w - kH1;
    T *sg = c2 + q.cells, *mg = sg + q.cells, *fc = mg + q.cells, *ic = fc + q.cells, *amp = ic + q.cells;
    int* e0 = reinterpret_cast<int*>(amp + kAmpSteps * q.npts);
    int* e1 = e0 + q.cells;
    const long long sh = (long long)shot * p.fstride + kOZ;
    const int* bx = p.inj.box + shot * 6;
    // the state with its halos (zero beyond the grid: the fields' own zero halos)
    for (int j = tid - kH1; j < n + kH1; j += blockDim.x) {
        us[j] = q.in_cur[sh + a + j];
        us[w + j] = j >= 0 && j < n ? q.in_prev[sh + a + j] : T(0);
        ps[j] = q.in_phz[sh + a + j];
        ps[w + j] = T(0);
    }
    for (int j = tid; j < n; j += blockDim.x) {
        const int k = a + j;
        c2[j] = p.c2[kOZ + k];
        sg[j] = p.sgz[k];
        mg[j] = p.mgz[k];
        fc[j] = p.fcz[k];
        ic[j] = MODE == kAdj ? p.ic[sh + k] : T(0);
        const bool in = p.inj.on && bx[0] <= 0 && bx[1] > 0 && k >= bx[4] && k < bx[5];
        const int* rp = p.inj.rowptr + (in ? p.inj.rpbase[shot] + k - bx[4] : 0);
        e0[j] = in ? rp[0] : 0;
        e1[j] = in ? rp[1] : 0;
    }
    // the neighbours' halos: cells j < R go to the left block's right halo, cells j >= n-R to the right's left
    const int nl = q.cells;  // cells of the left neighbour (only the last block may have fewer)
    T* left = rank > 0 ? cl.map_shared_rank(us, rank - 1) : nullptr;
    T* right = rank + 1 < nc ? cl.map_shared_rank(us, rank + 1) : nullptr;
    const bool ahead = MODE == kAdj && q.dw && n <= nt && tid < n;
    T dw_next = ahead && q.k0 % q.dw_period == 0
                    ? __ldcs(q.dw + (long long)((q.k0 - q.dw_k0) / q.dw_div) * q.field_stride + sh + a + tid) : T(0);
    cl.sync();
    int cur = 0;
    for (int i = 0; i < q.n; ++i) {
        const int k = q.k0 + q.dir * i;
        const T *uk = us + cur, *pk = ps + cur;
        T *un = us + (w - cur), *pn = ps + (w - cur);
        if (p.inj.on && i % kAmpSteps == 0) {  // the amplitudes of the next steps
            const T* src = p.inj.amp + (long long)shot * p.inj.amp_sstride;
            const int m = min(kAmpSteps, q.n - i) * q.npts;
            for (int c = tid; c < m; c += blockDim.x) {
                const int r = c / q.npts;
                amp[c] = src[(long long)(k + q.dir * r) * q.npts + c - r * q.npts];
            }
            __syncthreads();
        }
        const T* am = amp + (i % kAmpSteps) * q.npts;
        if (MODE == kFwd && q.ckpt && k % q.S == 0) {  // the step's inputs: u_{k-1}, u_k, Phi_z
            T* c = q.ckpt + (long long)(k / q.S) * 3 * q.field_stride + sh + a;
            for (int j = tid; j < n && rw < 0; j += nt) {
                c[j] = un[j];
                c[q.field_stride + j] = uk[j];
                c[2 * q.field_stride + j] = pk[j];
            }
        }
        if (MODE != kAdj && rw >= 0 && q.traces) {
            // traces of u_k, each in the order of its taps, read from the block that holds their cell
            auto sample = [&](int e, T& wt, T& v) {
                const int cell = (int)(__ldg(p.rec.off + e) - kOZ), b = __umulhi(cell, q.inv);
                wt = __ldg(p.rec.w + e);
                const T* ub = b == rank ? us : cl.map_shared_rank(us, b);
                v = ub[cur + cell - b * q.cells];
            };
            T* out = q.traces + (long long)shot * p.rec.tr_sstride + (long long)k * p.rec.nrec;
            const int* row = p.rec.rowptr + (long long)shot * p.rec.nrec;
            if (p.rec.nrec <= 4 * nc) {  // a warp per receiver: the lanes fetch its taps
                const int r = rank + nc * rw, lane = tid & 31;
                if (r < p.rec.nrec) {
                    const int e1r = __ldg(row + r + 1);
                    T acc = T(0);
                    for (int e = __ldg(row + r); e < e1r; e += 32) {
                        const int m = min(32, e1r - e);
                        T wt = T(0), v = T(0);
                        if (lane < m) sample(e + lane, wt, v);
                        for (int t = 0; t < m; ++t)
                            acc += __shfl_sync(0xffffffffu, wt, t) * __shfl_sync(0xffffffffu, v, t);
                    }
                    if (lane == 0) out[r] = acc;
                }
            } else {  // a thread per receiver, neighbouring receivers in one block
                const int per = (p.rec.nrec + nc - 1) / nc, rend = min(p.rec.nrec, (rank + 1) * per);
                for (int r = rank * per + tid - nt; r < rend; r += 32 * nrw) {
                    const int e1r = __ldg(row + r + 1);
                    T acc = T(0);
                    for (int e = __ldg(row + r); e < e1r; e += 8) {  // eight taps in flight
                        T wt[8], v[8];
#pragma unroll
                        for (int t = 0; t < 8; ++t) {
                            wt[t] = v[t] = T(0);
                            if (e + t < e1r) sample(e + t, wt[t], v[t]);
                        }
#pragma unroll
                        for (int t = 0; t < 8; ++t)
                            if (e + t < e1r) acc += wt[t] * v[t];
                    }
                    out[r] = acc;
                }
            }
        }
        const bool img = q.dw && k % q.dw_period == 0;
        const long long slot = img ? (long long)((k - q.dw_k0) / q.dw_div) * q.field_stride + sh + a : 0;
        // dWaveOp of the next imaged step, on its way while this one computes (one cell per thread)
        T dw_after = T(0);
        if (MODE == kAdj && ahead && i + 1 < q.n && (k - 1) % q.dw_period == 0)
            dw_after = __ldcs(q.dw + (long long)((k - 1 - q.dw_k0) / q.dw_div) * q.field_stride + sh + a + tid);
        for (int j = tid; j < n && rw < 0; j += nt) {
            const int c = a + j;
            const T dw = MODE == kAdj && img ? (ahead ? dw_next : __ldcs(q.dw + slot + j)) : T(0);
            const bool ok = c > 0 && c < p.nz - 1;
            const T sz = sg[j], uc = uk[j], uo = un[j], cc = c2[j];
            // Phi_z is zero outside the padding
            const bool near = c - R < p.pzl || c + R >= p.nz - p.pzr;
            T F = dd2<T, R>(uk + j, 1) * p.idz2 + (near ? dd1<T, R>(pk + j, 1) : T(0)) * p.idz;
            if (e1[j] > e0[j]) {
                T acc = T(0);
                for (int e = e0[j]; e < e1[j]; ++e) acc += __ldg(p.inj.w + e) * am[__ldg(p.inj.pt + e)];
                F += acc;
            }
            T unew, pnew = T(0);
            if (sz != T(0)) {
                const T dudz = dd1<T, R>(uk + j, 1) * p.idz;
                const T phz = pk[j];
                pnew = phz - p.dt * sz * (phz + dudz);
                const T fac2 = cc * F - (uo - T(2) * uc) * p.idt2 + sz * uo * p.i2dt;
                unew = fc[j] * fac2;
                if (!ok) { unew = T(0); pnew = T(0); }
            } else {
                unew = p.dt2 * cc * F - (uo - T(2) * uc);
                if (!ok) unew = T(0);
            }
            un[j] = unew;
            pn[j] = pnew;
            const int at = w - cur + j, pt = at + 2 * w;
            if (left && j < R) {
                left[at + nl] = unew;
                left[pt + nl] = pnew;
            }
            if (right && j >= n - R) {
                right[at - n] = unew;
                right[pt - n] = pnew;
            }
            if (MODE == kRecomp && img) {
                const T d = cc * F + (mg[j] - sz) * (unew - uo) * p.i2dt;
                __stcs(q.dw + slot + j, ok ? d : T(0));
            }
            if (MODE == kAdj && img) ic[j] += uc * dw;
        }
        cl.sync();  // the new fields and halos are complete, the old ones free
        cur = w - cur;
        dw_next = dw_after;
    }
    for (int j = tid; j < n; j += blockDim.x) {
        q.out_cur[sh + a + j] = us[cur + j];
        q.out_prev[sh + a + j] = us[w - cur + j];
        q.out_phz[sh + a + j] = ps[cur + j];
        if (MODE == kAdj) p.ic[sh + a + j] = ic[j];
    }
}

struct SweepShape {
    int nc, cells, threads;  // blocks per shot (0: none fits), cells per block, threads that step them
};
// the shape for a grid of nz cells, at most npts points and clusters of at most `most_nc` blocks
template <typename T>
SweepShape sweep1d_shape(int nz, int npts, int most_nc) {
    // a block's cells: in FP64 as few as give a few warps (the FP64 units bound the step: 2.4 us a step at
    // 100 cells a block, 3.5 at 250, where a launch per step takes 3.0), with sixteen blocks where eight
    // would hold more than 128 each; in FP32 a block's threads (1.5 us a step from 150 to 2000 cells);
    // more blocks for more receivers than a block's recording threads take at once
    const int want = sizeof(T) == 8 ? 64 : 512, most = sizeof(T) == 8 ? 160 : 2048;
    const int lim = std::min(most_nc, sizeof(T) == 8 && nz > 8 * 128 ? 16 : 8);
    SweepShape h{std::min({lim, std::max(ceil_div(nz, want), ceil_div(npts, 128)), ceil_div(nz, kH1)}), 0, 0};
    if (h.nc < 1) return SweepShape{};
    for (;; --h.nc) {
        h.cells = ceil_div(nz, h.nc);
        if (h.nc == 1 || nz - (h.nc - 1) * h.cells >= kH1) break;  // the last block feeds its neighbour's halo
    }
    h.threads = std::min(kThreads1 - 128, (h.cells + 31) / 32 * 32);
    if (h.cells > most || sweep1d_smem<T>(h.cells, npts) > 200 * 1024) return SweepShape{};
    return h;
}
// recording threads of a block: a warp per receiver for a few, else a thread per receiver
inline int sweep1d_recorders(const SweepShape& h, int nrec) {
    if (nrec <= 4 * h.nc) return 32 * ceil_div(nrec, h.nc);
    return std::min(kThreads1 - h.threads, (ceil_div(nrec, h.nc) + 31) / 32 * 32);
}

// launch configuration of a run (`attr`: room for its cluster attribute)
template <typename T>
cudaLaunchConfig_t sweep1d_config(const SweepShape& h, int nshot, int npts, int recorders, cudaLaunchAttribute* attr) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(h.nc * nshot);
    cfg.blockDim = dim3(h.threads + recorders);
    cfg.dynamicSmemBytes = sweep1d_smem<T>(h.cells, npts);
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim = {(unsigned)h.nc, 1, 1};
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

// whether the device places a cluster of the shape in one mode; sets the kernel's attributes
template <typename T, int R, int MODE>
bool sweep1d_placed(const SweepShape& h, int npts, int recorders) {
    if (sweep1d_smem<T>(h.cells, npts) > 48 * 1024 &&
        cudaFuncSetAttribute(wave1d_sweep_kernel<T, R, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024))
        return false;
    if (h.nc > 8 && cudaFuncSetAttribute(wave1d_sweep_kernel<T, R, MODE>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1))
        return false;
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = sweep1d_config<T>(h, 1, npts, recorders, &attr);
    int n = 0;
    return cudaOccupancyMaxActiveClusters(&n, wave1d_sweep_kernel<T, R, MODE>, &cfg) == cudaSuccess && n > 0;
}

}  // namespace

// Large launches step faster with a launch per step, whose blocks share the whole GPU: a run's blocks meet
// every step, and each reads the amplitudes of all receivers.  Measured against a launch per step (us a
// step of the whole gradient call): FP64 799 cells x 64 shots (65536 threads) 13.0 against 13.1, 96 shots
// 18.0 against 16.9, 32 shots 8.2 against 10.9; FP32 1520 x 96 (110592 threads) 6.9 against 8.0, 2220 x 64
// (122880) 8.3 against 7.8.  Receivers: FP64 799 x 32 shots x 400 (102400 of them times blocks) 9.3
// against 12.0, 64 shots (204800) 19.1 against 15.1; FP32 799 x 96 x 400 (153600) 7.2 against 8.4, 128
// shots (204800) 10.3 against 8.9.
template <typename T>
bool wave1d_sweeps(int nz, int nsrc, int nrec, int nshot) {
    const SweepShape h = sweep1d_shape<T>(nz, std::max(nsrc, nrec), 16);
    const long long blocks = (long long)h.nc * nshot;
    return h.nc > 0 && blocks * h.threads <= (sizeof(T) == 8 ? 65536 : 152 * 768) &&
           blocks * nrec <= (sizeof(T) == 8 ? 120000 : 180000);
}

template <typename T, int R>
int wave1d_prepare(int nz, int nsrc, int nrec) {
    for (int most_nc : {16, 8}) {
        const SweepShape h = sweep1d_shape<T>(nz, std::max(nsrc, nrec), most_nc);
        if (h.nc > 0 && sweep1d_placed<T, R, kFwd>(h, nsrc, sweep1d_recorders(h, nrec)) &&
            sweep1d_placed<T, R, kRecomp>(h, nsrc, sweep1d_recorders(h, nrec)) && sweep1d_placed<T, R, kAdj>(h, nrec, 0))
            return most_nc;
        cudaGetLastError();  // an attribute or shape that the device refuses is no error of the plan
    }
    return 0;
}

template <typename T, int R, int MODE>
void launch_wave1d_sweep(const WaveParams<T>& p, Sweep1d<T> q, cudaStream_t s) {
    const SweepShape h = sweep1d_shape<T>(p.nz, q.npts_max, q.most_nc);
    if (!p.inj.on) q.npts = 0;
    q.cells = h.cells;
    q.threads = h.threads;
    q.inv = 0xffffffffu / (unsigned)q.cells + 1;
    cudaLaunchAttribute attr;
    cudaLaunchConfig_t cfg =
        sweep1d_config<T>(h, p.nshot, q.npts, MODE != kAdj && q.traces ? sweep1d_recorders(h, p.rec.nrec) : 0, &attr);
    cfg.stream = s;
    cudaLaunchKernelEx(&cfg, wave1d_sweep_kernel<T, R, MODE>, p, q);
}

template <typename T, int R, int MODE>
void launch_wave1d(const WaveParams<T>& p, cudaStream_t s) {
    const int tb = 128;
    int ntile = ceil_div(p.nz, tb);
    int grid = ntile * p.nshot;
    if (MODE != kAdj && p.rec.nrec > 0 && p.rec.traces) grid += ceil_div((long long)p.nshot * p.rec.nrec, tb);
    wave1d_kernel<T, R, MODE><<<grid, tb, 0, s>>>(p, ntile);
}

template bool wave1d_sweeps<float>(int, int, int, int);
template bool wave1d_sweeps<double>(int, int, int, int);
#define PGB_INST1(T, R)                                                                  \
    template int wave1d_prepare<T, R>(int, int, int);                                                 \
    template void launch_wave1d_sweep<T, R, kFwd>(const WaveParams<T>&, Sweep1d<T>, cudaStream_t);    \
    template void launch_wave1d_sweep<T, R, kRecomp>(const WaveParams<T>&, Sweep1d<T>, cudaStream_t); \
    template void launch_wave1d_sweep<T, R, kAdj>(const WaveParams<T>&, Sweep1d<T>, cudaStream_t);    \
    template void launch_wave1d<T, R, kFwd>(const WaveParams<T>&, cudaStream_t);    \
    template void launch_wave1d<T, R, kRecomp>(const WaveParams<T>&, cudaStream_t); \
    template void launch_wave1d<T, R, kAdj>(const WaveParams<T>&, cudaStream_t);
PGB_INST1(float, 1)
PGB_INST1(float, 2)
PGB_INST1(float, 3)
PGB_INST1(float, 4)
PGB_INST1(double, 1)
PGB_INST1(double, 2)
PGB_INST1(double, 3)
PGB_INST1(double, 4)

}  // namespace pgb
