// Batched 1D leapfrog step (forward, recompute, adjoint modes) on the internal zero-halo layout
// of wave.cuh, for cda_time_scalar_1D (pysit/solvers/constant_density_acoustic/time/scalar/
// constant_density_acoustic_time_scalar_1D.h:78-130): one thread per cell.
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

}  // namespace

template <typename T, int R, int MODE>
void launch_wave1d(const WaveParams<T>& p, int bz, cudaStream_t s) {
    (void)bz;
    const int tb = 128;
    int ntile = ceil_div(p.nz, tb);
    int grid = ntile * p.nshot;
    if (MODE != kAdj && p.rec.nrec > 0 && p.rec.traces) grid += ceil_div((long long)p.nshot * p.rec.nrec, tb);
    wave1d_kernel<T, R, MODE><<<grid, tb, 0, s>>>(p, ntile);
}

#define PGB_INST1(T, R)                                                                  \
    template void launch_wave1d<T, R, kFwd>(const WaveParams<T>&, int, cudaStream_t);    \
    template void launch_wave1d<T, R, kRecomp>(const WaveParams<T>&, int, cudaStream_t); \
    template void launch_wave1d<T, R, kAdj>(const WaveParams<T>&, int, cudaStream_t);
PGB_INST1(float, 1)
PGB_INST1(float, 2)
PGB_INST1(float, 3)
PGB_INST1(float, 4)
PGB_INST1(double, 1)
PGB_INST1(double, 2)
PGB_INST1(double, 3)
PGB_INST1(double, 4)

}  // namespace pgb
