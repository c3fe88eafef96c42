// Pairs of neighbouring cells in registers, their vectors and z-windows, and the derivative
// weights of the step kernels' tiles.
#pragma once
#include "wave.cuh"

namespace pgb {
namespace {

// Pair arithmetic: two neighbouring cells per operation.  FP32 uses the packed f32x2
// instructions on 64-bit registers (one issue slot for two cells, each half rounded exactly
// like the scalar operation; the pairs stay packed from load to store, since taking them
// apart costs as many moves as the arithmetic saves); FP64 spells the pair out.
template <typename T> struct PairOps;
template <> struct PairOps<float> {
    using P = unsigned long long;
    static __device__ __forceinline__ P mk(float a, float b) {
        P d;
        asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
        return d;
    }
    static __device__ __forceinline__ float lo(P a) { return __uint_as_float((unsigned)a); }
    static __device__ __forceinline__ float hi(P a) { return __uint_as_float((unsigned)(a >> 32)); }
    static __device__ __forceinline__ P dup(float a) { return mk(a, a); }
    static __device__ __forceinline__ P add(P a, P b) {
        P d;
        asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
        return d;
    }
    static __device__ __forceinline__ P sub(P a, P b) {
        P d;
        asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
        return d;
    }
    static __device__ __forceinline__ P mul(P a, P b) {
        P d;
        asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
        return d;
    }
    static __device__ __forceinline__ P fma(P a, P b, P c) {
        P d;
        asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
        return d;
    }
};
template <> struct PairOps<double> {
    using P = double2;
    static __device__ __forceinline__ P mk(double a, double b) { return make_double2(a, b); }
    static __device__ __forceinline__ double lo(P a) { return a.x; }
    static __device__ __forceinline__ double hi(P a) { return a.y; }
    static __device__ __forceinline__ P dup(double a) { return make_double2(a, a); }
    static __device__ __forceinline__ P add(P a, P b) { return make_double2(a.x + b.x, a.y + b.y); }
    static __device__ __forceinline__ P sub(P a, P b) { return make_double2(a.x - b.x, a.y - b.y); }
    static __device__ __forceinline__ P mul(P a, P b) { return make_double2(a.x * b.x, a.y * b.y); }
    static __device__ __forceinline__ P fma(P a, P b, P c) {
        return make_double2(::fma(a.x, b.x, c.x), ::fma(a.y, b.y, c.y));
    }
};
// Notices a NaN or Inf among the pairs it is shown: FP32 adds 0 x each (a NaN stays), FP64 looks at
// the exponents (the FP64 units are what the FP64 kernels wait for)
template <typename T>
struct FiniteCheck {
    using O = PairOps<T>;
    typename O::P c;
    unsigned big = 0;
    __device__ __forceinline__ FiniteCheck() : c(O::dup(T(0))) {}
    __device__ __forceinline__ void see(typename O::P v) {
        if constexpr (sizeof(T) == 4) {
            c = O::fma(v, O::dup(T(0)), c);
        } else {
            auto e = [](double a) { return (unsigned)__double2hiint(a) & 0x7fffffffu; };
            big = max(big, max(e(v.x), e(v.y)));
        }
    }
    __device__ __forceinline__ bool bad() const {
        if constexpr (sizeof(T) == 4) return !(O::lo(c) + O::hi(c) == T(0));
        else return big >= 0x7ff00000u;
    }
};
// N pairs of neighbouring cells: a thread's vector along z
template <typename T, int N>
struct Pairs {
    typename PairOps<T>::P p[N];
};
__device__ __forceinline__ void ldp(Pairs<float, 2>& r, const float* q) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(q);
    r.p[0] = v.x; r.p[1] = v.y;
}
__device__ __forceinline__ void ldp(Pairs<float, 1>& r, const float* q) { r.p[0] = *reinterpret_cast<const unsigned long long*>(q); }
__device__ __forceinline__ void ldp(Pairs<double, 1>& r, const double* q) { r.p[0] = *reinterpret_cast<const double2*>(q); }
// the same through the read-only path: C^2 and m1, which no step kernel writes (see pdl_handover)
__device__ __forceinline__ void ldr(Pairs<float, 2>& r, const float* q) {
    const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2*>(q));
    r.p[0] = v.x; r.p[1] = v.y;
}
__device__ __forceinline__ void ldr(Pairs<float, 1>& r, const float* q) { r.p[0] = __ldg(reinterpret_cast<const unsigned long long*>(q)); }
__device__ __forceinline__ void ldr(Pairs<double, 1>& r, const double* q) { r.p[0] = __ldg(reinterpret_cast<const double2*>(q)); }
__device__ __forceinline__ void ldp(Pairs<double, 2>& r, const double* q) {
    r.p[0] = reinterpret_cast<const double2*>(q)[0];
    r.p[1] = reinterpret_cast<const double2*>(q)[1];
}
__device__ __forceinline__ void ldr(Pairs<double, 2>& r, const double* q) {
    r.p[0] = __ldg(reinterpret_cast<const double2*>(q));
    r.p[1] = __ldg(reinterpret_cast<const double2*>(q) + 1);
}
__device__ __forceinline__ void stp(double* q, const Pairs<double, 2>& r) {
    reinterpret_cast<double2*>(q)[0] = r.p[0];
    reinterpret_cast<double2*>(q)[1] = r.p[1];
}
__device__ __forceinline__ void stp_cs(double* q, const Pairs<double, 2>& r) {
    __stcs(reinterpret_cast<double2*>(q), r.p[0]);
    __stcs(reinterpret_cast<double2*>(q) + 1, r.p[1]);
}
__device__ __forceinline__ void stp(float* q, const Pairs<float, 2>& r) { *reinterpret_cast<ulonglong2*>(q) = make_ulonglong2(r.p[0], r.p[1]); }
__device__ __forceinline__ void stp(float* q, const Pairs<float, 1>& r) { *reinterpret_cast<unsigned long long*>(q) = r.p[0]; }
__device__ __forceinline__ void stp(double* q, const Pairs<double, 1>& r) { *reinterpret_cast<double2*>(q) = r.p[0]; }
__device__ __forceinline__ void stp_cs(float* q, const Pairs<float, 2>& r) { __stcs(reinterpret_cast<ulonglong2*>(q), make_ulonglong2(r.p[0], r.p[1])); }
__device__ __forceinline__ void stp_cs(float* q, const Pairs<float, 1>& r) { __stcs(reinterpret_cast<unsigned long long*>(q), r.p[0]); }
__device__ __forceinline__ void stp_cs(double* q, const Pairs<double, 1>& r) { __stcs(reinterpret_cast<double2*>(q), r.p[0]); }

// a thread's cells of one row with NB vectors of NP pairs on either side.  Taps an odd number
// of cells away straddle two pairs: in FP32 they are taken cell by cell (putting the pairs
// together costs more moves than the packed operation saves).
template <typename T, int NP, int NB>
struct Window {
    using O = PairOps<T>;
    using P = typename O::P;
    static constexpr int N = (2 * NB + 1) * NP;
    P e[N];
    __device__ __forceinline__ void load(const T* q, const Pairs<T, NP>* centre) {
#pragma unroll
        for (int j = 0; j <= 2 * NB; ++j) {
            Pairs<T, NP> a;
            if (j == NB && centre) a = *centre;
            else ldp(a, q + j * 2 * NP);
#pragma unroll
            for (int k = 0; k < NP; ++k) e[j * NP + k] = a.p[k];
        }
    }
    __device__ __forceinline__ T cell(int i) const { return i & 1 ? O::hi(e[i >> 1]) : O::lo(e[i >> 1]); }
    // the pair of cells i, i + 1
    __device__ __forceinline__ P at(int i) const { return i & 1 ? O::mk(cell(i), cell(i + 1)) : e[i >> 1]; }
    // acc + wd ((v_{c+d} - v_c) + (v_{c-d} - v_c)) for the pair at cell c
    __device__ __forceinline__ P d2(P acc, P wd, int c, int d) const {
        if (d & 1) {
            const P uc = e[c >> 1];
            const T a = (cell(c + d) - O::lo(uc)) + (cell(c - d) - O::lo(uc));
            const T b = (cell(c + 1 + d) - O::hi(uc)) + (cell(c + 1 - d) - O::hi(uc));
            return O::mk(::fma(O::lo(wd), a, O::lo(acc)), ::fma(O::hi(wd), b, O::hi(acc)));
        }
        return O::fma(wd, O::add(O::sub(e[(c + d) >> 1], e[c >> 1]), O::sub(e[(c - d) >> 1], e[c >> 1])), acc);
    }
    // acc + wd (v_{c+d} - v_{c-d})
    __device__ __forceinline__ P d1(P acc, P wd, int c, int d) const {
        if (d & 1)
            return O::mk(::fma(O::lo(wd), cell(c + d) - cell(c - d), O::lo(acc)),
                         ::fma(O::hi(wd), cell(c + 1 + d) - cell(c + 1 - d), O::hi(acc)));
        return O::fma(wd, O::sub(e[(c + d) >> 1], e[(c - d) >> 1]), acc);
    }
};

// weights of the derivatives over the first differences e_j = v_{j+1} - v_j (FP64 path):
// v'' = sum_j c_j (e_j - e_{-1-j}), j = 0..R-1, with c_j = sum_{m>j} w2_m
__host__ __device__ constexpr double c2sum(int R, int j) {
    double s = 0;
    for (int m = j + 1; m <= R; ++m) s += d2w(R, m);
    return s;
}

}  // namespace
}  // namespace pgb
