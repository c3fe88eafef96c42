// Device-side data layout and kernel parameters of the batched wave pipeline.
//
// Internal field layout (per shot, per field): a zero halo of HX = 4 rows on
// both x sides (2D/3D), HY = 4 rows on both y sides (3D), and along z a row
// pitch `ldz` (multiple of 32 elements) with the grid starting at z offset
// OZ = 4.  Cell (i, j, k) of the padded PySIT grid lives at
//     ((i + HX) * (ny + 2*HY) + (j + HY)) * ldz + OZ + k.
// The halos are never written with non-zero values, so the stencils read the
// reference's zero extension without bounds tests, rows start 128-byte
// aligned and z-vectors of 16 bytes are aligned.
#pragma once

#include "common.cuh"

namespace pgb {

constexpr int kHalo = 4;  // x/y halo rows and smem z halo (max stencil radius)
constexpr int kOZ = 4;    // z offset of cell k = 0 inside a row
constexpr int kTailZ = 12;  // zero cells kept after the last cell of a row (>= halo + vector - 1)

// bits of the device error word of a plan
#define PGB_ERR_TIMEOUT 1    // a bounded device wait expired
#define PGB_ERR_NONFINITE 2  // a NaN / Inf wavefield value (unstable time step)

template <typename T> struct V16;
template <> struct V16<float> { using type = float4; static constexpr int N = 4; };
template <> struct V16<double> { using type = double2; static constexpr int N = 2; };

// Kernel modes of the batched step.
enum StepMode : int {
    kFwd = 0,     // forward step; records traces of u_k
    kRecomp = 1,  // forward recompute; writes the imaging operand dWaveOp_k
    kAdj = 2,     // adjoint step driven by the residual; accumulates ic += q_k * dWaveOp_k
    kBorn = 3,    // 2D: scattered-field step with the Born source -m1 dWaveOp0_k inside the stencil
};

// Injection operator of one step: per shot a box of cells [x0,x1) x [y0,y1) x [z0,z1)
// with CSR rows over the box cells (x-major, z fastest); entries (point, weight).
// rhs(cell) = sum_e w[e] * amp[shot * amp_sstride + pt[e]].
template <typename T>
struct Inject {
    const int* box;          // [nshot][6]: x0, x1, y0, y1, z0, z1 (grid coords)
    const long long* rpbase; // [nshot] offset of the shot's first row pointer
    const int* rowptr;       // CSR row pointers (absolute entry indices)
    const int* pt;           // entry point index
    const T* w;              // entry weight
    const T* amp;            // amplitudes of this step for shot 0
    long long amp_sstride;   // amplitude stride between shots
    int on;                  // 0: no injection this step
};

// Trace recording of u_k: per (shot, receiver) a CSR row of taps.
template <typename T>
struct Record {
    const int* rowptr;       // [nshot*nrec + 1] absolute tap index (shot-major)
    const long long* off;    // tap offset inside a field (internal layout)
    const T* w;              // tap weight (sampling operator)
    T* traces;               // trace sample k of shot 0 receiver 0
    long long tr_sstride;    // stride between shots in the trace array
    int nrec;
    int lanes;               // threads per (shot, receiver): a power of two up to 32
};

template <typename T>
struct WaveParams {
    // geometry
    int nx, ny, nz;          // padded grid (ny = 1 in 2D)
    int ldz;                 // row pitch (elements)
    int rows_y;              // ny + 2*HY
    long long fstride;       // elements between consecutive shots of one field
    int hx, hy;              // halos (4 / 0 in 2D)
    int nshot;               // shots in this launch
    // wavefields (shot 0 base)
    T* u_prev;               // in: u_{k-1}; out: u_{k+1} (same cell, in place)
    const T* u_cur;          // u_k
    const T* phx_in; T* phx_out;
    const T* phy_in; T* phy_out;
    const T* phz_in; T* phz_out;
    const T* psi_in; T* psi_out;
    const T* c2;             // C^2, shared by all shots (internal layout)
    // PML (kernel convention) and mesh sigma maps, full length per axis
    const T *sgx, *sgy, *sgz;
    const T *mgx, *mgy, *mgz;
    const T *fcx, *fcy, *fcz;  // 2 dt^2 / (2 + dt s) of each axis' step sigmas alone (one_sigma_fac)
    int pxl, pxr, pyl, pyr, pzl, pzr;  // padding widths holding PML state
    // scalars
    T dt, dt2, idt2, i2dt, idx, idx2, idy, idy2, idz, idz2;
    // injection / recording / imaging
    Inject<T> inj;
    Record<T> rec;
    T* dw_out;               // kRecomp: imaging operand of this step (shot 0 base)
    const T* dw_in;          // kAdj: imaging operand of this step
    T* ic;                   // kAdj: imaging accumulator (shot 0 base)
    int image;               // kAdj: accumulate this step
    const T* m1;             // kBorn: edge-padded model perturbation (internal layout, shared by the shots);
                             // dw_in holds dWaveOp0_k
    int* err;                // device error word (PGB_ERR_* bits), may be NULL
    unsigned polls;          // tests of the wait that wait_fault adds (0: 64)
    int wait_fault;          // test aid: each 2D block first waits (bounded) on a barrier nothing arrives on
    int pf_next;             // 2D: blocks fetch the next shot's tile into L2
    int psi_c2;              // 3D: 1 = C^2 multiplies sigma_x sigma_y sigma_z psi (the reference), 0 = not
    int nan_check;           // kRecomp: flag non-finite u_{k+1} as kFwd does (a forward sweep that keeps dWaveOp)
};

template <typename T> __device__ __forceinline__ T rcp_(T x);
// FP32: the fast reciprocal (within ~1 ulp; the FP32 path's tolerances are 1e-4 / 1e-3);
// FP64 keeps the exact division of the reference
template <> __device__ __forceinline__ float rcp_(float x) { return __fdividef(1.0f, x); }
template <> __device__ __forceinline__ double rcp_(double x) { return 1.0 / x; }
// 2 dt^2 / (2 + dt s) with the rounding of the 2D (product with the reciprocal) and 3D (quotient) updates
template <typename T>
__device__ __forceinline__ T one_sigma_fac(int dim, T dt, T dt2, T s) {
    return dim == 2 ? (T(2) * dt2) * rcp_(::fma(dt, s, T(2))) : T(2) * dt2 / ::fma(dt, s, T(2));
}

// ---- helpers shared by the 2D kernels ---------------------------------------
// Programmatic dependent launch: consecutive step kernels of a stream.  A step kernel waits for the
// kernel before it to be complete, its writes visible, before it reads a wavefield, and then lets
// the next one start (its blocks take the slots that the running one leaves and wait in turn: the
// launch latency and the reads ahead of the wait overlap the running kernel).  What no step kernel
// writes (tables, sigmas, C^2, m1, injection operators) may be read before the wait, and through the
// read-only path; so may the amplitudes, since a memset or another kernel always stands between the
// steps that record traces and the adjoint steps that read the residual in their place.  Every wavefield, Phi, psi, dWaveOp and image is written by a kernel
// that may still run when this one starts: it is read after the wait and with ordinary loads, since
// __ldg is defined only for data that stay constant as long as the grid lives (the compiler may move
// it across the wait, and L1 need not drop its lines).
// Letting the next kernel start before the wait stacked several launches on the SMs: 141 x 81 cells
// in FP64 8.2 us a step instead of 7.1 without any overlap.
__device__ __forceinline__ void pdl_handover() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <typename... P, typename... A>
inline void launch_step(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// rhs of one cell from the injection operator of its shot
template <typename T>
__device__ __forceinline__ T inject_rhs(const Inject<T>& inj, const int* bx, int shot, int x, int z) {
    if (x < bx[0] || x >= bx[1] || z < bx[4] || z >= bx[5]) return T(0);
    int c = (x - bx[0]) * (bx[5] - bx[4]) + (z - bx[4]);
    const int* rp = inj.rowptr + inj.rpbase[shot];
    int e0 = __ldg(rp + c), e1 = __ldg(rp + c + 1);
    const T* amp = inj.amp + shot * inj.amp_sstride;
    T acc = T(0);
    int e = e0;
    // taps in groups of 8: the point indices and weights first, then the amplitudes, so that
    // a group's dependent loads are in flight together (the sum keeps the taps' order)
    for (; e + 8 <= e1; e += 8) {
        int pt[8];
        T w[8], a[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) { pt[q] = __ldg(inj.pt + e + q); w[q] = __ldg(inj.w + e + q); }
#pragma unroll
        for (int q = 0; q < 8; ++q) a[q] = __ldg(amp + pt[q]);
#pragma unroll
        for (int q = 0; q < 8; ++q) acc += w[q] * a[q];
    }
    for (; e < e1; ++e) acc += __ldg(inj.w + e) * __ldg(amp + __ldg(inj.pt + e));
    return acc;
}

template <typename T>
__device__ __forceinline__ T inject_rhs3(const Inject<T>& inj, const int* bx, int shot, int x,
                                         int y, int z) {
    if (x < bx[0] || x >= bx[1] || y < bx[2] || y >= bx[3] || z < bx[4] || z >= bx[5]) return T(0);
    long long c = ((long long)(x - bx[0]) * (bx[3] - bx[2]) + (y - bx[2])) * (bx[5] - bx[4]) + (z - bx[4]);
    const int* rp = inj.rowptr + inj.rpbase[shot];
    int e0 = __ldg(rp + c), e1 = __ldg(rp + c + 1);
    const T* amp = inj.amp + shot * inj.amp_sstride;
    T acc = T(0);
    for (int e = e0; e < e1; ++e) acc += __ldg(inj.w + e) * __ldg(amp + __ldg(inj.pt + e));
    return acc;
}

// Trace recorder: p.rec.lanes threads per (shot, receiver), 32 / lanes receivers per warp pass.
// Lane l sums taps l, l + lanes, ... in order, up to 8 of them with their loads in flight
// together; a fixed butterfly over the lanes adds the partial sums, so the result does not
// depend on scheduling.  Every lane of the warp takes part (the butterfly shuffles over it).
template <typename T>
__device__ __forceinline__ long long record_passes(const WaveParams<T>& p) {
    const int per = 32 / p.rec.lanes;
    return p.rec.traces ? ((long long)p.nshot * p.rec.nrec + per - 1) / per : 0;
}
template <typename T>
__device__ __forceinline__ void record_pass(const WaveParams<T>& p, long long pass) {
    constexpr int kTaps = 8;
    const int G = p.rec.lanes;
    const int lane = threadIdx.x & 31, l = lane & (G - 1);
    const long long id = pass * (32 / G) + lane / G;
    const bool mine = id < (long long)p.nshot * p.rec.nrec;
    int shot = 0;
    T acc = T(0);
    if (mine) {
        shot = (int)(id / p.rec.nrec);
        const int e1 = __ldg(p.rec.rowptr + id + 1);
        const T* u = p.u_cur + (long long)shot * p.fstride;
        for (int e = __ldg(p.rec.rowptr + id) + l; e < e1; e += kTaps * G) {
            long long off[kTaps];
            T w[kTaps], v[kTaps];
#pragma unroll
            for (int q = 0; q < kTaps; ++q) {
                const bool in = e + q * G < e1;
                off[q] = in ? __ldg(p.rec.off + e + q * G) : 0;
                w[q] = in ? __ldg(p.rec.w + e + q * G) : T(0);
            }
#pragma unroll
            for (int q = 0; q < kTaps; ++q) v[q] = e + q * G < e1 ? u[off[q]] : T(0);
#pragma unroll
            for (int q = 0; q < kTaps; ++q)
                if (e + q * G < e1) acc += w[q] * v[q];
        }
    }
    for (int m = G >> 1; m > 0; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
    if (mine && l == 0) p.rec.traces[shot * p.rec.tr_sstride + (id - (long long)shot * p.rec.nrec)] = acc;
}

// 2D tiles of one shot, shared by all shots: the device's form of the task table, interior
// tiles first
struct Tile2d {
    int x0, rows, zs, ncell;    // rows x0 .. x0+rows-1, cells zs .. zs+ncell-1
    int nzv, inv, kind, pad;    // vectors along z, ceil(2^16 / nzv), 0 interior / 1 PML shell / 2 shell, sigma_x zero
};
constexpr int kT2 = 128;  // threads of a block at most
// `strip`: x-rows per thread (1, 2 or 4); `threads`: of a block (32, 64 or kT2); `inj_cap`: cells of
// the largest tile's part of any shot's injection box
template <typename T, int R, int MODE>
void launch_wave2d_tiles(const WaveParams<T>& p, const Tile2d* tiles, int nint, int nshell, int strip, int threads,
                         int inj_cap, cudaStream_t s);
// cells of a thread along z: four (FP32 a 16-byte vector; FP64 two, whose window of first differences
// serves all four), two in the shell (two sets of columns and windows to hold)
constexpr int wave2d_cells(int pml) { return pml ? 2 : 4; }
// widest z-range of a tile of each kind: 32 16-byte vectors (FP32 shell: 8-byte ones)
constexpr int wave2d_seg(int dtype_bytes, int pml) { return dtype_bytes == 4 && !pml ? 128 : 64; }
// x-rows a block's threads take side by side, `strip` rows each
constexpr int wave2d_tile_rows(int pml, int strip, int threads, int zcells) {
    const int V = wave2d_cells(pml);
    return threads / ((zcells + V - 1) / V) * strip;
}
// 3D tiles of one shot, shared by all shots: the device's form of the task table, interior
// tiles first
struct Tile3d {
    int x0, x1, y0, y1;     // planes and rows
    int zs, ze, kind, inv;  // cells along z; 0 interior, 1 general shell, 2-4 faces; ceil(2^16 / vectors along z)
};
constexpr int kT3 = 128;                 // threads of a block at most
constexpr int kMaxInj3d = 160 * 1024;    // bytes of injection cells of a tile at most
// `planes`: x-planes per thread and round (1 or 4); `threads`: of a block (64 or kT3); `inj_cap`: cells of the largest tile's part of
// any shot's injection box
template <typename T, int R, int MODE>
void launch_wave3d_tiles(const WaveParams<T>& p, const Tile3d* tiles, int nint, int nshell, int planes, int threads,
                         int inj_cap, cudaStream_t s);
template <typename T, int R>
void wave3d_tile_prepare();
// widest z-range of a tile: 32 vectors
constexpr int wave3d_seg(int dtype_bytes) { return 32 * (16 / dtype_bytes); }
// y-rows of a tile of zcells z-cells: a warp takes 32 / vectors rows
constexpr int wave3d_task_rows(int dtype_bytes, int threads, int zcells) {
    const int V = 16 / dtype_bytes;
    return threads / 32 * (32 / ((zcells + V - 1) / V));
}
// A run of 1D steps in one launch (wave1d.cu)
template <typename T>
struct Sweep1d {
    const T *in_prev, *in_cur, *in_phz;  // state before the first step (shot 0)
    T *out_prev, *out_cur, *out_phz;     // and after the last
    int k0, n, dir;                      // first step, number of steps, +1 or -1
    int npts, npts_max;                  // injection points of this run; of any run of the plan
    int most_nc;                         // blocks per shot at most (wave1d_prepare)
    T* traces;                           // NULL, or the traces of step 0 of shot 0 (rows of p.rec.nrec)
    T* dw;                               // NULL, or dWaveOp: step k with k % dw_period == 0 in field (k - dw_k0) / dw_div
    int dw_period, dw_k0, dw_div;
    T* ckpt;                             // NULL, or the checkpoints: u_{k-1}, u_k, Phi_z of every S-th step
    int S;
    long long field_stride;              // elements between fields of a launch's shots
    int cells, threads;                  // cells per block and threads that step them (set by the launch)
    unsigned inv;                        // ceil(2^32 / cells): the block of a cell
};
// whether launches of nshot shots on a grid of nz cells run as sweeps
template <typename T>
bool wave1d_sweeps(int nz, int nsrc, int nrec, int nshot);
// readies the kernels on the device; the largest cluster limit (16 or 8 blocks) whose clusters it places,
// 0: none
template <typename T, int R>
int wave1d_prepare(int nz, int nsrc, int nrec);
template <typename T, int R, int MODE>
void launch_wave1d_sweep(const WaveParams<T>& p, Sweep1d<T> q, cudaStream_t s);
template <typename T, int R, int MODE>
void launch_wave1d(const WaveParams<T>& p, cudaStream_t s);

}  // namespace pgb
