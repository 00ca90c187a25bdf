// Axis-pass kernels of the Strang step and the device table builders.
//
// A Strang step of the reference, V/2 . F^-1 K F . V/2 (core/src/propagator.ixx:110-119),
// is executed as a chain of axis passes over psi in HBM.  With the interior
// half-kicks merged into full kicks (reference GPU batch, solver/src/vk_engine.ixx:611-633):
//
//   3D step:  X[inv x, V*M, fwd x]  Y[fwd y]  Z[fwd z, K/N, inv z]  Y[inv y]
//   2D step:  X[inv x, V*M, fwd x]  Y[fwd y, K/N, inv y]
//   1D step:  X[V*M, fwd x, K/N, inv x]
//
// so one step reads and writes psi 4 / 2 / 1 times and reads the potential
// phase table once.  All diagonal factors (potential phase, absorbing mask,
// kinetic phase, 1/N) are applied in FP64 whatever the storage precision.
#pragma once

#include <type_traits>

#include "ses_fft.cuh"

namespace sesk {

enum DiagKind : int { DG_NONE = 0, DG_HALF = 1, DG_FULL = 2 };

// Number of FP64 sums a k-space reduction produces:
// [0] sum|phi|^2  [1] sum k^2/(2m)|phi|^2  [2..4] sum k_a |phi|^2
constexpr int kRedK = 5;
// Real-space sums: [0] sum|psi|^2 [1] sum V|psi|^2 [2] sum_{x in [a,b)}|psi|^2
// [3..5] sum r_a|psi|^2 [6..8] sum r_a^2|psi|^2
constexpr int kRedR = 9;

struct Tables {
    const void* vtab;          // C128: cis(-V dt/2) as cx<double>; C64: cis(-V dt/2) - 1 as cx<float>
    const double* mask1[3];    // separable absorber profiles (all set or all null)
    const double* maskfull;    // non-separable absorber (nullable)
    const cx<double>* kd[3];   // per axis: cis(-k^2 dt/(2m)) - 1
    const double* kv[3];       // per axis: wavenumbers (fftfreq layout)
    // complex64 path: the same FP64-built per-axis tables rounded to FP32
    const float* mask1f[3];
    const cx<float>* kdf[3];
    double inv_mass;
    double kscale;             // 1/N, folded into the kinetic multiply
    // long 1D line (four-step layout N1 x N2); null / 0 otherwise
    const void* kfull;         // kinetic delta per stored k-space element (cx<T>)
    const void* tw4;           // W_N^{n1 k2} per element (cx<T>; complex64: FP32-rounded)
    const void* tw4l;          // complex64: FP32 remainder of tw4
    int long_n2;               // N2: stored element (k1, k2) is frequency k2 + N2 k1
    // dipole drive (drive.ixx:25-40): the per-axis factors of this pass's kick
    // psi *= cis(-theta (axis . r)), nx + ny + nz entries; null off
    const cx<double>* kick;
};

// complex64 phase multiplies in FP32 on the delta form: psi + psi*d, d = factor - 1.
__device__ __forceinline__ cx<float> add_mul(cx<float> p, cx<float> d) {  // p + p*d
    return mk<float>(fmaf(p.x, d.x, fmaf(-p.y, d.y, p.x)), fmaf(p.x, d.y, fmaf(p.y, d.x, p.y)));
}
// (1+a)(1+b) - 1 for the separable kinetic deltas
__device__ __forceinline__ cx<double> dmul1(cx<double> a, cx<double> b) { return a + b + a * b; }
__device__ __forceinline__ cx<float> dmul1f(cx<float> a, cx<float> b) {  // (1+a)(1+b) - 1
    return mk<float>(fmaf(a.x, b.x, fmaf(-a.y, b.y, a.x + b.x)), fmaf(a.x, b.y, fmaf(a.y, b.x, a.y + b.y)));
}

template <typename T>
struct PassArgs {
    const cx<T>* src;
    cx<T>* dst;
    int axis;  // 0 = x (contiguous lines), 1 = y, 2 = z
    int nx, ny, nz;
    long long nlines;
    // strided-axis addressing: line slot s -> base (s % nu) + (s / nu) * sw,
    // element stride se.  For the x axis: base = s * nx, se = 1.
    long long nu, sw, se;
    FastDiv fnu, fny, fnx;
    const cx<T>* stw;  // per-stage twiddle tables of the axis's plan, forward then reversed order (hi part)
    const cx<T>* stwl; // FP32: remainder (lo part) of the same tables
    // run-time parts of the pass program (the structure is the kernel's MODE)
    int d_load, d_mid, d_store;
    int m_load, m_mid, m_store;
    double out_scale;
    Tables tb;
    double* partials;
};
// Passed by value to every pass: with 816 bytes (the run-time plan's tables among them) the
// launches of a small step cost about 0.15 us more each than with these 352 (96 x 96 x 16
// complex128 step of four 13.2 -> 12.7 us, 32 x 32 x 16 of two 6.8 -> 6.5).
static_assert(sizeof(PassArgs<float>) <= 384 && sizeof(PassArgs<double>) <= 384, "launch arguments of a pass");

// Absorber value at flat index f, coordinates (i, j, k): m = mx[i] * (my[j] * mz[k]), in FP64.
template <typename T>
__device__ __forceinline__ double maskval(const Tables& tb, long long f, int i, int j, int k) {
    if (tb.maskfull) return tb.maskfull[f];
    return tb.mask1[0][i] * (tb.mask1[1][j] * tb.mask1[2][k]);
}

template <typename T>
__device__ __forceinline__ cx<T> apply_diag_tv(cx<T> v, int kind, cx<T> tab, int use_mask, double m);

// psi * (potential phase) * (mask) at flat index f, coordinates (i, j, k).
template <typename T>
__device__ __forceinline__ cx<T> apply_diag(cx<T> v, int kind, int use_mask, long long f, int i, int j,
                                            int k, const Tables& tb) {
    const cx<T> tab = kind != DG_NONE ? reinterpret_cast<const cx<T>*>(tb.vtab)[f] : v;
    return apply_diag_tv(v, kind, tab, use_mask, use_mask ? maskval<T>(tb, f, i, j, k) : 1.0);
}

// Same as apply_diag with the potential-table entry and mask value supplied
// by the caller (pipelined passes stage the table in shared memory).
//   DG_HALF: psi * h (* m)            h = cis(-V dt/2)
//   DG_FULL: (psi * h (* m)) * h      the kick between two steps, applied as the
//            half kick that ends one step (with the mask) followed by the half
//            kick that starts the next, in exactly that arithmetic -- so a run
//            of steps split into two calls gives the same bits as one call.
// The complex64 path multiplies in FP32 on the delta form psi + psi*d, d = h - 1.
template <typename T>
__device__ __forceinline__ cx<T> apply_diag_tv(cx<T> v, int kind, cx<T> tab, int use_mask, double m) {
    if constexpr (sizeof(T) == 4) {
        cx<float> p = v;
        if (kind != DG_NONE) p = add_mul(p, tab);
        if (use_mask) {  // p - p (1 - m): the FP32 rounding falls on the small 1 - m, not on m
            const float md = (float)(1.0 - m);
            p = mk<float>(fmaf(-p.x, md, p.x), fmaf(-p.y, md, p.y));
        }
        if (kind == DG_FULL) p = add_mul(p, tab);
        return p;
    } else {
        cx<double> p = v;
        if (kind != DG_NONE) p = p * tab;
        if (use_mask) p = mk<double>(p.x * m, p.y * m);
        if (kind == DG_FULL) p = p * tab;
        return p;
    }
}

// psi_k * K / N then conj (inverse FFT start); complex64: FP32 on the delta form.
__device__ __forceinline__ cx<float> kinetic_conj_f(cx<float> v, cx<float> d, double kscale) {
    return cconj(scale_d(add_mul(v, d), kscale));
}

template <typename T>
__device__ __forceinline__ cx<T> kinetic_apply(cx<T> v, cx<double> dother, const cx<double>* kda64,
                                               const cx<float>* kda32, int pos, double kscale) {
    if constexpr (sizeof(T) == 4) return kinetic_conj_f(v, dmul1f(narrow<float>(dother), kda32[pos]), kscale);
    else return kinetic_conj(v, dmul1(dother, kda64[pos]), kscale);
}


// psi_k * K(k) / N followed by the conjugation that starts the inverse FFT.
template <typename T>
__device__ __forceinline__ cx<T> kinetic_conj(cx<T> v, cx<double> d, double kscale) {
    cx<double> p = widen(v);
    p = p + p * d;
    return narrow<T>(mk<double>(p.x * kscale, -p.y * kscale));
}

// Kinetic multiply from a per-element delta table (long 1D lines).
template <typename T>
__device__ __forceinline__ cx<T> kinetic_full(cx<T> v, const void* kfull, long long idx, double kscale) {
    if constexpr (sizeof(T) == 4)
        return kinetic_conj_f(v, reinterpret_cast<const cx<float>*>(kfull)[idx], kscale);
    else
        return kinetic_conj(v, reinterpret_cast<const cx<double>*>(kfull)[idx], kscale);
}

// Kinetic multiply of element `pos` of an axis whose other two axes give the
// FP64 delta `dother`: complex128 -> FP64; complex64 -> FP32 delta form with
// the FP32-rounded tables (kda64 / kda32 are the axis's FP64 / FP32 deltas).
template <typename T>
__device__ __forceinline__ cx<T> kinetic_apply(cx<T> v, cx<double> dother, const cx<double>* kda64,
                                               const cx<float>* kda32, int pos, double kscale);

// kinetic_apply with the axis's delta at this element fetched beforehand (kde:
// the FP64 delta for complex128, the FP32-rounded one for complex64): the same
// arithmetic, so passes that prefetch their tables give the same bits.
template <typename T>
using KinDelta = typename std::conditional<sizeof(T) == 4, cx<float>, cx<double>>::type;

template <typename T>
__device__ __forceinline__ cx<T> kinetic_apply_pre(cx<T> v, cx<double> dother, KinDelta<T> kde, double kscale) {
    if constexpr (sizeof(T) == 4) return kinetic_conj_f(v, dmul1f(narrow<float>(dother), kde), kscale);
    else return kinetic_conj(v, dmul1(dother, kde), kscale);
}

template <typename T>
__device__ __forceinline__ KinDelta<T> kin_delta(const cx<double>* kda64, const cx<float>* kda32, int pos) {
    if constexpr (sizeof(T) == 4) return kda32[pos];
    else return kda64[pos];
}

template <int NR>
__device__ __forceinline__ void block_reduce_store(double (&acc)[NR], double* out) {
    __shared__ double red[32][NR];
#pragma unroll
    for (int q = 0; q < NR; ++q) {
        double v = acc[q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        acc[q] = v;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
#pragma unroll
        for (int q = 0; q < NR; ++q) red[warp][q] = acc[q];
    }
    __syncthreads();
    if (threadIdx.x < NR) {
        const int nw = (blockDim.x + 31) >> 5;
        double s = 0.0;
        for (int w = 0; w < nw; ++w) s += red[w][threadIdx.x];
        out[(size_t)blockIdx.x * NR + threadIdx.x] = s;
    }
}

// Accumulate k-space sums of one element: axis wavenumber ka, other two
// wavenumbers (kb, kc) in fixed axis slots.
__device__ __forceinline__ void acc_k(double (&acc)[kRedK], double w, const double* k3,
                                      double inv_mass) {
    const double ksq = k3[0] * k3[0] + k3[1] * k3[1] + k3[2] * k3[2];
    acc[0] += w;
    acc[1] += 0.5 * ksq * inv_mass * w;
    acc[2] += k3[0] * w;
    acc[3] += k3[1] * w;
    acc[4] += k3[2] * w;
}

// ---------------------------------------------------------------------------
// Pass programs.  Each program is its own kernel so every kernel holds at most
// two tile FFTs (register allocation stays local; no run-time program flags in
// the butterfly loops).
// ---------------------------------------------------------------------------
enum XMode : int {
    XM_FWD = 0,     // fwd x                                   (fft3 surface, energy copy)
    XM_INV = 1,     // inv x, scaled                           (fft3 surface)
    XM_START = 2,   // V/2, fwd x                              (first step of a batch)
    XM_MID = 3,     // inv x, V (* M), fwd x                   (between steps)
    XM_END = 4,     // inv x, V/2 (* M)                        (end of a batch)
    XM_1D = 5,      // V/2 or V (* M), fwd x, K/N, inv x, [V/2 (* M)]   (x only axis)
    XM_REDUCE = 6   // fwd x, k-space sums                     (1D energy)
};
// Strided programs.  SM_TW_* are the strided halves of a long 1D line run as a
// four-step transform (line of N = N1 N2 points stored as N1 x N2, x fastest):
// the y pass is the length-N2 transform with the twiddles W_N^{n1 k2} on its
// k-space side, the x pass (XM_1D) the length-N1 transform with the kinetic
// phase of frequency k2 + N2 k1 between forward and inverse.
enum SModeK : int {
    SM_FWD = 0,       // fwd y/z
    SM_INV = 1,       // inv y/z, scaled
    SM_FUSED = 2,     // fwd, K/N, inv                 (last axis)
    SM_REDUCE = 3,    // fwd, k-space sums
    SM_TW_START = 4,  // [V/2 (* M)], fwd y, * W        (long line: batch start, or k-space copy)
    SM_TW_MID = 5,    // * conj W, inv y, V (* M), fwd y, * W   (between steps)
    SM_TW_END = 6     // * conj W, inv y, V/2 (* M)     (batch end)
};
constexpr int kSModes = 7;

// Programmatic dependent launch: a pass kernel may be launched while the
// previous kernel of its stream drains; it waits here, before touching any
// field or argument table, until that kernel has completed and its writes are
// visible (a no-op for a normal launch).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// The grid as the real-space observables see it.
struct ObsArgs {
    long long N;
    int nx, ny;
    FastDiv fnx, fny;
    double x0, hx, y0, hy, z0, hz;
    double xlo, xhi;
};

template <typename S, typename D>
__global__ void convert_kernel(const cx<S>* __restrict__ src, cx<D>* dst, long long N) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N;
         i += (long long)gridDim.x * blockDim.x) {
        dst[i] = mk<D>((D)src[i].x, (D)src[i].y);
    }
}

}  // namespace sesk
