// Non-template kernels of the solver (table builders, final reductions).
// Included by ses_gpu.cu only: __global__ functions defined here have one
// definition in the library.
#pragma once

#include "ses_pass.cuh"

namespace sesk {

// Real-space observables: per-thread FP64 sums, one partial row per CTA.
// Points of a thread per trip: their loads (psi and V) are issued together, which
// keeps 16-64 KB per SM in flight; the indices come from 32-bit divisions by
// invariant integers (N < 2^31).  Bound by memory on large fields, by launch and
// reduction latency on small ones.
constexpr int kObsUnroll = 4;

// CTAs of obs_real_kernel: one trip each until kObsBlocks (fixed by N: deterministic sums).
inline unsigned obs_blocks(long long N, int most) {
    const long long b = (N + 256 * kObsUnroll - 1) / (256 * kObsUnroll);
    return (unsigned)(b < most ? b : most);
}

template <typename T>
__global__ void __launch_bounds__(256) obs_real_kernel(const cx<T>* __restrict__ psi,
                                                       const double* __restrict__ V, ObsArgs o,
                                                       double* partials) {
    double acc[kRedR];
#pragma unroll
    for (int q = 0; q < kRedR; ++q) acc[q] = 0.0;
    const long long stride = (long long)gridDim.x * blockDim.x * kObsUnroll;
    for (long long first = (long long)blockIdx.x * blockDim.x * kObsUnroll + threadIdx.x; first < o.N;
         first += stride) {
        cx<T> pv[kObsUnroll];
        double vv[kObsUnroll];
#pragma unroll
        for (int u = 0; u < kObsUnroll; ++u) {
            const long long idx = first + (long long)u * blockDim.x;
            const bool in = idx < o.N;
            pv[u] = in ? psi[idx] : mk<T>((T)0, (T)0);
            vv[u] = in ? V[idx] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < kObsUnroll; ++u) {
            const long long idx = first + (long long)u * blockDim.x;
            if (idx >= o.N) break;
            const uint32_t line = fdiv((uint32_t)idx, o.fnx);
            const int i = (int)((uint32_t)idx - line * (uint32_t)o.nx);
            const uint32_t k = fdiv(line, o.fny);
            const int j = (int)(line - k * (uint32_t)o.ny);
            const cx<double> p = widen(pv[u]);
            const double w = p.x * p.x + p.y * p.y;
            const double x = o.x0 + i * o.hx, y = o.y0 + j * o.hy, z = o.z0 + (double)(int)k * o.hz;
            acc[0] += w;
            acc[1] += vv[u] * w;
            if (x >= o.xlo && x < o.xhi) acc[2] += w;
            acc[3] += x * w;
            acc[4] += y * w;
            acc[5] += z * w;
            acc[6] += x * x * w;
            acc[7] += y * y * w;
            acc[8] += z * z * w;
        }
    }
    block_reduce_store<kRedR>(acc, partials);
}

// Fixed-order final sum of the n per-CTA partial rows of NR values, by one CTA of
// kFoldThreads threads: out[q] (and host[q], page-locked, when given) =
// sum_b rows[b][q].  The rows are read as one array, thread t at t, t + T, ... with
// T a multiple of NR, so that a thread stays in one column and every load is
// coalesced; then one warp per column adds the threads' sums.  Bound by latency (one
// thread per column reading row after row took 37 us for 592 rows; a 64^3 complex128
// relaxation, which sums after every step, went from 56 to 35 us a step).
constexpr int kFoldThreads = 1024;

template <int NR>
__device__ __forceinline__ void fold_rows(const double* __restrict__ rows, int n, double* out, double* host) {
    __shared__ double red[kFoldThreads];
    constexpr int T = kFoldThreads / NR * NR;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    if (t < T) {
        const long long total = (long long)n * NR;
        long long i = t;
        for (; i + 3 * T < total; i += 4 * T) {
#pragma unroll
            for (int u = 0; u < 4; ++u) s[u] += rows[i + u * T];
        }
        for (; i < total; i += T) s[0] += rows[i];
    }
    red[t] = (s[0] + s[1]) + (s[2] + s[3]);
    __syncthreads();
    if (warp < NR) {
        double v = 0.0;
        for (int j = warp + lane * NR; j < T; j += 32 * NR) v += red[j];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) {
            out[warp] = v;
            if (host) host[warp] = v;
        }
    }
}

// CTA 0: the nr_rows rows of kRedR real-space sums at `real`; CTA 1 (when launched):
// the nk_rows rows of kRedK k-space sums at `kspace`, into out + kRedR.  host: the
// same values in page-locked memory, valid once the stream has passed this kernel.
__global__ void __launch_bounds__(kFoldThreads)
    finalize_kernel(const double* __restrict__ real, int nr_rows, const double* __restrict__ kspace, int nk_rows,
                    double* out, double* host) {
    if (blockIdx.x == 0) fold_rows<kRedR>(real, nr_rows, out, host);
    else fold_rows<kRedK>(kspace, nk_rows, out + kRedR, host ? host + kRedR : nullptr);
}

// ---------------------------------------------------------------------------
// FP64 table builders.  Phase arguments use round-to-nearest intrinsics in the
// reference's evaluation order (no FMA contraction), so theta is bitwise the
// reference's: -0.5*V*dt (propagator.ixx:81) and
// -0.5*(kx^2+ky^2+kz^2)/mass*dt (propagator.ixx:95-96).
// ---------------------------------------------------------------------------
__device__ __forceinline__ double theta_v(double V, double dt) {
    return __dmul_rn(__dmul_rn(-0.5, V), dt);
}

__device__ __forceinline__ double theta_k(double ksq, double mass, double dt) {
    return __dmul_rn(__ddiv_rn(__dmul_rn(-0.5, ksq), mass), dt);
}

// cis(theta) - 1 without cancellation: (-2 sin^2(theta/2), sin(theta))
__device__ __forceinline__ cx<double> cis_minus_one(double th) {
    double s2, c2;
    sincos(0.5 * th, &s2, &c2);
    return mk<double>(-2.0 * s2 * s2, 2.0 * s2 * c2);
}

__global__ void build_vtab_c128(const double* __restrict__ V, cx<double>* out, long long N, double dt) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N;
         i += (long long)gridDim.x * blockDim.x) {
        double s, c;
        sincos(theta_v(V[i], dt), &s, &c);
        out[i] = mk<double>(c, s);
    }
}

__global__ void build_vtab_c64(const double* __restrict__ V, cx<float>* out, long long N, double dt) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N;
         i += (long long)gridDim.x * blockDim.x) {
        out[i] = narrow<float>(cis_minus_one(theta_v(V[i], dt)));
    }
}

// Per-axis factors cis(-theta a_q r_q) of the dipole kicks of several steps: kick s
// (blockIdx.y) has the x, y and z factors one after the other, n0 + n1 + n2 of them --
// a sincos per axis point and kick instead of one per cell.  delta: cis - 1
// (complex64), without cancellation.
constexpr int kKicks = 16;  // kicks per launch
struct KickArgs {
    int n[3];
    double axis[3], origin[3], h[3];
    double theta[kKicks];
};

__global__ void kick_factors(const KickArgs a, int delta, cx<double>* out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int total = a.n[0] + a.n[1] + a.n[2];
    if (i >= total) return;
    cx<double>* o = out + (size_t)blockIdx.y * total + i;
    int q = 0;
    while (i >= a.n[q]) i -= a.n[q++];
    const double ang = -a.theta[blockIdx.y] * (a.axis[q] * (a.origin[q] + i * a.h[q]));
    double s, c;
    if (delta) {
        *o = cis_minus_one(ang);
    } else {
        sincos(ang, &s, &c);
        *o = mk<double>(c, s);
    }
}

// Imaginary time (imaginary_time.ixx:71-95): real weights exp(-V dtau/2) and
// exp(-k^2 dtau/(2m)) in the tables' formats -- complex128 (w, 0), complex64
// the delta (w - 1, 0) from expm1, so small weights-minus-one stay accurate.
__global__ void build_vtab_imag_c128(const double* __restrict__ V, cx<double>* out, long long N, double dtau) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N;
         i += (long long)gridDim.x * blockDim.x)
        out[i] = mk<double>(exp(theta_v(V[i], dtau)), 0.0);
}

__global__ void build_vtab_imag_c64(const double* __restrict__ V, cx<float>* out, long long N, double dtau) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N;
         i += (long long)gridDim.x * blockDim.x)
        out[i] = mk<float>((float)expm1(theta_v(V[i], dtau)), 0.0f);
}

__global__ void build_axis_tables_imag(int n, double dtau, double mass, const double* kv, cx<double>* kd) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < n) kd[j] = mk<double>(expm1(theta_k(__dmul_rn(kv[j], kv[j]), mass, dtau)), 0.0);
}

// Smallest and largest potential value, for the range that one imaginary-time step can
// scale a field by: one row per CTA, then (one CTA) host[0] = min, host[1] = max.
__global__ void __launch_bounds__(256) value_range(const double* __restrict__ V, long long N, double* rows) {
    double lo = INFINITY, hi = -INFINITY;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < N; i += (long long)gridDim.x * 256) {
        lo = fmin(lo, V[i]);
        hi = fmax(hi, V[i]);
    }
    __shared__ double slo[256], shi[256];
    slo[threadIdx.x] = lo;
    shi[threadIdx.x] = hi;
    __syncthreads();
    for (int h = 128; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h) {
            slo[threadIdx.x] = fmin(slo[threadIdx.x], slo[threadIdx.x + h]);
            shi[threadIdx.x] = fmax(shi[threadIdx.x], shi[threadIdx.x + h]);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        rows[2 * blockIdx.x] = slo[0];
        rows[2 * blockIdx.x + 1] = shi[0];
    }
}

__global__ void value_range_fold(const double* __restrict__ rows, int n, double* host) {
    double lo = INFINITY, hi = -INFINITY;
    for (int i = threadIdx.x; i < n; i += 32) {
        lo = fmin(lo, rows[2 * i]);
        hi = fmax(hi, rows[2 * i + 1]);
    }
    for (int o = 16; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_down_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_down_sync(0xffffffffu, hi, o));
    }
    if (threadIdx.x == 0) {
        host[0] = lo;
        host[1] = hi;
    }
}

// psi *= 1 / sqrt(sum |psi|^2 dV), the sum taken from sums[0] on the device;
// sums[0] is kept for the energy estimate.
template <typename T>
__global__ void renormalize_kernel(cx<T>* psi, long long N, const double* __restrict__ sums, double dv) {
    const double s = 1.0 / sqrt(sums[0] * dv);
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N;
         i += (long long)gridDim.x * blockDim.x)
        psi[i] = scale_d(psi[i], s);
}

// |psi|^2 of the plane index `at` along `axis` (0/1/2) of an nx x ny x nz field,
// the other two axes in their own order (first the lower axis), as FP32.
template <typename T>
__global__ void density_slice_kernel(const cx<T>* __restrict__ psi, int nx, int ny, int nz, int axis, int at,
                                     float* out) {
    const int na = axis == 0 ? ny : nx, nb = axis == 2 ? ny : nz;
    const long long cnt = (long long)na * nb;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < cnt;
         t += (long long)gridDim.x * blockDim.x) {
        const int a = (int)(t % na), b = (int)(t / na);
        const int i = axis == 0 ? at : a, j = axis == 0 ? a : (axis == 1 ? at : b), k = axis == 2 ? at : b;
        const cx<double> p = widen(psi[i + (long long)nx * (j + (long long)ny * k)]);
        out[t] = (float)(p.x * p.x + p.y * p.y);
    }
}

// per-axis wavenumbers k_j = (2 pi / L) * (j if 2j < n else j - n)  (spectral.ixx:14-23)
// and kinetic deltas cis(-k^2 dt/(2m)) - 1
__global__ void build_axis_tables(double xmin, double xmax, int n, double dt, double mass,
                                  double* kv, cx<double>* kd) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < n) {
        const double dk = __ddiv_rn(2.0 * 3.14159265358979323846, __dsub_rn(xmax, xmin));
        const int shifted = (2 * j < n) ? j : j - n;
        const double k = __dmul_rn(dk, (double)shifted);
        kv[j] = k;
        kd[j] = cis_minus_one(theta_k(__dmul_rn(k, k), mass, dt));
    }
}

// Per-stage twiddles of a plan, forward order then reversed order: stage (R, Ns)
// holds w^{r k n/(Ns R)} at [r Ns + k], w = e^{-2 pi i/n}, from an FP64 sincospi
// (complex64: hi and the FP32 remainder lo).  Built here, not copied from the host:
// a copy from pageable memory waits for the stream.
struct StageRadices {
    int n, nst;
    int rad[2][kMaxStages];
};

__host__ __device__ inline int stage_entries(const StageRadices& s) {  // both orders
    int total = 0;
    for (int o = 0; o < 2; ++o) {
        int Ns = 1;
        for (int p = 0; p < s.nst; ++p) {
            total += s.rad[o][p] * Ns;
            Ns *= s.rad[o][p];
        }
    }
    return total;
}

template <typename T>
__global__ void build_stage_twiddles(const StageRadices s, int total, cx<T>* hi, cx<T>* lo) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= total) return;
    int i = e;
    for (int o = 0; o < 2; ++o) {
        int Ns = 1;
        for (int p = 0; p < s.nst; ++p) {
            const int R = s.rad[o][p];
            if (i < R * Ns) {
                const int r = i / Ns, k = i - r * Ns;
                const int t = r * k * (s.n / (Ns * R));  // < n
                double sn, cs;
                sincospi(-2.0 * (double)t / (double)s.n, &sn, &cs);
                const cx<T> h = mk<T>((T)cs, (T)sn);
                hi[e] = h;
                if (lo) lo[e] = mk<T>((T)(cs - (double)h.x), (T)(sn - (double)h.y));
                return;
            }
            i -= R * Ns;
            Ns *= R;
        }
    }
}

// Long 1D line of N = N1 N2 points in the four-step layout: the element stored
// at (k1, k2) after the forward transform (flat k1 + N1 k2) is frequency
// k = k2 + N2 k1; its kinetic delta is cis(-k_phys^2 dt/(2m)) - 1 with k_phys the
// line's fftfreq wavenumber kv[k].  The twiddle of element (n1, k2) is
// W_N^{n1 k2} = e^{-2 pi i (n1 k2 mod N)/N}, in FP64 (complex64: hi + lo parts).
template <typename T>
__global__ void build_long_tables(const double* __restrict__ kv, int n1, int n2, double dt, double mass,
                                  cx<T>* kfull, cx<T>* tw_hi, cx<T>* tw_lo) {
    const long long N = (long long)n1 * n2;
    for (long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x; f < N;
         f += (long long)gridDim.x * blockDim.x) {
        const long long a = f % n1, b = f / n1;  // (k1, k2) for kfull, (n1, k2) for the twiddle
        const double k = kv[b + (long long)n2 * a];
        const cx<double> d = cis_minus_one(theta_k(__dmul_rn(k, k), mass, dt));
        kfull[f] = mk<T>((T)d.x, (T)d.y);
        const long long t = (a * b) % N;
        double sn, cs;
        sincospi(-2.0 * (double)t / (double)N, &sn, &cs);
        tw_hi[f] = mk<T>((T)cs, (T)sn);
        if (tw_lo) tw_lo[f] = mk<T>((T)(cs - (double)(T)cs), (T)(sn - (double)(T)sn));
    }
}

// Full-N reference tables (propagator-tables surface).
__global__ void build_full_tables(const double* __restrict__ V, const double* __restrict__ kvx,
                                  const double* __restrict__ kvy, const double* __restrict__ kvz,
                                  int nx, int ny, long long N, double dt, double mass,
                                  cx<double>* half_v, cx<double>* kin) {
    for (long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x; f < N;
         f += (long long)gridDim.x * blockDim.x) {
        double s, c;
        if (half_v) {
            sincos(theta_v(V[f], dt), &s, &c);
            half_v[f] = mk<double>(c, s);
        }
        if (kin) {
            const long long line = f / nx;
            const int i = (int)(f - line * nx);
            const long long k = line / ny;
            const int j = (int)(line - k * ny);
            const double a = kvx[i], b = kvy[j], cz = kvz[k];
            const double ksq = __dadd_rn(__dadd_rn(__dmul_rn(a, a), __dmul_rn(b, b)), __dmul_rn(cz, cz));
            sincos(theta_k(ksq, mass, dt), &s, &c);
            kin[f] = mk<double>(c, s);
        }
    }
}

}  // namespace sesk
