// Axis passes of run-time plans: any axis length 2^a 3^b 5^c up to 4096 that has no
// compiled plan, the passes of dipole-driven steps, and whole runs of a 1D line.
//
// A length is a product of at most a few radices (two up to 256, three up to 4096
// for most lengths), and a pass is a sequence of stages: each thread takes a
// butterfly of R points into registers, transforms it and hands the points to the
// next stage through shared memory.  Two buffers take turns, so a stage costs one
// barrier and no value lives across it.  The last stage of a transform leaves a
// thread the points j + r n/R -- exactly what the first stage of a transform in the
// reversed radix order reads -- so where a pass runs two transforms (inverse,
// potential, forward; forward, kinetic, inverse) the diagonal multiply between them
// and both neighbouring stages happen in registers.  A line of n = R0 R1 takes two
// trips through shared memory for both its transforms.
//
// What bounds it: latency and instruction issue on fields in L2, HBM from about
// 100 MB on.  A tile is sized to 256 threads and at most 64 KB of buffers, so that
// 2 to 4 CTAs per SM cover each other's barriers (strided tiles keep rows of 64 bytes up to
// 200 KB of buffers: one CTA per SM for lines above 512 points); radices up to 10 run in a kernel
// of their own with 64 registers a thread in complex64.  Against the kernels this
// replaces (radices to 8, one to three more stages, two barriers each, twiddles
// gathered from one table): 120x100x90 complex128 step 190 -> 57 us, a 1024-point
// complex128 line 28.6 -> 5.3 us a step.
#pragma once

#include "ses_pass2.cuh"

namespace sesk {

constexpr int kLineThreads = 256;  // most threads of a CTA

// f(integral_constant<int, R>) for the plan's radix R <= RM (uniform in the CTA).
template <int RM, class F>
__device__ __forceinline__ void with_radix(int R, F&& f) {
    switch (R) {
        case 1: f(std::integral_constant<int, 1>()); break;
        case 2: f(std::integral_constant<int, 2>()); break;
        case 3: f(std::integral_constant<int, 3>()); break;
        case 4: f(std::integral_constant<int, 4>()); break;
        case 5: f(std::integral_constant<int, 5>()); break;
        case 6: f(std::integral_constant<int, 6>()); break;
        case 8: f(std::integral_constant<int, 8>()); break;
        case 9: f(std::integral_constant<int, 9>()); break;
        case 10: f(std::integral_constant<int, 10>()); break;
        case 12:
            if constexpr (RM >= 12) f(std::integral_constant<int, 12>());
            break;
        case 15:
            if constexpr (RM >= 15) f(std::integral_constant<int, 15>());
            break;
        case 16:
            if constexpr (RM >= 16) f(std::integral_constant<int, 16>());
            break;
        default: break;
    }
}

// A pass's arguments and the plan of its axis (kept out of PassArgs, which every other
// kernel takes too).
template <typename T>
struct LineArgs : PassArgs<T> {
    LinePlan g;
};

// Contiguous tiles: line l at l * pitch, one spare element after every 16, which
// spreads the writes of a first stage (R apart) over the banks.
__host__ __device__ constexpr int line_pad(int pos) { return pos + (pos >> 4); }

// The transforms of a tile.  CONTIG: butterflies run along the lines (consecutive
// threads, consecutive points), else across them (consecutive threads, consecutive
// lines).  rev: the first transform runs in the reversed radix order.  nmid: the
// number of times that cross<R>(i, l, j, nR, v) turns the end of a transform into the
// start of the next (i = 0 .. nmid - 1), each in the other order.  load<R> gives the
// first inputs, store<R> takes the last outputs: the R points j + r nR of line l at
// once, so that their loads leave together (one at a time behind the tests of a
// general kick, the 120x100x90 complex128 x pass took 39 us, this 28).
//
// The tile's shared memory: the pass's arguments (indexed at run time by the stages),
// then the two exchange buffers of g.buf.
template <typename T>
constexpr size_t line_args_bytes() {
    return (sizeof(LineArgs<T>) + 15) / 16 * 16;
}
__device__ __forceinline__ unsigned char* line_smem() {
    extern __shared__ __align__(16) unsigned char smraw[];
    return smraw;
}
template <typename T>
__device__ __forceinline__ const LineArgs<T>& line_args() {
    return *reinterpret_cast<const LineArgs<T>*>(line_smem());
}
template <typename T>
__device__ __forceinline__ cx<T>* line_bufs() {
    return reinterpret_cast<cx<T>*>(line_smem() + line_args_bytes<T>());
}
// Copies the arguments in and waits for the previous kernel of the stream.
template <typename T>
__device__ __forceinline__ void line_begin(const LineArgs<T>& args) {
    static_assert(sizeof(LineArgs<T>) % 4 == 0, "copied by words");
    const uint32_t* from = reinterpret_cast<const uint32_t*>(&args);
    uint32_t* to = reinterpret_cast<uint32_t*>(line_smem());
    for (int i = threadIdx.x; i < (int)(sizeof(LineArgs<T>) / 4); i += blockDim.x) to[i] = from[i];
    pdl_wait();
    __syncthreads();
}

struct LineStage {
    int o, p;          // radix order and stage in it
    int done, here;    // crossings before this stage, and made by it
    bool first, final; // the pass's first / last stage
    int turn;          // the exchange buffer it writes
};

template <class P, int R>
__device__ __forceinline__ void line_stage(P& pass, const LineStage c) {
    using T = typename P::type;
    constexpr bool CONTIG = P::kContig;
    const LineArgs<T>& a = line_args<T>();
    const LinePlan& g = a.g;
    cx<T>* bufs = line_bufs<T>();
    const int n = g.n, nR = n / R;
    const int nb = g.L * nR;
    const int Ns = g.Ns[c.o][c.p];
    const cx<T>* th = a.stw + g.toff[c.o][c.p];
    const cx<T>* tl = sizeof(T) == 4 ? a.stwl + g.toff[c.o][c.p] : nullptr;
    const cx<T>* from = bufs + (c.turn ^ 1) * g.buf;
    cx<T>* to = bufs + c.turn * g.buf;
#pragma unroll 1
    for (int b = (int)threadIdx.x; b < nb; b += (int)blockDim.x) {
        int l, j;
        if constexpr (CONTIG) {
            l = (int)fdiv((uint32_t)b, g.fnR[c.o][c.p]);
            j = b - l * nR;
        } else {
            l = b & (g.L - 1);
            j = b >> g.lshift;
        }
        cx<T> v[R];
        int k = 0;
        if (c.first) {
            pass.template load<R>(l, j, nR, v);
        } else {
            k = j - (int)fdiv((uint32_t)j, g.fNs[c.o][c.p]) * Ns;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int pos = j + r * nR;
                v[r] = CONTIG ? from[l * g.pitch + line_pad(pos)] : from[(pos << g.lshift) + l];
            }
#pragma unroll
            for (int r = 1; r < R; ++r) v[r] = twmul<T>(v[r], th, tl, r * Ns + k);
        }
        dft<T, R>(v);
#pragma unroll 1
        for (int i = 0; i < c.here; ++i) {
            pass.template cross<R>(c.done + i, l, j, nR, v);
            dft<T, R>(v);
        }
        if (c.final) {
            pass.template store<R>(l, j, nR, v);
        } else {  // a crossing's second half is the first stage of its transform (Ns = 1)
            const int base = c.here ? j * R : (j - k) * R + k;
            const int step = c.here ? 1 : Ns;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int pos = base + r * step;
                if constexpr (CONTIG) to[l * g.pitch + line_pad(pos)] = v[r];
                else to[(pos << g.lshift) + l] = v[r];
            }
        }
    }
}

template <int RM, class P>
__device__ __forceinline__ void line_transforms(P& pass, bool rev, int nmid) {
    const LinePlan& g = line_args<typename P::type>().g;
    const int nst = g.nst;
    LineStage c{rev ? 1 : 0, 0, 0, 0, true, false, 0};
    for (;;) {
        const bool last = c.p == nst - 1;
        // single-stage plans make every crossing here, others one per transform's end
        c.here = last ? (nst == 1 ? nmid - c.done : (c.done < nmid ? 1 : 0)) : 0;
        c.final = last && (nst == 1 || c.done == nmid);
        with_radix<RM>(g.rad[c.o][c.p], [&](auto rc) { line_stage<P, decltype(rc)::value>(pass, c); });
        if (c.final) return;
        __syncthreads();
        c.done += c.here;
        c.turn ^= 1;
        c.first = false;
        if (c.here) {
            c.o ^= 1;
            c.p = 1;
        } else {
            ++c.p;
        }
    }
}

// The dipole kick of a cell: cis(-theta (a . r)) as the product of three per-axis
// factors, read from the step's FP64 table (x, then y, then z entries; kick_factors in
// ses_aux.cuh): cis for complex128, cis - 1 for complex64, whose product is rounded to
// FP32 as a delta.
template <typename T>
__device__ __forceinline__ cx<double> kick_times(cx<double> a, cx<double> b) {
    if constexpr (sizeof(T) == 4) return dmul1(a, b);
    else return a * b;
}

// Potential (KIND), absorber (MASK: mrow[r nR] * myz) and dipole kick on the R points
// j + r nR of a line, straight-line code.
template <typename T, bool KICK, int KIND, bool MASK, int R>
__device__ __forceinline__ void line_diag_as(const cx<T>* tab, const double* mrow, double myz, const cx<double>* kx,
                                             cx<double> kyz, int nR, cx<T> (&v)[R]) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
        cx<T> t = v[r];
        if constexpr (KIND != DG_NONE) t = tab[r * nR];
        double m = 1.0;
        if constexpr (MASK) m = mrow[r * nR] * myz;
        v[r] = apply_diag_tv(v[r], KIND, t, MASK ? 1 : 0, m);
        if constexpr (KICK) {
            const cx<double> f = kick_times<T>(kx[r * nR], kyz);
            if constexpr (sizeof(T) == 4) v[r] = add_mul(v[r], narrow<float>(f));
            else v[r] = v[r] * f;
        }
    }
}

// The same for line (y, z) = (jy, kz) whose first point is flat index f0, the tests of
// the pass's program (kind, mask) made once per butterfly.
template <typename T, bool KICK, int R>
__device__ __forceinline__ void line_diag(const LineArgs<T>& a, int kind, int msk, long long f0, int j, int nR, int jy,
                                          int kz, cx<T> (&v)[R]) {
    const Tables& tb = a.tb;
    const cx<T>* tab = reinterpret_cast<const cx<T>*>(tb.vtab) + f0 + j;
    const double* mrow = nullptr;
    double myz = 1.0;
    if (msk) {
        mrow = tb.maskfull ? tb.maskfull + f0 + j : tb.mask1[0] + j;
        if (!tb.maskfull) myz = tb.mask1[1][jy] * tb.mask1[2][kz];
    }
    const cx<double>* kx = nullptr;
    cx<double> kyz = mk<double>(0.0, 0.0);
    if constexpr (KICK) {
        kx = tb.kick + j;
        kyz = kick_times<T>(tb.kick[a.nx + jy], tb.kick[a.nx + a.ny + kz]);
    }
    if (kind == DG_FULL) {
        if (msk) line_diag_as<T, KICK, DG_FULL, true, R>(tab, mrow, myz, kx, kyz, nR, v);
        else line_diag_as<T, KICK, DG_FULL, false, R>(tab, mrow, myz, kx, kyz, nR, v);
    } else if (kind == DG_HALF) {
        if (msk) line_diag_as<T, KICK, DG_HALF, true, R>(tab, mrow, myz, kx, kyz, nR, v);
        else line_diag_as<T, KICK, DG_HALF, false, R>(tab, mrow, myz, kx, kyz, nR, v);
    } else {
        if (msk) line_diag_as<T, KICK, DG_NONE, true, R>(tab, mrow, myz, kx, kyz, nR, v);
        else line_diag_as<T, KICK, DG_NONE, false, R>(tab, mrow, myz, kx, kyz, nR, v);
    }
}

template <typename T, int RM>
constexpr int line_min_ctas() {  // CTAs per SM the register allocation is sized for
    // complex128: 120x100x90 step 61 us with 2 (128 registers), 71 with 3 (80, spilling);
    // complex64: 128-point x passes with radix 16 on 3, radix 10 on 4, 6 to 27% faster than on 2
    return sizeof(T) == 8 ? 2 : (RM > 10 ? 3 : 4);
}

// The contiguous pass of a tile, modes as in XMode.
template <typename T, int MODE, bool KICK>
struct LineX {
    using type = T;
    static constexpr bool kContig = true;
    long long m0;  // first line of the tile
    double acc[kRedK];

    // coordinates of line l; lines past the end work on line 0
    __device__ __forceinline__ long long line(int l, int* j, int* k) const {
        const LineArgs<T>& a = line_args<T>();
        const long long m = m0 + l < a.nlines ? m0 + l : 0;
        *k = (int)fdiv((uint32_t)m, a.fny);
        *j = (int)(m - (long long)*k * a.ny);
        return m;
    }
    template <int R>
    __device__ __forceinline__ void diag(int kind, int msk, int l, int j, int nR, cx<T> (&v)[R]) const {
        const LineArgs<T>& a = line_args<T>();
        if (kind == DG_NONE && !msk && !KICK) return;
        int jy, kz;
        const long long m = line(l, &jy, &kz);
        line_diag<T, KICK, R>(a, kind, msk, m * a.g.n, j, nR, jy, kz, v);
    }
    template <int R>
    static __device__ __forceinline__ void conj_all(cx<T> (&v)[R]) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = cconj(v[r]);
    }
    template <int R>
    __device__ __forceinline__ void load(int l, int j, int nR, cx<T> (&v)[R]) {
        const LineArgs<T>& a = line_args<T>();
        const long long m = m0 + l < a.nlines ? m0 + l : 0;
        const cx<T>* src = a.src + m * a.g.n + j;
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = src[r * nR];
        if constexpr (MODE == XM_INV || MODE == XM_MID || MODE == XM_END) conj_all<R>(v);
        if constexpr (MODE == XM_START || MODE == XM_1D) diag<R>(a.d_load, a.m_load, l, j, nR, v);
    }
    template <int R>
    __device__ __forceinline__ void cross(int i, int l, int j, int nR, cx<T> (&v)[R]) {
        const LineArgs<T>& a = line_args<T>();
        if (MODE == XM_MID || (MODE == XM_1D && (i & 1))) {
            conj_all<R>(v);
            diag<R>(a.d_mid, a.m_mid, l, j, nR, v);
        } else if constexpr (MODE == XM_1D) {
            int jy, kz;
            line(l, &jy, &kz);
            const cx<double> dyz = dmul1(a.tb.kd[1][jy], a.tb.kd[2][kz]);
#pragma unroll
            for (int r = 0; r < R; ++r)
                v[r] = kinetic_apply(v[r], dyz, a.tb.kd[0], a.tb.kdf[0], j + r * nR, a.tb.kscale);
        }
    }
    template <int R>
    __device__ __forceinline__ void store(int l, int j, int nR, cx<T> (&v)[R]) {
        const LineArgs<T>& a = line_args<T>();
        if constexpr (MODE == XM_REDUCE) {
            if (m0 + l >= a.nlines) return;
            int jy, kz;
            line(l, &jy, &kz);
            const double ky = a.tb.kv[1][jy], kzv = a.tb.kv[2][kz];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const double k3[3] = {a.tb.kv[0][j + r * nR], ky, kzv};
                const cx<double> w = widen(v[r]);
                acc_k(acc, w.x * w.x + w.y * w.y, k3, a.tb.inv_mass);
            }
            return;
        }
        if constexpr (MODE == XM_INV) {
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = scale_d(cconj(v[r]), a.out_scale);
        }
        if constexpr (MODE == XM_END || MODE == XM_1D) {
            conj_all<R>(v);
            diag<R>(a.d_store, a.m_store, l, j, nR, v);
        }
        if (m0 + l < a.nlines) {
            cx<T>* dst = a.dst + (m0 + l) * a.g.n + j;
#pragma unroll
            for (int r = 0; r < R; ++r) dst[r * nR] = v[r];
        }
    }
};

// XM_1D runs `steps` steps of 1D lines in one launch: [d_load] fwd, K/N, inv {[d_mid]
// fwd, K/N, inv} ... [d_store], the field in registers and shared memory from the
// first load to the last store.
template <typename T, int MODE, int RM, bool KICK>
__global__ void __launch_bounds__(kLineThreads, (MODE == XM_1D || MODE == XM_REDUCE) ? 1 : line_min_ctas<T, RM>())
    line_x_kernel(const __grid_constant__ LineArgs<T> args, int steps) {
    line_begin(args);
    const LineArgs<T>& a = line_args<T>();
    LineX<T, MODE, KICK> pass{(long long)blockIdx.x * a.g.L, {0, 0, 0, 0, 0}};
    line_transforms<RM>(pass, MODE == XM_START, MODE == XM_MID ? 1 : (MODE == XM_1D ? 2 * steps - 1 : 0));
    if constexpr (MODE == XM_REDUCE) block_reduce_store<kRedK>(pass.acc, a.partials);
}

// The strided (y or z) pass of a tile, modes as in SModeK (SM_FWD, SM_INV, SM_FUSED,
// SM_REDUCE).  blockDim is a multiple of L: a thread stays on one line of the tile.
template <typename T, int MODE>
struct LineS {
    using type = T;
    static constexpr bool kContig = false;
    bool valid;
    long long base;  // of the thread's line (line 0 past the end)
    int c1, c2;      // the line's other two coordinates: y-pass (x, z), z-pass (x, y)
    double acc[kRedK];

    template <int R>
    __device__ __forceinline__ void load(int, int j, int nR, cx<T> (&v)[R]) {
        const LineArgs<T>& a = line_args<T>();
        const cx<T>* src = a.src + base + j * a.se;
        const long long step = nR * a.se;
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = src[r * step];
        if constexpr (MODE == SM_INV) {
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = cconj(v[r]);
        }
    }
    template <int R>
    __device__ __forceinline__ void cross(int, int, int j, int nR, cx<T> (&v)[R]) {
        const LineArgs<T>& a = line_args<T>();
        if constexpr (MODE == SM_FUSED) {
            const bool ypass = a.axis == 1;
            const cx<double>* kda = ypass ? a.tb.kd[1] : a.tb.kd[2];
            const cx<float>* kdaf = ypass ? a.tb.kdf[1] : a.tb.kdf[2];
            const cx<double> dother = dmul1(a.tb.kd[0][c1], ypass ? a.tb.kd[2][c2] : a.tb.kd[1][c2]);
            const double kscale = a.tb.kscale;
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = kinetic_apply(v[r], dother, kda, kdaf, j + r * nR, kscale);
        }
    }
    template <int R>
    __device__ __forceinline__ void store(int, int j, int nR, cx<T> (&v)[R]) {
        const LineArgs<T>& a = line_args<T>();
        if (!valid) return;
        if constexpr (MODE == SM_REDUCE) {
            const bool ypass = a.axis == 1;
            const double* kva = ypass ? a.tb.kv[1] : a.tb.kv[2];
            const double k1 = a.tb.kv[0][c1], k2 = ypass ? a.tb.kv[2][c2] : a.tb.kv[1][c2];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const double ka = kva[j + r * nR];
                const double k3[3] = {k1, ypass ? ka : k2, ypass ? k2 : ka};
                const cx<double> w = widen(v[r]);
                acc_k(acc, w.x * w.x + w.y * w.y, k3, a.tb.inv_mass);
            }
            return;
        }
        cx<T>* dst = a.dst + base + j * a.se;
        const long long step = nR * a.se;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if constexpr (MODE == SM_INV) v[r] = scale_d(cconj(v[r]), a.out_scale);
            if constexpr (MODE == SM_FUSED) v[r] = cconj(v[r]);
            dst[r * step] = v[r];
        }
    }
};

template <typename T, int MODE, int RM>
__global__ void __launch_bounds__(kLineThreads, MODE == SM_REDUCE ? 1 : line_min_ctas<T, RM>())
    line_s_kernel(const __grid_constant__ LineArgs<T> args) {
    line_begin(args);
    const LineArgs<T>& a = line_args<T>();
    const long long s = (long long)blockIdx.x * a.g.L + (threadIdx.x & (a.g.L - 1));
    const bool valid = s < a.nlines;
    const long long sc_ = valid ? s : 0;
    const long long w = (long long)fdiv((uint32_t)sc_, a.fnu);
    const long long u = sc_ - w * a.nu;
    int c1 = (int)u, c2 = (int)w;
    if (a.axis != 1) {
        c2 = (int)fdiv((uint32_t)u, a.fnx);
        c1 = (int)(u - (long long)c2 * a.nx);
    }
    LineS<T, MODE> pass{valid, u + w * a.sw, c1, c2, {0, 0, 0, 0, 0}};
    line_transforms<RM>(pass, false, MODE == SM_FUSED ? 1 : 0);
    if constexpr (MODE == SM_REDUCE) block_reduce_store<kRedK>(pass.acc, a.partials);
}

template <typename T>
using LineXKernel = void (*)(const LineArgs<T>, int);
template <typename T>
using LineSKernel = void (*)(const LineArgs<T>);

// The kernel of a mode for plans of radices up to rmax (ses_line_c64.cu, ses_line_c128.cu);
// kick: the modes that apply the potential in driven steps.
template <typename T>
LineXKernel<T> line_x(int mode, int rmax, bool kick);
template <typename T>
LineSKernel<T> line_s(int mode, int rmax);

}  // namespace sesk
