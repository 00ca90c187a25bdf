// Long 1D lines in one launch: the four-step transform of N = N1 N2 points (stored
// N1 x N2, element n1 + N1 n2) with the field held by one thread-block cluster for
// all steps of a call.
//
// CTA c of the CS CTAs owns the columns n1 in [c N1/CS, (c+1) N1/CS) for the length-N2
// transforms and the rows k2 in [c N2/CS, (c+1) N2/CS) for the length-N1 ones.  A step is
//
//   columns: fwd y, * W_N^{n1 k2}   -> rows of their owners (distributed shared memory)
//   rows:    fwd x, K/N, inv x      -> columns of their owners
//   columns: * conj W, inv y, V (M)
//
// with a cluster barrier after each exchange; the columns stay in registers from the
// inverse transform through the kick to the next forward one.  The arithmetic is
// that of the two-launch form (SM_TW_* and XM_1D passes), which stays for batches,
// which fill the chip with many lines, and for lines that a cluster cannot hold.
//
// What bounds it: the latency of two barriers and four line transforms a step, on
// CS of 148 SMs; the field, 512 KB at 65536 points complex64, never leaves them.  The
// two launches it replaces put 8 and 32 CTAs to work and cost 27.8 us a step there,
// this 9.1 on 16 CTAs (16.5 on 8, whose SMs bound it); 8192 points 11.1 -> 3.6.
#pragma once

#include <vector>

#include "ses_plane.cuh"

namespace sesk {

template <typename T, int N1, int E1, int N2, int E2, int CS>
struct LongShape {
    static constexpr int NC = N1 / CS, NR = N2 / CS;  // columns / rows of one CTA
    static constexpr int TL1 = N1 / E1, TL2 = N2 / E2;
    static constexpr int LPW = 32 / TL1;              // rows per warp
    static constexpr int NT = NC * TL2;               // threads: one column element group each
    static constexpr int SH = XPad<N1, E1>::SH, PM = XPad<N1, E1>::PM, PITCH = XPad<N1, E1>::PITCH;
    static constexpr int CP = NC + (sizeof(T) == 4 ? 8 : 0);  // column buffer pitch, as the cluster plane pass
    static constexpr size_t rows_bytes = ((size_t)NR * PITCH * sizeof(cx<T>) + 15) / 16 * 16;
    static constexpr size_t cols_bytes = ((size_t)N2 * CP * sizeof(cx<T>) + 15) / 16 * 16;
    static_assert(N1 % CS == 0 && N2 % CS == 0 && NT % 32 == 0 && NT <= 1024, "cluster tiling");
    static_assert(NR % LPW == 0 && NR * TL1 <= NT, "the rows of a CTA are whole warps of its threads");
    static __device__ __forceinline__ int col(int x) { return x + PM * (x >> SH); }
};

template <typename T, int N1, int E1, int X0, int X1, int X2, int N2, int E2, int Y0, int Y1, int Y2, int CS>
constexpr size_t long_smem() {
    using S = LongShape<T, N1, E1, N2, E2, CS>;
    return S::rows_bytes + S::cols_bytes + TwStage<T, X0, X1, X2>::bytes + TwStage<T, Y0, Y1, Y2>::bytes;
}

// ay: the strided pass's arguments (field, tables, program: d_load, d_mid, m_mid, d_store,
// m_store, y stage twiddles); ax: the x stage twiddles.
template <typename T, int N1, int E1, int X0, int X1, int X2, int N2, int E2, int Y0, int Y1, int Y2, int CS>
__global__ void __launch_bounds__(LongShape<T, N1, E1, N2, E2, CS>::NT, 1)
    long_line_kernel(const PassArgs<T> ay, const PassArgs<T> ax, int steps) {
    using S = LongShape<T, N1, E1, N2, E2, CS>;
    using SY = PlanShape<Y0, Y1, Y2>;
    constexpr bool PK = sizeof(T) == 4;
    constexpr uint32_t ES = sizeof(cx<T>);
    constexpr int YL = SY::last, XL = PlanShape<X0, X1, X2>::last;
    constexpr int TL1 = S::TL1, TL2 = S::TL2;
    extern __shared__ __align__(16) unsigned char smraw[];
    cx<T>* R = reinterpret_cast<cx<T>*>(smraw);
    cx<T>* C = reinterpret_cast<cx<T>*>(smraw + S::rows_bytes);
    cx<T>* twx = reinterpret_cast<cx<T>*>(smraw + S::rows_bytes + S::cols_bytes);
    cx<T>* twy = reinterpret_cast<cx<T>*>(smraw + S::rows_bytes + S::cols_bytes + TwStage<T, X0, X1, X2>::bytes);
    pdl_wait();
    TwStage<T, X0, X1, X2>::load(twx, ax.stw, ax.stwl);
    TwStage<T, Y0, Y1, Y2>::load(twy, ay.stw, ay.stwl);
    const int c = (int)cluster_ctarank();
    uint32_t rb[CS], cb[CS];
#pragma unroll
    for (int o = 0; o < CS; ++o) {
        rb[o] = cluster_map(R, (uint32_t)o);
        cb[o] = cluster_map(C, (uint32_t)o);
    }
    const int l = threadIdx.x % S::NC, q = threadIdx.x / S::NC, n1 = c * S::NC + l;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row = warp * S::LPW + lane / TL1, q1 = lane % TL1;
    const bool has_row = (int)threadIdx.x < S::NR * TL1;  // whole warps
    const int k2row = c * S::NR + row;
    XchCol<T, S::CP> xc{C + l};
    XchWarp<T, S::SH, S::PM> xw{R + row * S::PITCH};
    const Tables& tb = ay.tb;
    const cx<T>* vtab = reinterpret_cast<const cx<T>*>(tb.vtab);
    auto diag = [&](cx<T>(&v)[E2], int kind, int msk) {  // at the last-stage layout of the inverse transform
        if (kind == DG_NONE && !msk) return;
#pragma unroll
        for (int b = 0; b < E2 / YL; ++b)
#pragma unroll
            for (int r = 0; r < YL; ++r) {
                const int f = n1 + N1 * (q + TL2 * b + r * (N2 / YL));
                cx<T>& e = v[b * YL + r];
                e = apply_diag_tv(e, kind, kind != DG_NONE ? vtab[f] : e, msk, msk ? tb.maskfull[f] : 1.0);
            }
    };
    cx<T> v[E2];
#pragma unroll
    for (int b = 0; b < E2 / YL; ++b)
#pragma unroll
        for (int r = 0; r < YL; ++r) v[b * YL + r] = ay.src[n1 + N1 * (q + TL2 * b + r * (N2 / YL))];
    diag(v, ay.d_load, ay.m_load);
    cluster_barrier();  // every CTA runs and has its twiddles
#pragma unroll 1
    for (int s = 0; s < steps; ++s) {
        rfft_plan<T, N2, E2, Y0, Y1, Y2, true, PK>(v, q, twy, twy, xc);
#pragma unroll
        for (int b = 0; b < E2 / Y0; ++b)
#pragma unroll
            for (int r = 0; r < Y0; ++r) {
                const int k2 = q + TL2 * b + r * (N2 / Y0), o = k2 / S::NR;
                st_cluster(pick_base<CS>(rb, o) + (uint32_t)((k2 - o * S::NR) * S::PITCH + S::col(n1)) * ES,
                           tw4_mul<T>(v[b * Y0 + r], tb, n1 + N1 * k2));
            }
        cluster_barrier();
        if (has_row) {
            cx<T> u[E1];
#pragma unroll
            for (int b = 0; b < E1 / X0; ++b)
#pragma unroll
                for (int r = 0; r < X0; ++r) u[b * X0 + r] = xw.get(q1 + TL1 * b + r * (N1 / X0));
            __syncwarp();
            rfft_plan<T, N1, E1, X0, X1, X2, false, PK>(u, q1, twx, twx, xw);
#pragma unroll
            for (int b = 0; b < E1 / XL; ++b)
#pragma unroll
                for (int r = 0; r < XL; ++r)
                    u[b * XL + r] = kinetic_full<T>(u[b * XL + r], tb.kfull,
                                                    (long long)k2row * N1 + q1 + TL1 * b + r * (N1 / XL), tb.kscale);
            rfft_plan<T, N1, E1, X0, X1, X2, true, PK>(u, q1, twx, twx, xw);
#pragma unroll
            for (int b = 0; b < E1 / X0; ++b)
#pragma unroll
                for (int r = 0; r < X0; ++r) {  // the conjugate of the value: the column's inverse starts from it
                    const int x = q1 + TL1 * b + r * (N1 / X0), o = x / S::NC;
                    st_cluster(pick_base<CS>(cb, o) + (uint32_t)(k2row * S::CP + (x - o * S::NC)) * ES, u[b * X0 + r]);
                }
        }
        cluster_barrier();
#pragma unroll
        for (int b = 0; b < E2 / Y0; ++b)
#pragma unroll
            for (int r = 0; r < Y0; ++r) {
                const int k2 = q + TL2 * b + r * (N2 / Y0);
                v[b * Y0 + r] = tw4_mul<T>(xc.get(k2), tb, n1 + N1 * k2);
            }
        __syncthreads();  // the column's other threads have read their inputs before the first exchange
        rfft_plan<T, N2, E2, Y0, Y1, Y2, false, PK>(v, q, twy, twy, xc);
#pragma unroll
        for (int i = 0; i < E2; ++i) v[i] = cconj(v[i]);
        if (s + 1 < steps) diag(v, ay.d_mid, ay.m_mid);
    }
    diag(v, ay.d_store, ay.m_store);
#pragma unroll
    for (int b = 0; b < E2 / YL; ++b)
#pragma unroll
        for (int r = 0; r < YL; ++r) ay.dst[n1 + N1 * (q + TL2 * b + r * (N2 / YL))] = v[b * YL + r];
}

// A compiled long-line kernel and the x and y plans it was built with.
template <typename T>
struct LongEntry {
    int n1 = 0, n2 = 0, cs = 0, nt = 0;
    int xe = 0, xr[3] = {1, 1, 1};
    int ye = 0, yr[3] = {1, 1, 1};
    size_t smem = 0;
    void (*k)(const PassArgs<T>, const PassArgs<T>, int) = nullptr;
    bool usable = false;  // the device can hold such a cluster
};

template <typename T, int N1, int E1, int X0, int X1, int X2, int N2, int E2, int Y0, int Y1, int Y2, int CS>
LongEntry<T> make_long_entry() {
    LongEntry<T> e;
    e.n1 = N1;
    e.n2 = N2;
    e.cs = CS;
    e.nt = LongShape<T, N1, E1, N2, E2, CS>::NT;
    e.xe = E1;
    e.xr[0] = X0;
    e.xr[1] = X1;
    e.xr[2] = X2;
    e.ye = E2;
    e.yr[0] = Y0;
    e.yr[1] = Y1;
    e.yr[2] = Y2;
    e.smem = long_smem<T, N1, E1, X0, X1, X2, N2, E2, Y0, Y1, Y2, CS>();
    e.k = long_line_kernel<T, N1, E1, X0, X1, X2, N2, E2, Y0, Y1, Y2, CS>;
    cudaFuncSetAttribute(e.k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)e.smem);
    if (CS > 8) cudaFuncSetAttribute(e.k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(CS);
    cfg.blockDim = dim3((unsigned)e.nt);
    cfg.dynamicSmemBytes = e.smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CS;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int clusters = 0;
    e.usable = cudaOccupancyMaxActiveClusters(&clusters, e.k, &cfg) == cudaSuccess && clusters > 0;
    cudaGetLastError();
    return e;
}

void register_long_lines(std::vector<LongEntry<float>>& f, std::vector<LongEntry<double>>& d);

}  // namespace sesk
