// Strided passes with warp-owned lines: TMA in, transforms inside a warp, TMA out.
//
// A CTA holds a ring of tiles (L lines of N points, one row of L points per position),
// one producer thread and groups of warps that take the tiles in turn.  The producer
// loads a tile with swizzled TMA boxes, waits until the tile's warps have put their
// results back into it, stores it with TMA and reloads the buffer.  A warp owns whole
// lines: it waits for its tile, transforms in registers, exchanges between stages
// through its own lines' slots with __syncwarp only, and moves on -- no CTA barrier,
// so warps run at different phases of different tiles and loads, arithmetic and stores
// overlap across the whole ring.
//
// Bank conflicts: a tile row is 64 or 128 bytes, and the swizzle puts a 16-byte chunk
// of rows r .. r + 7 (r % 8 == 0) on 8 different chunk positions.  A phase of a warp's
// access covers one chunk of 8 rows, so it is free of conflicts when the 8 rows differ
// in their low three bits: rows in order at the load and store; position p of an
// exchange after a stage of radix R is kept in row p ^ ((p / R) mod 8), which has
// that property for the writes (R apart) and the reads (in order).  Both maps are
// linear over XOR, so a thread's row address is one XOR of a constant, and eight such
// values serve all its elements.
//
// What bounds it: HBM for the plain transforms (256^3 complex64: 268 MB in 46 us, 5.8
// TB/s), issue for the fused pass, whose two transforms cost about 90 instructions a
// point.  us, the fastest CTA-wide tile of ses_pass3.cuh (or the register path) ->
// this, forward y / fused z: complex64 256^3 55 -> 46 / 86 -> 64, 512^3 390 -> 400 /
// 788 -> 705, six fields of 128^3 41.5 -> 41 / 60.5 -> 52; complex128 256^3 99 -> 95 /
// 143 -> 108, six of 128^3 74.5 -> 69 / 121 -> 85.  Rows of 64 bytes and 12 to 16 warps
// for the 256-point lines, 128 bytes for shorter ones (rows of 64 at 128 points: y 15.8
// against 12.3); for the 512-point ones two groups of four warps hold 32 points a thread.
#pragma once

#include "ses_pass3.cuh"

namespace sesk {

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, int c0, int c1, uint32_t src) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(map), "r"(c0),
                 "r"(c1), "r"(src)
                 : "memory");
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, int c0, int c1, int c2, uint32_t src) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(map),
                 "r"(c0), "r"(c1), "r"(c2), "r"(src)
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int K>
__device__ __forceinline__ void bulk_wait_read() {  // all but the K newest groups have read their source
    asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(K) : "memory");
}
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// Shape of a pass: tile rows of RB bytes, NG groups of warps, NBUF tiles in the ring.
template <typename T, int N, int E, int R0, int R1, int RB, int NG, int NBUF>
struct Pass4Shape {
    static constexpr int TL = N / E;                      // threads per line
    static constexpr int L = RB / (int)sizeof(cx<T>);     // lines per tile
    static constexpr int LPW = 32 / TL;                   // lines per warp
    static constexpr int WT = L / LPW;                    // warps per tile
    static constexpr int NT = (WT * NG + 1) * 32;         // threads: the groups and the producer's warp
    static constexpr uint32_t TILE = (uint32_t)N * RB;
    static constexpr size_t tw_off = (size_t)NBUF * TILE;
    static constexpr size_t kd_off = tw_off + TwStage<T, R0, R1, 1>::bytes;  // the axis's kinetic deltas
    static constexpr size_t bar_off = kd_off + (size_t)N * sizeof(cx<T>);
    static constexpr size_t smem = bar_off + 2 * NBUF * 8;
    static_assert(RB == 64 || RB == 128, "the swizzles used");
    // A buffer always belongs to the same group, whose warps have then seen the buffer's
    // previous load: a wait by phase parity could otherwise take a load that is still in
    // flight, two phases back, for the one it waits for.
    static_assert(NBUF % NG == 0, "whole rounds of the groups in the ring");
    static_assert((N & (N - 1)) == 0 && TL >= 8 && TL <= 16 && R0 * R1 == N && R0 >= 8 && R1 >= 8, "two-stage plans");
    static_assert(L % LPW == 0 && (sizeof(T) == 8 || LPW % 2 == 0), "a warp's lines fill 16-byte chunks");
    static_assert(smem <= 227 * 1024, "shared memory");
};

// Byte offset of row `slot` in a tile without its line part (the swizzle's chunk bits
// are XORed with the line's chunk).
template <int RB>
__host__ __device__ constexpr uint32_t row4(uint32_t slot) {
    return slot * RB ^ ((RB == 64 ? (slot >> 1) & 3u : slot & 7u) << 4);
}
__host__ __device__ constexpr int log2c(int x) { return x <= 1 ? 0 : 1 + log2c(x / 2); }

template <typename T>
__device__ __forceinline__ cx<T> lds4(const unsigned char* sm, uint32_t off) {
    return *reinterpret_cast<const cx<T>*>(sm + off);
}
template <typename T>
__device__ __forceinline__ void sts4(unsigned char* sm, uint32_t off, cx<T> v) {
    *reinterpret_cast<cx<T>*>(sm + off) = v;
}

// Exchange between a stage of radix RP (the first: its outputs are positions j RP + r,
// j = q + TL b) and one of radix RN (inputs j + r N/RN).  kp, kg: the thread's row
// addresses of positions q RP and q.
template <typename T, int N, int E, int RP, int RN, int RB>
__device__ __forceinline__ void exchange4(cx<T> (&v)[E], unsigned char* sm, uint32_t kp, uint32_t kg) {
    constexpr int TL = N / E;
    constexpr int S = log2c(RP);
#pragma unroll
    for (int b = 0; b < E / RP; ++b)
#pragma unroll
        for (int r = 0; r < RP; ++r)
            sts4(sm, (kp ^ row4<RB>(r & 7)) + (uint32_t)((b * TL * RP + (r & ~7)) * RB), v[b * RP + r]);
    __syncwarp();
#pragma unroll
    for (int b = 0; b < E / RN; ++b)
#pragma unroll
        for (int r = 0; r < RN; ++r) {
            const int c = TL * b + r * (N / RN);
            v[b * RN + r] = lds4<T>(sm, (kg ^ row4<RB>((c >> S) & 7)) + (uint32_t)(c * RB));
        }
    __syncwarp();
}

template <typename T, int MODE, int N, int E, int R0, int R1, int RB, int NG, int NBUF, class F>
__device__ __forceinline__ void spass4_body(const F& f, const PipeArgs& pa) {
    using P = Pass4Shape<T, N, E, R0, R1, RB, NG, NBUF>;
    using S = PlanShape<R0, R1, 1>;
    using TW = TwStage<T, R0, R1, 1>;
    constexpr bool PK = sizeof(T) == 4;
    constexpr int TL = P::TL, L = P::L, WT = P::WT;
    constexpr int EW = (int)sizeof(cx<T>) / 8;
    extern __shared__ __align__(1024) unsigned char smraw4[];
    const cx<T>* tw = reinterpret_cast<const cx<T>*>(smraw4 + P::tw_off);
    const cx<T>* kds = reinterpret_cast<const cx<T>*>(smraw4 + P::kd_off);
    uint64_t* full = reinterpret_cast<uint64_t*>(smraw4 + P::bar_off);
    uint64_t* done = full + NBUF;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nmine = blockIdx.x < (unsigned)pa.ntiles ? (pa.ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    if (threadIdx.x == 0) {
        for (int b = 0; b < NBUF; ++b) {
            mbar_init(smem_u32(&full[b]), 1);
            mbar_init(smem_u32(&done[b]), WT);
        }
        fence_mbar_init();
    }
    if (nmine > 0) {
        const PassArgs<T>& a = f.args(blockIdx.x);
        TW::load(reinterpret_cast<cx<T>*>(smraw4 + P::tw_off), a.stw, a.stwl);
        if constexpr (MODE == SM_FUSED && !F::kMany) {  // members of a class may differ in theirs
            const cx<T>* kd;
            if constexpr (sizeof(T) == 4) kd = a.tb.kdf[a.axis];
            else kd = a.tb.kd[a.axis];
            cx<T>* to = reinterpret_cast<cx<T>*>(smraw4 + P::kd_off);
            for (int i = threadIdx.x; i < N; i += blockDim.x) to[i] = kd[i];
        }
    }
    __syncthreads();

    if (warp == WT * NG) {  // the producer
        if (lane != 0) return;
        auto coords = [&](int i, const CUtensorMap** map, int* x, int* z) {
            const uint32_t t = blockIdx.x + (uint32_t)i * gridDim.x;
            const int s0 = (int)f.local(t) * L;
            *map = f.tmap(t);
            if (pa.kind == 0) {
                const int nx = f.args(t).nx;
                *z = s0 / nx;
                *x = (s0 - *z * nx) * EW;
            } else {
                *z = 0;
                *x = s0 * EW;
            }
        };
        auto load = [&](int i) {
            const int buf = i % NBUF;
            const CUtensorMap* map;
            int x, z;
            coords(i, &map, &x, &z);
            const uint32_t bar = smem_u32(&full[buf]), dst = smem_u32(smraw4) + (uint32_t)buf * P::TILE;
            mbar_expect_tx(bar, P::TILE + pa.extra_tx);
            for (int bx = 0; bx < pa.nbox; ++bx) {
                const uint32_t d = dst + (uint32_t)(bx * pa.rows_per_box * RB);
                if (pa.kind == 0) tma_load_3d(d, map, x, bx * pa.rows_per_box, z, bar);
                else tma_load_2d(d, map, x, bx * pa.rows_per_box, bar);
            }
        };
        for (int i = 0; i < NBUF && i < nmine; ++i) load(i);
        for (int i = 0; i < nmine; ++i) {
            const int buf = i % NBUF;
            // the tile's warps give up after wait_limit: twice that covers them
            const long long lim = 2 * (pa.wait_limit > 0 ? pa.wait_limit : kWaitLimitCycles);
            if (!mbar_wait(smem_u32(&done[buf]), (uint32_t)((i / NBUF) & 1), lim)) {
                atomicOr(pa.err, 1u);
                // drain the loads in flight, a tile each (bounded: 50 ms is far beyond a load's time)
                const long long drain = lim < 100000000LL ? lim : 100000000LL;
                for (int j = i; j < nmine && j < i + NBUF; ++j)
                    (void)mbar_wait(smem_u32(&full[j % NBUF]), (uint32_t)((j / NBUF) & 1), drain);
                break;
            }
            const CUtensorMap* map;
            int x, z;
            coords(i, &map, &x, &z);
            const uint32_t src = smem_u32(smraw4) + (uint32_t)buf * P::TILE;
            for (int bx = 0; bx < pa.nbox; ++bx) {
                const uint32_t s = src + (uint32_t)(bx * pa.rows_per_box * RB);
                if (pa.kind == 0) tma_store_3d(map, x, bx * pa.rows_per_box, z, s);
                else tma_store_2d(map, x, bx * pa.rows_per_box, s);
            }
            bulk_commit();
            if (i >= 1 && i - 1 + NBUF < nmine) {  // the previous tile's buffer, once its store has read it
                bulk_wait_read<1>();
                load(i - 1 + NBUF);
            }
        }
        bulk_wait_all();
        return;
    }

    const int group = warp / WT;
    // complex64: the two lines of a 16-byte chunk sit on neighbouring lanes
    const int lw = sizeof(T) == 4 ? (lane & 1) + 2 * (lane / (2 * TL)) : lane / TL;
    const int q = sizeof(T) == 4 ? (lane >> 1) % TL : lane % TL;
    const int line = (warp % WT) * P::LPW + lw;
    const uint32_t lpart = (uint32_t)(line * (int)sizeof(cx<T>));  // chunk and word of the line
    const uint32_t kg0 = row4<RB>((uint32_t)q) ^ lpart;
    const uint32_t kp0 = row4<RB>((uint32_t)(q * R0) ^ (uint32_t)(q & 7)) ^ lpart;
    const uint32_t kr0 = row4<RB>((uint32_t)(q * R1) ^ (uint32_t)(q & 7)) ^ lpart;
    for (int i = group; i < nmine; i += NG) {
        const int buf = i % NBUF;
        const uint32_t t = blockIdx.x + (uint32_t)i * gridDim.x;
        const PassArgs<T>& a = f.args(t);
        const uint32_t off = (uint32_t)buf * P::TILE;
        const uint32_t kg = off + kg0, kp = off + kp0, kr = off + kr0;
        cx<double> dother = mk<double>(0.0, 0.0);
        const bool ypass = a.axis == 1;
        if constexpr (MODE == SM_FUSED) {
            const long long s = f.local(t) * L + line;
            const long long sc = s < a.nlines ? s : 0;
            const long long w = (long long)fdiv((uint32_t)sc, a.fnu);
            const long long u = sc - w * a.nu;
            int c1 = (int)u, c2 = (int)w;
            if (!ypass) {
                c2 = (int)fdiv((uint32_t)u, a.fnx);
                c1 = (int)(u - (long long)c2 * a.nx);
            }
            dother = dmul1(a.tb.kd[0][c1], ypass ? a.tb.kd[2][c2] : a.tb.kd[1][c2]);
        }
        if (!mbar_wait(smem_u32(&full[buf]), (uint32_t)((i / NBUF) & 1), pa.wait_limit)) {
            if (lane == 0) atomicOr(pa.err, 1u);
            return;
        }
        cx<T> v[E];
#pragma unroll
        for (int b = 0; b < E / R0; ++b)
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                const cx<T> e = lds4<T>(smraw4, kg + (uint32_t)((TL * b + r * (N / R0)) * RB));
                v[b * R0 + r] = MODE == SM_INV ? cconj(e) : e;
            }
        __syncwarp();  // the lines are reused for the exchanges
        rstage<T, N, E, TL, R0, 1, 0, PK>(v, q, tw, tw);
        exchange4<T, N, E, R0, R1, RB>(v, smraw4, kp, kg);
        rstage<T, N, E, TL, R1, R0, R0, PK>(v, q, tw, tw);
        if constexpr (MODE == SM_FUSED) {
            const cx<double>* kda = a.tb.kd[a.axis];
            const cx<float>* kdaf = a.tb.kdf[a.axis];
            if constexpr (!F::kMany) {
                if constexpr (sizeof(T) == 4) kdaf = kds;
                else kda = kds;
            }
#pragma unroll
            for (int b = 0; b < E / R1; ++b)
#pragma unroll
                for (int r = 0; r < R1; ++r)
                    v[b * R1 + r] = kinetic_apply(v[b * R1 + r], dother, kda, kdaf, q + TL * b + r * (N / R1), a.tb.kscale);
            rstage<T, N, E, TL, R1, 1, S::fwd_tables, PK>(v, q, tw, tw);
            exchange4<T, N, E, R1, R0, RB>(v, smraw4, kr, kg);
            rstage<T, N, E, TL, R0, R1, S::fwd_tables + R1, PK>(v, q, tw, tw);
#pragma unroll
            for (int b = 0; b < E / R0; ++b)
#pragma unroll
                for (int r = 0; r < R0; ++r)
                    sts4(smraw4, kg + (uint32_t)((TL * b + r * (N / R0)) * RB), cconj(v[b * R0 + r]));
        } else {
#pragma unroll
            for (int b = 0; b < E / R1; ++b)
#pragma unroll
                for (int r = 0; r < R1; ++r) {
                    cx<T> e = v[b * R1 + r];
                    if constexpr (MODE == SM_INV) e = scale_d(cconj(e), a.out_scale);
                    sts4(smraw4, kg + (uint32_t)((TL * b + r * (N / R1)) * RB), e);
                }
        }
        fence_proxy_async_smem();  // this lane's results before the tile's TMA store
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&done[buf]));
    }
}

template <typename T, int MODE, int N, int E, int R0, int R1, int RB, int NG, int NBUF>
__global__ void __launch_bounds__(Pass4Shape<T, N, E, R0, R1, RB, NG, NBUF>::NT, 1)
    spass4_kernel(const __grid_constant__ PassArgs<T> a, const __grid_constant__ CUtensorMap tmap, const PipeArgs pa) {
    pdl_wait();
    spass4_body<T, MODE, N, E, R0, R1, RB, NG, NBUF>(OneField<T>{a, &tmap}, pa);
}

// The fields of one shape class, per-instance arguments and tensor maps in global memory.
template <typename T, int MODE, int N, int E, int R0, int R1, int RB, int NG, int NBUF>
__global__ void __launch_bounds__(Pass4Shape<T, N, E, R0, R1, RB, NG, NBUF>::NT, 1)
    sbatch4_kernel(const PassArgs<T>* __restrict__ args, const CUtensorMap* maps, const BatchWork w, const PipeArgs pa) {
    pdl_wait();
    spass4_body<T, MODE, N, E, R0, R1, RB, NG, NBUF>(ManyFields<T>{args, maps, w}, pa);
}

}  // namespace sesk
