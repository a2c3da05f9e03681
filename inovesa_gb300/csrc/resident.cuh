// k_bres: many solver steps of chain-0 bunches in one launch, the density
// on the chip from the first step to the last (included by batch.cu after
// ring_fast.cuh; the lattices are those of k_bmaps0f, F_Y7, up to 256
// rows, bunches on their own).
//
// A thread-block cluster of C CTAs owns one bunch; CTA `rank` owns the R =
// N / C mesh rows from rank * R on, in shared memory twice: T, the density,
// and K, the rows after the y-kick with the halo rows of the neighbours.
// One step is
//
//   wake      every warp sums the wake of its own rows from the profile P
//             in shared memory (lane = N/32 source cells, one register
//             window of the Toeplitz table, sums by reduce-scatter) and
//             builds their composite 7-tap y-kick;
//   y-kick    T -> K, 8 columns per lane; at the edges of the CTA's rows
//             also into the neighbours' K;
//   drift, Fokker-Planck   K -> T, 4 columns per lane, a sliding window of
//             4 rows; the rows' Simpson sums into every CTA's P.
//
// What crosses CTAs (halo rows of K, the sums P) goes by asynchronous
// stores into distributed shared memory that complete on the receiver's
// mbarriers, so a step makes no trip to memory and no cluster barrier (a
// release over the cluster costs 400-500 cycles).  P is double-buffered: a
// CTA can send the next step's sums before another has read this step's,
// but not the sums after those, which need the other's own.  K's halo rows
// need one buffer: the next ones are sent by a CTA that has every row's
// sum, and a row's sum leaves after its warp has read K.  Every wait is
// bounded.  The same arithmetic per cell and the same order of every sum as
// k_bwake and k_bmaps0f: the same bits.
//
// Per step, measured: one 128-row bunch 6.7 us with the per-step kernels,
// 1.5 us here; 777 bunches of 64 rows 23.3 and 6.0; 256 of 256 rows 39.9
// and 29.8 (7 rounds of clusters, the last four bunches on larger ones).
// Bound by latency: 8 warps per SM leave 64 % of the issue slots empty, and
// the wake, the barriers and the row sums' way between the CTAs are a third of
// a step.
//
// Rows of T and K: [16 zeros][words 0, 2, 4 ..][16 zeros][words 1, 3, ..]
// (words of 4 columns): the y-kick's lanes (two words each, any shift) and
// the drift's (one word each) both read and write 8 consecutive lanes on
// 32 banks, and windows past the row's ends read zeros.
#pragma once

#include "vfps_internal.cuh"

namespace {

constexpr int RES_MAX_C = 16;
constexpr int RES_MAX_N = 256;

// N: mesh size, CPL: columns per lane of the drift, RW: rows of a run (the
// rows a group of N/CPL lanes walks in the drift)
template <int N_, int CPL_, int RW_>
struct ResShape {
    static constexpr int N = N_, CPL = CPL_, RW = RW_;
    static constexpr int NW = 8;                    // warps of a CTA
    static constexpr int NT = 32 * NW;
    static constexpr int WPL = CPL / 4;             // words per lane
    static constexpr int SEG = N / CPL;             // lanes a row
    static constexpr int RUNS = NT / SEG;           // runs of a CTA
    static constexpr int R = RUNS * RW;             // rows of a CTA
    static constexpr int C = N / R;                 // CTAs of a bunch
    static constexpr int KR = R / NW;               // a warp's kick rows
    static constexpr int KL = N / 8;                // kick lanes a row
    static constexpr int KS = 32 / KL;              // kick rows at a time
    static constexpr int RS = N + 32;               // floats of a row
    static constexpr int MPL = N / 32;              // source cells per lane
    // padded index of the Toeplitz tables: lanes MPL entries apart on an
    // odd stride
    static constexpr int LG = MPL == 2 ? 1 : MPL == 4 ? 2 : 3;
    static constexpr int WLEN = (N + R) + ((N + R) >> LG) + 1;
    static_assert(R * C == N && C <= RES_MAX_C && KR % KS == 0
                  && SEG <= 32 && N <= RES_MAX_N, "rows");
};

// float offsets of the dynamic shared memory; krows: rows of K (R and the
// widest halos of the launch's bunches)
template <typename S>
struct ResSmem {
    static __host__ __device__ constexpr uint32_t up4(uint32_t v)
    {
        return (v + 3) & ~3u;
    }
    uint32_t T, K, P, W, KT, st, sb, csr, sum, misc, bar, total;
    __host__ __device__ explicit ResSmem(int krows)
    {
        T = 0;
        K = T + uint32_t(S::R) * S::RS + 16;
        P = K + uint32_t(krows) * S::RS;
        W = P + 2 * S::N;
        KT = W + up4(S::WLEN);
        st = KT + up4(S::WLEN);
        sb = st + S::R * 8;
        csr = sb + up4(S::R * 5);
        sum = csr + up4(4 * S::C * S::NW);
        misc = sum + up4(S::R);
        bar = misc + 4;   // three mbarriers
        total = bar + 8;
    }
};

struct ResArgs {
    const BDev* bd;
    const uint32_t* list;      // bunches of this launch
    uint32_t nlist, nsteps;
    int krows;
    const float* tabs;
    const float* dwt;
    const float* wt;
    const RowStencil* st;
    const float* din;
    float* dout;
    const float* pin;
    float* pout;
    float* wake;
    float* factor;
    double* filling;
    unsigned long long* tickets;   // step counters, from wblk0[bunch] on
    const uint32_t* wblk0;
    CsrRec csr;
    int* status;
};

__device__ __forceinline__ uint32_t cluster_id_x()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
    return r;
}

__device__ __forceinline__ uint32_t cluster_count_x()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%nclusterid.x;" : "=r"(r));
    return r;
}

// asynchronous stores to shared memory of the cluster; their bytes complete
// on the barrier `bar` of the same CTA (both addresses from cluster_map)
__device__ __forceinline__ void cluster_send(uint32_t addr, float v,
                                             uint32_t bar)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f32"
                 " [%0], %1, [%2];"
                 :: "r"(addr), "f"(v), "r"(bar) : "memory");
}

__device__ __forceinline__ void cluster_send2(uint32_t addr, float2 v,
                                              uint32_t bar)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2"
                 ".f32 [%0], {%1, %2}, [%3];"
                 :: "r"(addr), "f"(v.x), "f"(v.y), "r"(bar) : "memory");
}

__device__ __forceinline__ void cluster_send4(uint32_t addr, float4 v,
                                              uint32_t bar)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4"
                 ".f32 [%0], {%1, %2, %3, %4}, [%5];"
                 :: "r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w),
                    "r"(bar) : "memory");
}

// every thread of the cluster (of the CTA, C = 1)
template <int C>
__device__ __forceinline__ void cluster_barrier()
{
    if constexpr (C > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;\n"
                     "barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        __syncthreads();
    }
}

// one arrival of this CTA's barrier
__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];"
                 :: "r"(smem_addr(bar)) : "memory");
}

// mbar_wait_bounded with the timer read only now and then: these waits are
// a few hundred cycles, and a timer read would delay seeing their end
__device__ __forceinline__ bool res_wait(uint64_t* bar, uint32_t parity)
{
    uint64_t t0 = 0;
    for (uint32_t i = 0; !mbar_try_wait(bar, parity); i++) {
        if ((i & 255u) == 255u) {
            const uint64_t now = global_ns();
            t0 = t0 ? t0 : now;
            if (now - t0 > WAIT_NS) {
                return false;
            }
        }
    }
    return true;
}

// Sums v[0..CNT) over groups of L lanes (L a power of two, CNT <= L):
// afterwards v[0] holds the sum of entry `ret` (lanes l, l' of a group that
// differ only below the last exchange hold the same entry; the lanes with
// l % (L / CNT) == 0 hold one entry each).  Lanes L/2 apart first, then
// L/4 .. 1; NEAR: neighbours before those (the lanes that hold the same
// entry differ in the bits 1 .. lg(L / CNT), (l >> 1) % (L / CNT) counts
// them)
template <int CNT, int L, bool NEAR = false>
__device__ __forceinline__ int reduce_scatter(float (&v)[CNT], int l)
{
    static_assert(CNT <= L, "one entry per lane at most");
    int at = 0;
    int o = NEAR ? 1 : L >> 1;
    constexpr int END = NEAR ? 1 : 0;
    auto next = [&] { o = NEAR && o == 1 ? L >> 1 : o >> 1; };
#pragma unroll
    for (int c = CNT; c > 1; c >>= 1, next()) {
        const bool up = (l & o) != 0;
#pragma unroll
        for (int i = 0; i < c / 2; i++) {
            const float send = up ? v[i] : v[i + c / 2];
            const float keep = up ? v[i + c / 2] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
        at += up ? c / 2 : 0;
    }
    if (NEAR && CNT == 1) {
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
        next();
    }
#pragma unroll
    for (; o > END; o >>= 1) {
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    }
    return at;
}

// compensated charge integral in the order of all kernels (a warp; every
// lane's value)
template <int N>
__device__ __forceinline__ double profile_charge(const float* P,
                                                 const float* ws, int lane)
{
    constexpr int K = N / 32 < 8 ? N / 32 : 8;
    FF f[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
        f[k] = ff_prod(P[32 * k + lane], ws[32 * k + lane]);
        if (N / 32 > K) {   // (512 rows)
            f[k] = ff_add(f[k], ff_prod(P[32 * (k + K) + lane],
                                        ws[32 * (k + K) + lane]));
        }
    }
    // over the lanes, all k at once (afterwards k's bits are the lane's
    // highest), then over k
    auto other = [](FF v, int o) {
        return FF{__shfl_xor_sync(0xffffffffu, v.hi, o),
                  __shfl_xor_sync(0xffffffffu, v.lo, o)};
    };
    int o = 16;
#pragma unroll
    for (int c = K / 2; c > 0; c >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int k = 0; k < c; k++) {
            const FF got = other(up ? f[k] : f[k + c], o);
            f[k] = ff_add(up ? f[k + c] : f[k], got);
        }
    }
    FF a = f[0];
#pragma unroll
    for (; o > 0; o >>= 1) {
        a = ff_add(a, other(a, o));
    }
#pragma unroll
    for (int q = 16; q > 16 / K; q >>= 1) {
        a = ff_add(a, other(a, q));
    }
    return double(a.hi) + double(a.lo);
}

// compensated sum over the rows of a warp's group, on the lanes `first` apart
// (row i of the group on lane i first), neighbours first; lane 0's value
__device__ __forceinline__ FF rows_sum(FF v, int first)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const FF u{__shfl_xor_sync(0xffffffffu, v.hi, o),
                   __shfl_xor_sync(0xffffffffu, v.lo, o)};
        v = o >= first ? ff_add(v, u) : v;
    }
    return v;
}

// and over `count` groups' sums (at most 128, a multiple of 4 or at most 32)
__device__ __forceinline__ float groups_sum(const float2* part, int count,
                                            int lane)
{
    auto at = [&](int i) {
        const float2 v = i < count ? part[i] : make_float2(0.f, 0.f);
        return FF{v.x, v.y};
    };
    FF v;
    if (count <= 32) {
        v = at(lane);
    } else {   // 64 or 128
        const int per = count / 32;
        v = ff_add(at(per * lane), at(per * lane + 1));
        if (per == 4) {
            v = ff_add(v, ff_add(at(4 * lane + 2), at(4 * lane + 3)));
        }
    }
    v = rows_sum(v, 1);
    return v.hi + v.lo;
}

// Whether the sign of a profile's charge needs the compensated sum (a warp;
// the same in every lane): an FP32 sum with the Simpson weights 1 4 2 .. 2 4 1
// (here halved), N / 32 + 5 roundings and those of the weights off at most,
// leaves no doubt above 1e-5 of the sum of magnitudes (NaN and infinities
// stay in doubt)
template <int N>
__device__ __forceinline__ bool charge_doubtful(const float* P, int lane)
{
    float a = 0.f, m = 0.f;
#pragma unroll
    for (int i = 0; i < N / 32; i++) {
        const float p = P[lane + 32 * i];
        const bool end = lane + 32 * i == 0 || lane + 32 * i == N - 1;
        const float w = end ? 0.5f : (lane & 1) ? 2.f : 1.f;
        a = fmaf(p, w, a);
        m = fmaf(fabsf(p), w, m);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        m += __shfl_xor_sync(0xffffffffu, m, o);
    }
    return !(a > 1e-5f * m);
}

// sum_m P[m] T(x - m) on rows xl .. xl + ROWS of this CTA, from the table
// Wt[k + (k >> LG)] = T(x0 + k - N), k = (x - x0) - m + N: lane l takes the
// source cells MPL l .. MPL l + MPL - 1 (their table entries slide through
// ROWS + MPL - 1 registers); every lane leaves with the sum of row xl + ret
template <typename S, int ROWS>
__device__ __forceinline__ int toeplitz_rows(const float* P, const float* Wt,
                                             int xl, int lane, float& sum)
{
    constexpr int MPL = S::MPL;
    const int m0 = MPL * lane;
    float p[MPL];
    if constexpr (MPL == 2) {
        const float2 q = *reinterpret_cast<const float2*>(P + m0);
        p[0] = q.x;
        p[1] = q.y;
    } else {
#pragma unroll
        for (int j = 0; j < MPL; j += 4) {
            const float4 q = *reinterpret_cast<const float4*>(P + m0 + j);
            p[j] = q.x;
            p[j + 1] = q.y;
            p[j + 2] = q.z;
            p[j + 3] = q.w;
        }
    }
    float w[ROWS + MPL - 1];
#pragma unroll
    for (int d = 0; d < ROWS + MPL - 1; d++) {
        const int k = xl + S::N - (MPL - 1) + d;   // less MPL lane
        w[d] = Wt[k + (k >> S::LG) - (MPL + 1) * lane];
    }
    float acc[ROWS];
#pragma unroll
    for (int i = 0; i < ROWS; i++) {
        acc[i] = p[0] * w[i + MPL - 1];
#pragma unroll
        for (int j = 1; j < MPL; j++) {
            acc[i] = fmaf(p[j], w[i + MPL - 1 - j], acc[i]);
        }
    }
    const int at = reduce_scatter<ROWS, 32>(acc, lane);
    sum = acc[0];
    return at;
}

// offset in a row of T or K of word f (4 columns)
template <typename S>
__device__ __forceinline__ int res_word(int f)
{
    return 16 + (f & 1) * (S::N / 2 + 16) + (f >> 1) * 4;
}

// 8 outputs of the 7-tap y-kick from the window v, whose first input is
// v[AL]
template <int AL>
__device__ __forceinline__ void res_kick8(const float (&v)[20],
                                          const float (&c)[7], float (&o)[8])
{
#pragma unroll
    for (int q = 0; q < 8; q++) {
        o[q] = c[0] * v[AL + q];
    }
#pragma unroll
    for (int k = 1; k < 7; k++) {
#pragma unroll
        for (int q = 0; q < 8; q++) {
            o[q] = fmaf(c[k], v[AL + q + k], o[q]);
        }
    }
}

// the stencil of a row's y-kick (ST) and the first 4 words of its window
struct ResKick {
    float4 q0, q1;
    float4 v[4];
};

template <int N, int CPL, int RW>
__global__ void __launch_bounds__(256, CPL == 8 ? 1 : 2)
k_bres(const __grid_constant__ ResArgs A)
{
    using S = ResShape<N, CPL, RW>;
    constexpr int SEG = S::SEG, R = S::R, C = S::C;
    constexpr int KR = S::KR, KL = S::KL, KS = S::KS;
    constexpr int RS = S::RS, NT = S::NT, NW = S::NW, WPL = S::WPL;
    extern __shared__ float4 smem4[];
    float* sm = reinterpret_cast<float*>(smem4);
    const ResSmem<S> L(A.krows);
    float* T = sm + L.T;
    float* K = sm + L.K;
    float* W = sm + L.W;
    float* KT = sm + L.KT;
    float* SB = sm + L.sb;              // RF stencils: shift, 4 weights
    float2* cpart = reinterpret_cast<float2*>(sm + L.csr);
    float* wsum = sm + L.sum;
    float* fac_s = sm + L.misc;
    // P of even and odd steps complete, halo rows of K complete
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + L.bar);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = C > 1 ? int(cluster_rank()) : 0;
    const uint32_t cl = C > 1 ? cluster_id_x() : blockIdx.x;
    const uint32_t ncl = C > 1 ? cluster_count_x() : gridDim.x;
    const int x0 = rank * R;            // the CTA's first row
    // drift: the lane's run of rows and words of columns
    const int l = lane & (SEG - 1);
    const int row0 = threadIdx.x / SEG * RW;
    const int f0 = l * WPL;                  // its first word
    // (a lane of two words has one of each half of a row)
    const int fo = res_word<S>(f0);
    constexpr int FG = N / 2 + 16;           // from the first to the second
    // y-kick: the warp's rows and the lane's pair of words
    const int krow0 = warp * KR;
    const int kl = lane & (KL - 1);
    float4* ST = reinterpret_cast<float4*>(sm + L.st);
    uint32_t k_lo = 0, k_hi = 0, kb_lo = 0, kb_hi = 0;
    if constexpr (C > 1) {
        if (rank > 0) {
            k_lo = cluster_map(smem_addr(K), rank - 1);
            kb_lo = cluster_map(smem_addr(bar + 2), rank - 1);
        }
        if (rank < C - 1) {
            k_hi = cluster_map(smem_addr(K), rank + 1);
            kb_hi = cluster_map(smem_addr(bar + 2), rank + 1);
        }
        if (threadIdx.x == 0) {
            mbar_init(&bar[0], NW);
            mbar_init(&bar[1], NW);
            mbar_init(&bar[2], 1);
            mbar_fence_init();
        }
    }
    uint32_t gs = 0;   // steps of this launch so far, over its bunches
    int bad = 0;       // a wait ran out
    // the zero words of T's rows
    for (int i = threadIdx.x; i < R * RS + 16; i += NT) {
        T[i] = 0.f;
    }

    for (uint32_t bi = cl; bi < A.nlist; bi += ncl) {
        const uint32_t b = A.list[bi];
        const BDev& BD = A.bd[b];
        const int hlo = BD.halo_lo, hhi = BD.halo_hi;
        const int it = int(BD.it), renorm = BD.renorm;
        const float wakescale = BD.wakescale, fillset = BD.fillset;
        const uint32_t prof_off = BD.prof_off;
        const bool has_wake = BD.flags & F_WAKE;
        const uint32_t koff = A.csr.every ? A.csr.off[b] : NO_CSR;
        const unsigned step0 =
            static_cast<unsigned>(A.tickets[A.wblk0[b]]);
        const float* ws = A.tabs + BD.tab_off + TAB_WS * N;
        const float h03 = ws[0];
        __syncthreads();   // the last bunch's P and T are stored
        // ---- the bunch's tables, profile and rows
        for (int i = threadIdx.x; i < N; i += NT) {
            sm[L.P + (gs & 1) * N + i] = A.pin[prof_off + i];
        }
        if (has_wake) {
            const int nmax = int(BD.nmax);
            const float* w = A.wt + BD.wt_off;
            for (int k = threadIdx.x; k < N + R; k += NT) {
                int i = (x0 + k - N) % nmax;
                i += i < 0 ? nmax : 0;
                W[k + (k >> S::LG)] = w[i];
            }
        }
        if (koff != NO_CSR) {
            for (int k = threadIdx.x + 1; k < N + R; k += NT) {
                KT[k + (k >> S::LG)] = A.csr.k[koff + x0 + k - 1];
            }
        }
        for (int i = threadIdx.x; i < R; i += NT) {
            const RowStencil r = A.st[BD.st_off + ST_RF * N + x0 + i];
            SB[5 * i] = __int_as_float(r.shift0);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                SB[5 * i + 1 + j] = r.w[j];
            }
        }
        // halo rows off the mesh are zero rows (nothing writes them)
        if (rank == 0) {
            for (int i = threadIdx.x; i < hlo * RS; i += NT) {
                K[i] = 0.f;
            }
        }
        if (rank == C - 1) {
            for (int i = threadIdx.x; i < hhi * RS; i += NT) {
                K[(hlo + R) * RS + i] = 0.f;
            }
        }
        {
            const float4* src = reinterpret_cast<const float4*>(
                A.din + BD.dens_off + size_t(x0) * N);
#pragma unroll 8
            for (int i = threadIdx.x; i < R * (N / 4); i += NT) {
                const int x = i / (N / 4), f = i % (N / 4);
                *reinterpret_cast<float4*>(T + x * RS + res_word<S>(f)) =
                    src[i];
            }
        }
        // the lane's Simpson weights (in units of h03), drift and
        // Fokker-Planck weights, and its windows in K
        const float* dw = A.dwt + BD.dw_off;
        float sw[CPL];
        float4 wd[WPL][4], fw[WPL][5];
        const float* kwin[WPL];
#pragma unroll
        for (int g = 0; g < WPL; g++) {
            const int y = 4 * (f0 + g);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                sw[4 * g + q] = y + q == 0 || y + q == N - 1
                                    ? 1.f : ((q & 1) ? 4.f : 2.f);
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                wd[g][j] = *reinterpret_cast<const float4*>(dw + j * N + y);
            }
#pragma unroll
            for (int o = 0; o < 5; o++) {
                fw[g][o] = *reinterpret_cast<const float4*>(dw + (5 + o) * N
                                                            + y);
            }
            kwin[g] = K + (row0 + hlo + __float_as_int(dw[4 * N + y])) * RS
                      + fo + g * FG;
        }
        __syncwarp();
        cluster_barrier<C>();   // tables complete; every CTA is running

        // the CSR power of step csr_step from its parts (warp 0 of rank 0,
        // one step later; two buffers, so that the next parts may arrive)
        bool csr_pending = false;
        unsigned csr_step = 0, csr_buf = 0;
        auto csr_store = [&] {
            if (!csr_pending) {
                return;
            }
            csr_pending = false;
            const float tot = groups_sum(cpart + csr_buf * C * NW, C * NW,
                                         lane);
            if (lane == 0) {
                const uint32_t slot = (csr_step / A.csr.every) % A.csr.cap;
                A.csr.power[size_t(slot) * A.csr.nb + b] = tot;
                if (b == 0) {
                    A.csr.steps[slot] = csr_step;
                }
            }
        };
        for (uint32_t t = 0; t < A.nsteps; t++, gs++) {
            const float* P = sm + L.P + (gs & 1) * N;
            const uint32_t pn = L.P + ((gs + 1) & 1) * N;   // the next one
            const unsigned step = step0 + t;
            const bool lastst = t + 1 == A.nsteps;
            const bool renorm_now = renorm > 0
                                    && (step % unsigned(renorm)) == 0;
            const bool csr_now = koff != NO_CSR && step % A.csr.every == 0;
            auto charge = [&] { return profile_charge<N>(P, ws, lane); };
            if (renorm_now && warp == 0) {
                const double q = charge();
                if (lane == 0) {
                    fac_s[0] = fillset > 0
                                   ? static_cast<float>(double(fillset) / q)
                                   : 0.f;
                }
            }
            // ---- wake sums of the warp's rows
            if (has_wake) {
                float sum;
                const int at = toeplitz_rows<S, KR>(P, W, krow0, lane, sum);
                if ((lane & (32 / KR - 1)) == 0) {
                    wsum[krow0 + at] = sum;
                }
            }
            if (__syncthreads_or(bad)) {
                bad = 1;
                break;
            }
            // ---- the composite y-kick of row threadIdx.x
            if (warp < (R + 31) / 32 && (R >= 32 || lane < R)) {
                const int x = threadIdx.x;
                const float fac = renorm_now ? fac_s[0] : 1.f;
                float wk = 0.f;
                RowStencil sa;
                if (has_wake) {
                    wk = __fmul_rn(wakescale, wsum[x]);
                    sa = make_stencil(wk, N, it);
                } else {
                    sa.shift0 = 0;
                    sa.w[0] = 1.f;
                    sa.w[1] = sa.w[2] = sa.w[3] = 0.f;
                }
                const float* sb = SB + 5 * x;
                float a[4], bw[4];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    a[j] = sa.w[j] * fac;
                    bw[j] = sb[1 + j];
                }
                const int s = sa.shift0 + __float_as_int(sb[0]);
                float c[7];
#pragma unroll
                for (int k = 0; k < 7; k++) {
                    float v = 0.f;
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        if (k - i >= 0 && k - i < 4) {
                            v = fmaf(a[i], bw[k - i], v);
                        }
                    }
                    c[k] = v;
                }
                ST[2 * x] = make_float4(__int_as_float(s), c[0], c[1], c[2]);
                ST[2 * x + 1] = make_float4(c[3], c[4], c[5], c[6]);
                if (lastst) {
                    A.wake[prof_off + x0 + x] = wk;
                }
            }
            __syncthreads();
            // ---- y-kick
            if constexpr (C > 1) {
                // this step's halo rows
                if (threadIdx.x == 0) {
                    mbar_arrive_expect_tx(
                        &bar[2], uint32_t((rank > 0 ? hlo : 0)
                                          + (rank < C - 1 ? hhi : 0))
                                     * uint32_t(N * 4));
                }
            }
            // window word 2 pw + (s >> 2) + j of row lx lies at w0 (j even)
            // or w1 (j odd), 4 floats on for every second word
            auto window = [&](int lx, int s, const float*& w0,
                              const float*& w1) {
                const float* w = T + lx * RS + 16 + 4 * kl + 4 * (s >> 3);
                w0 = w + ((s & 4) ? FG : 0);
                w1 = w + ((s & 4) ? 4 : FG);
            };
            auto in_pads = [](int s) { return s >= -32 && s <= 20; };
            auto shift = [&](int lx) {
                return __float_as_int(ST[2 * lx].x);
            };
            auto fetch = [&](int lx, int s, ResKick& f) {
                f.q0 = ST[2 * lx];
                f.q1 = ST[2 * lx + 1];
                const float *w0, *w1;
                window(lx, in_pads(s) ? s : 0, w0, w1);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    f.v[j] = *reinterpret_cast<const float4*>(
                        ((j & 1) ? w1 : w0) + (j >> 1) * 4);
                }
            };
            auto kick = [&](int lx, int s, const ResKick& f) {
                const float c[7] = {f.q0.y, f.q0.z, f.q0.w, f.q1.x, f.q1.y,
                                    f.q1.z, f.q1.w};
                float o[8];
                if (in_pads(s)) {
                    float v[20];
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        v[4 * j] = f.v[j].x;
                        v[4 * j + 1] = f.v[j].y;
                        v[4 * j + 2] = f.v[j].z;
                        v[4 * j + 3] = f.v[j].w;
                    }
                    if (s & 2) {
                        if (s & 1) {
                            const float *w0, *w1;
                            window(lx, s, w0, w1);
                            const float4 q = *reinterpret_cast<const float4*>(
                                w0 + 8);
                            v[16] = q.x;
                            v[17] = q.y;
                            v[18] = q.z;
                            v[19] = q.w;
                            res_kick8<3>(v, c, o);
                        } else {
                            res_kick8<2>(v, c, o);
                        }
                    } else {
                        if (s & 1) {
                            res_kick8<1>(v, c, o);
                        } else {
                            res_kick8<0>(v, c, o);
                        }
                    }
                } else {
                    // a window further off: every input checked
#pragma unroll
                    for (int q = 0; q < 8; q++) {
                        o[q] = 0.f;
                    }
#pragma unroll 1
                    for (int k = 0; k < 7; k++) {
                        const float ck = k == 0 ? c[0] : k == 1 ? c[1]
                            : k == 2 ? c[2] : k == 3 ? c[3]
                            : k == 4 ? c[4] : k == 5 ? c[5] : c[6];
#pragma unroll
                        for (int q = 0; q < 8; q++) {
                            const int y = 8 * kl + s + q + k;
                            const float v = unsigned(y) < unsigned(N)
                                ? T[lx * RS + res_word<S>(y >> 2) + (y & 3)]
                                : 0.f;
                            o[q] = k == 0 ? ck * v : fmaf(ck, v, o[q]);
                        }
                    }
                }
                float* k0 = K + (hlo + lx) * RS + 16 + 4 * kl;
                *reinterpret_cast<float4*>(k0) =
                    make_float4(o[0], o[1], o[2], o[3]);
                *reinterpret_cast<float4*>(k0 + FG) =
                    make_float4(o[4], o[5], o[6], o[7]);
            };
            {
                // the next row's stencil and window and the shift of the
                // one after it are on their way while a row is kicked
                constexpr int TURNS = KR / KS;
                const int lx0 = krow0 + lane / KL;
                auto row = [&](int i) {
                    return lx0 + min(i, TURNS - 1) * KS;
                };
                ResKick f[2];
                int s0 = shift(row(0)), s1 = shift(row(1));
                fetch(row(0), s0, f[0]);
#pragma unroll 2
                for (int i = 0; i < TURNS; i++) {
                    const int s2 = shift(row(i + 2));
                    fetch(row(i + 1), s1, f[(i + 1) & 1]);
                    kick(row(i), s0, f[i & 1]);
                    s0 = s1;
                    s1 = s2;
                }
            }
            __syncthreads();   // the CTA's rows of K
            if constexpr (C > 1) {
                // those among the neighbours' halo rows (by all threads: a
                // warp's asynchronous stores take some 50 cycles each)
                if (rank < C - 1) {
                    for (int i = threadIdx.x; i < hlo * (N / 4); i += NT) {
                        const int r = i / (N / 4);
                        const int at = res_word<S>(i % (N / 4));
                        cluster_send4(
                            k_hi + 4u * uint32_t(r * RS + at),
                            *reinterpret_cast<const float4*>(
                                K + (R + r) * RS + at), kb_hi);
                    }
                }
                if (rank > 0) {
                    for (int i = threadIdx.x; i < hhi * (N / 4); i += NT) {
                        const int r = i / (N / 4);
                        const int at = res_word<S>(i % (N / 4));
                        cluster_send4(
                            k_lo + 4u * uint32_t((hlo + R + r) * RS + at),
                            *reinterpret_cast<const float4*>(
                                K + (hlo + r) * RS + at), kb_lo);
                    }
                }
            }
            // ---- while the halo rows arrive: the step's charge (its sign
            // is watched; its value kept of the last step) and CSR power
            if (rank == 0 && warp == 0) {
                csr_store();   // the last step's
                if (lastst) {
                    const double q = charge();
                    if (lane == 0) {
                        A.filling[b] = q;
                        A.factor[b] = renorm_now ? fac_s[0] : 1.f;
                        if (fillset > 0 && !(q > 0)) {
                            atomicCAS(A.status, 0, VFPS_ERR_NUMERIC);
                        }
                    }
                } else if (fillset > 0 && charge_doubtful<N>(P, lane)) {
                    const double q = charge();
                    if (lane == 0 && !(q > 0)) {
                        atomicCAS(A.status, 0, VFPS_ERR_NUMERIC);
                    }
                }
            }
            if (csr_now) {
                // the warp's rows' part of the CSR power
                float v;
                const int at = toeplitz_rows<S, KR>(P, KT, krow0, lane, v);
                FF dot = FF{0.f, 0.f};
                if ((lane & (32 / KR - 1)) == 0) {
                    dot = ff_prod(P[x0 + krow0 + at], v);
                }
                dot = rows_sum(dot, 32 / KR);
                if (lane == 0) {
                    // (with the step's row sums)
                    float2* cp = cpart + ((t & 1) * C + rank) * NW + warp;
                    if (rank > 0) {
                        cluster_send2(cluster_map(smem_addr(cp), 0),
                                      make_float2(dot.hi, dot.lo),
                                      cluster_map(smem_addr(&bar[gs & 1]),
                                                  0));
                    } else {
                        *cp = make_float2(dot.hi, dot.lo);
                    }
                }
                csr_step = step;
                csr_buf = t & 1;
                csr_pending = true;
            }
            __syncwarp();
            if constexpr (C > 1) {
                // the runs whose windows reach into the halo rows
                if (row0 < hlo || row0 + RW + hhi > R) {
                    if (!res_wait(&bar[2], gs & 1)) {
                        bad = 1;
                    }
                }
            }
            // ---- drift, Fokker-Planck, row sums
            float* tp = T + row0 * RS + fo;
            const float* kp[WPL];
            float4 win[WPL][4];
#pragma unroll
            for (int g = 0; g < WPL; g++) {
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    win[g][j] = *reinterpret_cast<const float4*>(kwin[g]
                                                                 + j * RS);
                }
                kp[g] = kwin[g] + 3 * RS;
            }
            constexpr int U = RW < 8 ? RW : 8;   // rows per turn
#pragma unroll 1
            for (int r0 = 0; r0 < RW; r0 += U) {
                float ps[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    // the drift of the lane's columns in w[2 ..], the
                    // neighbours' around them (at the mesh edges the
                    // wrapped values meet zero weights)
                    float w[CPL + 4];
#pragma unroll
                    for (int g = 0; g < WPL; g++) {
                        win[g][(u + 3) & 3] =
                            *reinterpret_cast<const float4*>(kp[g]
                                                             + u * RS);
                        const float4 d = drift4(
                            win[g][u & 3], win[g][(u + 1) & 3],
                            win[g][(u + 2) & 3], win[g][(u + 3) & 3],
                            wd[g]);
                        w[2 + 4 * g] = d.x;
                        w[3 + 4 * g] = d.y;
                        w[4 + 4 * g] = d.z;
                        w[5 + 4 * g] = d.w;
                    }
                    const int lm = (l + SEG - 1) & (SEG - 1);
                    const int lp = (l + 1) & (SEG - 1);
                    w[0] = __shfl_sync(0xffffffffu, w[CPL], lm, SEG);
                    w[1] = __shfl_sync(0xffffffffu, w[CPL + 1], lm, SEG);
                    w[CPL + 2] = __shfl_sync(0xffffffffu, w[2], lp, SEG);
                    w[CPL + 3] = __shfl_sync(0xffffffffu, w[3], lp, SEG);
                    float o[CPL];
#pragma unroll
                    for (int k = 0; k < 5; k++) {
#pragma unroll
                        for (int g = 0; g < WPL; g++) {
                            const float f[4] = {fw[g][k].x, fw[g][k].y,
                                                fw[g][k].z, fw[g][k].w};
#pragma unroll
                            for (int q = 0; q < 4; q++) {
                                const int i = 4 * g + q;
                                o[i] = k == 0
                                           ? f[q] * w[i + k]
                                           : fmaf(f[q], w[i + k], o[i]);
                            }
                        }
                    }
#pragma unroll
                    for (int g = 0; g < WPL; g++) {
                        *reinterpret_cast<float4*>(tp + u * RS + g * FG) =
                            make_float4(o[4 * g], o[4 * g + 1],
                                        o[4 * g + 2], o[4 * g + 3]);
                    }
#pragma unroll
                    for (int g = 0; g < WPL; g++) {   // a word's sum
                        const float p0 = fmaf(sw[4 * g + 2], o[4 * g + 2],
                                              sw[4 * g] * o[4 * g]);
                        const float p1 = fmaf(sw[4 * g + 3], o[4 * g + 3],
                                              sw[4 * g + 1] * o[4 * g + 1]);
                        ps[u] = g == 0 ? p0 + p1 : ps[u] + (p0 + p1);
                    }
                }
#pragma unroll
                for (int g = 0; g < WPL; g++) {
                    kp[g] += U * RS;
                }
                tp += U * RS;
                // (a lane of one word: its neighbour's is added first)
                constexpr bool NEAR = WPL == 1;
                const int at = reduce_scatter<U, SEG, NEAR>(ps, l);
                constexpr int REP = SEG / U;  // lanes holding a row's sum
                const int rep = (NEAR ? l >> 1 : l) & (REP - 1);
                const int xr = row0 + r0 + at;
                float* pa = sm + pn + x0 + xr;
                const float v = h03 * ps[0];
                for (int c = rep; c < C; c += REP) {
                    if (c == rank) {
                        *pa = v;
                    } else {
                        cluster_send(
                            cluster_map(smem_addr(pa), c), v,
                            cluster_map(smem_addr(&bar[gs & 1]), c));
                    }
                }
            }
            // the CTA's rows of T and P (an arrival per warp), the others'
            // of P (their bytes)
            __syncwarp();
            if constexpr (C > 1) {
                if (threadIdx.x == 0) {
                    mbar_arrive_expect_tx(
                        &bar[gs & 1],
                        uint32_t(N - R) * 4u
                            + (csr_now && rank == 0
                                   ? uint32_t((C - 1) * NW) * 8u : 0u));
                } else if (lane == 0) {
                    mbar_arrive(&bar[gs & 1]);
                }
                if (!res_wait(&bar[gs & 1], (gs >> 1) & 1)) {
                    bad = 1;
                }
            } else {
                __syncthreads();
            }
        }
        if (__syncthreads_or(bad)) {
            bad = 1;
            break;
        }
        const float* P = sm + L.P + (gs & 1) * N;
        if (rank == 0 && warp == 0) {
            csr_store();
        }
        // ---- the new state
        {
            float4* dst = reinterpret_cast<float4*>(
                A.dout + BD.dens_off + size_t(x0) * N);
#pragma unroll 8
            for (int i = threadIdx.x; i < R * (N / 4); i += NT) {
                const int x = i / (N / 4), f = i % (N / 4);
                dst[i] = *reinterpret_cast<const float4*>(T + x * RS
                                                          + res_word<S>(f));
            }
        }
        for (int i = threadIdx.x; i < R; i += NT) {
            A.pout[prof_off + x0 + i] = P[x0 + i];
        }
        if (rank == 0 && threadIdx.x < N / wake_block_rows(N)) {
            // (every CTA of the cluster read its counter before the
            // barriers above)
            A.tickets[A.wblk0[b] + threadIdx.x] += A.nsteps;
        }
    }
    if (bad && threadIdx.x == 0) {
        atomicCAS(A.status, 0, VFPS_ERR_TIMEOUT);
    }
    __syncwarp();
    cluster_barrier<C>();   // no CTA leaves while another may send to it
}

}  // namespace
