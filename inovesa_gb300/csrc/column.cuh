// k_bcol: many solver steps of 512-row chain-0 bunches on regular lattices in
// one launch, the density on the chip from the first step to the last (included by batch.cu
// after resident.cuh, whose arguments and cluster primitives it shares).
//
// A cluster of 16 CTAs owns one bunch; CTA `rank` owns 32 mesh rows, one
// per lane of every warp, in shared memory twice (this step's density and
// the next one's) as lines of 32 rows per column: a lane reads its row's
// columns at any shift without bank conflicts, and with one read per output
// its window of the y-kick moves through registers.  A warp walks 32
// columns, two more on either side:
//
//   y-kick    7 taps, the row's weights in registers; the two rows beyond
//             either end of the CTA's come from a small array (their
//             densities arrive with the row sums);
//   drift     rows by shuffles, the column's weights from shared memory;
//   Fokker-Planck   the last 5 columns' drift in registers; row sums on the
//             way, the edge rows to the neighbours.
//   The warps of the lower energies need no tap at 2, those of the upper ones
//   none at -2: 4 taps and 3 shuffles a column (the two in the middle: all).
//
// One exchange per step: edge rows and row sums go by asynchronous stores
// that complete on the receiver's mbarrier of the step; the density, the
// edge rows and the profile are double-buffered.  A CTA sends into the
// buffer of step t + 2 only with every row sum of step t + 1, which the
// others send after they have read step t's.  Every wait is bounded.
//
// A step of one bunch, measured: 6.4 us here, 7.1 us with its CSR power (7.0
// and 7.8 with 5 taps for every warp); 8.6 and 12.1 us with the per-step
// kernels.  Seven clusters run at a time: seven bunches 6.4 us, 11.3 us with
// the per-step kernels.  Bound by instruction issue and shared memory
// together (16 warps on an SM: half the issue slots, 60 % of the cycles of
// its shared memory).  For meshes of up to 256 rows k_bres is faster (256
// rows: 4.2 us, 5.3 us this way): a row lies along its lanes there, and the
// drift needs no shuffles.
#pragma once

#include "resident.cuh"

namespace {

constexpr int res_up4(int v)
{
    return (v + 3) & ~3;
}

struct Col {
    static constexpr int N = 512;
    static constexpr int NW = 16;                   // warps of a CTA
    static constexpr int NT = 32 * NW;
    static constexpr int R = 32;                    // rows of a CTA
    static constexpr int C = N / R;                 // CTAs of a bunch
    static constexpr int RT = 4;                    // rows of a wake group
    static constexpr int GROUPS = (R + 4) / RT;     // with the halo rows
    static constexpr int CG = R / RT;               // of own rows
    static constexpr int Y = N / NW;                // columns of a warp
    static constexpr int YP = Y + 4;                // with two on each side
    static constexpr int UN = 12;                   // columns per turn
    static constexpr int DR = UN / 2;
    static constexpr int PAD = 16;    // zero lines before and after
    static constexpr int LINES = N + 2 * PAD;
    static constexpr int MPL = N / 32;              // source cells per lane
    // padded index of the Toeplitz tables: lanes MPL entries apart on an
    // odd stride
    static constexpr int LG = 4;
    static constexpr int WN = N + GROUPS * RT;
    static constexpr int WLEN = WN + (WN >> LG) + 1;
    static_assert(YP % UN == 0 && GROUPS <= NW && (R + 4) % RT == 0
                  && N == NT && C <= RES_MAX_C && MPL == 1 << LG, "shape");

    // float offsets of the dynamic shared memory
    static constexpr int TL = LINES * R;              // a density
    static constexpr int oT = 0;                      // [2]
    static constexpr int oDW = oT + 2 * TL;           // [NW][YP][12]
    static constexpr int oH = oDW + NW * YP * 12;     // [2][2][N][2]
    static constexpr int oP = oH + 8 * N;             // [2][N]
    static constexpr int oW = oP + 2 * N;
    static constexpr int oKT = oW + res_up4(WLEN);
    static constexpr int oST = oKT + res_up4(WLEN);       // [2][R + 4][4]
    static constexpr int oE = oST + 8 * (R + 4);      // [NW][YP][4]
    static constexpr int oPS = oE + NW * YP * 4;      // [NW][R]
    static constexpr int oSB = oPS + NW * R;          // [R + 4][5]
    static constexpr int oCSR = res_up4(oSB + 5 * (R + 4));   // [2][C][CG][2]
    static constexpr int oMISC = oCSR + 4 * C * CG;
    static constexpr int oBAR = oMISC + 4;            // two mbarriers
    static constexpr size_t BYTES = (oBAR + 4) * sizeof(float);
    static_assert(BYTES <= 227 * 1024, "shared memory of a CTA");
};

// cluster_send where addr is not 0
__device__ __forceinline__ void cluster_send_if(uint32_t to, uint32_t addr,
                                                float v, uint32_t bar)
{
    asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %0, 0;\n"
                 "@p st.async.shared::cluster.mbarrier::complete_tx::bytes"
                 ".f32 [%1], %2, [%3];\n}"
                 :: "r"(to), "r"(addr), "f"(v), "r"(bar) : "memory");
}

__global__ void __launch_bounds__(Col::NT, 1)
k_bcol(const __grid_constant__ ResArgs A)
{
    using S = Col;
    constexpr int N = S::N, NW = S::NW, NT = S::NT, R = S::R, C = S::C;
    constexpr int RT = S::RT, Y = S::Y, YP = S::YP, UN = S::UN, DR = S::DR;
    constexpr int PAD = S::PAD;
    extern __shared__ float4 smem4[];
    float* sm = reinterpret_cast<float*>(smem4);
    float* W = sm + S::oW;
    float* KT = sm + S::oKT;
    float4* ST = reinterpret_cast<float4*>(sm + S::oST);
    float* SB = sm + S::oSB;             // RF stencils: shift, 4 weights
    float2* cpart = reinterpret_cast<float2*>(sm + S::oCSR);
    float* fac_s = sm + S::oMISC;
    // P and halo rows of even and odd steps complete
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + S::oBAR);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = int(cluster_rank());
    const uint32_t cl = cluster_id_x(), ncl = cluster_count_x();
    const int x0 = rank * R;            // the CTA's first row
    const int ya = warp * Y;            // the warp's first column
    // the first two and the last two rows go to a neighbour: the lane's
    // place in its H, its barriers
    uint32_t h_to = 0, hb_to = 0;
    if (lane < 2 && rank > 0) {
        h_to = cluster_map(smem_addr(sm + S::oH + 2 * N + lane), rank - 1);
        hb_to = cluster_map(smem_addr(bar), rank - 1);
    }
    if (lane >= 30 && rank < C - 1) {
        h_to = cluster_map(smem_addr(sm + S::oH + lane - 30), rank + 1);
        hb_to = cluster_map(smem_addr(bar), rank + 1);
    }
    if (threadIdx.x == 0) {
        mbar_init(&bar[0], NW);
        mbar_init(&bar[1], NW);
        mbar_fence_init();
    }
    uint32_t gs = 0;   // steps of this launch so far, over its bunches
    int bad = 0;       // a wait ran out
    for (int i = threadIdx.x; i < int(2 * S::TL); i += NT) {
        sm[S::oT + i] = 0.f;
    }

    for (uint32_t bi = cl; bi < A.nlist; bi += ncl) {
        const uint32_t b = A.list[bi];
        const BDev& BD = A.bd[b];
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
        // ---- the bunch's rows (transposed by way of the other density)
        // and tables
        float* stage = sm + S::oT + ((gs + 1) & 1) * S::TL;
        {
            const float* src = A.din + BD.dens_off + size_t(x0) * N;
#pragma unroll 8
            for (int i = threadIdx.x; i < R * N; i += NT) {
                stage[(i / N) * (N + 1) + i % N] = __ldg(src + i);
            }
        }
        for (int i = threadIdx.x; i < N; i += NT) {
            sm[S::oP + (gs & 1) * N + i] = A.pin[prof_off + i];
        }
        for (int i = threadIdx.x; i < 4 * N; i += NT) {
            const int h = i / N, y = i % N;
            const int x = x0 + (h < 2 ? h - 2 : R + h - 2);
            float* at = sm + S::oH + (h >> 1) * 2 * N + 2 * y + (h & 1);
            if (unsigned(x) < unsigned(N)) {
                at[(gs & 1) * 4 * N] = A.din[BD.dens_off + size_t(x) * N + y];
            } else {
                // rows off the mesh are zero (nothing writes them)
                at[0] = at[4 * N] = 0.f;
            }
        }
        if (has_wake) {
            const int nmax = int(BD.nmax);
            const float* w = A.wt + BD.wt_off;
            for (int k = threadIdx.x; k < S::WN; k += NT) {
                int i = (x0 - 2 + k - N) % nmax;
                i += i < 0 ? nmax : 0;
                W[k + (k >> S::LG)] = w[i];
            }
        }
        if (koff != NO_CSR) {
            for (int k = threadIdx.x + 1; k < N + R; k += NT) {
                KT[k + (k >> S::LG)] = A.csr.k[koff + x0 + k - 1];
            }
        }
        for (int i = threadIdx.x; i < R + 4; i += NT) {
            const int x = min(max(x0 - 2 + i, 0), N - 1);
            const RowStencil r = A.st[BD.st_off + ST_RF * N + x];
            SB[5 * i] = __int_as_float(r.shift0);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                SB[5 * i + 1 + j] = r.w[j];
            }
        }
        // the warp's column table, entry e of column y = ya - 2 + e: the
        // drift's weights of column y for the rows -2..2, the
        // Fokker-Planck weights of column y - 2 for -2..2, as
        //   form 1  no taps at 2: -2..1 of both     (lower energies)
        //   form 2  no taps at -2: -1..2 of both    (upper energies)
        //   form 0  -2..1 of both, then both at 2
        int form;
        {
            const float* dw = A.dwt + BD.dw_off;
            auto drift = [&](int e, int o) {   // row o of column ya - 2 + e
                const int y = ya - 2 + e;
                float v = 0.f;
                if (unsigned(y) < unsigned(N)) {
                    const int j = o - __float_as_int(dw[4 * N + y]);
                    v = unsigned(j) < 4u ? dw[j * N + y] : 0.f;
                }
                return v;
            };
            auto fokker = [&](int e, int o) {   // of column ya - 4 + e
                return e >= 4 ? dw[(7 + o) * N + ya - 4 + e] : 0.f;
            };
            bool low = true, high = true;
            for (int e = lane; e < YP; e += 32) {
                low = low && drift(e, 2) == 0.f && fokker(e, 2) == 0.f;
                high = high && drift(e, -2) == 0.f && fokker(e, -2) == 0.f;
            }
            form = __all_sync(0xffffffffu, low) ? 1
                   : __all_sync(0xffffffffu, high) ? 2 : 0;
            const int o0 = form == 2 ? -1 : -2;
            float* wt = sm + S::oDW + warp * YP * 12;
            for (int i = lane; i < YP * 12; i += 32) {
                const int e = i / 12, k = i % 12;
                wt[i] = k < 4 ? drift(e, o0 + k)
                        : k < 8 ? fokker(e, o0 + k - 4)
                        : k == 8 ? drift(e, 2) : fokker(e, 2);
            }
        }
        __syncthreads();
        {
            float* T = sm + S::oT + (gs & 1) * S::TL;
            for (int y = warp; y < N; y += NW) {
                T[(PAD + y) * R + lane] = stage[lane * (N + 1) + y];
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < PAD * R; i += NT) {
            stage[i] = 0.f;
            stage[(PAD + N) * R + i] = 0.f;
        }
        cluster_barrier<S::C>();   // tables complete; every CTA is running

        // the CSR power of step csr_step from its parts (warp 0 of rank 0,
        // one step later; two buffers, so that the next parts may arrive)
        bool csr_pending = false;
        unsigned csr_step = 0, csr_buf = 0;
        auto csr_store = [&] {
            if (!csr_pending) {
                return;
            }
            csr_pending = false;
            const float tot = groups_sum(cpart + csr_buf * C * S::CG,
                                         C * S::CG, lane);
            if (lane == 0) {
                const uint32_t slot = (csr_step / A.csr.every) % A.csr.cap;
                A.csr.power[size_t(slot) * A.csr.nb + b] = tot;
                if (b == 0) {
                    A.csr.steps[slot] = csr_step;
                }
            }
        };
        for (uint32_t t = 0; t < A.nsteps; t++, gs++) {
            const float* P = sm + S::oP + (gs & 1) * N;
            const uint32_t pn = S::oP + ((gs + 1) & 1) * N;   // the next one
            const unsigned step = step0 + t;
            const bool lastst = t + 1 == A.nsteps;
            const bool renorm_now = renorm > 0
                                    && (step % unsigned(renorm)) == 0;
            const bool csr_now = koff != NO_CSR && step % A.csr.every == 0;
            auto charge = [&] { return profile_charge<N>(P, ws, lane); };
            if (renorm_now) {
                if (warp == 0) {
                    const double q = charge();
                    if (lane == 0) {
                        fac_s[0] = fillset > 0
                                       ? static_cast<float>(double(fillset)
                                                            / q)
                                       : 0.f;
                    }
                }
                __syncthreads();
            }
            // ---- wake sums of the warp's group of rows and their composite
            // y-kicks
            if (warp < S::GROUPS) {
                const int at = lane / (32 / RT);
                const int r = warp * RT + at;     // row x0 - 2 + r
                float wk = 0.f;
                RowStencil sa;
                if (has_wake) {
                    float sum;
                    toeplitz_rows<S, RT>(P, W, warp * RT, lane, sum);
                    wk = __fmul_rn(wakescale, sum);
                    sa = make_stencil(wk, N, it);
                } else {
                    sa.shift0 = 0;
                    sa.w[0] = 1.f;
                    sa.w[1] = sa.w[2] = sa.w[3] = 0.f;
                }
                if (lane % (32 / RT) == 0 && r < R + 4) {
                    const float fac = renorm_now ? fac_s[0] : 1.f;
                    const float* sb = SB + 5 * r;
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
                    // own rows by lane, then the halo rows -2 -1 R R+1
                    const int x = r - 2;
                    const int to = x < 0 ? R + r : x >= R ? r : x;
                    ST[to] = make_float4(__int_as_float(s), c[0], c[1],
                                         c[2]);
                    ST[R + 4 + to] = make_float4(c[3], c[4], c[5], c[6]);
                    if (lastst && unsigned(x) < unsigned(R)) {
                        A.wake[prof_off + x0 + x] = wk;
                    }
                }
            }
            if (csr_now) {
                // the CTA's rows' part of the CSR power, in groups of rows
                const int g = NW - 1 - warp;
                if (g < S::CG) {
                    float v;
                    const int at = toeplitz_rows<S, RT>(P, KT, g * RT, lane,
                                                        v);
                    FF dot = FF{0.f, 0.f};
                    if (lane % (32 / RT) == 0) {
                        dot = ff_prod(P[x0 + g * RT + at], v);
                    }
                    dot = rows_sum(dot, 32 / RT);
                    if (lane == 0) {
                        // (with the step's row sums)
                        float2* cp = cpart + ((t & 1) * C + rank) * S::CG + g;
                        if (rank > 0) {
                            cluster_send2(
                                cluster_map(smem_addr(cp), 0),
                                make_float2(dot.hi, dot.lo),
                                cluster_map(smem_addr(&bar[gs & 1]), 0));
                        } else {
                            *cp = make_float2(dot.hi, dot.lo);
                        }
                    }
                }
            }
            if (__syncthreads_or(bad)) {
                bad = 1;
                break;
            }
            // the step's charge (its sign is watched; its value kept of the
            // last step) and the last step's CSR power
            if (rank == 0 && warp == 0) {
                csr_store();
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
                csr_step = step;
                csr_buf = t & 1;
                csr_pending = true;
            }
            // ---- the halo rows' y-kick on the warp's columns
            float4* E = reinterpret_cast<float4*>(sm + S::oE) + warp * YP;
            const float* H = sm + S::oH + (gs & 1) * 4 * N;
#pragma unroll
            for (int i0 = 0; i0 < 4 * YP; i0 += 32) {
                const int i = i0 + lane;
                if (i < 4 * YP) {
                    const int h = i / YP, e = i - h * YP;
                    const float4 q0 = ST[R + h], q1 = ST[2 * R + 4 + h];
                    const float c[7] = {q0.y, q0.z, q0.w, q1.x, q1.y,
                                        q1.z, q1.w};
                    const int y = ya - 2 + e + __float_as_int(q0.x);
                    const float* hp = H + (h >> 1) * 2 * N + (h & 1);
                    float v = 0.f;
#pragma unroll
                    for (int k = 0; k < 7; k++) {
                        const float d = unsigned(y + k) < unsigned(N)
                                            ? hp[2 * (y + k)] : 0.f;
                        v = k == 0 ? c[0] * d : fmaf(c[k], d, v);
                    }
                    reinterpret_cast<float*>(E + e)[h] = v;
                }
            }
            __syncwarp();
            // ---- the columns
            const float* T = sm + S::oT + (gs & 1) * S::TL;
            float* Tn = sm + S::oT + ((gs + 1) & 1) * S::TL;
            const float4 q0 = ST[lane], q1 = ST[R + 4 + lane];
            const float c[7] = {q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
            const int s = __float_as_int(q0.x);
            const uint32_t hn = h_to + ((gs + 1) & 1) * 16u * N;
            const uint32_t hb = hb_to + (gs & 1) * 8u;
            auto walk = [&](auto far, auto form_) {
                constexpr bool FAR = decltype(far)::value != 0;
                constexpr int FORM = decltype(form_)::value;
                // element e of the row's window: line ya - 2 + s + e (far:
                // any shift; lines 0 and LINES - 1 are zero)
                int line = PAD + ya - 2 + s;
                const float* tp = T + (FAR ? 0 : line * R) + lane;
                auto load = [&](int e) {
                    return tp[(FAR ? min(max(line + e, 0), S::LINES - 1) : e)
                              * R];
                };
                float win[UN];
#pragma unroll
                for (int e = 0; e < UN - 1; e++) {
                    win[e] = load(e);
                }
                const float4* wt = reinterpret_cast<const float4*>(sm + S::oDW)
                                   + 3 * warp * YP;
                const float4* ep = E;
                float* to = Tn + (PAD + ya - 4) * R + lane;
                uint32_t hy = hn + 8u * uint32_t(ya - 4);
                // the row's sum over the warp's 8 words, neighbours first:
                // words -, 0, 1 of the first turn, 2 3 4 and 5 6 7 of the others
                float d[DR], ps = 0.f, odd = 0.f;
#pragma unroll 1
                for (int e0 = 0; e0 < YP; e0 += UN) {
                    float word[UN / 4] = {}, p0 = 0.f, p1 = 0.f;
                    const float wfirst = ya + e0 == 0 ? 1.f : 2.f;
                    const float wlast = ya + e0 + UN - 5 == N - 1 ? 1.f : 4.f;
#pragma unroll
                    for (int u = 0; u < UN; u++) {
                        win[(u + UN - 1) % UN] = load(u + UN - 1);
                        const float4 w0 = wt[3 * u], f0 = wt[3 * u + 1];
                        float2 at2 = make_float2(0.f, 0.f);
                        if (FORM == 0) {
                            at2 = *reinterpret_cast<const float2*>(
                                wt + 3 * u + 2);
                        }
                        const float4 ev = ep[u];
                        float kv = c[0] * win[u];
#pragma unroll
                        for (int k = 1; k < 7; k++) {
                            kv = fmaf(c[k], win[(u + k) % UN], kv);
                        }
                        // the rows -2 .. 2 around the lane's
                        float g[5];
                        g[2] = kv;
                        if (FORM != 2) {
                            g[0] = __shfl_up_sync(0xffffffffu, kv, 2);
                            g[0] = lane == 0 ? ev.x : lane == 1 ? ev.y : g[0];
                        }
                        g[1] = __shfl_up_sync(0xffffffffu, kv, 1);
                        g[1] = lane == 0 ? ev.y : g[1];
                        g[3] = __shfl_down_sync(0xffffffffu, kv, 1);
                        g[3] = lane == 31 ? ev.z : g[3];
                        if (FORM != 1) {
                            g[4] = __shfl_down_sync(0xffffffffu, kv, 2);
                            g[4] = lane == 31 ? ev.w
                                   : lane == 30 ? ev.z : g[4];
                        }
                        constexpr int O = FORM == 2 ? 1 : 0;
                        float v = w0.x * g[O];
                        v = fmaf(w0.y, g[O + 1], v);
                        v = fmaf(w0.z, g[O + 2], v);
                        v = fmaf(w0.w, g[O + 3], v);
                        if (FORM == 0) {
                            v = fmaf(at2.x, g[4], v);
                        }
                        d[u % DR] = v;
                        if (u >= 4 || e0 > 0) {
                            // Fokker-Planck of column ya - 4 + e0 + u
                            float o = f0.x * d[(u + 2 * DR - 4 + O) % DR];
                            o = fmaf(f0.y, d[(u + 2 * DR - 3 + O) % DR], o);
                            o = fmaf(f0.z, d[(u + 2 * DR - 2 + O) % DR], o);
                            o = fmaf(f0.w, d[(u + 2 * DR - 1 + O) % DR], o);
                            if (FORM == 0) {
                                o = fmaf(at2.y, v, o);
                            }
                            to[u * R] = o;
                            // (Simpson weights 1 4 2 .. 2 4 1; ya is even)
                            const float sw = u == 4 ? wfirst
                                : u == UN - 1 ? wlast : u & 1 ? 4.f : 2.f;
                            if (u % 4 == 0) {
                                p0 = sw * o;
                            } else if (u % 4 == 1) {
                                p1 = sw * o;
                            } else if (u % 4 == 2) {
                                p0 = fmaf(sw, o, p0);
                            } else {
                                p1 = fmaf(sw, o, p1);
                                word[u / 4] = p0 + p1;
                            }
                            cluster_send_if(h_to, hy + 8u * u, o, hb);
                        }
                    }
                    static_assert(YP == 3 * UN && UN == 12, "8 words");
                    if (e0 == 0) {
                        ps = word[1] + word[2];
                    } else if (e0 == UN) {
                        ps += word[0] + word[1];
                        odd = word[2];
                    } else {
                        ps += (odd + word[0]) + (word[1] + word[2]);
                    }
                    tp += FAR ? 0 : UN * R;
                    line += UN;
                    wt += 3 * UN;
                    ep += UN;
                    to += UN * R;
                    hy += 8u * UN;
                }
                sm[S::oPS + warp * R + lane] = ps;
            };
            if (__all_sync(0xffffffffu,
                           s >= 2 - PAD && s <= PAD - 1 - UN)) {
                if (form == 1) {
                    walk(IntC<0>{}, IntC<1>{});
                } else if (form == 2) {
                    walk(IntC<0>{}, IntC<2>{});
                } else {
                    walk(IntC<0>{}, IntC<0>{});
                }
            } else if (form == 1) {
                walk(IntC<1>{}, IntC<1>{});
            } else if (form == 2) {
                walk(IntC<1>{}, IntC<2>{});
            } else {
                walk(IntC<1>{}, IntC<0>{});
            }
            __syncthreads();
            // ---- the rows' sums, to every CTA
            {
                const int r = lane, to = warp;   // (a warp per CTA)
                float f[NW];
#pragma unroll
                for (int w = 0; w < NW; w++) {
                    f[w] = sm[S::oPS + w * R + r];
                }
#pragma unroll
                for (int o = 1; o < NW; o <<= 1) {
#pragma unroll
                    for (int w = 0; w < NW; w += 2 * o) {
                        f[w] += f[w + o];
                    }
                }
                const float v = h03 * f[0];
                float* pa = sm + pn + x0 + r;
                if (to == rank) {
                    *pa = v;
                } else {
                    cluster_send(cluster_map(smem_addr(pa), to), v,
                                 cluster_map(smem_addr(&bar[gs & 1]), to));
                }
            }
            __syncwarp();
            if (threadIdx.x == 0) {
                mbar_arrive_expect_tx(
                    &bar[gs & 1],
                    uint32_t(N - R) * 4u
                        + uint32_t((rank > 0) + (rank < C - 1))
                              * uint32_t(N * 8)
                        + (csr_now && rank == 0
                               ? uint32_t((C - 1) * S::CG) * 8u : 0u));
            } else if (lane == 0) {
                mbar_arrive(&bar[gs & 1]);
            }
            if (!res_wait(&bar[gs & 1], (gs >> 1) & 1)) {
                bad = 1;
            }
        }
        if (__syncthreads_or(bad)) {
            bad = 1;
            break;
        }
        const float* P = sm + S::oP + (gs & 1) * N;
        if (rank == 0 && warp == 0) {
            csr_store();
        }
        // ---- the new state (transposed by way of the other density)
        {
            const float* T = sm + S::oT + (gs & 1) * S::TL;
            float* out = sm + S::oT + ((gs + 1) & 1) * S::TL;
            for (int y = warp; y < N; y += NW) {
                out[lane * (N + 1) + y] = T[(PAD + y) * R + lane];
            }
            __syncthreads();
            float* dst = A.dout + BD.dens_off + size_t(x0) * N;
#pragma unroll 8
            for (int i = threadIdx.x; i < R * N; i += NT) {
                dst[i] = out[(i / N) * (N + 1) + i % N];
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
    cluster_barrier<S::C>();   // no CTA leaves while another may send to it
}

}  // namespace
