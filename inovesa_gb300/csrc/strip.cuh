// k_bstrip: chain 0 (wake kick, RF kick, drift, Fokker-Planck) of 512- and
// 1024-row meshes, one step per launch (included by batch.cu).
//
// A CTA takes a tile of rows, a warp of it a strip of the columns (5 strips
// of 512, 10 of 1024; 4 columns per lane, a lane more on either side), and
// walks down the rows on its own:
//
//   staging   the columns that the row's y-kick reads, whatever its shift,
//             into a ring of the warp by 16-byte asynchronous copies, WIN - 1
//             rows ahead (columns off the mesh are filled with zeros);
//   y-kick    both kicks as one 7-tap stencil (RowInfo7) of the 16-byte
//             words around the lane's columns; the shift is the same for
//             the whole warp.  TURN (512-row lattices that are not regular,
//             F_TURN): the words at the energy axis' ends whose second kick
//             reaches past them get the two kicks in turn, as from k_bmaps0
//             (what the first one moves off the axis does not come back with
//             the second).  The first and the last warp compute these before
//             they walk, two rows per lane (64 bunches of 512 rows: 46 us a
//             step without, 53 so, 60 with the kicks in turn on the way
//             down the rows);
//   drift     the last WIN kicked rows in registers; every column's weights
//             lie on the rows its shift reaches from the strip's lowest
//             shift on (WIN = 4 + the widest spread of shifts in a strip);
//   Fokker-Planck   5 taps, neighbours by shuffles; the new row to memory.
//
// Nothing is shared between warps but the words' sums at the end, so 15 to 20
// warps of an SM run without a barrier.  A step of 24 bunches of 1024 rows:
// 71 us on k_bmaps0f (8 warps around a ring of whole rows), 55 us here (29
// us for its bytes at the memory's rate); 64 bunches of 512 rows whose drift
// has no shift in common 77 (on k_bmaps0<4>) and 53 us.  Bound by instruction
// issue and latency together: 120 instructions a row and warp, of a row's
// chain of 500 cycles, at 54 % of the issue slots (20 warps at 96 registers).
#pragma once

namespace {

constexpr int STRIP_ROWS = 44;    // rows of a tile at most
// words at either end of the axis that F_TURN computes apart, and the shifts
// of the second y-kick they are enough for
constexpr int STRIP_ENDS = 4;
constexpr int STRIP_TURN = 13;

// strips of a mesh: the strip, the lane before it and the one after it are
// 28 lanes at most, so that 32 words of 4 hold the window of a row's y-kick
__host__ __device__ constexpr int strips(int n)
{
    return n / 102;
}

// the strip's first group of 4 columns
__host__ __device__ constexpr int strip_begin(int n, int k)
{
    return k * (n / 4) / strips(n);
}

// a warp's shared memory in floats: the ring, the rows' stencils
__host__ __device__ constexpr int strip_floats(int win)
{
    return win * 128 + (STRIP_ROWS + win) * 8;
}

// the row sums of the words of 4 columns, a row (4 more: the lanes that add a
// row read 16 bytes each)
__host__ __device__ constexpr int strip_words(int n)
{
    return n / 4 + 4;
}

// TURN, for the first and the last strip: the rows' words at the axis' ends
__host__ __device__ constexpr int strip_turn_floats(int win)
{
    return (STRIP_ROWS + win) * 4 * STRIP_ENDS;
}

constexpr size_t strip_smem(int n, int win, bool turn)
{
    return sizeof(float) * (strips(n) * strip_floats(win)
                            + STRIP_ROWS * strip_words(n)
                            + (turn ? 2 * strip_turn_floats(win) : 0));
}

// 16 bytes to shared memory, or 16 zero bytes
__device__ __forceinline__ void strip_copy(uint32_t to, const void* from,
                                           bool in)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                 :: "r"(to), "l"(from), "r"(in ? 16 : 0) : "memory");
}

// 4 outputs of the 7-tap y-kick from the window v, whose first input is v[AL]
template <int AL>
__device__ __forceinline__ float4 strip_kick(const float (&v)[16],
                                             const float (&c)[7])
{
    float o[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        o[q] = c[0] * v[AL + q];
    }
#pragma unroll
    for (int k = 1; k < 7; k++) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            o[q] = fmaf(c[k], v[AL + q + k], o[q]);
        }
    }
    return make_float4(o[0], o[1], o[2], o[3]);
}

// the same by the two kicks in turn (r: RowInfo), of word g of a row in memory;
// the first kick's outputs are zero off the mesh
template <int N>
__device__ __forceinline__ float4 strip_turn(const float* row, int g,
                                             const float4 (&r)[3])
{
    const float a[4] = {r[0].z, r[0].w, r[1].x, r[1].y};
    const float b[4] = {r[1].z, r[1].w, r[2].x, r[2].y};
    const int at = 4 * g + __float_as_int(r[0].x);    // column of c[0]
    const int q0 = 4 * g + __float_as_int(r[0].y);    // column of t[0]
    float c[10], t[7], o[4];
#pragma unroll
    for (int i = 0; i < 10; i++) {
        c[i] = unsigned(at + i) < unsigned(N) ? row[at + i] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < 7; i++) {
        float v = a[0] * c[i];
#pragma unroll
        for (int j = 1; j < 4; j++) {
            v = fmaf(a[j], c[i + j], v);
        }
        t[i] = unsigned(q0 + i) < unsigned(N) ? v : 0.f;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
        o[q] = b[0] * t[q];
#pragma unroll
        for (int i = 1; i < 4; i++) {
            o[q] = fmaf(b[i], t[q + i], o[q]);
        }
    }
    return make_float4(o[0], o[1], o[2], o[3]);
}

template <int N, int WIN, bool TURN = false>
__global__ void __launch_bounds__(32 * strips(N), N == 512 ? 3 : 2)
k_bstrip(const BDev* __restrict__ bd, const Tile* __restrict__ tiles,
         const float* __restrict__ tabs, const float* __restrict__ dwt,
         const RowInfo7* rinfo,   // (k_bwake may still write them)
         const RowInfo* rinfo2,
         const float* __restrict__ din, float* __restrict__ dout,
         float* __restrict__ pout)
{
    // taps of a column in the table (1024 rows: 4 columns have one shift)
    constexpr int TAPS = N == 1024 ? 5 : 4;
    constexpr int NS = strips(N);
    extern __shared__ float4 smem4[];
    float* sm = reinterpret_cast<float*>(smem4);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* ring = sm + warp * strip_floats(WIN);          // [WIN][128]
    float* info = ring + WIN * 128;                       // [ROWS + WIN][8]
    constexpr int PS = strip_words(N);
    float* psum = sm + NS * strip_floats(WIN);            // [ROWS][PS]
    // [ROWS + WIN][ENDS]
    static_assert(strip_floats(WIN) % 4 == 0 && PS % 4 == 0, "16-byte words");
    float4* ends = reinterpret_cast<float4*>(
        psum + STRIP_ROWS * PS + (warp ? strip_turn_floats(WIN) : 0));
    const Tile t = tiles[blockIdx.x];
    const BDev& B = bd[t.bunch];
    const int rows = int(t.rows);
    const int g0 = strip_begin(N, warp), g1 = strip_begin(N, warp + 1);
    const int g = g0 - 1 + lane;
    const bool in = unsigned(g) < unsigned(N / 4);
    const bool mine = g >= g0 && g < g1;
    const int y = 4 * g, yc = in ? y : 0;
    // ---- the lane's weights: drift taps on the rows from the strip's
    // lowest shift d0 on, Fokker-Planck, Simpson (in units of h03)
    const float* dw = dwt + B.dw_off;
    int sh[4], d0 = INT_MAX;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        sh[q] = __float_as_int(dw[TAPS * N + yc + q]);
        d0 = in && g <= g1 ? min(d0, sh[q]) : d0;
    }
    d0 = __reduce_min_sync(0xffffffffu, d0);
    float wd[WIN][4];
    float4 fw[5];
    {
        float tap[TAPS][4];
#pragma unroll
        for (int j = 0; j < TAPS; j++) {
            const float4 v = *reinterpret_cast<const float4*>(dw + j * N
                                                              + yc);
            tap[j][0] = v.x;
            tap[j][1] = v.y;
            tap[j][2] = v.z;
            tap[j][3] = v.w;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
#pragma unroll
            for (int j = 0; j < WIN; j++) {
                float v = 0.f;
#pragma unroll
                for (int k = 0; k < TAPS; k++) {
                    v = j - k == sh[q] - d0 && in ? tap[k][q] : v;
                }
                wd[j][q] = v;
            }
        }
#pragma unroll
        for (int o = 0; o < 5; o++) {
            fw[o] = *reinterpret_cast<const float4*>(
                dw + (TAPS + 1 + o) * N + yc);
        }
    }
    const float a0 = y == 0 ? 1.f : 2.f, a3 = y == N - 4 ? 1.f : 4.f;
    // ---- the kicked rows k0 .. k0 + nk - 1 of the mesh
    const int x0 = int(t.x0);
    const int k0 = x0 + d0, nk = rows + WIN - 1;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int i = lane; i < 2 * nk; i += 32) {
        const int x = k0 + (i >> 1);
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (unsigned(x) < unsigned(N)) {
            v = reinterpret_cast<const float4*>(rinfo + B.prof_off + x)[i & 1];
        }
        reinterpret_cast<float4*>(info)[i] = v;
    }
    __syncwarp();
    // row i of the ring, into slot `slot`
    const uint32_t ring_at = smem_addr(ring) + 16u * lane;
    const float* src = din + B.dens_off;
    const int c0 = 4 * (g0 - 1 + lane);
    auto issue = [&](int i, int slot) {
        if (i < nk) {
            const int x = k0 + i;
            const int c = c0 + (__float_as_int(info[8 * i]) & ~3);
            const bool ok = unsigned(x) < unsigned(N)
                            && unsigned(c) < unsigned(N);
            strip_copy(ring_at + 512u * slot, src + (ok ? x * N + c : 0), ok);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int i = 0; i < WIN - 1; i++) {
        issue(i, i);
    }
    // the row's word from the axis' end on (0 the outermost), where the first
    // `words` of them are computed apart
    int end = 0, words = 0;
    if (TURN && (warp == 0 || warp == NS - 1)) {
        static_assert(STRIP_ROWS + WIN - 1 <= 64, "two rows per lane");
        end = warp == 0 ? g : N / 4 - 1 - g;
        auto word = [&](int e) { return warp == 0 ? e : N / 4 - 1 - e; };
        float4 r[2][3];
        bool ok[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int i = lane + 32 * u, x = k0 + i;
            ok[u] = i < nk && unsigned(x) < unsigned(N);
#pragma unroll
            for (int q = 0; q < 3; q++) {
                r[u][q] = ok[u] ? reinterpret_cast<const float4*>(
                                      rinfo2 + B.prof_off + x)[q]
                                : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int e = 0; e < STRIP_ENDS; e++) {
                const int at = 4 * word(e) + __float_as_int(r[u][0].y);
                words = ok[u] && (at < 0 || at + 6 >= N) ? max(words, e + 1)
                                                         : words;
            }
        }
        words = __reduce_max_sync(0xffffffffu, words);
#pragma unroll 1
        for (int e = 0; e < words; e++) {
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int i = lane + 32 * u;
                if (i < nk) {
                    ends[STRIP_ENDS * i + e] =
                        ok[u] ? strip_turn<N>(src + (k0 + i) * N, word(e),
                                              r[u])
                              : make_float4(0.f, 0.f, 0.f, 0.f);
                }
            }
        }
        __syncwarp();
    }
    const bool apart = TURN && unsigned(end) < unsigned(words);
    float4 K[WIN];
    float* dst = dout + B.dens_off + size_t(x0) * N + yc;
    float* pto = psum + (in ? g : 0);
#pragma unroll 1
    for (int i0 = 0; i0 < nk; i0 += WIN) {
#pragma unroll
        for (int k = 0; k < WIN; k++) {
            const int i = i0 + k;
            if (i >= nk) {
                break;
            }
            asm volatile("cp.async.wait_group %0;" :: "n"(WIN - 2)
                         : "memory");
            __syncwarp();   // (every lane has read the row before)
            issue(i + WIN - 1, (k + WIN - 1) % WIN);
            // ---- y-kick
            const float4 q0 = *reinterpret_cast<const float4*>(info + 8 * i);
            const float4 q1 = *reinterpret_cast<const float4*>(info + 8 * i
                                                               + 4);
            const float c[7] = {q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
            const int s = __float_as_int(q0.x);
            // (the lanes past the strip's window read within the warp's
            // memory; their columns go unused)
            float v[16];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float4 u = reinterpret_cast<const float4*>(
                    ring + 128 * k)[lane + j];
                v[4 * j] = u.x;
                v[4 * j + 1] = u.y;
                v[4 * j + 2] = u.z;
                v[4 * j + 3] = u.w;
            }
            if (s & 2) {
                K[k] = s & 1 ? strip_kick<3>(v, c) : strip_kick<2>(v, c);
            } else {
                K[k] = s & 1 ? strip_kick<1>(v, c) : strip_kick<0>(v, c);
            }
            if (apart) {
                K[k] = ends[STRIP_ENDS * i + end];
            }
            if (i0 == 0 && k < WIN - 1) {
                continue;
            }
            // ---- drift
            float2 lo, hi;
#pragma unroll
            for (int j = 0; j < WIN; j++) {
                const float4 r = K[(k + 1 + j) % WIN];
                const float2 wl = make_float2(wd[j][0], wd[j][1]);
                const float2 wh = make_float2(wd[j][2], wd[j][3]);
                if (j == 0) {
                    lo = __fmul2_rn(wl, make_float2(r.x, r.y));
                    hi = __fmul2_rn(wh, make_float2(r.z, r.w));
                } else {
                    lo = __ffma2_rn(wl, make_float2(r.x, r.y), lo);
                    hi = __ffma2_rn(wh, make_float2(r.z, r.w), hi);
                }
            }
            // ---- Fokker-Planck
            float w[8];
            w[2] = lo.x;
            w[3] = lo.y;
            w[4] = hi.x;
            w[5] = hi.y;
            w[0] = __shfl_up_sync(0xffffffffu, hi.x, 1);
            w[1] = __shfl_up_sync(0xffffffffu, hi.y, 1);
            w[6] = __shfl_down_sync(0xffffffffu, lo.x, 1);
            w[7] = __shfl_down_sync(0xffffffffu, lo.y, 1);
            float o[4];
#pragma unroll
            for (int h = 0; h < 5; h++) {
                const float f[4] = {fw[h].x, fw[h].y, fw[h].z, fw[h].w};
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    o[q] = h == 0 ? f[q] * w[q] : fmaf(f[q], w[q + h], o[q]);
                }
            }
            if (mine) {
                *reinterpret_cast<float4*>(dst + (k - (WIN - 1)) * N) =
                    make_float4(o[0], o[1], o[2], o[3]);
            }
            // ---- the word's part of the row's sum
            if (mine) {
                pto[PS * (k - (WIN - 1))] = fmaf(2.f, o[2], a0 * o[0])
                                            + fmaf(a3, o[3], 4.f * o[1]);
            }
        }
        dst += WIN * N;
        pto += PS * WIN;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // the rows' sums, neighbours first: N / 128 words a lane, then the lanes
    const float h03 = tabs[B.tab_off + TAB_WS * N];
#pragma unroll 2
    for (int r = warp; r < rows; r += NS) {
        constexpr int Q = N / 512;   // 16-byte words of sums a lane
        float v = 0.f;
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const float4 f = *reinterpret_cast<const float4*>(
                psum + PS * r + 4 * (Q * lane + q));
            const float u = (f.x + f.y) + (f.z + f.w);
            v = q == 0 ? u : v + u;
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            v += __shfl_xor_sync(0xffffffffu, v, o);
        }
        if (lane == 0) {
            pout[B.prof_off + x0 + r] = h03 * v;
        }
    }
}

}  // namespace
