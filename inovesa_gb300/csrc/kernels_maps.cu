// Plain (one map per launch) SourceMap kernels.  Weights are evaluated in
// registers from the source coordinate -- the reference's per-cell
// (index, weight) tables (8 B per tap) are never materialised.
//
//  k_rotation  RotationMap::genHInfo + apply (src/SM/RotationMap.cpp:97-260)
//  k_kick_y    KickMap y-kick, one CTA per mesh row (src/SM/KickMap.cpp:244-266)
//  k_kick_x    KickMap x-kick (src/SM/KickMap.cpp:221-242)
//  k_fp        FokkerPlanckMap::apply (src/SM/FokkerPlanckMap.cpp:170-213)
#include <algorithm>
#include <cfloat>
#include <climits>

#include "vfps_internal.cuh"

namespace vfps {
namespace {

using namespace dev;

// Taps (i1, j1) of a source cell's neighbourhood, kept from one output row
// to the next: with the base's column unchanged and its row one further
// (small angles: nearly always), rows 1..IT-1 move up and only the last row
// is read.
template <int IT>
struct RotTaps {
    int x = INT_MIN, y = 0;
    float v[IT][IT];
    // taps off the mesh are 0
    __device__ __forceinline__ void move(const float* src,
                                         int n, int x1, int y1)
    {
        constexpr int h = (IT - 1) / 2;
        auto row = [&](int i1) {
            const int i0 = x1 + i1 - h;
            const float* p = src + size_t(i0 < 0 ? 0 : i0) * n;
#pragma unroll
            for (int j1 = 0; j1 < IT; j1++) {
                const int j0 = y1 + j1 - h;
                v[i1][j1] = unsigned(i0) < unsigned(n)
                                    && unsigned(j0) < unsigned(n)
                                ? p[j0] : 0.f;
            }
        };
        if (y1 == y && x1 == x + 1) {
#pragma unroll
            for (int i1 = 0; i1 + 1 < IT; i1++) {
#pragma unroll
                for (int j1 = 0; j1 < IT; j1++) {
                    v[i1][j1] = v[i1 + 1][j1];
                }
            }
            row(IT - 1);
        } else {
#pragma unroll
            for (int i1 = 0; i1 < IT; i1++) {
                row(i1);
            }
        }
        x = x1;
        y = y1;
    }
};

// A thread per column y and `rows` output rows.  Each output as in
// src/SM/RotationMap.cpp: the sum over the taps in order, no FMA.  A tap off
// the mesh adds fmul(0, w) = +-0, which changes nothing.
template <int IT, bool CLAMP>
__global__ void __launch_bounds__(128)
k_rotation(const float* in, float* __restrict__ out, uint32_t n,
           const float* __restrict__ qv, const float* __restrict__ pv,
           float dq, float dp, float zbq, float zbp, float cs, float sn,
           int rows)
{
    pdl_trigger();
    const uint32_t y0 = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t xa = blockIdx.y * rows;
    const uint32_t xe = min(n, xa + rows);
    pdl_wait();
    if (y0 >= n) {
        return;
    }
    const size_t nxy = size_t(n) * n;
    const float* src = in + blockIdx.z * nxy;
    float* dst = out + blockIdx.z * nxy + y0;
    const float p = pv[y0];
    const float snp = fmul(sn, p), csp = fmul(cs, p);
    const float cell0 = CLAMP ? *src : 0.f;
    constexpr int h = (IT - 1) / 2;
    RotTaps<IT> t;
    for (uint32_t x0 = xa; x0 < xe; x0++) {
        const float q = __ldg(qv + x0);
        const float x1r = fadd(fdiv(fsub(fmul(cs, q), snp), dq), zbq);
        const float y1r = fadd(fdiv(fadd(fmul(sn, q), csp), dp), zbp);
        int x1 = 0, y1 = 0;
        float xf, yf;
        const bool okx = base_index(x1r, n, &x1, &xf);
        const bool oky = base_index(y1r, n, &y1, &yf);
        const bool ok = okx && oky;
        float value = 0.f;
        if (ok) {
            float icq[4], icp[4];
            coefficients(icq, xf, IT);
            coefficients(icp, yf, IT);
            t.move(src, int(n), x1, y1);
#pragma unroll
            for (int i1 = 0; i1 < IT; i1++) {
#pragma unroll
                for (int j1 = 0; j1 < IT; j1++) {
                    value = fadd(value, fmul(t.v[i1][j1],
                                             fmul(icq[i1], icp[j1])));
                }
            }
        }
        if (CLAMP) {
            // src/SM/RotationMap.cpp:159-172: range of the 2x2 nearest
            // taps, starting from FLT_MIN / FLT_MAX; taps off the mesh read
            // cell 0
            float ceil_v = FLT_MIN, flor_v = FLT_MAX;
#pragma unroll
            for (int i1 = 1; i1 <= 2; i1++) {
#pragma unroll
                for (int j1 = 1; j1 <= 2; j1++) {
                    const int i0 = x1 + i1 - h, j0 = y1 + j1 - h;
                    const bool in_mesh = ok && unsigned(i0) < n
                                         && unsigned(j0) < n;
                    const float v = in_mesh ? t.v[i1 < IT ? i1 : 0]
                                                 [j1 < IT ? j1 : 0]
                                            : cell0;
                    ceil_v = (ceil_v < v) ? v : ceil_v;
                    flor_v = (v < flor_v) ? v : flor_v;
                }
            }
            const float c = (value < ceil_v) ? value : ceil_v;
            value = (c < flor_v) ? flor_v : c;
        }
        dst[size_t(x0) * n] = value;
    }
}

// The reference's CPU KickMap never clamps (its interpol_clamp flag only
// prints a notice, src/SM/KickMap.cpp:42-44), so the kick kernels follow
// that path and take no clamp argument.

// one CTA per (bunch, row x); offsets[b*n + x] in mesh units
__global__ void k_kick_y(const float* in, float* __restrict__ out,
                         const float* offsets, uint32_t n, int it)
{
    pdl_trigger();
    pdl_wait();
    const uint32_t row = blockIdx.x;
    const KickStencil s = kick_stencil(offsets[row], n, it);
    const float* src = in + size_t(row) * n;
    float* dst = out + size_t(row) * n;
    for (uint32_t y = threadIdx.x; y < n; y += blockDim.x) {
        float value = 0.f;
        for (int j = 0; j < it; j++) {
            const int ys = int(y) + s.shift[j];
            if (s.valid[j] && ys >= 0 && ys < int(n)) {
                value = fadd(value, fmul(src[ys], s.w[j]));
            }
        }
        dst[y] = value;
    }
}

// thread per cell; offsets[y] shared by all bunches
__global__ void k_kick_x(const float* in, float* __restrict__ out,
                         const float* offsets, uint32_t n, int it)
{
    pdl_trigger();
    pdl_wait();
    const uint32_t y = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t x = blockIdx.y;
    if (y >= n) {
        return;
    }
    const size_t nxy = size_t(n) * n;
    const float* src = in + blockIdx.z * nxy;
    const KickStencil s = kick_stencil(offsets[y], n, it);
    float value = 0.f;
    for (int j = 0; j < it; j++) {
        const int xs = int(x) + s.shift[j];
        if (s.valid[j] && xs >= 0 && xs < int(n)) {
            value = fadd(value, fmul(src[size_t(xs) * n + y], s.w[j]));
        }
    }
    out[blockIdx.z * nxy + size_t(x) * n + y] = value;
}

// thread per cell; stencil table idx/w [n][ip] shared by every row
__global__ void k_fp(const float* in, float* __restrict__ out,
                     const uint32_t* __restrict__ idx,
                     const float* __restrict__ w, uint32_t n, int ip)
{
    pdl_trigger();
    pdl_wait();
    const uint32_t y = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t x = blockIdx.y;
    if (y >= n) {
        return;
    }
    const size_t row = (blockIdx.z * size_t(n) + x) * n;
    float value = 0.f;
    for (int j = 0; j < ip; j++) {
        value = fadd(value, fmul(in[row + idx[y * ip + j]],
                                 w[y * ip + j]));
    }
    out[row + y] = value;
}

// ------------------------------------------------ row-sweep forms
// Meshes whose side is a multiple of 4 (up to PLAIN_V4_MAX) take these
// instead of the thread-per-cell kernels above: 16-byte row sweeps in and
// out, the stencils computed once per thread for its 4 columns and kept
// in registers, and rows staged in shared memory where a stencil reads
// along the row.  Every output is the same sum in the same order as the
// kernels above; a tap outside the mesh reads a zero pad instead of being
// skipped, and adds fmul(0, w) = +-0 (an exact no-op, because the sum is
// never -0).

// one output group: taps j < it of the aligned window v (AL: offset of
// the first tap of the first output)
template <int AL>
__device__ __forceinline__ float4 kick_row4(const float4 (&v4)[3],
                                            const float (&w)[4], int it)
{
    const float v[12] = {v4[0].x, v4[0].y, v4[0].z, v4[0].w,
                         v4[1].x, v4[1].y, v4[1].z, v4[1].w,
                         v4[2].x, v4[2].y, v4[2].z, v4[2].w};
    float o[4];
#pragma unroll
    for (int c = 0; c < 4; c++) {
        float value = 0.f;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (j < it) {
                value = fadd(value, fmul(v[AL + c + j], w[j]));
            }
        }
        o[c] = value;
    }
    return make_float4(o[0], o[1], o[2], o[3]);
}

// y-kick, one CTA per (bunch, row): the row in shared memory between zero
// pads of kick_pad(n) floats (a valid tap lies at most n/2 + 3 columns
// away), the stencil uniform over the row, 4 outputs per thread from 3
// aligned 16-byte reads (the window's alignment is the same for the whole
// row)
__host__ __device__ inline int kick_pad(uint32_t n)
{
    return int(((n / 2 + 3) & ~3u) + 16);
}

__global__ void k_kick_y4(const float* in, float* __restrict__ out,
                          const float* offsets, uint32_t n,
                          int it)
{
    pdl_trigger();
    pdl_wait();
    extern __shared__ float4 row4[];
    const uint32_t row = blockIdx.x;
    const KickStencil s = kick_stencil(offsets[row], n, it);
    const int pad4 = kick_pad(n) / 4, n4 = int(n / 4);
    const float4* src = reinterpret_cast<const float4*>(in + size_t(row) * n);
    float4* dst = reinterpret_cast<float4*>(out + size_t(row) * n);
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    const bool any = s.valid[0] || s.valid[1] || s.valid[2] || s.valid[3];
    if (!any) {   // no tap inside the mesh: the row is zero
        for (int i = threadIdx.x; i < n4; i += blockDim.x) {
            dst[i] = z;
        }
        return;
    }
    for (int i = threadIdx.x; i < 2 * pad4 + n4; i += blockDim.x) {
        const int k = i - pad4;
        row4[i] = (k >= 0 && k < n4) ? src[k] : z;
    }
    __syncthreads();
    // shift[0] lies in [-n/2 - 3, n/2): every window inside the pads
    const int s0 = s.shift[0];
    const int al = s0 & 3;
    const int b4 = pad4 + ((s0 - al) >> 2);
    for (int i = threadIdx.x; i < n4; i += blockDim.x) {
        const float4 v[3] = {row4[b4 + i], row4[b4 + i + 1],
                             row4[b4 + i + 2]};
        float4 o;
        switch (al) {
        case 0: o = kick_row4<0>(v, s.w, it); break;
        case 1: o = kick_row4<1>(v, s.w, it); break;
        case 2: o = kick_row4<2>(v, s.w, it); break;
        default: o = kick_row4<3>(v, s.w, it); break;
        }
        dst[i] = o;
    }
}

// the x-kick's stencils of every column, tap-major: shift[j][y], w[j][y]
// (the same function the kernels evaluate, computed once per set of
// offsets)
__global__ void k_kick_table(const float* offsets, uint32_t n,
                             int it, int* __restrict__ shift,
                             float* __restrict__ w)
{
    pdl_trigger();
    pdl_wait();
    const uint32_t y = blockIdx.x * blockDim.x + threadIdx.x;
    if (y >= n) {
        return;
    }
    const KickStencil s = kick_stencil(offsets[y], n, it);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        shift[j * n + y] = s.shift[j];
        w[j * n + y] = s.w[j];
    }
}

// x-kick: a CTA per block of rows and block of column groups of one bunch;
// each thread owns 4 columns (their stencils, one per column, loaded from
// the table in 16-byte words) and sweeps the rows.  Where the 4 columns take
// the same shifts, the 4 tap rows move through registers (one 16-byte read
// per output row; a row off the mesh is zero); column by column otherwise.
// 2048 x 2048: 15.6 us with every tap row read for every output and 3 rows
// per CTA, 13.2 us now (two passes over 16.8 MB at
// the memory's rate: 5 us).
__global__ void __launch_bounds__(128)
k_kick_x4(const float* in, float* __restrict__ out,
          const int* shtab, const float* wtab,
          uint32_t n, int it, int rows)
{
    pdl_trigger();
    const int n4 = int(n / 4);
    const size_t nxy = size_t(n) * n;
    const float* src = in + blockIdx.z * nxy;
    float* dst = out + blockIdx.z * nxy;
    const int xa = blockIdx.x * rows;
    const int xe = min(int(n), xa + rows);
    const int g = blockIdx.y * blockDim.x + threadIdx.x;
    pdl_wait();
    if (g >= n4) {
        return;
    }
    KickStencil s[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int4 sh = reinterpret_cast<const int4*>(shtab
                                                      + size_t(j) * n)[g];
        const float4 wv = reinterpret_cast<const float4*>(wtab
                                                          + size_t(j) * n)[g];
        s[0].shift[j] = sh.x;
        s[1].shift[j] = sh.y;
        s[2].shift[j] = sh.z;
        s[3].shift[j] = sh.w;
        s[0].w[j] = wv.x;
        s[1].w[j] = wv.y;
        s[2].w[j] = wv.z;
        s[3].w[j] = wv.w;
    }
    // (the shifts of one stencil are consecutive)
    const bool same = s[1].shift[0] == s[0].shift[0]
                      && s[2].shift[0] == s[0].shift[0]
                      && s[3].shift[0] == s[0].shift[0];
    if (same) {
        auto load = [&](int x) {
            return x >= 0 && x < int(n)
                       ? reinterpret_cast<const float4*>(src
                                                         + size_t(x) * n)[g]
                       : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        // (4 output rows per turn: their 4 new tap rows read together)
        const int x0 = s[0].shift[0];
        float4 v[7];
#pragma unroll
        for (int j = 0; j < 3; j++) {
            v[j] = load(xa + x0 + j);
        }
        for (int xb = xa; xb < xe; xb += 4) {
#pragma unroll
            for (int u = 0; u < 4; u++) {
                v[3 + u] = load(xb + u < xe ? xb + u + x0 + 3 : -1);
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    if (j < it) {
                        o.x = fadd(o.x, fmul(v[u + j].x, s[0].w[j]));
                        o.y = fadd(o.y, fmul(v[u + j].y, s[1].w[j]));
                        o.z = fadd(o.z, fmul(v[u + j].z, s[2].w[j]));
                        o.w = fadd(o.w, fmul(v[u + j].w, s[3].w[j]));
                    }
                }
                if (xb + u < xe) {
                    reinterpret_cast<float4*>(dst + size_t(xb + u) * n)[g] =
                        o;
                }
            }
#pragma unroll
            for (int j = 0; j < 3; j++) {
                v[j] = v[4 + j];
            }
        }
        return;
    }
    for (int x = xa; x < xe; x++) {
        float o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < 4; c++) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int xs = x + s[c].shift[j];
                if (j < it && xs >= 0 && xs < int(n)) {
                    o[c] = fadd(o[c], fmul(src[size_t(xs) * n + 4 * g + c],
                                           s[c].w[j]));
                }
            }
        }
        reinterpret_cast<float4*>(dst + size_t(x) * n)[g] =
            make_float4(o[0], o[1], o[2], o[3]);
    }
}

// Fokker-Planck: each thread owns 4 columns of `rows` rows and reads them
// with the 4 columns on either side (16-byte words); a column's taps are ip
// neighbours from offset d on (-2 or -1), its weights tap-major [4][n]; a
// column without a stencil (d = 0) is column 0 times 0, which says nothing of
// its neighbours where those are not finite.
// (Gathering every tap through an index table from rows staged in shared
// memory: 15.3 us for 2048 x 2048, 8.4 us now.)
template <int U>
__global__ void __launch_bounds__(128)
k_fp4(const float* in, float* __restrict__ out,
      const int* __restrict__ d4, const float* __restrict__ w4, uint32_t n,
      int ip, int rows)
{
    pdl_trigger();
    const int n4 = int(n / 4);
    const int xa = blockIdx.x * rows;
    const int xe = min(int(n), xa + rows);
    const int g = blockIdx.y * blockDim.x + threadIdx.x;
    int4 d = make_int4(0, 0, 0, 0);
    float4 wv[4];
    if (g < n4) {   // (the tables were uploaded when the map was made)
        d = __ldg(reinterpret_cast<const int4*>(d4) + g);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            wv[j] = __ldg(reinterpret_cast<const float4*>(w4 + size_t(j) * n)
                          + g);
        }
    }
    pdl_wait();
    if (g >= n4) {
        return;
    }
    const bool far[4] = {d.x == -2, d.y == -2, d.z == -2, d.w == -2};
    const bool none[4] = {d.x == 0, d.y == 0, d.z == 0, d.w == 0};
    const bool edge = none[0] || none[1] || none[2] || none[3];
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    const size_t base = (blockIdx.z * size_t(n) + xa) * n4 + g;
    const float4* src = reinterpret_cast<const float4*>(in) + base;
    float4* dst = reinterpret_cast<float4*>(out) + base;
    // (U rows per turn, all read first)
    for (int xb = xa; xb < xe; xb += U) {
        float4 a[U], b[U], c[U];
        float first[U];   // column 0, of a thread with stencil-less columns
#pragma unroll
        for (int u = 0; u < U; u++) {
            const bool in_row = xb + u < xe;
            first[u] = in_row && edge ? src[u * n4 - g].x : 0.f;
            a[u] = in_row && g > 0 ? src[u * n4 - 1] : z;
            b[u] = in_row ? src[u * n4] : z;
            c[u] = in_row && g + 1 < n4 ? src[u * n4 + 1] : z;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            // columns 4g - 2 .. 4g + 6
            const float v[9] = {a[u].z, a[u].w, b[u].x, b[u].y, b[u].z,
                                b[u].w, c[u].x, c[u].y, c[u].z};
            float o[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                float value = 0.f;
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    if (j < ip) {
                        const float w = k == 0 ? wv[j].x : k == 1 ? wv[j].y
                                        : k == 2 ? wv[j].z : wv[j].w;
                        value = fadd(value, fmul(far[k] ? v[k + j]
                                                        : v[k + j + 1], w));
                    }
                }
                o[k] = none[k] ? fadd(0.f, fmul(first[u], 0.f)) : value;
            }
            if (xb + u < xe) {
                dst[u * n4] = make_float4(o[0], o[1], o[2], o[3]);
            }
        }
        src += U * n4;
        dst += U * n4;
    }
}

// DynamicRFKickMap::apply (src/SM/DynamicRFKickMap.cpp:79-109 and
// RFKickMap::_calcKick, src/SM/RFKickMap.cpp:59-83): the modulation of
// apply number `step` -- phase = syncphase + N(0,1) phasenoise + modampl
// sin(2 pi modtimeincrement step), amplitude = 1 + N(0,1) amplnoise, the
// normals drawn by Box-Muller from Philox(step, seed) -- and the RF kick
// offsets of every row with it (identical for every bunch).
__global__ void k_dynrf(DynRf d, uint64_t step, const float* __restrict__ q,
                        float xcenter, float dq, float dp, float pscale,
                        uint32_t n, uint32_t nb, float* __restrict__ offset,
                        float* __restrict__ log)
{
    pdl_trigger();
    pdl_wait();
    const uint32_t ctr[4] = {uint32_t(step), uint32_t(step >> 32), 0u, 0u};
    const uint32_t key[2] = {d.seed, 0x5EED0001u};
    uint32_t r[4];
    philox4x32_10(ctr, key, r);
    // uniforms in (0, 1]
    const float u1 = (float(r[0] >> 8) + 1.f) * (1.f / 16777216.f);
    const float u2 = (float(r[1] >> 8) + 1.f) * (1.f / 16777216.f);
    const float rad = sqrtf(-2.f * logf(u1));
    float sn, cs;
    sincospif(2.f * u2, &sn, &cs);
    const float n1 = rad * cs, n2 = rad * sn;
    const float mod = d.modampl
        * static_cast<float>(sin(d.modtimedelta * double(step)));
    const float phase = d.syncphase + n1 * d.phasenoise + mod;
    const float ampl = 1.f + n2 * d.amplnoise;
    if (blockIdx.x == 0 && threadIdx.x == 0 && log) {
        log[0] = phase;
        log[1] = ampl;
    }
    for (uint32_t x = blockIdx.x * blockDim.x + threadIdx.x; x < n;
         x += gridDim.x * blockDim.x) {
        float o;
        if (d.linear) {
            const float phaseoffs = d.syncphase - phase;
            const float ta = tanf(d.angle);
            o = __fmul_rn(ta, __fsub_rn(xcenter, float(x)));
            o = __fadd_rn(o, __fdiv_rn(__fdiv_rn(__fmul_rn(ta, phaseoffs),
                                                 d.bl2phase), dq));
            o = __fmul_rn(o, ampl);
        } else {
            const float arg = __fadd_rn(__fmul_rn(q[x], d.bl2phase), phase);
            const float v = __fadd_rn(__fmul_rn(-ampl * d.v_rf, sinf(arg)),
                                      d.v0);
            o = __fdiv_rn(__fdiv_rn(__fmul_rn(d.revolutionpart, v), dp),
                          pscale);
        }
        for (uint32_t b = 0; b < nb; b++) {
            offset[size_t(b) * n + x] = o;
        }
    }
}

}  // namespace

void launch_dynrf(vfps_map* m)
{
    const vfps_ps* in = m->in;
    const uint32_t n = in->n;
    float* log = m->dyn_step < m->dyn_cap ? m->dyn_log.p + 2 * m->dyn_step
                                          : nullptr;
    pdl_launch(k_dynrf, dim3((n + 127) / 128), dim3(128), 0, in->ctx->stream,
               m->dyn, m->dyn_step, m->axis_q.p, in->ax[0].zerobin,
               in->ax[0].delta, in->ax[1].delta, in->ax[1].scale, n, in->nb,
               m->offset.p, log);
    m->dyn_step++;
}

void launch_rotation(const vfps_map* m)
{
    const vfps_ps* in = m->in;
    const uint32_t n = in->n;
    // rows per thread: one, unless the meshes give more than 8 CTAs per SM
    // with it; at most 16
    const size_t ctas = size_t((n + 127) / 128) * n * in->nb;
    const int rows = int(std::max<size_t>(
        1, std::min<size_t>(16, ctas / (8 * size_t(in->ctx->sm_count)))));
    void (*kernel)(const float*, float*, uint32_t, const float*, const float*,
                   float, float, float, float, float, float, int) =
        m->it == 1 ? k_rotation<1, false>
        : m->it == 2 ? k_rotation<2, false>
        : m->it == 3 ? k_rotation<3, false>
        : m->clamp ? k_rotation<4, true> : k_rotation<4, false>;
    pdl_launch(kernel, dim3((n + 127) / 128, (n + rows - 1) / rows, in->nb),
               dim3(128), 0, in->ctx->stream, in->data.p, m->out->data.p, n,
               in->axisv[0].p, in->axisv[1].p, in->ax[0].delta,
               in->ax[1].delta, in->ax[0].zerobin, in->ax[1].zerobin, m->cs,
               m->sn, rows);
}

// the row-sweep forms: sides that are a multiple of 4, up to this size
// (shared memory of the y-kick's padded row: 32 KiB at most, within the
// default limit)
constexpr uint32_t PLAIN_V4_MAX = 4096;

bool plain_v4(uint32_t n)
{
    return n % 4 == 0 && n <= PLAIN_V4_MAX;
}

// rows per CTA of k_kick_x4 and k_fp4: one, unless the meshes give more
// than 4 CTAs per SM with one; at most 8
int plain_rows(const vfps_ps* in)
{
    const uint32_t n = in->n;
    const size_t per = size_t(n) * in->nb * ((n / 4 + 127) / 128)
                       / (4 * size_t(in->ctx->sm_count));
    return int(std::max<size_t>(1, std::min<size_t>(8, per)));
}

void launch_kick(const vfps_map* m, const float* offset)
{
    const vfps_ps* in = m->in;
    const uint32_t n = in->n;
    cudaStream_t st = in->ctx->stream;
    const bool v4 = plain_v4(n) && !m->cells;
    if (v4 && m->axis == VFPS_AXIS_Y) {
        const int t4 = int(std::min<uint32_t>(256,
                                              ((n / 4 + 31) / 32) * 32));
        const size_t smem = (2 * size_t(kick_pad(n)) + n) * sizeof(float);
        pdl_launch(k_kick_y4, dim3(in->nb * n), dim3(t4), smem, st,
                   in->data.p, m->out->data.p, offset, n, m->it);
    } else if (v4) {
        if (!m->xtab_valid) {
            m->xshift.alloc(size_t(4) * n);
            m->xweight.alloc(size_t(4) * n);
            pdl_launch(k_kick_table, dim3((n + 127) / 128), dim3(128), 0, st,
                       offset, n, m->it, m->xshift.p, m->xweight.p);
            m->xtab_valid = true;
        }
        const int rows = plain_rows(in);
        const int t4 = int(std::min<uint32_t>(128,
                                              ((n / 4 + 31) / 32) * 32));
        pdl_launch(k_kick_x4,
                   dim3((n + rows - 1) / rows, (n / 4 + t4 - 1) / t4, in->nb),
                   dim3(t4), 0, st, in->data.p, m->out->data.p, m->xshift.p,
                   m->xweight.p, n, m->it, rows);
    } else if (m->axis == VFPS_AXIS_Y) {
        const int threads = n >= 256 ? 256 : ((n + 31) / 32) * 32;
        pdl_launch(k_kick_y, dim3(in->nb * n), dim3(threads), 0, st,
                   in->data.p, m->out->data.p, offset, n, m->it);
    } else {
        pdl_launch(k_kick_x, dim3((n + 127) / 128, n, in->nb), dim3(128), 0,
                   st, in->data.p, m->out->data.p, offset, n, m->it);
    }
}

void launch_fp(const vfps_map* m)
{
    const vfps_ps* in = m->in;
    const uint32_t n = in->n;
    cudaStream_t st = in->ctx->stream;
    if (plain_v4(n) && !m->cells) {
        const int rows = plain_rows(in);
        const int t4 = int(std::min<uint32_t>(128,
                                              ((n / 4 + 31) / 32) * 32));
        pdl_launch(rows > 1 ? k_fp4<4> : k_fp4<1>,
                   dim3((n + rows - 1) / rows, (n / 4 + t4 - 1) / t4, in->nb),
                   dim3(t4), 0, st, in->data.p, m->out->data.p, m->fp_d4.p,
                   m->fp_w4.p, n, m->ip, rows);
        return;
    }
    pdl_launch(k_fp, dim3((n + 127) / 128, n, in->nb), dim3(128), 0, st,
               in->data.p, m->out->data.p, m->fp_idx.p, m->fp_w.p, n, m->ip);
}

}  // namespace vfps
