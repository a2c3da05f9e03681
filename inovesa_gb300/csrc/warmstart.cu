// Learned warm start (no counterpart in the reference): a small network
// that proposes the equilibrium density of a bunch from its normalised
// current, gap ratio and damping time, trained on equilibria the solver
// itself produced.  Forward, backward and Adam kernels; every buffer is a
// device pointer owned by the caller (vfps_ws_net in vfps.h).
//
// Network (B samples, nin inputs, nh hidden units, nlat latent channels,
// npix output cells):
//   h1 = tanh(W1 x + b1)            W1 [nh][nin]
//   h2 = tanh(W2 h1 + b2)           W2 [nh][nh]
//   z  = W3 h2 + b3                 W3 [nlat][nh]
//   y  = bd + sum_k z_k Wd[k]       Wd [nlat][npix]: a transposed
//                                   convolution from a 1x1 latent map with
//                                   nlat channels to the full mesh
// Weights are read as BF16 (the Adam step keeps FP32 masters and writes
// the BF16 copies); all sums accumulate in FP32.  Loss: mean squared error
// against the target densities, L = sum (y - t)^2 / (B npix).
#include <algorithm>

#include <cuda_bf16.h>

#include "vfps_internal.cuh"

namespace {

constexpr int WS_THREADS = 256;
constexpr int WS_MLP_THREADS = 1024;   // of a sample's hidden layers
constexpr uint32_t WS_SLICES = 8;      // of a transposed layer's sums, most
constexpr size_t WS_SMEM = 227 * 1024; // shared memory of a CTA at most
constexpr uint32_t WS_LAT = 32;   // latent channels (nlat must equal it)

__device__ __forceinline__ float bf(const __nv_bfloat16* w, size_t i)
{
    return __bfloat162float(w[i]);
}

// rows of a layer, a warp each: f(j, sum_i W[j][i] a[i]) on lane 0, the
// weights read along the rows (coalesced), several rows in flight
template <typename F>
__device__ __forceinline__ void layer(const __nv_bfloat16* W, const float* a,
                                      uint32_t nout, uint32_t nin, F f)
{
    const uint32_t warps = blockDim.x >> 5, lane = threadIdx.x & 31;
#pragma unroll 4
    for (uint32_t j = threadIdx.x >> 5; j < nout; j += warps) {
        float s = 0.f;
        for (uint32_t i = lane; i < nin; i += 32) {
            s = fmaf(bf(W, size_t(j) * nin + i), a[i], s);
        }
        s = vfps::dev::warp_sum_f(s);
        if (lane == 0) {
            f(j, s);
        }
    }
}

// one CTA per sample: hidden layers and latent (18.0 us with a thread per
// unit reading its own weight row, 8.7 us with a warp per unit)
__global__ void k_ws_mlp_fwd(vfps_ws_net N, const float* __restrict__ x,
                             float* __restrict__ h1, float* __restrict__ h2,
                             float* __restrict__ z)
{
    const uint32_t b = blockIdx.x;
    extern __shared__ float ws_s[];
    float* xs = ws_s;                 // [nin]
    float* a1 = xs + N.nin;           // [nh]
    float* a2 = a1 + N.nh;            // [nh]
    const auto* W1 = static_cast<const __nv_bfloat16*>(N.w1);
    const auto* W2 = static_cast<const __nv_bfloat16*>(N.w2);
    const auto* W3 = static_cast<const __nv_bfloat16*>(N.w3);
    for (uint32_t i = threadIdx.x; i < N.nin; i += blockDim.x) {
        xs[i] = x[size_t(b) * N.nin + i];
    }
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < N.nh; j += blockDim.x) {
        float s = N.b1[j];
        for (uint32_t i = 0; i < N.nin; i++) {
            s = fmaf(bf(W1, size_t(j) * N.nin + i), xs[i], s);
        }
        a1[j] = tanhf(s);
        h1[size_t(b) * N.nh + j] = a1[j];
    }
    __syncthreads();
    layer(W2, a1, N.nh, N.nh, [&](uint32_t j, float s) {
        a2[j] = tanhf(s + N.b2[j]);
        h2[size_t(b) * N.nh + j] = a2[j];
    });
    __syncthreads();
    layer(W3, a2, N.nlat, N.nh, [&](uint32_t k, float s) {
        z[size_t(b) * N.nlat + k] = s + N.b3[k];
    });
}

// (64 samples of 256 x 256 pixels: 41.5 us with scalar reads of z, 30 us
// with 16-byte reads and the targets of 4 samples in flight; the
// multiply-adds alone take 4 us)
// y[b][p] = bd[p] + sum_k z[b][k] Wd[k][p]; with a target, also the loss
// gradient g = 2 (y - t) / (B npix) and per-CTA partial losses
__global__ void k_ws_decode(vfps_ws_net N, const float* __restrict__ z,
                            uint32_t B, const float* __restrict__ target,
                            float* __restrict__ y, float* __restrict__ g,
                            double* __restrict__ lpart)
{
    extern __shared__ float4 ws_s4[];
    float* zs = reinterpret_cast<float*>(ws_s4);      // [B][nlat]
    __shared__ double red[32];
    for (uint32_t i = threadIdx.x; i < B * N.nlat; i += blockDim.x) {
        zs[i] = z[i];
    }
    __syncthreads();
    const auto* Wd = static_cast<const __nv_bfloat16*>(N.wd);
    const float inv = 2.f / (float(B) * float(N.npix));
    double loss = 0;
    for (size_t p = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
         p < N.npix; p += size_t(gridDim.x) * blockDim.x) {
        float w[WS_LAT];
#pragma unroll
        for (uint32_t k = 0; k < WS_LAT; k++) {
            w[k] = bf(Wd, size_t(k) * N.npix + p);
        }
        const float bias = N.bd[p];
        // (the targets of 4 samples are on their way while their sums run)
        for (uint32_t b0 = 0; b0 < B; b0 += 4) {
            float t[4];
#pragma unroll
            for (uint32_t u = 0; u < 4; u++) {
                t[u] = target && b0 + u < B
                           ? target[size_t(b0 + u) * N.npix + p] : 0.f;
            }
#pragma unroll
            for (uint32_t u = 0; u < 4; u++) {
                const uint32_t b = b0 + u;
                if (b >= B) {
                    break;
                }
                float s = bias;
                const float4* zr = ws_s4 + b * (WS_LAT / 4);
#pragma unroll
                for (uint32_t k = 0; k < WS_LAT; k += 4) {
                    const float4 q = zr[k / 4];
                    s = fmaf(q.x, w[k], s);
                    s = fmaf(q.y, w[k + 1], s);
                    s = fmaf(q.z, w[k + 2], s);
                    s = fmaf(q.w, w[k + 3], s);
                }
                const size_t o = size_t(b) * N.npix + p;
                if (y) {
                    y[o] = s;
                }
                if (target) {
                    const float d = s - t[u];
                    g[o] = inv * d;
                    loss += double(d) * d;
                }
            }
        }
    }
    if (target) {
        loss = vfps::dev::block_sum(loss, red);
        if (threadIdx.x == 0) {
            lpart[blockIdx.x] = loss;
        }
    }
}

// Gradients of the decoder in one pass over g: dWd[k][p] = sum_b z[b][k]
// g[b][p], dbd[p] = sum_b g[b][p], and this CTA's part of dz[b][k] = sum_p
// Wd[k][p] g[b][p] (part[CTA][b][k]; k_ws_mlp_bwd adds the parts).
//
// A CTA takes tiles of WS_TILE pixels, g in chunks of WS_CHUNK samples in
// shared memory beside the tile's weights.  Thread = one pixel for dWd (32
// accumulators over the samples); for dz a chunk's 32 x 32 products are cut
// into 4 x 4 per thread (samples tb + 8 i, channels tk + 8 j: rows 260
// floats apart lie on 8 different groups of 4 banks) and the tile's pixels
// into 4 quarters, summed in FP32 over 32 pixels and in FP64 beyond.
// Every value of g and Wd is read from memory once; the form before, one
// CTA per (b, k), read g 32 times and Wd B times.  64 samples of 256 x 256
// pixels: 541 us for dz and 20 us for dWd before, 48 us together now; bound
// by shared-memory loads (8 16-byte loads per 64 multiply-adds of dz, 8 per
// 32 of dWd), with memory's floor at 5 us.
constexpr uint32_t WS_TILE = 256;
constexpr uint32_t WS_CHUNK = 32;
constexpr uint32_t WS_ROW = WS_TILE + 4;
constexpr uint32_t WS_MAX_CTAS = 304;   // two per SM

size_t bwd_smem(uint32_t B)
{
    return sizeof(float) * ((WS_LAT + WS_CHUNK) * WS_ROW
                            + size_t(B) * WS_LAT);
}

__global__ void __launch_bounds__(WS_TILE, 2)
k_ws_decode_bwd(vfps_ws_net N, vfps_ws_net G, const float* __restrict__ z,
                const float* __restrict__ g, uint32_t B,
                double* __restrict__ part)
{
    extern __shared__ float4 ws_s4[];
    float* wt = reinterpret_cast<float*>(ws_s4);   // [WS_LAT][WS_ROW]
    float* gt = wt + WS_LAT * WS_ROW;              // [WS_CHUNK][WS_ROW]
    float* zs = gt + WS_CHUNK * WS_ROW;            // [B][WS_LAT]
    for (uint32_t i = threadIdx.x; i < B * WS_LAT; i += WS_TILE) {
        zs[i] = z[i];
    }
    const auto* Wd = static_cast<const __nv_bfloat16*>(N.wd);
    float* dWd = const_cast<float*>(static_cast<const float*>(G.wd));
    float* dbd = const_cast<float*>(G.bd);
    double* mine = part + size_t(blockIdx.x) * B * WS_LAT;
    const uint32_t tid = threadIdx.x;
    const uint32_t quarter = tid >> 6, tb = (tid >> 3) & 7, tk = tid & 7;
    bool first = true;
    for (uint32_t p0 = blockIdx.x * WS_TILE; p0 < N.npix;
         p0 += gridDim.x * WS_TILE) {
        const uint32_t p = p0 + tid;
        const bool in = p < N.npix;
        __syncthreads();   // the last tile's weights are read
#pragma unroll 8
        for (uint32_t k = 0; k < WS_LAT; k++) {
            wt[k * WS_ROW + tid] = in ? bf(Wd, size_t(k) * N.npix + p) : 0.f;
        }
        float acc[WS_LAT];
#pragma unroll
        for (uint32_t k = 0; k < WS_LAT; k++) {
            acc[k] = 0.f;
        }
        float sb = 0.f;
        for (uint32_t b0 = 0; b0 < B; b0 += WS_CHUNK) {
            const uint32_t nb = min(B - b0, WS_CHUNK);
            __syncthreads();   // the last chunk is read
#pragma unroll 8
            for (uint32_t b = 0; b < WS_CHUNK; b++) {
                gt[b * WS_ROW + tid] =
                    in && b < nb ? g[size_t(b0 + b) * N.npix + p] : 0.f;
            }
            __syncthreads();
#pragma unroll 2
            for (uint32_t b = 0; b < nb; b++) {
                const float gv = gt[b * WS_ROW + tid];
                sb += gv;
                const float4* zr = reinterpret_cast<const float4*>(
                    zs + (b0 + b) * WS_LAT);
#pragma unroll
                for (uint32_t k = 0; k < WS_LAT; k += 4) {
                    const float4 q = zr[k / 4];
                    acc[k] = fmaf(q.x, gv, acc[k]);
                    acc[k + 1] = fmaf(q.y, gv, acc[k + 1]);
                    acc[k + 2] = fmaf(q.z, gv, acc[k + 2]);
                    acc[k + 3] = fmaf(q.w, gv, acc[k + 3]);
                }
            }
            float s0[4][4], s[4][4] = {};   // over 32 pixels each
#pragma unroll 1
            for (uint32_t h = 0; h < 2; h++) {
#pragma unroll
                for (int i = 0; i < 4; i++) {
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        s0[i][j] = s[i][j];
                        s[i][j] = 0.f;
                    }
                }
                const uint32_t at = quarter * 64 + h * 32;
#pragma unroll 2
                for (uint32_t c = 0; c < 32; c += 4) {
                    float4 gv[4], wv[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        gv[i] = *reinterpret_cast<const float4*>(
                            gt + (tb + 8 * i) * WS_ROW + at + c);
                        wv[i] = *reinterpret_cast<const float4*>(
                            wt + (tk + 8 * i) * WS_ROW + at + c);
                    }
#pragma unroll
                    for (int i = 0; i < 4; i++) {
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            s[i][j] = fmaf(wv[j].x, gv[i].x, s[i][j]);
                            s[i][j] = fmaf(wv[j].y, gv[i].y, s[i][j]);
                            s[i][j] = fmaf(wv[j].z, gv[i].z, s[i][j]);
                            s[i][j] = fmaf(wv[j].w, gv[i].w, s[i][j]);
                        }
                    }
                }
            }
            __syncthreads();   // the chunk is read: its place takes the sums
            float2* q = reinterpret_cast<float2*>(gt);   // [4][32 * 32]
#pragma unroll
            for (int i = 0; i < 4; i++) {
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    q[quarter * 1024 + (tb + 8 * i) * 32 + tk + 8 * j] =
                        make_float2(s0[i][j], s[i][j]);
                }
            }
            __syncthreads();
            for (uint32_t i = tid; i < nb * WS_LAT; i += WS_TILE) {
                double* m = mine + b0 * WS_LAT + i;
                double v = first ? 0. : *m;
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    v += double(q[u * 1024 + i].x);
                    v += double(q[u * 1024 + i].y);
                }
                *m = v;
            }
        }
        if (in) {
#pragma unroll
            for (uint32_t k = 0; k < WS_LAT; k++) {
                dWd[size_t(k) * N.npix + p] = acc[k];
            }
            dbd[p] = sb;
        }
        first = false;
    }
}

// back through the MLP, one CTA per sample (a chain of short sums, bound by
// latency: 15.4 us with 256 threads and one thread per sum, 12 us with 1024
// and the sums sliced, the parts of dz added as well): dz from its parts, then
// the per-sample deltas
//   d3 = dz, d2 = (W3^T d3) (1 - h2^2), d1 = (W2^T d2) (1 - h1^2),
// the sums cut into `slices` slices
constexpr size_t WS_BWD_FLOATS = 2 * (WS_MLP_THREADS / 32) * WS_LAT + WS_LAT;

// as many slices as fit beside the parts of dz and the units' deltas
// (layers of up to 6200 units: all eight)
uint32_t mlp_bwd_slices(uint32_t nh)
{
    const size_t rows = (WS_SMEM / sizeof(float) - WS_BWD_FLOATS) / nh;
    return uint32_t(std::min<size_t>(WS_SLICES, rows > 1 ? rows - 1 : 0));
}

size_t mlp_bwd_smem(uint32_t nh, uint32_t slices)
{
    return sizeof(float) * (WS_BWD_FLOATS + size_t(1 + slices) * nh);
}

__global__ void k_ws_mlp_bwd(vfps_ws_net N, const double* __restrict__ part,
                             uint32_t parts, uint32_t slices,
                             const float* __restrict__ h1,
                             const float* __restrict__ h2,
                             float* __restrict__ dz, float* __restrict__ d1,
                             float* __restrict__ d2)
{
    const uint32_t b = blockIdx.x, B = gridDim.x;
    extern __shared__ double ws_sd[];
    float* ws_s = reinterpret_cast<float*>(ws_sd);
    constexpr uint32_t NW = WS_MLP_THREADS / 32;
    double* red = ws_sd;                             // [NW][WS_LAT]
    float* s3 = ws_s + 2 * NW * WS_LAT;              // [nlat]
    float* s2 = s3 + N.nlat;                         // [nh]
    float* sl = s2 + N.nh;                           // [slices][nh]
    const auto* W2 = static_cast<const __nv_bfloat16*>(N.w2);
    const auto* W3 = static_cast<const __nv_bfloat16*>(N.w3);
    {
        const uint32_t k = threadIdx.x & 31, u = threadIdx.x >> 5;
        double s = 0;
#pragma unroll 8
        for (uint32_t c = u; c < parts; c += NW) {
            s += part[(size_t(c) * B + b) * WS_LAT + k];
        }
        red[u * WS_LAT + k] = s;
    }
    __syncthreads();
    if (threadIdx.x < WS_LAT) {
        double s = 0;
#pragma unroll
        for (uint32_t u = 0; u < NW; u++) {
            s += red[u * WS_LAT + threadIdx.x];
        }
        s3[threadIdx.x] = float(s);
        dz[size_t(b) * WS_LAT + threadIdx.x] = float(s);
    }
    __syncthreads();
    // out[i] = (sum_j W[j][i] a[j]) (1 - h[i]^2)
    auto back = [&](const __nv_bfloat16* W, const float* a, uint32_t nj,
                    const float* h, auto out) {
        const uint32_t per = (nj + slices - 1) / slices;
        for (uint32_t t = threadIdx.x; t < N.nh * slices;
             t += WS_MLP_THREADS) {
            const uint32_t i = t % N.nh, j0 = t / N.nh * per;
            float s = 0.f;
#pragma unroll 8
            for (uint32_t j = j0; j < min(nj, j0 + per); j++) {
                s = fmaf(bf(W, size_t(j) * N.nh + i), a[j], s);
            }
            sl[t] = s;
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < N.nh; i += WS_MLP_THREADS) {
            float s = 0.f;
            for (uint32_t u = 0; u < slices; u++) {
                s += sl[u * N.nh + i];
            }
            const float v = h[size_t(b) * N.nh + i];
            out(i, s * (1.f - v * v));
        }
        __syncthreads();
    };
    back(W3, s3, N.nlat, h2, [&](uint32_t i, float v) {
        s2[i] = v;
        d2[size_t(b) * N.nh + i] = v;
    });
    back(W2, s2, N.nh, h1,
         [&](uint32_t i, float v) { d1[size_t(b) * N.nh + i] = v; });
}

// dW[j][i] = sum_b d[b][j] a[b][i], db[j] = sum_b d[b][j] of the three MLP
// layers, one thread per weight (the layers are small: one launch of 9.9 us
// for three of 8.5, 8.7 and 6.6 us)
struct WsOuter {
    const float *d, *a;
    float *dW, *db;
    uint32_t nout, nin, first;   // first: its first thread
};

struct WsOuter3 {
    WsOuter l[3];
};

__global__ void k_ws_outer(const __grid_constant__ WsOuter3 A, uint32_t B)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const WsOuter& L = A.l[t >= A.l[2].first ? 2 : t >= A.l[1].first ? 1 : 0];
    const uint32_t i0 = t - L.first, nw = L.nout * L.nin;
    if (i0 < nw) {
        const uint32_t j = i0 / L.nin, i = i0 % L.nin;
        float s = 0.f;
#pragma unroll 8
        for (uint32_t b = 0; b < B; b++) {
            s = fmaf(L.d[size_t(b) * L.nout + j], L.a[size_t(b) * L.nin + i],
                     s);
        }
        L.dW[i0] = s;
    } else if (i0 < nw + L.nout) {
        const uint32_t j = i0 - nw;
        float s = 0.f;
#pragma unroll 8
        for (uint32_t b = 0; b < B; b++) {
            s += L.d[size_t(b) * L.nout + j];
        }
        L.db[j] = s;
    }
}

// Adam (Kingma & Ba 2015) on FP32 masters; writes the BF16 copies, all
// tensors of a network in one launch (12.8 us for 2.2 million parameters, the
// time of the largest alone; eight launches took 36 us).  Bound by memory.
struct WsAdam {
    float* w;
    const float* g;
    float *m, *v;
    __nv_bfloat16* w16;
    size_t count;
    uint32_t first;   // its first CTA
};
constexpr uint32_t WS_ADAM_MAX = 8;   // tensors of one launch
struct WsAdamList {
    WsAdam t[WS_ADAM_MAX];
    uint32_t n;
};
constexpr uint32_t WS_ADAM_CTA = 4 * WS_THREADS;   // elements of a CTA

__global__ void k_ws_adam(const __grid_constant__ WsAdamList L, float lr,
                          float b1, float b2, float eps, float c1, float c2)
{
    uint32_t k = 0;
    while (k + 1 < L.n && blockIdx.x >= L.t[k + 1].first) {
        k++;
    }
    const WsAdam& t = L.t[k];
    const size_t i0 = size_t(blockIdx.x - t.first) * WS_ADAM_CTA
                      + threadIdx.x;
    // (4 strided elements per thread, all loads first)
    float gi[4], mi[4], vi[4], wi[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const size_t i = i0 + u * WS_THREADS;
        if (i < t.count) {
            gi[u] = t.g[i];
            mi[u] = t.m[i];
            vi[u] = t.v[i];
            wi[u] = t.w[i];
        }
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const size_t i = i0 + u * WS_THREADS;
        if (i < t.count) {
            const float m = b1 * mi[u] + (1.f - b1) * gi[u];
            const float v = b2 * vi[u] + (1.f - b2) * gi[u] * gi[u];
            t.m[i] = m;
            t.v[i] = v;
            const float w = wi[u] - lr * (m / c1) / (sqrtf(v / c2) + eps);
            t.w[i] = w;
            if (t.w16) {
                t.w16[i] = __float2bfloat16_rn(w);
            }
        }
    }
}

// Scratch of the context for the CTAs' parts of dz.  A larger one takes its
// place; the old one stays until the context goes, as a captured graph may
// hold it.  The sizes are powers of two, so the old ones are together no
// larger than the newest: 64 MB in all at the largest call's (304 CTAs, 384
// samples).  Allocated in relaxed capture mode, so that a call under stream
// capture may be the first.
cudaError_t dz_scratch(vfps_ctx* ctx, size_t count, double** out)
{
    if (ctx->ws_part.empty() || ctx->ws_part.back().n < count) {
        size_t n = size_t(1) << 17;   // 1 MB
        while (n < count) {
            n *= 2;
        }
        try {
            ctx->ws_part.reserve(ctx->ws_part.size() + 1);
        } catch (const std::bad_alloc&) {
            return cudaErrorMemoryAllocation;
        }
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&mode);
        double* p = nullptr;
        const cudaError_t e = cudaMalloc(&p, n * sizeof(double));
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (e != cudaSuccess) {
            return e;
        }
        vfps::DevBuf<double> buf;
        buf.p = p;
        buf.n = n;
        ctx->ws_part.push_back(std::move(buf));
    }
    *out = ctx->ws_part.back().p;
    return cudaSuccess;
}

int ws_check(const vfps_ws_net* n)
{
    if (!n || n->nin == 0 || n->nh == 0 || n->nlat != WS_LAT
        || n->npix == 0 || !n->w1 || !n->b1 || !n->w2 || !n->b2 || !n->w3
        || !n->b3 || !n->wd || !n->bd) {
        return VFPS_ERR_INVALID_ARGUMENT;
    }
    return VFPS_OK;
}

int launched(vfps_ctx* ctx)
{
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        ctx->last_error = cudaGetErrorString(e);
        return VFPS_ERR_CUDA;
    }
    return VFPS_OK;
}

}  // namespace

extern "C" int vfps_ws_forward(vfps_ctx* ctx, const vfps_ws_net* net,
                               const float* x, uint32_t B, float* h1,
                               float* h2, float* z, float* y,
                               const float* target, float* g, double* lpart,
                               uint32_t nparts)
{
    if (!ctx || ws_check(net) || !x || !h1 || !h2 || !z || B == 0
        || (target && (!g || !lpart || nparts == 0))) {
        return VFPS_ERR_INVALID_ARGUMENT;
    }
    if (cudaSetDevice(ctx->device) != cudaSuccess) {
        return VFPS_ERR_CUDA;
    }
    const vfps_ws_net N = *net;
    const size_t s1 = sizeof(float) * (N.nin + 2 * N.nh);
    k_ws_mlp_fwd<<<B, WS_MLP_THREADS, s1, ctx->stream>>>(N, x, h1, h2, z);
    int rc = launched(ctx);
    if (rc) {
        return rc;
    }
    const size_t s2 = sizeof(float) * size_t(B) * N.nlat;
    const uint32_t grid = target ? nparts
        : uint32_t((N.npix + WS_THREADS - 1) / WS_THREADS);
    k_ws_decode<<<grid, WS_THREADS, s2, ctx->stream>>>(N, z, B, target, y, g,
                                                      lpart);
    return launched(ctx);
}

extern "C" int vfps_ws_backward(vfps_ctx* ctx, const vfps_ws_net* net,
                                const vfps_ws_net* grad, const float* x,
                                uint32_t B, const float* h1, const float* h2,
                                const float* z, const float* g, float* dz,
                                float* d1, float* d2)
{
    if (!ctx || ws_check(net) || ws_check(grad) || !x || !h1 || !h2 || !z
        || !g || !dz || !d1 || !d2 || B == 0) {
        return VFPS_ERR_INVALID_ARGUMENT;
    }
    if (cudaSetDevice(ctx->device) != cudaSuccess) {
        return VFPS_ERR_CUDA;
    }
    const vfps_ws_net N = *net, G = *grad;
    cudaStream_t st = ctx->stream;
    // the limits on the samples (the forward pass's) and on the hidden units,
    // before the first launch writes into the caller's gradients
    const uint32_t slices = mlp_bwd_slices(N.nh);
    if (size_t(B) * N.nlat * sizeof(float) > 48 * 1024
        || (size_t(N.nlat) + N.nh) * sizeof(float) > 48 * 1024) {
        ctx->last_error = cudaGetErrorString(cudaErrorInvalidValue);
        return VFPS_ERR_CUDA;
    }
    const size_t sz = bwd_smem(B);
    const uint32_t ctas = uint32_t(std::min<size_t>(
        WS_MAX_CTAS, (size_t(N.npix) + WS_TILE - 1) / WS_TILE));
    double* part = nullptr;
    cudaError_t e = vfps::allow_smem(k_ws_decode_bwd);
    if (e == cudaSuccess) {
        e = vfps::allow_smem(k_ws_mlp_bwd);
    }
    if (e == cudaSuccess) {
        e = dz_scratch(ctx, size_t(ctas) * B * WS_LAT, &part);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        ctx->last_error = cudaGetErrorString(e);
        return e == cudaErrorMemoryAllocation ? VFPS_ERR_OUT_OF_MEMORY
                                              : VFPS_ERR_CUDA;
    }
    k_ws_decode_bwd<<<ctas, WS_TILE, sz, st>>>(N, G, z, g, B, part);
    int rc = launched(ctx);
    if (rc) {
        return rc;
    }
    k_ws_mlp_bwd<<<B, WS_MLP_THREADS, mlp_bwd_smem(N.nh, slices), st>>>(
        N, part, ctas, slices, h1, h2, dz, d1, d2);
    rc = launched(ctx);
    if (rc) {
        return rc;
    }
    auto mut = [](const void* p) {
        return const_cast<float*>(static_cast<const float*>(p));
    };
    WsOuter3 L = {{
        {dz, h2, mut(G.w3), mut(G.b3), N.nlat, N.nh, 0},
        {d2, h1, mut(G.w2), mut(G.b2), N.nh, N.nh, 0},
        {d1, x, mut(G.w1), mut(G.b1), N.nh, N.nin, 0},
    }};
    uint32_t tot = 0;
    for (auto& o : L.l) {
        o.first = tot;
        tot += o.nout * o.nin + o.nout;
    }
    k_ws_outer<<<(tot + 127) / 128, 128, 0, st>>>(L, B);
    return launched(ctx);
}

namespace {

int adam(vfps_ctx* ctx, WsAdamList& L, float lr, float beta1, float beta2,
         float eps, uint32_t step)
{
    if (cudaSetDevice(ctx->device) != cudaSuccess) {
        return VFPS_ERR_CUDA;
    }
    const float c1 = 1.f - powf(beta1, float(step));
    const float c2 = 1.f - powf(beta2, float(step));
    size_t ctas = 0;
    for (uint32_t k = 0; k < L.n; k++) {
        L.t[k].first = uint32_t(ctas);
        ctas += (L.t[k].count + WS_ADAM_CTA - 1) / WS_ADAM_CTA;
    }
    if (ctas > 0x7fffffffu) {
        ctx->last_error = "too many parameters";
        return VFPS_ERR_INVALID_ARGUMENT;
    }
    k_ws_adam<<<unsigned(ctas), WS_THREADS, 0, ctx->stream>>>(
        L, lr, beta1, beta2, eps, c1, c2);
    return launched(ctx);
}

}  // namespace

extern "C" int vfps_ws_adam(vfps_ctx* ctx, float* w, const float* g,
                            float* m, float* v, void* w_bf16, size_t count,
                            float lr, float beta1, float beta2, float eps,
                            uint32_t step)
{
    if (!ctx || !w || !g || !m || !v || count == 0 || step == 0) {
        return VFPS_ERR_INVALID_ARGUMENT;
    }
    WsAdamList L{};
    L.n = 1;
    L.t[0] = {w, g, m, v, static_cast<__nv_bfloat16*>(w_bf16), count, 0};
    return adam(ctx, L, lr, beta1, beta2, eps, step);
}

extern "C" int vfps_ws_adam_list(vfps_ctx* ctx, uint32_t n,
                                 const vfps_ws_param* p, float lr,
                                 float beta1, float beta2, float eps,
                                 uint32_t step)
{
    if (!ctx || !p || n == 0 || n > WS_ADAM_MAX || step == 0) {
        return VFPS_ERR_INVALID_ARGUMENT;
    }
    WsAdamList L{};
    L.n = n;
    for (uint32_t k = 0; k < n; k++) {
        if (!p[k].w || !p[k].g || !p[k].m || !p[k].v || p[k].count == 0) {
            return VFPS_ERR_INVALID_ARGUMENT;
        }
        L.t[k] = {p[k].w, p[k].g, p[k].m, p[k].v,
                  static_cast<__nv_bfloat16*>(p[k].w_bf16),
                  size_t(p[k].count), 0};
    }
    return adam(ctx, L, lr, beta1, beta2, eps, step);
}
