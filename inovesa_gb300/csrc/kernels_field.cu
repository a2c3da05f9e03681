// ElectricField kernels (src/PS/ElectricField.cpp:133-263).
//
// The reference computes the wake potential as c2r(Z * r2c(padded
// profile)) with unnormalised FFTW transforms, multiplying only the bins
// below nmax/2.  That is a circular convolution of the padded profile with
//   w[d] = Re Z_0 + 2 sum_{k=1}^{floor(nmax/2)-1} Re(Z_k e^{+2 pi i k d/nmax}),
// so the wake is the Toeplitz product  wake_b[x] = s sum_{b',m}
// proj_b'[m] w[(pos_b + x - pos_b' - m) mod nmax]  with s = wakescaling/nmax.
// w is built once per field in FP64; no FFT runs per step.
#include "vfps_internal.cuh"

namespace vfps {
namespace {

// w[d] in FP64 from the float impedance table, rounded to float at the end
__global__ void k_wake_table(const float* __restrict__ z, uint32_t nmax,
                             float* __restrict__ wtab)
{
    const uint32_t d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= nmax) {
        return;
    }
    double acc = double(z[0]);
    const uint32_t kmax = nmax / 2;  // bins k < nmax/2 are multiplied
    double part = 0;
    for (uint32_t k = 1; k < kmax; k++) {
        const uint64_t r = (uint64_t(k) * d) % nmax;
        double s, c;
        sincospi(2.0 * double(r) / double(nmax), &s, &c);
        part += double(z[2 * k]) * c - double(z[2 * k + 1]) * s;
    }
    acc += 2.0 * part;
    wtab[d] = static_cast<float>(acc);
}

constexpr int FW = 8;   // warps per CTA of the wake and CSR sums

// wake[b][x] = scale * sum_{b2,m} proj[b2][m] w[(pos_b - pos_b2 + x - m) mod nmax]:
// a CTA per 32 outputs x of bunch b (one per lane), its warps splitting
// the source cells m in chunks of 32 (chunk c to warp c mod FW).  Each
// chunk's FP32 partial is added in FP64, the warps' sums in a fixed order.
// The profile and the table's n + 31 entries that the outputs reach sit in
// shared memory (n = 2048: 16.2 us with the table read through L1 and its
// index wrapped per product, 8.3 us); TAB false: meshes whose table does
// not fit there
template <bool TAB>
__global__ void __launch_bounds__(FW * 32)
k_wake(const float* proj, const float* __restrict__ wtab,
       const uint32_t* __restrict__ pos, float* __restrict__ wake,
       uint32_t nb, uint32_t n, uint32_t nmax, float scale)
{
    extern __shared__ float sp[];
    float* sw = sp + n;   // sw[k] = w[(base + k) mod nmax]
    __shared__ double red[FW][32];
    dev::pdl_trigger();
    const uint32_t b = blockIdx.y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t x = blockIdx.x * 32 + lane;
    const long long nm = nmax;
    double acc = 0;
    for (uint32_t b2 = 0; b2 < nb; b2++) {
        // distance of output 32 blockIdx.x from source cell 0
        const long long at = (long long)pos[b] - (long long)pos[b2]
                             + blockIdx.x * 32ll;
        if (b2 > 0) {
            __syncthreads();
        }
        if (TAB) {
            long long k0 = (at - (long long)(n - 1)) % nm;
            k0 += k0 < 0 ? nm : 0;
            uint32_t k = static_cast<uint32_t>((k0 + threadIdx.x) % nm);
            const uint32_t step = (FW * 32) % nmax;
            for (uint32_t i = threadIdx.x; i < n + 31; i += FW * 32) {
                sw[i] = __ldg(wtab + k);
                k += step;
                k -= k >= nmax ? nmax : 0;
            }
        }
        if (b2 == 0) {
            dev::pdl_wait();   // the profiles (tables and positions stand)
        }
        for (uint32_t i = threadIdx.x; i < n; i += FW * 32) {
            sp[i] = proj[size_t(b2) * n + i];
        }
        __syncthreads();
        if (x < n) {
            for (uint32_t m0 = 32u * warp; m0 < n; m0 += 32u * FW) {
                const uint32_t me = min(n, m0 + 32u);
                float part = 0.f;
                if (TAB) {
                    const float* wv = sw + (n - 1) + lane;
                    if (me == m0 + 32u) {
#pragma unroll
                        for (uint32_t u = 0; u < 32; u++) {
                            part = fmaf(sp[m0 + u],
                                        wv[-int(m0) - int(u)], part);
                        }
                    } else {
                        for (uint32_t m = m0; m < me; m++) {
                            part = fmaf(sp[m], wv[-int(m)], part);
                        }
                    }
                } else {
                    const long long d0 = (at + lane - (long long)m0) % nm;
                    uint32_t d = static_cast<uint32_t>(d0 < 0 ? d0 + nm
                                                              : d0);
                    for (uint32_t m = m0; m < me; m++) {
                        part = fmaf(sp[m], __ldg(wtab + d), part);
                        d = (d == 0) ? nmax - 1 : d - 1;
                    }
                }
                acc += part;
            }
        }
    }
    red[warp][lane] = acc;
    __syncthreads();
    if (warp == 0 && x < n) {
        double sum = 0;
#pragma unroll
        for (int w = 0; w < FW; w++) {
            sum += red[w][lane];
        }
        wake[size_t(b) * n + x] = __fmul_rn(scale, static_cast<float>(sum));
    }
}

__global__ void k_pad(const float* __restrict__ proj,
                      const uint32_t* __restrict__ pos,
                      float* __restrict__ padded, uint32_t n)
{
    const uint32_t b = blockIdx.y;
    const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x < n) {
        padded[pos[b] + x] = proj[size_t(b) * n + x];
    }
}

// one lane per frequency bin k <= nmax/2 (32 bins per CTA) of bunch
// blockIdx.y: FF_k = sum_m p[m] e^{-2 pi i k m / nmax}, spectrum = coef_k
// |FF_k|^2.  The warps split the source cells in chunks of 32 (chunk c to
// warp c mod FW); a chunk is two runs of 16 cells, each the FP32 sum with
// the lane's own 16 factors e^{-2 pi i k u / nmax} (registers) times the
// factor of the run's first cell (the table), the chunks added in FP64.
// (The table read for every cell, 16 KiB of it staged per CTA, met up to
// 32-way bank conflicts: 8.1 us for n = 256, nmax = 2048 and 20.0 us for
// 2048, 8192, each with a memset before; 8.0 and 15.3 us now, without.)
// The CTAs' powers are added in order by the bunch's last CTA to finish.
__global__ void __launch_bounds__(FW * 32)
k_csr(const float* proj, const float2* __restrict__ tw,
      const float* __restrict__ coef, float* __restrict__ spectrum,
      double* __restrict__ part, unsigned* __restrict__ done,
      double* __restrict__ power, uint32_t n, uint32_t nmax, float fdelta)
{
    extern __shared__ float sp[];   // the profile, zeros up to 32 cells more
    __shared__ double red[2][FW][32];
    dev::pdl_trigger();
    const uint32_t b = blockIdx.y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t k = blockIdx.x * 32 + lane;
    const bool in = k <= nmax / 2;
    float2 f[16];
    {
        uint32_t idx = 0;
#pragma unroll
        for (int u = 0; u < 16; u++) {
            f[u] = in ? __ldg(tw + idx) : make_float2(0.f, 0.f);
            idx += k;
            idx -= in && idx >= nmax ? nmax : 0;
        }
    }
    const uint32_t n32 = (n + 31) & ~31u;
    dev::pdl_wait();
    for (uint32_t i = threadIdx.x; i < n32; i += blockDim.x) {
        sp[i] = i < n ? proj[size_t(b) * n + i] : 0.f;
    }
    __syncthreads();
    double re = 0, im = 0;
    if (in) {
        uint32_t idx = static_cast<uint32_t>((uint64_t(32u * warp) * k)
                                             % nmax);
        const uint32_t s16 = static_cast<uint32_t>((uint64_t(16) * k) % nmax);
        const uint32_t s32 = static_cast<uint32_t>(
            (uint64_t(32u * FW - 16u) * k) % nmax);
        for (uint32_t m0 = 32u * warp; m0 < n; m0 += 32u * FW) {
            float pre = 0.f, pim = 0.f;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const float2 t = __ldg(tw + idx);
                idx += h ? s32 : s16;
                idx -= idx >= nmax ? nmax : 0;
                float a = 0.f, c = 0.f;
                const float4* p4 = reinterpret_cast<const float4*>(
                    sp + m0 + 16 * h);
#pragma unroll
                for (int u = 0; u < 16; u += 4) {
                    const float4 q = p4[u / 4];
                    a = fmaf(q.x, f[u].x, a);
                    c = fmaf(q.x, f[u].y, c);
                    a = fmaf(q.y, f[u + 1].x, a);
                    c = fmaf(q.y, f[u + 1].y, c);
                    a = fmaf(q.z, f[u + 2].x, a);
                    c = fmaf(q.z, f[u + 2].y, c);
                    a = fmaf(q.w, f[u + 3].x, a);
                    c = fmaf(q.w, f[u + 3].y, c);
                }
                // (a - i c) (cos - i sin)
                pre = fmaf(a, t.x, pre);
                pre = fmaf(-c, t.y, pre);
                pim = fmaf(-a, t.y, pim);
                pim = fmaf(-c, t.x, pim);
            }
            re += pre;
            im += pim;
        }
    }
    red[0][warp][lane] = re;
    red[1][warp][lane] = im;
    __syncthreads();
    if (warp == 0) {
        double pw = 0;
        if (in) {
            double R = 0, I = 0;
#pragma unroll
            for (int w = 0; w < FW; w++) {
                R += red[0][w][lane];
                I += red[1][w][lane];
            }
            const float sv = __fmul_rn(coef[k], static_cast<float>(R * R
                                                                 + I * I));
            spectrum[size_t(b) * nmax + k] = sv;
            pw = double(fdelta) * double(sv);
        }
        pw = dev::warp_sum(pw);
        unsigned last = 0;
        if (lane == 0) {
            part[size_t(b) * gridDim.x + blockIdx.x] = pw;
            __threadfence();
            last = atomicAdd(done + b, 1u) == gridDim.x - 1;
        }
        last = __shfl_sync(0xffffffffu, last, 0);
        if (last) {
            __threadfence();
            double sum = 0;
            for (uint32_t i = lane; i < gridDim.x; i += 32) {
                sum += __ldcg(part + size_t(b) * gridDim.x + i);
            }
            sum = dev::warp_sum(sum);
            if (lane == 0) {
                power[b] = sum;
                done[b] = 0;   // for the next launch
            }
        }
    }
}

__global__ void k_twiddle(float2* tw, uint32_t nmax)
{
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < nmax) {
        double s, c;
        sincospi(2.0 * double(j) / double(nmax), &s, &c);
        tw[j] = make_float2(static_cast<float>(c), static_cast<float>(s));
    }
}

}  // namespace

void launch_wake_table(vfps_field* f)
{
    const uint32_t nmax = static_cast<uint32_t>(f->nmax);
    cudaStream_t st = f->ps->ctx->stream;
    k_wake_table<<<(nmax + 127) / 128, 128, 0, st>>>(f->z.p, nmax, f->wtab.p);
    VFPS_LAUNCHED();
    k_twiddle<<<(nmax + 127) / 128, 128, 0, st>>>(
        reinterpret_cast<float2*>(f->twiddle.p), nmax);
    VFPS_LAUNCHED();
}

void launch_wake_table_raw(vfps_ctx* ctx, const float* z, size_t nmax,
                           float* out)
{
    const uint32_t m = static_cast<uint32_t>(nmax);
    k_wake_table<<<(m + 127) / 128, 128, 0, ctx->stream>>>(z, m, out);
    VFPS_LAUNCHED();
}

void launch_wake(vfps_field* f)
{
    vfps_ps* ps = f->ps;
    const uint32_t n = ps->n;
    // profile and table within the default 48 KiB (with the static part)
    const size_t tab = (2 * size_t(n) + 31) * sizeof(float);
    const bool fits = tab <= 44 * 1024;
    pdl_launch(fits ? k_wake<true> : k_wake<false>,
               dim3((n + 31) / 32, ps->nb), dim3(FW * 32),
               fits ? tab : n * sizeof(float), ps->ctx->stream,
               ps->proj[0].p, f->wtab.p, f->d_pos.p, f->wake.p, ps->nb, n,
               static_cast<uint32_t>(f->nmax), f->wakescale);
}

void launch_pad(vfps_field* f)
{
    vfps_ps* ps = f->ps;
    VFPS_CUDA(cudaMemsetAsync(f->padded.p, 0, f->padded.bytes(),
                              ps->ctx->stream));
    dim3 grid((ps->n + 127) / 128, ps->nb);
    k_pad<<<grid, 128, 0, ps->ctx->stream>>>(ps->proj[0].p, f->d_pos.p,
                                             f->padded.p, ps->n);
    VFPS_LAUNCHED();
}

void launch_csr(vfps_field* f)
{
    vfps_ps* ps = f->ps;
    const uint32_t nmax = static_cast<uint32_t>(f->nmax);
    cudaStream_t st = ps->ctx->stream;
    const size_t smem = ((size_t(ps->n) + 31) & ~size_t(31)) * sizeof(float);
    pdl_launch(k_csr, dim3(csr_ctas(f->nmax), ps->nb), dim3(FW * 32), smem,
               st, ps->proj[0].p,
               reinterpret_cast<const float2*>(f->twiddle.p), f->csr_coef.p,
               f->spectrum.p, f->csr_part.p, f->csr_done.p, f->power.p,
               ps->n, nmax, f->freq_delta);
}

}  // namespace vfps
