// PhaseSpace kernels: Gaussian start, x/y projections, integral,
// normalisation and moments (src/PS/PhaseSpace.cpp:200-372,457-501).
// Sums feeding the wake and the charge integral accumulate in FP64; the
// per-lane partial sums of at most 8 cells stay in FP32 so that the FP64
// pipe (slow on GB300) sees n/256 additions per row.
#include "vfps_internal.cuh"

namespace vfps {
namespace {

__global__ void k_fill_gaussian(float* __restrict__ data,
                                const float* __restrict__ gx,
                                const float* __restrict__ gy, uint32_t nb,
                                uint32_t n)
{
    const size_t nxy = size_t(n) * n;
    const size_t total = nxy * nb;
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < total;
         i += size_t(gridDim.x) * blockDim.x) {
        const size_t c = i % nxy;
        data[i] = __fmul_rn(gx[c / n], gy[c % n]);
    }
}

// one warp per row: proj[row] = sum_y data[row][y] ws[y], 8 cells per lane
// (32 apart, all read first) in FP32, then FP64 (the order of
// vfps_charge_noalloc)
__global__ void k_project_x(const float* data,
                            const float* __restrict__ ws,
                            float* __restrict__ proj,
                            double* __restrict__ proj64, uint32_t rows,
                            uint32_t n)
{
    dev::pdl_trigger();
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    dev::pdl_wait();
    if (warp >= rows) {
        return;
    }
    const float* r = data + size_t(warp) * n;
    double acc = 0;
#pragma unroll 2
    for (uint32_t y0 = lane; y0 < n; y0 += 256) {
        float v[8], w[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const uint32_t y = y0 + 32 * u;
            v[u] = y < n ? r[y] : 0.f;
            w[u] = y < n ? __ldg(ws + y) : 0.f;
        }
        float part = 0;
#pragma unroll
        for (int u = 0; u < 8; u++) {
            part = fmaf(v[u], w[u], part);
        }
        acc += part;
    }
    acc = dev::warp_sum(acc);
    if (lane == 0) {
        proj[warp] = static_cast<float>(acc);
        if (proj64) {
            proj64[warp] = acc;
        }
    }
}

// proj[b][y] = sum_x data[b][x][y] ws[x]: a CTA per 32 columns of a bunch
// and slice of `rows` rows, its 32 warps taking rows 32 apart (8 rows in
// FP32, then FP64); the slices' sums are added in order by the last CTA of
// the columns.  (A thread per column, every row in sequence: 33 us for 256
// rows and 260 us for 2048; now 6.1 and 12.6 us, 31 us with one slice.)
__global__ void __launch_bounds__(1024)
k_project_y(const float* data, const float* __restrict__ ws,
            float* __restrict__ proj, double* __restrict__ part,
            unsigned* __restrict__ done, uint32_t n, uint32_t rows)
{
    __shared__ double red[32][33];
    __shared__ bool last;
    dev::pdl_trigger();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t y = blockIdx.x * 32 + lane;
    const uint32_t b = blockIdx.y, slices = gridDim.z;
    const uint32_t xa = blockIdx.z * rows, xe = min(n, xa + rows);
    dev::pdl_wait();
    double acc = 0;
    if (y < n) {
        const float* d = data + size_t(b) * n * n + y;
        for (uint32_t x0 = xa + warp; x0 < xe; x0 += 32 * 8) {
            float v[8], w[8];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const uint32_t x = x0 + 32 * u;
                v[u] = x < xe ? d[size_t(x) * n] : 0.f;
                w[u] = x < xe ? __ldg(ws + x) : 0.f;
            }
            float p = 0;
#pragma unroll
            for (int u = 0; u < 8; u++) {
                p = fmaf(v[u], w[u], p);
            }
            acc += p;
        }
    }
    red[warp][lane] = acc;
    __syncthreads();
    // column `warp` of the CTA: the warps' sums, one per lane
    acc = dev::warp_sum(red[lane][warp]);
    const uint32_t yw = blockIdx.x * 32 + warp;
    if (slices > 1) {
        const size_t at = size_t(b) * n + yw;
        if (lane == 0 && yw < n) {
            part[blockIdx.z * (size_t(gridDim.y) * n) + at] = acc;
            __threadfence();
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned* c = done + b * gridDim.x + blockIdx.x;
            last = atomicAdd(c, 1u) == slices - 1;
            if (last) {
                *c = 0;   // for the next launch
            }
        }
        __syncthreads();
        if (!last || lane != 0 || yw >= n) {
            return;
        }
        __threadfence();
        acc = 0;
        for (uint32_t z = 0; z < slices; z++) {
            acc += __ldcg(part + z * (size_t(gridDim.y) * n) + at);
        }
    }
    if (lane == 0 && yw < n) {
        proj[size_t(b) * n + yw] = static_cast<float>(acc);
    }
}

// single block: filling[b] = sum_x proj64[b][x] ws[x]; filling[nb] = total.
// Several bunches at a time, `wpb` warps each
__global__ void k_integrate(const double* proj64,
                            const float* __restrict__ ws,
                            const float* __restrict__ fillset,
                            double* __restrict__ filling, uint32_t nb,
                            uint32_t n, uint32_t wpb, int* status)
{
    __shared__ double red[8];
    dev::pdl_trigger();
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t at_once = 8 / wpb;
    dev::pdl_wait();
    double total = 0;
    for (uint32_t b0 = 0; b0 < nb; b0 += at_once) {
        const uint32_t b = b0 + warp / wpb;
        double acc = 0;
        if (b < nb) {
            const double* p = proj64 + size_t(b) * n;
#pragma unroll 4
            for (uint32_t x = (warp % wpb) * 32 + lane; x < n;
                 x += 32 * wpb) {
                acc += p[x] * double(__ldg(ws + x));
            }
        }
        acc = dev::warp_sum(acc);
        if (lane == 0) {
            red[warp] = acc;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (uint32_t u = 0; u < at_once && b0 + u < nb; u++) {
                double f = 0;
                for (uint32_t w = 0; w < wpb; w++) {
                    f += red[u * wpb + w];
                }
                filling[b0 + u] = f;
                total += f;
                // watchdog: a populated bunch must keep a finite, positive
                // charge
                if (fillset[b0 + u] > 0 && !(f > 0) && status) {
                    atomicCAS(status, 0, VFPS_ERR_NUMERIC);
                }
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        filling[nb] = total;
    }
}

__global__ void k_normalize(float* __restrict__ data,
                            const float* __restrict__ fillset,
                            const double* filling, uint32_t nb, size_t nxy)
{
    dev::pdl_trigger();
    const size_t total = nxy * nb;
    dev::pdl_wait();
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < total;
         i += size_t(gridDim.x) * blockDim.x) {
        const uint32_t b = static_cast<uint32_t>(i / nxy);
        const float fs = fillset[b];
        data[i] = fs > 0 ? data[i] * static_cast<float>(double(fs) / filling[b])
                         : 0.f;
    }
}

// one block per bunch: average, variance, rms of one axis
__global__ void k_moments(const float* proj,
                          const float* __restrict__ axisv,
                          const float* __restrict__ fillset,
                          const double* filling, float delta,
                          uint32_t nb, uint32_t n, float* __restrict__ mom)
{
    __shared__ double scratch[32];
    __shared__ double avg_s;
    dev::pdl_trigger();
    const uint32_t b = blockIdx.x;
    const bool pop = fillset[b] > 0;
    dev::pdl_wait();
    double a = 0;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        a += double(proj[size_t(b) * n + i]) * double(axisv[i]);
    }
    a = dev::block_sum(a, scratch);
    if (threadIdx.x == 0) {
        avg_s = pop ? a * double(delta) / filling[b] : 0.0;
    }
    __syncthreads();
    const double avg = avg_s;
    double v = 0;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        const double d = double(axisv[i]) - avg;
        v += double(proj[size_t(b) * n + i]) * d * d;
    }
    v = dev::block_sum(v, scratch);
    if (threadIdx.x == 0) {
        const double var = pop ? v * double(delta) / filling[b] : 0.0;
        mom[0 * nb + b] = static_cast<float>(avg);
        mom[1 * nb + b] = static_cast<float>(var);
        mom[2 * nb + b] = static_cast<float>(sqrt(var));
    }
}

int grid_for(size_t total, int threads)
{
    const size_t blocks = (total + threads - 1) / threads;
    return static_cast<int>(blocks < 65535 * 16 ? blocks : 65535 * 16);
}

}  // namespace

void launch_fill_gaussian(vfps_ps* ps, const float* gx, const float* gy)
{
    const size_t total = size_t(ps->nb) * ps->n * ps->n;
    k_fill_gaussian<<<grid_for(total, 256), 256, 0, ps->ctx->stream>>>(
        ps->data.p, gx, gy, ps->nb, ps->n);
    VFPS_LAUNCHED();
}

void launch_project_x(vfps_ps* ps, const float* data)
{
    const uint32_t rows = ps->nb * ps->n;
    const int threads = 256;
    const int blocks = (rows * 32 + threads - 1) / threads;
    pdl_launch(k_project_x, dim3(blocks), dim3(threads), 0, ps->ctx->stream,
               data ? data : ps->data.p, ps->ws.p, ps->proj[0].p,
               ps->proj64.p, rows, ps->n);
}

void launch_project_y(vfps_ps* ps)
{
    const uint32_t slices = project_y_slices(ps->ctx, ps->nb, ps->n);
    const uint32_t rows = (ps->n + slices - 1) / slices;
    pdl_launch(k_project_y, dim3((ps->n + 31) / 32, ps->nb, slices),
               dim3(1024), 0, ps->ctx->stream, ps->data.p, ps->ws.p,
               ps->proj[1].p, ps->py_part.p, ps->py_done.p, ps->n, rows);
}

void launch_integrate(vfps_ps* ps)
{
    const uint32_t wpb = ps->nb == 1 ? 8 : ps->nb == 2 ? 4
                         : ps->nb <= 4 ? 2 : 1;
    pdl_launch(k_integrate, dim3(1), dim3(256), 0, ps->ctx->stream,
               ps->proj64.p, ps->ws.p, ps->fillset.p, ps->filling.p, ps->nb,
               ps->n, wpb, ps->ctx->d_status);
}

void launch_normalize(vfps_ps* ps)
{
    const size_t nxy = size_t(ps->n) * ps->n;
    pdl_launch(k_normalize, dim3(grid_for(nxy * ps->nb, 256)), dim3(256), 0,
               ps->ctx->stream, ps->data.p, ps->fillset.p, ps->filling.p,
               ps->nb, nxy);
}

void launch_moments(vfps_ps* ps, int axis)
{
    // (FP64 sums: as many threads as cells, up to 1024)
    const int threads = ps->n <= 256 ? 256 : 1024;
    pdl_launch(k_moments, dim3(ps->nb), dim3(threads), 0, ps->ctx->stream,
               ps->proj[axis].p, ps->axisv[axis].p, ps->fillset.p,
               ps->filling.p, ps->ax[axis].delta, ps->nb, ps->n,
               ps->moments.p + size_t(axis) * 3 * ps->nb);
}

}  // namespace vfps
