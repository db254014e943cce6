// fields.cu -- the tracer fields between their device layouts and the caller's P(3,lx,ly,lz) arrays
// of doubles (component fastest).  The conversion runs on the device, chunk by chunk through a
// staging buffer, so the host only receives (or sends) finished arrays: converted by the host, one
// P of a 160^3 box took 20 ms, against 6 ms for the transfer into fresh pages.
#include "common.cuh"
#include "fields.h"
#include "host_pages.h"

namespace lbg {
namespace {

constexpr int BLOCK = 256;

// out[e] = component e % 3 of record e / 3: consecutive threads write consecutive doubles
__global__ void __launch_bounds__(BLOCK) k_pack32(const float4 *__restrict__ src, double *__restrict__ out, unsigned n)
{
    const unsigned e = blockIdx.x * BLOCK + threadIdx.x;
    if (e >= 3u * n) return;
    out[e] = (double)reinterpret_cast<const float *>(src)[4u * (e / 3u) + e % 3u];
}

__global__ void __launch_bounds__(BLOCK) k_pack64(const double *__restrict__ x, const double *__restrict__ y,
                                                  const double *__restrict__ z, double *__restrict__ out, unsigned n)
{
    const unsigned e = blockIdx.x * BLOCK + threadIdx.x;
    if (e >= 3u * n) return;
    const unsigned i = e / 3u, d = e % 3u;
    out[e] = (d == 0 ? x : (d == 1 ? y : z))[i];
}

__global__ void __launch_bounds__(BLOCK) k_unpack32(const double *__restrict__ in, float4 *__restrict__ dst, unsigned n)
{
    const unsigned i = blockIdx.x * BLOCK + threadIdx.x;
    if (i >= n) return;
    dst[i] = make_float4((float)in[3u * i], (float)in[3u * i + 1], (float)in[3u * i + 2], 0.0f);
}

__global__ void __launch_bounds__(BLOCK) k_unpack64(const double *__restrict__ in, double *__restrict__ x,
                                                    double *__restrict__ y, double *__restrict__ z, unsigned n)
{
    const unsigned i = blockIdx.x * BLOCK + threadIdx.x;
    if (i >= n) return;
    x[i] = in[3u * i];
    y[i] = in[3u * i + 1];
    z[i] = in[3u * i + 2];
}

unsigned blocks(size_t n) { return (unsigned)((n + BLOCK - 1) / BLOCK); }

}  // namespace

namespace {
cudaError_t pack(const Field3 &f, size_t at, unsigned n, double *stage, cudaStream_t s)
{
    if (f.rec) k_pack32<<<blocks(3 * (size_t)n), BLOCK, 0, s>>>(f.rec + at, stage, n);
    else k_pack64<<<blocks(3 * (size_t)n), BLOCK, 0, s>>>(f.comp[0] + at, f.comp[1] + at, f.comp[2] + at, stage, n);
    return cudaGetLastError();
}
}  // namespace

cudaError_t fields_to_host(const Field3 &a, const Field3 &b, long long N, double *stage, double *host_a, double *host_b,
                           cudaStream_t s)
{
    const size_t doubles = 3 * (size_t)N, bytes = sizeof(double) * doubles;
    cudaError_t e = pack(a, 0, (unsigned)N, stage, s);
    if (e == cudaSuccess) e = pack(b, 0, (unsigned)N, stage + doubles, s);
    if (e != cudaSuccess) return e;
    if (host_b == host_a + doubles) {   // one array: one copy
        ready_pages({{host_a, 2 * bytes}});
        e = cudaMemcpyAsync(host_a, stage, 2 * bytes, cudaMemcpyDeviceToHost, s);
    } else {
        ready_pages({{host_a, bytes}, {host_b, bytes}});
        e = cudaMemcpyAsync(host_a, stage, bytes, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaMemcpyAsync(host_b, stage + doubles, bytes, cudaMemcpyDeviceToHost, s);
    }
    return e == cudaSuccess ? cudaStreamSynchronize(s) : e;
}

cudaError_t field_to_host(const Field3 &f, long long N, double *stage, size_t chunk, double *host, cudaStream_t s)
{
    for (size_t at = 0; at < (size_t)N; at += chunk) {
        const unsigned n = (unsigned)((size_t)N - at < chunk ? (size_t)N - at : chunk);
        cudaError_t e = pack(f, at, n, stage, s);
        if (at == 0) ready_pages({{host, sizeof(double) * 3 * (size_t)N}});
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(host + 3 * at, stage, sizeof(double) * 3 * n, cudaMemcpyDeviceToHost, s);
        if (e != cudaSuccess) return e;
    }
    return cudaStreamSynchronize(s);
}

cudaError_t field_from_host(const Field3 &f, long long N, double *stage, size_t chunk, const double *host, cudaStream_t s)
{
    for (size_t at = 0; at < (size_t)N; at += chunk) {
        const unsigned n = (unsigned)((size_t)N - at < chunk ? (size_t)N - at : chunk);
        cudaError_t e = cudaMemcpyAsync(stage, host + 3 * at, sizeof(double) * 3 * n, cudaMemcpyHostToDevice, s);
        if (e != cudaSuccess) return e;
        if (f.rec) k_unpack32<<<blocks(n), BLOCK, 0, s>>>(stage, f.rec + at, n);
        else k_unpack64<<<blocks(n), BLOCK, 0, s>>>(stage, f.comp[0] + at, f.comp[1] + at, f.comp[2] + at, n);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    return cudaStreamSynchronize(s);
}

}  // namespace lbg
