// fields.h -- transfers of tracer fields (fields.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace lbg {

// A three-component field on the device: float4 records (rec), or three arrays of doubles (comp).
struct Field3 {
    float4 *rec;
    double *comp[3];
};

// nodes converted at a time; `stage` below holds 3 doubles of each (12 MiB at most)
constexpr size_t FIELD_CHUNK = 1u << 19, FIELD_CHUNK_LEAST = 1u << 12;   // the least: where the device has no room
inline size_t field_chunk_nodes(long long N) { return (size_t)N < FIELD_CHUNK ? (size_t)N : FIELD_CHUNK; }
// host[3 i + d] = component d of node i (and back), waiting for the stream; `chunk` nodes of stage
cudaError_t field_to_host(const Field3 &f, long long N, double *stage, size_t chunk, double *host, cudaStream_t s);
// both fields of a box of half a chunk at most at once (a: host_a, b: host_b), with 6 doubles of stage per node
cudaError_t fields_to_host(const Field3 &a, const Field3 &b, long long N, double *stage, double *host_a, double *host_b,
                           cudaStream_t s);
cudaError_t field_from_host(const Field3 &f, long long N, double *stage, size_t chunk, const double *host, cudaStream_t s);

}  // namespace lbg
