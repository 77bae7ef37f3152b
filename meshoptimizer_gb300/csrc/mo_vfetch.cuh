// mo_vfetch.cuh - vertex-buffer compaction after simplification, on device data
// (src/vfetchoptimizer.cpp:7-71, src/indexgenerator.cpp:555-578).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

namespace mogpu
{

// scratch words vertexOrder needs
size_t vertexOrderScratchWords(size_t index_count, size_t vertex_count);

// order[v] = new index of vertex v in order of first use by indices; mark_unused: ~0u if unused (else
// left as it is, and the scratch keeps the vertices in their new order, vertexOrderList). counters: 5
// device words, read by takeOrderCount.
void vertexOrder(unsigned int* order, bool mark_unused, const unsigned int* indices, size_t index_count, size_t vertex_count, unsigned int* scratch,
    unsigned int* counters, cudaStream_t stream);
unsigned int* vertexOrderList(unsigned int* scratch, size_t vertex_count);

// waits for the stream; the used vertex count, or an exception if an index is out of range
unsigned int takeOrderCount(const unsigned int* counters, cudaStream_t stream);

// destination[order[v]] = vertices[v] for used vertices (vertex_size bytes each; the buffers must not
// overlap) and indices[i] = order[indices[i]]; nothing if an index is out of range
void compactVertices(void* destination, const void* vertices, size_t vertex_count, size_t vertex_size, unsigned int* indices, size_t index_count,
    const unsigned int* order, const unsigned int* list, const unsigned int* counters, cudaStream_t stream);

// scratch words positionRemap needs
size_t positionRemapScratchWords(size_t vertex_count);

// remap[i] = smallest vertex index whose position (the first 3 floats of each stride_f-float
// vertex) compares equal to vertex i's. counters: [1] nonzero if the table overflowed.
void positionRemap(unsigned int* remap, const float* positions, size_t vertex_count, size_t stride_f, unsigned int* scratch, unsigned int* counters,
    cudaStream_t stream);

} // namespace mogpu
