// mo_batch.cuh - persistent multi-mesh simplification (one CTA per mesh, device work queue).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

namespace mogpu
{

// attributes with weight > 0 of a batched mesh (rescaleAttributes :605-621, :2410-2421): source
// column and weight of each used attribute
struct BatchAttr
{
	unsigned int src[32];
	float weight[32];
};

// one mesh of a batch; device pointers
struct BatchDesc
{
	const unsigned int* indices;
	const float* positions;
	unsigned int* out;
	unsigned int index_count;
	unsigned int vertex_count; // of the vertex buffer the indices address
	unsigned int stride_f;     // position stride in floats
	unsigned int target_index_count;
	float target_error;
	unsigned int options;
	const float* attributes;   // nullptr: positions only
	const unsigned char* lock; // vertex_lock, nullptr: none
	const BatchAttr* amap;     // used attributes (ac of them)
	unsigned int attr_stride_f;
	unsigned int ac;
};

struct BatchResult
{
	unsigned int index_count;
	float result_error;
	unsigned int passes;
	unsigned int status; // 0 ok, 2 invalid index, 3 a decision round made no progress, 4 its scratch was too small; and the bits below
};
constexpr unsigned int kBatchInSlab = 0x100; // the mesh ran in its CTA's slab
constexpr unsigned int kBatchBeyond = 0x200; // it had more vertices or a larger capacity than expected

// Memory of one mesh. smem: shared memory it is expected to need beside its attribute rows (rows), which
// go there too where they fit, else into the CTA's slab; slab: memory of either kind in which it runs
// whatever it turns out to need.
struct BatchBytes
{
	size_t smem, rows, slab;
};
BatchBytes batchBytes(const BatchDesc& d, bool narrow);

// whether a mesh's ids fit the kernels' 16-bit form: its indices, and its (local) vertices, of which a
// sparse mesh (option bit 1) has one per index at most
constexpr size_t kNarrowIndices = 60000;
constexpr size_t kNarrowVertices = 24000; // their table has at most 32,768 slots
inline bool batchNarrow(const BatchDesc& d)
{
	const bool few = d.vertex_count <= kNarrowVertices || ((d.options & (1u << 1)) && d.index_count <= kNarrowVertices);
	return d.index_count <= kNarrowIndices && few;
}

// whether a mesh needs the full-option kernel: a sparse subset (option bit 1), attributes,
// vertex_lock or Permissive (option bit 5)
inline bool batchNeedsFull(const BatchDesc& d)
{
	return d.ac || d.lock || (d.options & ((1u << 1) | (1u << 5)));
}

// the kernel's forms (mo_batch_kernel.cuh)
typedef void (*BatchKernel)(const BatchDesc*, unsigned int, unsigned int*, BatchResult*, char*, size_t, unsigned int);
BatchKernel batchKernelLean(int threads);
BatchKernel batchKernelFull(int threads);
BatchKernel batchKernelWide(bool full);

// resident CTAs per SM for a thread count, dynamic shared memory size and kernel form
int batchBlocksPerSM(int threads, unsigned int smem_bytes, bool full, bool narrow);

// full: the instantiation with every option; otherwise the positions-only one. narrow: every mesh is
// narrow. Every CTA has slab_bytes of slabs, the largest mesh's at least, or none where smem_bytes are that.
void launchBatch(const BatchDesc* d_descs, unsigned int count, unsigned int* d_ticket, BatchResult* d_results, char* d_slabs, size_t slab_bytes,
    unsigned int smem_bytes, unsigned int blocks, int threads, bool full, bool narrow, cudaStream_t stream);

} // namespace mogpu
