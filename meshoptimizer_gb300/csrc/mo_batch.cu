// mo_batch.cu - the host side of the batch kernel (mo_batch_kernel.cuh): which form runs, the memory a
// mesh needs, and the launch.
#include "mo_batch_kernel.cuh"

#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>

namespace mogpu
{

template <class IX>
BatchBytes bytesOf(const BatchDesc& d)
{
	const bool sparse = (d.options & kOptSparse) != 0;
	const size_t I = d.index_count, bound = localVertexBound(I, d.vertex_count, sparse), V = expectedVertices(I, bound, sparse);
	BatchBytes b;
	b.smem = hotBytes<IX>(I, V, bound, expectedCapacity(I), sparse);
	b.rows = rowBytes<IX>(V, d.ac);
	b.slab = rowBytes<IX>(bound, d.ac) + hotBytes<IX>(I, bound, bound, std::max(I + 4, expectedCapacity(I)), sparse);
	return b;
}

BatchBytes batchBytes(const BatchDesc& d, bool narrow)
{
	return narrow ? bytesOf<unsigned short>(d) : bytesOf<unsigned int>(d);
}

BatchKernel batchKernel(int threads, bool full, bool narrow)
{
	return narrow ? (full ? batchKernelFull(threads) : batchKernelLean(threads)) : batchKernelWide(full);
}

int batchThreads(int threads, bool narrow)
{
	return narrow ? (threads == 128 || threads == 512 ? threads : 256) : 512;
}

// the dynamic shared-memory limit of every batch kernel instance is raised once, to the
// device's opt-in maximum: setting it per launch would race between threads launching batches
// with different sizes
void raiseSmemLimits()
{
	static std::once_flag once;
	std::call_once(once, [] {
		int dev = 0, optin = 0;
		cudaGetDevice(&dev);
		cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
		int limit = optin - 4096; // room for the kernel's static shared memory
		for (bool full : {false, true})
		{
			for (int threads : {128, 256, 512})
				cudaFuncSetAttribute((const void*)batchKernel(threads, full, true), cudaFuncAttributeMaxDynamicSharedMemorySize, limit);
			cudaFuncSetAttribute((const void*)batchKernel(512, full, false), cudaFuncAttributeMaxDynamicSharedMemorySize, limit);
		}
	});
}

void launchBatch(const BatchDesc* d_descs, unsigned int count, unsigned int* d_ticket, BatchResult* d_results, char* d_slabs, size_t slab_bytes,
    unsigned int smem_bytes, unsigned int blocks, int threads, bool full, bool narrow, cudaStream_t stream)
{
	raiseSmemLimits();
	MO_CUDA_CHECK(cudaMemsetAsync(d_ticket, 0, sizeof(unsigned int), stream));
	const BatchKernel kBatch = batchKernel(threads, full, narrow);
	MO_LAUNCH(kBatch, blocks, batchThreads(threads, narrow), smem_bytes, stream, d_descs, count, d_ticket, d_results, d_slabs, slab_bytes, smem_bytes);
	MO_CUDA_CHECK(cudaGetLastError());
}

// occupancy per (device, threads, shared memory, variant), queried once each: driver queries
// are not free, and a batch call makes one
int batchBlocksPerSM(int threads, unsigned int smem_bytes, bool full, bool narrow)
{
	raiseSmemLimits();
	static std::mutex lock;
	static std::map<std::tuple<int, int, unsigned int, bool, bool>, int> known;
	int dev = 0;
	cudaGetDevice(&dev);
	const auto key = std::make_tuple(dev, threads, smem_bytes, full, narrow);
	{
		std::lock_guard<std::mutex> g(lock);
		auto it = known.find(key);
		if (it != known.end())
			return it->second;
	}
	int n = 0;
	cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, (const void*)batchKernel(threads, full, narrow), batchThreads(threads, narrow), smem_bytes);
	std::lock_guard<std::mutex> g(lock);
	known[key] = n;
	return n;
}

} // namespace mogpu
