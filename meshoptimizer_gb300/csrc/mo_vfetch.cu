// mo_vfetch.cu - the compaction step that follows the simplifier in its callers, on device data:
// meshopt_optimizeVertexFetchRemap / meshopt_optimizeVertexFetch (src/vfetchoptimizer.cpp:7-71)
// and meshopt_generatePositionRemap (src/indexgenerator.cpp:555-578).
//
// The reference walks the index buffer once and numbers vertices as they are first seen. Here
// the same order comes from two data-parallel steps: the first index position of every vertex
// (atomicMin), and a scan over the index positions that are first uses, whose value there is that
// vertex's new index. Vertices then move from the new order's side, so only used ones are read and
// neighbouring threads write neighbouring bytes. The position remap
// is an open-addressing table keyed by position in which the smallest vertex index of each
// position wins (atomicMin), which is the vertex the reference's sequential insertion keeps.
#include "mo_vfetch.cuh"
#include "mo_common.cuh"
#include "mo_grid.cuh"
#include "mo_prims.cuh"
#include "mo_probe.cuh"

#include <algorithm>
#include <atomic>
#include <stdexcept>

namespace mogpu
{

namespace
{

constexpr int kThreads = 256;

__device__ __forceinline__ size_t gtidv()
{
	return (size_t)blockIdx.x * blockDim.x + threadIdx.x;
}

// first[v] = smallest index position that references v; out-of-range indices raise *bad
__global__ void kFirstPosition(const unsigned int* __restrict__ idx, size_t n, size_t vcount, unsigned int* first, unsigned int* bad)
{
	size_t p = gtidv();
	if (p >= n)
		return;
	unsigned int v = idx[p];
	if (v >= vcount)
	{
		atomicOr(bad, 1u);
		return;
	}
	atomicMin(&first[v], (unsigned int)p);
}

constexpr unsigned int kOrderTile = kThreads * 4;

// counters: used vertices, bad indices, the grid barrier's two words and its error flag
constexpr int kCounters = 5;

// order[v] = rank of v's first use among the index positions that are first uses, list[rank] = v: one
// cooperative launch, each block over a run of tiles, counting them, then (behind the grid barrier)
// adding up the counts before it and ranking them. A flag per position, its three-launch scan and a
// pass over all vertices before it moved 16 bytes per index and 8 per vertex more, in five launches. The
// gathers of first are what counts where indices are in no order, so what they gave is kept from the count
// for the ranks, four bits per tile: 2M vertices, 6M random indices, the order alone 143 us with the
// gathers done twice, 116 so (131 in five launches).
__global__ void __launch_bounds__(kThreads) kVertexOrder(const unsigned int* __restrict__ idx, size_t n, size_t vcount, const unsigned int* __restrict__ first,
    unsigned int* __restrict__ order, unsigned int* __restrict__ list, unsigned int* sums, unsigned int* counters)
{
	__shared__ unsigned int smem[kThreads / 32 + 1];
	const size_t tiles = (n + kOrderTile - 1) / kOrderTile, per = (tiles + gridDim.x - 1) / gridDim.x;
	const size_t t0 = min(tiles, (size_t)blockIdx.x * per), t1 = min(tiles, t0 + per);
	auto firstUses = [&](size_t t) {
		const size_t p = t * kOrderTile + threadIdx.x * 4;
		unsigned int uses = 0, v[4];
#pragma unroll
		for (int j = 0; j < 4; ++j)
			v[j] = p + j < n ? idx[p + j] : ~0u;
#pragma unroll
		for (int j = 0; j < 4; ++j)
			uses |= (v[j] < vcount && first[v[j]] == (unsigned int)(p + j)) ? 1u << j : 0u;
		return uses;
	};
	unsigned int c = 0;
	unsigned long long kept = 0; // of the first 16 tiles
	for (size_t t = t0; t < t1; ++t)
	{
		const unsigned int uses = firstUses(t);
		c += __popc(uses);
		if (t - t0 < 16)
			kept |= (unsigned long long)uses << (t - t0) * 4;
	}
	unsigned int total;
	blockExclusiveScan<kThreads>(c, smem, &total);
	if (threadIdx.x == 0)
		sums[blockIdx.x] = total;
	gridBarrierOnce(counters + 2, counters + 4);
	if (__ldcg(counters + 4))
		return; // a barrier wait ran out: nothing is written from incomplete sums
	unsigned int before = 0, base;
	for (unsigned int q = threadIdx.x; q < blockIdx.x; q += kThreads)
		before += __ldcg(sums + q);
	blockExclusiveScan<kThreads>(before, smem, &base);
	for (size_t t = t0; t < t1; ++t)
	{
		const unsigned int uses = t - t0 < 16 ? (unsigned int)(kept >> (t - t0) * 4) & 15u : firstUses(t);
		__syncthreads(); // every thread has read the previous scan's shared words
		unsigned int r = base + blockExclusiveScan<kThreads>(__popc(uses), smem, &total);
#pragma unroll
		for (int j = 0; j < 4; ++j)
			if (uses >> j & 1u)
			{
				const unsigned int v = idx[t * kOrderTile + threadIdx.x * 4 + j];
				order[v] = r;
				if (list)
					list[r] = v;
				++r;
			}
		base += total;
	}
	if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0)
		counters[0] = base;
}

// indices to the new order; nothing where an index is bad or the order is incomplete
__global__ void kRewriteIndices(unsigned int* idx, size_t n, const unsigned int* __restrict__ order, const unsigned int* __restrict__ counters)
{
	size_t p = gtidv();
	if (p < n && !counters[1] && !counters[4])
		idx[p] = order[idx[p]];
}

// row r of the new order from vertex list[r], by 2^log_lanes threads per row in units of T (a divisor
// of the vertex size that both buffers are aligned to)
template <class T>
__global__ void kMoveVertices(const T* __restrict__ src, unsigned int units, unsigned int log_lanes, const unsigned int* __restrict__ list,
    const unsigned int* __restrict__ counters, T* __restrict__ dst)
{
	const size_t t = gtidv(), r = t >> log_lanes;
	if (r >= counters[0] || counters[1] || counters[4])
		return;
	const size_t from = (size_t)list[r] * units, to = r * units;
	for (unsigned int u = (unsigned int)t & ((1u << log_lanes) - 1u); u < units; u += 1u << log_lanes)
		dst[to + u] = src[from + u];
}

__device__ __forceinline__ unsigned int keyBits(float f)
{
	unsigned int u = __float_as_uint(f);
	return u == 0x80000000u ? 0u : u; // -0 hashes as +0 (they compare equal)
}

__device__ __forceinline__ unsigned int mixBits(unsigned int h)
{
	h ^= h >> 16;
	h *= 0x7feb352du;
	h ^= h >> 15;
	h *= 0x846ca68bu;
	h ^= h >> 16;
	return h;
}

// position table: a vertex claims an empty slot or, finding a slot whose vertex has an equal
// position, lowers it to its own index if smaller; slot[i] records where vertex i landed
__global__ void kPositionInsert(const float* __restrict__ pos, size_t stride_f, size_t n, unsigned int* table, unsigned int mask, unsigned int* __restrict__ slot,
    unsigned int* fail)
{
	size_t vi = gtidv();
	if (vi >= n)
		return;
	unsigned int i = (unsigned int)vi;
	const float* p = pos + vi * stride_f;
	float x = p[0], y = p[1], z = p[2];
	unsigned int h = mixBits(keyBits(x) * 0x9e3779b1u ^ mixBits(keyBits(y) + 0x85ebca6bu) ^ mixBits(keyBits(z) * 0xc2b2ae35u + 1u));
	unsigned int b = h & mask;
	for (unsigned int probe = 0; probe <= mask; ++probe)
	{
		unsigned int cur = table[b];
		if (cur == ~0u)
		{
			unsigned int prev = atomicCAS(&table[b], ~0u, i);
			if (prev == ~0u)
			{
				slot[i] = b;
				return;
			}
			cur = prev;
		}
		const float* q = pos + (size_t)cur * stride_f;
		if (q[0] == x && q[1] == y && q[2] == z)
		{
			atomicMin(&table[b], i);
			slot[i] = b;
			return;
		}
		b = (b + probe + 1) & mask;
	}
	atomicOr(fail, 1u);
	slot[i] = ~0u;
}

__global__ void kPositionRemap(const unsigned int* __restrict__ table, const unsigned int* __restrict__ slot, size_t n, unsigned int* __restrict__ remap)
{
	size_t i = gtidv();
	if (i >= n)
		return;
	unsigned int s = slot[i];
	remap[i] = s == ~0u ? (unsigned int)i : table[s];
}

size_t alignWords(size_t n)
{
	return (n + 63) & ~size_t(63);
}

} // namespace

constexpr unsigned int kOrderBlocksMax = 4096; // words for the blocks' sums

// co-resident blocks of kVertexOrder on the current device, queried once
unsigned int orderBlocks()
{
	constexpr int kDevices = 64;
	static std::atomic<unsigned int> cache[kDevices];
	int dev = 0, sms = 0, occ = 0;
	MO_CUDA_CHECK(cudaGetDevice(&dev));
	unsigned int c = dev < kDevices ? cache[dev].load(std::memory_order_relaxed) : 0u;
	if (c)
		return c;
	MO_CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
	MO_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kVertexOrder, kThreads, 0));
	c = std::min(kOrderBlocksMax, unsigned(std::max(1, sms) * std::max(1, std::min(occ, 4))));
	if (dev < kDevices)
		cache[dev].store(c, std::memory_order_relaxed);
	return c;
}

size_t vertexOrderScratchWords(size_t index_count, size_t vertex_count)
{
	return alignWords(vertex_count) + alignWords(std::min(index_count, vertex_count)) + kOrderBlocksMax + 64;
}

unsigned int* vertexOrderList(unsigned int* scratch, size_t vertex_count)
{
	return scratch + alignWords(vertex_count);
}

void vertexOrder(unsigned int* order, bool mark_unused, const unsigned int* indices, size_t index_count, size_t vertex_count, unsigned int* scratch,
    unsigned int* counters, cudaStream_t stream)
{
	unsigned int* first = scratch;
	unsigned int* list = vertexOrderList(scratch, vertex_count);
	unsigned int* sums = list + alignWords(std::min(index_count, vertex_count));
	if (mark_unused)
		list = nullptr; // the order itself is wanted
	MO_CUDA_CHECK(cudaMemsetAsync(counters, 0, kCounters * sizeof(unsigned int), stream));
	if (vertex_count && mark_unused)
		MO_CUDA_CHECK(cudaMemsetAsync(order, 0xFF, vertex_count * sizeof(unsigned int), stream));
	if (!index_count)
		return;
	if (vertex_count)
		MO_CUDA_CHECK(cudaMemsetAsync(first, 0xFF, vertex_count * sizeof(unsigned int), stream));
	MO_LAUNCH(kFirstPosition, gridFor(index_count, kThreads), kThreads, 0, stream, indices, index_count, vertex_count, first, &counters[1]);
	const size_t tiles = (index_count + kOrderTile - 1) / kOrderTile, cap = orderBlocks(), per = (tiles + cap - 1) / cap;
	const unsigned int blocks = unsigned((tiles + per - 1) / per);
	const unsigned int* cfirst = first;
	void* params[] = {(void*)&indices, (void*)&index_count, (void*)&vertex_count, (void*)&cfirst, (void*)&order, (void*)&list, (void*)&sums, (void*)&counters};
	cudaEvent_t e0 = probeBegin("kVertexOrder", stream);
	MO_CUDA_CHECK(cudaLaunchCooperativeKernel((const void*)kVertexOrder, dim3(blocks), dim3(kThreads), params, 0, stream));
	probeEnd(e0, stream);
}

unsigned int takeOrderCount(const unsigned int* counters, cudaStream_t stream)
{
	unsigned int h[kCounters];
	MO_CUDA_CHECK(cudaMemcpyAsync(h, counters, sizeof(h), cudaMemcpyDeviceToHost, stream));
	MO_CUDA_CHECK(cudaStreamSynchronize(stream));
	probe().collect();
	if (h[1])
		throw std::invalid_argument("an index is out of range of vertex_count");
	if (h[4])
		throw std::runtime_error("grid barrier wait limit reached in the vertex order");
	return h[0];
}

template <class T>
void moveUnits(void* destination, const void* vertices, size_t rows, size_t vertex_size, const unsigned int* list, const unsigned int* counters, cudaStream_t stream)
{
	const unsigned int units = unsigned(vertex_size / sizeof(T));
	unsigned int log_lanes = 0;
	while (log_lanes < 5 && (1u << log_lanes) < units)
		++log_lanes;
	MO_LAUNCH(kMoveVertices<T>, gridFor(rows << log_lanes, kThreads), kThreads, 0, stream, static_cast<const T*>(vertices), units, log_lanes, list, counters,
	    static_cast<T*>(destination));
}

void compactVertices(void* destination, const void* vertices, size_t vertex_count, size_t vertex_size, unsigned int* indices, size_t index_count,
    const unsigned int* order, const unsigned int* list, const unsigned int* counters, cudaStream_t stream)
{
	if (!index_count)
		return;
	// the widest unit that divides the vertices and that both buffers are aligned to
	const size_t align = vertex_size | reinterpret_cast<uintptr_t>(destination) | reinterpret_cast<uintptr_t>(vertices);
	const size_t rows = std::min(vertex_count, index_count);
	if (rows)
	{
		if (align % 16 == 0)
			moveUnits<uint4>(destination, vertices, rows, vertex_size, list, counters, stream);
		else if (align % 8 == 0)
			moveUnits<uint2>(destination, vertices, rows, vertex_size, list, counters, stream);
		else if (align % 4 == 0)
			moveUnits<unsigned int>(destination, vertices, rows, vertex_size, list, counters, stream);
		else
			moveUnits<unsigned char>(destination, vertices, rows, vertex_size, list, counters, stream);
	}
	MO_LAUNCH(kRewriteIndices, gridFor(index_count, kThreads), kThreads, 0, stream, indices, index_count, order, counters);
}

size_t positionRemapScratchWords(size_t vertex_count)
{
	size_t buckets = 1;
	while (buckets < vertex_count + vertex_count / 4)
		buckets *= 2;
	return alignWords(buckets) + alignWords(vertex_count) + 64;
}

void positionRemap(unsigned int* remap, const float* positions, size_t vertex_count, size_t stride_f, unsigned int* scratch, unsigned int* counters,
    cudaStream_t stream)
{
	size_t buckets = 1;
	while (buckets < vertex_count + vertex_count / 4)
		buckets *= 2;
	unsigned int* table = scratch;
	unsigned int* slot = table + alignWords(buckets);
	MO_CUDA_CHECK(cudaMemsetAsync(counters, 0, 2 * sizeof(unsigned int), stream));
	if (!vertex_count)
		return;
	MO_CUDA_CHECK(cudaMemsetAsync(table, 0xFF, buckets * sizeof(unsigned int), stream));
	MO_LAUNCH(kPositionInsert, gridFor(vertex_count, kThreads), kThreads, 0, stream, positions, stride_f, vertex_count, table, unsigned(buckets - 1), slot,
	    &counters[1]);
	MO_LAUNCH(kPositionRemap, gridFor(vertex_count, kThreads), kThreads, 0, stream, table, slot, vertex_count, remap);
}

} // namespace mogpu
