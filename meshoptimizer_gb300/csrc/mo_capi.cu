// mo_capi.cu - the C ABI (include/meshopt_gb300.h): drop-in entry points with the
// signatures of meshoptimizer.h, plus device-resident and diagnostic additions.
//
// Each calling thread owns one Simplifier (device scratch arena) and one CUDA stream, so
// concurrent callers do not share mutable state (the reference is reentrant too,
// meshoptimizer.h:1206-1210).
#include "../../include/meshopt_gb300.h"

#include "mo_common.cuh"
#include "mo_probe.cuh"
#include "mo_simplify.cuh"
#include "mo_batch.cuh"
#include "mo_vfetch.cuh"
#include "mo_groups.cuh"
#include "mo_meshlets.cuh"

#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <thread>
#include <tuple>
#include <memory>
#include <mutex>
#include <numeric>
#include <vector>
#include <new>
#include <string>

namespace
{

using namespace mogpu;

struct HostStaging
{
	void* ptr = nullptr;
	size_t cap = 0;
	~HostStaging()
	{
		if (ptr)
			cudaFreeHost(ptr);
	}
	void* ensure(size_t bytes)
	{
		if (bytes <= cap)
			return ptr;
		if (ptr)
			cudaFreeHost(ptr);
		ptr = nullptr;
		cap = 0;
		size_t want = bytes + bytes / 4 + 4096;
		MO_CUDA_CHECK(cudaMallocHost(&ptr, want));
		cap = want;
		return ptr;
	}
};

struct DeviceBuffer
{
	void* ptr = nullptr;
	size_t cap = 0;
	~DeviceBuffer()
	{
		if (ptr)
			cudaFree(ptr);
	}
	void* ensure(size_t bytes)
	{
		if (bytes <= cap)
			return ptr;
		if (ptr)
			cudaFree(ptr);
		ptr = nullptr;
		cap = 0;
		size_t want = bytes + bytes / 4 + 256;
		MO_CUDA_CHECK(cudaMalloc(&ptr, want));
		cap = want;
		return ptr;
	}
};

struct ThreadState
{
	int status = meshoptgpu_StatusOk;
	std::string message;
	int device = -1;
	cudaStream_t stream = nullptr;
	std::unique_ptr<Simplifier> simplifier;
	DeviceBuffer inputs;
	RunResult last;
	PhaseTimes times;
	bool timing = false;
	// batched path
	DeviceBuffer batch_meta, batch_slabs, batch_io, compact_scratch, group_scratch, update_io, meshlet_scratch;
	HostStaging batch_host, batch_meta_host;
	int batch_threads = 0;          // 0: autotune
	int sms = 1;                    // the device's SM count
	unsigned int batch_smem = 0;    // 0: default budget
	// drop-in calls with at most this many indices run on the batch kernel as a batch of one;
	// (size_t)-1: the autotuner picks the route per size class (see routeAndRun)
	size_t dropin_batch_limit = ~size_t(0);
	bool autotune = true; // the single-mesh path's launch shape and the drop-in route are timed per size class
	// drop-in copies on a stream of their own, in the order the setup first reads them:
	// positions, indices, attributes (one stream takes the whole host link, so a second one would
	// only slow the first inputs down). Events: positions, attributes, indices copied.
	cudaStream_t copy_stream = nullptr;
	cudaEvent_t copy_done[3] = {nullptr, nullptr, nullptr};
	// the second launch of a batch whose meshes need both forms of the kernel
	cudaStream_t batch_stream = nullptr;
	cudaEvent_t batch_event = nullptr;
	size_t batch_in_shared = 0, batch_in_slab = 0; // meshes of the last batch by where they ran
	size_t batch_slab_limit = ~size_t(0); // bytes of slabs a batch may allocate where its meshes can do without (the server's)

	void ensureBatchStream()
	{
		if (!batch_stream)
			MO_CUDA_CHECK(cudaStreamCreateWithFlags(&batch_stream, cudaStreamNonBlocking));
		if (!batch_event)
			MO_CUDA_CHECK(cudaEventCreateWithFlags(&batch_event, cudaEventDisableTiming));
	}

	void ensureCopyStreams()
	{
		if (!copy_stream)
			MO_CUDA_CHECK(cudaStreamCreateWithFlags(&copy_stream, cudaStreamNonBlocking));
		for (int i = 0; i < 3; ++i)
			if (!copy_done[i])
				MO_CUDA_CHECK(cudaEventCreateWithFlags(&copy_done[i], cudaEventDisableTiming));
	}

	void releaseStreams()
	{
		for (int i = 0; i < 3; ++i)
		{
			if (copy_done[i])
				cudaEventDestroy(copy_done[i]);
			copy_done[i] = nullptr;
		}
		if (copy_stream)
			cudaStreamDestroy(copy_stream);
		copy_stream = nullptr;
		if (batch_event)
			cudaEventDestroy(batch_event);
		batch_event = nullptr;
		if (batch_stream)
			cudaStreamDestroy(batch_stream);
		batch_stream = nullptr;
	}

	~ThreadState()
	{
		simplifier.reset();
		releaseStreams();
		if (stream)
			cudaStreamDestroy(stream);
	}

	void ensure()
	{
		int dev = 0;
		MO_CUDA_CHECK(cudaGetDevice(&dev));
		if (simplifier && device == dev)
			return;
		simplifier.reset();
		releaseStreams();
		if (stream)
			cudaStreamDestroy(stream);
		stream = nullptr;
		device = dev;
		MO_CUDA_CHECK(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
		MO_CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
		simplifier.reset(new Simplifier(dev));
		const char* at = getenv("MESHOPTGPU_AUTOTUNE");
		autotune = !(at && atoi(at) == 0) && !getenv("MESHOPTGPU_PERFORM_BLOCKS_PER_SM");
	}
};

// per-thread state, freed when the thread exits (server workers) or on request
thread_local std::unique_ptr<ThreadState> tls;

ThreadState& state()
{
	if (!tls)
		tls.reset(new ThreadState());
	return *tls;
}

void setStatus(int status, const std::string& msg)
{
	ThreadState& s = state();
	s.status = status;
	s.message = msg;
	if (status != meshoptgpu_StatusOk)
		fprintf(stderr, "meshopt_gb300: %s\n", msg.c_str());
}

const unsigned int kSupportedOptions =
    kOptLockBorder | kOptErrorAbsolute | kOptRegularize | kOptRegularizeLight | kOptSparse | kOptPermissive | kOptPrune | kOptInternalDebug;
// the one-CTA-per-mesh batch kernel implements every option but the component pruning and the
// debug output
const unsigned int kBatchOptions = kOptLockBorder | kOptErrorAbsolute | kOptRegularize | kOptRegularizeLight | kOptSparse | kOptPermissive;

// argument checks of meshopt_simplifyEdge (:2348-2357); returns an error message or empty
std::string checkArgs(size_t index_count, size_t vertex_positions_stride, size_t target_index_count, float target_error,
    size_t vertex_attributes_stride, const float* attribute_weights, size_t attribute_count, unsigned int options)
{
	if (index_count % 3 != 0)
		return "index_count must be a multiple of 3";
	if (vertex_positions_stride < 12 || vertex_positions_stride > 256 || vertex_positions_stride % 4 != 0)
		return "vertex_positions_stride must be in [12, 256] and a multiple of 4";
	if (target_index_count > index_count)
		return "target_index_count must not exceed index_count";
	if (!(target_error >= 0))
		return "target_error must be >= 0";
	if (attribute_count > (size_t)kMaxAttributes)
		return "attribute_count must be <= 32";
	if (attribute_count && (vertex_attributes_stride < attribute_count * 4 || vertex_attributes_stride > 256 || vertex_attributes_stride % 4 != 0))
		return "vertex_attributes_stride must be in [4*attribute_count, 256] and a multiple of 4";
	for (size_t i = 0; i < attribute_count; ++i)
		if (!(attribute_weights[i] >= 0))
			return "attribute weights must be >= 0";
	if (options & ~kSupportedOptions)
		return "option bits 0x" + [](unsigned v) {
			char b[16];
			snprintf(b, sizeof(b), "%x", v);
			return std::string(b);
		}(options & ~kSupportedOptions) + " are not implemented on the GPU path";
	return std::string();
}

int statusOf(const std::exception& e)
{
	if (auto ce = dynamic_cast<const CudaError*>(&e))
		return ce->code == cudaErrorMemoryAllocation ? meshoptgpu_StatusOutOfMemory : meshoptgpu_StatusCudaError;
	if (dynamic_cast<const std::invalid_argument*>(&e))
		return meshoptgpu_StatusInvalidArgument;
	if (dynamic_cast<const std::bad_alloc*>(&e))
		return meshoptgpu_StatusOutOfMemory;
	return meshoptgpu_StatusCudaError;
}

size_t failHost(unsigned int* destination, const unsigned int* indices, size_t index_count, float* result_error, int status, const std::string& msg)
{
	setStatus(status, msg);
	if (destination && indices && destination != indices)
		memmove(destination, indices, index_count * sizeof(unsigned int));
	if (result_error)
		*result_error = 0.f;
	return index_count;
}

size_t align256(size_t v)
{
	return (v + 255) & ~size_t(255);
}

// host bytes of `count` records of `stride` bytes of which the first `used` are read: the last
// record ends after its used bytes, as the reference reads it (an interleaved array may end
// there, and a copy of whole strides would read, or write back, past the caller's buffer)
size_t stridedExtent(size_t count, size_t stride, size_t used)
{
	return count ? (count - 1) * stride + used : 0;
}

struct HostCopy
{
	void* dst;
	const void* src;
	size_t bytes;
};

// Host threads for the batch path's packing and scattering copies (memory-bound host loops),
// started on first use and kept for the process (never joined: the threads only ever wait for
// the next job). One job at a time: a caller that finds the pool busy copies on its own thread.
class CopyPool
{
public:
	static CopyPool& get()
	{
		static CopyPool* pool = new CopyPool(); // left to the process: no teardown order at exit
		return *pool;
	}

	// copies[0, n) in `parts` contiguous runs given by cut (cut[0] = 0, cut[parts] = n); the calling
	// thread takes the last run. False when the pool is busy (nothing copied).
	bool run(const HostCopy* copies, const std::vector<size_t>& cut)
	{
		std::unique_lock<std::mutex> own(busy_, std::try_to_lock);
		if (!own.owns_lock())
			return false;
		const size_t parts = cut.size() - 1;
		{
			std::lock_guard<std::mutex> g(m_);
			while (workers_.size() + 1 < parts)
			{
				const size_t id = workers_.size();
				workers_.emplace_back([this, id]() { work(id); });
				workers_.back().detach();
			}
			copies_ = copies;
			cut_ = cut;
			pending_ = parts - 1;
			++generation_;
		}
		cv_.notify_all();
		copyRun(copies, cut[parts - 1], cut[parts]);
		std::unique_lock<std::mutex> g(m_);
		done_.wait(g, [&]() { return pending_ == 0; });
		return true;
	}

	static void copyRun(const HostCopy* copies, size_t b, size_t e)
	{
		for (size_t i = b; i < e; ++i)
			memcpy(copies[i].dst, copies[i].src, copies[i].bytes);
	}

private:
	void work(size_t id)
	{
		size_t seen = 0;
		for (;;)
		{
			const HostCopy* copies;
			size_t b, e;
			{
				std::unique_lock<std::mutex> g(m_);
				cv_.wait(g, [&]() { return generation_ != seen; });
				seen = generation_;
				if (id + 1 >= cut_.size() - 1)
					continue; // this job has fewer runs than workers
				copies = copies_;
				b = cut_[id];
				e = cut_[id + 1];
			}
			copyRun(copies, b, e);
			std::lock_guard<std::mutex> g(m_);
			if (--pending_ == 0)
				done_.notify_one();
		}
	}

	std::mutex busy_, m_;
	std::condition_variable cv_, done_;
	std::vector<std::thread> workers_;
	const HostCopy* copies_ = nullptr;
	std::vector<size_t> cut_;
	size_t generation_ = 0, pending_ = 0;
};

// Host memcpy of many pieces, spread over up to 16 threads in contiguous runs of about equal
// bytes when there is enough to copy (one thread per 256 KiB at least: one host thread copies
// about 10 GB/s, the link to the GPU takes 200).
void parallelCopies(const HostCopy* copies, size_t n)
{
	size_t total = 0;
	for (size_t i = 0; i < n; ++i)
		total += copies[i].bytes;
	const unsigned int hw = std::max(1u, std::thread::hardware_concurrency());
	const size_t threads = std::min<size_t>(std::min<size_t>(16, hw), total >> 18);
	if (threads <= 1)
	{
		CopyPool::copyRun(copies, 0, n);
		return;
	}
	std::vector<size_t> cut(1, 0);
	size_t acc = 0;
	const size_t share = total / threads;
	for (size_t i = 0; i < n && cut.size() < threads; ++i)
	{
		acc += copies[i].bytes;
		if (acc >= share * cut.size())
			cut.push_back(i + 1);
	}
	cut.push_back(n);
	if (!CopyPool::get().run(copies, cut))
		CopyPool::copyRun(copies, 0, n);
}

void parallelCopies(const std::vector<HostCopy>& copies)
{
	parallelCopies(copies.data(), copies.size());
}

// Offsets of distinct (pointer, bytes) keys in insertion order: an open-addressing table over a
// flat array (no allocation per key), for packing the arrays that meshes of a batch share once.
class PieceTable
{
public:
	explicit PieceTable(size_t keys)
	{
		size_t cap = 16;
		while (cap < 2 * keys)
			cap <<= 1;
		slots_.assign(cap, Slot{nullptr, 0, 0});
	}
	// the offset stored for (p, bytes), or ~0 after storing `at` for it
	size_t findOrInsert(const void* p, size_t bytes, size_t at)
	{
		const size_t mask = slots_.size() - 1;
		size_t h = (reinterpret_cast<uintptr_t>(p) * 0x9E3779B97F4A7C15ull ^ bytes * 0xC2B2AE3D27D4EB4Full) >> 17;
		for (;; ++h)
		{
			Slot& sl = slots_[h & mask];
			if (!sl.p)
			{
				sl = Slot{p, bytes, at};
				return ~size_t(0);
			}
			if (sl.p == p && sl.bytes == bytes)
				return sl.at;
		}
	}

private:
	struct Slot
	{
		const void* p;
		size_t bytes, at;
	};
	std::vector<Slot> slots_;
};

// Runs a small mesh (device pointers) on the batch kernel when the mesh's options allow; returns
// false to leave it to the single-mesh path.
bool smallMeshOnBatch(ThreadState& s, const MeshDesc& m, unsigned int* d_out, cudaStream_t st);

// A drop-in or device call's simplification (device pointers): on the batch kernel or the
// single-mesh path, as the calling thread's drop-in limit or the autotuner decides; the result
// in d_out and s.last.
void routeAndRun(ThreadState& s, const MeshDesc& m, unsigned int* d_out, cudaStream_t st, bool allow_batch);

// the index count above which routeAndRun sends every drop-in call to the single-mesh path
size_t singlePathAbove(const ThreadState& s);

size_t simplifyHost(unsigned int* destination, const unsigned int* indices, size_t index_count, const float* vertex_positions, size_t vertex_count,
    size_t vertex_positions_stride, const float* vertex_attributes, size_t vertex_attributes_stride, const float* attribute_weights, size_t attribute_count,
    const unsigned char* vertex_lock, size_t target_index_count, float target_error, unsigned int options, float* result_error)
{
	std::string bad = checkArgs(index_count, vertex_positions_stride, target_index_count, target_error, vertex_attributes_stride, attribute_weights,
	    attribute_count, options);
	if (!bad.empty())
		return failHost(destination, indices, index_count, result_error,
		    (options & ~kSupportedOptions) ? meshoptgpu_StatusUnsupported : meshoptgpu_StatusInvalidArgument, bad);
	bool split = false; // inputs copied on the copy streams too
	try
	{
		ThreadState& s = state();
		s.ensure();
		// device copies of the inputs, laid out back to back in one buffer
		size_t b_idx = align256(index_count * 4), b_pos = align256(vertex_count * vertex_positions_stride);
		size_t b_attr = attribute_count ? align256(vertex_count * vertex_attributes_stride) : 0;
		size_t b_lock = vertex_lock ? align256(vertex_count) : 0;
		size_t b_out = align256(index_count * 4);
		char* base = static_cast<char*>(s.inputs.ensure(b_idx + b_pos + b_attr + b_lock + b_out + 256));
		unsigned int* d_idx = reinterpret_cast<unsigned int*>(base);
		float* d_pos = reinterpret_cast<float*>(base + b_idx);
		float* d_attr = attribute_count ? reinterpret_cast<float*>(base + b_idx + b_pos) : nullptr;
		unsigned char* d_lock = vertex_lock ? reinterpret_cast<unsigned char*>(base + b_idx + b_pos + b_attr) : nullptr;
		unsigned int* d_out = reinterpret_cast<unsigned int*>(base + b_idx + b_pos + b_attr + b_lock);
		cudaStream_t st = s.stream;
		// large meshes on the single-mesh path: the copies on the copy stream, positions first (the
		// setup's first kernels read only them), then indices, then attributes; the setup waits for
		// each where it first reads it
		const size_t pos_bytes = stridedExtent(vertex_count, vertex_positions_stride, 12);
		const size_t attr_bytes = d_attr ? stridedExtent(vertex_count, vertex_attributes_stride, attribute_count * 4) : 0;
		split = index_count * 4 + pos_bytes + attr_bytes >= (size_t(1) << 20) && index_count > singlePathAbove(s);
		if (split)
		{
			s.ensureCopyStreams();
			if (vertex_count)
				MO_CUDA_CHECK(cudaMemcpyAsync(d_pos, vertex_positions, pos_bytes, cudaMemcpyHostToDevice, s.copy_stream));
			MO_CUDA_CHECK(cudaEventRecord(s.copy_done[0], s.copy_stream));
			if (index_count)
				MO_CUDA_CHECK(cudaMemcpyAsync(d_idx, indices, index_count * 4, cudaMemcpyHostToDevice, s.copy_stream));
			MO_CUDA_CHECK(cudaEventRecord(s.copy_done[2], s.copy_stream));
			if (d_attr)
				MO_CUDA_CHECK(cudaMemcpyAsync(d_attr, vertex_attributes, attr_bytes, cudaMemcpyHostToDevice, s.copy_stream));
			MO_CUDA_CHECK(cudaEventRecord(s.copy_done[1], s.copy_stream));
			MO_CUDA_CHECK(cudaStreamWaitEvent(st, s.copy_done[0], 0));
		}
		else
		{
			if (index_count)
				MO_CUDA_CHECK(cudaMemcpyAsync(d_idx, indices, index_count * 4, cudaMemcpyHostToDevice, st));
			if (vertex_count)
				MO_CUDA_CHECK(cudaMemcpyAsync(d_pos, vertex_positions, pos_bytes, cudaMemcpyHostToDevice, st));
			if (d_attr)
				MO_CUDA_CHECK(cudaMemcpyAsync(d_attr, vertex_attributes, attr_bytes, cudaMemcpyHostToDevice, st));
		}
		if (d_lock)
			MO_CUDA_CHECK(cudaMemcpyAsync(d_lock, vertex_lock, vertex_count, cudaMemcpyHostToDevice, st));

		MeshDesc m;
		m.indices = d_idx;
		m.index_count = index_count;
		m.positions = d_pos;
		m.vertex_count = vertex_count;
		m.positions_stride = vertex_positions_stride;
		m.attributes = d_attr;
		m.attributes_stride = vertex_attributes_stride;
		m.weights = attribute_weights;
		m.attribute_count = attribute_count;
		m.lock = d_lock;
		m.target_index_count = target_index_count;
		m.target_error = target_error;
		m.options = options;
		m.attributes_ready = split ? s.copy_done[1] : nullptr;
		m.indices_ready = split ? s.copy_done[2] : nullptr;
		routeAndRun(s, m, d_out, st, !split);
		if (s.last.index_count)
			MO_CUDA_CHECK(cudaMemcpyAsync(destination, d_out, s.last.index_count * 4, cudaMemcpyDeviceToHost, st));
		MO_CUDA_CHECK(cudaStreamSynchronize(st));
		if (split) // the caller's index and attribute buffers are read to the end before returning
		{
			MO_CUDA_CHECK(cudaEventSynchronize(s.copy_done[1]));
			MO_CUDA_CHECK(cudaEventSynchronize(s.copy_done[2]));
		}
		if (result_error)
			*result_error = s.last.result_error;
		setStatus(meshoptgpu_StatusOk, "");
		return s.last.index_count;
	}
	catch (const std::exception& e)
	{
		if (split)
		{
			ThreadState& s = state();
			cudaEventSynchronize(s.copy_done[0]);
			cudaEventSynchronize(s.copy_done[1]);
			cudaEventSynchronize(s.copy_done[2]);
		}
		return failHost(destination, indices, index_count, result_error, statusOf(e), e.what());
	}
}

// ---------------------------------------------------------------- the update mode

// meshopt_simplifyWithUpdate on host buffers. The vertex data goes to the device as one region
// when positions and attributes overlap (one interleaved buffer, as the reference's tests pass
// it) or as two, and comes back the same way after the write-back.
size_t updateHost(unsigned int* indices, size_t index_count, float* vertex_positions, size_t vertex_count, size_t vertex_positions_stride,
    float* vertex_attributes, size_t vertex_attributes_stride, const float* attribute_weights, size_t attribute_count, const unsigned char* vertex_lock,
    size_t target_index_count, float target_error, unsigned int options, float* result_error)
{
	std::string bad = checkArgs(index_count, vertex_positions_stride, target_index_count, target_error, vertex_attributes_stride, attribute_weights,
	    attribute_count, options);
	if (!bad.empty())
		return failHost(indices, indices, index_count, result_error,
		    (options & ~kSupportedOptions) ? meshoptgpu_StatusUnsupported : meshoptgpu_StatusInvalidArgument, bad);
	try
	{
		ThreadState& s = state();
		s.ensure();
		const size_t pbytes = stridedExtent(vertex_count, vertex_positions_stride, 12);
		const size_t abytes = attribute_count ? stridedExtent(vertex_count, vertex_attributes_stride, attribute_count * 4) : 0;
		const char* P = reinterpret_cast<const char*>(vertex_positions);
		const char* A = reinterpret_cast<const char*>(vertex_attributes);
		const bool joint = abytes && A < P + pbytes && P < A + abytes;
		const char* lo = joint ? std::min(P, A) : P;
		const size_t span = joint ? size_t(std::max(P + pbytes, A + abytes) - lo) : pbytes;
		size_t b_idx = align256(index_count * 4), b_v = align256(span), b_a = joint ? 0 : align256(abytes), b_lock = vertex_lock ? align256(vertex_count) : 0;
		char* base = static_cast<char*>(s.update_io.ensure(b_idx + b_v + b_a + b_lock + 256));
		unsigned int* d_idx = reinterpret_cast<unsigned int*>(base);
		char* d_v = base + b_idx;
		float* d_pos = reinterpret_cast<float*>(d_v + (P - lo));
		float* d_attr = abytes ? (joint ? reinterpret_cast<float*>(d_v + (A - lo)) : reinterpret_cast<float*>(base + b_idx + b_v)) : nullptr;
		unsigned char* d_lock = vertex_lock ? reinterpret_cast<unsigned char*>(base + b_idx + b_v + b_a) : nullptr;
		cudaStream_t st = s.stream;
		if (index_count)
			MO_CUDA_CHECK(cudaMemcpyAsync(d_idx, indices, index_count * 4, cudaMemcpyHostToDevice, st));
		if (span)
			MO_CUDA_CHECK(cudaMemcpyAsync(d_v, lo, span, cudaMemcpyHostToDevice, st));
		if (abytes && !joint)
			MO_CUDA_CHECK(cudaMemcpyAsync(d_attr, A, abytes, cudaMemcpyHostToDevice, st));
		if (d_lock)
			MO_CUDA_CHECK(cudaMemcpyAsync(d_lock, vertex_lock, vertex_count, cudaMemcpyHostToDevice, st));
		MeshDesc m;
		m.indices = d_idx;
		m.index_count = index_count;
		m.positions = d_pos;
		m.vertex_count = vertex_count;
		m.positions_stride = vertex_positions_stride;
		m.attributes = d_attr;
		m.attributes_stride = vertex_attributes_stride;
		m.weights = attribute_weights;
		m.attribute_count = attribute_count;
		m.lock = d_lock;
		m.target_index_count = target_index_count;
		m.target_error = target_error;
		m.options = options | kOptInternalSolve;
		m.update_positions = d_pos;
		m.update_attributes = d_attr;
		s.last = s.simplifier->run(m, d_idx, st, s.timing ? &s.times : nullptr);
		if (s.last.index_count)
			MO_CUDA_CHECK(cudaMemcpyAsync(indices, d_idx, s.last.index_count * 4, cudaMemcpyDeviceToHost, st));
		if (span)
			MO_CUDA_CHECK(cudaMemcpyAsync(const_cast<char*>(lo), d_v, span, cudaMemcpyDeviceToHost, st));
		if (abytes && !joint)
			MO_CUDA_CHECK(cudaMemcpyAsync(vertex_attributes, d_attr, abytes, cudaMemcpyDeviceToHost, st));
		MO_CUDA_CHECK(cudaStreamSynchronize(st));
		if (result_error)
			*result_error = s.last.result_error;
		setStatus(meshoptgpu_StatusOk, "");
		return s.last.index_count;
	}
	catch (const std::exception& e)
	{
		return failHost(indices, indices, index_count, result_error, statusOf(e), e.what());
	}
}

// ---------------------------------------------------------------- batched path

const size_t kBatchSmemDefault = 110 * 1024;    // shared-memory budget per CTA (two CTAs per SM)
const size_t kBatchSlabTotal = size_t(16) << 30; // global slabs for meshes beyond the budget

// threads per CTA, shared-memory budget per CTA, and whether the shared memory under that budget is sized
// for the most a mesh can need rather than for what it is expected to
struct BatchShape
{
	int threads = 0;
	size_t budget = 0;
	bool sure = false;
};

// The fastest shapes of a class: for meshes as expected, and for batches with many that need more (ribbons
// and separate quads, whose edges are borders; flat shaded groups, with three vertices per triangle), which
// shared memory sized by the expectation sends to the slab after their setup or part of it. What the
// class's last batch was like says which one is next. 4,096 ribbons of 120 / 200 triangles 1.44 / 2.01 ms
// by the expectation and 0.82 / 1.04 by the most they can need; flat groups of 60 / 200 triangles 0.80 /
// 1.75 and 0.57 / 0.96.
struct BatchShapes
{
	BatchShape as_expected, beyond;
	bool timed_beyond = false, last_beyond = false;
};

struct BatchTuner
{
	std::mutex lock;
	// (device, size class, the batch has more meshes than SMs, full form) -> fastest shape: a mesh that has
	// an SM to itself wants many threads, a batch that fills the GPU many CTAs (4,096 groups with what their
	// size class's single meshes had been given: 2.09 ms against 1.43), and the lean and full forms differ
	// in registers (4,096 meshes of 384 triangles with five attributes, with what positions-only ones had
	// been given: 2.63 ms against 1.66)
	std::map<std::tuple<int, int, bool, bool>, BatchShapes> shape;
} g_tuner;

// the shared-memory budgets the batch autotuner times (four, two and one CTAs per SM; a smaller largest
// mesh leaves room for more)
const size_t kBatchSmemBudgets[3] = {54 * 1024, kBatchSmemDefault, 216 * 1024};

int sizeClass(size_t max_index_count)
{
	int c = 0;
	while ((size_t(1) << c) < max_index_count)
		++c;
	return c;
}

// The used attributes (weight > 0, :2410-2421) of a batched mesh, deduplicated across the
// batch: meshes with the same weights share one map in device memory.
struct AttrMaps
{
	std::vector<BatchAttr> maps;
	std::map<std::string, int> index;

	// returns the map's index (or -1 when no attribute has a positive weight); ac = used count
	int add(const float* weights, size_t count, unsigned int& ac)
	{
		BatchAttr a;
		memset(&a, 0, sizeof(a));
		ac = 0;
		for (size_t k = 0; k < count; ++k)
			if (weights[k] > 0)
			{
				a.src[ac] = unsigned(k);
				a.weight[ac] = weights[k];
				ac++;
			}
		if (ac == 0)
			return -1;
		std::string key(reinterpret_cast<const char*>(&a), sizeof(a));
		auto it = index.find(key);
		if (it != index.end())
			return it->second;
		maps.push_back(a);
		index.emplace(key, int(maps.size()) - 1);
		return int(maps.size()) - 1;
	}
};

// The kernel descriptor of one batched mesh (device pointers); amap is patched by runBatch.
BatchDesc makeDesc(const meshoptgpu_BatchMesh& m, const unsigned int* indices, const float* positions, const float* attributes,
    const unsigned char* lock, unsigned int* out, AttrMaps& maps, int& attr_index)
{
	BatchDesc d{};
	d.indices = indices;
	d.positions = positions;
	d.out = out;
	d.index_count = unsigned(m.index_count);
	d.vertex_count = unsigned(m.vertex_count);
	d.stride_f = unsigned(m.vertex_positions_stride / 4);
	d.target_index_count = unsigned(m.target_index_count);
	d.target_error = m.target_error;
	d.options = m.options;
	d.lock = lock;
	unsigned int ac = 0;
	attr_index = m.attribute_count ? maps.add(m.attribute_weights, m.attribute_count, ac) : -1;
	d.attributes = ac ? attributes : nullptr;
	d.attr_stride_f = ac ? unsigned(m.vertex_attributes_stride / 4) : 0;
	d.ac = ac;
	d.amap = nullptr;
	return d;
}

// whether a mesh's output leaves its indices as they are, so that the call can be repeated
bool apart(const unsigned int* out, const unsigned int* indices, size_t index_count)
{
	return std::less_equal<const unsigned int*>()(out + index_count, indices) || std::less_equal<const unsigned int*>()(indices + index_count, out);
}

// Runs descs (device pointers) through the persistent kernel; results in the same order.
// attr_of[i] indexes maps.maps for descs[i] (-1: none).
// Meshes whose ids need 32 bits run in a launch of their own, beside the others': that form has no
// shared-memory path, and one such mesh in a batch would take it from all others (4,096 meshes of 384
// triangles and one of 24,100 vertices that uses 221 of them: 3.43 ms in one launch).
void runBatch(ThreadState& s, std::vector<BatchDesc>& descs, const AttrMaps& maps, const std::vector<int>& attr_of, std::vector<BatchResult>& results,
    cudaStream_t st)
{
	const size_t n = descs.size();
	results.assign(n, BatchResult{0, 0.f, 0, 0});
	s.batch_in_shared = s.batch_in_slab = 0;
	if (n == 0)
		return;
	// the wide meshes, then the others, each with the largest first so the queue's tail is short; results
	// are mapped back below
	std::vector<unsigned int> perm(n);
	size_t wide = 0;
	{
		// by eighths of a power of two: one counting pass, where a sort of 4,096 took 0.1 ms of the call
		constexpr size_t kSizes = 512;
		std::vector<unsigned short> place(n);
		size_t start[2 * kSizes + 1] = {};
		for (size_t i = 0; i < n; ++i)
		{
			const size_t v = size_t(descs[i].index_count) + 8;
			const unsigned int e = 60 - __builtin_clzll(v); // v >> e is 8 to 15
			const size_t size = size_t(e) * 8 + (v >> e) - 8;
			place[i] = (unsigned short)(kSizes - 1 - std::min(kSizes - 1, size) + (batchNarrow(descs[i]) ? kSizes : 0));
			++start[place[i] + 1];
		}
		for (size_t k = 0; k < 2 * kSizes; ++k)
			start[k + 1] += start[k];
		wide = start[kSizes];
		for (size_t i = 0; i < n; ++i)
			perm[start[place[i]]++] = (unsigned int)i;
	}
	std::vector<BatchDesc> ordered(n);
	std::vector<BatchBytes> bytes(n);
	struct Part // the meshes of one form of the kernel
	{
		size_t first, count;
		bool narrow, full;
		size_t slab, max_index_count;
		int threads;
		size_t budget;
		bool sure, repeatable;
	} parts[2] = {{0, wide, false, false, 0, 0, 0, 0, false, true}, {wide, n - wide, true, false, 0, 0, 0, 0, false, true}};
	for (Part& p : parts)
		for (size_t i = p.first; i < p.first + p.count; ++i)
		{
			ordered[i] = descs[perm[i]];
			bytes[i] = batchBytes(ordered[i], p.narrow);
			p.full = p.full || batchNeedsFull(ordered[i]);
			const BatchDesc& d = ordered[i]; // in place: its indices are its output after a launch
			p.repeatable = p.repeatable && apart(d.out, d.indices, d.index_count);
			p.slab = std::max(p.slab, bytes[i].slab);
			p.max_index_count = std::max<size_t>(p.max_index_count, ordered[i].index_count);
		}
	// a budget's dynamic shared memory: the largest mesh that fits it, with its attribute rows or without, by
	// what meshes are expected to need or (sure) by the most they can
	auto footprint = [&](const Part& p, size_t budget, bool sure) {
		size_t most = 0;
		if (p.narrow)
			for (size_t i = p.first; i < p.first + p.count; ++i)
			{
				const BatchBytes& b = bytes[i];
				const size_t all = sure ? b.slab : b.smem + b.rows;
				most = std::max(most, all <= budget ? all : (b.smem <= budget ? b.smem : size_t(0)));
			}
		return unsigned((most + 15) & ~size_t(15));
	};
	const int sms = s.sms;

	// device metadata: descriptors, results, the tickets, the attribute maps; descriptors and
	// maps go up in one copy from pinned staging
	const size_t nm = maps.maps.size();
	const size_t off_res = align256(n * sizeof(BatchDesc)), off_ticket = off_res + align256(n * sizeof(BatchResult));
	const size_t off_maps = off_ticket + 256;
	size_t meta = off_maps + align256(nm * sizeof(BatchAttr));
	char* mbase = static_cast<char*>(s.batch_meta.ensure(meta));
	BatchDesc* d_descs = reinterpret_cast<BatchDesc*>(mbase);
	BatchResult* d_res = reinterpret_cast<BatchResult*>(mbase + off_res);
	unsigned int* d_ticket = reinterpret_cast<unsigned int*>(mbase + off_ticket);
	BatchAttr* d_maps = reinterpret_cast<BatchAttr*>(mbase + off_maps);
	for (size_t i = 0; i < n; ++i)
		ordered[i].amap = attr_of[perm[i]] >= 0 ? d_maps + attr_of[perm[i]] : nullptr;
	char* hmeta = static_cast<char*>(s.batch_meta_host.ensure(meta));
	memcpy(hmeta, ordered.data(), n * sizeof(BatchDesc));
	if (nm)
		memcpy(hmeta + off_maps, maps.maps.data(), nm * sizeof(BatchAttr));
	MO_CUDA_CHECK(cudaMemcpyAsync(d_descs, hmeta, n * sizeof(BatchDesc), cudaMemcpyHostToDevice, st));
	if (nm)
		MO_CUDA_CHECK(cudaMemcpyAsync(d_maps, hmeta + off_maps, nm * sizeof(BatchAttr), cudaMemcpyHostToDevice, st));

	// a launch: shared memory per CTA, the CTAs, and each one's slab, if a mesh may need one. Where the slabs
	// would exceed the limit, shared memory is for the most that every mesh of up to kBatchSmemDefault can
	// need, which are then sure to need no slab.
	struct Plan
	{
		unsigned int smem, blocks;
		size_t slab;
	};
	auto plan = [&](const Part& p, const BatchShape& c, size_t limit) {
		Plan r{footprint(p, c.budget, c.sure), 0, 0};
		r.slab = p.slab > r.smem ? p.slab : 0;
		if (r.slab > limit && p.narrow)
		{
			for (size_t i = p.first; i < p.first + p.count; ++i)
				if (bytes[i].slab <= kBatchSmemDefault)
					r.smem = std::max(r.smem, unsigned((bytes[i].slab + 15) & ~size_t(15)));
			r.slab = p.slab > r.smem ? p.slab : 0;
		}
		const int per_sm = std::max(1, batchBlocksPerSM(c.threads, r.smem, p.full, p.narrow));
		size_t blocks = std::min<size_t>(size_t(per_sm) * sms, p.count);
		if (r.slab)
			blocks = std::max<size_t>(1, std::min(blocks, limit / r.slab));
		r.blocks = unsigned(blocks);
		return r;
	};
	auto launch = [&](const Part& p, int threads, const Plan& r, char* slabs, cudaStream_t on) {
		launchBatch(d_descs + p.first, unsigned(p.count), d_ticket + (p.narrow ? 1 : 0), d_res + p.first, slabs, r.slab, r.smem, r.blocks, threads, p.full, p.narrow, on);
	};
	const size_t limit = std::min(s.batch_slab_limit, kBatchSlabTotal);

	auto many = [](size_t beyond, size_t count) { return beyond > count / 16; };
	bool tuned = false;
	std::tuple<int, int, bool, bool> cls;
	for (Part& p : parts)
	{
		if (!p.count)
			continue;
		p.threads = s.batch_threads;
		p.budget = s.batch_smem ? s.batch_smem : kBatchSmemDefault;
		if (!p.narrow || (p.threads && s.batch_smem))
			continue; // the 32-bit form has one shape
		// the block size and the shared-memory budget the caller left open are autotuned per size
		// class: the first batch of a class times every candidate pair on its own meshes
		// (identical results; not with meshes simplified in place) and keeps the fastest
		cls = std::make_tuple(s.device, sizeClass(p.max_index_count), p.count > size_t(sms), p.full);
		BatchShapes shapes;
		bool known = false;
		{
			std::lock_guard<std::mutex> g(g_tuner.lock);
			auto it = g_tuner.shape.find(cls);
			if (it != g_tuner.shape.end())
				shapes = it->second, known = true;
		}
		auto trials = [&](bool sure) {
			BatchShape best = sure ? shapes.as_expected : BatchShape{p.threads ? p.threads : 256, p.budget, false};
			cudaEvent_t e0, e1;
			MO_CUDA_CHECK(cudaEventCreate(&e0));
			MO_CUDA_CHECK(cudaEventCreate(&e1));
			auto timed = [&](const BatchShape& c, bool warm) {
				const Plan r = plan(p, c, limit);
				char* slabs = r.slab ? static_cast<char*>(s.batch_slabs.ensure(r.blocks * r.slab)) : nullptr;
				if (warm)
					launch(p, c.threads, r, slabs, st);
				float least = 1e30f;
				for (int rep = 0; rep < (p.count > size_t(sms) ? 1 : 3); ++rep) // short launches: the fastest of three
				{
					MO_CUDA_CHECK(cudaEventRecord(e0, st));
					launch(p, c.threads, r, slabs, st);
					MO_CUDA_CHECK(cudaEventRecord(e1, st));
					MO_CUDA_CHECK(cudaEventSynchronize(e1));
					float ms = 0;
					MO_CUDA_CHECK(cudaEventElapsedTime(&ms, e0, e1));
					least = std::min(least, ms);
				}
				return least;
			};
			// a shape for the most a mesh can need is taken unless it is clearly the slower: it runs no setup twice
			float best_ms = sure ? 1.1f * timed(best, false) : 1e30f;
			for (int t : {128, 256, 512})
			{
				if (p.threads && t != p.threads)
					continue;
				bool warm = true; // a form's first launch also loads its code
				for (size_t b : kBatchSmemBudgets)
				{
					if ((s.batch_smem && b != s.batch_smem) || (sure && footprint(p, b, true) <= footprint(p, b, false)))
						continue;
					const BatchShape c{t, b, sure};
					const float ms = timed(c, warm);
					warm = false;
					if (ms < best_ms)
						best_ms = ms, best = c;
				}
			}
			cudaEventDestroy(e0);
			cudaEventDestroy(e1);
			return best;
		};
		// trials need meshes that a launch leaves as they are, and room for slabs: else the shape that is
		// known, or the default, which is not kept
		const bool trial = p.repeatable && p.slab <= limit;
		if (!known && !trial)
			continue;
		if (!known)
		{
			shapes.as_expected = trials(false);
			BatchResult* const seen = reinterpret_cast<BatchResult*>(hmeta + off_res) + p.first;
			MO_CUDA_CHECK(cudaMemcpyAsync(seen, d_res + p.first, p.count * sizeof(BatchResult), cudaMemcpyDeviceToHost, st));
			MO_CUDA_CHECK(cudaStreamSynchronize(st));
			shapes.last_beyond = many(std::count_if(seen, seen + p.count, [](const BatchResult& r) { return (r.status & kBatchBeyond) != 0; }), p.count);
		}
		if (shapes.last_beyond && !shapes.timed_beyond && trial)
		{
			shapes.beyond = trials(true);
			shapes.timed_beyond = true;
		}
		const BatchShape use = shapes.last_beyond && shapes.timed_beyond ? shapes.beyond : shapes.as_expected;
		p.threads = p.threads ? p.threads : use.threads;
		p.budget = s.batch_smem ? p.budget : use.budget;
		p.sure = use.sure;
		tuned = true;
		std::lock_guard<std::mutex> g(g_tuner.lock);
		g_tuner.shape[cls] = shapes;
	}

	// both parts at once, the wide one from a stream of its own
	const bool both = parts[0].count && parts[1].count;
	Plan plans[2] = {};
	size_t slab_bytes[2] = {0, 0};
	for (int q = 1; q >= 0; --q) // the narrow part's slabs, if any, leave the rest of the limit to the wide one
		if (parts[q].count)
		{
			const BatchShape c{parts[q].threads, parts[q].budget, parts[q].sure};
			const size_t share = both && q == 1 ? limit / 2 : limit - std::min(limit, slab_bytes[1]);
			plans[q] = plan(parts[q], c, share);
			slab_bytes[q] = align256(plans[q].blocks * plans[q].slab);
		}
	char* slabs = slab_bytes[0] + slab_bytes[1] ? static_cast<char*>(s.batch_slabs.ensure(slab_bytes[0] + slab_bytes[1])) : nullptr;
	if (both)
	{
		s.ensureBatchStream();
		MO_CUDA_CHECK(cudaEventRecord(s.batch_event, st));
		MO_CUDA_CHECK(cudaStreamWaitEvent(s.batch_stream, s.batch_event, 0));
	}
	try
	{
		if (parts[0].count)
			launch(parts[0], parts[0].threads, plans[0], slabs, both ? s.batch_stream : st);
		if (parts[1].count)
			launch(parts[1], parts[1].threads, plans[1], slabs + slab_bytes[0], st);
		if (both)
		{
			MO_CUDA_CHECK(cudaEventRecord(s.batch_event, s.batch_stream));
			MO_CUDA_CHECK(cudaStreamWaitEvent(st, s.batch_event, 0));
		}
	}
	catch (...)
	{
		if (both)
			cudaStreamSynchronize(s.batch_stream); // the caller's buffers are its own again when the call returns
		throw;
	}
	const BatchResult* tmp = reinterpret_cast<const BatchResult*>(hmeta + off_res);
	MO_CUDA_CHECK(cudaMemcpyAsync(hmeta + off_res, d_res, n * sizeof(BatchResult), cudaMemcpyDeviceToHost, st));
	MO_CUDA_CHECK(cudaStreamSynchronize(st));
	probe().collect();
	size_t slab = 0, beyond = 0;
	for (size_t i = 0; i < n; ++i)
	{
		const unsigned int where = tmp[i].status;
		slab += where / kBatchInSlab & 1;
		beyond += i >= wide ? where / kBatchBeyond & 1 : 0;
		BatchResult& r = results[perm[i]];
		r = tmp[i];
		r.status = where & 0xff;
	}
	s.batch_in_slab = slab;
	s.batch_in_shared = n - slab;
	if (tuned)
	{
		std::lock_guard<std::mutex> g(g_tuner.lock);
		g_tuner.shape[cls].last_beyond = many(beyond, parts[1].count);
	}
}

// argument checks of a batched mesh: those of meshopt_simplifyEdge (:2348-2357), then the
// batch kernel's option set unless the mesh may take the single-mesh path
bool smallMeshOnBatch(ThreadState& s, const MeshDesc& m, unsigned int* d_out, cudaStream_t st)
{
	if (s.timing || m.index_count == 0 || (m.options & ~kBatchOptions) || m.vertex_count >= (size_t(1) << 32))
		return false;
	meshoptgpu_BatchMesh bm{};
	bm.index_count = m.index_count;
	bm.vertex_count = m.vertex_count;
	bm.vertex_positions_stride = m.positions_stride;
	bm.target_index_count = m.target_index_count;
	bm.target_error = m.target_error;
	bm.options = m.options;
	bm.vertex_attributes_stride = m.attributes_stride;
	bm.attribute_weights = m.weights;
	bm.attribute_count = m.attribute_count;
	AttrMaps maps;
	std::vector<int> attr_of(1);
	std::vector<BatchDesc> descs{makeDesc(bm, m.indices, m.positions, m.attributes, m.lock, d_out, maps, attr_of[0])};
	std::vector<BatchResult> res;
	runBatch(s, descs, maps, attr_of, res, st);
	if (res[0].status == 2)
		throw std::invalid_argument("index out of range of vertex_count");
	if (res[0].status)
		throw std::runtime_error(res[0].status == 3 ? "collapse decision round made no progress" : "batch scratch too small");
	s.last = RunResult();
	s.last.index_count = res[0].index_count;
	s.last.result_error = res[0].result_error;
	return true;
}

// ---------------------------------------------------------------- autotuning of the single-mesh path
//
// Per size class of the mesh (its index count's bit length, and whether it has attributes), the
// first call that can be repeated (its destination does not alias its indices, no update mode,
// Prune or debug bit) times the candidates on the call's own mesh and keeps the fastest for the
// class; the results are identical whatever the choice, so the call returns the last candidate's.
// Later calls of the class take the choice. Tuned:
//  * the pass kernels' launch shape: blocks per SM, one or two;
//  * the drop-in route for meshes between kDropinBatchAlways and kDropinSingleAlways indices: the
//    batch kernel (one CTA does the whole mesh) or the single-mesh path (multi-CTA pass loop).
constexpr size_t kTuneMinIndices = 3000;       // below: the default shape (nothing to gain)
constexpr size_t kDropinBatchAlways = 3000;    // up to here drop-in calls take the batch kernel
constexpr size_t kDropinSingleAlways = 98304;  // above here the single-mesh path
constexpr size_t kDropinDefault = 15000;       // the route of calls that cannot be timed

struct ShapeTuner
{
	std::mutex lock;
	std::map<std::tuple<int, int, int>, int> shape;  // -> blocks per SM
	std::map<std::tuple<int, int, int>, bool> batch;                         // -> batch kernel faster
} g_shapes;

std::tuple<int, int, int> shapeKey(const ThreadState& s, const MeshDesc& m)
{
	return std::make_tuple(s.device, sizeClass(m.index_count), m.attribute_count ? 1 : 0);
}

bool repeatable(const ThreadState& s, const MeshDesc& m, const unsigned int* d_out)
{
	return s.autotune && !s.timing && apart(d_out, m.indices, m.index_count) &&
	       !(m.options & (kOptPrune | kOptInternalDebug | kOptInternalSolve)) && m.index_count > m.target_index_count;
}

float timedMs(cudaStream_t st, const std::function<void()>& f, int reps)
{
	cudaEvent_t e0, e1;
	MO_CUDA_CHECK(cudaEventCreate(&e0));
	MO_CUDA_CHECK(cudaEventCreate(&e1));
	float best = 1e30f;
	for (int r = 0; r < reps; ++r)
	{
		MO_CUDA_CHECK(cudaEventRecord(e0, st));
		f();
		MO_CUDA_CHECK(cudaEventRecord(e1, st));
		MO_CUDA_CHECK(cudaEventSynchronize(e1));
		float ms = 0;
		MO_CUDA_CHECK(cudaEventElapsedTime(&ms, e0, e1));
		best = std::min(best, ms);
	}
	cudaEventDestroy(e0);
	cudaEventDestroy(e1);
	return best;
}

// the single-mesh path with its size class's tuned launch shape (tuning it first if it has none)
void runSingle(ThreadState& s, const MeshDesc& m, unsigned int* d_out, cudaStream_t st)
{
	Simplifier& sp = *s.simplifier;
	if (!s.autotune)
	{
		s.last = sp.run(m, d_out, st, s.timing ? &s.times : nullptr);
		return;
	}
	const auto key = shapeKey(s, m);
	{
		std::lock_guard<std::mutex> g(g_shapes.lock);
		auto it = g_shapes.shape.find(key);
		if (it != g_shapes.shape.end())
		{
			sp.setPassShape(it->second);
			s.last = sp.run(m, d_out, st, s.timing ? &s.times : nullptr);
			return;
		}
	}
	if (!repeatable(s, m, d_out) || m.index_count < kTuneMinIndices)
	{
		sp.setPassShape(0);
		s.last = sp.run(m, d_out, st, s.timing ? &s.times : nullptr);
		return;
	}
	const int reps = 2; // the faster of two runs per candidate
	int best_bps = 1;
	float best = 1e30f;
	for (int bps = std::max(1, sp.performBlocksPerSMMax()); bps >= 1; --bps)
	{
		sp.setPassShape(bps);
		const float ms = timedMs(st, [&]() { s.last = sp.run(m, d_out, st); }, reps);
		if (ms < best)
			best = ms, best_bps = bps;
	}
	sp.setPassShape(best_bps);
	std::lock_guard<std::mutex> g(g_shapes.lock);
	g_shapes.shape[key] = best_bps;
}

size_t singlePathAbove(const ThreadState& s)
{
	if (s.dropin_batch_limit != ~size_t(0))
		return s.dropin_batch_limit;
	return s.autotune ? kDropinSingleAlways : kDropinDefault;
}

void routeAndRun(ThreadState& s, const MeshDesc& m, unsigned int* d_out, cudaStream_t st, bool allow_batch)
{
	const bool batchable = allow_batch && !s.timing && m.index_count && !(m.options & ~kBatchOptions) && m.vertex_count < (size_t(1) << 32);
	if (!batchable)
	{
		runSingle(s, m, d_out, st);
		return;
	}
	if (s.dropin_batch_limit != ~size_t(0) || !s.autotune)
	{
		// a fixed limit: the caller's (meshoptgpu_setDropinBatchLimit), or the default
		const size_t limit = s.dropin_batch_limit != ~size_t(0) ? s.dropin_batch_limit : kDropinDefault;
		if (m.index_count > limit || !smallMeshOnBatch(s, m, d_out, st))
			runSingle(s, m, d_out, st);
		return;
	}
	if (m.index_count <= kDropinBatchAlways && smallMeshOnBatch(s, m, d_out, st))
		return;
	if (m.index_count > kDropinSingleAlways)
	{
		runSingle(s, m, d_out, st);
		return;
	}
	const auto key = shapeKey(s, m);
	int route = -1; // 1: batch kernel, 0: single-mesh path
	{
		std::lock_guard<std::mutex> g(g_shapes.lock);
		auto it = g_shapes.batch.find(key);
		if (it != g_shapes.batch.end())
			route = it->second ? 1 : 0;
	}
	if (route < 0 && !repeatable(s, m, d_out))
		route = m.index_count <= kDropinDefault ? 1 : 0;
	if (route < 0)
	{
		// each route once untimed (its own first-call tuning), then each timed
		smallMeshOnBatch(s, m, d_out, st);
		runSingle(s, m, d_out, st);
		const float tb = timedMs(st, [&]() { smallMeshOnBatch(s, m, d_out, st); }, 2);
		const float ts = timedMs(st, [&]() { runSingle(s, m, d_out, st); }, 2);
		std::lock_guard<std::mutex> g(g_shapes.lock);
		g_shapes.batch[key] = tb < ts;
		return; // d_out and s.last hold the single-mesh path's result, identical to the batch kernel's
	}
	if (route == 1 && smallMeshOnBatch(s, m, d_out, st))
		return;
	runSingle(s, m, d_out, st);
}

std::string checkBatchMesh(const meshoptgpu_BatchMesh& m, bool any_option = false)
{
	if (m.attribute_count && (!m.vertex_attributes || !m.attribute_weights))
		return "vertex_attributes and attribute_weights are required when attribute_count > 0";
	std::string bad = checkArgs(m.index_count, m.vertex_positions_stride, m.target_index_count, m.target_error, m.vertex_attributes_stride,
	    m.attribute_weights, m.attribute_count, m.options);
	if (!bad.empty())
		return bad;
	if (!any_option && (m.options & ~kBatchOptions))
		return "batched meshes support every option but Prune and InternalDebug";
	if (m.index_count >= (size_t(1) << 32) || m.vertex_count >= (size_t(1) << 32))
		return "batched meshes must have fewer than 2^32 indices and vertices";
	return std::string();
}

int batchCheckStatus(const meshoptgpu_BatchMesh& m, bool any_option = false)
{
	return (m.options & ~(any_option ? kSupportedOptions : kBatchOptions)) ? meshoptgpu_StatusUnsupported : meshoptgpu_StatusInvalidArgument;
}

int finishBatch(const std::vector<BatchResult>& res, size_t* counts, float* errors)
{
	int status = meshoptgpu_StatusOk;
	for (size_t i = 0; i < res.size(); ++i)
	{
		if (counts)
			counts[i] = res[i].index_count;
		if (errors)
			errors[i] = res[i].result_error;
		if (res[i].status)
			status = res[i].status >= 3 ? meshoptgpu_StatusCudaError : meshoptgpu_StatusInvalidArgument;
	}
	if (status == meshoptgpu_StatusInvalidArgument)
		setStatus(status, "a batched mesh has an index out of range of its vertex_count");
	else if (status != meshoptgpu_StatusOk)
		setStatus(status, "a batched mesh's decision round made no progress, or its scratch was too small");
	else
		setStatus(meshoptgpu_StatusOk, "");
	return status;
}

// ---------------------------------------------------------------- serving

struct ServerRequest
{
	BatchDesc desc;
	std::vector<float> weights; // attribute weights, copied at submission
	size_t index_count = 0, vertex_count = 0;
	size_t reserve = 0, slab = 0;
	std::chrono::steady_clock::time_point submitted, completed;
	bool done = false;
	int status = meshoptgpu_StatusOk;
	size_t result_count = 0;
	float result_error = 0.f;
};

struct ServerImpl
{
	meshoptgpu_ServerConfig cfg;
	int device = 0;
	int sms = 1;
	std::mutex m;
	// One waiting worker is woken for a request, and wakes the next while requests are left: all of them
	// for each took longer than the submission (2,000 requests of 512 triangles from one thread, whose
	// batches are shorter than a round of wake-ups: 33 ms, 7.6 with one)
	std::condition_variable cv_small, cv_large, cv_done;
	std::deque<ServerRequest*> small_q, large_q;
	std::vector<std::unique_ptr<ServerRequest>> reqs; // index = ticket
	size_t reserved = 0, peak_reserved = 0;
	unsigned long long completed = 0, batches = 0, singles = 0, inflight = 0, peak_inflight = 0;
	bool stop = false;
	std::vector<std::thread> threads;

	void wake() // with the lock held
	{
		if (!small_q.empty())
			cv_small.notify_one();
		if (!large_q.empty())
			cv_large.notify_one();
	}
};

const size_t kServerBudgetDefault = size_t(40) << 30;

// device bytes a request holds while it runs on the batch path: a slab, or for a mesh that shared memory
// holds whatever it needs, no more than its share of the batch's descriptors and results
size_t batchReserve(size_t slab)
{
	return slab <= kBatchSmemDefault ? 4096 : slab;
}

void publish(ServerImpl& S, std::vector<ServerRequest*>& done_reqs, size_t release)
{
	std::lock_guard<std::mutex> g(S.m);
	auto now = std::chrono::steady_clock::now();
	for (ServerRequest* r : done_reqs)
	{
		r->done = true;
		r->completed = now;
	}
	S.completed += done_reqs.size();
	S.inflight -= done_reqs.size();
	S.reserved -= release;
	S.cv_done.notify_all();
	S.wake();
}

void batchWorker(ServerImpl* S)
{
	cudaSetDevice(S->device);
	ThreadState& ts = state();
	ts.batch_threads = S->cfg.batch_threads;
	for (;;)
	{
		std::vector<ServerRequest*> take;
		size_t reserve = 0;
		{
			std::unique_lock<std::mutex> lk(S->m);
			S->cv_small.wait(lk, [&] {
				if (S->stop)
					return true;
				return !S->small_q.empty() && S->reserved + S->small_q.front()->reserve <= S->cfg.memory_budget;
			});
			if (S->stop && S->small_q.empty())
				return;
			// continuous batching: everything that arrived since this worker last launched, in
			// arrival order, while the memory budget and the batch limit allow
			size_t least = 0, most = 0; // a CTA's slab: where shared memory may be too small, and for all
			while (!S->small_q.empty() && take.size() < size_t(S->cfg.max_batch))
			{
				ServerRequest* r = S->small_q.front();
				const size_t nl = std::max(least, r->slab <= kBatchSmemDefault ? size_t(0) : r->slab);
				const size_t blocks = std::min<size_t>(take.size() + 1, size_t(S->sms) * 4);
				if (S->reserved + blocks * nl + 4096 * (take.size() + 1) > S->cfg.memory_budget && !take.empty())
					break;
				least = nl;
				most = std::max(most, r->slab);
				take.push_back(r);
				S->small_q.pop_front();
			}
			// slabs for all where there is room: shared memory can then be sized by what meshes are expected
			// to need, for more CTAs per SM
			const size_t blocks = std::min<size_t>(take.size(), size_t(S->sms) * 4), fixed = 4096 * take.size();
			ts.batch_slab_limit = blocks * (S->reserved + blocks * most + fixed <= S->cfg.memory_budget ? most : least);
			reserve = ts.batch_slab_limit + fixed;
			S->reserved += reserve;
			S->peak_reserved = std::max(S->peak_reserved, S->reserved);
			S->inflight += take.size();
			S->peak_inflight = std::max(S->peak_inflight, S->inflight);
			S->batches++;
			S->wake();
		}
		std::vector<BatchDesc> descs(take.size());
		std::vector<int> attr_of(take.size(), -1);
		AttrMaps maps;
		for (size_t i = 0; i < take.size(); ++i)
		{
			descs[i] = take[i]->desc;
			unsigned int ac = 0;
			if (!take[i]->weights.empty())
				attr_of[i] = maps.add(take[i]->weights.data(), take[i]->weights.size(), ac);
		}
		std::vector<BatchResult> res;
		try
		{
			ts.ensure();
			runBatch(ts, descs, maps, attr_of, res, ts.stream);
			for (size_t i = 0; i < take.size(); ++i)
			{
				take[i]->result_count = res[i].index_count;
				take[i]->result_error = res[i].result_error;
				take[i]->status = res[i].status ? meshoptgpu_StatusInvalidArgument : meshoptgpu_StatusOk;
			}
		}
		catch (const std::exception& e)
		{
			for (ServerRequest* r : take)
				r->status = statusOf(e);
			fprintf(stderr, "meshopt_gb300: server batch failed: %s\n", e.what());
		}
		publish(*S, take, reserve);
	}
}

void largeWorker(ServerImpl* S)
{
	cudaSetDevice(S->device);
	ThreadState& ts = state();
	try
	{
		ts.ensure();
		Tuning t = ts.simplifier->tuning();
		t.perform_grid_cap = S->cfg.perform_blocks;
		ts.simplifier->setTuning(t);
	}
	catch (const std::exception& e)
	{
		fprintf(stderr, "meshopt_gb300: server worker setup failed: %s\n", e.what());
	}
	for (;;)
	{
		ServerRequest* r = nullptr;
		{
			std::unique_lock<std::mutex> lk(S->m);
			S->cv_large.wait(lk, [&] {
				if (S->stop)
					return true;
				return !S->large_q.empty() && S->reserved + S->large_q.front()->reserve <= S->cfg.memory_budget;
			});
			if (S->stop && S->large_q.empty())
				return;
			r = S->large_q.front();
			S->large_q.pop_front();
			S->reserved += r->reserve;
			S->peak_reserved = std::max(S->peak_reserved, S->reserved);
			S->inflight++;
			S->peak_inflight = std::max(S->peak_inflight, S->inflight);
			S->singles++;
			S->wake();
		}
		try
		{
			ts.ensure();
			MeshDesc m;
			m.indices = r->desc.indices;
			m.index_count = r->index_count;
			m.positions = r->desc.positions;
			m.vertex_count = r->vertex_count;
			m.positions_stride = size_t(r->desc.stride_f) * 4;
			m.target_index_count = r->desc.target_index_count;
			m.target_error = r->desc.target_error;
			m.options = r->desc.options;
			m.lock = r->desc.lock;
			if (!r->weights.empty())
			{
				m.attributes = r->desc.attributes;
				m.attributes_stride = size_t(r->desc.attr_stride_f) * 4;
				m.weights = r->weights.data();
				m.attribute_count = r->weights.size();
			}
			RunResult rr = ts.simplifier->run(m, r->desc.out, ts.stream);
			r->result_count = rr.index_count;
			r->result_error = rr.result_error;
			r->status = meshoptgpu_StatusOk;
		}
		catch (const std::exception& e)
		{
			r->status = statusOf(e);
			fprintf(stderr, "meshopt_gb300: server request failed: %s\n", e.what());
		}
		std::vector<ServerRequest*> one{r};
		publish(*S, one, r->reserve);
	}
}

} // namespace

extern "C" {

size_t meshopt_simplifyWithUpdate(unsigned int* indices, size_t index_count, float* vertex_positions, size_t vertex_count, size_t vertex_positions_stride,
    float* vertex_attributes, size_t vertex_attributes_stride, const float* attribute_weights, size_t attribute_count, const unsigned char* vertex_lock,
    size_t target_index_count, float target_error, unsigned int options, float* result_error)
{
	return updateHost(indices, index_count, vertex_positions, vertex_count, vertex_positions_stride, vertex_attributes, vertex_attributes_stride,
	    attribute_weights, attribute_count, vertex_lock, target_index_count, target_error, options, result_error);
}

size_t meshoptgpu_simplifyWithUpdateDevice(unsigned int* indices, size_t index_count, float* vertex_positions, size_t vertex_count,
    size_t vertex_positions_stride, float* vertex_attributes, size_t vertex_attributes_stride, const float* attribute_weights, size_t attribute_count,
    const unsigned char* vertex_lock, size_t target_index_count, float target_error, unsigned int options, float* result_error, void* stream)
{
	std::string bad = checkArgs(index_count, vertex_positions_stride, target_index_count, target_error, vertex_attributes_stride, attribute_weights,
	    attribute_count, options);
	if (!bad.empty())
	{
		setStatus((options & ~kSupportedOptions) ? meshoptgpu_StatusUnsupported : meshoptgpu_StatusInvalidArgument, bad);
		if (result_error)
			*result_error = 0.f;
		return index_count;
	}
	try
	{
		ThreadState& s = state();
		s.ensure();
		cudaStream_t st = static_cast<cudaStream_t>(stream);
		MeshDesc m;
		m.indices = indices;
		m.index_count = index_count;
		m.positions = vertex_positions;
		m.vertex_count = vertex_count;
		m.positions_stride = vertex_positions_stride;
		m.attributes = attribute_count ? vertex_attributes : nullptr;
		m.attributes_stride = vertex_attributes_stride;
		m.weights = attribute_weights;
		m.attribute_count = attribute_count;
		m.lock = vertex_lock;
		m.target_index_count = target_index_count;
		m.target_error = target_error;
		m.options = options | kOptInternalSolve;
		m.update_positions = vertex_positions;
		m.update_attributes = attribute_count ? vertex_attributes : nullptr;
		s.last = s.simplifier->run(m, indices, st, s.timing ? &s.times : nullptr);
		MO_CUDA_CHECK(cudaStreamSynchronize(st));
		if (result_error)
			*result_error = s.last.result_error;
		setStatus(meshoptgpu_StatusOk, "");
		return s.last.index_count;
	}
	catch (const std::exception& e)
	{
		setStatus(statusOf(e), e.what());
		if (result_error)
			*result_error = 0.f;
		return index_count;
	}
}

int meshoptgpu_simplifyBatch(const meshoptgpu_BatchMesh* meshes, size_t mesh_count, size_t* result_index_counts, float* result_errors, void* stream)
{
	for (size_t i = 0; i < mesh_count; ++i)
	{
		std::string bad = checkBatchMesh(meshes[i]);
		if (!bad.empty())
		{
			int st = batchCheckStatus(meshes[i]);
			setStatus(st, "mesh " + std::to_string(i) + ": " + bad);
			return st;
		}
	}
	try
	{
		ThreadState& s = state();
		s.ensure();
		std::vector<BatchDesc> descs(mesh_count);
		std::vector<int> attr_of(mesh_count);
		AttrMaps maps;
		for (size_t i = 0; i < mesh_count; ++i)
		{
			const meshoptgpu_BatchMesh& m = meshes[i];
			descs[i] = makeDesc(m, m.indices, m.vertex_positions, m.vertex_attributes, m.vertex_lock, m.destination, maps, attr_of[i]);
		}
		std::vector<BatchResult> res;
		runBatch(s, descs, maps, attr_of, res, static_cast<cudaStream_t>(stream));
		return finishBatch(res, result_index_counts, result_errors);
	}
	catch (const std::exception& e)
	{
		setStatus(statusOf(e), e.what());
		return statusOf(e);
	}
}

int meshoptgpu_simplifyBatchHost(const meshoptgpu_BatchMesh* meshes, size_t mesh_count, size_t* result_index_counts, float* result_errors)
{
	for (size_t i = 0; i < mesh_count; ++i)
	{
		std::string bad = checkBatchMesh(meshes[i]);
		if (!bad.empty())
		{
			int st = batchCheckStatus(meshes[i]);
			setStatus(st, "mesh " + std::to_string(i) + ": " + bad);
			return st;
		}
	}
	try
	{
		ThreadState& s = state();
		s.ensure();
		// pack inputs into one pinned buffer (16-byte aligned pieces): per mesh its indices, and
		// every distinct vertex, attribute and lock array once (meshes of a sparse group share
		// them); outputs follow all inputs on the device
		size_t in_bytes = 0, out_words = 0;
		PieceTable shared(3 * mesh_count);
		std::vector<std::pair<const void*, size_t>> pieces; // (source, bytes) in pack order
		pieces.reserve(2 * mesh_count);
		auto place = [&](const void* p, size_t bytes, bool dedupe) -> size_t {
			if (!p || !bytes)
				return ~size_t(0);
			const size_t at = in_bytes;
			if (dedupe)
			{
				const size_t seen = shared.findOrInsert(p, bytes, at);
				if (seen != ~size_t(0))
					return seen;
			}
			in_bytes = (in_bytes + bytes + 15) & ~size_t(15);
			pieces.push_back({p, bytes});
			return at;
		};
		std::vector<size_t> off_idx(mesh_count), off_pos(mesh_count), off_attr(mesh_count), off_lock(mesh_count), off_out(mesh_count);
		for (size_t i = 0; i < mesh_count; ++i)
		{
			const meshoptgpu_BatchMesh& m = meshes[i];
			off_idx[i] = place(m.indices, m.index_count * 4, false);
			off_pos[i] = place(m.vertex_positions, stridedExtent(m.vertex_count, m.vertex_positions_stride, 12), true);
			off_attr[i] = m.attribute_count ? place(m.vertex_attributes, stridedExtent(m.vertex_count, m.vertex_attributes_stride, m.attribute_count * 4), true)
			                                : ~size_t(0);
			off_lock[i] = place(m.vertex_lock, m.vertex_count, true);
			off_out[i] = out_words;
			out_words += m.index_count;
		}
		char* h = static_cast<char*>(s.batch_host.ensure(in_bytes + 16));
		char* d = static_cast<char*>(s.batch_io.ensure(align256(in_bytes) + out_words * 4 + 256));
		unsigned int* d_out = reinterpret_cast<unsigned int*>(d + align256(in_bytes));
		cudaStream_t st = s.stream;
		{
			// packed and uploaded in chunks of about a quarter of the bytes (4 MiB at least): the
			// upload of one chunk runs while the next one is packed
			std::vector<HostCopy> copies;
			copies.reserve(pieces.size());
			size_t at = 0;
			for (auto& pc : pieces)
			{
				copies.push_back(HostCopy{h + at, pc.first, pc.second});
				at = (at + pc.second + 15) & ~size_t(15);
			}
			const size_t chunk = std::max<size_t>(size_t(4) << 20, in_bytes / 4);
			for (size_t b = 0; b < copies.size();)
			{
				size_t e = b, bytes = 0;
				while (e < copies.size() && (e == b || bytes < chunk))
					bytes += copies[e++].bytes;
				parallelCopies(copies.data() + b, e - b);
				const size_t lo = static_cast<size_t>(static_cast<char*>(copies[b].dst) - h);
				const size_t hi = e < copies.size() ? static_cast<size_t>(static_cast<char*>(copies[e].dst) - h) : in_bytes;
				MO_CUDA_CHECK(cudaMemcpyAsync(d + lo, h + lo, hi - lo, cudaMemcpyHostToDevice, st));
				b = e;
			}
		}
		std::vector<BatchDesc> descs(mesh_count);
		std::vector<int> attr_of(mesh_count);
		AttrMaps maps;
		auto at = [&](size_t off) { return off == ~size_t(0) ? nullptr : d + off; };
		for (size_t i = 0; i < mesh_count; ++i)
			descs[i] = makeDesc(meshes[i], reinterpret_cast<const unsigned int*>(at(off_idx[i])), reinterpret_cast<const float*>(at(off_pos[i])),
			    reinterpret_cast<const float*>(at(off_attr[i])), reinterpret_cast<const unsigned char*>(at(off_lock[i])), d_out + off_out[i], maps,
			    attr_of[i]);
		std::vector<BatchResult> res;
		runBatch(s, descs, maps, attr_of, res, st);
		// results back in one copy (the packed outputs), then scattered to the callers' buffers
		unsigned int* hout = static_cast<unsigned int*>(s.batch_host.ensure(std::max(in_bytes + 16, out_words * 4 + 16)));
		MO_CUDA_CHECK(cudaMemcpyAsync(hout, d_out, out_words * 4, cudaMemcpyDeviceToHost, st));
		MO_CUDA_CHECK(cudaStreamSynchronize(st));
		std::vector<HostCopy> copies(mesh_count);
		for (size_t i = 0; i < mesh_count; ++i)
			copies[i] = HostCopy{meshes[i].destination, hout + off_out[i], size_t(res[i].index_count) * 4};
		parallelCopies(copies);
		return finishBatch(res, result_index_counts, result_errors);
	}
	catch (const std::exception& e)
	{
		setStatus(statusOf(e), e.what());
		return statusOf(e);
	}
}

int meshoptgpu_simplifyGroups(unsigned int* destination, const unsigned int* indices, const size_t* group_offsets, size_t group_count,
    const float* vertex_positions, size_t vertex_count, size_t vertex_positions_stride, const float* vertex_attributes, size_t vertex_attributes_stride,
    const float* attribute_weights, size_t attribute_count, const unsigned int* position_remap, unsigned char* locks, const unsigned char* vertex_lock,
    const size_t* target_index_counts, float target_error, unsigned int options, size_t* result_index_counts, float* result_errors, void* stream)
{
	if (!position_remap || !locks || (group_count && (!group_offsets || !target_index_counts)))
	{
		setStatus(meshoptgpu_StatusInvalidArgument, "position_remap, locks, group_offsets and target_index_counts are required");
		return meshoptgpu_StatusInvalidArgument;
	}
	std::vector<meshoptgpu_BatchMesh> meshes(group_count);
	for (size_t g = 0; g < group_count; ++g)
	{
		meshoptgpu_BatchMesh& m = meshes[g];
		m = meshoptgpu_BatchMesh{};
		if (group_offsets[g + 1] < group_offsets[g])
		{
			setStatus(meshoptgpu_StatusInvalidArgument, "group_offsets must not decrease");
			return meshoptgpu_StatusInvalidArgument;
		}
		m.indices = indices + group_offsets[g];
		m.index_count = group_offsets[g + 1] - group_offsets[g];
		m.vertex_positions = vertex_positions;
		m.vertex_count = vertex_count;
		m.vertex_positions_stride = vertex_positions_stride;
		m.target_index_count = target_index_counts[g];
		m.target_error = target_error;
		m.options = options | kOptSparse;
		m.destination = destination + group_offsets[g];
		m.vertex_attributes = vertex_attributes;
		m.vertex_attributes_stride = vertex_attributes_stride;
		m.attribute_weights = attribute_weights;
		m.attribute_count = attribute_count;
		m.vertex_lock = locks;
		std::string bad = checkBatchMesh(m);
		if (!bad.empty())
		{
			int st = batchCheckStatus(m);
			setStatus(st, "group " + std::to_string(g) + ": " + bad);
			return st;
		}
	}
	try
	{
		ThreadState& s = state();
		s.ensure();
		cudaStream_t st = static_cast<cudaStream_t>(stream);
		// offsets (device, 64-bit), the claim tables, the error word
		const size_t lock_bytes = groupLockScratchBytes(vertex_count, group_count);
		char* base = static_cast<char*>(s.group_scratch.ensure(lock_bytes + (group_count + 1) * 8 + 512));
		unsigned long long* d_off = reinterpret_cast<unsigned long long*>(base + lock_bytes);
		unsigned int* d_bad = reinterpret_cast<unsigned int*>(base + lock_bytes + ((group_count + 1) * 8 + 255) / 256 * 256);
		std::vector<unsigned long long> off(group_offsets, group_offsets + group_count + 1);
		unsigned long long* h_off = static_cast<unsigned long long*>(s.batch_host.ensure(off.size() * 8));
		memcpy(h_off, off.data(), off.size() * 8);
		MO_CUDA_CHECK(cudaMemcpyAsync(d_off, h_off, off.size() * 8, cudaMemcpyHostToDevice, st));
		groupLocks(locks, indices, d_off, group_count, position_remap, vertex_lock, vertex_count, base, d_bad, st);
		std::vector<BatchDesc> descs(group_count);
		std::vector<int> attr_of(group_count);
		AttrMaps maps;
		for (size_t g = 0; g < group_count; ++g)
		{
			const meshoptgpu_BatchMesh& m = meshes[g];
			descs[g] = makeDesc(m, m.indices, m.vertex_positions, m.vertex_attributes, m.vertex_lock, m.destination, maps, attr_of[g]);
		}
		std::vector<BatchResult> res;
		runBatch(s, descs, maps, attr_of, res, st);
		unsigned int hbad = 0;
		MO_CUDA_CHECK(cudaMemcpyAsync(h_off, d_bad, 4, cudaMemcpyDeviceToHost, st));
		MO_CUDA_CHECK(cudaStreamSynchronize(st));
		memcpy(&hbad, h_off, 4);
		if (hbad)
		{
			setStatus(meshoptgpu_StatusInvalidArgument, "an index or a position_remap entry is out of range of vertex_count");
			return meshoptgpu_StatusInvalidArgument;
		}
		return finishBatch(res, result_index_counts, result_errors);
	}
	catch (const std::exception& e)
	{
		setStatus(statusOf(e), e.what());
		return statusOf(e);
	}
}

int meshoptgpu_buildMeshletsFlexGroups(unsigned int* meshlets, unsigned int* meshlet_vertices, unsigned char* meshlet_triangles,
    const size_t* meshlet_offsets, size_t* meshlet_counts, const unsigned int* indices, const size_t* group_offsets, size_t group_count,
    const float* vertex_positions, size_t vertex_count, size_t vertex_positions_stride, size_t max_vertices, size_t min_triangles, size_t max_triangles,
    float cone_weight, float split_factor, int optimize_level, void* stream)
{
	// the reference's argument checks (src/clusterizer.cpp:1039-1049), as errors
	std::string bad;
	if (group_count && (!group_offsets || !meshlet_offsets || !meshlet_counts))
		bad = "group_offsets, meshlet_offsets and meshlet_counts are required";
	else if (vertex_positions_stride < 12 || vertex_positions_stride > 256 || vertex_positions_stride % 4)
		bad = "vertex_positions_stride must be 12..256 and a multiple of 4";
	else if (max_vertices < 3 || max_vertices > 256)
		bad = "max_vertices must be 3..256";
	else if (min_triangles < 1 || min_triangles > max_triangles || max_triangles > 512)
		bad = "need 1 <= min_triangles <= max_triangles <= 512";
	else if (!(cone_weight >= 0.f && cone_weight <= 1.f))
		bad = "cone_weight must be in [0, 1]";
	else if (!(split_factor >= 0.f))
		bad = "split_factor must be >= 0";
	else if (vertex_count >= (size_t(1) << 32))
		bad = "vertex_count must be below 2^32";
	else if (optimize_level < -1 || optimize_level > 9)
		bad = "optimize_level must be -1 (none) or 0..9";
	for (size_t g = 0; bad.empty() && g < group_count; ++g)
	{
		const size_t n = group_offsets[g + 1] - group_offsets[g];
		if (group_offsets[g + 1] < group_offsets[g] || n % 3)
			bad = "group " + std::to_string(g) + ": index counts must be multiples of 3 and offsets must not decrease";
		else if (meshlet_offsets[g + 1] < meshlet_offsets[g] || meshlet_offsets[g + 1] - meshlet_offsets[g] < meshletBound(n, max_vertices, min_triangles))
			bad = "group " + std::to_string(g) + ": fewer meshlet rows than meshopt_buildMeshletsBound(index_count, max_vertices, min_triangles)";
		else if (n >= (size_t(1) << 31))
			bad = "group " + std::to_string(g) + ": index count must be below 2^31";
		else if (n && (!vertex_count || !vertex_positions)) // the kernel reads vertex 0 in the place of a bad index
			bad = "an index is out of range of vertex_count";
	}
	if (!bad.empty())
	{
		setStatus(meshoptgpu_StatusInvalidArgument, bad);
		return meshoptgpu_StatusInvalidArgument;
	}
	if (!group_count)
	{
		setStatus(meshoptgpu_StatusOk, "");
		return meshoptgpu_StatusOk;
	}
	try
	{
		ThreadState& s = state();
		s.ensure();
		cudaStream_t st = static_cast<cudaStream_t>(stream);
		// per group: index offsets, meshlet rows, scratch offsets (64-bit, device); counts and the error word
		const size_t G = group_count;
		std::vector<unsigned long long> host((G + 1) * 3, 0);
		unsigned long long scratch = 0;
		unsigned int max_index_count = 0;
		for (size_t g = 0; g <= G; ++g)
		{
			host[g] = group_offsets[g];
			host[(G + 1) + g] = meshlet_offsets[g];
			host[2 * (G + 1) + g] = scratch;
			if (g < G)
			{
				scratch += meshletScratchBytes(group_offsets[g + 1] - group_offsets[g]);
				max_index_count = std::max(max_index_count, unsigned(group_offsets[g + 1] - group_offsets[g]));
			}
		}
		const size_t meta = ((host.size() * 8 + 255) / 256) * 256, words = ((G + 1) * 4 + 255) / 256 * 256;
		char* base = static_cast<char*>(s.meshlet_scratch.ensure(meta + words + scratch + 256));
		unsigned long long* d_meta = reinterpret_cast<unsigned long long*>(base);
		unsigned int* d_counts = reinterpret_cast<unsigned int*>(base + meta);
		unsigned int* d_err = d_counts + G;
		char* d_scratch = base + meta + words;
		void* h = s.batch_host.ensure(host.size() * 8 + (G + 1) * 4);
		memcpy(h, host.data(), host.size() * 8);
		MO_CUDA_CHECK(cudaMemcpyAsync(d_meta, h, host.size() * 8, cudaMemcpyHostToDevice, st));
		MO_CUDA_CHECK(cudaMemsetAsync(d_err, 0, 4, st));
		MeshletBatch b;
		b.indices = indices;
		b.offsets = d_meta;
		b.groups = unsigned(G);
		b.positions = vertex_positions;
		b.stride_f = unsigned(vertex_positions_stride / 4);
		b.vertex_count = unsigned(vertex_count);
		b.max_vertices = unsigned(max_vertices);
		b.min_triangles = unsigned(min_triangles);
		b.max_triangles = unsigned(max_triangles);
		b.cone_weight = cone_weight;
		b.split_factor = split_factor;
		b.meshlets = meshlets;
		b.meshlet_base = d_meta + (G + 1);
		b.mverts = meshlet_vertices;
		b.mtris = meshlet_triangles;
		b.counts = d_counts;
		b.scratch = d_scratch;
		b.scratch_off = d_meta + 2 * (G + 1);
		b.error = d_err;
		b.max_index_count = max_index_count;
		b.optimize_level = optimize_level;
		b.rows = meshlet_offsets[G];
		buildMeshletsBatch(b, st);
		unsigned int* hc = reinterpret_cast<unsigned int*>(static_cast<char*>(h) + host.size() * 8);
		MO_CUDA_CHECK(cudaMemcpyAsync(hc, d_counts, (G + 1) * 4, cudaMemcpyDeviceToHost, st));
		MO_CUDA_CHECK(cudaStreamSynchronize(st));
		if (hc[G] & 1u)
		{
			setStatus(meshoptgpu_StatusInvalidArgument, "an index is out of range of vertex_count");
			return meshoptgpu_StatusInvalidArgument;
		}
		if (hc[G])
		{
			setStatus(meshoptgpu_StatusInternal, "meshlet construction exceeded a bound it keeps (tree depth or output size)");
			return meshoptgpu_StatusInternal;
		}
		for (size_t g = 0; g < G; ++g)
			meshlet_counts[g] = hc[g];
		setStatus(meshoptgpu_StatusOk, "");
		return meshoptgpu_StatusOk;
	}
	catch (const std::exception& e)
	{
		setStatus(statusOf(e), e.what());
		return statusOf(e);
	}
}

size_t meshoptgpu_optimizeVertexFetchRemapDevice(unsigned int* destination, const unsigned int* indices, size_t index_count, size_t vertex_count,
    void* stream)
{
	try
	{
		if (vertex_count && !destination)
			throw std::invalid_argument("destination is required");
		if (vertex_count >= (size_t(1) << 32) || index_count >= (size_t(1) << 32))
			throw std::invalid_argument("counts must be below 2^32");
		ThreadState& s = state();
		cudaStream_t st = static_cast<cudaStream_t>(stream);
		unsigned int* scratch = static_cast<unsigned int*>(s.compact_scratch.ensure((vertexOrderScratchWords(index_count, vertex_count) + 64) * 4));
		unsigned int* counters = scratch + vertexOrderScratchWords(index_count, vertex_count);
		vertexOrder(destination, true, indices, index_count, vertex_count, scratch, counters, st);
		const unsigned int used = takeOrderCount(counters, st);
		setStatus(meshoptgpu_StatusOk, "");
		return used;
	}
	catch (const std::exception& e)
	{
		setStatus(statusOf(e), e.what());
		return 0;
	}
}

size_t meshoptgpu_optimizeVertexFetchDevice(void* destination, unsigned int* indices, size_t index_count, const void* vertices, size_t vertex_count,
    size_t vertex_size, void* stream)
{
	try
	{
		if (vertex_size == 0 || vertex_size > 256)
			throw std::invalid_argument("vertex_size must be in [1, 256]");
		if (vertex_count >= (size_t(1) << 32) || index_count >= (size_t(1) << 32))
			throw std::invalid_argument("counts must be below 2^32");
		ThreadState& s = state();
		cudaStream_t st = static_cast<cudaStream_t>(stream);
		// scratch: the order table, the vertex-order scratch, counters, and for an in-place call
		// a copy of the vertices
		const size_t ow = (vertex_count + 63) & ~size_t(63), sw = vertexOrderScratchWords(index_count, vertex_count);
		const size_t copy_bytes = destination == vertices ? vertex_count * vertex_size : 0;
		char* base = static_cast<char*>(s.compact_scratch.ensure((ow + sw + 64) * 4 + copy_bytes + 256));
		unsigned int* order = reinterpret_cast<unsigned int*>(base);
		unsigned int* scratch = order + ow;
		unsigned int* counters = scratch + sw;
		const void* src = vertices;
		if (copy_bytes)
		{
			void* copy = base + (ow + sw + 64) * 4;
			MO_CUDA_CHECK(cudaMemcpyAsync(copy, vertices, copy_bytes, cudaMemcpyDeviceToDevice, st));
			src = copy;
		}
		// the moves are queued behind the order and do nothing if an index is bad, so the call waits once
		vertexOrder(order, false, indices, index_count, vertex_count, scratch, counters, st);
		compactVertices(destination, src, vertex_count, vertex_size, indices, index_count, order, vertexOrderList(scratch, vertex_count), counters, st);
		const unsigned int used = takeOrderCount(counters, st);
		setStatus(meshoptgpu_StatusOk, "");
		return used;
	}
	catch (const std::exception& e)
	{
		setStatus(statusOf(e), e.what());
		return 0;
	}
}

int meshoptgpu_generatePositionRemapDevice(unsigned int* destination, const float* vertex_positions, size_t vertex_count, size_t vertex_positions_stride,
    void* stream)
{
	try
	{
		if (vertex_positions_stride < 12 || vertex_positions_stride > 256 || vertex_positions_stride % 4 != 0)
			throw std::invalid_argument("vertex_positions_stride must be in [12, 256] and a multiple of 4");
		if (vertex_count >= (size_t(1) << 32))
			throw std::invalid_argument("vertex_count must be below 2^32");
		ThreadState& s = state();
		cudaStream_t st = static_cast<cudaStream_t>(stream);
		const size_t sw = positionRemapScratchWords(vertex_count);
		unsigned int* scratch = static_cast<unsigned int*>(s.compact_scratch.ensure((sw + 64) * 4));
		unsigned int* counters = scratch + sw;
		positionRemap(destination, vertex_positions, vertex_count, vertex_positions_stride / 4, scratch, counters, st);
		unsigned int h[2];
		MO_CUDA_CHECK(cudaMemcpyAsync(h, counters, sizeof(h), cudaMemcpyDeviceToHost, st));
		MO_CUDA_CHECK(cudaStreamSynchronize(st));
		probe().collect();
		if (h[1])
			throw std::runtime_error("position table overflow");
		setStatus(meshoptgpu_StatusOk, "");
		return meshoptgpu_StatusOk;
	}
	catch (const std::exception& e)
	{
		setStatus(statusOf(e), e.what());
		return statusOf(e);
	}
}

meshoptgpu_Server* meshoptgpu_serverCreate(const meshoptgpu_ServerConfig* config)
{
	try
	{
		std::unique_ptr<ServerImpl> S(new ServerImpl());
		meshoptgpu_ServerConfig c = config ? *config : meshoptgpu_ServerConfig{};
		c.memory_budget = c.memory_budget ? c.memory_budget : kServerBudgetDefault;
		c.batch_workers = c.batch_workers > 0 ? c.batch_workers : 8;
		c.large_workers = c.large_workers > 0 ? c.large_workers : 8;
		c.large_index_count = c.large_index_count ? c.large_index_count : 30000;
		c.max_batch = c.max_batch > 0 ? c.max_batch : 2048;
		c.batch_threads = (c.batch_threads == 128 || c.batch_threads == 256 || c.batch_threads == 512) ? c.batch_threads : 256;
		c.perform_blocks = c.plain ? 0 : (c.perform_blocks > 0 ? c.perform_blocks : 64);
		S->cfg = c;
		MO_CUDA_CHECK(cudaGetDevice(&S->device));
		MO_CUDA_CHECK(cudaDeviceGetAttribute(&S->sms, cudaDevAttrMultiProcessorCount, S->device));
		ServerImpl* raw = S.get();
		if (!c.plain)
			for (int i = 0; i < c.batch_workers; ++i)
				S->threads.emplace_back(batchWorker, raw);
		for (int i = 0; i < (c.plain ? 1 : c.large_workers); ++i)
			S->threads.emplace_back(largeWorker, raw);
		setStatus(meshoptgpu_StatusOk, "");
		return reinterpret_cast<meshoptgpu_Server*>(S.release());
	}
	catch (const std::exception& e)
	{
		setStatus(statusOf(e), e.what());
		return nullptr;
	}
}

void meshoptgpu_serverDestroy(meshoptgpu_Server* server)
{
	if (!server)
		return;
	ServerImpl* S = reinterpret_cast<ServerImpl*>(server);
	{
		std::unique_lock<std::mutex> lk(S->m);
		S->cv_done.wait(lk, [&] { return S->small_q.empty() && S->large_q.empty() && S->inflight == 0; });
		S->stop = true;
		S->cv_small.notify_all();
		S->cv_large.notify_all();
	}
	for (std::thread& t : S->threads)
		t.join();
	delete S;
}

long long meshoptgpu_serverSubmit(meshoptgpu_Server* server, const meshoptgpu_BatchMesh* mesh)
{
	if (!server || !mesh)
		return -meshoptgpu_StatusInvalidArgument;
	ServerImpl* S = reinterpret_cast<ServerImpl*>(server);
	std::string bad = checkBatchMesh(*mesh, true);
	if (!bad.empty())
	{
		int st = batchCheckStatus(*mesh, true);
		setStatus(st, bad);
		return -st;
	}
	std::unique_ptr<ServerRequest> r(new ServerRequest());
	AttrMaps unused;
	int attr_index = -1;
	r->desc = makeDesc(*mesh, mesh->indices, mesh->vertex_positions, mesh->vertex_attributes, mesh->vertex_lock, mesh->destination, unused, attr_index);
	if (r->desc.ac)
		r->weights.assign(mesh->attribute_weights, mesh->attribute_weights + mesh->attribute_count);
	r->index_count = mesh->index_count;
	r->vertex_count = mesh->vertex_count;
	// meshes up to large_index_count indices go to the batch kernel (one CTA per mesh, shared
	// memory or a global slab); larger ones, and the options the batch kernel does not have,
	// take the multi-CTA single-mesh path
	bool large = S->cfg.plain || mesh->index_count > S->cfg.large_index_count || (mesh->options & ~kBatchOptions);
	if (!large)
		r->slab = batchBytes(r->desc, batchNarrow(r->desc)).slab;
	r->reserve = large ? Simplifier::workspaceBytes(mesh->index_count, mesh->vertex_count, r->desc.ac) : batchReserve(r->slab);
	if (r->reserve > S->cfg.memory_budget)
	{
		setStatus(meshoptgpu_StatusOutOfMemory, "request needs more device scratch than the server's memory budget");
		return -meshoptgpu_StatusOutOfMemory;
	}
	r->submitted = std::chrono::steady_clock::now();
	std::lock_guard<std::mutex> g(S->m);
	long long ticket = (long long)S->reqs.size();
	(large ? S->large_q : S->small_q).push_back(r.get());
	S->reqs.push_back(std::move(r));
	(large ? S->cv_large : S->cv_small).notify_one();
	return ticket;
}

int meshoptgpu_serverWait(meshoptgpu_Server* server, long long ticket, size_t* result_index_count, float* result_error, double* latency_ms)
{
	if (!server)
		return meshoptgpu_StatusInvalidArgument;
	ServerImpl* S = reinterpret_cast<ServerImpl*>(server);
	std::unique_lock<std::mutex> lk(S->m);
	if (ticket < 0 || ticket >= (long long)S->reqs.size())
		return meshoptgpu_StatusInvalidArgument;
	ServerRequest* r = S->reqs[size_t(ticket)].get();
	S->cv_done.wait(lk, [&] { return r->done; });
	if (result_index_count)
		*result_index_count = r->result_count;
	if (result_error)
		*result_error = r->result_error;
	if (latency_ms)
		*latency_ms = std::chrono::duration<double, std::milli>(r->completed - r->submitted).count();
	return r->status;
}

void meshoptgpu_serverStats(meshoptgpu_Server* server, unsigned long long* out5)
{
	ServerImpl* S = reinterpret_cast<ServerImpl*>(server);
	std::lock_guard<std::mutex> g(S->m);
	out5[0] = S->completed;
	out5[1] = S->batches;
	out5[2] = S->singles;
	out5[3] = S->peak_reserved;
	out5[4] = S->peak_inflight;
}

void meshoptgpu_setBatchConfig(int threads, unsigned int smem_bytes)
{
	ThreadState& s = state();
	s.batch_threads = (threads == 128 || threads == 256 || threads == 512) ? threads : 0;
	s.batch_smem = smem_bytes;
}

void meshoptgpu_setDropinBatchLimit(size_t max_index_count)
{
	state().dropin_batch_limit = max_index_count;
}

void meshoptgpu_getLastBatchPlacement(size_t* in_shared_memory, size_t* in_global_memory)
{
	const ThreadState& s = state();
	if (in_shared_memory)
		*in_shared_memory = s.batch_in_shared;
	if (in_global_memory)
		*in_global_memory = s.batch_in_slab;
}

int meshoptgpu_setDeviceLoop(int enabled)
{
	try
	{
		ThreadState& s = state();
		s.ensure();
		Tuning t = s.simplifier->tuning();
		t.device_loop = enabled != 0;
		s.simplifier->setTuning(t);
		return meshoptgpu_StatusOk;
	}
	catch (const std::exception& e)
	{
		setStatus(statusOf(e), e.what());
		return statusOf(e);
	}
}

int meshoptgpu_probeBarrierWait(int once, unsigned int blocks, unsigned int wait_limit, unsigned int* timed_out)
{
	try
	{
		ThreadState& s = state();
		s.ensure();
		if (blocks < 2 || blocks > coopScanCapacity() || wait_limit == 0 || wait_limit > (1u << 20) || !timed_out)
			throw std::invalid_argument("probeBarrierWait: blocks must be 2..resident blocks, wait_limit 1..2^20, timed_out non-null");
		*timed_out = probeBarrierWait(once == 2 ? 2 : once != 0, blocks, wait_limit, s.stream);
		setStatus(meshoptgpu_StatusOk, "");
		return meshoptgpu_StatusOk;
	}
	catch (const std::exception& e)
	{
		setStatus(statusOf(e), e.what());
		return statusOf(e);
	}
}

int meshoptgpu_getBatchThreads(void)
{
	ThreadState& s = state();
	if (s.batch_threads)
		return s.batch_threads;
	std::lock_guard<std::mutex> g(g_tuner.lock);
	return g_tuner.shape.empty() ? 0 : g_tuner.shape.rbegin()->second.as_expected.threads;
}

int meshoptgpu_getTuning(size_t index_count, size_t attribute_count, int* out4)
{
	if (!out4)
		return 0;
	int dev = 0;
	cudaGetDevice(&dev);
	const auto key = std::make_tuple(dev, sizeClass(index_count), attribute_count ? 1 : 0);
	int found = 0;
	out4[0] = out4[1] = 0;
	out4[2] = -1;
	out4[3] = 0;
	{
		std::lock_guard<std::mutex> g(g_shapes.lock);
		auto it = g_shapes.shape.find(key);
		if (it != g_shapes.shape.end())
		{
			out4[0] = it->second;
			out4[1] = 0;
			found = 1;
		}
		auto jt = g_shapes.batch.find(key);
		if (jt != g_shapes.batch.end())
			out4[2] = jt->second ? 1 : 0;
	}
	{
		std::lock_guard<std::mutex> g(g_tuner.lock);
		for (const auto& it : g_tuner.shape) // in order of the size class
			if (std::get<0>(it.first) == dev)
				out4[3] = int(it.second.as_expected.budget / 1024);
	}
	return found;
}

} // extern "C"

namespace
{

} // namespace

extern "C" {

size_t meshopt_simplify(unsigned int* destination, const unsigned int* indices, size_t index_count, const float* vertex_positions, size_t vertex_count,
    size_t vertex_positions_stride, size_t target_index_count, float target_error, unsigned int options, float* result_error)
{
	return simplifyHost(destination, indices, index_count, vertex_positions, vertex_count, vertex_positions_stride, nullptr, 0, nullptr, 0, nullptr,
	    target_index_count, target_error, options, result_error);
}

size_t meshopt_simplifyWithAttributes(unsigned int* destination, const unsigned int* indices, size_t index_count, const float* vertex_positions,
    size_t vertex_count, size_t vertex_positions_stride, const float* vertex_attributes, size_t vertex_attributes_stride, const float* attribute_weights,
    size_t attribute_count, const unsigned char* vertex_lock, size_t target_index_count, float target_error, unsigned int options, float* result_error)
{
	return simplifyHost(destination, indices, index_count, vertex_positions, vertex_count, vertex_positions_stride, vertex_attributes,
	    vertex_attributes_stride, attribute_weights, attribute_count, vertex_lock, target_index_count, target_error, options, result_error);
}

float meshopt_simplifyScale(const float* vertex_positions, size_t vertex_count, size_t vertex_positions_stride)
{
	if (vertex_positions_stride < 12 || vertex_positions_stride > 256 || vertex_positions_stride % 4 != 0)
	{
		setStatus(meshoptgpu_StatusInvalidArgument, "vertex_positions_stride must be in [12, 256] and a multiple of 4");
		return 0.f;
	}
	try
	{
		ThreadState& s = state();
		s.ensure();
		float* d_pos = static_cast<float*>(s.inputs.ensure(align256(vertex_count * vertex_positions_stride) + 256));
		if (vertex_count)
			MO_CUDA_CHECK(cudaMemcpyAsync(d_pos, vertex_positions, stridedExtent(vertex_count, vertex_positions_stride, 12), cudaMemcpyHostToDevice, s.stream));
		float r = s.simplifier->scale(d_pos, vertex_count, vertex_positions_stride, s.stream);
		setStatus(meshoptgpu_StatusOk, "");
		return r;
	}
	catch (const std::exception& e)
	{
		setStatus(statusOf(e), e.what());
		return 0.f;
	}
}

int meshoptgpu_getLastStatus(void)
{
	return state().status;
}

const char* meshoptgpu_getLastMessage(void)
{
	return state().message.c_str();
}

int meshoptgpu_getLastPassStats(meshoptgpu_PassStats* out, int max_passes)
{
	ThreadState& s = state();
	int n = s.last.passes < kMaxPassStats ? s.last.passes : kMaxPassStats;
	for (int i = 0; i < n && i < max_passes; ++i)
	{
		const PassStats& p = s.last.pass[i];
		out[i] = meshoptgpu_PassStats{p.triangles, p.candidates, p.evaluated, p.done, p.skipped, p.invalid, p.stop, p.rounds, p.active, p.windows};
	}
	return s.last.passes;
}

int meshoptgpu_getLastRoundTrace(unsigned int* active, float* micros, int max_rounds)
{
	const RunResult& r = state().last;
	int n = int(r.round_trace.size());
	for (int i = 0; i < n && i < max_rounds; ++i)
	{
		active[i] = r.round_trace[i].first;
		micros[i] = r.round_trace[i].second;
	}
	return n;
}

int meshoptgpu_getLastPassPhaseTimes(float* out, int max_passes)
{
	const RunResult& r = state().last;
	int n = int(r.pass_phase_ms.size());
	for (int i = 0; i < n && i < max_passes; ++i)
		memcpy(out + 5 * i, r.pass_phase_ms[i].data(), 5 * sizeof(float));
	return n;
}

void meshoptgpu_setTiming(int enabled)
{
	state().timing = enabled != 0;
}

int meshoptgpu_getLastPhaseTimes(float* out16)
{
	const PhaseTimes& t = state().times;
	float v[8] = {t.setup, t.adjacency, t.pick, t.rank, t.sort, t.perform, t.apply, t.total};
	memcpy(out16, v, sizeof(v));
	memcpy(out16 + 8, state().last.perform_phase_ms, sizeof(v));
	return 16;
}

size_t meshoptgpu_simplifyDevice(unsigned int* destination, const unsigned int* indices, size_t index_count, const float* vertex_positions,
    size_t vertex_count, size_t vertex_positions_stride, const float* vertex_attributes, size_t vertex_attributes_stride, const float* attribute_weights,
    size_t attribute_count, const unsigned char* vertex_lock, size_t target_index_count, float target_error, unsigned int options, float* result_error,
    void* stream)
{
	std::string bad = checkArgs(index_count, vertex_positions_stride, target_index_count, target_error, vertex_attributes_stride, attribute_weights,
	    attribute_count, options);
	cudaStream_t st = static_cast<cudaStream_t>(stream);
	auto fail = [&](int status, const std::string& msg) {
		setStatus(status, msg);
		if (destination != indices && index_count)
			cudaMemcpyAsync(destination, indices, index_count * 4, cudaMemcpyDeviceToDevice, st);
		if (result_error)
			*result_error = 0.f;
		return index_count;
	};
	if (!bad.empty())
		return fail((options & ~kSupportedOptions) ? meshoptgpu_StatusUnsupported : meshoptgpu_StatusInvalidArgument, bad);
	try
	{
		ThreadState& s = state();
		s.ensure();
		MeshDesc m;
		m.indices = indices;
		m.index_count = index_count;
		m.positions = vertex_positions;
		m.vertex_count = vertex_count;
		m.positions_stride = vertex_positions_stride;
		m.attributes = vertex_attributes;
		m.attributes_stride = vertex_attributes_stride;
		m.weights = attribute_weights;
		m.attribute_count = attribute_count;
		m.lock = vertex_lock;
		m.target_index_count = target_index_count;
		m.target_error = target_error;
		m.options = options;
		routeAndRun(s, m, destination, st, true);
		if (result_error)
			*result_error = s.last.result_error;
		setStatus(meshoptgpu_StatusOk, "");
		return s.last.index_count;
	}
	catch (const std::exception& e)
	{
		return fail(statusOf(e), e.what());
	}
}

void meshoptgpu_setKernelProfile(const char* kernel_name)
{
	LaunchProbe& p = probe();
	p.selected = kernel_name ? kernel_name : "";
	p.timed_launches = 0;
	p.timed_ms = 0;
}

void meshoptgpu_getKernelProfile(unsigned long long* launches, double* total_ms)
{
	LaunchProbe& p = probe();
	if (launches)
		*launches = p.timed_launches;
	if (total_ms)
		*total_ms = p.timed_ms;
}

unsigned long long meshoptgpu_getLaunchCount(void)
{
	return probe().launches;
}

size_t meshoptgpu_workspaceBytes(size_t index_count, size_t vertex_count, size_t attribute_count)
{
	return Simplifier::workspaceBytes(index_count, vertex_count, attribute_count);
}

void meshoptgpu_releaseThreadResources(void)
{
	tls.reset();
}

} // extern "C"
