// mo_batch_kernel.cuh - many small meshes simplified in one persistent launch: the kernel, instantiated
// by mo_batch_lean.cu, mo_batch_full.cu and mo_batch_wide.cu (one translation unit each, so that they
// compile side by side).
//
// Each CTA takes meshes from a device work queue (an atomic ticket) and runs the whole
// edge-collapse simplification of one mesh (meshopt_simplifyEdge, src/simplifier.cpp:2344-2626) with
// block-level phases.
//
// What bounds it is latency: chains of dependent accesses to a mesh's few hundred vertices, between
// barriers. So the mesh lives in shared memory, with 16-bit ids so that two CTAs with a 1,024-triangle
// group of cluster LOD or four with a 512-triangle mesh share an SM, and the code for it is compiled
// apart from the code for a mesh in the CTA's slab of global memory, so that its loads are shared-memory
// loads (as generic ones they made the whole kernel 10 to 20% slower). Measured with 32-bit ids in memory
// addressed generically, the mesh in shared memory only where the largest fits whole: 4,096 meshes of 510
// triangles 1.43 ms and 0.82 since (the kernel alone 0.53); 2,048 groups of 1,024 triangles with attributes
// 3.67 ms and 1.88.
#pragma once

#include <cmath>
#include <type_traits>

#include "mo_common.cuh"
#include "mo_prims.cuh"
#include "mo_probe.cuh"
#include "mo_batch.cuh"

namespace mogpu
{

namespace
{

// A mesh's vertex and triangle ids, in 16 bits where they and the table slots kept in their place fit.
template <class IX>
struct Pair2;
template <>
struct Pair2<unsigned short>
{
	typedef ushort2 T;
	typedef unsigned int Mark; // a round's tag over a sorted position; or a commit's position over its target
	static __device__ __forceinline__ T make(unsigned int x, unsigned int y) { return make_ushort2((unsigned short)x, (unsigned short)y); }
};
template <>
struct Pair2<unsigned int>
{
	typedef uint2 T;
	typedef unsigned long long Mark;
	static __device__ __forceinline__ T make(unsigned int x, unsigned int y) { return make_uint2(x, y); }
};

constexpr unsigned int kSortKeys = 2560;  // values of sortKey
// Candidates of a pass's expected window that a warp walks alone. A walk takes about 200 cycles for each
// that is not locked, a round 3,000 whatever its size, and a pass six rounds. Walks up to 0 / 160 / 192 /
// 224 / 256 / 512 candidates: one mesh of 510 triangles 194 / 190 / 168 / 166 / 171 / 181 us; 4,096 of
// 510 triangles 1.17 / 1.12 / 1.07 / 1.00 / 1.02 / 1.01 ms; 2,048 groups of 1,024 triangles 1.92 / 1.89 /
// 1.90 / 1.90 / 1.99 / 2.05 ms.
constexpr unsigned int kWalk = 224;
// Where a walk hands over to the rounds, if the stop rules let it come so far (most candidates' flips are
// rejected). One mesh of 16,700 triangles that looks at 15,000 candidates in each of two passes to remove
// 100 triangles: 14.7 ms with a walk to their end, 4.8 so.
constexpr unsigned int kWalkEnd = 2 * kWalk;
// Candidates within the error limit that a longer pass's warp walks alone: all of them are looked at, where
// about half of the window above are. Up to 0 / 32 / 64 / 96 / 160 candidates, 4,096 meshes of 1,682
// triangles to an error of 1e-3 3.37 / 3.31 / 3.39 / 3.54 / 3.55 ms (5.27 with the window by the goal alone,
// one mesh of 512 triangles 0.104 and 0.076); no difference at 0 and 1e-4.
constexpr unsigned int kWalkLimit = 32;

template <class IX>
struct CtaWork
{
	IX* idx;                         // I: current result indices (compacted in place)
	float4* pos;                     // V: rescaled positions
	IX* remap;                       // V
	IX* wedge;                       // V
	IX* loop;                        // V
	IX* loopback;                    // V
	unsigned char* kind;             // V
	unsigned char* staged;           // V: the permissive kinds while they are found
	Quadric* vq;                     // V
	unsigned int* adj_off;           // V + 2: list starts; counts and then cursors while lists are built
	typename Pair2<IX>::T* adj;      // I
	IX* cr;                          // V: the pass's moves
	unsigned int* table;             // H
	IX* cv0;                         // cap
	IX* cv1;                         // cap
	unsigned int* cerr;              // cap
	IX* order;                       // cap
	IX* hist;                        // kSortKeys + 2: the sort's counters: its keys, or 8 warps x 256 digits
	typename Pair2<IX>::Mark* minT;  // V: earliest undecided candidate touching the vertex; 0 once a commit took it
	typename Pair2<IX>::Mark* minS;  // V: ... that moves the vertex
	typename Pair2<IX>::Mark* moved; // V: the commit that moved the vertex and where to; all ones: none
	unsigned char* status;           // cap: decision per sorted position
	IX* sort_tmp;                    // cap: the sort's first digit pass; then the window's undecided candidates
	unsigned int* back;              // V: sparse meshes, local vertex -> vertex of the shared buffer
	float* attr;                     // V * ac: rescaled attributes
	Quadric* aq;                     // V: attribute quadrics (per wedge)
	float4* ag;                      // V * ac: attribute gradients
};

__host__ __device__ inline size_t alignUp(size_t v, size_t a)
{
	return (v + a - 1) & ~(a - 1);
}

__host__ __device__ inline size_t hashBucketsFor(size_t count)
{
	size_t b = 1;
	while (b < count + count / 4)
		b *= 2;
	return b;
}

// vertices a mesh's workspace is carved for: its own, or for a sparse mesh at most one per index
__host__ __device__ inline size_t localVertexBound(size_t I, size_t vertex_count, bool sparse)
{
	return sparse ? (I < vertex_count ? I : vertex_count) : vertex_count;
}

// Memory handed out front to back; what lies past the limit is not to be used (ok() is false then), and
// without a base it only counts.
struct Region
{
	char* base;
	size_t limit;
	size_t off = 0;

	__host__ __device__ Region(char* b, size_t l) : base(b), limit(l) {}
	template <class T>
	__host__ __device__ void take(T*& ptr, size_t count)
	{
		ptr = reinterpret_cast<T*>(base + off);
		off = alignUp(off + count * sizeof(T), 16);
	}
	__host__ __device__ bool ok() const { return off <= limit; }
};

// A mesh's workspace is carved in steps, each when its size is known: the index arrays, the arrays of
// its V (local) vertices (a sparse mesh's are counted first), and, in the place of the position table,
// the candidates of its collapse capacity. The attribute rows have a region of their own, beside the
// rest where they fit, else in the slab.
template <class IX>
__host__ __device__ inline void carveIndices(CtaWork<IX>& w, Region& r, size_t I)
{
	r.take(w.idx, I);
	r.take(w.adj, I);
}

// a sparse mesh's first-use table, in the place of its vertex arrays
__host__ __device__ inline size_t sparseTableBytes(size_t vertex_bound)
{
	return hashBucketsFor(vertex_bound ? vertex_bound : 1) * 8;
}

template <class IX>
__host__ __device__ inline void carveVertices(CtaWork<IX>& w, Region& r, size_t V, bool sparse)
{
	r.take(w.pos, V);
	r.take(w.remap, V);
	r.take(w.wedge, V);
	r.take(w.loop, V);
	r.take(w.loopback, V);
	r.take(w.back, sparse ? V : 0);
	r.take(w.kind, V);
	r.take(w.staged, V);
	r.take(w.vq, V);
	r.take(w.adj_off, V + 2);
	r.take(w.cr, V);
	r.take(w.minT, V);
	r.take(w.minS, V);
	r.take(w.moved, V);
}

template <class IX>
__host__ __device__ inline void carveRows(CtaWork<IX>& w, Region& r, size_t V, size_t ac)
{
	r.take(w.attr, V * ac);
	r.take(w.aq, ac ? V : 0);
	r.take(w.ag, V * ac);
}

template <class IX>
__host__ __device__ inline void carveTable(CtaWork<IX>& w, Region& r, size_t V)
{
	r.take(w.table, hashBucketsFor(V ? V : 1));
}

template <class IX>
__host__ __device__ inline void carveCandidates(CtaWork<IX>& w, Region& r, size_t cap)
{
	r.take(w.cv0, cap);
	r.take(w.cv1, cap);
	r.take(w.cerr, cap);
	r.take(w.order, cap);
	r.take(w.sort_tmp, cap);
	r.take(w.hist, kSortKeys + 2);
	r.take(w.status, cap);
}

// bytes of everything but the attribute rows, and of those
template <class IX>
__host__ __device__ inline size_t hotBytes(size_t I, size_t V, size_t vertex_bound, size_t cap, bool sparse)
{
	CtaWork<IX> w;
	Region r(nullptr, 0);
	carveIndices(w, r, I);
	const size_t table = r.off + (sparse ? sparseTableBytes(vertex_bound) : 0);
	carveVertices(w, r, V, sparse);
	Region t = r;
	carveTable(w, t, V);
	carveCandidates(w, r, cap);
	const size_t most = t.off > r.off ? t.off : r.off;
	return most > table ? most : table;
}

template <class IX>
__host__ __device__ inline size_t rowBytes(size_t V, size_t ac)
{
	CtaWork<IX> w;
	Region r(nullptr, 0);
	carveRows(w, r, V, ac);
	return r.off;
}

// What a mesh is expected to need: a square patch of a surface has one vertex for two triangles and half
// its perimeter's (1,024 triangles: 560; 589 are allowed for), and its capacity (boundEdgeCollapses) is
// about two thirds of its indices (all of them where every edge is on a border). A mesh that needs more
// than the launch's shared memory runs in the slab, after its setup up to there; where many do, launches
// are sized for the most a mesh can need.
inline size_t expectedVertices(size_t I, size_t bound, bool sparse)
{
	if (!sparse)
		return bound;
	const size_t v = I / 6 + size_t(std::sqrt(double(I))) * 5 / 4 + 10;
	return v < bound ? v : bound;
}

__host__ __device__ inline size_t expectedCapacity(size_t I)
{
	return I - I * 3 / 10 + 16;
}

// whether a mesh had more vertices or a larger capacity than that
__device__ inline bool beyondExpected(unsigned int V, unsigned int I, unsigned int cap, bool sparse)
{
	const unsigned int x = V > I / 6 + 10 ? V - I / 6 - 10 : 0u; // beside 1.25 times the root of I
	return cap > expectedCapacity(I) || (sparse && (unsigned long long)x * x * 16 > 25ull * I);
}

// ---------------------------------------------------------------- block helpers

// exclusive scan of data[0..n) in place over the block; returns the total
template <int NT, unsigned int STRIDE = 1, class T>
__device__ unsigned int blockScanArray(T* data, unsigned int n, unsigned int* red)
{
	// each thread scans a contiguous run; one block scan of the run totals
	const unsigned int per = (n + NT - 1) / NT;
	const unsigned int b = min(n, threadIdx.x * per), e = min(n, b + per);
	unsigned int sum = 0;
	for (unsigned int i = b; i < e; ++i)
		sum += data[i * STRIDE];
	unsigned int tot;
	unsigned int run = blockExclusiveScan<NT>(sum, red, &tot);
	for (unsigned int i = b; i < e; ++i)
	{
		const unsigned int v = data[i * STRIDE];
		data[i * STRIDE] = T(run);
		run += v;
	}
	__syncthreads();
	return tot;
}

// One pass of a stable LSD radix sort of candidate indices on 8 bits of their sort key: up to 8
// warps each own a contiguous segment, count its digits (counters digit-major, then warp, so
// one scan gives every (digit, warp) its start), and scatter the segment in order. Equal digits
// keep segment order and index order inside a segment. src == nullptr: the identity.
template <int NT, class IX>
__device__ void blockDigitPass(const unsigned int* cerr, const IX* src, IX* dst, unsigned int C, int shift, IX* cnt, unsigned int* red)
{
	constexpr unsigned int NW = NT / 32 < 8 ? NT / 32 : 8; // counters: NW * 256 words
	const unsigned int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const unsigned int seg = (C + NW - 1) / NW;
	const unsigned int s0 = min(C, warp * seg), s1 = warp < NW ? min(C, s0 + seg) : s0;
	for (unsigned int i = threadIdx.x; i < NW * 256; i += NT)
		cnt[i] = 0;
	__syncthreads();
	for (unsigned int b = s0; b < s1; b += 32)
	{
		unsigned int x = b + lane;
		bool valid = x < s1;
		unsigned int v = valid ? (src ? (unsigned int)src[x] : x) : 0u;
		unsigned int d = valid ? ((sortKey(cerr[v]) >> shift) & 255u) : 256u + lane;
		unsigned int peers = __match_any_sync(0xffffffffu, d);
		if (valid && lane == (unsigned int)(__ffs(peers) - 1))
			cnt[d * NW + warp] += IX(__popc(peers));
		__syncwarp();
	}
	__syncthreads();
	blockScanArray<NT>(cnt, NW * 256, red);
	for (unsigned int b = s0; b < s1; b += 32)
	{
		unsigned int x = b + lane;
		bool valid = x < s1;
		unsigned int v = valid ? (src ? (unsigned int)src[x] : x) : 0u;
		unsigned int d = valid ? ((sortKey(cerr[v]) >> shift) & 255u) : 256u + lane;
		unsigned int peers = __match_any_sync(0xffffffffu, d);
		unsigned int leader = __ffs(peers) - 1;
		unsigned int base = 0;
		if (valid && lane == leader)
		{
			base = cnt[d * NW + warp];
			cnt[d * NW + warp] = IX(base + __popc(peers));
		}
		base = __shfl_sync(0xffffffffu, base, leader);
		if (valid)
			dst[base + __popc(peers & ((1u << lane) - 1u))] = IX(v);
		__syncwarp();
	}
	__syncthreads();
}

// The same order for ids of 16 bits by one count of the whole key (kSortKeys counters, two to a word), a
// scatter, and a rank inside each key by index, its entries having come in any order. It has half the
// barriers of the digit passes and no chains of warp votes: 20k cycles of a 510-triangle mesh's 270k for
// its four passes, where they took 50k. False, with nothing written to dst, when more than kSameKey
// candidates share a key, whose ranking would then be the longer (a flat mesh's errors are all zero).
constexpr unsigned int kSameKey = 128;

template <int NT, class IX>
__device__ bool blockCountSort(const unsigned int* cerr, IX* tmp, IX* dst, unsigned char* slot, unsigned int C, IX* cnt, unsigned int* red)
{
	unsigned int* const word = reinterpret_cast<unsigned int*>(cnt);
	for (unsigned int i = threadIdx.x; i < (kSortKeys + 2) / 2; i += NT)
		word[i] = 0;
	__syncthreads();
	bool many = false;
	for (unsigned int c = threadIdx.x; c < C; c += NT)
	{
		const unsigned int key = sortKey(cerr[c]), half = (key & 1) * 16;
		const unsigned int at = atomicAdd(&word[key / 2], 1u << half) >> half & 0xffffu;
		many |= at >= kSameKey;
		slot[c] = (unsigned char)at;
	}
	if (__syncthreads_or(many))
		return false;
	blockScanArray<NT>(cnt, kSortKeys + 1, red);
	for (unsigned int c = threadIdx.x; c < C; c += NT)
		tmp[cnt[sortKey(cerr[c])] + slot[c]] = IX(c);
	__syncthreads();
	for (unsigned int c = threadIdx.x; c < C; c += NT)
	{
		const unsigned int key = sortKey(cerr[c]), b = cnt[key], e = cnt[key + 1];
		unsigned int at = b;
		for (unsigned int x = b; x < e; ++x)
			at += tmp[x] < c;
		dst[at] = IX(c);
	}
	__syncthreads();
	return true;
}

template <int NT>
__device__ unsigned int blockSum(unsigned int v, unsigned int* red)
{
	unsigned int tot;
	blockExclusiveScan<NT>(v, red, &tot);
	__syncthreads();
	return tot;
}

__device__ __forceinline__ unsigned int mix32b(unsigned int h)
{
	h ^= h >> 16;
	h *= 0x7feb352du;
	h ^= h >> 15;
	h *= 0x846ca68bu;
	h ^= h >> 16;
	return h;
}

__device__ __forceinline__ unsigned int posBitsB(float f)
{
	unsigned int u = __float_as_uint(f);
	return u == 0x80000000u ? 0u : u;
}

// ordered min/max folds, see rescalePositions :551-567 (leftmost of equal values, NaN skipped)
__device__ __forceinline__ float fmin_l(float l, float r)
{
	return l > r ? r : l;
}

__device__ __forceinline__ float fmax_l(float l, float r)
{
	return l < r ? r : l;
}

// ---------------------------------------------------------------- one mesh

extern __shared__ __align__(16) char smem[];

// FULL = false compiles out the sparse subset, attributes, vertex_lock and Permissive, so that
// positions-only batches run the lean instantiation
template <int NT, bool FULL, class IX, bool FAST>
__device__ bool simplifyMesh(const BatchDesc& d, BatchResult* out, Region mem, Region rows)
{
	// mem: the mesh's memory; rows: what the attribute rows take when mem has no room for them. False
	// when mem is too small (nothing is written then). FAST: mem is the block's shared memory, and named
	// as such, so that its loads and atomics are not generic ones.
	if constexpr (FAST)
		mem.base = smem;
	CtaWork<IX> w;
	__shared__ unsigned int s_red[64];
	unsigned int* const red = s_red;
	typedef typename Pair2<IX>::T IX2;
	constexpr IX kNone = IX(~0u); // no loop, no slot
	constexpr unsigned int kWhere = FAST ? 0u : kBatchInSlab;
	const unsigned int tid = threadIdx.x;
	const unsigned int I = d.index_count;
	const float* P = d.positions;
	const unsigned int sf = d.stride_f;
	const unsigned int ac = FULL ? d.ac : 0;
	const unsigned char* const vlock = FULL ? d.lock : nullptr;
	const bool sparse = FULL && (d.options & kOptSparse) != 0;
	carveIndices(w, mem, I);
	if (!mem.ok())
		return false;
	__shared__ unsigned int s_flag, s_unique;
	__shared__ float s_mm[NT / 32][6];
	__shared__ float s_minv[3], s_scale, s_extent;
	__shared__ unsigned int s_cap, s_count, s_trunc, s_done, s_errbits, s_stall;
	__shared__ unsigned long long s_cut;
	__shared__ unsigned int s_sums[3][33];
	__shared__ unsigned int s_window;
	__shared__ unsigned int s_walk[4]; // sorted positions walked, and the stop rules' terms up to there

	if (tid == 0)
		s_flag = 0, s_stall = 0;
	__syncthreads();
	for (unsigned int i = tid; i < I; i += NT)
	{
		unsigned int v = d.indices[i];
		w.idx[i] = IX(v);
		if (v >= d.vertex_count)
			s_flag = 1;
	}
	__syncthreads();
	if (s_flag)
	{
		if (tid == 0)
			*out = BatchResult{I, 0.f, 0, 2u | kWhere};
		for (unsigned int i = tid; i < I; i += NT)
			d.out[i] = d.indices[i];
		return true;
	}

	// ---- sparse subset (buildSparseRemap :242-294): local ids in order of first use. A
	// 64-bit table keyed by the shared-buffer vertex keeps its first index position (atomicMin);
	// the positions that are first uses, ranked by a block scan, give the local ids.
	unsigned int V = d.vertex_count;
	if (sparse)
	{
		const size_t bound = localVertexBound(I, d.vertex_count, true);
		if (mem.off + sparseTableBytes(bound) > mem.limit)
			return false;
		unsigned long long* t64 = reinterpret_cast<unsigned long long*>(mem.base + mem.off);
		const unsigned int HS = (unsigned int)hashBucketsFor(bound ? bound : 1);
		const unsigned int smask = HS - 1;
		for (unsigned int i = tid; i < HS; i += NT)
			t64[i] = ~0ull;
		__syncthreads();
		for (unsigned int p = tid; p < I; p += NT)
		{
			unsigned int v = d.indices[p]; // the shared buffer's id
			unsigned long long key = ((unsigned long long)v << 32) | p;
			unsigned int b = mix32b(v) & smask, slot = 0;
			for (unsigned int probe = 0; probe <= smask; ++probe)
			{
				unsigned long long cur = t64[b];
				if (cur == ~0ull)
				{
					unsigned long long prev = atomicCAS(&t64[b], ~0ull, key);
					if (prev == ~0ull)
					{
						slot = b;
						break;
					}
					cur = prev;
				}
				if ((unsigned int)(cur >> 32) == v)
				{
					atomicMin(&t64[b], key);
					slot = b;
					break;
				}
				b = (b + probe + 1) & smask;
			}
			w.adj[p].x = IX(slot);
		}
		__syncthreads();
		for (unsigned int p = tid; p < I; p += NT)
			w.adj[p].y = IX(t64[w.adj[p].x]); // first position of this vertex
		__syncthreads();
		// the table is dead from here: the vertex arrays take its place
		for (unsigned int p = tid; p < I; p += NT)
			w.adj[p].x = w.adj[p].y == p;
		__syncthreads();
		unsigned int unique = I ? blockScanArray<NT, 2>(&w.adj[0].x, I, red) : 0u;
		carveVertices(w, mem, unique, true);
		if (!mem.ok())
			return false;
		for (unsigned int p = tid; p < I; p += NT)
		{
			const IX2 a = w.adj[p];
			if (a.y == p)
				w.back[a.x] = d.indices[p];
			w.idx[p] = w.adj[a.y].x;
		}
		if (tid == 0)
			s_unique = unique;
		__syncthreads();
		V = s_unique;
	}
	else
	{
		carveVertices(w, mem, V, false);
		if (!mem.ok())
			return false;
	}
	auto src = [&](unsigned int i) { return sparse ? w.back[i] : i; };
	if (FULL && ac)
	{
		Region with = mem, rest = mem;
		carveRows(w, with, V, ac);
		rest.off = with.off;
		carveCandidates(w, rest, expectedCapacity(I));
		if (FAST && rest.ok())
			mem = with;
		else
		{
			carveRows(w, rows, V, ac);
			if (!rows.ok())
				return false;
		}
	}
	{
		Region t = mem;
		carveTable(w, t, V);
		if (!t.ok())
			return false;
	}

	// ---- position remap (buildPositionRemap :195-214) in a block-local hash table
	const unsigned int H = (unsigned int)hashBucketsFor(V ? V : 1), mask = H - 1;
	for (unsigned int i = tid; i < H; i += NT)
		w.table[i] = ~0u;
	__syncthreads();
	for (unsigned int i = tid; i < V; i += NT)
	{
		const float* p = P + (size_t)src(i) * sf;
		float x = p[0], y = p[1], z = p[2];
		unsigned int h = mix32b(posBitsB(x) * 0x9e3779b1u ^ mix32b(posBitsB(y) + 0x85ebca6bu) ^ mix32b(posBitsB(z) * 0xc2b2ae35u + 1u));
		unsigned int b = h & mask, slot = ~0u;
		for (unsigned int probe = 0; probe <= mask; ++probe)
		{
			unsigned int cur = w.table[b];
			if (cur == ~0u)
			{
				unsigned int prev = atomicCAS(&w.table[b], ~0u, i);
				if (prev == ~0u)
				{
					slot = b;
					break;
				}
				cur = prev;
			}
			const float* q = P + (size_t)src(cur) * sf;
			if (q[0] == x && q[1] == y && q[2] == z)
			{
				atomicMin(&w.table[b], i);
				slot = b;
				break;
			}
			b = (b + probe + 1) & mask;
		}
		w.remap[i] = IX(slot); // slot for now
	}
	__syncthreads();
	for (unsigned int i = tid; i < V; i += NT)
	{
		const IX s = w.remap[i];
		w.remap[i] = IX(s == kNone ? i : w.table[s]);
	}
	__syncthreads();
	// wedge cycle (:229-239): dup i -> previous member of its class (or the primary); the
	// primary -> largest duplicate
	for (unsigned int i = tid; i < V; i += NT)
	{
		w.wedge[i] = IX(i);
		w.adj_off[i] = 0; // the class's largest duplicate
	}
	__syncthreads();
	for (unsigned int i = tid; i < V; i += NT)
	{
		unsigned int r = w.remap[i];
		if (r == i)
			continue;
		unsigned int pred = r;
		for (unsigned int j = r + 1; j < i; ++j)
			if (w.remap[j] == r)
				pred = j;
		w.wedge[i] = IX(pred);
		atomicMax(&w.adj_off[r], i);
	}
	__syncthreads();
	for (unsigned int i = tid; i < V; i += NT)
		if (w.remap[i] == i && w.adj_off[i])
			w.wedge[i] = IX(w.adj_off[i]);
	__syncthreads();

	// ---- rescale (rescalePositions :544-603): ordered folds over contiguous thread chunks
	{
		float mn[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, mx[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
		unsigned int per = (V + NT - 1) / NT, b0 = min(V, tid * per), b1 = min(V, b0 + per);
		for (unsigned int i = b0; i < b1; ++i)
		{
			const float* p = P + (size_t)src(i) * sf;
			for (int j = 0; j < 3; ++j)
			{
				mn[j] = mn[j] > p[j] ? p[j] : mn[j];
				mx[j] = mx[j] < p[j] ? p[j] : mx[j];
			}
		}
		for (int o = 1; o < 32; o <<= 1)
			for (int j = 0; j < 3; ++j)
			{
				float a = __shfl_down_sync(0xffffffffu, mn[j], o), c = __shfl_down_sync(0xffffffffu, mx[j], o);
				if ((tid & 31) + o < 32 && ((tid & (2 * o - 1)) == 0))
					mn[j] = fmin_l(mn[j], a), mx[j] = fmax_l(mx[j], c);
			}
		if ((tid & 31) == 0)
			for (int j = 0; j < 3; ++j)
				s_mm[tid >> 5][j] = mn[j], s_mm[tid >> 5][3 + j] = mx[j];
		__syncthreads();
		if (tid == 0)
		{
			for (int q = 1; q < NT / 32; ++q)
				for (int j = 0; j < 3; ++j)
					s_mm[0][j] = fmin_l(s_mm[0][j], s_mm[q][j]), s_mm[0][3 + j] = fmax_l(s_mm[0][3 + j], s_mm[q][3 + j]);
			float extent = 0.f;
			extent = (s_mm[0][3] - s_mm[0][0]) < extent ? extent : (s_mm[0][3] - s_mm[0][0]);
			extent = (s_mm[0][4] - s_mm[0][1]) < extent ? extent : (s_mm[0][4] - s_mm[0][1]);
			extent = (s_mm[0][5] - s_mm[0][2]) < extent ? extent : (s_mm[0][5] - s_mm[0][2]);
			s_extent = extent;
			s_scale = extent == 0 ? 0.f : 1.f / extent;
			for (int j = 0; j < 3; ++j)
				s_minv[j] = s_mm[0][j];
		}
		__syncthreads();
		for (unsigned int i = tid; i < V; i += NT)
		{
			const float* p = P + (size_t)src(i) * sf;
			w.pos[i] = make_float4((p[0] - s_minv[0]) * s_scale, (p[1] - s_minv[1]) * s_scale, (p[2] - s_minv[2]) * s_scale, 0.f);
		}
		// rescaleAttributes (:605-621): weighted copies of the used attributes
		if constexpr (FULL)
			if (ac)
				for (unsigned int x = tid; x < V * ac; x += NT)
				{
					unsigned int i = x / ac, k = x - i * ac;
					w.attr[x] = d.attributes[(size_t)src(i) * d.attr_stride_f + d.amap->src[k]] * d.amap->weight[k];
				}
	}

	// ---- raw adjacency (updateEdgeAdjacency :52-109, no remap): corner lists, unordered. Lists are built
	// with their counts one place up: after the scan adj_off[v + 1] is v's start, and the cursor that ends
	// as the next one's.
	for (unsigned int i = tid; i < V + 2; i += NT)
		w.adj_off[i] = 0;
	__syncthreads();
	for (unsigned int p = tid; p < I; p += NT)
		atomicAdd(&w.adj_off[w.idx[p] + 1], 1u);
	__syncthreads();
	blockScanArray<NT>(w.adj_off, V + 2, red);
	for (unsigned int p = tid; p < I; p += NT)
	{
		unsigned int v = w.idx[p];
		unsigned int s = atomicAdd(&w.adj_off[v + 1], 1u);
		unsigned int f = p / 3, c = p - f * 3;
		w.adj[s] = Pair2<IX>::make(w.idx[f * 3 + (c == 2 ? 0 : c + 1)], w.idx[f * 3 + (c == 0 ? 2 : c - 1)]);
	}
	__syncthreads();

	// ---- classification (classifyVertices :364-542, open edges from each vertex's own list)
	for (unsigned int v = tid; v < V; v += NT)
	{
		unsigned int b = w.adj_off[v], e = w.adj_off[v + 1];
		bool degen = false;
		for (unsigned int j = b; j < e; ++j)
			degen |= w.adj[j].x == v;
		unsigned int outc = 0, outt = ~0u, inc = 0, ins = ~0u;
		if (!degen)
			for (unsigned int j = b; j < e; ++j)
			{
				const IX2 ej = w.adj[j];
				bool bk = false, fwd = false;
				for (unsigned int q = b; q < e; ++q)
				{
					const IX2 eq = w.adj[q];
					bk |= eq.y == ej.x;
					fwd |= eq.x == ej.y;
				}
				if (!bk)
					outc++, outt = ej.x;
				if (!fwd)
					inc++, ins = ej.y;
			}
		w.loop[v] = IX(degen ? v : (outc == 0 ? ~0u : (outc == 1 ? outt : v)));
		w.loopback[v] = IX(degen ? v : (inc == 0 ? ~0u : (inc == 1 ? ins : v)));
	}
	__syncthreads();
	for (unsigned int i = tid; i < V; i += NT)
	{
		unsigned int r = w.remap[i], wi = w.wedge[r];
		unsigned char k;
		if (wi == r)
		{
			const IX openi = w.loopback[r], openo = w.loop[r];
			if (openi == kNone && openo == kNone)
				k = kManifold;
			else if (openi != kNone && openo != kNone && w.remap[openi] == w.remap[openo] && openi != r)
				k = kSeam;
			else if (openi != r && openo != r)
				k = kBorder;
			else
				k = kLocked;
		}
		else if (w.wedge[wi] == r)
		{
			const IX openiv = w.loopback[r], openov = w.loop[r], openiw = w.loopback[wi], openow = w.loop[wi];
			if (openiv != kNone && openiv != r && openov != kNone && openov != r && openiw != kNone && openiw != wi && openow != kNone && openow != wi)
				k = (w.remap[openiv] == w.remap[openow] && w.remap[openov] == w.remap[openiw] && w.remap[openiv] != w.remap[openov]) ? kSeam : kLocked;
			else
				k = kLocked;
		}
		else
			k = kLocked;
		w.kind[i] = k;
	}
	__syncthreads();
	if (FULL && (d.options & kOptPermissive))
	{
		// Permissive (:481-515): a seam or locked primary becomes Complex unless a wedge is
		// protected or has a half-edge with no opposite in position space (hasEdge :345-362);
		// the new kinds are staged, then copied to wedges
		for (unsigned int i = tid; i < V; i += NT)
		{
			unsigned char k = w.kind[i];
			unsigned char nk = k;
			if (w.remap[i] == i && (k == kSeam || k == kLocked))
			{
				bool protect = false;
				unsigned int v = i;
				do
				{
					protect |= vlock && (vlock[src(v)] & kVertexProtect) != 0;
					v = w.wedge[v];
				} while (v != i);
				do
				{
					for (unsigned int j = w.adj_off[v]; j < w.adj_off[v + 1] && !protect; ++j)
					{
						// hasEdge(nx -> v) over the wedges of nx
						unsigned int a = w.adj[j].x, rb = w.remap[v], u = a;
						bool found = false;
						do
						{
							for (unsigned int q = w.adj_off[u]; q < w.adj_off[u + 1] && !found; ++q)
								found = w.remap[w.adj[q].x] == rb;
							u = w.wedge[u];
						} while (u != a && !found);
						protect |= !found;
					}
					v = w.wedge[v];
				} while (v != i);
				nk = protect ? k : (unsigned char)kComplex;
			}
			w.staged[i] = nk;
		}
		__syncthreads();
		for (unsigned int i = tid; i < V; i += NT)
		{
			unsigned char k = w.kind[i];
			if (k == kSeam || k == kLocked)
				w.kind[i] = w.staged[w.remap[i]];
		}
		__syncthreads();
	}
	if (vlock)
	{
		// vertex_lock (:517-531): a locked wedge locks its whole position
		for (unsigned int i = tid; i < V; i += NT)
			if (vlock[src(i)] & kVertexLock)
				w.kind[w.remap[i]] = kLocked;
		__syncthreads();
		for (unsigned int i = tid; i < V; i += NT)
			if (w.kind[w.remap[i]] == kLocked)
				w.kind[i] = kLocked;
		__syncthreads();
	}
	if (d.options & kOptLockBorder)
	{
		for (unsigned int i = tid; i < V; i += NT)
			if (w.kind[i] == kBorder)
				w.kind[i] = kLocked;
		__syncthreads();
	}

	// ---- capacity (boundEdgeCollapses :1292-1308) from the raw degrees
	{
		unsigned int dual = 0;
		for (unsigned int i = tid; i < V; i += NT)
		{
			unsigned char k = w.kind[i];
			dual += (k == kManifold || k == kSeam) ? (w.adj_off[i + 1] - w.adj_off[i]) : 0;
		}
		unsigned int tot = blockSum<NT>(dual, red);
		if (tid == 0)
			s_cap = I - tot / 2 + 3;
		__syncthreads();
		carveCandidates(w, mem, s_cap);
		if (!mem.ok())
			return false;
	}

	// ---- corner lists in corner order (remapped for the position quadrics, raw for the
	// attribute quadrics), then the quadric folds (:1057-1179)
	auto cornerLists = [&](bool remapped) {
		for (unsigned int i = tid; i < V + 2; i += NT)
			w.adj_off[i] = 0;
		__syncthreads();
		for (unsigned int p = tid; p < I; p += NT)
			atomicAdd(&w.adj_off[(remapped ? w.remap[w.idx[p]] : w.idx[p]) + 1], 1u);
		__syncthreads();
		blockScanArray<NT>(w.adj_off, V + 2, red);
		for (unsigned int p = tid; p < I; p += NT)
		{
			unsigned int v = remapped ? w.remap[w.idx[p]] : w.idx[p];
			w.adj[atomicAdd(&w.adj_off[v + 1], 1u)].x = IX(p);
		}
		__syncthreads();
		for (unsigned int v = tid; v < V; v += NT)
		{
			// insertion sort of the vertex's corners (few per vertex)
			unsigned int b = w.adj_off[v], e = w.adj_off[v + 1];
			for (unsigned int j = b + 1; j < e; ++j)
			{
				const IX x = w.adj[j].x;
				unsigned int q = j;
				while (q > b && w.adj[q - 1].x > x)
				{
					w.adj[q].x = w.adj[q - 1].x;
					--q;
				}
				w.adj[q].x = x;
			}
		}
		__syncthreads();
	};
	cornerLists(true);
	{
		const float factor = (d.options & kOptRegularizeLight) ? 1e-2f : ((d.options & kOptRegularize) ? 1e-1f : 1e-7f);
		for (unsigned int r = tid; r < V; r += NT)
		{
			if (w.remap[r] != r)
			{
				stquadric(w.vq, r, qzero());
				continue;
			}
			unsigned int b = w.adj_off[r], e = w.adj_off[r + 1];
			Quadric Q = qzero();
			for (unsigned int j = b; j < e; ++j)
			{
				unsigned int f = w.adj[j].x / 3;
				unsigned int i0 = w.idx[f * 3 + 0], i1 = w.idx[f * 3 + 1], i2 = w.idx[f * 3 + 2];
				float4 a0 = w.pos[i0], a1 = w.pos[i1], a2 = w.pos[i2];
				Quadric F = qtriangle(V3{a0.x, a0.y, a0.z}, V3{a1.x, a1.y, a1.z}, V3{a2.x, a2.y, a2.z}, 1.f);
				qadd(Q, F);
			}
			bool priority = vlock && (vlock[src(r)] & kVertexPriority) != 0;
			float wt = Q.w * (priority ? 1.0f : factor);
			float4 pr = w.pos[r];
			Quadric Pq = qpoint(pr.x, pr.y, pr.z, wt);
			qadd(Q, Pq);
			unsigned int lastf = ~0u;
			for (unsigned int j = b; j < e; ++j)
			{
				unsigned int f = w.adj[j].x / 3;
				if (f == lastf)
					continue;
				lastf = f;
				for (int ed = 0; ed < 3; ++ed)
				{
					unsigned int i0 = w.idx[f * 3 + ed], i1 = w.idx[f * 3 + (ed == 2 ? 0 : ed + 1)];
					unsigned char k0 = w.kind[i0], k1 = w.kind[i1];
					bool b0 = k0 == kBorder || k0 == kSeam, b1 = k1 == kBorder || k1 == kSeam;
					if (!b0 && !b1)
						continue;
					if (b0 && w.loop[i0] != i1)
						continue;
					if (b1 && w.loopback[i1] != i0)
						continue;
					bool to0 = w.remap[i0] == r, to1 = w.remap[i1] == r;
					if (!to0 && !to1)
						continue;
					unsigned int i2 = w.idx[f * 3 + (ed == 0 ? 2 : ed - 1)];
					float weight = (k0 == kBorder || k1 == kBorder) ? 10.f : 0.5f;
					float4 a0 = w.pos[i0], a1 = w.pos[i1], a2 = w.pos[i2];
					V3 p0{a0.x, a0.y, a0.z}, p1{a1.x, a1.y, a1.z}, p2{a2.x, a2.y, a2.z};
					Quadric E = qedge(p0, p1, p2, weight);
					Quadric Tq = qtriangle(p0, p1, p2, weight);
					Tq.w = 0;
					qadd(E, Tq);
					if (to0)
						qadd(Q, E);
					if (to1)
						qadd(Q, E);
				}
			}
			stquadric(w.vq, r, Q);
		}
	}
	__syncthreads();
	if constexpr (FULL)
	{
		if (ac)
		{
			// fillAttributeQuadrics (:1159-1179): per wedge over its faces in face order (each vertex is owned
			// by one thread); the gradients add up in registers where there are few and room for them, else in
			// place
			cornerLists(false);
			for (unsigned int v = tid; v < V; v += NT)
			{
				float4* G = w.ag + (size_t)v * ac;
				Quadric Q = qzero();
				auto faces = [&](auto limit, float4* to) {
					for (unsigned int j = w.adj_off[v]; j < w.adj_off[v + 1]; ++j)
					{
						unsigned int f = w.adj[j].x / 3;
						unsigned int i0 = w.idx[f * 3 + 0], i1 = w.idx[f * 3 + 1], i2 = w.idx[f * 3 + 2];
						float4 a0 = w.pos[i0], a1 = w.pos[i1], a2 = w.pos[i2];
						addAttributeQuadric<decltype(limit)::value>(Q, to, (int)ac, V3{a0.x, a0.y, a0.z}, V3{a1.x, a1.y, a1.z}, V3{a2.x, a2.y, a2.z},
						    w.attr + (size_t)i0 * ac, w.attr + (size_t)i1 * ac, w.attr + (size_t)i2 * ac);
					}
				};
				if (NT > 128 && ac <= 8)
				{
					float4 g[8];
#pragma unroll
					for (int k = 0; k < 8; ++k)
						g[k] = make_float4(0.f, 0.f, 0.f, 0.f);
					faces(std::integral_constant<int, 8>(), g);
#pragma unroll
					for (int k = 0; k < 8; ++k)
						if (k < (int)ac)
							G[k] = g[k];
				}
				else
				{
					for (unsigned int k = 0; k < ac; ++k)
						G[k] = make_float4(0.f, 0.f, 0.f, 0.f);
					faces(std::integral_constant<int, 32>(), G);
				}
				stquadric(w.aq, v, Q);
			}
			__syncthreads();
		}
	}

	// ---- pass loop (:2493-2541)
	const float error_scale = (d.options & kOptErrorAbsolute) ? s_extent : 1.f;
	const float error_limit = (d.target_error * d.target_error) / (error_scale * error_scale);
	unsigned int result_count = I;
	float result_error = 0.f;
	unsigned int passes = 0;

	while (result_count > d.target_index_count)
	{
		const unsigned int T = result_count / 3;

		// adjacency of the current result, welded by remap (unordered lists)
		for (unsigned int i = tid; i < V + 2; i += NT)
			w.adj_off[i] = 0;
		__syncthreads();
		for (unsigned int p = tid; p < result_count; p += NT)
			atomicAdd(&w.adj_off[w.remap[w.idx[p]] + 1], 1u);
		__syncthreads();
		blockScanArray<NT>(w.adj_off, V + 2, red);
		for (unsigned int t = tid; t < T; t += NT)
		{
			unsigned int a = w.remap[w.idx[t * 3 + 0]], b = w.remap[w.idx[t * 3 + 1]], c = w.remap[w.idx[t * 3 + 2]];
			w.adj[atomicAdd(&w.adj_off[a + 1], 1u)] = Pair2<IX>::make(b, c);
			w.adj[atomicAdd(&w.adj_off[b + 1], 1u)] = Pair2<IX>::make(c, a);
			w.adj[atomicAdd(&w.adj_off[c + 1], 1u)] = Pair2<IX>::make(a, b);
		}
		__syncthreads();

		// pick (pickEdgeCollapses :1310-1372): each thread takes a contiguous run of triangles,
		// counts its candidates, and after one block scan emits them in triangle order; the
		// capacity check stops at the first triangle that has no room for three more
		if (tid == 0)
			s_trunc = ~0u;
		{
			// 0: no candidate, 1: i0 onto i1, 2: i1 onto i0, 3: either way
			auto pickEdgeB = [&](unsigned int i0, unsigned int i1) -> unsigned int {
				unsigned int r0 = w.remap[i0], r1 = w.remap[i1];
				if (r0 == r1)
					return 0;
				unsigned int k0 = w.kind[i0], k1 = w.kind[i1];
				bool c01 = canCollapse(k0, k1), c10 = canCollapse(k1, k0);
				if (!(c01 | c10))
					return 0;
				if (hasOpposite(k0, k1) && r1 > r0)
					return 0;
				if ((k0 == kBorder || k0 == kSeam) && k1 != kManifold && w.loop[i0] != i1)
					return 0;
				if ((k1 == kBorder || k1 == kSeam) && k0 != kManifold && w.loopback[i1] != i0)
					return 0;
				return (c01 ? 1u : 0u) | (c10 ? 2u : 0u);
			};
			// what the first 10 triangles of a run give is kept for the emission, two bits per edge
			const unsigned int per = (T + NT - 1) / NT;
			const unsigned int t0 = min(T, tid * per), t1 = min(T, t0 + per);
			unsigned int n = 0;
			unsigned long long codes = 0;
			auto edge = [&](unsigned int t, unsigned int e, unsigned int& i0, unsigned int& i1) {
				i0 = w.idx[t * 3 + e], i1 = w.idx[t * 3 + (e == 2 ? 0 : e + 1)];
			};
			for (unsigned int t = t0; t < t1; ++t)
				for (unsigned int e = 0; e < 3; ++e)
				{
					unsigned int i0, i1;
					edge(t, e, i0, i1);
					const unsigned int code = pickEdgeB(i0, i1);
					n += code != 0;
					if (t - t0 < 10)
						codes |= (unsigned long long)code << ((t - t0) * 6 + e * 2);
				}
			unsigned int tot;
			unsigned int o = blockExclusiveScan<NT>(n, red, &tot);
			if (tid == 0)
				s_count = tot;
			for (unsigned int t = t0; t < t1; ++t)
			{
				if (o + 3 > s_cap)
				{
					atomicMin(&s_trunc, o);
					break;
				}
				for (unsigned int e = 0; e < 3; ++e)
				{
					unsigned int i0, i1;
					edge(t, e, i0, i1);
					const unsigned int code = t - t0 < 10 ? (unsigned int)(codes >> ((t - t0) * 6 + e * 2)) & 3u : pickEdgeB(i0, i1);
					if (code)
					{
						w.cv0[o] = IX(code == 2 ? i1 : i0), w.cv1[o] = IX(code == 2 ? i0 : i1), w.cerr[o] = code == 3;
						o++;
					}
				}
			}
			__syncthreads();
		}
		const unsigned int C = min(s_count, s_trunc);
		if (C == 0)
			break;

		// rank (rankEdgeCollapses :1374-1450)
		for (unsigned int c = tid; c < C; c += NT)
		{
			unsigned int i0 = w.cv0[c], i1 = w.cv1[c];
			bool bidi = w.cerr[c] != 0;
			float4 a0 = w.pos[i0], a1 = w.pos[i1];
			V3 p0{a0.x, a0.y, a0.z}, p1{a1.x, a1.y, a1.z};
			float ei = qerror(ldquadric(w.vq, w.remap[i0]), p1);
			float ej = bidi ? qerror(ldquadric(w.vq, w.remap[i1]), p0) : FLT_MAX;
			if (ac)
			{
				auto term = [&](unsigned int v, unsigned int t) {
					float4 pt = w.pos[t];
					return qerrorAttr(ldquadric(w.aq, v), w.ag + (size_t)v * ac, (int)ac, V3{pt.x, pt.y, pt.z}, w.attr + (size_t)t * ac);
				};
				ei += term(i0, i1);
				ej += bidi ? term(i1, i0) : 0;
				if (w.kind[i0] == kSeam)
				{
					unsigned int s0 = w.wedge[i0];
					IX s1 = w.loop[i0] == i1 ? w.loopback[s0] : w.loop[s0];
					s1 = s1 != kNone ? s1 : w.wedge[i1];
					ei += term(s0, s1);
					ej += bidi ? term(s1, s0) : 0;
				}
				else
				{
					if (FULL && w.kind[i0] == kComplex)
						for (unsigned int v = w.wedge[i0]; v != i0; v = w.wedge[v])
							ei += term(v, complexTarget<IX>(v, i1, w.remap, w.loop, w.loopback));
					if (FULL && w.kind[i1] == kComplex && bidi)
						for (unsigned int v = w.wedge[i1]; v != i1; v = w.wedge[v])
							ej += term(v, complexTarget<IX>(v, i0, w.remap, w.loop, w.loopback));
				}
			}
			bool rev = bidi & (ej < ei);
			w.cv0[c] = IX(rev ? i1 : i0);
			w.cv1[c] = IX(rev ? i0 : i1);
			w.cerr[c] = __float_as_uint(ej < ei ? ej : ei);
		}
		// sort (sortEdgeCollapses :1452-1496): the same stable order on the 12-bit key, by a count of the
		// keys, else as two stable 8-bit digit passes (low byte, then the high four bits)
		bool sorted = false;
		if constexpr (sizeof(IX) == 2)
			sorted = blockCountSort<NT>(w.cerr, w.sort_tmp, w.order, w.status, C, w.hist, red);
		if (!sorted)
		{
			blockDigitPass<NT>(w.cerr, (const IX*)nullptr, w.sort_tmp, C, 0, w.hist, red);
			blockDigitPass<NT>(w.cerr, (const IX*)w.sort_tmp, w.order, C, 8, w.hist, red);
		}
		// perform (performEdgeCollapses :1498-1636). A pass that is expected to look at few candidates is
		// walked in sorted order by one warp, four flip tests at a time; a longer one, and what a walk has not
		// come to by kWalkEnd, goes in block-level decision rounds: a candidate is decided once nothing earlier
		// in sorted order can change its outcome (the rule of the multi-CTA path's performPass), over a window
		// of sorted order that grows until the stop rules fire; the stop rules are a prefix scan of the
		// decisions. A warp keeps the undecided ones of every NT / 32nd position, so a round needs two barriers
		// only: marks are complete, decisions are complete.
		typedef typename Pair2<IX>::Mark Mark;
		constexpr unsigned int kTagShift = sizeof(Mark) * 4;
		constexpr Mark kFree = Mark(~0ull);
		const unsigned int goal = (result_count - d.target_index_count) / 3;
		for (unsigned int i = tid; i < V; i += NT)
			w.cr[i] = IX(i), w.minT[i] = kFree, w.minS[i] = kFree, w.moved[i] = kFree;
		for (unsigned int k = tid; k < C; k += NT)
			w.status[k] = kUndecided;
		if (tid == 0)
			s_cut = ~0ull, s_done = 0, s_errbits = __float_as_uint(result_error);
		const unsigned int warp = tid / 32, lane = tid & 31;
		if (warp == 0)
		{
			// The window the pass is expected to need: by its goal, and where that is not a short walk, up to the
			// first candidate of a key beyond the error limit's, which ends the pass (a 32-way search).
			unsigned int window = (unsigned int)min((unsigned long long)C, 2ull * (goal / 2) + 64ull);
			if (window > kWalk)
			{
				const unsigned int key = sortKey(__float_as_uint(error_limit));
				unsigned int lo = 0, hi = C;
				while (lo < hi)
				{
					const unsigned int step = (hi - lo + 31) / 32, at = lo + (lane + 1) * step - 1;
					const unsigned int m = __ballot_sync(0xffffffffu, at >= hi || sortKey(w.cerr[w.order[at]]) > key);
					const unsigned int f = m ? __ffs(m) - 1 : 32;
					hi = min(hi, lo + (f + 1) * step - 1);
					lo = min(hi, lo + f * step);
				}
				window = hi < kWalkLimit ? 0 : min(max(window, (unsigned int)NT), min(C, hi + 1));
			}
			else
				window = 0;
			if (lane == 0)
				s_window = window;
		}
		__syncthreads();
		// where a commit takes the position of its source
		auto moveTarget = [&](unsigned int r0, unsigned int i0, unsigned int i1) -> unsigned int {
			if (FULL && w.kind[i0] == kComplex)
				return complexTarget<IX>(r0, i1, w.remap, w.loop, w.loopback);
			if (w.kind[i0] == kSeam)
			{
				const unsigned int s0 = w.wedge[i0];
				IX s1 = w.loop[i0] == i1 ? w.loopback[s0] : w.loop[s0];
				s1 = s1 != kNone ? s1 : w.wedge[i1];
				return s0 == r0 ? (unsigned int)s1 : i1;
			}
			return i1;
		};
		auto stopReason = [&](float e, unsigned long long T, unsigned long long F, unsigned int M) -> unsigned int {
			if (e > error_limit)
				return 1;
			if (T >= goal)
				return 2;
			if (T > goal / 6 && e > __uint_as_float(M))
			{
				const unsigned long long eg = goal / 2 + F;
				const float error_goal = eg < C ? 1.5f * __uint_as_float(w.cerr[w.order[eg]]) : FLT_MAX;
				if (e > error_goal)
					return 3;
			}
			return 0;
		};
		const unsigned int window = s_window; // 0: walked
		if (tid == 0)
			s_walk[0] = 0, s_walk[1] = 0, s_walk[2] = 0, s_walk[3] = __float_as_uint(result_error);
		if (!window)
		{
			if (warp == 0)
			{
				unsigned int T = 0, F = 0, M = __float_as_uint(result_error), base = 0;
				bool stopped = false;
				for (; base < min(C, kWalkEnd) && !stopped; base += 32)
				{
					unsigned int i0 = 0, i1 = 0, r0 = 0, r1 = 0, eb = 0;
					if (base + lane < C)
					{
						const unsigned int c = w.order[base + lane];
						i0 = w.cv0[c], i1 = w.cv1[c], eb = w.cerr[c];
						r0 = w.remap[i0], r1 = w.remap[i1];
					}
					const float err = __uint_as_float(eb);
					const unsigned int tris = w.kind[i0] == kBorder ? 1u : 2u;
					unsigned int open = C - base < 32 ? (1u << (C - base)) - 1u : ~0u; // not passed yet
					while (open)
					{
						const bool locked = w.minT[r0] == 0 || w.minT[r1] == 0;
						const unsigned int stops = __ballot_sync(0xffffffffu, stopReason(err, T, F, M) != 0) & open;
						const unsigned int before = stops ? (stops & (0u - stops)) - 1u : ~0u;
						unsigned int todo = __ballot_sync(0xffffffffu, !locked) & open & before;
						if (!todo)
						{
							if (stops)
							{
								stopped = true;
								const unsigned int at = __ffs(stops) - 1;
								if (lane == at)
									s_cut = (unsigned long long)(base + at) << 2 | stopReason(err, T, F, M);
							}
							break;
						}
						// the first four at once, eight lanes each, as if each were the next
						unsigned int from[4];
						for (unsigned int g = 0; g < 4; ++g)
						{
							from[g] = todo ? __ffs(todo) - 1 : 32;
							todo &= todo - 1;
						}
						const unsigned int g = lane / 8, mine = g == 0 ? from[0] : (g == 1 ? from[1] : (g == 2 ? from[2] : from[3]));
						const unsigned int sub = lane & 7;
						const unsigned int q0 = __shfl_sync(0xffffffffu, r0, mine & 31), q1 = __shfl_sync(0xffffffffu, r1, mine & 31);
						// what the ones before it may move
						const unsigned int a0 = __shfl_sync(0xffffffffu, q0, 0), a1 = __shfl_sync(0xffffffffu, q1, 0);
						const unsigned int b0 = __shfl_sync(0xffffffffu, q0, 8), b1 = __shfl_sync(0xffffffffu, q1, 8);
						const unsigned int c0 = __shfl_sync(0xffffffffu, q0, 16), c1 = __shfl_sync(0xffffffffu, q1, 16);
						unsigned int after = 0; // bits of the ones before it whose commit it depends on
						if (q0 == a0 || q0 == a1 || q1 == a0 || q1 == a1)
							after |= 1;
						if (q0 == b0 || q0 == b1 || q1 == b0 || q1 == b1)
							after |= 2;
						if (q0 == c0 || q0 == c1 || q1 == c0 || q1 == c1)
							after |= 4;
						bool flip = false;
						if (mine < 32)
						{
							const float4 p0 = w.pos[q0], p1 = w.pos[q1];
							const V3 v0{p0.x, p0.y, p0.z}, v1{p1.x, p1.y, p1.z};
							const unsigned int e = w.adj_off[q0 + 1];
							for (unsigned int j = w.adj_off[q0] + sub; j < e; j += 8)
							{
								const IX2 ed = w.adj[j];
								const Mark mx = w.moved[ed.x], my = w.moved[ed.y];
								after |= (ed.x == a0 || ed.y == a0 ? 1u : 0u) | (ed.x == b0 || ed.y == b0 ? 2u : 0u) | (ed.x == c0 || ed.y == c0 ? 4u : 0u);
								const unsigned int va = mx != kFree ? (unsigned int)IX(mx) : (unsigned int)ed.x;
								const unsigned int vb = my != kFree ? (unsigned int)IX(my) : (unsigned int)ed.y;
								if (flip || va == q1 || vb == q1 || va == vb)
									continue;
								const float4 pa = w.pos[va], pb = w.pos[vb];
								flip = triFlip(V3{pa.x, pa.y, pa.z}, V3{pb.x, pb.y, pb.z}, v0, v1);
							}
						}
						after &= (1u << g) - 1u;
						const unsigned int flips = __ballot_sync(0xffffffffu, flip);
						const unsigned int after0 = __ballot_sync(0xffffffffu, after & 1), after1 = __ballot_sync(0xffffffffu, after & 2),
						                   after2 = __ballot_sync(0xffffffffu, after & 4);
						// in order, as long as none depends on a commit of these and the stop rules do not fire
						unsigned int commits = 0;
						for (unsigned int x = 0; x < 4; ++x)
						{
							if (from[x] == 32)
								break;
							const unsigned int group = 0xFFu << (x * 8);
							if (((commits & 1) && (after0 & group)) || ((commits & 2) && (after1 & group)) || ((commits & 4) && (after2 & group)))
								break;
							const unsigned int upto = 2u << from[x];
							if (x && (__ballot_sync(0xffffffffu, stopReason(err, T, F, M) != 0) & open & (upto - 1u)))
								break;
							open &= ~(upto - 1u);
							if (flips & group)
							{
								++F;
								continue;
							}
							commits |= 1u << x;
							T += __shfl_sync(0xffffffffu, tris, from[x]);
							const unsigned int me = __shfl_sync(0xffffffffu, eb, from[x]);
							if (__uint_as_float(me) == __uint_as_float(me))
								M = max(M, me);
						}
						bool commit = false;
						for (unsigned int x = 0; x < 4; ++x)
							commit |= (commits >> x & 1) && lane == from[x];
						if (commit)
						{
							const unsigned int k = base + lane;
							w.moved[r0] = Mark(k) << kTagShift | moveTarget(r0, i0, i1);
							w.minT[r0] = 0;
							w.minT[r1] = 0;
							w.status[k] = kCommit;
						}
						__syncwarp();
					}
				}
				if (lane == 0)
					s_walk[0] = stopped ? C : base, s_walk[1] = T, s_walk[2] = F, s_walk[3] = M;
			}
		}
		__syncthreads();
		if (s_walk[0] < C)
		{
			// rounds are numbered within the pass, which sets all marks free: a pass has at most a round per
			// candidate, and later rounds' tags are smaller
			unsigned int round = 0;
			auto mark = [&](unsigned int k, unsigned int r0, unsigned int r1) {
				const Mark m = ((kFree >> kTagShift) - (round + 1)) << kTagShift | k;
				atomicMin(&w.minT[r0], m);
				atomicMin(&w.minT[r1], m);
				atomicMin(&w.minS[r0], m);
			};
			unsigned int carryT = s_walk[1], carryF = s_walk[2], carryM = s_walk[3];
			unsigned int K0 = s_walk[0], K1 = min(C, K0 ? max(2 * K0, (unsigned int)NT) : window);
			for (;;)
			{
				// the warp's undecided candidates: beyond 32 a list in the warp's share of sort_tmp, then one per lane
				const unsigned int share = (K1 - K0) / (NT / 32), extra = (K1 - K0) % (NT / 32);
				IX* const list = w.sort_tmp + warp * share + min(warp, extra);
				unsigned int n = share + (warp < extra);
				unsigned int lk = 0, lr0 = 0, lr1 = 0;
				for (unsigned int x = lane; x < n; x += 32)
				{
					lk = K0 + x * (NT / 32) + warp;
					const unsigned int c = w.order[lk];
					lr0 = w.remap[w.cv0[c]], lr1 = w.remap[w.cv1[c]];
					list[x] = IX(lk);
					mark(lk, lr0, lr1);
				}
				bool inlanes = n <= 32;
				const unsigned int rounds = round + K1 - K0;
				__syncthreads();
				for (;;)
				{
					++round;
					const Mark tag = ((kFree >> kTagShift) - round) << kTagShift;
					for (unsigned int base = 0; base < n; base += 32)
					{
						// the earliest on both endpoints go on to the flip test (one a commit took is decided below)
						bool pass = false;
						if (base + lane < n)
						{
							if (!inlanes)
							{
								lk = list[base + lane];
								const unsigned int c = w.order[lk];
								lr0 = w.remap[w.cv0[c]], lr1 = w.remap[w.cv1[c]];
							}
							pass = w.minT[lr0] == (tag | lk) && w.minT[lr1] == (tag | lk);
						}
						unsigned int todo = __ballot_sync(0xffffffffu, pass);
						while (todo)
						{
							// four at a time, eight lanes each. One walk over the one-ring: an undecided earlier
							// candidate that moves a vertex of it makes the candidate wait; else the flip test sees
							// the ring as moved by earlier commits, and the candidate is rejected or commits
							unsigned int from = 32;
							for (unsigned int g = 0; g < 4; ++g)
							{
								if (lane / 8 == g && todo)
									from = __ffs(todo) - 1;
								todo &= todo - 1;
							}
							const bool valid = from < 32;
							const unsigned int k = __shfl_sync(0xffffffffu, lk, from & 31), r0 = __shfl_sync(0xffffffffu, lr0, from & 31),
							                   r1 = __shfl_sync(0xffffffffu, lr1, from & 31);
							const unsigned int sub = lane & 7, group = 0xFFu << (lane & 24);
							unsigned int b = 0, e = 0;
							if (valid)
								b = w.adj_off[r0], e = w.adj_off[r0 + 1];
							const float4 a0 = w.pos[r0], a1 = w.pos[r1];
							const V3 v0{a0.x, a0.y, a0.z}, v1{a1.x, a1.y, a1.z};
							bool wait = false, flip = false;
							auto waits = [&](unsigned int v) {
								const Mark m = w.minS[v];
								return m >= tag && m < (tag | k);
							};
							auto now = [&](unsigned int v) {
								const Mark m = ((volatile Mark*)w.moved)[v];
								return (unsigned int)(m >> kTagShift) < k ? (unsigned int)IX(m) : v;
							};
							for (unsigned int j = b + sub; j < e; j += 8)
							{
								const IX2 ed = w.adj[j];
								wait |= waits(ed.x) | waits(ed.y);
								const unsigned int va = now(ed.x), vb = now(ed.y);
								if (wait || flip || va == r1 || vb == r1 || va == vb)
									continue;
								const float4 pa = w.pos[va], pb = w.pos[vb];
								flip = triFlip(V3{pa.x, pa.y, pa.z}, V3{pb.x, pb.y, pb.z}, v0, v1);
							}
							wait = (__ballot_sync(0xffffffffu, wait) & group) != 0;
							flip = (__ballot_sync(0xffffffffu, flip) & group) != 0;
							if (valid && !wait && sub == 0)
							{
								unsigned char decision = kSkipFlip;
								if (!flip)
								{
									const unsigned int c = w.order[k], i0 = w.cv0[c], i1 = w.cv1[c];
									w.moved[r0] = Mark(k) << kTagShift | moveTarget(r0, i0, i1);
									w.minT[r0] = 0;
									w.minT[r1] = 0;
									decision = kCommit;
								}
								w.status[k] = decision;
							}
							__syncwarp();
						}
					}
					__syncthreads();
					// the candidates still undecided: locked if a commit took an endpoint (any commit on one is
					// earlier), else they mark for the next round; the list closes up in place
					unsigned int left = 0;
					for (unsigned int base = 0; base < n; base += 32)
					{
						bool keep = false;
						if (base + lane < n)
						{
							if (!inlanes)
								lk = list[base + lane];
							if (w.status[lk] == kUndecided)
							{
								if (!inlanes)
								{
									const unsigned int c = w.order[lk];
									lr0 = w.remap[w.cv0[c]], lr1 = w.remap[w.cv1[c]];
								}
								keep = w.minT[lr0] != 0 && w.minT[lr1] != 0;
								if (keep)
									mark(lk, lr0, lr1);
								else
									w.status[lk] = kSkipLocked;
							}
						}
						const unsigned int m = __ballot_sync(0xffffffffu, keep);
						if (inlanes)
						{
							// undecided ones stay in their lanes
							n = m ? 32 - __clz(m) : 0;
							left = n;
						}
						else
						{
							if (keep)
								list[left + __popc(m & ((1u << lane) - 1u))] = IX(lk);
							left += __popc(m);
							__syncwarp();
						}
					}
					if (!inlanes && left <= 32)
					{
						inlanes = true;
						if (lane < left)
						{
							lk = list[lane];
							const unsigned int c = w.order[lk];
							lr0 = w.remap[w.cv0[c]], lr1 = w.remap[w.cv1[c]];
						}
					}
					n = left;
					if (!__syncthreads_or(left != 0))
						break;
					if (round >= rounds)
					{
						if (tid == 0)
							s_stall = 1;
						break;
					}
				}
				__syncthreads();
				// stop rules over [K0, K1): contiguous thread chunks, block scan, carried prefix
				const unsigned int len = K1 - K0, per = (len + NT - 1) / NT;
				const unsigned int t0 = min(K1, K0 + tid * per), t1 = min(K1, t0 + per);
				unsigned int sT = 0, sF = 0, sM = 0;
				for (unsigned int k = t0; k < t1; ++k)
				{
					unsigned char st = w.status[k];
					unsigned int c = w.order[k];
					float e = __uint_as_float(w.cerr[c]);
					if (st == kCommit)
					{
						sT += w.kind[w.cv0[c]] == kBorder ? 1u : 2u;
						if (e == e)
							sM = max(sM, w.cerr[c]);
					}
					sF += st == kSkipFlip;
				}
				const uint3 sums = blockScan3(sT, sF, sM, s_sums);
				unsigned long long T = (unsigned long long)carryT + sT, F = (unsigned long long)carryF + sF;
				unsigned int M = max(carryM, sM);
				for (unsigned int k = t0; k < t1; ++k)
				{
					unsigned int c = w.order[k];
					float e = __uint_as_float(w.cerr[c]);
					const unsigned int reason = stopReason(e, T, F, M);
					if (reason)
					{
						atomicMin(&s_cut, ((unsigned long long)k << 2) | reason);
						break;
					}
					unsigned char st = w.status[k];
					if (st == kCommit)
					{
						T += w.kind[w.cv0[c]] == kBorder ? 1u : 2u;
						if (e == e)
							M = max(M, w.cerr[c]);
					}
					F += st == kSkipFlip;
				}
				__syncthreads();
				if (s_cut != ~0ull || K1 == C || s_stall)
					break;
				carryT += sums.x;
				carryF += sums.y;
				carryM = max(carryM, sums.z);
				K0 = K1;
				K1 = (unsigned int)min((unsigned long long)C, 2ull * K1);
			}
		}
		// apply the committed prefix: collapse_remap writes, done count, result error
		{
			const unsigned int cut = s_cut == ~0ull ? C : (unsigned int)(s_cut >> 2);
			unsigned int done = 0, em = 0;
			for (unsigned int k = tid; k < cut; k += NT)
			{
				if (w.status[k] != kCommit)
					continue;
				unsigned int c = w.order[k];
				unsigned int i0 = w.cv0[c], i1 = w.cv1[c];
				if (FULL && w.kind[i0] == kComplex)
				{
					unsigned int v = i0;
					do
					{
						w.cr[v] = IX(complexTarget<IX>(v, i1, w.remap, w.loop, w.loopback));
						v = w.wedge[v];
					} while (v != i0);
				}
				else if (w.kind[i0] == kSeam)
				{
					unsigned int s0 = w.wedge[i0];
					IX s1 = w.loop[i0] == i1 ? w.loopback[s0] : w.loop[s0];
					s1 = s1 != kNone ? s1 : w.wedge[i1];
					w.cr[i0] = IX(i1);
					w.cr[s0] = s1;
				}
				else
					w.cr[i0] = IX(i1);
				done++;
				float e = __uint_as_float(w.cerr[c]);
				if (e == e)
					em = max(em, w.cerr[c]);
			}
			done = __reduce_add_sync(0xffffffffu, done);
			em = __reduce_max_sync(0xffffffffu, em);
			if ((tid & 31) == 0 && done)
			{
				atomicAdd(&s_done, done);
				atomicMax(&s_errbits, em);
			}
		}
		__syncthreads();
		result_error = __uint_as_float(s_errbits);
		passes++;
		if (s_done == 0 || s_stall)
			break;

		// updateQuadrics (:1638-1673): every target receives at most one source per pass. The
		// moved wedges of one commit all belong to its source position (whose primary always
		// moves), and no other commit targets their targets, so each moved primary merges the
		// attribute quadrics of its wedges in increasing vertex order, as the reference's vertex
		// loop does
		for (unsigned int i = tid; i < V; i += NT)
		{
			unsigned int t = w.cr[i];
			if (t == i || w.remap[i] != i)
				continue;
			unsigned int r1 = w.remap[t];
			Quadric Q = ldquadric(w.vq, r1);
			qadd(Q, ldquadric(w.vq, i));
			stquadric(w.vq, r1, Q);
			if constexpr (FULL)
			{
				if (ac)
				{
					unsigned int last = 0;
					bool firstw = true;
					for (;;)
					{
						unsigned int best = ~0u, v = i;
						do
						{
							if ((firstw || v > last) && v < best)
								best = v;
							v = w.wedge[v];
						} while (v != i);
						if (best == ~0u)
							break;
						unsigned int tb = w.cr[best];
						if (tb != best)
						{
							Quadric A = ldquadric(w.aq, tb);
							qadd(A, ldquadric(w.aq, best));
							stquadric(w.aq, tb, A);
							for (unsigned int q = 0; q < ac; ++q)
							{
								float4 g = w.ag[(size_t)tb * ac + q], h = w.ag[(size_t)best * ac + q];
								g.x += h.x, g.y += h.y, g.z += h.z, g.w += h.w;
								w.ag[(size_t)tb * ac + q] = g;
							}
						}
						last = best;
						firstw = false;
					}
				}
			}
		}
		// remapEdgeLoops (:1845-1864), in place
		for (unsigned int i = tid; i < V; i += NT)
		{
			IX* arrs[2] = {w.loop, w.loopback};
			for (int q = 0; q < 2; ++q)
			{
				IX* L = arrs[q];
				const IX l = L[i];
				if (l == kNone)
					continue;
				const IX r = w.cr[l];
				if (i == r)
				{
					const IX ll = L[l];
					L[i] = ll != kNone ? w.cr[ll] : kNone;
				}
				else
					L[i] = r;
			}
		}
		__syncthreads();
		// remapIndexBuffer (:1811-1843): in-place order-preserving compaction by chunks
		unsigned int written = 0;
		for (unsigned int base = 0; base < T; base += NT)
		{
			unsigned int t = base + tid;
			unsigned int v0 = 0, v1 = 0, v2 = 0;
			bool keep = false;
			if (t < T)
			{
				v0 = w.cr[w.idx[t * 3]], v1 = w.cr[w.idx[t * 3 + 1]], v2 = w.cr[w.idx[t * 3 + 2]];
				unsigned int r0 = w.remap[v0], r1 = w.remap[v1], r2 = w.remap[v2];
				keep = r0 != r1 && r0 != r2 && r1 != r2;
			}
			unsigned int tot;
			unsigned int ex = blockExclusiveScan<NT>(keep ? 1u : 0u, red, &tot);
			if (keep)
			{
				unsigned int o = (written + ex) * 3;
				w.idx[o] = IX(v0), w.idx[o + 1] = IX(v1), w.idx[o + 2] = IX(v2);
			}
			written += tot;
			__syncthreads();
		}
		result_count = written * 3;
	}

	for (unsigned int i = tid; i < result_count; i += NT)
		d.out[i] = src(w.idx[i]);
	if (tid == 0)
		*out = BatchResult{result_count, sqrtf(result_error) * error_scale, passes, (s_stall ? 3u : 0u) | kWhere | (beyondExpected(V, I, s_cap, sparse) ? kBatchBeyond : 0u)};
	return true;
}

// The kernel's forms: lean and full, 16-bit ids in 128, 256 or 512 threads, 32-bit ids in 512. Warps per
// SM they are compiled for: full meshes too large for shared memory wait on their slab, so their form (128
// threads) wants warps more than registers (2,048 groups of 1,024 triangles in the slab with 16 / 20 / 24 /
// 32 / 40 warps: 3.68 / 3.50 / 3.32 / 2.95 / 2.98 ms); the others sum attribute gradients in registers.
template <int NT, bool FULL>
constexpr int kBatchWarps = NT == 512 ? (FULL ? 16 : 32) : (FULL && NT == 128 ? 32 : 16);

template <int NT, bool FULL, class IX>
__global__ void __launch_bounds__(NT, (kBatchWarps<NT, FULL>) * 32 / NT) kBatch(const BatchDesc* __restrict__ descs, unsigned int count, unsigned int* ticket,
    BatchResult* results, char* slabs, size_t slab_bytes, unsigned int smem_bytes)
{
	__shared__ unsigned int s_job;
	char* const slab = slabs + (size_t)blockIdx.x * slab_bytes;
	for (;;)
	{
		if (threadIdx.x == 0)
			s_job = atomicAdd(ticket, 1u);
		__syncthreads();
		unsigned int job = s_job;
		if (job >= count)
			break;
		const BatchDesc d = descs[job];
		// in shared memory, its attribute rows there or in the slab; where that is too small, in the slab (a
		// mesh that needs 32-bit ids is larger than any shared memory)
		const size_t bound = localVertexBound(d.index_count, d.vertex_count, FULL && (d.options & kOptSparse) != 0);
		// (a launch without slabs has shared memory for the most any of its meshes can need)
		const size_t rows = FULL && d.ac ? min(rowBytes<IX>(bound, d.ac), slab_bytes) : 0;
		bool done = false;
		if constexpr (sizeof(IX) == 2)
		{
			done = simplifyMesh<NT, FULL, IX, true>(d, &results[job], Region(nullptr, smem_bytes), Region(slab, rows));
			__syncthreads();
		}
		if (!done)
			done = simplifyMesh<NT, FULL, IX, false>(d, &results[job], Region(slab + rows, slab_bytes - rows), Region(slab, rows));
		if (!done && threadIdx.x == 0)
			results[job] = BatchResult{0, 0.f, 0, 4};
		__syncthreads();
	}
}

} // namespace

} // namespace mogpu
