// mo_meshlets.cu - meshopt_buildMeshletsFlex (src/clusterizer.cpp:1035-1224) for many index
// subsets of one vertex buffer: the re-clusterization a cluster-LOD builder runs on every
// simplified group (demo/clusterlod.h:266-296).
//
// The algorithm is a serial greedy: every step appends the best triangle next to the current
// meshlet, and the choice depends on all earlier ones. Here one warp builds one group's meshlets,
// and groups run side by side. Inside a group, lane 0 runs the order-dependent bookkeeping (the
// area sum, the kd-tree, seeds, appends, list removal) exactly as the reference orders it, and
// the warp shares the wide steps:
//  - group-local vertex ids in first-use order (a hash table keyed by vertex, a warp scan);
//  - every vertex's triangle list in face order (ranks among equal vertices from match_any, so
//    corners enter their lists in corner order, as the reference's fill loop does);
//  - the triangle cones; the kd-tree, built only when a step first needs it;
//  - the neighbour search of every step. The reference scans the live triangle lists of all
//    meshlet vertices; here the distinct triangles in them are kept as a frontier, and the lanes
//    score those. The smallest (priority, score) is the reference's first best triangle unless
//    two tie exactly; then the tied ones' scan positions (meshlet vertex, list entry) decide. A
//    NaN score breaks that ordering, so a step that meets one is scanned again by lane 0 alone,
//    in the reference's order;
//  - the list removals and frontier insertions of the appended triangle;
//  - each meshlet vertex's best seed neighbour when a meshlet ends.
// The reference keys its per-vertex arrays by the caller's vertex index; nothing in its result
// depends on that numbering, only on vertex identity and on the order vertices enter a meshlet,
// so group-local ids give the same meshlets.
//
// A step is a chain of dependent instructions (one issue in 7 cycles per warp, three warps per
// scheduler), and a level takes about one group's chain, so what counts is the instructions of a
// step and that every group of a level is resident: the arrays that steps write are packed into
// shared memory (16-bit ids in groups below 65,535 corners: 13 KB for 512 triangles, 14 groups per
// SM). 2,048 simplified groups of 512 triangles with the reorder, whole call: 5.84 ms with all
// meshlet vertices' lists scanned at every step, lane 0 doing the appends and the tree built for
// every group; 1.48 ms now (1.92 with the lists and the reorder's shifts still on lane 0; 0.1 more
// with every array in the group's scratch).
#include "mo_meshlets.cuh"
#include "mo_common.cuh"
#include "mo_prims.cuh"
#include "mo_probe.cuh"

#include <algorithm>
#include <float.h>
#include <type_traits>

namespace mogpu
{

namespace
{

constexpr unsigned int kMaxSeeds = 256; // kMeshletMaxSeeds, :27
constexpr unsigned int kAddSeeds = 4;   // kMeshletAddSeeds, :28
constexpr int kMaxDepth = 50;           // kMeshletMaxTreeDepth, :31
constexpr unsigned int kLeafSize = 8;   // :1090
#ifndef MO_FLEX_POOL_MAX
#define MO_FLEX_POOL_MAX 40960
#endif
constexpr size_t kPoolMax = MO_FLEX_POOL_MAX; // shared memory of one group at most
#ifndef MO_FLEX_TABLE_MAX
#define MO_FLEX_TABLE_MAX 16384
#endif
constexpr size_t kPoolTableMax = MO_FLEX_TABLE_MAX; // ... of its vertex table

struct Cone
{
	float px, py, pz, nx, ny, nz;
};

// kd-tree node (:473-485): axis 3 = leaf of `children` points (this node and the ones after);
// a branch's right subtree starts children + 1 nodes after it
struct KDNode
{
	unsigned int word; // split (float bits) or point index
	unsigned int axis;
	unsigned int children;
};

size_t align256(size_t n)
{
	return (n + 255) & ~size_t(255);
}

__host__ __device__ inline unsigned int tableSize(unsigned int I)
{
	unsigned int h = 64;
	while (h < 2 * I)
		h *= 2;
	return h;
}

// per-triangle and per-vertex words of a group, in 16 bits where every id and count fits
struct Narrow
{
	typedef unsigned short Id;
	typedef ushort2 Vertex;
	typedef ushort4 Triangle;
};

struct Wide
{
	typedef unsigned int Id;
	typedef uint2 Vertex;
	typedef uint4 Triangle;
};

// states of a triangle
enum : unsigned char
{
	kTriFree = 0,     // live, not next to the current meshlet
	kTriFrontier = 1, // live, in the frontier
	kTriEmitted = 2,
};

// one group's scratch, carved from its base in a fixed order (host and device agree)
template <class K>
struct Scratch
{
	typedef typename K::Id Id;
	unsigned int *hkey, *gid, *vbest, *seeds, *kdrank;
	Id *hid, *hcnt, *lid, *lpos; // hash table: local id per slot; corners per vertex; per corner: vertex, place in its list
	Id *adj, *off, *kdidx, *kdtmp;
	typename K::Vertex* vert;  // {live triangles, index in the current meshlet (all ones: none)}
	typename K::Triangle* tri; // {vertices}
	unsigned char* state;      // of each triangle
	// the frontier, its first kFrontSlots triangles and the others: {vertices, triangle} and apex
	typename K::Triangle *front, *front_more;
	float *apex, *apex_more; // apex x of every slot, then y, then z
	unsigned int more;       // stride of apex_more
	float *cent, *norm;      // cone apex and axis, 3 floats per triangle
	float* area;
	KDNode* nodes;
	Id* mvl;             // the current meshlet's vertices
	unsigned char* mtri; // and its triangles, as places among them

	static __device__ __forceinline__ Id none() { return Id(~0u); }
};

constexpr unsigned int kFrontSlots = 128; // a multiple of the warp; a 128-triangle meshlet's frontier is 20 to 60

// the arrays that steps write, for shared memory (a line of L1 that is stored to is read again from
// L2, while the arrays that only setup writes stay in L1)
template <class K>
__host__ __device__ inline size_t carveHot(Scratch<K>& s, char* base, unsigned int F, unsigned int U)
{
	size_t o = 0;
	auto take = [&](auto*& ptr, size_t count) {
		if (base)
			ptr = reinterpret_cast<std::remove_reference_t<decltype(ptr)>>(base + o);
		o += (count * sizeof(*ptr) + 15) & ~size_t(15);
	};
	take(s.front, kFrontSlots);
	take(s.apex, kFrontSlots * 3);
	take(s.vert, U);
	take(s.adj, size_t(F) * 3);
	take(s.tri, F);
	take(s.state, F);
	take(s.off, U);
	return o;
}

// slots of the vertex table in shared memory, where it fits there before the arrays above
__host__ __device__ inline unsigned int sharedTableSize(unsigned int I)
{
	unsigned int h = 64;
	while (h < I + I / 4)
		h *= 2;
	return h;
}

template <class K>
__host__ __device__ inline size_t carve(Scratch<K>& s, char* base, unsigned int I)
{
	typedef typename K::Id Id;
	const unsigned int F = I / 3, H = tableSize(I);
	size_t o = 0;
	auto take = [&](auto*& ptr, size_t count) {
		ptr = base ? reinterpret_cast<std::remove_reference_t<decltype(ptr)>>(base + o) : nullptr;
		o += (count * sizeof(*ptr) + 15) & ~size_t(15);
	};
	take(s.hkey, H);
	take(s.hid, H);
	take(s.hcnt, I);
	take(s.lid, I);
	take(s.lpos, I);
	take(s.gid, I);
	take(s.vbest, 256 * 3);
	take(s.seeds, kMaxSeeds);
	take(s.kdrank, F);
	take(s.adj, I);
	take(s.off, I);
	take(s.kdidx, F);
	take(s.kdtmp, F);
	take(s.vert, I);
	take(s.tri, F);
	take(s.state, F);
	take(s.front, kFrontSlots);
	take(s.front_more, F);
	take(s.apex, kFrontSlots * 3);
	take(s.apex_more, size_t(F) * 3);
	s.more = F;
	take(s.cent, size_t(F) * 3);
	take(s.norm, size_t(F) * 3);
	take(s.area, F);
	take(s.nodes, size_t(F) * 2);
	take(s.mvl, 256);
	take(s.mtri, 512 * 3);
	return o;
}

__device__ __forceinline__ unsigned int hashVertex(unsigned int v)
{
	v ^= v >> 16;
	v *= 0x7feb352du;
	v ^= v >> 15;
	v *= 0x846ca68bu;
	v ^= v >> 16;
	return v;
}

__device__ __forceinline__ float dist3(float ax, float ay, float az, float bx, float by, float bz)
{
	float dx = ax - bx, dy = ay - by, dz = az - bz;
	return sqrtf(dx * dx + dy * dy + dz * dz);
}

// getMeshletScore, :173-179
__device__ __forceinline__ float meshletScore(float distance, float spread, float cone_weight, float expected_radius)
{
	float cone = 1.f - spread * cone_weight;
	float clamped = cone < 1e-3f ? 1e-3f : cone;
	return (1 + distance / expected_radius * (1 - cone_weight)) * clamped;
}

// topology priority of a candidate triangle (:318-335)
template <class K>
__device__ __forceinline__ int neighborPriority(const Scratch<K>& s, const typename K::Triangle& t)
{
	const typename K::Vertex a = s.vert[t.x], b = s.vert[t.y], c = s.vert[t.z];
	const typename K::Id no = Scratch<K>::none();
	int extra = (a.y == no) + (b.y == no) + (c.y == no);
	unsigned int la = a.x, lb = b.x, lc = c.x;
	if (extra == 0)
		return 0;
	if (la == 1 || lb == 1 || lc == 1)
		return 1;
	if ((la == 2) + (lb == 2) + (lc == 2) >= 2)
		return 1 + extra;
	return 2 + extra;
}

// what a step scores triangles with. With a cone weight of 0 the axes cancel out of the score
// (1 - spread * 0 is 1 for any finite spread), so they are read only otherwise, or where one of the
// group's is not finite.
struct ScoreArgs
{
	Cone mc;
	float cone_weight, radius;
	bool axes;
};

template <class K>
__device__ __forceinline__ float neighborScore(const Scratch<K>& s, unsigned int t, float x, float y, float z, const ScoreArgs& a)
{
	float distance = dist3(x, y, z, a.mc.px, a.mc.py, a.mc.pz);
	float spread = 0.f;
	if (a.axes)
	{
		const float* n = s.norm + (size_t)t * 3;
		spread = n[0] * a.mc.nx + n[1] * a.mc.ny + n[2] * a.mc.nz;
	}
	return meshletScore(distance, spread, a.cone_weight, a.radius);
}

// slot i of the frontier
template <class K>
__device__ __forceinline__ typename K::Triangle frontAt(const Scratch<K>& s, unsigned int i, float& x, float& y, float& z)
{
	if (i < kFrontSlots)
	{
		x = s.apex[i], y = s.apex[kFrontSlots + i], z = s.apex[2 * kFrontSlots + i];
		return s.front[i];
	}
	const float* m = s.apex_more + (i - kFrontSlots);
	x = m[0], y = m[s.more], z = m[2 * (size_t)s.more];
	return s.front_more[i - kFrontSlots];
}

template <class K>
__device__ __forceinline__ void frontSet(const Scratch<K>& s, unsigned int i, const typename K::Triangle& f, float x, float y, float z)
{
	if (i < kFrontSlots)
	{
		s.apex[i] = x, s.apex[kFrontSlots + i] = y, s.apex[2 * kFrontSlots + i] = z;
		s.front[i] = f;
		return;
	}
	float* m = s.apex_more + (i - kFrontSlots);
	m[0] = x, m[s.more] = y, m[2 * (size_t)s.more] = z;
	s.front_more[i - kFrontSlots] = f;
}

// getNeighborTriangle, :302-362, in the reference's scan order (lane 0 only)
template <class K>
__device__ unsigned int neighborSerial(const Scratch<K>& s, unsigned int vcount, const ScoreArgs& a)
{
	unsigned int best = ~0u;
	int best_priority = 5;
	float best_score = FLT_MAX;
	for (unsigned int i = 0; i < vcount; ++i)
	{
		unsigned int v = s.mvl[i];
		const typename K::Id* list = s.adj + s.off[v];
		const unsigned int n = s.vert[v].x;
		for (unsigned int j = 0; j < n; ++j)
		{
			unsigned int t = list[j];
			int priority = neighborPriority(s, s.tri[t]);
			if (priority > best_priority)
				continue;
			const float* c = s.cent + (size_t)t * 3;
			float score = neighborScore(s, t, c[0], c[1], c[2], a);
			if (priority < best_priority || score < best_score)
			{
				best = t;
				best_priority = priority;
				best_score = score;
			}
		}
	}
	return best;
}

// floats (no NaN, no -0) as unsigned integers of the same order
__device__ __forceinline__ unsigned int orderedBits(float f)
{
	const unsigned int u = __float_as_uint(f);
	return u ^ ((unsigned int)((int)u >> 31) | 0x80000000u);
}

// The same choice from the frontier by the whole warp; *slot is its place there. *nan is set when a
// score was NaN (the warp's answer is then not the reference's).
template <class K>
__device__ unsigned int neighborWarp(const Scratch<K>& s, unsigned int fn, const ScoreArgs& a, unsigned int* slot, bool* nan)
{
	const unsigned int lane = threadIdx.x & 31;
	unsigned int best = ~0u, at = 0;
	int bp = 6;
	float bs = FLT_MAX;
	bool sawnan = false, tie = false;
	for (unsigned int i = lane; i < fn; i += 32)
	{
		float x, y, z;
		const typename K::Triangle f = frontAt(s, i, x, y, z);
		const int priority = neighborPriority(s, f);
		if (priority > bp)
			continue;
		const float score = neighborScore(s, f.w, x, y, z, a) + 0.f;
		sawnan |= score != score;
		if (priority < bp || score < bs)
		{
			best = f.w;
			at = i;
			bp = priority;
			bs = score;
			tie = false;
		}
		else
			tie |= score == bs;
	}
	// one reduction where the best scores are all in [1, 2^64): then (priority, score) fits a word
	const unsigned int from1 = __float_as_uint(bs) - 0x3f800000u;
	unsigned int win;
	int P;
	if (__any_sync(0xffffffffu, sawnan || (best != ~0u && from1 >> 29)))
	{
		*nan = __any_sync(0xffffffffu, sawnan);
		P = (int)__reduce_min_sync(0xffffffffu, (unsigned int)bp);
		const unsigned int key = bp == P && best != ~0u ? orderedBits(bs) : ~0u;
		const unsigned int least = __reduce_min_sync(0xffffffffu, key);
		win = __ballot_sync(0xffffffffu, best != ~0u && key == least);
	}
	else
	{
		*nan = false;
		const unsigned int key = best != ~0u ? (unsigned int)bp << 29 | from1 : ~0u;
		const unsigned int least = __reduce_min_sync(0xffffffffu, key);
		win = __ballot_sync(0xffffffffu, key == least);
		P = (int)(least >> 29);
	}
	if ((win & (win - 1)) || (fn > 32 && __any_sync(0xffffffffu, tie && (win >> lane & 1u))))
	{
		const unsigned int Kmin = orderedBits(__shfl_sync(0xffffffffu, bs, __ffs(win) - 1));
		// several are equally good: the first one in scan order
		unsigned long long first = ~0ull;
		for (unsigned int i = lane; i < fn; i += 32)
		{
			float px, py, pz;
			const typename K::Triangle tr = frontAt(s, i, px, py, pz);
			const unsigned int t = tr.w;
			if (neighborPriority(s, tr) != P || orderedBits(neighborScore(s, t, px, py, pz, a) + 0.f) != Kmin)
				continue;
			const typename K::Vertex va = s.vert[tr.x], vb = s.vert[tr.y], vc = s.vert[tr.z];
			unsigned int v = tr.x, y = va.y;
			if (vb.y < y)
				v = tr.y, y = vb.y;
			if (vc.y < y)
				v = tr.z, y = vc.y;
			const typename K::Id* list = s.adj + s.off[v];
			unsigned int j = 0;
			for (const unsigned int n = s.vert[v].x; j < n && list[j] != t; ++j)
				;
			const unsigned long long key64 = (unsigned long long)y << 32 | j;
			if (key64 < first)
			{
				first = key64;
				best = t;
				at = i;
			}
		}
		unsigned long long m = first;
		for (int o = 16; o > 0; o >>= 1)
		{
			const unsigned long long x = __shfl_xor_sync(0xffffffffu, m, o);
			m = x < m ? x : m;
		}
		const unsigned int w = __ffs(__ballot_sync(0xffffffffu, first == m)) - 1;
		*slot = __shfl_sync(0xffffffffu, at, w);
		return __shfl_sync(0xffffffffu, best, w);
	}
	const unsigned int w = __ffs(win) - 1;
	*slot = __shfl_sync(0xffffffffu, at, w);
	return __shfl_sync(0xffffffffu, best, w);
}

// kdtreeBuild, :532-581, depth first on an explicit stack, by the whole warp: a subtree's nodes
// start where the previous one in that order ended, and a right subtree records its distance from
// its parent when it starts, which is after the whole left subtree. Every lane holds the stack.
// The statistics run in point order, one axis per lane, on points the warp loads 32 at a time.
template <class K>
__device__ void kdBuild(const Scratch<K>& s, unsigned int F, unsigned int* err)
{
	typedef typename K::Id Id;
	// the points in the frontier's memory where they fit: it is empty when the tree is built
	Id* const points = size_t(F) * sizeof(Id) <= kFrontSlots * sizeof(typename K::Triangle) ? reinterpret_cast<Id*>(s.front) : s.kdidx;
	const unsigned int lane = threadIdx.x & 31, below = (1u << lane) - 1u;
	struct Task
	{
		unsigned int start, count, parent;
		int depth;
	} stack[kMaxDepth + 8];
	int top = 0;
	stack[top++] = Task{0, F, ~0u, 0};
	for (unsigned int i = lane; i < F; i += 32)
		points[i] = Id(i);
	__syncwarp();
	unsigned int next = 0;
	while (top > 0)
	{
		const Task t = stack[--top];
		const unsigned int offset = next;
		if (t.parent != ~0u && lane == 0)
			s.nodes[t.parent].children = offset - t.parent - 1;
		Id* idx = points + t.start;
		bool leaf = t.count <= kLeafSize;
		float split = 0.f;
		unsigned int axis = 0, middle = 0;
		if (!leaf)
		{
			// Welford's mean and sum of squares, :544-560: lane k (mod 3) runs axis k
			const unsigned int k = lane % 3;
			float mean = 0.f, var = 0.f;
			for (unsigned int base = 0; base < t.count; base += 32)
			{
				const unsigned int i = base + lane;
				const float* c = s.cent + (size_t)(i < t.count ? idx[i] : idx[0]) * 3;
				const float px = c[0], py = c[1], pz = c[2];
				const float runs = 1.f / float(i + 1);
				const unsigned int m = min(32u, t.count - base);
#pragma unroll 8
				for (unsigned int j = 0; j < m; ++j)
				{
					const float x = __shfl_sync(0xffffffffu, px, j), y = __shfl_sync(0xffffffffu, py, j), z = __shfl_sync(0xffffffffu, pz, j);
					const float r = __shfl_sync(0xffffffffu, runs, j);
					const float p = k == 0 ? x : (k == 1 ? y : z);
					float delta = p - mean;
					mean += delta * r;
					var += delta * (p - mean);
				}
			}
			const float v0 = __shfl_sync(0xffffffffu, var, 0), v1 = __shfl_sync(0xffffffffu, var, 1), v2 = __shfl_sync(0xffffffffu, var, 2);
			axis = (v0 >= v1 && v0 >= v2) ? 0 : (v1 >= v2 ? 1 : 2);
			split = __shfl_sync(0xffffffffu, mean, axis);
			// kdtreePartition, :487-506, swaps point i with the first point not below the split, for i
			// in order. Points below it end up in front in order. For the others, let f(j) be the point
			// at the boundary before step j: step i leaves f(i) in place i and makes f(i + 1) point i
			// itself, or, when that one is below the split, what step m + 1 left in place m + 1, where m
			// is the number of points below the split before i: f(i + 1) = f(m + 1).
			if (t.count <= 32)
			{
				const bool valid = lane < t.count;
				const Id x = valid ? idx[lane] : Id(0);
				const bool less = valid && s.cent[(size_t)x * 3 + axis] < split;
				const unsigned int bal = __ballot_sync(0xffffffffu, less);
				middle = __popc(bal);
				unsigned int j = lane == middle ? t.count : lane;
				if (lane >= middle && valid)
					while (bal >> (j - 1) & 1u)
						j = __popc(bal & ((1u << (j - 1)) - 1u)) + 1;
				const Id y = Id(__shfl_sync(0xffffffffu, (unsigned int)x, (j - 1) & 31));
				__syncwarp();
				if (less)
					idx[__popc(bal & below)] = x;
				if (valid && lane >= middle)
					idx[lane] = y;
				__syncwarp();
			}
			else
			{
				unsigned int m = 0;
				for (unsigned int base = 0; base < t.count; base += 32)
				{
					const unsigned int i = base + lane;
					const bool valid = i < t.count;
					const Id x = valid ? idx[i] : Id(0);
					const bool less = valid && s.cent[(size_t)x * 3 + axis] < split;
					const unsigned int bal = __ballot_sync(0xffffffffu, less);
					const unsigned int rank = m + __popc(bal & below);
					if (valid)
						s.kdrank[i] = rank << 1 | (less ? 1u : 0u);
					if (less)
						s.kdtmp[rank] = x;
					m += __popc(bal);
				}
				middle = m;
				__syncwarp();
				for (unsigned int q = middle + lane; q < t.count; q += 32)
				{
					unsigned int j = q == middle ? t.count : q; // the last boundary point, or f(q)
					for (unsigned int guard = 0; guard <= t.count; ++guard)
					{
						const unsigned int r = s.kdrank[j - 1];
						if (!(r & 1u))
							break;
						j = (r >> 1) + 1;
					}
					s.kdtmp[q] = idx[j - 1];
				}
				__syncwarp();
				for (unsigned int i = lane; i < t.count; i += 32)
					idx[i] = s.kdtmp[i];
				__syncwarp();
			}
			leaf = middle <= kLeafSize / 2 || middle >= t.count - kLeafSize / 2 || t.depth >= kMaxDepth;
		}
		if (leaf)
		{
			// kdtreeBuildLeaf, :508-530
			for (unsigned int i = lane; i < t.count; i += 32)
				s.nodes[offset + i] = KDNode{idx[i], 3u, i ? ~0u >> 2 : t.count};
			next = offset + t.count;
			continue;
		}
		if (lane == 0)
			s.nodes[offset] = KDNode{__float_as_uint(split), axis, 0u};
		next = offset + 1;
		if (top + 2 > kMaxDepth + 8)
		{
			if (lane == 0)
				atomicOr(err, 2u);
			break;
		}
		stack[top++] = Task{t.start + middle, t.count - middle, offset, t.depth + 1};
		stack[top++] = Task{t.start, middle, ~0u, t.depth + 1};
	}
	__syncwarp();
}

// kdtreeNearest, :583-639, on an explicit stack in the recursion's order (lane 0): a branch
// leaves "its second child, if the split is within the best distance then" under its first
// child; emptied leaves and branches are switched off on the way
template <class K>
__device__ void kdNearest(const Scratch<K>& s, const float* pos, unsigned int* result, float* limit)
{
	struct Frame
	{
		unsigned int node;
		float dist; // >= 0: a deferred second child, visited if dist <= limit; < 0: visit
	} stack[2 * kMaxDepth + 8];
	int top = 0;
	stack[top++] = Frame{0, -1.f};
	while (top > 0)
	{
		Frame f = stack[--top];
		if (f.dist >= 0.f && !(f.dist <= *limit))
			continue;
		const unsigned int root = f.node;
		KDNode& node = s.nodes[root];
		if (node.children == 0)
			continue;
		if (node.axis == 3)
		{
			bool inactive = true;
			for (unsigned int i = 0; i < node.children; ++i)
			{
				unsigned int index = s.nodes[root + i].word;
				if (s.state[index] == kTriEmitted)
					continue;
				inactive = false;
				const float* c = s.cent + (size_t)index * 3;
				float d = dist3(c[0], c[1], c[2], pos[0], pos[1], pos[2]);
				if (d < *limit)
				{
					*result = index;
					*limit = d;
				}
			}
			if (inactive)
				node.children = 0;
		}
		else
		{
			float delta = pos[node.axis] - __uint_as_float(node.word);
			unsigned int first = (delta <= 0) ? 0 : node.children;
			unsigned int second = first ^ node.children;
			if ((s.nodes[root + 1 + first].children | s.nodes[root + 1 + second].children) == 0)
				node.children = 0;
			if (top + 2 > 2 * kMaxDepth + 8)
				return;
			// a NaN delta is never <= limit, so that child is skipped as the recursion skips it
			stack[top++] = Frame{root + 1 + second, delta != delta ? FLT_MAX : fabsf(delta)};
			stack[top++] = Frame{root + 1 + first, -1.f};
		}
	}
}

// kdtreeNearest without the tree: the nearest live triangle, by the whole warp. The search finds a
// triangle at the smallest distance: a subtree it skips lies beyond a plane further away than the
// best so far, and rounding keeps that order (no distance is below its own axis difference, which
// is not below the plane's) while no square over- or underflows. So a single nearest triangle is the
// search's result; with several equally near ones, or values outside that range (*sure = false),
// its order decides.
// A tree cost 0.65M cycles per group of 512 triangles and its search 0.15M; a scan takes 5k.
constexpr unsigned int kNearestScan = 4096; // triangles of a group at most: above, the tree's search is shorter
template <class K>
__device__ unsigned int nearestScan(const Scratch<K>& s, unsigned int F, const Cone& mc, float* distance, bool* sure)
{
	const unsigned int lane = threadIdx.x & 31;
	unsigned int best = ~0u;
	float bd = FLT_MAX;
	bool tie = false;
#pragma unroll 4
	for (unsigned int t = lane; t < F; t += 32)
	{
		if (s.state[t] == kTriEmitted)
			continue;
		const float* c = s.cent + (size_t)t * 3;
		const float d = dist3(c[0], c[1], c[2], mc.px, mc.py, mc.pz);
		tie = d < bd ? false : (tie || d == bd);
		if (d < bd)
		{
			bd = d;
			best = t;
		}
	}
	const unsigned int key = __float_as_uint(bd); // not negative
	const unsigned int least = __reduce_min_sync(0xffffffffu, key);
	const unsigned int win = __ballot_sync(0xffffffffu, key == least && best != ~0u);
	*distance = __uint_as_float(least);
	*sure = (win & (win - 1)) == 0 && !__any_sync(0xffffffffu, tie && (win >> lane & 1u)) && *distance > 1e-15f && fabsf(mc.px) <= 1e15f &&
	        fabsf(mc.py) <= 1e15f && fabsf(mc.pz) <= 1e15f && win;
	return win ? __shfl_sync(0xffffffffu, best, __ffs(win) - 1) : ~0u;
}

// meshopt_optimizeMeshletLevel (src/meshletutils.cpp:366-554) on one meshlet, by one warp. At every
// position the scan over the remaining triangles runs 32 at a time (the stop after the level-th edge
// match found with a ballot, then the first best score up to it), and the triangles before the
// chosen one shift up together; 8-bit timestamps and valences wrap as the reference's do. The
// rotations and the renumbering need only each vertex's first use, so every triangle is done at once.
struct MeshletOpt
{
	unsigned int tri[512]; // three 8-bit corners
	unsigned int valence[256];
	unsigned int first[256];
	unsigned char cache[256];
};

__device__ __forceinline__ unsigned int packCorners(unsigned int a, unsigned int b, unsigned int c)
{
	return a | b << 8 | c << 16;
}

__device__ void optimizeMeshletWarp(unsigned int* verts, unsigned char* tris, unsigned int vc, unsigned int tc, int level, MeshletOpt& o)
{
	const unsigned int lane = threadIdx.x & 31, below = (1u << lane) - 1u;
	const unsigned char cutoff = 3;
	for (unsigned int v = lane; v < vc; v += 32)
	{
		o.cache[v] = 0;
		o.valence[v] = 0;
		o.first[v] = ~0u;
	}
	__syncwarp();
	for (unsigned int j = lane; j < tc; j += 32)
	{
		const unsigned int a = tris[j * 3], b = tris[j * 3 + 1], c = tris[j * 3 + 2];
		o.tri[j] = packCorners(a, b, c);
		atomicAdd(&o.valence[a], 1u);
		atomicAdd(&o.valence[b], 1u);
		atomicAdd(&o.valence[c], 1u);
	}
	__syncwarp();
	unsigned char cache_last = 128;
	for (unsigned int i = 0; i < tc; ++i)
	{
		unsigned int next = 0, word = 0;
		int next_score = -1, edges = 0;
		bool done = false;
		for (unsigned int j0 = i; j0 < tc && !done; j0 += 32)
		{
			const unsigned int j = j0 + lane;
			const bool valid = j < tc;
			int score = -2, match = 0;
			unsigned int w = 0;
			if (valid)
			{
				w = o.tri[j];
				const unsigned int a = w & 255u, b = w >> 8 & 255u, c = w >> 16;
				unsigned char ad = (unsigned char)(cache_last - o.cache[a]);
				unsigned char bd = (unsigned char)(cache_last - o.cache[b]);
				unsigned char cd = (unsigned char)(cache_last - o.cache[c]);
				match = (ad < cutoff) + (bd < cutoff) + (cd < cutoff);
				if (level)
				{
					int va = o.valence[a] & 0xFF, vb = o.valence[b] & 0xFF, vcc = o.valence[c] & 0xFF;
					int vmin = va < vb ? va : vb;
					vmin = vcc < vmin ? vcc : vmin;
					score = (match * 1024 + (1023 - ad - bd - cd)) * 256 + (255 - vmin);
				}
				else
					score = match;
			}
			// the scan stops at the edge match that makes `level` of them (the first one at level 0)
			const unsigned int em = __ballot_sync(0xffffffffu, valid && match >= 2);
			const int need = level ? level - edges : 1;
			unsigned int last = 31;
			if (__popc(em) >= need)
			{
				unsigned int m = em;
				for (int q = 1; q < need; ++q)
					m &= m - 1;
				last = __ffs(m) - 1;
				done = true;
			}
			edges += __popc(em & (last == 31 ? 0xffffffffu : ((2u << last) - 1u)));
			// the first best score among the scanned ones
			const int mine = valid && lane <= last ? score : -2;
			const int bs = __reduce_max_sync(0xffffffffu, mine);
			if (bs > next_score)
			{
				const unsigned int at = __ffs(__ballot_sync(0xffffffffu, mine == bs)) - 1;
				next = j0 + at;
				next_score = bs;
				word = __shfl_sync(0xffffffffu, w, at);
			}
		}
		for (unsigned int top = next; top > i; top = top > i + 32 ? top - 32 : i)
		{
			// place p takes the triangle before it
			const bool moves = top >= lane && top - lane > i;
			const unsigned int x = moves ? o.tri[top - lane - 1] : 0u;
			__syncwarp();
			if (moves)
				o.tri[top - lane] = x;
			__syncwarp();
		}
		if (lane == 0)
		{
			const unsigned int a = word & 255u, b = word >> 8 & 255u, c = word >> 16;
			o.tri[i] = word;
			unsigned char stamp = (unsigned char)(cache_last + 1);
			o.cache[a] = o.cache[b] = o.cache[c] = stamp;
			o.valence[a] = (o.valence[a] - 1) & 0xFF;
			o.valence[b] = (o.valence[b] - 1) & 0xFF;
			o.valence[c] = (o.valence[c] - 1) & 0xFF;
		}
		cache_last++;
		__syncwarp();
	}
	if (level >= 1)
	{
		// a vertex is seen from its first triangle on; the edges compared below are the same whichever
		// corner a triangle starts at
		for (unsigned int i = lane; i < tc; i += 32)
		{
			const unsigned int w = o.tri[i];
			atomicMin(&o.first[w & 255u], i);
			atomicMin(&o.first[w >> 8 & 255u], i);
			atomicMin(&o.first[w >> 16], i);
		}
		__syncwarp();
		for (unsigned int base = 0; base < tc; base += 32)
		{
			const unsigned int i = base + lane;
			unsigned int w = 0;
			if (i < tc)
			{
				w = o.tri[i];
				const unsigned int a = w & 255u, b = w >> 8 & 255u, c = w >> 16;
				const bool sa = o.first[a] < i, sb = o.first[b] < i, sc = o.first[c] < i;
				if (!sa && sb && !sc)
					w = packCorners(b, c, a);
				else if (!sa && !sb && !sc)
				{
					bool ab = false, bc = false, ca = false;
					for (unsigned int j = i + 1; j < tc && j <= i + cutoff; ++j)
					{
						const unsigned int x = o.tri[j];
						const unsigned int oa = x & 255u, ob = x >> 8 & 255u, oc = x >> 16;
						ab |= (oa == b && ob == a) || (ob == b && oc == a) || (oc == b && oa == a);
						bc |= (oa == c && ob == b) || (ob == c && oc == b) || (oc == c && oa == b);
						ca |= (oa == a && ob == c) || (ob == a && oc == c) || (oc == a && oa == c);
					}
					if (ab && !bc)
						w = packCorners(b, c, a);
					else if ((ab && !ca) || (!ab && bc && !ca))
						w = packCorners(c, a, b);
				}
			}
			__syncwarp(); // the next triangles of this step were read above
			if (i < tc)
				o.tri[i] = w;
			__syncwarp();
		}
	}
	// vertices renumbered in first-use order; the valence words now hold the new numbers
	for (unsigned int v = lane; v < vc; v += 32)
		o.first[v] = ~0u;
	__syncwarp();
	for (unsigned int k = lane; k < tc * 3; k += 32)
		atomicMin(&o.first[o.tri[k / 3] >> (k % 3 * 8) & 255u], k);
	__syncwarp();
	unsigned int n = 0;
	unsigned int moved[8]; // this lane's vertices by new number, at most 256 / 32
#pragma unroll
	for (int q = 0; q < 8; ++q)
		moved[q] = 0;
	for (unsigned int base = 0; base < tc * 3; base += 32)
	{
		const unsigned int k = base + lane;
		const unsigned int v = k < tc * 3 ? o.tri[k / 3] >> (k % 3 * 8) & 255u : 0u;
		const bool first = k < tc * 3 && o.first[v] == k;
		const unsigned int m = __ballot_sync(0xffffffffu, first);
		if (first)
			o.valence[v] = n + __popc(m & below);
		n += __popc(m);
	}
	__syncwarp();
#pragma unroll
	for (int q = 0; q < 8; ++q)
	{
		const unsigned int v = q * 32 + lane;
		if (v < vc && o.first[v] != ~0u)
			moved[q] = verts[v];
	}
	__syncwarp();
#pragma unroll
	for (int q = 0; q < 8; ++q)
	{
		const unsigned int v = q * 32 + lane;
		if (v < vc && o.first[v] != ~0u)
			verts[o.valence[v]] = moved[q];
	}
	for (unsigned int k = lane; k < tc * 3; k += 32)
		tris[k] = (unsigned char)o.valence[o.tri[k / 3] >> (k % 3 * 8) & 255u];
	__syncwarp();
}

// Group-local vertex ids in first-use order, each corner's id and its place in its vertex's triangle
// list, and the corners of every vertex; false if there are more than `cap` vertices. A step takes 32
// corners: the first of each vertex among them finds or enters it in the table.
template <class K>
__device__ __forceinline__ bool assignIds(const MeshletBatch& b, const Scratch<K>& s, const unsigned int* indices, unsigned int I, unsigned int* hkey,
    typename K::Id* hid, typename K::Id* hcnt, unsigned int H, unsigned int cap, unsigned int& U)
{
	typedef typename K::Id Id;
	const unsigned int lane = threadIdx.x, below = (1u << lane) - 1u;
	for (unsigned int h = lane; h < H; h += 32)
		hkey[h] = ~0u;
	__syncwarp();
	U = 0;
	unsigned int ahead = lane < I ? indices[lane] : 0u;
	for (unsigned int base = 0; base < I; base += 32)
	{
		const unsigned int p = base + lane;
		const bool valid = p < I;
		unsigned int v = ahead;
		ahead = p + 32 < I ? indices[p + 32] : 0u;
		if (valid && v >= b.vertex_count)
		{
			atomicOr(b.error, 1u);
			v = 0;
		}
		const unsigned int peers = __match_any_sync(0xffffffffu, valid ? v : ~0u); // no vertex is ~0
		const unsigned int leader = __ffs(peers) - 1;
		unsigned int h = hashVertex(v) & (H - 1), k = ~0u;
		if (valid && lane == leader)
			for (unsigned int probe = 0; probe < H; ++probe)
			{
				k = atomicCAS(&hkey[h], ~0u, v);
				if (k == ~0u || k == v)
					break;
				h = (h + 1) & (H - 1);
			}
		const bool fresh = valid && lane == leader && k == ~0u;
		const unsigned int m = __ballot_sync(0xffffffffu, fresh);
		if (U + __popc(m) > cap)
			return false;
		unsigned int id = 0, count = 0;
		if (valid && lane == leader)
		{
			if (fresh)
			{
				id = U + __popc(m & below);
				hid[h] = Id(id);
				s.gid[id] = v;
			}
			else
			{
				id = hid[h];
				count = hcnt[id];
			}
			hcnt[id] = Id(count + __popc(peers));
		}
		U += __popc(m);
		id = __shfl_sync(0xffffffffu, id, leader);
		count = __shfl_sync(0xffffffffu, count, leader);
		if (valid)
		{
			s.lid[p] = Id(id);
			s.lpos[p] = Id(count + __popc(peers & below));
		}
		__syncwarp();
	}
	return true;
}

// one group with its ids assigned: everything after
template <class K>
__device__ __forceinline__ void buildGroup(const MeshletBatch& b, const Scratch<K>& s, const unsigned long long g, unsigned int I, unsigned int U)
{
	typedef typename K::Id Id;
	typedef typename K::Vertex Vertex;
	typedef typename K::Triangle Triangle;
	const unsigned int lane = threadIdx.x;
	const unsigned int below = (1u << lane) - 1u;
	const unsigned int F = I / 3;
	const unsigned long long i0 = b.offsets[g];
	unsigned int* out = b.meshlets + b.meshlet_base[g] * 4;
	const unsigned long long out_rows = b.meshlet_base[g + 1] - b.meshlet_base[g];
	unsigned int* mverts = b.mverts + i0;
	unsigned char* mtris = b.mtris + i0;

	// ---- triangle lists per vertex, in face order (corner order)
	const Id none = Scratch<K>::none();
	bool degenerate = false; // a triangle that names a vertex twice
	for (unsigned int t = lane; t < F; t += 32)
	{
		Triangle tr;
		tr.x = s.lid[t * 3], tr.y = s.lid[t * 3 + 1], tr.z = s.lid[t * 3 + 2], tr.w = Id(t);
		s.tri[t] = tr;
		s.state[t] = kTriFree;
		degenerate |= tr.x == tr.y || tr.x == tr.z || tr.y == tr.z;
	}
	degenerate = __any_sync(0xffffffffu, degenerate);
	__syncwarp();
	for (unsigned int p = lane; p < I; p += 32)
		s.adj[s.off[s.lid[p]] + s.lpos[p]] = Id(p / 3);

	// ---- triangle cones (computeTriangleCones, :201-241)
	bool finite = true, small = F <= kNearestScan;
	for (unsigned int t = lane; t < F; t += 32)
	{
		const Triangle tr = s.tri[t];
		const float* p0 = b.positions + size_t(b.stride_f) * s.gid[tr.x];
		const float* p1 = b.positions + size_t(b.stride_f) * s.gid[tr.y];
		const float* p2 = b.positions + size_t(b.stride_f) * s.gid[tr.z];
		float p10[3] = {p1[0] - p0[0], p1[1] - p0[1], p1[2] - p0[2]};
		float p20[3] = {p2[0] - p0[0], p2[1] - p0[1], p2[2] - p0[2]};
		float nx = p10[1] * p20[2] - p10[2] * p20[1];
		float ny = p10[2] * p20[0] - p10[0] * p20[2];
		float nz = p10[0] * p20[1] - p10[1] * p20[0];
		float area = sqrtf(nx * nx + ny * ny + nz * nz);
		float inv = (area == 0.f) ? 0.f : 1.f / area;
		float* c = s.cent + size_t(t) * 3;
		float* n = s.norm + size_t(t) * 3;
		c[0] = (p0[0] + p1[0] + p2[0]) / 3.f;
		c[1] = (p0[1] + p1[1] + p2[1]) / 3.f;
		c[2] = (p0[2] + p1[2] + p2[2]) / 3.f;
		n[0] = nx * inv;
		n[1] = ny * inv;
		n[2] = nz * inv;
		finite = finite && fabsf(n[0]) <= FLT_MAX && fabsf(n[1]) <= FLT_MAX && fabsf(n[2]) <= FLT_MAX;
		small = small && fabsf(c[0]) <= 1e15f && fabsf(c[1]) <= 1e15f && fabsf(c[2]) <= 1e15f;
		s.area[t] = area;
	}
	ScoreArgs sa;
	sa.cone_weight = b.cone_weight;
	sa.axes = b.cone_weight != 0.f || __any_sync(0xffffffffu, !finite);
	const bool tame = __all_sync(0xffffffffu, small); // nearestScan's answers hold
	__syncwarp();

	// ---- mesh area in face order (lane 0), the corner, the first seed
	float mesh_area = 0.f;
	if (lane == 0)
	{
#pragma unroll 8
		for (unsigned int t = 0; t < F; ++t)
			mesh_area += s.area[t];
		float tri_area_avg = mesh_area / float(F) * 0.5f;
		sa.radius = sqrtf(tri_area_avg * float(b.max_triangles)) * 0.5f;
	}
	sa.radius = __shfl_sync(0xffffffffu, sa.radius, 0);
	const float radius = sa.radius;
	// the smallest of each coordinate, NaN skipped (the sign of a zero does not reach the distances)
	float cx = FLT_MAX, cy = FLT_MAX, cz = FLT_MAX;
	for (unsigned int t = lane; t < F; t += 32)
	{
		const float* c = s.cent + size_t(t) * 3;
		cx = cx > c[0] ? c[0] : cx;
		cy = cy > c[1] ? c[1] : cy;
		cz = cz > c[2] ? c[2] : cz;
	}
	for (int o = 16; o > 0; o >>= 1)
	{
		const float x = __shfl_xor_sync(0xffffffffu, cx, o), y = __shfl_xor_sync(0xffffffffu, cy, o), z = __shfl_xor_sync(0xffffffffu, cz, o);
		cx = cx > x ? x : cx;
		cy = cy > y ? y : cy;
		cz = cz > z ? z : cz;
	}
	// the first triangle with the smallest distance to it; a NaN first distance keeps triangle 0
	unsigned int initial = ~0u;
	{
		float bd = 0.f;
		bool nan0 = false;
		for (unsigned int t = lane; t < F; t += 32)
		{
			const float* c = s.cent + size_t(t) * 3;
			const float d = dist3(c[0], c[1], c[2], cx, cy, cz);
			nan0 |= t == 0 && d != d;
			if (d == d && (initial == ~0u || d < bd))
			{
				initial = t;
				bd = d;
			}
		}
		const unsigned int key = initial == ~0u ? ~0u : orderedBits(bd);
		const unsigned int m = __reduce_min_sync(0xffffffffu, key);
		initial = __reduce_min_sync(0xffffffffu, key == m && initial != ~0u ? initial : ~0u);
		if (__any_sync(0xffffffffu, nan0) || initial == ~0u)
			initial = 0;
	}
	__syncwarp();

	// ---- the greedy loop (:1125-1216); every lane holds the same meshlet state
	unsigned int m_voff = 0, m_toff = 0, m_vc = 0, m_tc = 0; // the current meshlet
	unsigned int offset = 0, seed_count = 0;
	unsigned int fn = 0; // triangles in the frontier
	bool tree = false;   // the kd-tree is built
	Cone acc = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
	// the current meshlet's row, vertices and triangles
	auto writeMeshlet = [&]() {
		if (offset >= out_rows || m_voff + m_vc > I || m_toff + m_tc * 3 > I)
		{
			if (lane == 0)
				atomicOr(b.error, 4u);
			return;
		}
		if (lane < 4)
			out[offset * 4 + lane] = lane == 0 ? m_voff : (lane == 1 ? m_toff : (lane == 2 ? m_vc : m_tc));
		for (unsigned int j = lane; j < m_vc; j += 32)
			mverts[m_voff + j] = s.gid[s.mvl[j]];
		for (unsigned int j = lane; j < m_tc * 3; j += 32)
			mtris[m_toff + j] = s.mtri[j];
	};
	for (unsigned int step = 0; step < F; ++step) // with every triangle emitted there is no next one
	{
		// getMeshletCone, :181-199
		sa.mc = acc;
		{
			float center_scale = m_tc == 0 ? 0.f : 1.f / float(m_tc);
			sa.mc.px *= center_scale;
			sa.mc.py *= center_scale;
			sa.mc.pz *= center_scale;
			if (sa.axes)
			{
				float len = sa.mc.nx * sa.mc.nx + sa.mc.ny * sa.mc.ny + sa.mc.nz * sa.mc.nz;
				float axis_scale = len == 0.f ? 0.f : 1.f / sqrtf(len);
				sa.mc.nx *= axis_scale;
				sa.mc.ny *= axis_scale;
				sa.mc.nz *= axis_scale;
			}
		}
		unsigned int best = ~0u, slot = ~0u;
		if (offset == 0 && m_tc == 0)
			best = initial;
		else if (fn)
		{
			bool nan = false;
			best = neighborWarp(s, fn, sa, &slot, &nan);
			if (nan)
			{
				if (lane == 0)
					best = neighborSerial(s, m_vc, sa);
				best = __shfl_sync(0xffffffffu, best, 0);
				slot = ~0u;
			}
		}
		bool split = false;
		if (best == ~0u)
		{
			// no adjacent triangle: the nearest unemitted one (kdtreeNearest)
			float distance = FLT_MAX;
			bool sure = false;
			if (tame)
				best = nearestScan(s, F, sa.mc, &distance, &sure);
			if (!sure)
			{
				if (!tree)
					kdBuild(s, F, b.error);
				tree = true;
				best = ~0u;
				distance = FLT_MAX;
				if (lane == 0)
				{
					const float pos[3] = {sa.mc.px, sa.mc.py, sa.mc.pz};
					kdNearest(s, pos, &best, &distance);
				}
				best = __shfl_sync(0xffffffffu, best, 0);
				distance = __shfl_sync(0xffffffffu, distance, 0);
			}
			split = m_tc >= b.min_triangles && b.split_factor > 0 && distance > radius * b.split_factor;
		}
		if (best == ~0u)
			break;
		__syncwarp();
		Triangle bt = s.tri[best];
		Id y0 = s.vert[bt.x].y, y1 = s.vert[bt.y].y, y2 = s.vert[bt.z].y;
		int extra = (y0 == none) + (y1 == none) + (y2 == none);
		if (split || m_vc + extra > b.max_vertices || m_tc >= b.max_triangles)
		{
			// each meshlet vertex's neighbour with the smallest live count (appendSeedTriangles,
			// :364-430, inner loop), then the seed bookkeeping in vertex order on lane 0
			for (unsigned int i = lane; i < m_vc; i += 32)
			{
				unsigned int v = s.mvl[i];
				const Id* list = s.adj + s.off[v];
				const unsigned int n = s.vert[v].x;
				unsigned int bn = ~0u, bn_live = ~0u;
				for (unsigned int j = 0; j < n; ++j)
				{
					unsigned int t = list[j];
					const Triangle tr = s.tri[t];
					unsigned int l = s.vert[tr.x].x + s.vert[tr.y].x + s.vert[tr.z].x;
					if (l < bn_live)
					{
						bn = t;
						bn_live = l;
					}
				}
				float score = 0.f;
				if (bn != ~0u)
				{
					const float* c = s.cent + size_t(bn) * 3;
					score = dist3(c[0], c[1], c[2], cx, cy, cz);
				}
				s.vbest[i * 3 + 0] = bn;
				s.vbest[i * 3 + 1] = bn_live;
				s.vbest[i * 3 + 2] = __float_as_uint(score);
			}
			__syncwarp();
			if (lane == 0)
			{
				// pruneSeedTriangles, :432-445
				unsigned int r = 0;
				for (unsigned int i = 0; i < seed_count; ++i)
				{
					unsigned int sd = s.seeds[i];
					s.seeds[r] = sd;
					r += s.state[sd] != kTriEmitted;
				}
				seed_count = (r + kAddSeeds <= kMaxSeeds) ? r : kMaxSeeds - kAddSeeds;
				unsigned int bs[kAddSeeds], bl[kAddSeeds];
				float bsc[kAddSeeds];
				for (unsigned int i = 0; i < kAddSeeds; ++i)
				{
					bs[i] = ~0u;
					bl[i] = ~0u;
					bsc[i] = FLT_MAX;
				}
				for (unsigned int i = 0; i < m_vc; ++i)
				{
					unsigned int bn = s.vbest[i * 3 + 0];
					if (bn == ~0u)
						continue;
					unsigned int live = s.vbest[i * 3 + 1];
					float score = __uint_as_float(s.vbest[i * 3 + 2]);
					for (unsigned int j = 0; j < kAddSeeds; ++j)
						if (live < bl[j] || (live == bl[j] && score <= bsc[j]))
						{
							bs[j] = bn;
							bl[j] = live;
							bsc[j] = score;
							break;
						}
				}
				for (unsigned int i = 0; i < kAddSeeds; ++i)
					if (bs[i] != ~0u)
						s.seeds[seed_count++] = bs[i];
				// selectSeedTriangle, :447-471
				unsigned int bseed = ~0u, blive = ~0u;
				float bscore = FLT_MAX;
				for (unsigned int i = 0; i < seed_count; ++i)
				{
					unsigned int sd = s.seeds[i];
					const Triangle tr = s.tri[sd];
					unsigned int live = s.vert[tr.x].x + s.vert[tr.y].x + s.vert[tr.z].x;
					const float* c = s.cent + size_t(sd) * 3;
					float score = dist3(c[0], c[1], c[2], cx, cy, cz);
					if (live < blive || (live == blive && score < bscore))
					{
						bseed = sd;
						blive = live;
						bscore = score;
					}
				}
				if (bseed != ~0u && bseed != best)
				{
					best = bseed;
					slot = ~0u;
				}
			}
			best = __shfl_sync(0xffffffffu, best, 0);
			slot = __shfl_sync(0xffffffffu, slot, 0);
			seed_count = __shfl_sync(0xffffffffu, seed_count, 0);
			bt = s.tri[best];
			y0 = s.vert[bt.x].y, y1 = s.vert[bt.y].y, y2 = s.vert[bt.z].y;
			extra = (y0 == none) + (y1 == none) + (y2 == none);
		}

		bool in_front = s.state[best] == kTriFrontier;
		// appendMeshlet, :243-300
		if (m_vc + extra > b.max_vertices || m_tc >= b.max_triangles || split)
		{
			writeMeshlet();
			for (unsigned int j = lane; j < m_vc; j += 32)
				s.vert[s.mvl[j]].y = none;
			for (unsigned int i = lane; i < fn; i += 32)
			{
				float x, y, z;
				s.state[frontAt(s, i, x, y, z).w] = kTriFree;
			}
			fn = 0;
			in_front = false;
			y0 = y1 = y2 = none;
			m_voff += m_vc;
			m_toff += m_tc * 3;
			m_vc = 0;
			m_tc = 0;
			offset++;
			acc = Cone{0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
			__syncwarp();
		}
		const unsigned int v0 = bt.x, v1 = bt.y, v2 = bt.z;
		const bool n0 = y0 == none, n1 = y1 == none && v1 != v0, n2 = y2 == none && v2 != v0 && v2 != v1;
		const unsigned int l0 = n0 ? m_vc : y0;
		const unsigned int l1 = n1 ? m_vc + n0 : (v1 == v0 ? l0 : y1);
		const unsigned int l2 = n2 ? m_vc + n0 + n1 : (v2 == v0 ? l0 : (v2 == v1 ? l1 : y2));
		__syncwarp(); // every lane has read the words written below
		if (lane < 3)
		{
			const unsigned int v = lane == 0 ? v0 : (lane == 1 ? v1 : v2), l = lane == 0 ? l0 : (lane == 1 ? l1 : l2);
			if (lane == 0 ? n0 : (lane == 1 ? n1 : n2))
			{
				s.vert[v].y = Id(l);
				s.mvl[l] = Id(v);
			}
			s.mtri[m_tc * 3 + lane] = (unsigned char)l;
		}
		m_vc += n0 + n1 + n2;
		m_tc++;
		// its place in the frontier: the first triangle that joins takes it, else the last one does
		if (in_front)
			for (unsigned int base = 0; base < fn && slot == ~0u; base += 32)
			{
				float x, y, z;
				const unsigned int hit = __ballot_sync(0xffffffffu, base + lane < fn && frontAt(s, base + lane, x, y, z).w == best);
				if (hit)
					slot = base + __ffs(hit) - 1;
			}
		if (lane == 0)
			s.state[best] = kTriEmitted;
		// and its vertices' lists (swap with the last, :1177-1199), and the other live triangles of
		// vertices new to the meshlet join the frontier: eight lanes per vertex, every entry read once
		if (!degenerate)
		{
			const unsigned int k = lane >> 3;
			const unsigned int v = k == 0 ? v0 : (k == 1 ? v1 : v2);
			const bool fresh = k == 0 ? n0 : (k == 1 ? n1 : n2 && k == 2);
			const unsigned int n = k < 3 ? s.vert[v].x : 0u;
			Id* list = s.adj + s.off[v];
			__syncwarp();
			for (unsigned int j = lane & 7; __any_sync(0xffffffffu, j < n); j += 8)
			{
				bool add = false;
				unsigned int t = 0;
				Triangle tr;
				float x = 0.f, y = 0.f, z = 0.f;
				if (j < n)
				{
					t = list[j];
					if (t == best)
					{
						list[j] = list[n - 1];
						s.vert[v].x = Id(n - 1);
					}
					else if (fresh)
					{
						// a triangle of two new vertices joins with the first
						const float* c = s.cent + size_t(t) * 3;
						tr = s.tri[t];
						x = c[0], y = c[1], z = c[2];
						add = s.state[t] == kTriFree && !(k >= 1 && n0 && (tr.x == v0 || tr.y == v0 || tr.z == v0)) &&
						      !(k == 2 && n1 && (tr.x == v1 || tr.y == v1 || tr.z == v1));
					}
				}
				const unsigned int m = __ballot_sync(0xffffffffu, add);
				if (m)
				{
					const unsigned int r = __popc(m & below);
					if (add)
					{
						frontSet(s, in_front ? (r ? fn + r - 1 : slot) : fn + r, tr, x, y, z);
						s.state[t] = kTriFrontier;
					}
					fn += __popc(m) - in_front;
					in_front = false;
				}
			}
		}
		else
		{
			// a triangle may name a vertex twice, and its list then holds it twice: in order, one lane
			__syncwarp();
			if (lane == 0)
				for (int k = 0; k < 3; ++k)
				{
					const unsigned int v = k == 0 ? v0 : (k == 1 ? v1 : v2);
					Id* list = s.adj + s.off[v];
					const unsigned int n = s.vert[v].x;
					for (unsigned int i = 0; i < n; ++i)
						if (list[i] == best)
						{
							list[i] = list[n - 1];
							s.vert[v].x = Id(n - 1);
							break;
						}
				}
			__syncwarp();
			if (lane == 0)
				for (int k = 0; k < 3; ++k)
				{
					const unsigned int v = k == 0 ? v0 : (k == 1 ? v1 : v2);
					const Id* list = s.adj + s.off[v];
					for (unsigned int j = 0, n = (k == 0 ? n0 : (k == 1 ? n1 : n2)) ? s.vert[v].x : 0u; j < n; ++j)
						if (s.state[list[j]] == kTriFree)
						{
							const float* c = s.cent + size_t(list[j]) * 3;
							frontSet(s, fn++, s.tri[list[j]], c[0], c[1], c[2]);
							s.state[list[j]] = kTriFrontier;
						}
				}
			fn = __shfl_sync(0xffffffffu, fn, 0);
		}
		if (in_front)
		{
			--fn;
			if (lane == 0 && slot != fn)
			{
				float x, y, z;
				const Triangle f = frontAt(s, fn, x, y, z);
				frontSet(s, slot, f, x, y, z);
			}
		}
		__syncwarp();
		const float* c = s.cent + size_t(best) * 3;
		acc.px += c[0];
		acc.py += c[1];
		acc.pz += c[2];
		if (sa.axes)
		{
			const float* n = s.norm + size_t(best) * 3;
			acc.nx += n[0];
			acc.ny += n[1];
			acc.nz += n[2];
		}
	}
	if (m_tc)
	{
		writeMeshlet();
		offset++;
	}
	if (lane == 0)
		b.counts[g] = offset;
}

template <class K>
__global__ void __launch_bounds__(32) kMeshletsFlex(MeshletBatch b, unsigned int pool_bytes)
{
	typedef typename K::Id Id;
	extern __shared__ __align__(16) char pool[];
	__shared__ Id mvl[256];
	__shared__ unsigned char mtri[512 * 3];
	const unsigned int lane = threadIdx.x;
	const unsigned int g = blockIdx.x;
	const unsigned long long i0 = b.offsets[g];
	const unsigned int I = unsigned(b.offsets[g + 1] - i0) / 3 * 3, F = I / 3;
	const unsigned int* indices = b.indices + i0;
	if (F == 0)
	{
		if (lane == 0)
			b.counts[g] = 0;
		return;
	}
	Scratch<K> s;
	carve(s, b.scratch + b.scratch_off[g], I);
	s.mvl = mvl;
	s.mtri = mtri;

	// the vertex table in shared memory, before the hot arrays need it, or in the scratch
	unsigned int U = 0;
	bool done = false;
	const unsigned int HS = sharedTableSize(I);
	if (size_t(HS) * (4 + sizeof(Id)) < pool_bytes)
	{
		unsigned int* hkey = reinterpret_cast<unsigned int*>(pool);
		Id* hid = reinterpret_cast<Id*>(hkey + HS);
		Id* count = hid + HS;
		const unsigned int cap = unsigned((pool_bytes - size_t(HS) * (4 + sizeof(Id))) / sizeof(Id));
		done = assignIds(b, s, indices, I, hkey, hid, count, HS, cap, U);
		if (done)
		{
			__syncwarp();
			for (unsigned int v = lane; v < U; v += 32)
				s.hcnt[v] = count[v];
		}
		__syncwarp();
	}
	if (!done)
		assignIds(b, s, indices, I, s.hkey, s.hid, s.hcnt, tableSize(I), ~0u, U);
	__syncwarp();
	// list offsets and live counts, then the rest, with the arrays a step reads in shared memory
	// where they fit
	auto vertices = [&](const Scratch<K>& a) {
		unsigned int run = 0;
		for (unsigned int base = 0; base < U; base += 32)
		{
			const unsigned int v = base + lane;
			unsigned int c = v < U ? s.hcnt[v] : 0u, x = c;
			for (int o = 1; o < 32; o <<= 1)
			{
				unsigned int y = __shfl_up_sync(0xffffffffu, x, o);
				if (lane >= (unsigned)o)
					x += y;
			}
			if (v < U)
			{
				a.off[v] = Id(run + x - c);
				typename K::Vertex w;
				w.x = Id(c), w.y = Scratch<K>::none();
				a.vert[v] = w;
			}
			run += __shfl_sync(0xffffffffu, x, 31);
		}
		__syncwarp();
	};
	Scratch<K> hot = s;
	if (carveHot(hot, pool, F, U) <= pool_bytes)
	{
		vertices(hot);
		buildGroup(b, hot, g, I, U);
	}
	else
	{
		vertices(s);
		buildGroup(b, s, g, I, U);
	}
}

// meshopt_optimizeMeshletLevel on every meshlet, as clusterize runs it (demo/clusterlod.h:292-300):
// one warp per meshlet row of the batch; a row past its group's meshlet count has nothing to do
__global__ void __launch_bounds__(32) kOptimizeMeshlets(MeshletBatch b, unsigned long long rows)
{
	__shared__ MeshletOpt opt;
	for (unsigned long long r = blockIdx.x; r < rows; r += gridDim.x)
	{
		// the group whose rows hold r: the last g with meshlet_base[g] <= r
		unsigned int lo = 0, hi = b.groups;
		while (hi - lo > 1)
		{
			unsigned int mid = (lo + hi) / 2;
			if (b.meshlet_base[mid] <= r)
				lo = mid;
			else
				hi = mid;
		}
		const unsigned int g = lo;
		const unsigned long long k = r - b.meshlet_base[g];
		if (k >= b.counts[g])
			continue;
		const unsigned long long i0 = b.offsets[g];
		const unsigned int I = unsigned(b.offsets[g + 1] - i0) / 3 * 3;
		const unsigned int* row = b.meshlets + r * 4;
		const unsigned int vo = row[0], to = row[1], vc = row[2], tc = row[3];
		if (vc <= 256 && tc <= 512 && vo + vc <= I && to + tc * 3 <= I)
			optimizeMeshletWarp(b.mverts + i0 + vo, b.mtris + i0 + to, vc, tc, b.optimize_level, opt);
	}
}

} // namespace

size_t meshletBound(size_t index_count, size_t max_vertices, size_t max_triangles)
{
	size_t conservative = max_vertices - 2;
	size_t by_vertices = (index_count + conservative - 1) / conservative;
	size_t by_triangles = (index_count / 3 + max_triangles - 1) / max_triangles;
	return by_vertices > by_triangles ? by_vertices : by_triangles;
}

size_t meshletScratchBytes(size_t index_count)
{
	// the wide layout's, which holds either
	Scratch<Wide> s;
	return align256(carve(s, nullptr, unsigned(index_count / 3 * 3)));
}

template <class K>
void launchFlex(const MeshletBatch& b, unsigned int pool, cudaStream_t stream)
{
	MO_LAUNCH((kMeshletsFlex<K>), b.groups, 32, pool, stream, b, pool);
}

void buildMeshletsBatch(const MeshletBatch& b, cudaStream_t stream)
{
	if (!b.groups)
		return;
	const unsigned int F = b.max_index_count / 3;
	const bool narrow = b.max_index_count < 65535;
	// shared memory for the largest group's hot arrays, with 3 vertices for 4 triangles (a patch of a
	// surface has about one for two; a group with more keeps them in its scratch), and for its vertex
	// table where that is small. Above kPoolMax too few groups would fit an SM.
	const unsigned int U = F - F / 4 + 3;
	Scratch<Narrow> sn;
	Scratch<Wide> sw;
	size_t want = narrow ? carveHot(sn, nullptr, F, U) : carveHot(sw, nullptr, F, U);
	const size_t table = sharedTableSize(b.max_index_count) * (narrow ? 6 : 8) + U * (narrow ? 2 : 4) + 16;
	if (table <= kPoolTableMax)
		want = std::max(want, table);
	const unsigned int pool = want <= kPoolMax ? unsigned(want) : 0u;
	if (narrow)
		launchFlex<Narrow>(b, pool, stream);
	else
		launchFlex<Wide>(b, pool, stream);
	if (b.optimize_level >= 0 && b.rows)
		MO_LAUNCH(kOptimizeMeshlets, unsigned(std::min(b.rows, 0x7fffffffull)), 32, 0, stream, b, b.rows);
	MO_CUDA_CHECK(cudaGetLastError());
}

} // namespace mogpu
