// On-device BVH construction: per-mesh BLAS (8-wide, quantised) and per-scene TLAS (binary) with a
// refit path for pose updates. The per-item logic lives in bvh_core.hpp.
//
// Replaces the OptiX acceleration-structure builds of reference src/scene/GASBuilder.hpp:31-100 and
// src/scene/Scene.cpp:131-190 (where any pose change triggers a full IAS rebuild plus a stream sync).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <stdexcept>
#include <string>
#include <vector>

#include "bvh_core.hpp"
#include "collapse.cuh"
#include "kernels.hpp"
#include "sah_build.hpp"

namespace rgl {

namespace {

#define RGL_CUDA_OK(expr)                                                                                                      \
	do {                                                                                                                       \
		cudaError_t e_ = (expr);                                                                                               \
		if (e_ != cudaSuccess) {                                                                                               \
			throw std::runtime_error(std::string("CUDA error in BVH build: ") + cudaGetErrorString(e_) + " at " #expr);        \
		}                                                                                                                      \
	} while (0)

__device__ __forceinline__ uint32_t orderedBits(float f)
{
	uint32_t u = __float_as_uint(f);
	return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__host__ __device__ __forceinline__ float orderedFloat(uint32_t u)
{
	uint32_t v = (u & 0x80000000u) ? (u & 0x7fffffffu) : ~u;
#if defined(__CUDA_ARCH__)
	return __uint_as_float(v);
#else
	float f;
	__builtin_memcpy(&f, &v, 4);
	return f;
#endif
}

// Triangle boxes, centroids and, if asked for, the centroid bounds: 6 ordered uints, the minima xyz
// complemented so that all of them start at zero and grow, then the maxima xyz.
__global__ void kTriBounds(const float* __restrict__ v, const int32_t* __restrict__ idx, int nTris, float4* lo, float4* hi,
                           uint32_t* cbounds)
{
	__shared__ uint32_t sh[6];
	if (threadIdx.x < 6) {
		sh[threadIdx.x] = 0u;
	}
	__syncthreads();
	int t = blockIdx.x * blockDim.x + threadIdx.x;
	if (t < nTris) {
		const float* a = v + 3 * (size_t) idx[3 * t];
		const float* b = v + 3 * (size_t) idx[3 * t + 1];
		const float* c = v + 3 * (size_t) idx[3 * t + 2];
		float4 l = make_float4(fminf(fminf(a[0], b[0]), c[0]), fminf(fminf(a[1], b[1]), c[1]), fminf(fminf(a[2], b[2]), c[2]), 0.f);
		float4 h = make_float4(fmaxf(fmaxf(a[0], b[0]), c[0]), fmaxf(fmaxf(a[1], b[1]), c[1]), fmaxf(fmaxf(a[2], b[2]), c[2]), 0.f);
		lo[t] = l;
		hi[t] = h;
		if (cbounds != nullptr) {
			float cx = 0.5f * (l.x + h.x), cy = 0.5f * (l.y + h.y), cz = 0.5f * (l.z + h.z);
			atomicMax(&sh[0], ~orderedBits(cx));
			atomicMax(&sh[1], ~orderedBits(cy));
			atomicMax(&sh[2], ~orderedBits(cz));
			atomicMax(&sh[3], orderedBits(cx));
			atomicMax(&sh[4], orderedBits(cy));
			atomicMax(&sh[5], orderedBits(cz));
		}
	}
	__syncthreads();
	if (cbounds != nullptr && threadIdx.x < 6) {
		atomicMax(&cbounds[threadIdx.x], sh[threadIdx.x]);
	}
}

// The keys, and their digits counted for the sort (kKeyPasses x 256 counts): a launch and a read of the keys
// less than counting them on their own (3 us and a gap of 2 for 32,768 triangles).
constexpr int kKeyBits = 30, kKeyPasses = 4;
constexpr int kMortonItems = 4;
__global__ void __launch_bounds__(256) kMorton(const float4* __restrict__ lo, const float4* __restrict__ hi, int n, const uint32_t* cbounds,
                                               uint32_t* codes, uint32_t* ids, uint32_t* digitCounts)
{
	__shared__ uint32_t sh[kKeyPasses][256];
#pragma unroll
	for (int p = 0; p < kKeyPasses; ++p) {
		sh[p][threadIdx.x] = 0u;
	}
	__syncthreads();
	const Box cb{orderedFloat(~cbounds[0]), orderedFloat(~cbounds[1]), orderedFloat(~cbounds[2]),
	             orderedFloat(cbounds[3]), orderedFloat(cbounds[4]), orderedFloat(cbounds[5])};
#pragma unroll
	for (int k = 0; k < kMortonItems; ++k) {
		const int t = (blockIdx.x * kMortonItems + k) * 256 + threadIdx.x;
		if (t < n) {
			const float4 l = lo[t], h = hi[t];
			const uint32_t code = morton30(0.5f * (l.x + h.x), 0.5f * (l.y + h.y), 0.5f * (l.z + h.z), cb);
			codes[t] = code;
			ids[t] = (uint32_t) t;
#pragma unroll
			for (int p = 0; p < kKeyPasses; ++p) {
				atomicAdd(&sh[p][(code >> (8 * p)) & 255u], 1u);
			}
		}
	}
	__syncthreads();
#pragma unroll
	for (int p = 0; p < kKeyPasses; ++p) {
		if (sh[p][threadIdx.x] != 0u) {
			atomicAdd(&digitCounts[p * 256 + threadIdx.x], sh[p][threadIdx.x]);
		}
	}
}

// Boxes of aligned groups of 1, 2, 4, ... sorted primitives, level after level: level k holds
// ceil(n / 2^k) boxes (lo, hi).
struct BoxPyramid
{
	float4 *lo, *hi;
};
__host__ __device__ inline size_t pyramidBoxes(int n) { return 2 * (size_t) n + 32; }

// Unions that pass over NaN, with an empty box that is neutral for infinite ones too: a node's box does not
// depend on the order in which its parts are united.
__device__ __forceinline__ Box pyramidUnion(const Box& a, const Box& b)
{
	return Box{fminf(a.lox, b.lox), fminf(a.loy, b.loy), fminf(a.loz, b.loz), fmaxf(a.hix, b.hix), fmaxf(a.hiy, b.hiy), fmaxf(a.hiz, b.hiz)};
}
__device__ __forceinline__ Box pyramidEmpty()
{
	const float inf = __builtin_huge_valf();
	return Box{inf, inf, inf, -inf, -inf, -inf};
}

constexpr int kPyramidTile = 512; // primitives per block; the last block to finish adds the levels above
constexpr int kPyramidThreads = 256;
__device__ __forceinline__ Box pyramidBox(const BoxPyramid& py, size_t i)
{
	const float4 l = __ldcg(py.lo + i), h = __ldcg(py.hi + i);
	return Box{l.x, l.y, l.z, h.x, h.y, h.z};
}
__device__ __forceinline__ void setPyramidBox(const BoxPyramid& py, size_t i, const Box& b)
{
	__stcg(py.lo + i, make_float4(b.lox, b.loy, b.loz, 0.0f));
	__stcg(py.hi + i, make_float4(b.hix, b.hiy, b.hiz, 0.0f));
}
// The levels above the boxes of s, whose level has `count` boxes in all and begins at `at` less `count`: the
// block's boxes are those from `first` on, a tile at most. Leaves `count` and `at` at the last level made, at
// most kPyramidTile boxes wide in this block.
__device__ __forceinline__ void tileLevels(const BoxPyramid& py, Box* s, int first, int& count, size_t& at)
{
	for (int width = kPyramidTile; count > 1 && width > 1; width >>= 1) {
		const int mine = min(count - first, width), c = (count + 1) >> 1, f = first >> 1;
		Box b;
		const int i = threadIdx.x;
		const bool has = 2 * i < mine;
		if (has) {
			b = 2 * i + 1 < mine ? pyramidUnion(s[2 * i], s[2 * i + 1]) : s[2 * i];
		}
		__syncthreads();
		if (has) {
			s[i] = b;
			setPyramidBox(py, at + f + i, b);
		}
		__syncthreads();
		at += c;
		count = c;
		first = f;
	}
}

__global__ void __launch_bounds__(kPyramidThreads) kBoxPyramid(const uint32_t* __restrict__ ids, const float4* __restrict__ lo,
                                                               const float4* __restrict__ hi, int n, BoxPyramid py, uint32_t* ticket)
{
	static_assert(kPyramidTile == 2 * kPyramidThreads, "a pair per thread");
	__shared__ Box s[kPyramidTile];
	__shared__ bool last;
	const int first = blockIdx.x * kPyramidTile;
#pragma unroll
	for (int k = 0; k < 2; ++k) {
		const int local = k * kPyramidThreads + (int) threadIdx.x, i = first + local;
		if (i < n) {
			const uint32_t id = ids[i];
			const float4 l = lo[id], h = hi[id];
			s[local] = Box{l.x, l.y, l.z, h.x, h.y, h.z};
			setPyramidBox(py, i, s[local]);
		}
	}
	__syncthreads();
	int count = n;
	size_t at = (size_t) n; // the next level's first box
	tileLevels(py, s, first, count, at);
	if (count <= 1) {
		return; // one tile: all levels are there
	}
	if (threadIdx.x == 0) {
		__threadfence();
		last = atomicAdd(ticket, 1u) == gridDim.x - 1;
		__threadfence();
	}
	__syncthreads();
	if (!last) {
		return;
	}
	while (count > kPyramidTile) {
		const int c = (count + 1) >> 1;
		const size_t below = at - count;
		for (int i = threadIdx.x; i < c; i += kPyramidThreads) {
			const Box a = pyramidBox(py, below + 2 * i);
			setPyramidBox(py, at + i, 2 * i + 1 < count ? pyramidUnion(a, pyramidBox(py, below + 2 * i + 1)) : a);
		}
		__syncthreads();
		at += c;
		count = c;
	}
	for (int i = threadIdx.x; i < count; i += kPyramidThreads) {
		s[i] = pyramidBox(py, at - count + i);
	}
	__syncthreads();
	tileLevels(py, s, 0, count, at);
}

// The binary nodes: children and range of node i from the sorted keys, its box from at most two pyramid
// boxes per level. Every load of a box is known from the range alone, so a node waits for four levels at a
// time. Climbing from the leaves, the second child to arrive uniting both, was a chain of an atomic and two
// loads per depth (32,768 triangles: 32 us after 11 for children and ranges; now 14 and 6 for the pyramid).
__global__ void kLbvh(const uint32_t* __restrict__ codes, int n, BinNode* bin, int32_t* rangeFirst, int32_t* rangeLast, BoxPyramid py)
{
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n - 1) {
		return;
	}
	int32_t l, r, f, la;
	lbvhInternal(i, codes, n, l, r, f, la);
	rangeFirst[i] = f;
	rangeLast[i] = la;
	Box b = pyramidEmpty();
	constexpr int kLevels = 4;
	size_t at = 0;
	int count = n;
	for (int lo = f, hi = la + 1; lo < hi;) {
		Box part[2 * kLevels];
#pragma unroll
		for (int k = 0; k < kLevels; ++k) {
			part[2 * k] = part[2 * k + 1] = pyramidEmpty();
			if (lo < hi) {
				if (lo & 1) {
					part[2 * k] = pyramidBox(py, at + lo);
					++lo;
				}
				if (hi & 1) {
					--hi;
					part[2 * k + 1] = pyramidBox(py, at + hi);
				}
			}
			at += count;
			count = (count + 1) >> 1;
			lo >>= 1;
			hi >>= 1;
		}
#pragma unroll
		for (int k = 0; k < 2 * kLevels; ++k) {
			b = pyramidUnion(b, part[k]);
		}
	}
	float4* p = reinterpret_cast<float4*>(bin + i);
	p[0] = make_float4(b.lox, b.loy, b.loz, __int_as_float(l));
	p[1] = make_float4(b.hix, b.hiy, b.hiz, __int_as_float(r));
}

// Counters of one collapse: three depth counters used in turn (see kCollapse).
struct CollapseState
{
	collapsedev::DepthCounter depth[3];
};

// What the collapse tells the host about the stages before it.
struct BuildStages
{
	const uint32_t* sah;       // control words of the SAH topology, or null
	const int32_t* sortFailed; // flag of the radix sort, or null
	BuildReport* report;       // mapped host memory
};

// The whole collapse of a binary tree over n primitives in one cooperative launch, depth by depth with
// a grid barrier between (one launch per depth, sixteen between host checks of the queue, before). A
// depth adds to its own counter; the counter after next is cleared meanwhile, when nobody reads it.
// `st` is zero at the start. A SAH topology that is not complete is not collapsed: the report says so.
// levelStarts (optional) receives the first node of every depth and the node count, up to levelCap
// entries. 131,072 triangles: sixteen launches 516 us, one 100 us, with the leaf records written at the
// end, eight blocks per SM instead of four and the choices below 90 us (8 us a depth, see collapse.cuh
// for what bounds it; the barriers 1.4 each).
constexpr int kCollapseThreads = 128;
__global__ void __launch_bounds__(kCollapseThreads) kCollapse(CollapseInputs in, collapsedev::CollapseTarget out, int n, CollapseState* st,
                                                              int32_t* levelStarts, int32_t* nLevels, int levelCap, BuildStages stages)
{
	cooperative_groups::grid_group grid = cooperative_groups::this_grid();
	// Neighbouring nodes go to different SMs.
	const uint32_t warp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x, warps = gridDim.x * (kCollapseThreads / 32);
	const uint32_t group = (threadIdx.x & 31u) >> 3;
	const bool first = blockIdx.x == 0 && threadIdx.x == 0;
	uint32_t start = 0, end = 1, leaves = 0;
	int level = 0;
	volatile BuildReport* report = stages.report;
	if (stages.sah != nullptr) {
		const uint32_t nodes = stages.sah[kSahNodes], error = stages.sah[kSahError];
		if (first) {
			report->sahNodes = nodes;
			report->sahError = error;
		}
		if (error != 0u || nodes != (uint32_t) (n - 1)) {
			if (first) {
				report->done = 1;
				__threadfence_system();
			}
			return; // every block sees the same words
		}
	}
	for (; start < end; ++level) {
		collapsedev::DepthCounter* ctr = &st->depth[level % 3];
		if (first) {
			st->depth[(level + 1) % 3] = 0;
			if (levelStarts != nullptr && level < levelCap) {
				levelStarts[level] = (int32_t) start;
			}
		}
		for (uint32_t at = start + 4 * warp; at < end; at += 4 * warps) {
			const uint32_t idx = at + group;
			const bool valid = idx < end;
			collapsedev::CollapseTask task{0, 0};
			if (valid) {
				task = level == 0 ? collapsedev::rootTask(in.bin, n) : out.queue[idx];
			}
			if (in.vertices != nullptr) {
				collapsedev::collapseGroups<true>(valid, idx, task, in, out, ctr, end, leaves, (uint32_t) n);
			} else {
				collapsedev::collapseGroups<false>(valid, idx, task, in, out, ctr, end, leaves, (uint32_t) n);
			}
		}
		grid.sync();
		// Stable until the depth after next clears it, so every block takes the same decision.
		const collapsedev::DepthCounter got = *(volatile collapsedev::DepthCounter*) ctr;
		start = end;
		end += (uint32_t) got;
		leaves += (uint32_t) (got >> 32);
		if (end > (uint32_t) n || leaves > (uint32_t) n) {
			break; // not a proper tree; the host sees the counts
		}
	}
	if (in.vertices != nullptr && end <= (uint32_t) n && leaves == (uint32_t) n) { // every record has its position
		for (uint32_t i = blockIdx.x * kCollapseThreads + threadIdx.x; i < leaves; i += gridDim.x * kCollapseThreads) {
			collapsedev::writeTriangle(in, out.tris, i);
		}
	}
	if (first) {
		report->nodes = end;
		report->leaves = leaves;
		report->sortFailed = stages.sortFailed != nullptr ? *stages.sortFailed : 0;
		const float4* root = reinterpret_cast<const float4*>(in.bin);
		const float4 lo = n > 1 ? root[0] : in.triLo[0], hi = n > 1 ? root[1] : in.triHi[0];
		report->box[0] = lo.x;
		report->box[1] = lo.y;
		report->box[2] = lo.z;
		report->box[3] = hi.x;
		report->box[4] = hi.y;
		report->box[5] = hi.z;
		report->done = 1;
		__threadfence_system();
		if (levelStarts != nullptr && level < levelCap) {
			levelStarts[level] = (int32_t) end;
			*nLevels = level;
		}
	}
}

inline int blocks(int n, int b) { return (n + b - 1) / b; }

struct WideBuildResult
{
	uint32_t nodeCount;
	Box bounds;
};

// Where a collapse records the first node of every depth (device): levelCap entries and the depths.
struct LevelRecord
{
	int32_t* starts = nullptr;
	int32_t* count = nullptr;
	int capacity = 0;
};

void launchCollapse(CollapseInputs in, collapsedev::CollapseTarget out, int n, CollapseState* state, LevelRecord levels, BuildStages stages,
                    cudaStream_t s)
{
	static const int most = [] { // blocks that fit the device at once, as the grid barrier needs
		int dev = 0, sms = 0, perSm = 0;
		RGL_CUDA_OK(cudaGetDevice(&dev));
		RGL_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
		RGL_CUDA_OK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kCollapse, kCollapseThreads, 0));
		return sms * std::min(perSm, 8);
	}();
	// The widest depths hold about n / 5 nodes, 16 at a time per block; a small tree takes fewer blocks.
	int grid = std::max(1, std::min(most, n / 80));
	void* args[] = {&in, &out, &n, &state, &levels.starts, &levels.count, &levels.capacity, &stages};
	RGL_CUDA_OK(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(&kCollapse), dim3(grid), dim3(kCollapseThreads), args, 0, s));
	countLaunch();
}

// Wide BVH over n primitive boxes lo/hi (device), written on stream s: the binary topology (binned SAH, or
// with the centroid bounds cb, 6 words of kTriBounds, Morton codes, onesweep sort, LBVH and box
// pyramid), then the collapse into 8-wide nodes (one launch). Leaf records are triangles (dV/dI given) or
// primitive indices (dV null). `levels` optionally receives the first node index of every depth and the
// node count. The host waits once, for the report of the last kernel, so s is synchronised at the end.
WideBuildResult buildWide(const float4* lo, const float4* hi, const uint32_t* cb, int n, const float* dV, const int32_t* dI, int leafMax,
                          WideNode* outNodes, TriRecord* outLeaves, Box* outBoxes, cudaStream_t s, LevelRecord levels = {})
{
	const bool sah = cb == nullptr;
	BuildScratch scratch(s);
	uint32_t *codes = nullptr, *ids = nullptr, *ticket = nullptr;
	uint8_t* sortScratch = nullptr;
	BinNode* bin = nullptr;
	int32_t *rf = nullptr, *rl = nullptr, *err = nullptr;
	BoxPyramid pyramid{nullptr, nullptr};
	collapsedev::CollapseTask* queue = nullptr;
	CollapseState* state = nullptr;
	scratch.carve([&](BuildScratch::Carver& place) {
		place(state, 1); // cleared together: state, err, ticket and the start of the sort's scratch
		place(err, 1);
		place(ticket, 1);
		if (!sah) {
			place(sortScratch, sortPairsScratchBytes(n, kKeyBits));
			place(codes, n);
			place(pyramid.lo, pyramidBoxes(n));
			place(pyramid.hi, pyramidBoxes(n));
		}
		place(ids, n);
		place(bin, n);
		place(rf, n);
		place(rl, n);
		place(queue, n);
	});
	const uint8_t* cleared = sah ? reinterpret_cast<const uint8_t*>(ticket + 1) : sortScratch + sortPairsZeroBytes(n, kKeyBits);
	RGL_CUDA_OK(cudaMemsetAsync(state, 0, cleared - reinterpret_cast<const uint8_t*>(state), s));

	BuildScratch sahScratch(s);
	const uint32_t* sahControl = nullptr;
	if (sah) {
		sahControl = enqueueSahTopology(sahScratch, lo, hi, n, bin, rf, rl, ids, s);
	} else {
		kMorton<<<blocks(n, kMortonItems * 256), 256, 0, s>>>(lo, hi, n, cb, codes, ids, reinterpret_cast<uint32_t*>(sortScratch));
		countLaunch();
		sortCountedPairs(codes, ids, n, kKeyBits, sortScratch, err, s);
		if (n > 1) {
			kBoxPyramid<<<blocks(n, kPyramidTile), kPyramidThreads, 0, s>>>(ids, lo, hi, n, pyramid, ticket);
			countLaunch();
			kLbvh<<<blocks(n - 1, 128), 128, 0, s>>>(codes, n, bin, rf, rl, pyramid);
			countLaunch();
		}
	}
	HostReport report;
	const CollapseInputs ci{bin, rf, rl, reinterpret_cast<const int32_t*>(ids), lo, hi, dV, dI, leafMax};
	const BuildStages stages{sahControl, err, report.device()};
	const volatile BuildReport& r = *report.host();
	launchCollapse(ci, collapsedev::CollapseTarget{outNodes, outLeaves, outBoxes, queue}, n, state, levels, stages, s);
	RGL_CUDA_OK(cudaStreamSynchronize(s));
	scratch.waited();
	sahScratch.waited();
	if (r.done == 0) {
		throw std::runtime_error("BVH build: the collapse did not report");
	}
	if (r.sahError != 0) {
		throw std::runtime_error("SAH build: a partition or range stack index left its range");
	}
	if (stages.sah != nullptr && r.sahNodes != (uint32_t) (n - 1)) {
		throw std::runtime_error("SAH build: " + std::to_string(r.sahNodes) + " binary nodes for " + std::to_string(n) + " primitives");
	}
	if (r.sortFailed != 0) {
		throw std::runtime_error("BVH build: radix sort look-back did not complete");
	}
	if (r.leaves != (uint32_t) n || r.nodes > (uint32_t) n) {
		throw std::runtime_error("BVH build: collapse produced an inconsistent tree (leaf records " + std::to_string(r.leaves) + ", nodes " +
		                         std::to_string(r.nodes) + ")");
	}
	return WideBuildResult{r.nodes, Box{r.box[0], r.box[1], r.box[2], r.box[3], r.box[4], r.box[5]}};
}

void allocBlas(BlasBuild& out, int nTris, cudaStream_t s)
{
	// A rebuild (an animated entity) reuses the previous storage when it is large enough.
	if (out.nodes == nullptr || out.nodeCapacity < (uint32_t) nTris) {
		freeBlas(out);
		out.nodes = static_cast<WideNode*>(allocateStorage(sizeof(WideNode) * (size_t) nTris, s));
		out.tris = static_cast<TriRecord*>(allocateStorage(sizeof(TriRecord) * (size_t) nTris, s));
		out.nodeCapacity = (uint32_t) nTris;
	}
}

} // namespace

void buildBlas(const float* dVertices, int nVertices, const int32_t* dIndices, int nTris, BlasBuild& out, cudaStream_t s, bool sah)
{
	(void) nVertices;
	if (nTris <= 0) {
		throw std::invalid_argument("mesh without triangles");
	}
	const int T = nTris;
	BuildScratch scratch(s);
	float4 *lo = nullptr, *hi = nullptr;
	uint32_t* cb = nullptr;
	scratch.carve([&](BuildScratch::Carver& place) {
		place(lo, T);
		place(hi, T);
		if (!sah) {
			place(cb, 6);
		}
	});
	allocBlas(out, T, s);
	out.triCount = T;
	if (!sah) {
		RGL_CUDA_OK(cudaMemsetAsync(cb, 0, 6 * sizeof(uint32_t), s));
	}
	kTriBounds<<<blocks(T, 256), 256, 0, s>>>(dVertices, dIndices, T, lo, hi, cb);
	countLaunch();
	const WideBuildResult r = buildWide(lo, hi, cb, T, dVertices, dIndices, kLeafMaxTris, out.nodes, out.tris, nullptr, s);
	scratch.waited();
	out.nodeCount = r.nodeCount;
	out.bounds[0] = r.bounds.lox;
	out.bounds[1] = r.bounds.loy;
	out.bounds[2] = r.bounds.loz;
	out.bounds[3] = r.bounds.hix;
	out.bounds[4] = r.bounds.hiy;
	out.bounds[5] = r.bounds.hiz;
}

void buildBlasHost(const float* hVertices, int nVertices, const int32_t* hIndices, int nTris, BlasBuild& out)
{
	(void) nVertices;
	if (nTris <= 0) {
		throw std::invalid_argument("mesh without triangles");
	}
	const int T = nTris;
	std::vector<Box> boxes(T);
	std::vector<float4> lo(T), hi(T);
	for (int t = 0; t < T; ++t) {
		const float* a = hVertices + 3 * hIndices[3 * t];
		const float* b = hVertices + 3 * hIndices[3 * t + 1];
		const float* c = hVertices + 3 * hIndices[3 * t + 2];
		Box bx{std::min(a[0], std::min(b[0], c[0])), std::min(a[1], std::min(b[1], c[1])), std::min(a[2], std::min(b[2], c[2])),
		       std::max(a[0], std::max(b[0], c[0])), std::max(a[1], std::max(b[1], c[1])), std::max(a[2], std::max(b[2], c[2]))};
		boxes[t] = bx;
		lo[t] = make_float4(bx.lox, bx.loy, bx.loz, 0.0f);
		hi[t] = make_float4(bx.hix, bx.hiy, bx.hiz, 0.0f);
	}
	const SahTree tree = buildBinnedSahTree(boxes);
	std::vector<WideNode> wide(T);
	std::vector<TriRecord> tris(T);
	uint32_t wideCounter = 1, triCounter = 0;
	std::vector<int2> qa(T), qb(T);
	uint32_t qaCount = 1, qbCount = 0;
	qa[0] = make_int2(T == 1 ? ~0 : 0, 0);
	CollapseInputs in{tree.bin.data(), tree.rangeFirst.data(), tree.rangeLast.data(), tree.sortedIds.data(), lo.data(), hi.data(),
	                  hVertices, hIndices, kLeafMaxTris};
	while (qaCount > 0) {
		qbCount = 0;
		CollapseOutputs o{wide.data(), tris.data(), &wideCounter, &triCounter, qb.data(), &qbCount, nullptr};
		for (uint32_t i = 0; i < qaCount; ++i) {
			collapseItem(qa[i].x, (uint32_t) qa[i].y, in, o);
		}
		std::swap(qa, qb);
		qaCount = qbCount;
	}
	if (triCounter != (uint32_t) T || wideCounter > (uint32_t) T) {
		throw std::runtime_error("BLAS build: collapse produced an inconsistent tree");
	}
	allocBlas(out, T, nullptr);
	RGL_CUDA_OK(cudaMemcpy(out.nodes, wide.data(), sizeof(WideNode) * wideCounter, cudaMemcpyHostToDevice));
	RGL_CUDA_OK(cudaMemcpy(out.tris, tris.data(), sizeof(TriRecord) * (size_t) T, cudaMemcpyHostToDevice));
	out.nodeCount = wideCounter;
	out.triCount = T;
	const Box root = T == 1 ? boxes[0] : Box{tree.bin[0].lox, tree.bin[0].loy, tree.bin[0].loz, tree.bin[0].hix, tree.bin[0].hiy, tree.bin[0].hiz};
	out.bounds[0] = root.lox;
	out.bounds[1] = root.loy;
	out.bounds[2] = root.loz;
	out.bounds[3] = root.hix;
	out.bounds[4] = root.hiy;
	out.bounds[5] = root.hiz;
}

void freeBlas(BlasBuild& b)
{
	freeStorage(b.nodes);
	freeStorage(b.tris);
	b.nodes = nullptr;
	b.tris = nullptr;
	b.nodeCapacity = 0;
}

namespace {

// TLAS refit after pose changes, one block: depth by depth from the leaves up, every wide node takes
// the union of its children's boxes (child nodes' stored boxes, instances' world boxes) and
// re-quantises its children in a new frame with the builder's arithmetic. Topology and slots stay.
__global__ void __launch_bounds__(256) kRefitTlas(WideNode* nodes, const TriRecord* __restrict__ leaves, Box* boxes,
                                                  const InstanceRec* __restrict__ inst, const int32_t* __restrict__ levelStarts,
                                                  const int32_t* __restrict__ nLevelsWord)
{
	const int nLevels = *nLevelsWord;
	for (int L = nLevels - 1; L >= 0; --L) {
		const int a = levelStarts[L], b = levelStarts[L + 1];
		for (int i = a + (int) threadIdx.x; i < b; i += blockDim.x) {
			WideNode w = nodes[i];
			Box cbx[kWideArity];
			uint32_t present = 0;
			Box nb = emptyBox();
			for (int k = 0; k < kWideArity; ++k) {
				const bool internal = (w.imask >> k) & 1u;
				if (!internal && w.meta[k] == 0) {
					continue;
				}
				if (internal) {
					cbx[k] = boxes[w.childBase + (uint32_t) __popc(w.imask & ((1u << k) - 1u))];
				} else {
					const InstanceRec& r = inst[leaves[w.triBase + (w.meta[k] & 31u)].primId];
					cbx[k] = Box{r.lox, r.loy, r.loz, r.hix, r.hiy, r.hiz};
				}
				present |= 1u << k;
				nb = unite(nb, cbx[k]);
			}
			setWideFrame(w, nb);
			for (int k = 0; k < kWideArity; ++k) {
				if ((present >> k) & 1u) {
					quantizeChild(w, k, cbx[k]);
				} else {
					clearChild(w, k);
				}
			}
			nodes[i] = w;
			boxes[i] = nb;
		}
		__syncthreads();
	}
}

// Shared-memory layout of the one-block collapse over n primitives (16-byte aligned parts): primitive
// boxes lo[n] | hi[n] | binary nodes[n - 1] | queue[n] | sorted ids[n] | ranges first[n - 1],
// last[n - 1] | depth counters[3].
struct SmallCollapseLayout
{
	size_t lo, hi, bin, queue, ids, rf, rl, ctr, bytes;
};
__host__ __device__ SmallCollapseLayout smallCollapseLayout(int n)
{
	auto up = [](size_t b) { return (b + 15) & ~size_t{15}; };
	const size_t m = (size_t) (n > 1 ? n - 1 : 1);
	SmallCollapseLayout L;
	L.lo = 0;
	L.hi = L.lo + up(sizeof(float4) * (size_t) n);
	L.bin = L.hi + up(sizeof(float4) * (size_t) n);
	L.queue = L.bin + up(sizeof(BinNode) * m);
	L.ids = L.queue + up(sizeof(collapsedev::CollapseTask) * (size_t) n);
	L.rf = L.ids + up(sizeof(int32_t) * (size_t) n);
	L.rl = L.rf + up(sizeof(int32_t) * m);
	L.ctr = L.rl + up(sizeof(int32_t) * m);
	L.bytes = L.ctr + up(3 * sizeof(collapsedev::DepthCounter));
	return L;
}

// The wide collapse of a small binary tree by one block, depth by depth (as kCollapse, with block
// barriers). The tree, the primitive boxes, the queue and the counters live in shared memory, so each
// depth costs shared-memory latency, not a chain of global loads. Records the first node of every depth
// and the number of depths. 94 instances: 172 us with one thread per node.
constexpr int kSmallThreads = 256;
__global__ void __launch_bounds__(kSmallThreads) kCollapseSmall(CollapseInputs gin, WideNode* wide, TriRecord* leaves, Box* boxes,
                                                                const InstanceRec* __restrict__ inst, EnterRec* enter,
                                                                int32_t* levelStarts, int32_t* nLevels, int n)
{
	extern __shared__ __align__(16) uint8_t smem[];
	const SmallCollapseLayout L = smallCollapseLayout(n);
	float4* lo = reinterpret_cast<float4*>(smem + L.lo);
	float4* hi = reinterpret_cast<float4*>(smem + L.hi);
	BinNode* bin = reinterpret_cast<BinNode*>(smem + L.bin);
	collapsedev::CollapseTask* queue = reinterpret_cast<collapsedev::CollapseTask*>(smem + L.queue);
	int32_t* ids = reinterpret_cast<int32_t*>(smem + L.ids);
	int32_t* rf = reinterpret_cast<int32_t*>(smem + L.rf);
	int32_t* rl = reinterpret_cast<int32_t*>(smem + L.rl);
	collapsedev::DepthCounter* depth = reinterpret_cast<collapsedev::DepthCounter*>(smem + L.ctr);
	for (int i = threadIdx.x; i < n; i += blockDim.x) {
		lo[i] = gin.triLo[i];
		hi[i] = gin.triHi[i];
		ids[i] = gin.sortedIds[i];
	}
	for (int i = threadIdx.x; i < n - 1; i += blockDim.x) {
		bin[i] = gin.bin[i];
		rf[i] = gin.rangeFirst[i];
		rl[i] = gin.rangeLast[i];
	}
	if (threadIdx.x < 3) {
		depth[threadIdx.x] = 0;
	}
	__syncthreads();
	const CollapseInputs in{bin, rf, rl, ids, lo, hi, nullptr, nullptr, gin.leafMax};
	const collapsedev::CollapseTarget out{wide, leaves, boxes, queue};
	const uint32_t warp = threadIdx.x >> 5, warps = blockDim.x >> 5, group = (threadIdx.x & 31u) >> 3;
	uint32_t start = 0, end = 1, done = 0;
	int level = 0;
	for (; start < end; ++level) {
		collapsedev::DepthCounter* ctr = &depth[level % 3];
		if (threadIdx.x == 0) {
			depth[(level + 1) % 3] = 0;
			levelStarts[level] = (int32_t) start; // n + 2 entries: every depth holds a node
		}
		for (uint32_t at = start + 4 * warp; at < end; at += 4 * warps) {
			const uint32_t idx = at + group;
			const bool valid = idx < end;
			collapsedev::CollapseTask task{0, 0};
			if (valid) {
				task = level == 0 ? collapsedev::rootTask(bin, n) : queue[idx];
			}
			collapsedev::collapseGroups<false>(valid, idx, task, in, out, ctr, end, done, (uint32_t) n);
		}
		__syncthreads();
		const collapsedev::DepthCounter got = *(volatile collapsedev::DepthCounter*) ctr;
		start = end;
		end += (uint32_t) got;
		done += (uint32_t) (got >> 32);
		if (end > (uint32_t) n || done > (uint32_t) n) {
			break; // not a proper tree
		}
	}
	if (threadIdx.x == 0) {
		levelStarts[level] = (int32_t) end;
		*nLevels = level;
	}
	for (int i = threadIdx.x; i < n; i += blockDim.x) {
		const int32_t k = leaves[i].primId; // written by this block before its last barrier
		enter[i] = enterRecord(inst[k], k);
	}
}

// Enter records of the TLAS's leaf records (after a build or a refit of more than kSahSmallMax instances;
// the one-block collapse writes them itself).
__global__ void kEnterRecords(const TriRecord* __restrict__ leaves, const InstanceRec* __restrict__ inst, int n, EnterRec* enter)
{
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n) {
		const int32_t k = leaves[i].primId;
		enter[i] = enterRecord(inst[k], k);
	}
}

} // namespace

// The TLAS is a wide BVH over the instances' world boxes, one instance per leaf child, built on the
// device like a mesh BLAS (binned SAH topology, then the wide collapse with one instance per leaf).
// The node range of every depth (contiguous: the collapse allocates nodes depth by depth) drives the
// refit kernel.
namespace {

// Shared memory of the one-block kernels, set outside any capture and for the largest scene: the limit is the
// kernel's, so a small scene must not lower it under a large one.
void prepareSmallTlas()
{
	static const bool done = [] {
		prepareSahBlock();
		RGL_CUDA_OK(cudaFuncSetAttribute(kCollapseSmall, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smallCollapseLayout(kSahSmallMax).bytes));
		return true;
	}();
	(void) done;
}

// The rebuild of up to kSahSmallMax instances from their device records: two launches, no host
// interaction, so a captured frame can hold it.
void rebuildTlas(const InstanceRec* dInst, TlasBuild& t, cudaStream_t s)
{
	const int n = t.nInstances;
	enqueueSahTopologySmall(dInst, t.lo, t.hi, n, t.bin, t.rangeFirst, t.rangeLast, t.sortedIds, s);
	const CollapseInputs ci{t.bin, t.rangeFirst, t.rangeLast, reinterpret_cast<const int32_t*>(t.sortedIds), t.lo, t.hi, nullptr, nullptr, 1};
	kCollapseSmall<<<1, kSmallThreads, smallCollapseLayout(n).bytes, s>>>(ci, t.nodes, t.leaves, reinterpret_cast<Box*>(t.boxes), dInst,
	                                                                      t.enter, t.levelStarts, t.nLevels, n);
	countLaunch();
}

} // namespace

void buildTlas(const InstanceRec* hInst, const InstanceRec* dInst, int n, TlasBuild& t, cudaStream_t s)
{
	if (n > 0) {
		allocateTlas(t, n);
	}
	t.nInstances = n;
	t.nodeCount = 0;
	if (n <= 0) {
		return;
	}
	if (n <= kSahSmallMax) {
		prepareSmallTlas();
		rebuildTlas(dInst, t, s);
		return;
	}
	std::vector<float4> hLo(n), hHi(n);
	for (int i = 0; i < n; ++i) {
		const InstanceRec& r = hInst[i];
		hLo[i] = make_float4(r.lox, r.loy, r.loz, 0.0f);
		hHi[i] = make_float4(r.hix, r.hiy, r.hiz, 0.0f);
	}
	BuildScratch scratch(s);
	float4 *lo = nullptr, *hi = nullptr;
	scratch.carve([&](BuildScratch::Carver& place) {
		place(lo, n);
		place(hi, n);
	});
	// Pageable sources: each copy is staged before the call returns.
	RGL_CUDA_OK(cudaMemcpyAsync(lo, hLo.data(), sizeof(float4) * (size_t) n, cudaMemcpyHostToDevice, s));
	RGL_CUDA_OK(cudaMemcpyAsync(hi, hHi.data(), sizeof(float4) * (size_t) n, cudaMemcpyHostToDevice, s));
	const WideBuildResult r = buildWide(lo, hi, nullptr, n, nullptr, nullptr, 1, t.nodes, t.leaves, reinterpret_cast<Box*>(t.boxes), s,
	                                    LevelRecord{t.levelStarts, t.nLevels, t.levelCapacity});
	scratch.waited();
	t.nodeCount = r.nodeCount;
	kEnterRecords<<<blocks(n, 128), 128, 0, s>>>(t.leaves, dInst, n, t.enter);
	countLaunch();
}

void updateTlas(const InstanceRec* dInst, TlasBuild& t, cudaStream_t s)
{
	if (t.nInstances <= 0) {
		return;
	}
	if (t.nInstances <= kSahSmallMax) {
		rebuildTlas(dInst, t, s);
	} else {
		refitTlas(dInst, t, s);
	}
}

void refitTlas(const InstanceRec* dInst, TlasBuild& t, cudaStream_t s)
{
	if (t.nInstances <= 0) {
		return;
	}
	kRefitTlas<<<1, 256, 0, s>>>(t.nodes, t.leaves, reinterpret_cast<Box*>(t.boxes), dInst, t.levelStarts, t.nLevels);
	kEnterRecords<<<blocks(t.nInstances, 128), 128, 0, s>>>(t.leaves, dInst, t.nInstances, t.enter);
	countLaunch(2);
}

} // namespace rgl
