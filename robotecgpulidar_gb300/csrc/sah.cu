// On-device binned SAH topology for mesh BLASes: the binary tree of the host builder
// (sah_build.hpp buildBinnedSahTree), computed on the GPU with the same float arithmetic, so the
// device tree equals the host tree node for node and the sorted primitive order equals the host's.
//
// Replaces OptiX's GAS build of reference src/scene/GASBuilder.hpp:31-100 (optixAccelBuild), which
// runs on the device; the wide collapse and quantisation that follow are bvh_core.hpp's.
//
// Algorithm (after Wald 2007, binned SAH, 32 bins per axis; parallel top-down):
//  * ranges of more than kBigTask primitives are split level by level, each by many blocks, all levels in
//    one cooperative launch (kSahLevels): one warp per range evaluates the 3 x 31 split candidates from
//    the range's bins; a pass over the elements counts how many go left and gathers the children's bounds;
//    a second one puts them in their place (stable: counts of earlier chunks, then a block scan) and adds
//    them to their child's bins (shared-memory atomics, then the range's);
//  * ranges of 2..kBigTask primitives are built to the leaves by one block each, in shared memory
//    (kSahBlock); blocks take ranges until none is left.
// Exactness: boxes and centroid bounds are min/max (order free); the centroid, the bin index, the
// half areas and the split costs use the host's expressions with round-to-nearest intrinsics and no
// FMA contraction; among equal costs the first candidate in (axis, bin) order wins, as in the host's
// strict comparison; partitions are stable; a range whose centroids all coincide splits in the
// middle. Node numbering differs from the host's (atomics instead of a depth-first counter); the
// collapse does not depend on it.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <stdexcept>
#include <string>

#include "bvh_core.hpp"
#include "kernels.hpp"

namespace rgl {

struct SahTask
{
	int32_t lo, hi, node, pad; // sorted positions [lo, hi), binary node index
};

struct SahSplit
{
	int32_t axis, bin, nLeft, pad; // axis -1: split in the middle
};

namespace {

#define RGL_SAH_OK(expr)                                                                                                       \
	do {                                                                                                                       \
		cudaError_t e_ = (expr);                                                                                               \
		if (e_ != cudaSuccess) {                                                                                               \
			throw std::runtime_error(std::string("CUDA error in SAH build: ") + cudaGetErrorString(e_) + " at " #expr);        \
		}                                                                                                                      \
	} while (0)

constexpr int kBins = 32;
constexpr int kBinWords = 7;                    // lo xyz (ordered bits, complemented), hi xyz (ordered bits), count: empty is 0
constexpr int kTaskBinWords = 3 * kBins * kBinWords;
// Larger ranges split in the level loop, the others are built by a block each. 131,072 triangles, 2,048 /
// 1,024 / 512: levels 166 / 194 / 222 us, blocks 231 / 143 / 120 us, before the bins were filled out of step.
constexpr int kBigTask = 1024;
constexpr int kMeshThreads = 512;
constexpr int kChunk = 512;                     // elements per block in the level loop: 256 blocks for 131,072 triangles
constexpr int kThreads = 256;
constexpr int kItems = kChunk / kThreads;       // 2 elements per thread
constexpr int kSmallTask = 32;                  // ranges up to this size: one warp
constexpr int kWarps = kThreads / 32;
constexpr uint32_t kEmptyLo = 0xffffffffu;      // identity of min over ordered bits
constexpr uint32_t kEmptyHi = 0u;               // identity of max
constexpr float kInf = __builtin_huge_valf();

__device__ __forceinline__ uint32_t ordered(float f)
{
	const uint32_t u = __float_as_uint(f);
	return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float unordered(uint32_t u) { return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u); }

// The host's expressions (sah_build.hpp), without contraction.
__device__ __forceinline__ float halfAreaOf(float lx, float ly, float lz, float hx, float hy, float hz)
{
	const float dx = __fsub_rn(hx, lx), dy = __fsub_rn(hy, ly), dz = __fsub_rn(hz, lz);
	return __fadd_rn(__fadd_rn(__fmul_rn(dx, dy), __fmul_rn(dy, dz)), __fmul_rn(dz, dx));
}
__device__ __forceinline__ int binOf(float c, float cmin, float scale)
{
	const int b = (int) __fmul_rn(__fsub_rn(c, cmin), scale); // >= 0 for finite input; clamped for any
	return b < 0 ? 0 : (b < kBins - 1 ? b : kBins - 1);
}
__device__ __forceinline__ float comp3(const float4& v, int a) { return a == 0 ? v.x : (a == 1 ? v.y : v.z); }

// Node box and centroid bounds of a range, 12 ordered words: box lo xyz, box hi xyz, centroid lo
// xyz, centroid hi xyz.
struct Bounds12
{
	uint32_t w[12];
	__device__ __forceinline__ void clear()
	{
#pragma unroll
		for (int k = 0; k < 12; ++k) {
			w[k] = (k < 3 || (k >= 6 && k < 9)) ? kEmptyLo : kEmptyHi;
		}
	}
	__device__ __forceinline__ void add(const float4& l, const float4& h, const float4& c)
	{
		w[0] = min(w[0], ordered(l.x));
		w[1] = min(w[1], ordered(l.y));
		w[2] = min(w[2], ordered(l.z));
		w[3] = max(w[3], ordered(h.x));
		w[4] = max(w[4], ordered(h.y));
		w[5] = max(w[5], ordered(h.z));
		w[6] = min(w[6], ordered(c.x));
		w[7] = min(w[7], ordered(c.y));
		w[8] = min(w[8], ordered(c.z));
		w[9] = max(w[9], ordered(c.x));
		w[10] = max(w[10], ordered(c.y));
		w[11] = max(w[11], ordered(c.z));
	}
	__device__ __forceinline__ void warpReduce()
	{
#pragma unroll
		for (int k = 0; k < 12; ++k) {
			const bool isMin = k < 3 || (k >= 6 && k < 9);
			w[k] = isMin ? __reduce_min_sync(0xffffffffu, w[k]) : __reduce_max_sync(0xffffffffu, w[k]);
		}
	}
};
__device__ __forceinline__ bool isMinWord(int k) { return k < 3 || (k >= 6 && k < 9); }

// Binning frame of one axis: valid when the centroids spread along it (the host's ext > 0).
struct AxisFrame
{
	float cmin, scale;
	bool valid;
};
__device__ __forceinline__ AxisFrame axisFrame(const uint32_t* b12, int a)
{
	AxisFrame f;
	f.cmin = unordered(b12[6 + a]);
	const float ext = __fsub_rn(unordered(b12[9 + a]), f.cmin);
	f.valid = ext > 0.0f;
	f.scale = f.valid ? __fdiv_rn((float) kBins, ext) : 0.0f;
	return f;
}

// Adds an element to its bin of every axis. Neighbouring elements of a mesh share bins, and 32 lanes adding
// to one word take turns; so every lane goes through the axes and words from a place of its own: a value is
// turned by the lane's number, as the word it goes to (131,072 triangles of a terrain: levels 183 us in step,
// 167 so, block ranges 141 and 122; 94 instances 32 and 27).
__device__ __forceinline__ void addToBins(uint32_t* bins, const float4& l, const float4& h, const float4& c, const AxisFrame (&fr)[3])
{
	const uint32_t lane = threadIdx.x & 31u, turn = lane % 6u, third = lane % 3u;
	uint32_t v[6] = {~ordered(l.x), ~ordered(l.y), ~ordered(l.z), ordered(h.x), ordered(h.y), ordered(h.z)};
#pragma unroll
	for (int by = 1; by < 6; by <<= 1) {
		uint32_t t[6];
#pragma unroll
		for (int j = 0; j < 6; ++j) {
			t[j] = (turn & (uint32_t) by) != 0u ? v[(j + by) % 6] : v[j];
		}
#pragma unroll
		for (int j = 0; j < 6; ++j) {
			v[j] = t[j];
		}
	}
	int at[3];
#pragma unroll
	for (int a = 0; a < 3; ++a) {
		at[a] = fr[a].valid ? (a * kBins + binOf(comp3(c, a), fr[a].cmin, fr[a].scale)) * kBinWords : -1;
	}
	const int first = third == 0u ? at[0] : (third == 1u ? at[1] : at[2]), second = third == 0u ? at[1] : (third == 1u ? at[2] : at[0]),
	          last = third == 0u ? at[2] : (third == 1u ? at[0] : at[1]);
	const int order[3] = {first, second, last};
#pragma unroll
	for (int a = 0; a < 3; ++a) {
		if (order[a] < 0) {
			continue;
		}
		uint32_t* bin = bins + order[a];
#pragma unroll
		for (uint32_t j = 0; j < 6; ++j) {
			atomicMax(bin + (turn + j < 6u ? turn + j : turn + j - 6u), v[j]);
		}
		atomicAdd(bin + 6, 1u);
	}
}

// Best split of a range from its bins (3 x 32 x 7 words, any address space) and bounds, by one warp:
// the candidate between bins b-1 and b of axis a costs halfArea(left) * nLeft + halfArea(right) * nRight;
// candidates with an empty side are skipped; the lowest cost wins, the first in (axis, b) order among
// equal costs. Returns axis -1 when no axis has spread centroids.
__device__ SahSplit warpBestSplit(const uint32_t* bins, const uint32_t* b12, int lane)
{
	float bestCost = kInf;
	int bestKey = 1 << 30, bestLeft = 0;
	uint32_t v[3][kBinWords]; // all at once: the loads do not wait for each other
#pragma unroll
	for (int a = 0; a < 3; ++a) {
#pragma unroll
		for (int k = 0; k < kBinWords; ++k) {
			const uint32_t word = bins[(a * kBins + lane) * kBinWords + k];
			v[a][k] = k < 3 ? ~word : word;
		}
	}
#pragma unroll
	for (int a = 0; a < 3; ++a) {
		const AxisFrame f = axisFrame(b12, a);
		if (!f.valid) {
			continue;
		}
		// inclusive prefix (bins 0..lane) and suffix (bins lane..31)
		uint32_t p[kBinWords], q[kBinWords];
#pragma unroll
		for (int k = 0; k < kBinWords; ++k) {
			p[k] = v[a][k];
			q[k] = v[a][k];
		}
#pragma unroll
		for (int off = 1; off < 32; off <<= 1) {
#pragma unroll
			for (int k = 0; k < kBinWords; ++k) {
				const uint32_t up = __shfl_up_sync(0xffffffffu, p[k], off);
				const uint32_t dn = __shfl_down_sync(0xffffffffu, q[k], off);
				if (lane >= off) {
					p[k] = k < 3 ? min(p[k], up) : (k < 6 ? max(p[k], up) : p[k] + up);
				}
				if (lane + off < 32) {
					q[k] = k < 3 ? min(q[k], dn) : (k < 6 ? max(q[k], dn) : q[k] + dn);
				}
			}
		}
		// left side of candidate `lane` = prefix of lane - 1
		uint32_t l[kBinWords];
#pragma unroll
		for (int k = 0; k < kBinWords; ++k) {
			l[k] = __shfl_up_sync(0xffffffffu, p[k], 1);
		}
		const uint32_t lc = l[6], rc = q[6];
		if (lane >= 1 && lc != 0u && rc != 0u) {
			const float ha = halfAreaOf(unordered(l[0]), unordered(l[1]), unordered(l[2]), unordered(l[3]), unordered(l[4]), unordered(l[5]));
			const float hb = halfAreaOf(unordered(q[0]), unordered(q[1]), unordered(q[2]), unordered(q[3]), unordered(q[4]), unordered(q[5]));
			const float cost = __fadd_rn(__fmul_rn(ha, (float) lc), __fmul_rn(hb, (float) rc));
			if (cost < bestCost) {
				bestCost = cost;
				bestKey = a * kBins + lane;
				bestLeft = (int) lc;
			}
		}
	}
	// warp argmin over (cost, key)
#pragma unroll
	for (int off = 16; off >= 1; off >>= 1) {
		const float oc = __shfl_xor_sync(0xffffffffu, bestCost, off);
		const int ok = __shfl_xor_sync(0xffffffffu, bestKey, off);
		const int ol = __shfl_xor_sync(0xffffffffu, bestLeft, off);
		if (oc < bestCost || (oc == bestCost && ok < bestKey)) {
			bestCost = oc;
			bestKey = ok;
			bestLeft = ol;
		}
	}
	SahSplit s;
	if (bestKey >= (1 << 30)) {
		s.axis = -1;
		s.bin = 0;
		s.nLeft = 0;
	} else {
		s.axis = bestKey / kBins;
		s.bin = bestKey % kBins;
		s.nLeft = bestLeft;
	}
	s.pad = 0;
	return s;
}

// ------------------------------------------------------------------ level loop (ranges > kBigTask)

// One range of at most kBigTask primitives: its order, its task and the control words.
__global__ void kSahInit(int n, uint32_t* sorted, SahTask* blockTasks, uint32_t* ctr)
{
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n) {
		sorted[i] = (uint32_t) i;
	}
	if (i < kSahWords) {
		ctr[i] = i == kSahNodes || i == kSahBlocks ? 1u : 0u; // the root
	}
	if (i == 0) {
		blockTasks[0] = SahTask{0, n, 0, 0};
	}
}

// Block-wide exclusive scan of one int per thread; returns the prefix and the block total.
template<int WARPS = kWarps>
__device__ __forceinline__ int blockExclusiveScan(int v, int* sW, int& total)
{
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	int incl = v;
#pragma unroll
	for (int off = 1; off < 32; off <<= 1) {
		const int u = __shfl_up_sync(0xffffffffu, incl, off);
		if (lane >= off) {
			incl += u;
		}
	}
	if (lane == 31) {
		sW[warp] = incl;
	}
	__syncthreads();
	int before = 0;
	total = 0;
	for (int w = 0; w < WARPS; ++w) {
		const int x = sW[w];
		before += w < warp ? x : 0;
		total += x;
	}
	__syncthreads();
	return before + incl - v;
}

// Where nodes go.
struct NodeSink
{
	BinNode* bin;
	int32_t* rangeFirst;
	int32_t* rangeLast;
	uint32_t* ctr; // control words, or null (a one-block build: no other block, nobody reads the error word)
	__device__ __forceinline__ void error() const
	{
		if (ctr != nullptr) {
			atomicExch(&ctr[kSahError], 1u);
		}
	}
	__device__ __forceinline__ void write(int node, int lo, int hi, const uint32_t* b12, int32_t left, int32_t right) const
	{
		float4* p = reinterpret_cast<float4*>(bin + node);
		p[0] = make_float4(unordered(b12[0]), unordered(b12[1]), unordered(b12[2]), __int_as_float(left));
		p[1] = make_float4(unordered(b12[3]), unordered(b12[4]), unordered(b12[5]), __int_as_float(right));
		rangeFirst[node] = lo;
		rangeLast[node] = hi - 1;
	}
};

// What a range's warp decides: the split, and the children's places among the next level's ranges (-1:
// not one of them).
struct LevelSplit
{
	SahSplit split;
	int32_t child[2];
};

// Memory of the level loop; pairs are used in turn by the levels.
struct SahLevels
{
	int n;
	uint32_t *ids[2], *sorted;
	SahTask *tasks[2], *blockTasks;
	uint32_t *bounds[2], *bins;
	int32_t *chunkBase[2], *chunkTask[2]; // first chunk of every range and the chunks; range of every chunk
	int32_t* chunkLeft;                   // left elements of a chunk
	LevelSplit* splits;
	int maxBig;
	BinNode* bin;
	int32_t *rangeFirst, *rangeLast;
	uint32_t* ctr;
};

// Adds a block's bounds to those of up to two ranges, null for none (every thread calls it; ends with a
// barrier).
template<int RANGES>
__device__ __forceinline__ void blockAddBounds(Bounds12 (&b)[RANGES], uint32_t (*sRed)[kWarps][12], uint32_t* const (&out)[RANGES])
{
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
	for (int r = 0; r < RANGES; ++r) {
		if (out[r] == nullptr) {
			continue;
		}
		b[r].warpReduce();
		if (lane == 0) {
#pragma unroll
			for (int k = 0; k < 12; ++k) {
				sRed[r][warp][k] = b[r].w[k];
			}
		}
	}
	__syncthreads();
#pragma unroll
	for (int r = 0; r < RANGES; ++r) {
		const int k = (int) threadIdx.x - 32 * r; // one warp each
		if (out[r] != nullptr && k >= 0 && k < 12) {
			uint32_t v = sRed[r][0][k];
#pragma unroll
			for (int w = 1; w < kWarps; ++w) {
				v = isMinWord(k) ? min(v, sRed[r][w][k]) : max(v, sRed[r][w][k]);
			}
			if (isMinWord(k)) {
				atomicMin(&out[r][k], v);
			} else {
				atomicMax(&out[r][k], v);
			}
		}
	}
	__syncthreads();
}

__device__ __forceinline__ float4 centroidOf(const float4& l, const float4& h)
{
	return make_float4(__fmul_rn(0.5f, __fadd_rn(l.x, h.x)), __fmul_rn(0.5f, __fadd_rn(l.y, h.y)), __fmul_rn(0.5f, __fadd_rn(l.z, h.z)), 0.0f);
}

__device__ __forceinline__ void clearBins(uint32_t* bins, int first, int step, int words = kTaskBinWords)
{
	for (int k = first; k < words; k += step) {
		bins[k] = 0u;
	}
}

// A block's bins of a range added to the range's; the block's are empty afterwards.
__device__ __forceinline__ void flushBins(uint32_t* sb, uint32_t* tb)
{
	for (int k = threadIdx.x; k < 3 * kBins; k += kThreads) {
		uint32_t* bb = sb + k * kBinWords;
		if (bb[6] == 0u) {
			continue;
		}
		uint32_t* g = tb + k * kBinWords;
#pragma unroll
		for (int w = 0; w < 6; ++w) {
			atomicMax(&g[w], bb[w]);
		}
		atomicAdd(&g[6], bb[6]);
		clearBins(bb, 0, 1, kBinWords);
	}
}

// All levels in one cooperative launch. A level has three phases with a grid barrier after each:
//  1. one warp per range: the split from the range's bins, its node, its children;
//  2. by chunks of kChunk elements: how many go left, and the children's bounds;
//  3. by chunks: the elements to their places, and into their child's bins.
// A block works through consecutive chunks and hands its bounds and bins on when the range changes.
// What bounds a level of a mesh of 100,000 triangles is not its data (4 MB, in L2) but the phases after
// each other: as six launches (chunk table, bounds, bins, split, count, scatter) a level took 27 us, and
// the host had to guess how many levels to queue; here it takes 17 (split 3.2, count 3, scatter 6,
// barriers 1 to 2 each) and less since, 167 us in all for 131,072 triangles against 245.
__global__ void __launch_bounds__(kThreads, 2) kSahLevels(const float4* __restrict__ lo, const float4* __restrict__ hi, SahLevels L)
{
	__shared__ uint32_t sBins[2][kTaskBinWords];
	__shared__ uint32_t sRed[2][kWarps][12];
	__shared__ int sW[kWarps];
	cooperative_groups::grid_group grid = cooperative_groups::this_grid();
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int thread = (int) (blockIdx.x * kThreads + threadIdx.x), threads = (int) (gridDim.x * kThreads);
	clearBins(sBins[0], (int) threadIdx.x, kThreads, 2 * kTaskBinWords);

	// The root: its order, bounds and bins.
	const int rootChunks = (L.n + kChunk - 1) / kChunk;
	if (blockIdx.x == 0) {
		if (threadIdx.x < kSahWords) {
			L.ctr[threadIdx.x] = threadIdx.x == kSahNodes || threadIdx.x == kSahLevel ? 1u : 0u;
		}
		if (threadIdx.x < 12) {
			L.bounds[0][threadIdx.x] = isMinWord((int) threadIdx.x) ? kEmptyLo : kEmptyHi;
		}
		if (threadIdx.x == 0) {
			L.tasks[0][0] = SahTask{0, L.n, 0, 0};
			L.chunkBase[0][0] = 0;
			L.chunkBase[0][1] = rootChunks;
		}
	}
	clearBins(L.bins, thread, threads, L.maxBig * kTaskBinWords);
	Bounds12 b[1];
	b[0].clear();
	for (int i = thread; i < L.n; i += threads) {
		if (i < rootChunks) {
			L.chunkTask[0][i] = 0;
		}
		L.ids[0][i] = (uint32_t) i;
		const float4 l = lo[i], h = hi[i];
		b[0].add(l, h, centroidOf(l, h));
	}
	grid.sync();
	blockAddBounds<1>(b, sRed, {L.bounds[0]});
	grid.sync();
	{
		AxisFrame fr[3];
#pragma unroll
		for (int a = 0; a < 3; ++a) {
			fr[a] = axisFrame(L.bounds[0], a);
		}
		for (int i = thread; i < L.n; i += threads) {
			const float4 l = lo[i], h = hi[i];
			addToBins(sBins[0], l, h, centroidOf(l, h), fr);
		}
		__syncthreads();
		flushBins(sBins[0], L.bins);
	}
	grid.sync();

	for (int level = 0;; ++level) {
		const int now = level & 1, then = now ^ 1;
		SahTask* const tasks = L.tasks[now];
		SahTask* const next = L.tasks[then];
		uint32_t* const bounds = L.bounds[now];
		uint32_t* const childBounds = L.bounds[then];
		const uint32_t* const ids = L.ids[now];
		const int32_t* const chunkBase = L.chunkBase[now];
		// Counts of three levels in turn: this one's, the next one's, and one that nobody reads now.
		uint32_t* const counts = L.ctr + kSahLevel;
		const int nTasks = (int) *(volatile uint32_t*) &counts[level % 3];
		if (nTasks == 0) {
			break;
		}
		if (thread == 0) {
			counts[(level + 2) % 3] = 0u;
		}
		for (int w = thread >> 5; w < nTasks; w += threads >> 5) {
			const SahTask tk = tasks[w];
			const uint32_t* b12 = bounds + (size_t) w * 12;
			uint32_t* tb = L.bins + (size_t) w * kTaskBinWords;
			LevelSplit s{warpBestSplit(tb, b12, lane), {-1, -1}};
			if (s.split.axis < 0) {
				s.split.nLeft = (tk.lo + tk.hi) / 2 - tk.lo;
			}
			__syncwarp();
			clearBins(tb, lane, 32); // for the next level's range of this number
			if (lane == 0) {
				const int cut[3] = {tk.lo, tk.lo + s.split.nLeft, tk.hi};
				uint32_t inner[2], big[2], block[2];
#pragma unroll
				for (int c = 0; c < 2; ++c) {
					const int cnt = cut[c + 1] - cut[c];
					inner[c] = cnt > 1 ? 1u : 0u;
					big[c] = cnt > kBigTask ? 1u : 0u;
					block[c] = inner[c] - big[c];
				}
				uint32_t node = atomicAdd(&L.ctr[kSahNodes], inner[0] + inner[1]);
				uint32_t slot = atomicAdd(&counts[(level + 1) % 3], big[0] + big[1]);
				uint32_t blockSlot = atomicAdd(&L.ctr[kSahBlocks], block[0] + block[1]);
				int32_t child[2];
#pragma unroll
				for (int c = 0; c < 2; ++c) {
					child[c] = inner[c] != 0u ? (int32_t) node : ~cut[c];
					const SahTask range{cut[c], cut[c + 1], child[c], 0};
					if (big[c] != 0u) {
						s.child[c] = (int32_t) slot;
						next[slot] = range;
						uint32_t* cb = childBounds + (size_t) slot * 12;
#pragma unroll
						for (int k = 0; k < 12; ++k) {
							cb[k] = isMinWord(k) ? kEmptyLo : kEmptyHi;
						}
					} else if (block[c] != 0u) {
						L.blockTasks[blockSlot] = range;
					}
					node += inner[c];
					slot += big[c];
					blockSlot += block[c];
				}
				L.splits[w] = s;
				NodeSink{L.bin, L.rangeFirst, L.rangeLast, L.ctr}.write(tk.node, tk.lo, tk.hi, b12, child[0], child[1]);
			}
			__syncwarp();
		}
		grid.sync();

		const int nNext = (int) *(volatile uint32_t*) &counts[(level + 1) % 3];
		const int nChunks = chunkBase[nTasks];
		const int run = (nChunks + (int) gridDim.x - 1) / (int) gridDim.x;
		const int c0 = min((int) blockIdx.x * run, nChunks), c1 = min(c0 + run, nChunks);
		const int t0 = c0 < c1 ? L.chunkTask[now][c0] : 0;
		{
			Bounds12 side[2];
			side[0].clear();
			side[1].clear();
			for (int c = c0, t = t0; c < c1; ++c) {
				const SahTask tk = tasks[t];
				const LevelSplit s = L.splits[t];
				const AxisFrame f = s.split.axis >= 0 ? axisFrame(bounds + (size_t) t * 12, s.split.axis) : AxisFrame{0.0f, 0.0f, false};
				const int start = tk.lo + (c - chunkBase[t]) * kChunk, end = min(tk.hi, start + kChunk);
				int cnt = 0;
#pragma unroll
				for (int q = 0; q < kItems; ++q) {
					const int i = start + q * kThreads + (int) threadIdx.x;
					if (i < end) {
						const uint32_t id = ids[i];
						const float4 l = lo[id], h = hi[id], cen = centroidOf(l, h);
						const bool left = s.split.axis < 0 ? i < tk.lo + s.split.nLeft
						                                   : binOf(comp3(cen, s.split.axis), f.cmin, f.scale) < s.split.bin;
						cnt += left ? 1 : 0;
						if (left) {
							side[0].add(l, h, cen);
						} else {
							side[1].add(l, h, cen);
						}
					}
				}
				cnt = __reduce_add_sync(0xffffffffu, cnt);
				if (lane == 0) {
					sW[warp] = cnt;
				}
				__syncthreads();
				if (threadIdx.x == 0) {
					int sum = 0;
					for (int w = 0; w < kWarps; ++w) {
						sum += sW[w];
					}
					L.chunkLeft[c] = sum;
				}
				__syncthreads();
				if (c + 1 == c1 || c + 1 == chunkBase[t + 1]) { // the range ends here
					uint32_t* const to[2] = {s.child[0] >= 0 ? childBounds + (size_t) s.child[0] * 12 : nullptr,
					                         s.child[1] >= 0 ? childBounds + (size_t) s.child[1] * 12 : nullptr};
					blockAddBounds<2>(side, sRed, to);
					side[0].clear();
					side[1].clear();
					++t;
				}
			}
		}
		if (blockIdx.x == gridDim.x - 1) { // the next level's chunk table
			int32_t* base = L.chunkBase[then];
			int carry = 0;
			for (int first = 0; first < nNext; first += kThreads) {
				const int t = first + (int) threadIdx.x;
				const int v = t < nNext ? (next[t].hi - next[t].lo + kChunk - 1) / kChunk : 0;
				int total;
				const int before = blockExclusiveScan(v, sW, total);
				if (t < nNext) {
					base[t] = carry + before;
					for (int k = 0; k < v; ++k) {
						L.chunkTask[then][carry + before + k] = t;
					}
				}
				carry += total;
			}
			if (threadIdx.x == 0) {
				base[nNext] = carry;
			}
		}
		grid.sync();

		AxisFrame fr[2][3];
		for (int c = c0, t = t0; c < c1; ++c) {
			const SahTask tk = tasks[t];
			const LevelSplit s = L.splits[t];
			const AxisFrame f = s.split.axis >= 0 ? axisFrame(bounds + (size_t) t * 12, s.split.axis) : AxisFrame{0.0f, 0.0f, false};
			if (c == c0 || c == chunkBase[t]) {
#pragma unroll
				for (int q = 0; q < 2; ++q) {
#pragma unroll
					for (int a = 0; a < 3; ++a) {
						fr[q][a] = s.child[q] >= 0 ? axisFrame(childBounds + (size_t) s.child[q] * 12, a) : AxisFrame{0.0f, 0.0f, false};
					}
				}
			}
			const int start = tk.lo + (c - chunkBase[t]) * kChunk, end = min(tk.hi, start + kChunk);
			// left elements of the range's earlier chunks
			int before = 0;
			for (int k = chunkBase[t] + (int) threadIdx.x; k < c; k += kThreads) {
				before += L.chunkLeft[k];
			}
			int leftBefore, total;
			(void) blockExclusiveScan(before, sW, leftBefore);
			// this thread's run of kItems consecutive elements
			const int p0 = start + (int) threadIdx.x * kItems;
			uint32_t id[kItems];
			float4 l[kItems], h[kItems];
			bool left[kItems];
			int mine = 0;
#pragma unroll
			for (int q = 0; q < kItems; ++q) {
				const int p = p0 + q;
				left[q] = false;
				if (p < end) {
					id[q] = ids[p];
					l[q] = lo[id[q]];
					h[q] = hi[id[q]];
					left[q] = s.split.axis < 0 ? p < tk.lo + s.split.nLeft
					                           : binOf(comp3(centroidOf(l[q], h[q]), s.split.axis), f.cmin, f.scale) < s.split.bin;
					mine += left[q] ? 1 : 0;
				}
			}
			int rank = leftBefore + blockExclusiveScan(mine, sW, total);
#pragma unroll
			for (int q = 0; q < kItems; ++q) {
				const int p = p0 + q;
				if (p < end) {
					// left: lo + (left elements before p); right: lo + nLeft + (right elements before p)
					const int dst = left[q] ? tk.lo + rank : tk.lo + s.split.nLeft + (p - tk.lo - rank);
					rank += left[q] ? 1 : 0;
					if (dst < tk.lo || dst >= tk.hi) {
						atomicExch(&L.ctr[kSahError], 1u);
						continue;
					}
					if (s.child[left[q] ? 0 : 1] >= 0) {
						L.ids[then][dst] = id[q];
						if (left[q]) {
							addToBins(sBins[0], l[q], h[q], centroidOf(l[q], h[q]), fr[0]);
						} else {
							addToBins(sBins[1], l[q], h[q], centroidOf(l[q], h[q]), fr[1]);
						}
					} else {
						L.sorted[dst] = id[q];
					}
				}
			}
			if (c + 1 == c1 || c + 1 == chunkBase[t + 1]) { // the range ends here
				__syncthreads();
#pragma unroll
				for (int q = 0; q < 2; ++q) {
					if (s.child[q] >= 0) {
						flushBins(sBins[q], L.bins + (size_t) s.child[q] * kTaskBinWords);
					}
				}
				__syncthreads();
				++t;
			}
		}
		if (nNext == 0) {
			break; // the same in every block
		}
		grid.sync();
	}
}

// ------------------------------------------------------------------ block phase (ranges 2..kBigTask)

// A block builds its range to the leaves in shared memory, its elements' boxes held there from the start:
//  * ranges above kMidTask elements: split by the whole block, one after another (a handful);
//  * ranges of 33..kMidTask: one warp each, all ranges of a depth side by side;
//  * ranges up to 32: one warp each, one element per lane, all subranges of a depth at once (smallBuild).
// What bounds a block is the chain of splits below each other, so what matters is that splits which do
// not depend on each other run together. With every range above 32 split by the whole block in turn and
// every subrange of a small one split alone, the ranges of 131,072 triangles took 885 us, 94 instances 58;
// side by side 255 (ranges of up to 2,048), with ranges of up to 1,024 and segmented scans in the smallest
// 141, with bins filled out of step 122; 94 instances 27.
constexpr int kMidTask = 256;

template<int CAPACITY, int THREADS>
struct BlockShared
{
	static constexpr int kBlockThreads = THREADS, kBlockWarps = THREADS / 32;
	static constexpr int kMaxMid = CAPACITY / (kSmallTask + 1) + 1, kMaxSmall = CAPACITY / 2, kMaxStack = CAPACITY / (kMidTask + 1) + 1;
	float box[6][CAPACITY];                        // by local element: lo xyz, hi xyz
	uint32_t gid[CAPACITY];                        // by local element: primitive
	uint16_t ids[CAPACITY], tmp[CAPACITY];         // local elements in sorted order
	uint32_t bins[kBlockWarps][kTaskBinWords];     // per warp; the first also for whole-block splits
	int4 stack[kMaxStack];                         // ranges above kMidTask, disjoint
	int4 mid[2][kMaxMid];                          // ranges of 33..kMidTask of this depth and the next
	int4 small[kMaxSmall];                         // ranges of 2..32
	uint32_t red[kBlockWarps][12];
	uint32_t bounds[12];
	int scan[kBlockWarps];
	uint8_t perm[kBlockWarps][3][32];
	int top, nMid[2], nSmall;
	uint32_t nextNode, taken;
	int4 cur;
	SahSplit split;

	__device__ __forceinline__ void add(Bounds12& b, int e) const
	{
		const float4 l = make_float4(box[0][e], box[1][e], box[2][e], 0.0f), h = make_float4(box[3][e], box[4][e], box[5][e], 0.0f);
		b.add(l, h, make_float4(centroid(e, 0), centroid(e, 1), centroid(e, 2), 0.0f));
	}
	// The host's centroid expression.
	__device__ __forceinline__ float centroid(int e, int a) const { return __fmul_rn(0.5f, __fadd_rn(box[a][e], box[3 + a][e])); }
	__device__ __forceinline__ void bin(uint32_t* to, int e, const AxisFrame (&fr)[3]) const
	{
		const float4 l = make_float4(box[0][e], box[1][e], box[2][e], 0.0f), h = make_float4(box[3][e], box[4][e], box[5][e], 0.0f);
		addToBins(to, l, h, make_float4(centroid(e, 0), centroid(e, 1), centroid(e, 2), 0.0f), fr);
	}
	__device__ __forceinline__ bool left(int e, int pos, int first, const SahSplit& s, const AxisFrame& f) const
	{
		return s.axis < 0 ? pos < first + s.nLeft : binOf(centroid(e, s.axis), f.cmin, f.scale) < s.bin;
	}
};

// One thread: the node of range [a, b) split after nLeft elements, and its children queued by size.
// Positions are the block's; `base` is the block's first sorted position.
template<class SHARED>
__device__ __forceinline__ void emitRange(SHARED& S, int a, int b, int node, int nLeft, const uint32_t* b12, int base, int midList,
                                          const NodeSink& out)
{
	const int cut[3] = {a, a + nLeft, b};
	int32_t child[2];
#pragma unroll
	for (int q = 0; q < 2; ++q) {
		child[q] = cut[q + 1] - cut[q] == 1 ? ~(base + cut[q]) : (int32_t) atomicAdd(&S.nextNode, 1u);
	}
	out.write(node, base + a, base + b, b12, child[0], child[1]);
#pragma unroll
	for (int q = 0; q < 2; ++q) {
		const int n = cut[q + 1] - cut[q];
		const int4 r = make_int4(cut[q], cut[q + 1], child[q], 0);
		if (n > kMidTask) {
			if (S.top < S.kMaxStack) { // whole-block splits only: no other thread pushes
				S.stack[S.top++] = r;
			} else {
				out.error();
			}
		} else if (n > kSmallTask) {
			const int k = atomicAdd(&S.nMid[midList], 1);
			if (k < S.kMaxMid) {
				S.mid[midList][k] = r;
			} else {
				out.error();
			}
		} else if (n >= 2) {
			const int k = atomicAdd(&S.nSmall, 1);
			if (k < S.kMaxSmall) {
				S.small[k] = r;
			} else {
				out.error();
			}
		}
	}
}

// A range of 33..kMidTask elements split by one warp.
template<class SHARED>
__device__ void warpSplit(SHARED& S, const int4 range, int base, int midList, const NodeSink& out)
{
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int a = range.x, b = range.y;
	uint32_t* bins = S.bins[warp];
	Bounds12 bd;
	bd.clear();
	for (int i = a + lane; i < b; i += 32) {
		S.add(bd, S.ids[i]);
	}
	bd.warpReduce();
	clearBins(bins, lane, 32);
	AxisFrame fr[3];
#pragma unroll
	for (int ax = 0; ax < 3; ++ax) {
		fr[ax] = axisFrame(bd.w, ax);
	}
	__syncwarp();
	for (int i = a + lane; i < b; i += 32) {
		S.bin(bins, S.ids[i], fr);
	}
	__syncwarp();
	SahSplit s = warpBestSplit(bins, bd.w, lane);
	if (s.axis < 0) {
		s.nLeft = (a + b) / 2 - a;
	}
	const AxisFrame f = s.axis >= 0 ? (s.axis == 0 ? fr[0] : (s.axis == 1 ? fr[1] : fr[2])) : AxisFrame{0.0f, 0.0f, false};
	// stable partition, 32 elements at a time
	int before = 0; // left elements of the earlier ones
	for (int i0 = a; i0 < b; i0 += 32) {
		const int i = i0 + lane;
		const uint16_t e = i < b ? S.ids[i] : (uint16_t) 0;
		const bool l = i < b && S.left(e, i, a, s, f);
		const uint32_t m = __ballot_sync(0xffffffffu, l);
		const int rank = before + __popc(m & ((1u << lane) - 1u));
		const int dst = l ? a + rank : a + s.nLeft + (i - a - rank);
		if (i < b) {
			if (dst >= a && dst < b) {
				S.tmp[dst] = e;
			} else {
				out.error();
			}
		}
		before += __popc(m);
	}
	__syncwarp();
	for (int i = a + lane; i < b; i += 32) {
		S.ids[i] = S.tmp[i];
	}
	if (lane == 0) {
		emitRange(S, a, b, range.z, s.nLeft, bd.w, base, midList, out);
	}
	__syncwarp();
}

// A range of 2..32 elements built to its leaves by one warp: lane j holds the element at position j, and
// all subranges of a depth are split together, per axis by a sort of the subrange's elements by bin and a
// segmented scan of their boxes from either end; the best of the candidates, in the host's order, is its
// split.
template<class SHARED>
__device__ void smallBuild(SHARED& S, const int4 range, int base, const NodeSink& out)
{
	constexpr uint32_t kAll = 0xffffffffu;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int a = range.x, cnt = range.y - range.x;
	const bool has = lane < cnt;
	int e = has ? S.ids[a + lane] : 0;
	uint32_t w[6]; // box, ordered bits
	float c[3];
#pragma unroll
	for (int k = 0; k < 6; ++k) {
		w[k] = has ? ordered(S.box[k][e]) : 0u;
	}
#pragma unroll
	for (int k = 0; k < 3; ++k) {
		c[k] = has ? S.centroid(e, k) : 0.0f;
	}
	int x = 0, y = has ? cnt : 0, node = range.z; // this lane's subrange and its node
	for (;;) {
		const int len = y - x;
		const bool active = has && len >= 2;
		const int longest = __reduce_max_sync(kAll, active ? len : 0);
		if (longest == 0) {
			break;
		}
		// Bounds of the subrange: combined towards its last lane, which then tells the others.
		uint32_t b12[12];
#pragma unroll
		for (int k = 0; k < 6; ++k) {
			b12[k] = w[k];
		}
#pragma unroll
		for (int k = 0; k < 3; ++k) {
			b12[6 + k] = b12[9 + k] = ordered(c[k]);
		}
		for (int off = 1; off < longest; off <<= 1) {
			const bool mine = lane - off >= x;
#pragma unroll
			for (int k = 0; k < 12; ++k) {
				const uint32_t v = __shfl_up_sync(kAll, b12[k], off);
				const uint32_t u = isMinWord(k) ? min(b12[k], v) : max(b12[k], v);
				b12[k] = mine ? u : b12[k];
			}
		}
		const int last = active ? y - 1 : lane;
#pragma unroll
		for (int k = 0; k < 12; ++k) {
			b12[k] = __shfl_sync(kAll, b12[k], last);
		}
		// The subrange's elements in order of their bins, one order per axis: a bin's place is the number of
		// smaller ones, counted bit by bit with ballots.
		const uint32_t below = (1u << lane) - 1u;
		const uint32_t segment = active ? ((y < 32 ? 1u << y : 0u) - 1u) & ~((1u << x) - 1u) : 1u << lane;
		uint32_t myBin[3];
		bool valid[3];
#pragma unroll
		for (int ax = 0; ax < 3; ++ax) {
			const AxisFrame f = axisFrame(b12, ax);
			valid[ax] = f.valid;
			myBin[ax] = f.valid ? (uint32_t) binOf(c[ax], f.cmin, f.scale) : 0u;
			uint32_t less = 0, equal = segment;
#pragma unroll
			for (int bit = 4; bit >= 0; --bit) {
				const bool one = ((myBin[ax] >> bit) & 1u) != 0u;
				const uint32_t ones = __ballot_sync(kAll, one);
				less |= one ? equal & ~ones : 0u;
				equal &= one ? ones : ~ones;
			}
			S.perm[warp][ax][(active ? x : lane) + __popc(less) + __popc(equal & below)] = (uint8_t) lane;
		}
		__syncwarp();
		// Boxes of everything up to a place and from it on; a split after a place is a candidate when the next
		// element is in another bin.
		uint32_t L[3][6], R[3][6], bin[3];
#pragma unroll
		for (int ax = 0; ax < 3; ++ax) {
			const int src = S.perm[warp][ax][lane];
			bin[ax] = __shfl_sync(kAll, myBin[ax], src);
#pragma unroll
			for (int q = 0; q < 6; ++q) {
				L[ax][q] = R[ax][q] = __shfl_sync(kAll, w[q], src);
			}
		}
		for (int off = 1; off < longest; off <<= 1) {
			const bool up = lane - off >= x, down = lane + off < y;
#pragma unroll
			for (int ax = 0; ax < 3; ++ax) {
#pragma unroll
				for (int q = 0; q < 6; ++q) {
					const uint32_t l = __shfl_up_sync(kAll, L[ax][q], off), r = __shfl_down_sync(kAll, R[ax][q], off);
					if (up) {
						L[ax][q] = q < 3 ? min(L[ax][q], l) : max(L[ax][q], l);
					}
					if (down) {
						R[ax][q] = q < 3 ? min(R[ax][q], r) : max(R[ax][q], r);
					}
				}
			}
		}
		// The lane's best candidate as (cost, axis and bin, left count); among equal costs the first (axis, bin)
		// is the smaller word.
		float bestCost = kInf;
		uint32_t bestKey = 0xffffffffu;
		const int lc = lane + 1 - x, rc = y - lane - 1;
#pragma unroll
		for (int ax = 0; ax < 3; ++ax) {
			uint32_t r[6];
#pragma unroll
			for (int q = 0; q < 6; ++q) {
				r[q] = __shfl_down_sync(kAll, R[ax][q], 1);
			}
			const uint32_t nextBin = __shfl_down_sync(kAll, bin[ax], 1);
			if (active && valid[ax] && rc > 0 && nextBin != bin[ax]) {
				const float ha = halfAreaOf(unordered(L[ax][0]), unordered(L[ax][1]), unordered(L[ax][2]), unordered(L[ax][3]), unordered(L[ax][4]),
				                            unordered(L[ax][5]));
				const float hb = halfAreaOf(unordered(r[0]), unordered(r[1]), unordered(r[2]), unordered(r[3]), unordered(r[4]), unordered(r[5]));
				const float cost = __fadd_rn(__fmul_rn(ha, (float) lc), __fmul_rn(hb, (float) rc));
				if (cost < bestCost) {
					bestCost = cost;
					bestKey = ((uint32_t) (ax * kBins) + bin[ax] + 1u) << 8 | (uint32_t) lc;
				}
			}
		}
		__syncwarp();
		// The best of the subrange, as its bounds.
		for (int off = 1; off < longest; off <<= 1) {
			const float oc = __shfl_up_sync(kAll, bestCost, off);
			const uint32_t ok = __shfl_up_sync(kAll, bestKey, off);
			if (lane - off >= x && (oc < bestCost || (oc == bestCost && ok < bestKey))) {
				bestCost = oc;
				bestKey = ok;
			}
		}
		bestKey = __shfl_sync(kAll, bestKey, last);
		const bool middle = bestKey == 0xffffffffu;
		const int nLeft = middle ? len / 2 : (int) (bestKey & 0xffu);
		const uint32_t key = bestKey >> 8;
		const uint32_t axis = key / kBins, cut = key % kBins; // a cut after bin 31 has no right side
		const uint32_t mine = axis == 0u ? myBin[0] : (axis == 1u ? myBin[1] : myBin[2]);
		const bool goLeft = active && (middle ? lane < x + nLeft : mine < cut);
		// stable partition within the subrange
		const uint32_t fromX = ~((1u << x) - 1u);
		const int leftRank = __popc(__ballot_sync(kAll, goLeft) & below & fromX);
		int dst = !active ? lane : (goLeft ? x + leftRank : x + nLeft + (lane - x - leftRank));
		if (dst < 0 || dst >= 32) {
			out.error();
			dst = lane;
		}
		S.perm[warp][0][dst] = (uint8_t) lane;
		// Nodes: each subrange's first lane writes it and takes numbers for its inner children.
		const bool leads = active && lane == x;
		int32_t child[2] = {~(base + a + x), ~(base + a + x + nLeft)};
		const uint32_t wantL = __ballot_sync(kAll, leads && nLeft > 1), wantR = __ballot_sync(kAll, leads && len - nLeft > 1);
		uint32_t first = 0;
		if (lane == 0 && (wantL | wantR) != 0u) {
			first = atomicAdd(&S.nextNode, (uint32_t) (__popc(wantL) + __popc(wantR)));
		}
		first = __shfl_sync(kAll, first, 0);
		if (leads) {
			if (nLeft > 1) {
				child[0] = (int32_t) (first + (uint32_t) __popc(wantL & below));
			}
			if (len - nLeft > 1) {
				child[1] = (int32_t) (first + (uint32_t) __popc(wantL) + (uint32_t) __popc(wantR & below));
			}
			out.write(node, base + a + x, base + a + y, b12, child[0], child[1]);
		}
		__syncwarp();
		const int32_t cl = __shfl_sync(kAll, child[0], x), cr = __shfl_sync(kAll, child[1], x);
		const int src = S.perm[warp][0][lane];
		__syncwarp();
		e = __shfl_sync(kAll, e, src);
#pragma unroll
		for (int q = 0; q < 6; ++q) {
			w[q] = __shfl_sync(kAll, w[q], src);
		}
#pragma unroll
		for (int q = 0; q < 3; ++q) {
			c[q] = __shfl_sync(kAll, c[q], src);
		}
		if (active) {
			const int mid = x + nLeft;
			node = lane < mid ? cl : cr;
			(lane < mid ? y : x) = mid;
		}
	}
	if (has) {
		S.ids[a + lane] = (uint16_t) e;
	}
	__syncwarp();
}

// One range of at most the capacity, by the whole block; see kSahBlock.
template<class SHARED>
__device__ __forceinline__ void buildRange(SHARED& S, const SahTask task, const SahTask* tasks, const InstanceRec* inst, float4* gLo,
                                           float4* gHi, uint32_t* sorted, const NodeSink& out)
{
	const int base = task.lo, cnt = task.hi - task.lo;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
		const uint32_t id = tasks != nullptr ? sorted[base + i] : (uint32_t) i;
		float4 l, h;
		if (inst != nullptr) {
			const InstanceRec& r = inst[id];
			l = make_float4(r.lox, r.loy, r.loz, 0.0f);
			h = make_float4(r.hix, r.hiy, r.hiz, 0.0f);
			gLo[id] = l;
			gHi[id] = h;
		} else {
			l = gLo[id];
			h = gHi[id];
		}
		S.gid[i] = id;
		S.ids[i] = (uint16_t) i;
		S.box[0][i] = l.x;
		S.box[1][i] = l.y;
		S.box[2][i] = l.z;
		S.box[3][i] = h.x;
		S.box[4][i] = h.y;
		S.box[5][i] = h.z;
	}
	if (threadIdx.x == 0) {
		S.top = S.nMid[0] = S.nMid[1] = S.nSmall = 0;
		// A range of cnt primitives has cnt - 1 nodes: its own, and the rest numbered from here.
		S.nextNode = out.ctr != nullptr ? atomicAdd(&out.ctr[kSahNodes], (uint32_t) (cnt - 2)) : 1u;
		const int4 r = make_int4(0, cnt, task.node, 0);
		if (cnt > kMidTask) {
			S.stack[S.top++] = r;
		} else if (cnt > kSmallTask) {
			S.mid[0][S.nMid[0]++] = r;
		} else if (cnt >= 2) {
			S.small[S.nSmall++] = r;
		}
	}
	__syncthreads();
	for (;;) {
		// Every thread reads the stack's top between two barriers, so none sees the pop or the pushes of
		// this turn.
		const int top = S.top;
		const int4 cur = S.stack[top > 0 ? top - 1 : 0];
		__syncthreads();
		if (top == 0) {
			break;
		}
		const int a = cur.x, b = cur.y, node = cur.z;
		if (threadIdx.x == 0) {
			S.top = top - 1;
		}
		// bounds
		Bounds12 bd;
		bd.clear();
		for (int i = a + (int) threadIdx.x; i < b; i += blockDim.x) {
			S.add(bd, S.ids[i]);
		}
		bd.warpReduce();
		if (lane == 0) {
#pragma unroll
			for (int k = 0; k < 12; ++k) {
				S.red[warp][k] = bd.w[k];
			}
		}
		clearBins(S.bins[0], (int) threadIdx.x, S.kBlockThreads);
		__syncthreads();
		if (threadIdx.x < 12) {
			const int k = threadIdx.x;
			uint32_t v = S.red[0][k];
			for (int w = 1; w < S.kBlockWarps; ++w) {
				v = isMinWord(k) ? min(v, S.red[w][k]) : max(v, S.red[w][k]);
			}
			S.bounds[k] = v;
		}
		__syncthreads();
		// bins
		AxisFrame fr[3];
#pragma unroll
		for (int ax = 0; ax < 3; ++ax) {
			fr[ax] = axisFrame(S.bounds, ax);
		}
		for (int i = a + (int) threadIdx.x; i < b; i += blockDim.x) {
			S.bin(S.bins[0], S.ids[i], fr);
		}
		__syncthreads();
		if (warp == 0) {
			SahSplit s = warpBestSplit(S.bins[0], S.bounds, lane);
			if (s.axis < 0) {
				s.nLeft = (a + b) / 2 - a;
			}
			if (lane == 0) {
				S.split = s;
			}
		}
		__syncthreads();
		const SahSplit s = S.split;
		// stable partition of [a, b): runs of consecutive elements per thread
		const int per = (b - a + S.kBlockThreads - 1) / S.kBlockThreads;
		const int p0 = a + (int) threadIdx.x * per;
		const int p1 = min(b, p0 + per);
		const AxisFrame f = s.axis >= 0 ? (s.axis == 0 ? fr[0] : (s.axis == 1 ? fr[1] : fr[2])) : AxisFrame{0.0f, 0.0f, false};
		int mine = 0;
		for (int p = p0; p < p1; ++p) {
			mine += S.left(S.ids[p], p, a, s, f) ? 1 : 0;
		}
		int total;
		int rank = blockExclusiveScan<SHARED::kBlockWarps>(mine, S.scan, total);
		for (int p = p0; p < p1; ++p) {
			const uint16_t e = S.ids[p];
			const bool gl = S.left(e, p, a, s, f);
			const int dst = gl ? a + rank : a + s.nLeft + (p - a - rank);
			rank += gl ? 1 : 0;
			if (dst < a || dst >= b) {
				out.error();
				continue;
			}
			S.tmp[dst] = e;
		}
		__syncthreads();
		for (int i = a + (int) threadIdx.x; i < b; i += blockDim.x) {
			S.ids[i] = S.tmp[i];
		}
		if (threadIdx.x == 0) {
			emitRange(S, a, b, node, s.nLeft, S.bounds, base, 0, out);
		}
		__syncthreads();
	}
	// ranges of 33..kMidTask, depth by depth
	for (int list = 0;; list ^= 1) {
		const int m = min(S.nMid[list], S.kMaxMid);
		if (m == 0) {
			break;
		}
		for (int k = warp; k < m; k += S.kBlockWarps) {
			warpSplit(S, S.mid[list][k], base, list ^ 1, out);
		}
		__syncthreads();
		if (threadIdx.x == 0) {
			S.nMid[list] = 0; // this list takes the depth after next
		}
		__syncthreads();
	}
	// ranges of up to 32 elements
	for (int k = warp; k < min(S.nSmall, S.kMaxSmall); k += S.kBlockWarps) {
		smallBuild(S, S.small[k], base, out);
	}
	__syncthreads();
	for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
		sorted[base + i] = S.gid[S.ids[i]];
	}
}

// tasks: ranges that the blocks take in turn, or null for a one-block build of primitives [0, n) in the given order. Boxes
// come from gLo / gHi, or, for a TLAS, from the instance records, and are then stored there for the collapse.
template<class SHARED>
__global__ void __launch_bounds__(SHARED::kBlockThreads) kSahBlock(const SahTask* __restrict__ tasks, int n, const InstanceRec* __restrict__ inst,
                                                           float4* gLo, float4* gHi, uint32_t* __restrict__ sorted, NodeSink out)
{
	extern __shared__ __align__(16) uint8_t smem[];
	SHARED& S = *reinterpret_cast<SHARED*>(smem);
	if (tasks == nullptr) {
		buildRange(S, SahTask{0, n, 0, 0}, nullptr, inst, gLo, gHi, sorted, out);
		return;
	}
	const uint32_t count = out.ctr[kSahBlocks];
	for (;;) {
		if (threadIdx.x == 0) {
			S.taken = atomicAdd(&out.ctr[kSahTaken], 1u);
		}
		__syncthreads();
		const uint32_t k = S.taken;
		if (k >= count) {
			return;
		}
		buildRange(S, tasks[k], tasks, inst, gLo, gHi, sorted, out);
		__syncthreads();
	}
}

// Ranges of a mesh, one block per SM (88 KB of shared memory would let two in, 115 registers for each of 512
// threads do not); and the one block of a TLAS.
using MeshShared = BlockShared<kBigTask, kMeshThreads>;
using TlasShared = BlockShared<kSahSmallMax, 512>;

// Blocks of a kernel that fit the device at once.
template<class Kernel>
int residentBlocks(Kernel kernel, int threads, size_t shared)
{
	int dev = 0, sms = 0, perSm = 0;
	RGL_SAH_OK(cudaGetDevice(&dev));
	RGL_SAH_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
	RGL_SAH_OK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kernel, threads, shared));
	return sms * perSm;
}

inline int blocksFor(int n, int b) { return (n + b - 1) / b; }

} // namespace

void prepareSahBlock()
{
	static const bool done = [] {
		RGL_SAH_OK(cudaFuncSetAttribute(kSahBlock<TlasShared>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) sizeof(TlasShared)));
		return true;
	}();
	(void) done;
}

const uint32_t* enqueueSahTopology(BuildScratch& scratch, const float4* lo, const float4* hi, int n, BinNode* bin, int32_t* rangeFirst,
                                   int32_t* rangeLast, uint32_t* sortedIds, cudaStream_t stream)
{
	if (n < 2) {
		RGL_SAH_OK(cudaMemsetAsync(sortedIds, 0, sizeof(uint32_t), stream));
		return nullptr;
	}
	SahLevels L{};
	L.n = n;
	L.maxBig = n / (kBigTask + 1) + 1; // disjoint ranges above kBigTask
	const int maxChunks = n / kChunk + L.maxBig + 1;
	scratch.carve([&](BuildScratch::Carver& place) {
		place(L.ctr, kSahWords);
		place(L.blockTasks, n / 2 + 1); // disjoint ranges of at least 2
		if (n <= kBigTask) {
			return;
		}
		for (int k = 0; k < 2; ++k) {
			place(L.ids[k], n);
			place(L.tasks[k], L.maxBig);
			place(L.bounds[k], (size_t) L.maxBig * 12);
			place(L.chunkBase[k], L.maxBig + 1);
			place(L.chunkTask[k], maxChunks);
		}
		place(L.bins, (size_t) L.maxBig * kTaskBinWords);
		place(L.chunkLeft, maxChunks);
		place(L.splits, L.maxBig);
	});
	L.sorted = sortedIds;
	L.bin = bin;
	L.rangeFirst = rangeFirst;
	L.rangeLast = rangeLast;
	if (n <= kBigTask) {
		kSahInit<<<blocksFor(n, 256), 256, 0, stream>>>(n, sortedIds, L.blockTasks, L.ctr);
	} else {
		static const int most = residentBlocks(kSahLevels, kThreads, 0); // the grid barrier needs all of them
		void* args[] = {&lo, &hi, &L};
		RGL_SAH_OK(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(&kSahLevels), dim3(std::min(most, maxChunks)),
		                                       dim3(kThreads), args, 0, stream));
	}
	countLaunch();
	// Blocks take ranges until none is left: their number is known on the device only.
	static const int meshBlocks = [] {
		RGL_SAH_OK(cudaFuncSetAttribute(kSahBlock<MeshShared>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) sizeof(MeshShared)));
		return residentBlocks(kSahBlock<MeshShared>, kMeshThreads, sizeof(MeshShared));
	}();
	kSahBlock<MeshShared><<<std::min(blocksFor(n, 32), meshBlocks), kMeshThreads, sizeof(MeshShared), stream>>>(
	    L.blockTasks, n, nullptr, const_cast<float4*>(lo), const_cast<float4*>(hi), sortedIds, NodeSink{bin, rangeFirst, rangeLast, L.ctr});
	countLaunch();
	return L.ctr;
}

void enqueueSahTopologySmall(const InstanceRec* inst, float4* lo, float4* hi, int n, BinNode* bin, int32_t* rangeFirst, int32_t* rangeLast,
                             uint32_t* sortedIds, cudaStream_t s)
{
	if (n <= 0 || n > kSahSmallMax) {
		throw std::runtime_error("SAH build: one-block topology takes 1.." + std::to_string(kSahSmallMax) + " primitives");
	}
	kSahBlock<TlasShared><<<1, TlasShared::kBlockThreads, sizeof(TlasShared), s>>>(nullptr, n, inst, lo, hi, sortedIds, NodeSink{bin, rangeFirst, rangeLast, nullptr});
	countLaunch();
}

} // namespace rgl
