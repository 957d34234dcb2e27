// On-device binned SAH topology for mesh BLASes: the binary tree of the host builder
// (sah_build.hpp buildBinnedSahTree), computed on the GPU with the same float arithmetic, so the
// device tree equals the host tree node for node and the sorted primitive order equals the host's.
//
// Replaces OptiX's GAS build of reference src/scene/GASBuilder.hpp:31-100 (optixAccelBuild), which
// runs on the device; the wide collapse and quantisation that follow are bvh_core.hpp's.
//
// Algorithm (after Wald 2007, binned SAH, 32 bins per axis; parallel top-down):
//  * ranges of more than kBigTask primitives are split level by level, each by many blocks: a bounds
//    pass (node box and centroid bounds), a binning pass (per-bin boxes and counts, shared-memory
//    atomics flushed to the range's global bins), one warp per range evaluating the 3 x 31 split
//    candidates, and a stable partition (per-chunk counts, then a scatter that ranks each chunk's
//    elements with a block scan);
//  * ranges of 2..kBigTask primitives are built to the leaves by one block each, in shared memory:
//    ranges above kSmallTask split with block-wide passes, smaller ones by one warp each, which keeps
//    its elements in registers and partitions them with ballots.
// Exactness: boxes and centroid bounds are min/max (order free); the centroid, the bin index, the
// half areas and the split costs use the host's expressions with round-to-nearest intrinsics and no
// FMA contraction; among equal costs the first candidate in (axis, bin) order wins, as in the host's
// strict comparison; partitions are stable; a range whose centroids all coincide splits in the
// middle. Node numbering differs from the host's (atomics instead of a depth-first counter); the
// collapse does not depend on it.
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
constexpr int kBinWords = 7;                    // lo xyz, hi xyz (ordered bits), count
constexpr int kTaskBinWords = 3 * kBins * kBinWords;
constexpr int kBigTask = 2048;                  // larger ranges split in the level loop
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

// Best split of a range from its bins (3 x 32 x 7 words, any address space) and bounds, by one warp:
// the candidate between bins b-1 and b of axis a costs halfArea(left) * nLeft + halfArea(right) * nRight;
// candidates with an empty side are skipped; the lowest cost wins, the first in (axis, b) order among
// equal costs. Returns axis -1 when no axis has spread centroids.
__device__ SahSplit warpBestSplit(const uint32_t* bins, const uint32_t* b12, int lane)
{
	float bestCost = kInf;
	int bestKey = 1 << 30, bestLeft = 0;
	for (int a = 0; a < 3; ++a) {
		const AxisFrame f = axisFrame(b12, a);
		if (!f.valid) {
			continue;
		}
		const uint32_t* bb = bins + (a * kBins + lane) * kBinWords;
		uint32_t v[kBinWords];
#pragma unroll
		for (int k = 0; k < kBinWords; ++k) {
			v[k] = bb[k];
		}
		// inclusive prefix (bins 0..lane) and suffix (bins lane..31)
		uint32_t p[kBinWords], q[kBinWords];
#pragma unroll
		for (int k = 0; k < kBinWords; ++k) {
			p[k] = v[k];
			q[k] = v[k];
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

// Writes binary node `node` over sorted positions [lo, hi) split at lo + nLeft, allocates its
// children's node indices and returns them (a leaf child is ~position).
__device__ __forceinline__ void emitNode(int node, int lo, int hi, int nLeft, const uint32_t* b12, BinNode* bin, int32_t* rangeFirst,
                                         int32_t* rangeLast, uint32_t* ctr, int32_t& left, int32_t& right)
{
	const int mid = lo + nLeft;
	left = (mid - lo == 1) ? ~lo : (int32_t) atomicAdd(&ctr[kSahNodes], 1u);
	right = (hi - mid == 1) ? ~mid : (int32_t) atomicAdd(&ctr[kSahNodes], 1u);
	BinNode bn;
	bn.lox = unordered(b12[0]);
	bn.loy = unordered(b12[1]);
	bn.loz = unordered(b12[2]);
	bn.hix = unordered(b12[3]);
	bn.hiy = unordered(b12[4]);
	bn.hiz = unordered(b12[5]);
	bn.left = left;
	bn.right = right;
	bin[node] = bn;
	rangeFirst[node] = lo;
	rangeLast[node] = hi - 1;
}

// ------------------------------------------------------------------ level loop (ranges > kBigTask)

__global__ void kSahInit(const float4* __restrict__ lo, const float4* __restrict__ hi, int n, float4* __restrict__ cen,
                         uint32_t* __restrict__ idsA, uint32_t* __restrict__ sorted, SahTask* levelTasks, SahTask* blockTasks, uint32_t* ctr)
{
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i < kSahWords) {
		const bool big = n > kBigTask;
		ctr[i] = i == kSahNodes ? 1u : (i == (big ? kSahNext : kSahBlocks) ? 1u : 0u);
		if (i == 0) {
			*(big ? levelTasks : blockTasks) = SahTask{0, n, 0, 0}; // the root
		}
	}
	if (i < n) {
		const float4 l = lo[i], h = hi[i];
		cen[i] = make_float4(__fmul_rn(0.5f, __fadd_rn(l.x, h.x)), __fmul_rn(0.5f, __fadd_rn(l.y, h.y)), __fmul_rn(0.5f, __fadd_rn(l.z, h.z)),
		                     0.0f);
		idsA[i] = (uint32_t) i;
		sorted[i] = (uint32_t) i;
	}
}

// The level's task count (what the level before counted), the chunk prefix sums of its ranges and their
// bounds cleared (one block). The kernels of a level read the count from the control words, so levels
// follow each other without the host.
__global__ void kSahLevelPrep(const SahTask* __restrict__ tasks, int32_t* chunkBase, uint32_t* bounds, uint32_t* ctr)
{
	__shared__ int32_t sWarp[32];
	__shared__ int32_t sCarry;
	const int nTasks = (int) ctr[kSahNext];
	__syncthreads();
	if (threadIdx.x == 0) {
		sCarry = 0;
		ctr[kSahCur] = (uint32_t) nTasks;
		ctr[kSahNext] = 0u;
	}
	for (int i = threadIdx.x; i < nTasks * 12; i += blockDim.x) {
		bounds[i] = isMinWord(i % 12) ? kEmptyLo : kEmptyHi;
	}
	__syncthreads();
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	for (int base = 0; base < nTasks; base += blockDim.x) {
		const int t = base + (int) threadIdx.x;
		const int v = t < nTasks ? (tasks[t].hi - tasks[t].lo + kChunk - 1) / kChunk : 0;
		int incl = v;
		for (int off = 1; off < 32; off <<= 1) {
			const int u = __shfl_up_sync(0xffffffffu, incl, off);
			if (lane >= off) {
				incl += u;
			}
		}
		if (lane == 31) {
			sWarp[warp] = incl;
		}
		__syncthreads();
		if (warp == 0) {
			const int nw = blockDim.x / 32;
			int w = lane < nw ? sWarp[lane] : 0;
			for (int off = 1; off < 32; off <<= 1) {
				const int u = __shfl_up_sync(0xffffffffu, w, off);
				if (lane >= off) {
					w += u;
				}
			}
			if (lane < nw) {
				sWarp[lane] = w; // inclusive over warps
			}
		}
		__syncthreads();
		const int warpBase = warp > 0 ? sWarp[warp - 1] : 0;
		if (t < nTasks) {
			chunkBase[t] = sCarry + warpBase + incl - v;
		}
		__syncthreads();
		if (threadIdx.x == 0) {
			sCarry += sWarp[blockDim.x / 32 - 1];
		}
		__syncthreads();
	}
	if (threadIdx.x == 0) {
		chunkBase[nTasks] = sCarry;
	}
}

// Range of chunk c: the task whose chunk prefix covers it.
__device__ __forceinline__ bool chunkRange(const int32_t* chunkBase, const uint32_t* ctr, const SahTask* tasks, int c, int& t, int& start,
                                           int& end, int& first)
{
	const int nTasks = (int) ctr[kSahCur];
	if (nTasks == 0 || c >= chunkBase[nTasks]) {
		return false;
	}
	int lo = 0, hi = nTasks; // chunkBase[lo] <= c < chunkBase[hi]
	while (hi - lo > 1) {
		const int mid = (lo + hi) >> 1;
		if (chunkBase[mid] <= c) {
			lo = mid;
		} else {
			hi = mid;
		}
	}
	t = lo;
	first = chunkBase[lo];
	start = tasks[lo].lo + (c - first) * kChunk;
	end = min(tasks[lo].hi, start + kChunk);
	return true;
}

__device__ __forceinline__ void blockReduceBounds(Bounds12& b, uint32_t (*sRed)[12], uint32_t* out)
{
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	b.warpReduce();
	if (lane == 0) {
#pragma unroll
		for (int k = 0; k < 12; ++k) {
			sRed[warp][k] = b.w[k];
		}
	}
	__syncthreads();
	if (threadIdx.x < 12) {
		const int k = threadIdx.x;
		uint32_t v = sRed[0][k];
		for (int w = 1; w < kWarps; ++w) {
			v = isMinWord(k) ? min(v, sRed[w][k]) : max(v, sRed[w][k]);
		}
		if (isMinWord(k)) {
			atomicMin(&out[k], v);
		} else {
			atomicMax(&out[k], v);
		}
	}
}

__global__ void __launch_bounds__(kThreads) kSahBounds(const SahTask* __restrict__ tasks, const uint32_t* ctr, const int32_t* __restrict__ chunkBase,
                                                       const uint32_t* __restrict__ ids, const float4* __restrict__ lo,
                                                       const float4* __restrict__ hi, const float4* __restrict__ cen, uint32_t* bounds,
                                                       uint32_t* bins)
{
	__shared__ uint32_t sRed[kWarps][12];
	int t, start, end, first;
	if (!chunkRange(chunkBase, ctr, tasks, blockIdx.x, t, start, end, first)) {
		return;
	}
	if ((int) blockIdx.x == first) { // the range's first chunk clears its bins for the binning pass
		uint32_t* tb = bins + (size_t) t * kTaskBinWords;
		for (int k = threadIdx.x; k < kTaskBinWords; k += blockDim.x) {
			const int w = k % kBinWords;
			tb[k] = w < 3 ? kEmptyLo : (w < 6 ? kEmptyHi : 0u);
		}
	}
	Bounds12 b;
	b.clear();
	for (int i = start + (int) threadIdx.x; i < end; i += blockDim.x) {
		const uint32_t id = ids[i];
		b.add(lo[id], hi[id], cen[id]);
	}
	blockReduceBounds(b, sRed, bounds + (size_t) t * 12);
}

__global__ void __launch_bounds__(kThreads) kSahBins(const SahTask* __restrict__ tasks, const uint32_t* ctr, const int32_t* __restrict__ chunkBase,
                                                     const uint32_t* __restrict__ ids, const float4* __restrict__ lo,
                                                     const float4* __restrict__ hi, const float4* __restrict__ cen,
                                                     const uint32_t* __restrict__ bounds, uint32_t* bins)
{
	__shared__ uint32_t sb[kTaskBinWords];
	int t, start, end, first;
	if (!chunkRange(chunkBase, ctr, tasks, blockIdx.x, t, start, end, first)) {
		return;
	}
	for (int k = threadIdx.x; k < kTaskBinWords; k += blockDim.x) {
		const int w = k % kBinWords;
		sb[k] = w < 3 ? kEmptyLo : (w < 6 ? kEmptyHi : 0u);
	}
	const uint32_t* b12 = bounds + (size_t) t * 12;
	AxisFrame fr[3];
#pragma unroll
	for (int a = 0; a < 3; ++a) {
		fr[a] = axisFrame(b12, a);
	}
	__syncthreads();
	for (int i = start + (int) threadIdx.x; i < end; i += blockDim.x) {
		const uint32_t id = ids[i];
		const float4 l = lo[id], h = hi[id], c = cen[id];
#pragma unroll
		for (int a = 0; a < 3; ++a) {
			if (!fr[a].valid) {
				continue;
			}
			uint32_t* bb = sb + (a * kBins + binOf(comp3(c, a), fr[a].cmin, fr[a].scale)) * kBinWords;
			atomicMin(&bb[0], ordered(l.x));
			atomicMin(&bb[1], ordered(l.y));
			atomicMin(&bb[2], ordered(l.z));
			atomicMax(&bb[3], ordered(h.x));
			atomicMax(&bb[4], ordered(h.y));
			atomicMax(&bb[5], ordered(h.z));
			atomicAdd(&bb[6], 1u);
		}
	}
	__syncthreads();
	uint32_t* tb = bins + (size_t) t * kTaskBinWords;
	for (int k = threadIdx.x; k < 3 * kBins; k += blockDim.x) {
		const uint32_t* bb = sb + k * kBinWords;
		if (bb[6] == 0u) {
			continue;
		}
		uint32_t* g = tb + k * kBinWords;
		atomicMin(&g[0], bb[0]);
		atomicMin(&g[1], bb[1]);
		atomicMin(&g[2], bb[2]);
		atomicMax(&g[3], bb[3]);
		atomicMax(&g[4], bb[4]);
		atomicMax(&g[5], bb[5]);
		atomicAdd(&g[6], bb[6]);
	}
}

// One warp per range: the split, the node, its children (next level, block phase or leaves).
__global__ void kSahSplit(const SahTask* __restrict__ tasks, const uint32_t* __restrict__ bounds,
                          const uint32_t* __restrict__ bins, SahSplit* splits, BinNode* bin, int32_t* rangeFirst, int32_t* rangeLast,
                          SahTask* next, SahTask* blockTasks, uint32_t* ctr)
{
	const int w = (int) ((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
	const int lane = threadIdx.x & 31;
	if (w >= (int) ctr[kSahCur]) {
		return;
	}
	const SahTask tk = tasks[w];
	const uint32_t* b12 = bounds + (size_t) w * 12;
	SahSplit s = warpBestSplit(bins + (size_t) w * kTaskBinWords, b12, lane);
	if (s.axis < 0) {
		s.nLeft = (tk.lo + tk.hi) / 2 - tk.lo;
	}
	if (lane == 0) {
		splits[w] = s;
		int32_t left, right;
		emitNode(tk.node, tk.lo, tk.hi, s.nLeft, b12, bin, rangeFirst, rangeLast, ctr, left, right);
		const int mid = tk.lo + s.nLeft;
		const int cl[2] = {left, right};
		const int r0[2] = {tk.lo, mid}, r1[2] = {mid, tk.hi};
		for (int c = 0; c < 2; ++c) {
			const int cnt = r1[c] - r0[c];
			if (cnt < 2) {
				continue;
			}
			const SahTask child{r0[c], r1[c], cl[c], 0};
			if (cnt > kBigTask) {
				next[atomicAdd(&ctr[kSahNext], 1u)] = child;
			} else {
				blockTasks[atomicAdd(&ctr[kSahBlocks], 1u)] = child;
			}
		}
	}
}

__device__ __forceinline__ bool goesLeft(uint32_t id, int pos, const SahTask& tk, const SahSplit& s, const AxisFrame& f,
                                         const float4* __restrict__ cen)
{
	if (s.axis < 0) {
		return pos < tk.lo + s.nLeft;
	}
	return binOf(comp3(cen[id], s.axis), f.cmin, f.scale) < s.bin;
}

__global__ void __launch_bounds__(kThreads) kSahPartCount(const SahTask* __restrict__ tasks, const uint32_t* ctr,
                                                          const int32_t* __restrict__ chunkBase, const uint32_t* __restrict__ ids,
                                                          const float4* __restrict__ cen, const uint32_t* __restrict__ bounds,
                                                          const SahSplit* __restrict__ splits, int32_t* chunkLeft)
{
	__shared__ int sW[kWarps];
	int t, start, end, first;
	if (!chunkRange(chunkBase, ctr, tasks, blockIdx.x, t, start, end, first)) {
		return;
	}
	const SahTask tk = tasks[t];
	const SahSplit s = splits[t];
	const AxisFrame f = s.axis >= 0 ? axisFrame(bounds + (size_t) t * 12, s.axis) : AxisFrame{0.0f, 0.0f, false};
	int cnt = 0;
	for (int i = start + (int) threadIdx.x; i < end; i += blockDim.x) {
		cnt += goesLeft(ids[i], i, tk, s, f, cen) ? 1 : 0;
	}
	cnt = __reduce_add_sync(0xffffffffu, cnt);
	if ((threadIdx.x & 31) == 0) {
		sW[threadIdx.x >> 5] = cnt;
	}
	__syncthreads();
	if (threadIdx.x == 0) {
		int sum = 0;
		for (int w = 0; w < kWarps; ++w) {
			sum += sW[w];
		}
		chunkLeft[blockIdx.x] = sum;
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

__global__ void __launch_bounds__(kThreads) kSahPartScatter(const SahTask* __restrict__ tasks, uint32_t* ctr,
                                                            const int32_t* __restrict__ chunkBase, const uint32_t* __restrict__ ids,
                                                            const float4* __restrict__ cen, const uint32_t* __restrict__ bounds,
                                                            const SahSplit* __restrict__ splits, const int32_t* __restrict__ chunkLeft,
                                                            uint32_t* __restrict__ idsOut, uint32_t* __restrict__ sorted)
{
	__shared__ int sW[kWarps];
	int t, start, end, first;
	if (!chunkRange(chunkBase, ctr, tasks, blockIdx.x, t, start, end, first)) {
		return;
	}
	const SahTask tk = tasks[t];
	const SahSplit s = splits[t];
	const AxisFrame f = s.axis >= 0 ? axisFrame(bounds + (size_t) t * 12, s.axis) : AxisFrame{0.0f, 0.0f, false};
	// left elements of the range's earlier chunks
	int before = 0;
	for (int c = first + (int) threadIdx.x; c < (int) blockIdx.x; c += blockDim.x) {
		before += chunkLeft[c];
	}
	int dummy;
	before = __reduce_add_sync(0xffffffffu, before);
	if ((threadIdx.x & 31) == 0) {
		sW[threadIdx.x >> 5] = before;
	}
	__syncthreads();
	int leftBefore = 0;
	for (int w = 0; w < kWarps; ++w) {
		leftBefore += sW[w];
	}
	__syncthreads();
	// this thread's run of kItems consecutive elements
	const int p0 = start + (int) threadIdx.x * kItems;
	uint32_t id[kItems];
	bool fl[kItems];
	int mine = 0;
#pragma unroll
	for (int k = 0; k < kItems; ++k) {
		const int p = p0 + k;
		fl[k] = false;
		id[k] = 0;
		if (p < end) {
			id[k] = ids[p];
			fl[k] = goesLeft(id[k], p, tk, s, f, cen);
			mine += fl[k] ? 1 : 0;
		}
	}
	int rank = leftBefore + blockExclusiveScan(mine, sW, dummy);
#pragma unroll
	for (int k = 0; k < kItems; ++k) {
		const int p = p0 + k;
		if (p < end) {
			// left: lo + (left elements before p); right: lo + nLeft + (right elements before p)
			const int dst = fl[k] ? tk.lo + rank : tk.lo + s.nLeft + (p - tk.lo - rank);
			rank += fl[k] ? 1 : 0;
			if (dst < tk.lo || dst >= tk.hi) {
				atomicExch(&ctr[kSahError], 1u);
				continue;
			}
			idsOut[dst] = id[k];
			sorted[dst] = id[k];
		}
	}
}

// ------------------------------------------------------------------ block phase (ranges 2..kBigTask)

// A block builds its range to the leaves in shared memory, its elements' boxes held there from the start:
//  * ranges above kMidTask elements: split by the whole block, one after another (a handful);
//  * ranges of 33..kMidTask: one warp each, all ranges of a depth side by side;
//  * ranges up to 32: one warp each, one element per lane, all subranges of a depth at once (smallBuild).
// What bounds a block is the chain of splits below each other, so what matters is that splits which do
// not depend on each other run together. With every range above 32 split by the whole block in turn and
// every subrange of a small one split alone, the 131,072-triangle mesh took 885 us here, 94 instances 58.
constexpr int kBlockThreads = 512;
constexpr int kBlockGrid = 152; // one block per SM, by shared memory
constexpr int kBlockWarps = kBlockThreads / 32;
constexpr int kMidTask = 256;

struct BlockShared
{
	float box[6][kBigTask];                        // by local element: lo xyz, hi xyz
	uint32_t gid[kBigTask];                        // by local element: primitive
	uint16_t ids[kBigTask], tmp[kBigTask];         // local elements in sorted order
	uint32_t bins[kBlockWarps][kTaskBinWords];     // per warp; the first also for whole-block splits
	int4 stack[16];                                // ranges above kMidTask: disjoint, at most kBigTask / 257
	int4 mid[2][kBigTask / (kSmallTask + 1) + 1];  // ranges of 33..kMidTask of this depth and the next
	int4 small[kBigTask / 2];                      // ranges of 2..32
	uint32_t red[kBlockWarps][12];
	uint32_t bounds[12];
	int scan[kBlockWarps];
	uint8_t perm[kBlockWarps][32];
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
#pragma unroll
		for (int a = 0; a < 3; ++a) {
			if (!fr[a].valid) {
				continue;
			}
			uint32_t* bb = to + (a * kBins + binOf(centroid(e, a), fr[a].cmin, fr[a].scale)) * kBinWords;
			atomicMin(&bb[0], ordered(box[0][e]));
			atomicMin(&bb[1], ordered(box[1][e]));
			atomicMin(&bb[2], ordered(box[2][e]));
			atomicMax(&bb[3], ordered(box[3][e]));
			atomicMax(&bb[4], ordered(box[4][e]));
			atomicMax(&bb[5], ordered(box[5][e]));
			atomicAdd(&bb[6], 1u);
		}
	}
	__device__ __forceinline__ bool left(int e, int pos, int first, const SahSplit& s, const AxisFrame& f) const
	{
		return s.axis < 0 ? pos < first + s.nLeft : binOf(centroid(e, s.axis), f.cmin, f.scale) < s.bin;
	}
};

// Where a block's nodes go.
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

__device__ __forceinline__ void clearBins(uint32_t* bins, int first, int step)
{
	for (int k = first; k < kTaskBinWords; k += step) {
		const int w = k % kBinWords;
		bins[k] = w < 3 ? kEmptyLo : (w < 6 ? kEmptyHi : 0u);
	}
}

// One thread: the node of range [a, b) split after nLeft elements, and its children queued by size.
// Positions are the block's; `base` is the block's first sorted position.
__device__ __forceinline__ void emitRange(BlockShared& S, int a, int b, int node, int nLeft, const uint32_t* b12, int base, int midList,
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
			if (S.top < 16) { // whole-block splits only: no other thread pushes
				S.stack[S.top++] = r;
			} else {
				out.error();
			}
		} else if (n > kSmallTask) {
			const int k = atomicAdd(&S.nMid[midList], 1);
			if (k <= kBigTask / (kSmallTask + 1)) {
				S.mid[midList][k] = r;
			} else {
				out.error();
			}
		} else if (n >= 2) {
			const int k = atomicAdd(&S.nSmall, 1);
			if (k < kBigTask / 2) {
				S.small[k] = r;
			} else {
				out.error();
			}
		}
	}
}

// A range of 33..kMidTask elements split by one warp.
__device__ void warpSplit(BlockShared& S, const int4 range, int base, int midList, const NodeSink& out)
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
// all subranges of a depth are split together. Every lane takes its own element's bin as the last one left
// of a split (the splits between two neighbouring elements' bins are the same split; the host takes the
// first, after the left one's bin) and gathers both sides' boxes from its subrange, element by element,
// along each axis; the best of the subrange's candidates, in the host's order, is its split.
__device__ void smallBuild(BlockShared& S, const int4 range, int base, const NodeSink& out)
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
		// Bounds of the subrange: every lane goes once around it.
		uint32_t b12[12];
#pragma unroll
		for (int k = 0; k < 6; ++k) {
			b12[k] = w[k];
		}
#pragma unroll
		for (int k = 0; k < 3; ++k) {
			b12[6 + k] = b12[9 + k] = ordered(c[k]);
		}
		int j = lane;
		for (int k = 1; k < longest; ++k) {
			j = j + 1 < y ? j + 1 : x;
			const int src = active ? j : lane; // once around: further turns meet the same elements again
#pragma unroll
			for (int q = 0; q < 6; ++q) {
				const uint32_t v = __shfl_sync(kAll, w[q], src);
				b12[q] = q < 3 ? min(b12[q], v) : max(b12[q], v);
			}
#pragma unroll
			for (int q = 0; q < 3; ++q) {
				const uint32_t v = ordered(__shfl_sync(kAll, c[q], src));
				b12[6 + q] = min(b12[6 + q], v);
				b12[9 + q] = max(b12[9 + q], v);
			}
		}
		uint32_t myBin[3], packed = 0;
		bool valid[3];
#pragma unroll
		for (int ax = 0; ax < 3; ++ax) {
			const AxisFrame f = axisFrame(b12, ax);
			valid[ax] = f.valid;
			myBin[ax] = f.valid ? (uint32_t) binOf(c[ax], f.cmin, f.scale) : 0u;
			packed |= myBin[ax] << (8 * ax);
		}
		// Both sides of this lane's candidate on each axis.
		uint32_t L[3][6], R[3][6];
		int lc[3] = {1, 1, 1};
#pragma unroll
		for (int ax = 0; ax < 3; ++ax) {
#pragma unroll
			for (int q = 0; q < 6; ++q) {
				L[ax][q] = w[q];
				R[ax][q] = q < 3 ? kEmptyLo : kEmptyHi;
			}
		}
		j = lane;
		for (int k = 1; k < longest; ++k) {
			j = j + 1 < y ? j + 1 : x;
			const int src = active ? j : lane;
			const bool counts = k < len;
			const uint32_t theirs = __shfl_sync(kAll, packed, src);
			uint32_t v[6];
#pragma unroll
			for (int q = 0; q < 6; ++q) {
				v[q] = __shfl_sync(kAll, w[q], src);
			}
#pragma unroll
			for (int ax = 0; ax < 3; ++ax) {
				const bool l = ((theirs >> (8 * ax)) & 0xffu) <= myBin[ax];
				lc[ax] += l && counts ? 1 : 0;
#pragma unroll
				for (int q = 0; q < 6; ++q) {
					const uint32_t empty = q < 3 ? kEmptyLo : kEmptyHi;
					const uint32_t vl = l ? v[q] : empty, vr = l ? empty : v[q];
					L[ax][q] = q < 3 ? min(L[ax][q], vl) : max(L[ax][q], vl);
					R[ax][q] = q < 3 ? min(R[ax][q], vr) : max(R[ax][q], vr);
				}
			}
		}
		// The lane's best candidate as (cost bits, axis and bin, left count): costs are not negative, so their
		// bits are ordered, and among equal costs the first (axis, bin) is the smaller word.
		float bestCost = kInf;
		uint32_t bestKey = 0xffffffffu;
#pragma unroll
		for (int ax = 0; ax < 3; ++ax) {
			const int rc = len - lc[ax];
			if (active && valid[ax] && rc > 0) {
				const float ha = halfAreaOf(unordered(L[ax][0]), unordered(L[ax][1]), unordered(L[ax][2]), unordered(L[ax][3]), unordered(L[ax][4]),
				                            unordered(L[ax][5]));
				const float hb = halfAreaOf(unordered(R[ax][0]), unordered(R[ax][1]), unordered(R[ax][2]), unordered(R[ax][3]), unordered(R[ax][4]),
				                            unordered(R[ax][5]));
				const float cost = __fadd_rn(__fmul_rn(ha, (float) lc[ax]), __fmul_rn(hb, (float) rc));
				if (cost < bestCost) {
					bestCost = cost;
					bestKey = ((uint32_t) (ax * kBins) + myBin[ax] + 1u) << 8 | (uint32_t) lc[ax];
				}
			}
		}
		__syncwarp();
		// The best of the subrange.
		const float mineCost = bestCost;
		const uint32_t mineKey = bestKey;
		j = lane;
		for (int k = 1; k < longest; ++k) {
			j = j + 1 < y ? j + 1 : x;
			const int src = active ? j : lane;
			const float oc = __shfl_sync(kAll, mineCost, src);
			const uint32_t ok = __shfl_sync(kAll, mineKey, src);
			if (oc < bestCost || (oc == bestCost && ok < bestKey)) {
				bestCost = oc;
				bestKey = ok;
			}
		}
		const bool middle = bestKey == 0xffffffffu;
		const int nLeft = middle ? len / 2 : (int) (bestKey & 0xffu);
		const uint32_t key = bestKey >> 8;
		const uint32_t axis = key / kBins, cut = key % kBins; // a cut after bin 31 has no right side
		const uint32_t mine = axis == 0u ? myBin[0] : (axis == 1u ? myBin[1] : myBin[2]);
		const bool goLeft = active && (middle ? lane < x + nLeft : mine < cut);
		// stable partition within the subrange
		const uint32_t below = (1u << lane) - 1u, fromX = ~((1u << x) - 1u);
		const int leftRank = __popc(__ballot_sync(kAll, goLeft) & below & fromX);
		int dst = !active ? lane : (goLeft ? x + leftRank : x + nLeft + (lane - x - leftRank));
		if (dst < 0 || dst >= 32) {
			out.error();
			dst = lane;
		}
		S.perm[warp][dst] = (uint8_t) lane;
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
		const int src = S.perm[warp][lane];
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

// One range of at most kBigTask primitives, by the whole block; see kSahBlock.
__device__ __forceinline__ void buildRange(BlockShared& S, const SahTask task, const SahTask* tasks, const InstanceRec* inst, float4* gLo,
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
		clearBins(S.bins[0], (int) threadIdx.x, kBlockThreads);
		__syncthreads();
		if (threadIdx.x < 12) {
			const int k = threadIdx.x;
			uint32_t v = S.red[0][k];
			for (int w = 1; w < kBlockWarps; ++w) {
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
		const int per = (b - a + kBlockThreads - 1) / kBlockThreads;
		const int p0 = a + (int) threadIdx.x * per;
		const int p1 = min(b, p0 + per);
		const AxisFrame f = s.axis >= 0 ? (s.axis == 0 ? fr[0] : (s.axis == 1 ? fr[1] : fr[2])) : AxisFrame{0.0f, 0.0f, false};
		int mine = 0;
		for (int p = p0; p < p1; ++p) {
			mine += S.left(S.ids[p], p, a, s, f) ? 1 : 0;
		}
		int total;
		int rank = blockExclusiveScan<kBlockWarps>(mine, S.scan, total);
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
		const int m = min(S.nMid[list], kBigTask / (kSmallTask + 1) + 1);
		if (m == 0) {
			break;
		}
		for (int k = warp; k < m; k += kBlockWarps) {
			warpSplit(S, S.mid[list][k], base, list ^ 1, out);
		}
		__syncthreads();
		if (threadIdx.x == 0) {
			S.nMid[list] = 0; // this list takes the depth after next
		}
		__syncthreads();
	}
	// ranges of up to 32 elements
	for (int k = warp; k < min(S.nSmall, kBigTask / 2); k += kBlockWarps) {
		smallBuild(S, S.small[k], base, out);
	}
	__syncthreads();
	for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
		sorted[base + i] = S.gid[S.ids[i]];
	}
}

// tasks: ranges that the blocks take in turn, or null for a one-block build of primitives [0, n) in the given order. Boxes
// come from gLo / gHi, or, for a TLAS, from the instance records, and are then stored there for the collapse.
__global__ void __launch_bounds__(kBlockThreads) kSahBlock(const SahTask* __restrict__ tasks, int n, const InstanceRec* __restrict__ inst,
                                                           float4* gLo, float4* gHi, uint32_t* __restrict__ sorted, NodeSink out)
{
	extern __shared__ __align__(16) uint8_t smem[];
	BlockShared& S = *reinterpret_cast<BlockShared*>(smem);
	if (tasks == nullptr) {
		buildRange(S, SahTask{0, n, 0, 0}, nullptr, inst, gLo, gHi, sorted, out);
		return;
	}
	if (out.ctr[kSahNext] != 0u) {
		return; // the levels are not done: nothing is taken yet
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

inline int blocksFor(int n, int b) { return (n + b - 1) / b; }

} // namespace

void prepareSahBlock()
{
	static const bool done = [] {
		RGL_SAH_OK(cudaFuncSetAttribute(kSahBlock, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) sizeof(BlockShared)));
		return true;
	}();
	(void) done;
}

SahTopology::SahTopology(const float4* lo, const float4* hi, int n, BinNode* bin, int32_t* rangeFirst, int32_t* rangeLast,
                         uint32_t* sortedIds, cudaStream_t stream)
    : lo_(lo), hi_(hi), n_(n), bin_(bin), rangeFirst_(rangeFirst), rangeLast_(rangeLast), sorted_(sortedIds), stream_(stream), scratch_(stream)
{
	maxBig_ = n / (kBigTask + 1) + 1;       // disjoint ranges above kBigTask
	const int maxBlock = n / 2 + 1;          // disjoint ranges of at least 2
	const int maxChunks = n / kChunk + maxBig_ + 1;
	scratch_.carve([&](BuildScratch::Carver& place) {
		place(cen_, n);
		place(idsCur_, n);
		place(idsNext_, n);
		place(cur_, maxBig_);
		place(next_, maxBig_);
		place(blockTasks_, maxBlock);
		place(splits_, maxBig_);
		place(bounds_, (size_t) maxBig_ * 12);
		place(bins_, (size_t) maxBig_ * kTaskBinWords);
		place(chunkBase_, maxBig_ + 1);
		place(chunkLeft_, maxChunks);
		place(ctr_, kSahWords);
	});
	kSahInit<<<blocksFor(n, 256), 256, 0, stream>>>(lo, hi, n, cen_, idsCur_, sortedIds, cur_, blockTasks_, ctr_);
	countLaunch();
	if (n < 2) {
		ctr_ = nullptr;
		return;
	}
	// As many levels as an even tree takes and two more (a level with nothing left costs six empty
	// launches, about 12 us; a look at what is left about 20).
	while (n > kBigTask && (kBigTask << levels_) < n) {
		++levels_;
	}
	levels_ += levels_ > 0 ? 2 : 0;
}

void SahTopology::enqueue()
{
	if (ctr_ == nullptr) {
		return;
	}
	const int grid = n_ / kChunk + maxBig_ + 1; // bound on a level's chunks; blocks past them return
	for (int l = 0; l < levels_; ++l) {
		kSahLevelPrep<<<1, 1024, 0, stream_>>>(cur_, chunkBase_, bounds_, ctr_);
		kSahBounds<<<grid, kThreads, 0, stream_>>>(cur_, ctr_, chunkBase_, idsCur_, lo_, hi_, cen_, bounds_, bins_);
		kSahBins<<<grid, kThreads, 0, stream_>>>(cur_, ctr_, chunkBase_, idsCur_, lo_, hi_, cen_, bounds_, bins_);
		kSahSplit<<<blocksFor(maxBig_ * 32, 128), 128, 0, stream_>>>(cur_, bounds_, bins_, splits_, bin_, rangeFirst_, rangeLast_, next_,
		                                                             blockTasks_, ctr_);
		kSahPartCount<<<grid, kThreads, 0, stream_>>>(cur_, ctr_, chunkBase_, idsCur_, cen_, bounds_, splits_, chunkLeft_);
		kSahPartScatter<<<grid, kThreads, 0, stream_>>>(cur_, ctr_, chunkBase_, idsCur_, cen_, bounds_, splits_, chunkLeft_, idsNext_, sorted_);
		countLaunch(6);
		std::swap(cur_, next_);
		std::swap(idsCur_, idsNext_);
	}
	levels_ = 4; // of a tree that is deeper
	// Blocks take ranges until none is left: their number is known on the device only.
	prepareSahBlock();
	kSahBlock<<<std::min(n_ / 2 + 1, kBlockGrid), kBlockThreads, sizeof(BlockShared), stream_>>>(
	    blockTasks_, n_, nullptr, const_cast<float4*>(lo_), const_cast<float4*>(hi_), sorted_, NodeSink{bin_, rangeFirst_, rangeLast_, ctr_});
	countLaunch();
}

static_assert(kBigTask == kSahSmallMax, "one block builds ranges up to kSahSmallMax primitives");

void enqueueSahTopologySmall(const InstanceRec* inst, float4* lo, float4* hi, int n, BinNode* bin, int32_t* rangeFirst, int32_t* rangeLast,
                             uint32_t* sortedIds, cudaStream_t s)
{
	if (n <= 0 || n > kSahSmallMax) {
		throw std::runtime_error("SAH build: one-block topology takes 1.." + std::to_string(kSahSmallMax) + " primitives");
	}
	kSahBlock<<<1, kBlockThreads, sizeof(BlockShared), s>>>(nullptr, n, inst, lo, hi, sortedIds, NodeSink{bin, rangeFirst, rangeLast, nullptr});
	countLaunch();
}

} // namespace rgl
