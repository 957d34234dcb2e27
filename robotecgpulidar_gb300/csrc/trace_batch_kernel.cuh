// Device side of the persistent batch traversal: the task functions of the two packings (a task's
// samples spread over the lanes, or one lane per beam) and the kernel template. Included by
// trace_batch.cu, which instantiates the kernels.
#pragma once

#include "trace_kernel.cuh"

namespace rgl {
namespace {

using namespace tracedev;

__device__ __forceinline__ void loadRay(const BatchJob* __restrict__ job, uint32_t beam, Mat34& ray, float& minRange, float& maxRange)
{
	ray = loadMat(job->p.rays + beam);
	if (job->hasRayTransform) {
		Mat34 tf;
#pragma unroll
		for (int r = 0; r < 3; ++r) {
#pragma unroll
			for (int c = 0; c < 4; ++c) {
				tf.m[r][c] = job->rayTransform.m[r][c];
			}
		}
		ray = mul(tf, ray);
	}
	if (job->p.ranges) {
		const float* rg = job->p.ranges + 2 * (job->p.nRanges == 1 ? 0u : beam);
		minRange = rg[0];
		maxRange = rg[1];
	} else {
		minRange = job->inlineRange[0];
		maxRange = job->inlineRange[1];
	}
}

// A traced sample in the warp's pool: distance and hit, with SHADING also intensity and triangle.
template<bool SHADING>
struct PoolEntry;
template<>
struct PoolEntry<false>
{
	uint2 w;
	__device__ __forceinline__ void set(const SampleVal& v) { w = make_uint2(__float_as_uint(v.dist), (uint32_t) v.inst); }
	__device__ __forceinline__ SampleVal get() const { return SampleVal{__uint_as_float(w.x), (int32_t) w.y, 0.0f, -1}; }
};
template<>
struct PoolEntry<true>
{
	uint4 w;
	__device__ __forceinline__ void set(const SampleVal& v)
	{
		w = make_uint4(__float_as_uint(v.dist), (uint32_t) v.inst, __float_as_uint(v.intensity), (uint32_t) v.tri);
	}
	__device__ __forceinline__ SampleVal get() const
	{
		return SampleVal{__uint_as_float(w.x), (int32_t) w.y, __uint_as_float(w.z), (int32_t) w.w};
	}
};

// Lane groups: the S samples of a beam on S adjacent lanes, 32 / S beams per task; the group's first lane
// takes the samples in order from the others and writes the beam's returns, with the beam's pose still in
// its registers. For up to kLaneGroupSamples samples a beam (see there).
template<bool SHADING>
__device__ __forceinline__ void laneGroupTask(const BatchJob* __restrict__ job, int first, int beams, const SceneView& sc, DevStack& st,
                                              int lane)
{
	const int S = job->p.nSamples;
	const int g = (int) (((uint32_t) lane * job->sampleMagic) >> 16); // lane / S
	const int s = lane - g * S;
	const bool valid = g < beams;
	const int local = first + (valid ? g : 0);
	uint32_t beam = 0;
	Mat34 ray = Mat34::identity();
	float minRange = 0.0f, maxRange = 0.0f;
	SampleVal v{job->p.farNonHitDistance, kNoHit, 0.0f, -1};
	if (valid) {
		beam = job->order ? __ldg(job->order + local) : (uint32_t) local;
		loadRay(job, beam, ray, minRange, maxRange);
		// A masked ray is not cast: all its samples are far non-hits (reference optixPrograms.cu:55-58).
		if (!(job->p.rayMask && job->p.rayMask[beam] == 0)) {
			const Mat34 traced = SHADING ? distortRay(job->p, beam, ray) : ray;
			const Mat34 sr = (s == 0) ? traced : mul(traced, loadMat(job->samples + s));
			v = traceSample<SHADING>(job->p, sc, sr, minRange, maxRange, st, s);
		}
	}
	const bool leader = valid && s == 0;
	ReturnReducer red;
	red.init(job->p.farNonHitDistance);
	for (int k = 0; k < S; ++k) {
		SampleVal cur;
		cur.dist = __shfl_sync(0xffffffffu, v.dist, lane + k);
		cur.inst = __shfl_sync(0xffffffffu, v.inst, lane + k);
		cur.intensity = SHADING ? __shfl_sync(0xffffffffu, v.intensity, lane + k) : 0.0f;
		cur.tri = SHADING ? __shfl_sync(0xffffffffu, v.tri, lane + k) : -1;
		if (leader) {
			red.add(k, cur);
		}
	}
	if (leader) {
		writeReturns<SHADING>(job->p, sc, job->samples, beam, ray, red);
	}
}

// Pooled samples: beams [first, first + beams) of a job in visiting order, by one warp: the beams' samples, numbered
// beam by beam, go 32 at a time to the lanes, which leave what they hit in the warp's pool in shared
// memory; then lane k selects and writes the returns of beam k. The lanes of a round hold neighbouring
// samples of neighbouring beams, no lane idles because a beam's samples do not divide 32, and the
// selection and the field writes run once for all beams of the task with one beam per lane. (With
// each beam's samples on its own min(S, 32) lanes and one selecting lane per beam, 5 samples a beam
// left 2 of 32 lanes idle and wrote with 6, 58 samples left 3 idle per round and wrote with 1.)
template<bool SHADING>
__device__ __forceinline__ void pooledTask(const BatchJob* __restrict__ job, int first, int beams, const SceneView& sc, DevStack& st,
                                           PoolEntry<SHADING>* pool, int lane)
{
	const int nSamples = job->p.nSamples;
	const uint32_t magic = job->sampleMagic;
	const int total = beams * nSamples;
	for (int base = 0; base < total; base += 32) {
		const int i = base + lane;
		if (i < total) {
			const int k = (int) (((uint32_t) i * magic) >> 16); // i / nSamples
			const int s = i - k * nSamples;
			const int local = first + k;
			const uint32_t beam = job->order ? __ldg(job->order + local) : (uint32_t) local;
			Mat34 ray;
			float minRange, maxRange;
			loadRay(job, beam, ray, minRange, maxRange);
			SampleVal v{job->p.farNonHitDistance, kNoHit, 0.0f, -1};
			// A masked ray is not cast: all its samples are far non-hits (reference optixPrograms.cu:55-58).
			if (!(job->p.rayMask && job->p.rayMask[beam] == 0)) {
				if (SHADING) {
					ray = distortRay(job->p, beam, ray);
				}
				if (s != 0) {
					ray = mul(ray, loadMat(job->samples + s));
				}
				v = traceSample<SHADING>(job->p, sc, ray, minRange, maxRange, st, s);
			}
			pool[i].set(v);
		}
		__syncwarp();
	}
	if (lane < beams) {
		ReturnReducer red;
		red.init(job->p.farNonHitDistance);
		const PoolEntry<SHADING>* mine = pool + lane * nSamples;
		for (int s = 0; s < nSamples; ++s) {
			red.add(s, mine[s].get());
		}
		const int local = first + lane;
		const uint32_t beam = job->order ? __ldg(job->order + local) : (uint32_t) local;
		Mat34 ray;
		float minRange, maxRange;
		loadRay(job, beam, ray, minRange, maxRange);
		writeReturns<SHADING>(job->p, sc, job->samples, beam, ray, red);
	}
	__syncwarp();
}

template<bool SHADING>
__device__ __forceinline__ void serialTask(const BatchJob* __restrict__ job, int first, const SceneView& sc, DevStack& st, int lane)
{
	const int local = first + lane;
	if (local >= job->p.nRays) {
		return;
	}
	const uint32_t beam = job->order ? __ldg(job->order + local) : (uint32_t) local;
	Mat34 ray;
	float minRange, maxRange;
	loadRay(job, beam, ray, minRange, maxRange);
	ReturnReducer red;
	red.init(job->p.farNonHitDistance);
	const int nSamples = job->p.nSamples;
	const Mat34 traced = SHADING ? distortRay(job->p, beam, ray) : ray;
	const bool cast = !(job->p.rayMask && job->p.rayMask[beam] == 0);
	for (int s = 0; s < nSamples; ++s) {
		SampleVal v{job->p.farNonHitDistance, kNoHit, 0.0f, -1};
		if (cast) {
			const Mat34 sr = (s == 0) ? traced : mul(traced, loadMat(job->samples + s));
			v = traceSample<SHADING>(job->p, sc, sr, minRange, maxRange, st, s);
		}
		red.add(s, v);
	}
	writeReturns<SHADING>(job->p, sc, job->samples, beam, ray, red);
}

// MODE 0: lane groups; MODE 1: one lane per beam; MODE 2: pooled samples.
// REGS caps registers per thread: 64, 80 and 96 keep eight, six and five 128-thread blocks resident
// per SM (more warps to hide latency, possibly with spills); 128 avoids spills in the variants that
// hold more state. The tuner picks.
template<int MODE, bool SHADING, int REGS>
__global__ void __maxnreg__(REGS) kTraceBatch(const BatchJob* __restrict__ jobs, const int32_t* __restrict__ taskBase, int nJobs,
                                              uint32_t* counter, int chunk)
{
	// Dynamic shared memory: stack columns | the warps' sample pools (pooled samples) | task bases.
	extern __shared__ __align__(16) uint2 dyn[];
	PoolEntry<SHADING>* pool = reinterpret_cast<PoolEntry<SHADING>*>(dyn + kSmemStack * blockDim.x);
	int32_t* sBase = reinterpret_cast<int32_t*>(pool + (MODE == 2 ? (blockDim.x / 32) * kPoolSamples : 0));
	pool += (threadIdx.x >> 5) * kPoolSamples;
	for (int i = threadIdx.x; i <= nJobs; i += blockDim.x) {
		sBase[i] = taskBase[i];
	}
	__syncthreads();
	const int total = sBase[nJobs];
	const int lane = threadIdx.x & 31;

	uint2 spill[kLocalStack];
	DevStack st;
	st.sm = dyn + threadIdx.x;
	st.spill = spill;
	st.stride = blockDim.x;
	st.sp = 0;
	st.overflow = false;

	for (;;) {
		uint32_t t0 = 0;
		if (lane == 0) {
			t0 = atomicAdd(counter, (uint32_t) chunk);
		}
		t0 = __shfl_sync(0xffffffffu, t0, 0);
		if (t0 >= (uint32_t) total) {
			break;
		}
		const int tEnd = min((int) t0 + chunk, total);
		for (int t = (int) t0; t < tEnd; ++t) {
			int lo = 0, hi = nJobs;
			while (hi - lo > 1) {
				const int mid = (lo + hi) >> 1;
				if (sBase[mid] <= t) {
					lo = mid;
				} else {
					hi = mid;
				}
			}
			const BatchJob* job = jobs + lo;
			const SceneView sc = *job->p.scene;
			const int first = (t - sBase[lo]) * job->beamsPerTask;
			const int beams = min(job->beamsPerTask, job->p.nRays - first);
			if (MODE == 0) {
				laneGroupTask<SHADING>(job, first, beams, sc, st, lane);
			} else if (MODE == 1) {
				serialTask<SHADING>(job, first, sc, st, lane);
			} else {
				pooledTask<SHADING>(job, first, beams, sc, st, pool, lane);
			}
			if (st.overflow) {
				if (job->p.errorFlag) {
					*(volatile int32_t*) job->p.errorFlag = 1; // an error slot in mapped host memory
				}
				st.overflow = false;
				st.sp = 0;
			}
		}
	}
	// Every task is handed out: a traversal launched after this one with programmatic stream
	// serialization may start its blocks as this grid's blocks exit (the first warp of each block to
	// get here triggers for the block). The next launch reads nothing this one writes.
	asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
	// Launched that way itself, a launch ends only after the launch before it has completed: later work
	// on the stream, which waits for this launch, then also follows every earlier one, and each
	// launch's counter block is re-armed before the stream reaches the next launch that uses it. A
	// launch without a programmatic predecessor passes this at once.
	asm volatile("griddepcontrol.wait;" ::: "memory");
	// The last block to finish re-arms both counters for the next launch, so no launch needs a memset
	// first: every block has left the task loop when it counts itself finished.
	__syncthreads();
	if (threadIdx.x == 0) {
		__threadfence();
		if (atomicAdd(counter + 1, 1u) == gridDim.x - 1) {
			atomicExch(counter, 0u);
			atomicExch(counter + 1, 0u);
		}
	}
}

} // namespace
} // namespace rgl
