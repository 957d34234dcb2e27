// CPU harness of csrc/beam_tasks.hpp.
#include "beam_tasks.hpp"

extern "C" int beams_per_task(int samples, int beams, int64_t launchBeams, int64_t residentWarps, int cells)
{
	return rgl::beamsPerTask(samples, beams, launchBeams, residentWarps, cells);
}

extern "C" int lane_group_samples() { return rgl::kLaneGroupSamples; }
extern "C" int pool_samples() { return rgl::kPoolSamples; }
extern "C" uint32_t sample_factor(int samples) { return rgl::sampleFactor(samples); }
