// Cutting a traversal launch's beams into tasks, one warp's work each (trace_batch.cu), as host-only
// functions so that a CPU test checks them too.
#pragma once

#include <algorithm>
#include <cstdint>

namespace rgl {

// Lane groups take patterns of up to this many samples, pooled samples the larger ones. From 17 samples on a
// group leaves up to half of the lanes idle and the selection, done by one lane per beam, weighs more: 58
// samples on two rounds of 32 lanes took 2276 us for 65,536 beams over 1M triangles, pooled 1195 us. Below,
// groups keep the beam's pose in registers: 5 samples took 302 us for 262,144 beams in groups, pooled 327 us
// (six beams a task); 9 / 13 / 16 samples for 20,000 beams of a plain scene 39 / 50 / 50 us in groups, pooled
// 86 / 88 / 91 us (one beam a task, as the pool's rule has it) and 41 / 54 / 54 us with 3 / 2 / 2.
constexpr int kLaneGroupSamples = 16;
// Samples that a warp keeps in shared memory between tracing a task's beams and selecting their returns: 6
// beams of 58, the default pattern. With shading a block of 256 threads keeps 45 KB so, and 25 KB of stacks.
constexpr int kPoolSamples = 352;
constexpr int kResidentWarps = 16; // per SM, at 128 registers

// Beams per task of a job with `samples` rays a beam and `beams` beams, with samples spread over the lanes (one
// lane per beam always takes 32). launchBeams: beams of all jobs of the launch; residentWarps: of the device.
// A launch that does not fill the chip twice over takes fewer beams per task, because a warp ends with its
// slowest ray and fewer rays diverge less: with 32 beams, 16, 8 and 1 per task, 3,600 beams took 35 / 33
// / 37 / 32 us, 32,768 beams 39 / 37 / 36 / 101 us, 76,920 beams 112 / 97 / 99 / 365 us, 131,072 beams 92
// / 89 / 98 / 474 us. What L2 holds does not matter, a pose may: 32,768 beams in tasks of 4 / 7 / 14 / 32 took
// 49 / 46 / 48 / 54 us over twelve poses in the plain scene and 94 / 100 / 119 / 143 in a hilly one (37 / 40 /
// 45 against 33 / 35 / 42 in tasks of 7 / 14 / 32 with L2 written over before every run), but 58 / 48 / 49 in
// tasks of 7 / 14 / 32 from the plain scene's centre, facing along an axis. Pooled samples want about eight
// tasks per warp (58 samples, 65,536 beams: 1221 / 1001 / 916 / 928 / 1010 us with 1 / 2 / 3 / 4 / 6 beams
// per task): fewer leave a long tail.
// `cells`: direction cells that the beams fill (launchCountCells on their sorted keys, 0: not known). The
// beams of a cell, less than 0.4 degrees apart in azimuth, take nearly the same walk, so a warp takes them
// together however small the launch: a ring of 3,000 / 12,000 / 30,000 beams took 27 / 29 / 29 us in
// tasks of 1 / 3 / 7 beams, 21 us in tasks of 2 / 10 / 16 and more.
inline int beamsPerTask(int samples, int beams, int64_t launchBeams, int64_t residentWarps, int cells)
{
	if (samples > kLaneGroupSamples) {
		return (int) std::max<int64_t>(1, std::min<int64_t>(launchBeams / (8 * residentWarps), std::min(32, kPoolSamples / samples)));
	}
	int64_t want = (launchBeams + 2 * residentWarps - 1) / (2 * residentWarps);
	if (cells > 0) {
		want = std::max<int64_t>(want, beams / cells);
	}
	return (int) std::max<int64_t>(1, std::min<int64_t>(want, 32 / samples));
}

// Factor of a division by a pattern's samples: i / samples = (i * factor) >> 16 for every sample i of a task.
inline uint32_t sampleFactor(int samples) { return (uint32_t) ((65536 + samples - 1) / samples); }

} // namespace rgl
