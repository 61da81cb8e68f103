/*
 * lane.cuh -- launch interface of the lane kernel (lane.cu).
 */
#ifndef BBT_LANE_CUH
#define BBT_LANE_CUH

#include <cuda_runtime.h>
#include <stdint.h>

#include "classify.cuh"

namespace bbt {

/* The warp kernel takes reads above this many bases in windows of up to 256 frames
 * (lane_long_item): a window costs the latency of h probes and the hashing of 256
 * frames however few of them decide the read, so windows pay where the earliest
 * decision is some 200 frames away.  Against steps of 32 or 64 frames, 8,000 reads of
 * one length over a 3.4 MB filter / a 2.1 GB one: 600 bases 177 against 119 us / 208
 * against 175, 1,000 bases 187 against 164 / 262 against 253, 1,600 bases 202 against
 * 236 / 351 against 372, 5,000 bases 404 against 633 / 944 against 1032.  Ragged reads
 * (50 to 300 bases, 5 % of 300 to 10,000) take the same time with this limit as with
 * one of 384 (8,000 over the small filter: 255 us, steps alone 659). */
constexpr uint32_t kWindowBases = 1536;

/* Device scratch of a launch: the indexes of the batch's long reads (n * mates
 * entries) and lane_counters(nf) counters, zeroed by the launch. */
struct LaneScratch {
	uint32_t *list;
	unsigned long long *ctr;
};

/* Whether the lane kernel takes these filters and options, and whether it is the
 * faster one for a batch of so many reads. */
bool lane_supports(const FilterDev *hf, uint32_t nf, uint32_t streak_thr, uint64_t total_reads);
bool lane_pays(const FilterDev *hf, uint32_t nf, uint64_t total_reads, bool scores);

/* Counters of a launch (which is a kernel per filter, after one that lists long
 * reads). */
inline size_t lane_counters(uint32_t nf)
{
	return 1 + 2 * (size_t)nf;
}

/* Hits of a batch (sa NULL), or the scores of every (read, filter) into
 * sa->scores, and with `hits` both in one walk (count: hits alone).  With two or more filters the hit words are ORed into and must be
 * zeroed before. */
cudaError_t launch_lane(const ClassifyArgs &a, const FilterDev *hf, const ScoreArgs *sa,
		bool hits, const LaneScratch &ls, int num_sms, bool count, cudaStream_t s);

} // namespace bbt

#endif
