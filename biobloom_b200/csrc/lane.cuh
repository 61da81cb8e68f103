/*
 * lane.cuh -- launch interface of the lane kernel (lane.cu).
 */
#ifndef BBT_LANE_CUH
#define BBT_LANE_CUH

#include <cuda_runtime.h>
#include <stdint.h>

#include "classify.cuh"

namespace bbt {

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
