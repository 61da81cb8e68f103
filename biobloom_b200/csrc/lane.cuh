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

/* What lane_list_kernel finds of a batch's lengths: reads above kLaneMaxBases, reads
 * above kLaneShortBases up to there, bases of the others and the longest of these. */
enum { kLaneLong, kLaneMid, kLaneBases, kLaneLongest, kLaneStats };
constexpr uint32_t kLaneMaxBases = 1024, kLaneShortBases = 384;

/* Whether the lane kernel takes a batch of so many reads with these lengths.  Where
 * one read in 64 is long the other kernels wait for the last of these (the lane kernel
 * starts with them), whatever the short ones are. */
__host__ __device__ inline bool lane_takes(const LaneRule &r, const unsigned long long *st,
		uint64_t reads)
{
	if (st[kLaneMid] * r.mids > reads || st[kLaneLong] * r.longs > reads)
		return false;
	if (st[kLaneLong] * 64 >= reads)
		return true;
	const uint64_t shorts = reads - st[kLaneLong] - st[kLaneMid];
	return st[kLaneBases] <= r.mean * shorts &&
			(!r.even || 5 * st[kLaneBases] >= 4 * st[kLaneLongest] * shorts);
}

#if defined(__CUDACC__)
/* A batch that is decided on the device: is it the lane kernel's? */
__device__ __forceinline__ bool lane_has(const ClassifyArgs &a)
{
	return lane_takes(a.lane_rule, a.lane_stats, a.n * a.mates);
}
#endif

/* Device scratch of a launch: the indexes of the batch's reads above kLaneShortBases
 * (n * mates entries: those above kLaneMaxBases from the front, the others from the
 * back) and lane_counters(nf) counters, of which the first kLaneStats are the
 * counts. */
struct LaneScratch {
	uint32_t *list;
	unsigned long long *ctr;
};

/* Whether the lane kernel can take these filters and options at all, and which
 * batches it is the faster one for. */
bool lane_supports(const FilterDev *hf, uint32_t nf, uint32_t streak_thr, uint64_t total_reads);
struct LaneAim {
	bool scores;   /* every frame is walked (BESTHIT, SCORES) */
	bool quick;    /* decided after few frames: LENGTH, thresholds above 0.3 */
	bool harmonic, length;
	bool host;     /* the lengths are read on the host (filter-major path) */
};
LaneRule lane_rule(const FilterDev *hf, uint32_t nf, const LaneAim &aim, uint64_t reads);

/* Counters of a launch (which is a kernel per filter, after one that lists the
 * longer reads). */
inline size_t lane_counters(uint32_t nf)
{
	return kLaneStats + 2 * (size_t)nf;
}

/* The list and the counts, which every launch_lane over the batch reads. */
cudaError_t launch_lane_list(const ClassifyArgs &a, const LaneScratch &ls, int num_sms,
		cudaStream_t s);

/* Hits of a batch (sa NULL), or the scores of every (read, filter) into sa->scores,
 * and with `hits` both in one walk (count: hits alone).  With two or more filters the
 * hit words are ORed into and must be zeroed before. */
cudaError_t launch_lane(const ClassifyArgs &a, const FilterDev *hf, const ScoreArgs *sa,
		bool hits, const LaneScratch &ls, int num_sms, bool count, cudaStream_t s);

} // namespace bbt

#endif
