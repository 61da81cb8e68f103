/*
 * lane.cu -- classification and scoring with one read per lane.
 *
 * The warp kernels (classify.cu, twopass.cu) give a read to a warp: 32 frames
 * are hashed and probed at once and the SeqEval machine runs on the ballots.
 * That costs each lane a whole k-mer of hashing for the few frames it owns and
 * the warp ~100 instructions of bit arithmetic per 32 frames, and probes
 * frames after the decision.  Here every lane walks a read of its own, eight
 * bases at a time: the rolling hash costs two table reads and ~16 instructions
 * a frame, the walk is the reference's own loop (lane_walk.cuh), and a warp
 * instruction still serves 32 frames, of 32 reads.
 *
 * A frame's filter bits are read level by level, all lanes together: level i
 * for the frames of the step whose levels 0..i-1 are set, which are the words
 * BloomFilter::contains reads.
 *
 * Work.  A launch per filter, one after another, so that the whole GPU probes
 * one filter at a time and a filter that fits L2 stays there; warps take chunks
 * of 32 reads from a counter.  A warp keeps its next items (base position,
 * length, thresholds: computed 32 at a time) in shared memory and hands them to
 * lanes as these finish.  Reads above 1024 bases, and most above 384 (lane_mids),
 * would leave a lane working long after its warp and are evaluated by whole warps,
 * before the others: a small kernel lists them.  The grid is full whatever the batch,
 * for the list (28,000 listed reads of 600 bases with one warp a chunk, 880 warps:
 * 680 us against 351), and chunks are handed to a part of each block (LaneShare): left
 * to the warps that come first they end up on some of the SMs (20,000 reads of 150
 * bases over a 3.4 MB filter 140 us against 95).
 */
#include "lane.cuh"

#include <algorithm>

#include "bbt.h"
#include "lane_item.cuh"

namespace bbt {

namespace {

constexpr int kLaneWarps = 8;     /* warps per block */
/* Blocks per SM the registers leave room for: 3 give a thread 80, which hold
 * eight frames' hashes and words in flight (with 4 blocks the steps spill, and
 * the spilled words cost more L2 and L1 than the warps bring: 11.8 against 10.1
 * ms on the ten 68 MB filters). */
constexpr int kLaneMinBlocks = 3;
/* Frames hashed and probed together.  8: fewer instructions around the probes;
 * 4 probes 3% fewer frames in vain and measured slower everywhere (0.72 against
 * 0.62 ms per 1M reads over the 3.4 MB filter, 10.1 against 8.7 on the ten). */
constexpr int kLaneSub = 8;
constexpr int kLaneRefill = 3;    /* idle lanes before a warp hands out reads (1 to 6: within 1%) */

/* One launch: one filter, whose constants are kernel parameters (constant
 * operands of the probe arithmetic, where registers would cost warps). */
struct LaneArgs {
	ClassifyArgs a;
	ScoreArgs sa;
	const uint32_t *list;
	const unsigned long long *stats;
	unsigned long long *ctr;    /* next chunk, next listed read */
	uint64_t chunks;
	uint32_t f;                 /* the filter's index */
	LaneFilter F;
};

/* What a lane needs of its read once per eight bases or less, and the bases
 * behind it, in shared memory: registers go to the probes in flight. */
template <int MODE>
struct LaneWarp {
	uint64_t base[32];          /* queue of items: first base in its mate array, */
	uint32_t read[32], len[32];
	int32_t thres[32], anti_thres[32];
	uint64_t my_base[32];       /* the same of the lanes' reads */
	uint32_t my_read[32], my_len[32];
	int32_t my_thres[32], my_anti_thres[32];
	uint32_t nib[4][32];        /* nibbles of the last 32 bases, 8 to a word */
	uint32_t first;             /* the next chunk is the warp's own */
	double hthres[MODE == SCORE_HARMONIC ? 32 : 1], my_hthres[MODE == SCORE_HARMONIC ? 32 : 1];
};

/* What a block's warps make of the batch's lengths.  Of a batch with fewer chunks than
 * warps, the first warps of each block take them, so that the SMs share them evenly:
 * without listed reads each its own first one, the others from the counter.  The
 * warps that have no chunks join in on the list only where it is long (more than
 * four reads a chunk): the longest reads, which the launch waits for, go faster
 * without (50,000 ragged reads over 2.1 GB, 2,500 of them listed: 404 us against
 * 436). */
struct LaneShare {
	uint32_t nlong, listed;     /* listed reads above kLaneMaxBases, and all */
	uint32_t max_bases;         /* of a lane's read */
	uint32_t warps;             /* of a block that take chunks */
	uint32_t own;               /* chunks that the counter does not give out */
	uint32_t help;              /* warps without chunks take listed reads */
	uint32_t go;                /* the batch is this kernel's */
};

/* The reads above kLaneShortBases (LaneScratch::list) and the counts of the
 * batch's lengths. */
__global__ void __launch_bounds__(256) lane_list_kernel(ClassifyArgs a, uint32_t *list,
		unsigned long long *stats)
{
	__shared__ uint64_t sums[8];
	__shared__ uint32_t tops[8], at[2][8], first[2];
	const uint64_t total = a.n * a.mates;
	const int lane = threadIdx.x & 31;
	const unsigned below = (1u << lane) - 1u;
	const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
	uint32_t bases = 0, longest = 0; /* this thread's reads: at most 2^32 / stride of them */
	for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < total; base += stride) {
		const uint64_t r = base + threadIdx.x;
		uint64_t len = 0;
		if (r < total) {
			const uint32_t mate = r >= a.n ? 1u : 0u;
			const uint64_t i = r - (mate ? a.n : 0);
			len = a.off[mate][i + 1] - a.off[mate][i];
		}
		if (len <= kLaneShortBases) {
			bases += (uint32_t)len;
			longest = max(longest, (uint32_t)len);
		}
		if (!__syncthreads_or(len > kLaneShortBases))
			continue;
		/* places in the list: one atomic addition of the block for each kind */
		const unsigned lm = __ballot_sync(kFull, len > kLaneMaxBases);
		const unsigned mm = __ballot_sync(kFull, len > kLaneShortBases) & ~lm;
		if (lane == 0) {
			at[0][threadIdx.x >> 5] = __popc(lm);
			at[1][threadIdx.x >> 5] = __popc(mm);
		}
		__syncthreads();
		if (threadIdx.x < 2) {
			uint32_t n = 0;
			for (int i = 0; i < 8; ++i) {
				const uint32_t c = at[threadIdx.x][i];
				at[threadIdx.x][i] = n;
				n += c;
			}
			first[threadIdx.x] = n ? (uint32_t)atomicAdd(stats + (threadIdx.x ? kLaneMid : kLaneLong),
					(unsigned long long)n) : 0u;
		}
		__syncthreads();
		if ((lm >> lane) & 1u)
			list[first[0] + at[0][threadIdx.x >> 5] + __popc(lm & below)] = (uint32_t)r;
		else if ((mm >> lane) & 1u)
			list[total - 1 - (first[1] + at[1][threadIdx.x >> 5] + __popc(mm & below))] = (uint32_t)r;
		__syncthreads(); /* read before the next ones are written */
	}
	const uint64_t sum = __reduce_add_sync(kFull, bases & 0xFFFFu) +
			((uint64_t)__reduce_add_sync(kFull, bases >> 16) << 16);
	longest = __reduce_max_sync(kFull, longest);
	if (lane == 0) {
		sums[threadIdx.x >> 5] = sum;
		tops[threadIdx.x >> 5] = longest;
	}
	__syncthreads();
	if (threadIdx.x == 0) {
		uint64_t all = 0;
		for (int i = 0; i < 8; ++i) {
			all += sums[i];
			longest = max(longest, tops[i]);
		}
		if (all) {
			atomicAdd(stats + kLaneBases, (unsigned long long)all);
			atomicMax(stats + kLaneLongest, (unsigned long long)longest);
		}
	}
}

/* Whether lanes take the reads of kLaneShortBases to kLaneMaxBases too, rather than
 * warps from the list: a lane costs a third of the instructions, but the launch then
 * lasts as long as a lane with the longest of them.  Over a filter in L2, 500,000
 * ragged reads with 7,000 of these take 902 us by warps and 1087 by lanes, 28,000
 * reads of 600 bases 351 and 260, 250,000 of them 2481 and 808; over one in HBM
 * 250,000 ragged reads 1296 and 1519, 160,000 reads of 600 bases 1967 and 1878 (scores,
 * which walk every frame: 4463 and 4596, 250,000 of 1,000 bases 11669 and 12848). */
template <bool SCORE>
__device__ __forceinline__ bool lane_mids(bool in_l2, unsigned long long mids, uint64_t reads)
{
	return in_l2 ? mids >= 25000u : !SCORE && mids * 8u > reads;
}

/* Items of chunk c, reads [32c, 32c + 32), into the warp's queue: those long
 * enough for a frame and of at most max_bases; the result of a read without
 * frames is written here.  Returns their number. */
template <int MODE, int WHAT, bool PACKED>
__device__ __forceinline__ int lane_queue(const LaneArgs &g, LaneWarp<MODE> &w, uint64_t c,
		uint32_t max_bases, int lane)
{
	constexpr bool SCORE = WHAT != kLaneHits, HITS = WHAT != kLaneScores;
	const ClassifyArgs &a = g.a;
	const uint64_t r = c * 32 + lane;
	const bool in = r < a.n * a.mates;
	uint64_t b = 0, l = 0, i = 0;
	uint32_t mate = 0;
	if (in) {
		mate = r >= a.n ? 1u : 0u;
		i = r - (mate ? a.n : 0);
		const uint64_t o = a.off[mate][i];
		l = a.off[mate][i + 1] - o;
		b = o - a.off_base[mate];
	}
	if (in && l < g.F.k) {
		if (SCORE) {
			ScoreState st;
			score_init(st);
			g.sa.scores[mate][i * a.nf + g.f] = MODE == SCORE_BINOMIAL
					? binomial_score(l, g.F.k, 0, 0.0, lane) : score_value<MODE>(st, l, g.F.k, 0.0, lane);
		}
		if (HITS && a.nf == 1)
			a.hits[mate][i] = 0;
	}
	const bool mine = in && l >= g.F.k && l <= max_bases;
	const unsigned m = __ballot_sync(kFull, mine);
	if (mine) {
		const int q = __popc(m & ((1u << lane) - 1u));
		const uint32_t frames = (uint32_t)l - g.F.k + 1u;
		w.base[q] = b;
		w.read[q] = (uint32_t)r;
		w.len[q] = (uint32_t)l;
		if (HITS) {
			int32_t t, at;
			double ht;
			lane_thresholds<MODE>(t, at, ht, a.score, a.one_minus, a.min_len,
					MODE == SCORE_BINOMIAL ? a.bthres[g.f * a.bthres_rows + frames] : 0u, frames,
					(uint32_t)l);
			w.thres[q] = t;
			w.anti_thres[q] = at;
			if (MODE == SCORE_HARMONIC)
				w.hthres[q] = ht;
		}
		/* its first bases into L1 by the time a lane takes it */
		const void *p = PACKED
				? (const void *)(reinterpret_cast<const uint32_t *>(a.seq[mate]) + (b >> 4))
				: (const void *)(a.seq[mate] + b);
		asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
	}
	__syncwarp();
	return __popc(m);
}

/* A decision into the read's hit words. */
__device__ __forceinline__ void lane_write(const LaneArgs &g, uint32_t read, int decided)
{
	const ClassifyArgs &a = g.a;
	const uint32_t mate = read >= a.n ? 1u : 0u;
	const uint64_t i = read - (mate ? a.n : 0);
	if (a.nf == 1)
		a.hits[mate][i] = decided == EVAL_ACCEPT ? 1u : 0u;
	else if (decided == EVAL_ACCEPT)
		atomicOr((unsigned long long *)&a.hits[mate][i * a.words + (g.f >> 6)],
				1ull << (g.f & 63u));
}

template <bool COUNT>
__device__ __forceinline__ void lane_count(const ClassifyArgs &a, unsigned long long (&acc)[3],
		int lane)
{
	if (!COUNT)
		return;
#pragma unroll
	for (int j = 0; j < 3; ++j)
		for (int o = 16; o; o >>= 1)
			acc[j] += __shfl_xor_sync(kFull, acc[j], o);
	if (lane == 0) {
		if (a.probes)
			atomicAdd(a.probes, acc[0]);
		if (a.frames)
			atomicAdd(a.frames, acc[1]);
		if (a.alg_probes)
			atomicAdd(a.alg_probes, acc[2]);
	}
}

template <int MODE, int WHAT, bool COUNT, bool PACKED>
__global__ void __launch_bounds__(kLaneWarps * 32, kLaneMinBlocks) lane_kernel(
		const __grid_constant__ LaneArgs g)
{
	constexpr bool SCORE = WHAT != kLaneHits, HITS = WHAT != kLaneScores;
	__shared__ LaneWarp<MODE> warps[kLaneWarps];
	__shared__ LaneTables tab;
	__shared__ LaneShare sh;
	__shared__ double terms[MODE == SCORE_HARMONIC ? kHarmTerms : 1];
	const ClassifyArgs &a = g.a;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	LaneWarp<MODE> &w = warps[warp];
	unsigned long long acc[3] = {0, 0, 0}; /* words read, frames hashed, words of the
	                                          sequential algorithm */
	if (threadIdx.x == 0) {
		const unsigned long long nmid = g.stats[kLaneMid];
		const bool mids = lane_mids<SCORE>(g.F.keep != 0, nmid, a.n * a.mates);
		sh.nlong = (uint32_t)g.stats[kLaneLong];
		sh.listed = sh.nlong + (mids ? 0u : (uint32_t)nmid);
		sh.max_bases = mids ? kLaneMaxBases : kLaneShortBases;
		sh.own = sh.listed ? 0u : gridDim.x * kLaneWarps;
		sh.warps = (uint32_t)min((uint64_t)kLaneWarps,
				(g.chunks + gridDim.x - 1) / gridDim.x);
		sh.help = sh.listed > 4u * g.chunks;
		sh.go = !a.lane_stats || lane_has(a);
	}
	__syncthreads();
	if (!sh.go)
		return;
	if (warp == 0)
		lane_tables<PACKED>(tab, g.F.k, lane);
	if (MODE == SCORE_HARMONIC && threadIdx.x < kHarmTerms)
		terms[threadIdx.x] = harmonic_term(threadIdx.x);
	__syncthreads();

	/* listed reads, a warp each */
	if (sh.listed && (warp < (int)sh.warps || sh.help)) {
		for (;;) {
			uint32_t it = 0;
			if (lane == 0)
				it = (uint32_t)atomicAdd(g.ctr + 1, 1ull);
			it = __shfl_sync(kFull, it, 0);
			if (it >= sh.listed)
				break;
			const uint32_t r = g.list[it < sh.nlong ? it
			                                        : (uint32_t)(a.n * a.mates) - 1u - (it - sh.nlong)];
			const int d = lane_long_item<MODE, WHAT, COUNT, PACKED>(a, &g.sa, g.F, g.f, tab, r,
					&w.nib[0][0], lane, COUNT ? acc : nullptr);
			if (HITS && lane == 0)
				lane_write(g, r, d);
			__syncwarp();
		}
	}

	/* the others, a lane each */
	const int32_t k = (int32_t)g.F.k;
	const uint64_t pol = lane_policy(g.F.keep != 0);
	if (lane == 0)
		w.first = !sh.listed;
	__syncwarp();
	bool more = warp < (int)sh.warps;
	int qi = 0, qn = 0;         /* queue: next item, items */
	bool active = false;
	bool open = false;          /* both: the decision has not fallen */
	uint32_t pos = 0, run = 0;
	uint64_t F = 0, R = 0;
	LaneEval<MODE> ev;
	LaneScore<MODE> sc;
	for (;;) {
		unsigned idle = __ballot_sync(kFull, !active);
		if (idle == kFull || __popc(idle) >= kLaneRefill) {
			while (idle) {
				if (qi == qn) {
					if (!more)
						break;
					unsigned long long c = (unsigned long long)warp * gridDim.x + blockIdx.x;
					if (lane == 0) {
						if (!w.first)
							c = sh.own + atomicAdd(g.ctr, 1ull);
						w.first = 0;
					}
					c = __shfl_sync(kFull, c, 0);
					more = c < g.chunks;
					if (!more)
						break;
					qn = lane_queue<MODE, WHAT, PACKED>(g, w, c, sh.max_bases, lane);
					qi = 0;
					if (!qn)
						continue;
				}
				const int n = min(__popc(idle), qn - qi);
				const int rank = __popc(idle & ((1u << lane) - 1u));
				if (!active && rank < n) {
					const int q = qi + rank;
					w.my_base[lane] = w.base[q];
					w.my_read[lane] = w.read[q];
					w.my_len[lane] = w.len[q];
#pragma unroll
					for (int j = 0; j < 4; ++j)
						w.nib[j][lane] = 0;
					if (SCORE)
						sc.start();
					if (HITS) {
						ev.start();
						if (WHAT == kLaneBoth)
							open = true;
						w.my_thres[lane] = w.thres[q];
						w.my_anti_thres[lane] = w.anti_thres[q];
						if (MODE == SCORE_HARMONIC)
							w.my_hthres[lane] = w.hthres[q];
					}
					pos = run = 0;
					F = tab.f0;
					R = tab.r0;
					active = true;
				}
				qi += n;
				__syncwarp(); /* items read before the queue is written again */
				idle = __ballot_sync(kFull, !active);
			}
			if (idle == kFull)
				break; /* nothing left */
		}

		/* eight bases: the frames that end at them; rolling table entries
		 * out << 2 | in, one nibble each */
		uint32_t V = 0, pairs = 0;
		if (active) {
			const uint32_t nb = min(8u, w.my_len[lane] - pos);
			const uint32_t mate = w.my_read[lane] >= a.n ? 1u : 0u;
			uint32_t nib, bad;
			lane_bases<PACKED>(a, mate, w.my_base[lane] + pos, nb, nib, bad);
			V = lane_valid(bad, nb, run, g.F.k);
			if (COUNT)
				acc[1] += __popc(V);
			/* the bases k before: nibbles from word q8 back, shifted */
			const uint32_t q8 = (g.F.k + 7u) >> 3, at = pos >> 3;
			const uint32_t lo = w.nib[(at - q8) & 3u][lane];
			const uint32_t hi = q8 == 1u ? nib : w.nib[(at - q8 + 1u) & 3u][lane];
			w.nib[at & 3u][lane] = nib;
			pairs = nib | (__funnelshift_r(lo, hi, 4u * (8u * q8 - g.F.k)) << 2);
			if (HITS) {
				ev.thres = w.my_thres[lane];
				ev.anti_thres = w.my_anti_thres[lane];
				if (MODE == SCORE_HARMONIC)
					ev.hthres = w.my_hthres[lane];
			}
		}
		int decided = EVAL_OPEN;
		int32_t p0 = (int32_t)pos - k + 1;
#pragma unroll 1
		for (int s = 0; s < 8 / kLaneSub; ++s, p0 += kLaneSub) {
			constexpr uint32_t kMask = (1u << kLaneSub) - 1u;
			const uint32_t Vs = !SCORE && decided ? 0u : V & kMask;
			V >>= kLaneSub;
			uint64_t canon[kLaneSub];
#pragma unroll
			for (int j = 0; j < kLaneSub; ++j) {
				const uint32_t e = (pairs >> (4 * j)) & 15u;
				F = rol1(F) ^ tab.fw[e];
				R = ror1(R) ^ tab.rc[e];
				canon[j] = F < R ? F : R;
			}
			pairs = kLaneSub == 8 ? 0u : pairs >> ((4 * kLaneSub) & 31);
			/* frames to probe: not below the skip window's end, not masked */
			const int32_t sk = (MODE == SCORE_LENGTH ? 0 : SCORE ? sc.skip_end : ev.skip_end) - p0;
			uint32_t live = sk <= 0 ? Vs : sk >= kLaneSub ? 0u : Vs & (kMask << sk);
			if (a.dust[0] && live) {
				const uint32_t mate = w.my_read[lane] >= a.n ? 1u : 0u;
#pragma unroll
				for (int j = 0; j < kLaneSub; ++j)
					if (((live >> j) & 1u) && dust_low(a.dust[mate],
							w.my_base[lane] + (uint64_t)(int64_t)(p0 + j)))
						live &= ~(1u << j);
			}
			uint32_t cost[COUNT ? kLaneSub : 1];
			live = lane_levels<COUNT, kLaneSub>(g.F, canon, live, pol, cost);
			if (SCORE && Vs)
				sc.template step<kLaneSub>(Vs, live, p0, k, (int32_t)a.streak_thr, terms);
			if (HITS && Vs && (WHAT != kLaneBoth || open)) {
				uint32_t vis = 0;
				decided = ev.template step<kLaneSub>(Vs, live, p0, k, (int32_t)a.streak_thr,
						terms, COUNT ? &vis : nullptr);
				if (COUNT)
					for (int j = 0; j < kLaneSub; ++j) {
						acc[0] += cost[j];
						acc[2] += ((vis >> j) & 1u) ? cost[j] : 0u;
					}
			}
		}
		pos += 8u;
		const bool done = active && ((!SCORE && decided != EVAL_OPEN) || pos >= w.my_len[lane]);
		if (SCORE) {
			const uint32_t read = w.my_read[lane], len = w.my_len[lane];
			const uint32_t mate = read >= a.n ? 1u : 0u;
			double *out = done ? g.sa.scores[mate] + (read - (mate ? a.n : 0)) * a.nf + g.f : nullptr;
			ScoreState st;
			sc.result(st);
			if (MODE == SCORE_BINOMIAL) {
				/* the binomial tail is summed by the warp, one read after another */
				for (unsigned m = __ballot_sync(kFull, done); m; m &= m - 1u) {
					const int l = __ffs(m) - 1;
					const uint32_t hits = __shfl_sync(kFull, (uint32_t)st.score, l);
					const uint32_t ln = __shfl_sync(kFull, len, l);
					const double v = binomial_score(ln, g.F.k, hits, g.sa.fpr[g.f], lane);
					if (lane == l)
						*out = v;
				}
			} else if (done) {
				*out = score_value<MODE>(st, len, g.F.k, 0.0, lane);
			}
		}
		/* both: the decision when it falls, or with the score */
		if (HITS && (WHAT == kLaneBoth ? active && open && (decided != EVAL_OPEN || done) : done)) {
			lane_write(g, w.my_read[lane], decided);
			open = false;
		}
		active = active && !done;
	}
	lane_count<COUNT>(a, acc, lane);
}

template <int MODE, int WHAT, bool COUNT>
cudaError_t launch_mode(const LaneArgs &g, int num_sms, cudaStream_t s)
{
	auto kern = g.a.packed ? lane_kernel<MODE, WHAT, COUNT, true>
	                       : lane_kernel<MODE, WHAT, COUNT, false>;
	int per_sm = 0;
	cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kLaneWarps * 32, 0);
	/* no more shared memory carved out than the blocks use: the rest is L1, which
	 * holds the reads' bases and the probes on their way (8.65 -> 8.26 ms on the
	 * ten 68 MB filters) */
	cudaFuncAttributes at;
	if (e == cudaSuccess)
		e = cudaFuncGetAttributes(&at, kern);
	if (e == cudaSuccess)
		e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
				(int)std::min<size_t>(100, (per_sm * (at.sharedSizeBytes + 1024) * 100 +
				(228 << 10) - 1) / (228 << 10)));
	if (e != cudaSuccess)
		return e;
	const uint64_t need = (g.a.n * g.a.mates + kLaneWarps - 1) / kLaneWarps;
	const uint64_t full = (uint64_t)std::max(per_sm, 1) * num_sms;
	kern<<<(unsigned)std::min(need, full), kLaneWarps * 32, 0, s>>>(g);
	return cudaGetLastError();
}

template <int WHAT, bool COUNT>
cudaError_t launch_lane_as(const LaneArgs &g, int num_sms, cudaStream_t s)
{
	switch (g.a.scoring) {
	case BBT_SCORE_LENGTH: return launch_mode<SCORE_LENGTH, WHAT, COUNT>(g, num_sms, s);
	case BBT_SCORE_HARMONIC: return launch_mode<SCORE_HARMONIC, WHAT, COUNT>(g, num_sms, s);
	case BBT_SCORE_BINOMIAL: return launch_mode<SCORE_BINOMIAL, WHAT, COUNT>(g, num_sms, s);
	default: return launch_mode<SCORE_SIMPLE, WHAT, COUNT>(g, num_sms, s);
	}
}

} // namespace

bool lane_supports(const FilterDev *hf, uint32_t nf, uint32_t streak_thr, uint64_t total_reads)
{
	if (streak_thr < 1 || streak_thr > 0x7fffffffu || total_reads >= (1ull << 32))
		return false;
	for (uint32_t i = 0; i < nf; ++i)
		if (hf[i].k > 32 || (hf[i].m >> 5) >= (1ull << 30))
			return false;
	return true;
}

/* Where the lane kernel is the faster one for every mixture of lengths, and where that
 * depends on them.  A launch lasts as long as its longest read's lane (95 us for 150
 * bases over a filter in L2, 154 over one in HBM, for any batch of up to some 28,000
 * reads), the other kernels' time grows with the bases; ragged reads below are 50 to 300
 * bases, log-uniform.
 *
 * Measured with SIMPLE scoring at 0.15, three hashes and k = 25 unless said otherwise.
 *
 * - one filter in L2: from 20,000 reads on where these are short and of much the same
 *   length (20,000 / 28,000 / 40,000 reads, 3.4 MB: 150 bases 95 / 93 / 106 us against
 *   115 / 135 / 166, 300 bases 145 / 151 / 172 against 144 / 173 / 217, 600 bases 258 /
 *   260 / 300 against 206 / 254 / 327, ragged 154 / 153 / 171 against 119 / 139 / 176),
 *   from 40,000 on always, with more than four hashes from 60,000 (six, 40,000 reads: 600
 *   bases 448 against 397, ragged 218 against 200); scores, every frame of which is walked,
 *   from 20,000, or 28,000 (20,000 ragged reads, six hashes: 232 against 183).  With LENGTH
 *   scoring, whose windows are short, only without long reads (60,000 ragged reads with
 *   them 890 against 771).
 * - two to four that fit L2 together: the filter-major passes hash a read once for all of
 *   them.  Four of 3.4 MB, 28,000 / 50,000 reads: 150 bases 270 / 326 us against 297 /
 *   466, 600 bases 914 / 1110 against 946 / 1608; 28,000 / 100,000 ragged ones 501 / 874
 *   against 334 / 805.  Scores of ragged reads 522 against 448 at 28,000, 571 against 577
 *   at 40,000.  The filter-major path asks from 40,000 reads on, where the answer costs less
 *   than it brings (28,000 of 150 bases 321 against 302).
 * - more that fit L2 together: likewise, and a launch's latency for each.  Ten of 3.4 MB
 *   meet at 50,000 reads (150 bases 751 against 872, 300 bases 1423 against 1634), thirty
 *   at 75,000 (80,000: 3007 against 3478); scores at 20,000 (150 bases 611 against 639) and
 *   42,000 (50,000 of 50 bases: 816 against 1014).  100,000 ragged reads over ten 2149
 *   against 1626, and one long read would make every launch wait.
 * - filters that each fit L2 but not together: the passes miss L2 as well.  Ten of 68 MB,
 *   from 28,000 reads on (50 bases 354 us against 400, 150 bases 852 against 1195, 1,000
 *   bases 4765 against 7503; 20,000 of 50 bases 336 against 288), ragged ones from 60,000
 *   (28,000 / 40,000: 1442 / 1575 against 1162 / 1404).  Scores of reads of which 5 % have
 *   300 to 10,000 bases: 28,000 5204 us against 4976, 40,000 5378 against 5780.
 * - one filter in HBM: a lane waits longer for its probes.  28,000 / 80,000 / 160,000 reads,
 *   2.1 GB: 100 bases 116 / 216 / 331 us against 144 / 281 / 508, 150 bases 154 / 305 / 487
 *   against 164 / 339 / 616, 300 bases 265 / 569 / 940 against 240 / 535 / 996; 40,000 /
 *   60,000 ragged ones 248 / 305 against 205 / 275; threshold 0.8, 100,000 of 150 bases 567
 *   against 518.  Scores: 100 bases 185 / 437 / 653
 *   against 210 / 456 / 841, 150 bases 266 / 691 / 1053 against 286 / 655 / 1211, 300 bases
 *   515 / 1437 / 2190 against 501 / 1234 / 2375.
 * - several, one or more of them in HBM: the read-major kernel's probes of all filters
 *   overlap.  3.4 MB and 2.1 GB, 28,000 / 40,000 ragged reads 334 / 383 us against 249 /
 *   315, scores of 50,000 / 160,000 reads of 150 bases 543 / 1310 against 490 / 1406.
 * - several filters and early decisions: the passes and the read-major kernel stop at
 *   them for all filters at once.  Four of 3.4 MB, threshold 0.8: 28,000 reads of 300 bases
 *   529 us against 388; LENGTH, 100,000 ragged reads with long ones 4740 against 2422, best
 *   hits of 20,000 of 150 bases over ten 606 against 419.  HARMONIC scoring of long reads:
 *   100,000 ragged ones, best hits over four 9364 against 6559. */
LaneRule lane_rule(const FilterDev *hf, uint32_t nf, const LaneAim &aim, uint64_t reads)
{
	const uint64_t always = ~0ull;
	const uint32_t none = ~0u, any = 0, free = ~0u;
	const bool scores = aim.scores;
	uint64_t bytes = 0, most = 0;
	uint32_t h = 0;
	for (uint32_t i = 0; i < nf; ++i) {
		bytes += hf[i].m / 8;
		most = std::max(most, hf[i].m / 8);
		h = std::max(h, hf[i].h);
	}
	if (nf > 1 && aim.quick)
		return {most > kLaneKeepBytes ? 160000u : 150000u, always, 64, none, free, true};
	if (most > kLaneKeepBytes && nf > 1)
		return {160000, always, 8, aim.harmonic ? none : 8, free, false};
	if (most > kLaneKeepBytes)
		return {28000, aim.length ? always : 160000, 8, any, 130, true};
	if (nf == 1 && scores)
		return {aim.length ? 28000u : 20000u, h > 4 || aim.length ? 28000u : 20000u, any, any, free,
				true};
	if (nf == 1) {
		const uint32_t sure = h > 4 || aim.length ? 60000 : 40000;
		const bool few = reads < sure;
		return {20000, aim.length ? always : sure, few ? 8 : any, aim.length ? none : any,
				reads < 28000 ? 170u : few ? 250u : free, few};
	}
	if (bytes > kLaneKeepBytes && aim.harmonic)
		return {28000, always, 64, none, free, true};
	if (bytes > kLaneKeepBytes)
		return {28000, 60000, any, scores && reads < 40000 ? 64 : any, free, true};
	if (nf <= 4)
		return {aim.host ? 40000u : 20000u, aim.harmonic ? always : scores ? 40000u : 150000u,
				aim.harmonic ? 64u : reads < 40000 ? 8u : any, aim.harmonic ? none : any,
				reads < 28000 ? 120u : free, true};
	if (scores)
		return {nf <= 10 ? (aim.host ? 28000 : 20000) : std::max<uint64_t>(28000, 1400ull * nf),
				always, 64, none, free, true};
	return {std::max<uint64_t>(std::min<uint64_t>(60000, 5000ull * nf), 2500ull * nf), always, 64,
			none, free, true};
}

cudaError_t launch_lane_list(const ClassifyArgs &a, const LaneScratch &ls, int num_sms,
		cudaStream_t s)
{
	const uint64_t total = a.n * a.mates;
	cudaError_t e = cudaMemsetAsync(ls.ctr, 0, kLaneStats * sizeof(unsigned long long), s);
	if (e != cudaSuccess || total == 0)
		return e;
	const uint64_t need = (total + 255) / 256;
	lane_list_kernel<<<(unsigned)std::min<uint64_t>(need, (uint64_t)num_sms * 8), 256, 0, s>>>(a,
			ls.list, ls.ctr);
	return cudaGetLastError();
}

cudaError_t launch_lane(const ClassifyArgs &a, const FilterDev *hf, const ScoreArgs *sa,
		bool hits, const LaneScratch &ls, int num_sms, bool count, cudaStream_t s)
{
	const uint64_t total = a.n * a.mates;
	if (total == 0)
		return cudaSuccess;
	LaneArgs g;
	g.ctr = ls.ctr + kLaneStats;
	cudaError_t e = cudaMemsetAsync(g.ctr, 0, 2 * (size_t)a.nf * sizeof(unsigned long long), s);
	if (e != cudaSuccess)
		return e;
	g.a = a;
	g.sa = sa ? *sa : ScoreArgs();
	g.list = ls.list;
	g.stats = ls.ctr;
	g.chunks = (total + 31) / 32;
	for (g.f = 0; g.f < a.nf; ++g.f, g.ctr += 2) {
		g.F = lane_filter(hf[g.f]);
		e = sa ? (hits ? launch_lane_as<kLaneBoth, false>(g, num_sms, s)
		               : launch_lane_as<kLaneScores, false>(g, num_sms, s))
		  : count ? launch_lane_as<kLaneHits, true>(g, num_sms, s)
		          : launch_lane_as<kLaneHits, false>(g, num_sms, s);
		if (e != cudaSuccess)
			return e;
	}
	return cudaSuccess;
}

} // namespace bbt
