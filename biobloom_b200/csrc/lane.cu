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
 * lanes as these finish.  Reads above LaneArgs::max_bases would leave a lane working
 * long after its warp and are evaluated by whole warps, before the others: a
 * small kernel lists them.
 */
#include "lane.cuh"

#include <algorithm>

#include "bbt.h"
#include "lane_item.cuh"

namespace bbt {

namespace {

constexpr int kLaneWarps = 8;     /* warps per block */
/* Blocks per SM the registers leave room for: 3 give a thread 80, which hold
 * eight frames' hashes and words in flight without spills (4 blocks spill, and
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
	const unsigned long long *nlong;
	unsigned long long *ctr;    /* next chunk, next long read */
	uint64_t chunks;
	uint32_t f;                 /* the filter's index */
	LaneFilter F;
	uint32_t max_bases;         /* of a lane's read */
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
	double hthres[MODE == SCORE_HARMONIC ? 32 : 1], my_hthres[MODE == SCORE_HARMONIC ? 32 : 1];
};

/* Indexes of the reads above max_bases. */
__global__ void lane_long_kernel(ClassifyArgs a, uint32_t max_bases, uint32_t *list,
		unsigned long long *nlong)
{
	const uint64_t total = a.n * a.mates;
	const int lane = threadIdx.x & 31;
	const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
	for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < total; base += stride) {
		const uint64_t r = base + threadIdx.x;
		bool is_long = false;
		if (r < total) {
			const uint32_t mate = r >= a.n ? 1u : 0u;
			const uint64_t i = r - (mate ? a.n : 0);
			is_long = a.off[mate][i + 1] - a.off[mate][i] > max_bases;
		}
		const unsigned m = __ballot_sync(kFull, is_long);
		if (m) {
			unsigned long long b = 0;
			if (lane == 0)
				b = atomicAdd(nlong, (unsigned long long)__popc(m));
			b = __shfl_sync(kFull, b, 0);
			if (is_long)
				list[b + __popc(m & ((1u << lane) - 1u))] = (uint32_t)r;
		}
	}
}

/* Items of chunk c, reads [32c, 32c + 32), into the warp's queue: those long
 * enough for a frame and not on the long list; the result of a read without
 * frames is written here.  Returns their number. */
template <int MODE, int WHAT, bool PACKED>
__device__ __forceinline__ int lane_queue(const LaneArgs &g, LaneWarp<MODE> &w, uint64_t c, int lane)
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
	const bool mine = in && l >= g.F.k && l <= g.max_bases;
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
	__shared__ double terms[MODE == SCORE_HARMONIC ? kHarmTerms : 1];
	const ClassifyArgs &a = g.a;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	LaneWarp<MODE> &w = warps[warp];
	unsigned long long acc[3] = {0, 0, 0}; /* words read, frames hashed, words of the
	                                          sequential algorithm */
	if (warp == 0)
		lane_tables<PACKED>(tab, g.F.k, lane);
	if (MODE == SCORE_HARMONIC && threadIdx.x < kHarmTerms)
		terms[threadIdx.x] = harmonic_term(threadIdx.x);
	__syncthreads();

	/* long reads, a warp each */
	const unsigned long long nlong = *g.nlong;
	if (nlong) {
		for (;;) {
			unsigned long long it = 0;
			if (lane == 0)
				it = atomicAdd(g.ctr + 1, 1ull);
			it = __shfl_sync(kFull, it, 0);
			if (it >= nlong)
				break;
			const uint32_t r = g.list[it];
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
	bool more = true;
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
					unsigned long long c = 0;
					if (lane == 0)
						c = atomicAdd(g.ctr, 1ull);
					c = __shfl_sync(kFull, c, 0);
					more = c < g.chunks;
					if (!more)
						break;
					qn = lane_queue<MODE, WHAT, PACKED>(g, w, c, lane);
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
	const uint64_t need = (g.chunks + kLaneWarps - 1) / kLaneWarps;
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

/* Whether a filter of the call fits L2. */
static bool lane_in_l2(const FilterDev *hf, uint32_t nf)
{
	for (uint32_t i = 0; i < nf; ++i)
		if (hf[i].m / 8 <= kLaneKeepBytes)
			return true;
	return false;
}

/* A lane's read takes its time (82 us for 150 bases over a filter in L2, 115-138 us
 * over one in HBM, the same for any batch of up to 37,888 reads); the other kernels'
 * time grows with the batch and reaches that at about 20k reads in L2 (82 us) and 28k
 * in HBM (122 us per 24k, 151 per 32k).  So it does with a few filters (four: 267
 * against 270 us at 20k) and with many that do not fit L2 together (ten of 68 MB: 927
 * against 836 at 20k).  Many that do fit are another matter: the filter-major passes
 * hash a read once for all of them and find them all in L2, the lane kernel pays a
 * launch's latency for each.  Ten of 3.4 MB meet at 50k reads (852 against 867 us;
 * 20k: 433 against 637), thirty at 60k (2584 against 2575; 20k: 954 against 1865).
 * Scores are walked per filter either way: ten meet at 20k (621 against 634), thirty
 * at 28k (1852 against 1857; 20k: 1410 against 1843). */
bool lane_pays(const FilterDev *hf, uint32_t nf, uint64_t total_reads, bool scores)
{
	if (!lane_in_l2(hf, nf))
		return total_reads >= 28000;
	uint64_t bytes = 0;
	for (uint32_t i = 0; i < nf; ++i)
		bytes += hf[i].m / 8;
	if (nf <= 4 || bytes > kLaneKeepBytes)
		return total_reads >= 20000;
	if (scores)
		return total_reads >= (nf <= 10 ? 20000u : 28000u);
	return total_reads >= std::min<uint64_t>(60000, 5000ull * nf);
}

cudaError_t launch_lane(const ClassifyArgs &a, const FilterDev *hf, const ScoreArgs *sa,
		bool hits, const LaneScratch &ls, int num_sms, bool count, cudaStream_t s)
{
	const uint64_t total = a.n * a.mates;
	if (total == 0)
		return cudaSuccess;
	cudaError_t e = cudaMemsetAsync(ls.ctr, 0, lane_counters(a.nf) * sizeof(unsigned long long), s);
	if (e != cudaSuccess)
		return e;
	LaneArgs g;
	g.max_bases = lane_in_l2(hf, a.nf) ? kLaneMaxBases : kLaneMaxBasesHbm;
	const uint64_t need = (total + 255) / 256;
	lane_long_kernel<<<(unsigned)std::min<uint64_t>(need, (uint64_t)num_sms * 8), 256, 0, s>>>(a,
			g.max_bases, ls.list, ls.ctr);
	if ((e = cudaGetLastError()) != cudaSuccess)
		return e;
	g.a = a;
	g.sa = sa ? *sa : ScoreArgs();
	g.list = ls.list;
	g.nlong = ls.ctr;
	g.chunks = (total + 31) / 32;
	g.ctr = ls.ctr + 1;
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
