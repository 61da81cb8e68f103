/*
 * lane_walk.cuh -- the SeqEval walks of one read by one thread, a few frames
 * at a time (the lane kernel, lane.cu).  Compiled for the device and for the
 * host, where tests run them against the CPU oracle.
 *
 * A step takes up to 8 consecutive frames: bit j of V is set when frame p0 + j
 * exists and holds only ACGT, bit j of H when it was probed and is in the
 * filter.  Frames are visited in order exactly as the reference's loops visit
 * them (Common/SeqEval.h:37-114, 116-193, 218-290, 295-332 for the decisions,
 * 334-491 for the scores), so a frame that a skip window opened inside the
 * step covers may have been probed in vain, and its H bit is not read.
 * Frames below LaneEval::skip_end are not probed at all.
 *
 * streak_thr is at least 1 (with 0 every miss opens a window; those runs take
 * the warp kernels).  Reads are short enough for 32-bit counters.
 */
#ifndef BBT_LANE_WALK_CUH
#define BBT_LANE_WALK_CUH

#include "seqeval_chunk.cuh"

namespace bbt {

/* HARMONIC: what the hit after s earlier hits of its streak adds, 0.5 for
 * s = 0 and 1 - 1/(1 + s) for s < kHarmTerms, from a table of harmonic_add's
 * own values (the same IEEE operations), so that a hit costs one addition. */
constexpr int kHarmTerms = 64;
BBT_HD double harmonic_term(uint32_t s)
{
	return harmonic_add(0.0, s); /* 0.0 + t is t */
}

BBT_HD double lane_harmonic(double score, uint32_t streak, const double *terms)
{
	if (streak >= kHarmTerms)
		return harmonic_add(score, streak);
#if defined(__CUDA_ARCH__)
	return __dadd_rn(score, terms[streak]);
#else
	return score + terms[streak];
#endif
}

/* Bit v mod m of a filter of m = 32 m5 bits, m5 < 2^30: the index of its 32-bit
 * word, (v >> 5) mod m5 (the bit is v & 31 of it).  u = v >> 5 < 2^59 and
 * inv = floor((2^64 - 1) / m5), so floor(u inv / 2^64) is u / m5 rounded down or
 * one less, and the remainder one subtraction away: a subtract and an unsigned
 * minimum.  32-bit operations on the low word, where reduce() takes the 64-bit
 * product, compare and select; the four multiplications go to another pipe than
 * the shifts and logic that bound the kernel.  m5 is at least 2: no partial sum
 * below leaves 64 bits. */
BBT_HD uint32_t lane_word(uint64_t v, uint32_t m5, uint32_t inv_hi, uint32_t inv_lo)
{
	const uint32_t ul = (uint32_t)(v >> 5), uh = (uint32_t)(v >> 37);
#if defined(__CUDA_ARCH__)
	const uint32_t low = __umulhi(ul, inv_lo);
#else
	const uint32_t low = (uint32_t)(((uint64_t)ul * inv_lo) >> 32);
#endif
	const uint64_t t = (uint64_t)ul * inv_hi + low + (uint64_t)uh * inv_lo;
	const uint32_t q = uh * inv_hi + (uint32_t)(t >> 32);
	const uint32_t r = ul - q * m5;
#if defined(__CUDA_ARCH__)
	return min(r, r - m5);
#else
	return r < r - m5 ? r : r - m5;
#endif
}

/* The frames that end at the next nb (at most 8) bases of a read and hold only
 * ACGT: bit j of `bad` is set when base j is not ACGT, `run` counts the valid
 * bases up to here and moves on. */
BBT_HD uint32_t lane_valid(uint32_t bad, uint32_t nb, uint32_t &run, uint32_t k)
{
	const uint32_t in = low_mask((int)nb);
	bad &= in;
	uint32_t V = 0;
	if (!bad) {
		const uint32_t need = run + 1u >= k ? 0u : k - 1u - run;
		V = need >= 8u ? 0u : 0xFFu << need;
		run += 8u;
	} else {
#pragma unroll
		for (int j = 0; j < 8; ++j) {
			run = ((bad >> j) & 1u) ? 0u : run + 1u;
			V |= (run >= k ? 1u : 0u) << j;
		}
	}
	return V & in;
}

/*
 * The frames of a step by masks instead of one by one, for the usual step: its
 * valid frames follow the last visited one without a gap (frame 0 of the masks
 * is prev + 1), and streak_thr is at most 15.  A window that opens inside the
 * step covers the rest of it (k >= N), so every frame but the hits before it
 * adds one to the misses, whether probed, in a window or the trigger.
 */
struct LaneMasks {
	uint32_t hits;   /* hits that count */
	uint32_t again;  /* those that continue a streak */
	int32_t n;       /* frames */
	int32_t streak, skip_end; /* after the step */
};

template <int N>
BBT_HD bool lane_masks(LaneMasks &o, uint32_t V, uint32_t H, int32_t p0, int32_t prev,
		int32_t streak, int32_t skip_end, int32_t k, int32_t streak_thr)
{
	const int32_t n0 = prev + 1 - p0;
	if ((uint32_t)n0 >= (uint32_t)N || streak_thr > 15 || k < N)
		return false;
	const uint32_t U = V >> n0;
	if (!(U & 1u) || (U & (U + 1u)) || (U << n0) != V)
		return false;
	const int32_t sk = skip_end - (prev + 1);
	const uint32_t W = sk <= 0 ? 0u : sk >= N ? U : U & ((1u << sk) - 1u);
	const uint32_t h = (H >> n0) & U & ~W;
	const uint32_t miss = U & ~W & ~h;
	/* bits 16 up: this step; below: the streak that reaches it */
	const uint32_t st = streak > 15 ? 15u : (uint32_t)streak;
	const uint32_t x = (h << 16) | (0xFFFFu & ~(0xFFFFu >> st));
	uint32_t run = x << 1;
	for (int32_t q = 2; q <= streak_thr; ++q)
		run &= x << q;
	const uint32_t trig = miss & (run >> 16);
	const uint32_t below = (trig & (0u - trig)) - 1u; /* all ones without a trigger */
	o.hits = h & below;
	o.again = o.hits & ((h << 1) | (streak > 0 ? 1u : 0u));
	o.n = popc32(U);
	o.skip_end = skip_end;
	if (trig) {
		o.streak = 0;
		o.skip_end = prev + 1 + popc32(below) + k;
	} else {
		o.streak = miss ? o.n - 1 - highbit32(miss) : streak + o.n - popc32(W);
	}
	return true;
}

/* The decision walk of one (read, filter). */
template <int MODE>
struct LaneEval {
	int32_t score;      /* SIMPLE half units, BINOMIAL 2 per hit, LENGTH current match */
	int32_t thres;      /* accept when score >= thres after a hit */
	int32_t anti;
	int32_t anti_thres; /* reject when anti >= anti_thres after it grew (LENGTH: bases) */
	int32_t streak;
	int32_t skip_end;   /* frames below this belong to a skip window */
	int32_t prev;       /* last visited frame, -1 before the first */
	double hscore, hthres;

	BBT_HD void start()
	{
		score = anti = streak = skip_end = 0;
		prev = -1;
		hscore = 0.0;
	}

	/* EVAL_* after the frames; vis (optional): the frames the reference probes. */
	template <int N>
	BBT_HD int step(uint32_t V, uint32_t H, int32_t p0, int32_t k, int32_t streak_thr,
			const double *terms, uint32_t *vis = nullptr)
	{
		int d = EVAL_OPEN;
		if (MODE == SCORE_LENGTH) {
#pragma unroll
			for (int j = 0; j < N; ++j) {
				if (d == EVAL_OPEN && ((V >> j) & 1u)) {
					const int32_t p = p0 + j;
					if (anti_thres - p + score < thres) {
						d = EVAL_REJECT;
					} else {
						if (vis)
							*vis |= 1u << j;
						const int32_t m = p == prev + 1 ? score : 0;
						score = ((H >> j) & 1u) ? (m == 0 ? k : m + 1) : 0;
						prev = p;
						if (score >= thres)
							d = EVAL_ACCEPT;
					}
				}
			}
			return d;
		}
		if (prev < 0 && V)
			prev = p0 + lowbit32(V) - 1; /* leading frames that are not valid count nothing */
		LaneMasks m;
		if (MODE != SCORE_HARMONIC && !vis &&
				lane_masks<N>(m, V, H, p0, prev, streak, skip_end, k, streak_thr)) {
			const int32_t nh = popc32(m.hits);
			const int32_t sc = score + nh + (MODE == SCORE_BINOMIAL ? nh : popc32(m.again));
			const int32_t an = anti + m.n - nh;
			const bool acc = nh && sc >= thres, rej = m.n > nh && an >= anti_thres;
			if (!(acc && rej)) { /* both: which comes first, below */
				score = sc;
				anti = an;
				streak = m.streak;
				skip_end = m.skip_end;
				prev += m.n;
				return acc ? EVAL_ACCEPT : rej ? EVAL_REJECT : EVAL_OPEN;
			}
		}
#pragma unroll
		for (int j = 0; j < N; ++j) {
			if (d == EVAL_OPEN && ((V >> j) & 1u)) {
				const int32_t p = p0 + j;
				bool more = false; /* anti grew */
				if (p < skip_end) {
					++anti;
					more = true;
				} else {
					const int32_t gap = p - prev - 1;
					if (gap) {
						anti += gap;
						streak = 0;
						more = true;
					}
					if (!(more && anti >= anti_thres)) {
						if (vis)
							*vis |= 1u << j;
						if ((H >> j) & 1u) {
							if (MODE == SCORE_HARMONIC) {
								hscore = lane_harmonic(hscore, (uint32_t)streak, terms);
								if (hthres <= hscore)
									d = EVAL_ACCEPT;
							} else {
								score += (MODE == SCORE_BINOMIAL || streak) ? 2 : 1;
								if (score >= thres)
									d = EVAL_ACCEPT;
							}
							++streak;
						} else {
							if (streak >= streak_thr)
								skip_end = p + k;
							streak = 0;
							++anti;
							more = true;
						}
					}
				}
				prev = p;
				if (more && anti >= anti_thres && d == EVAL_OPEN)
					d = EVAL_REJECT;
			}
		}
		return d;
	}
};

/* Thresholds of a read of `frames` frames (len bases): those of simple_init,
 * harmonic_init, binomial_simple_init (bthres: the read's accept count) and
 * length_init. */
template <int MODE>
BBT_HD void lane_thresholds(int32_t &thres, int32_t &anti_thres, double &hthres, double score,
		double one_minus, uint32_t min_len, uint32_t bthres, uint32_t frames, uint32_t len)
{
	hthres = 0.0;
	if (MODE == SCORE_LENGTH) {
		thres = min_len > 0x3fffffffu ? 0x3fffffff : (int32_t)min_len;
		anti_thres = (int32_t)len;
	} else if (MODE == SCORE_HARMONIC) {
		SeqState s;
		harmonic_init(s, score, one_minus, frames);
		hthres = s.thres;
		thres = 0;
		anti_thres = (int32_t)s.anti_thres; /* floor of at most frames */
	} else {
		SimpleState s;
		if (MODE == SCORE_BINOMIAL)
			binomial_simple_init(s, bthres, frames);
		else
			simple_init(s, score, one_minus, frames);
		thres = s.thres2;
		anti_thres = s.anti_thres;
	}
}

/* The exhaustive walk of one (read, filter): SeqEval::evalScore's loops. */
template <int MODE>
struct LaneScore {
	int32_t score;    /* SIMPLE half units, BINOMIAL hits, LENGTH run */
	int32_t streak;
	int32_t skip_end; /* frames below this are visited without a probe */
	int32_t prev;
	double hscore;

	BBT_HD void start()
	{
		score = streak = skip_end = 0;
		prev = -1; /* any value: there is no streak to break yet */
		hscore = 0.0;
	}

	template <int N>
	BBT_HD void step(uint32_t V, uint32_t H, int32_t p0, int32_t k, int32_t streak_thr,
			const double *terms)
	{
		LaneMasks m;
		if ((MODE == SCORE_SIMPLE || MODE == SCORE_BINOMIAL) &&
				lane_masks<N>(m, V, H, p0, prev, streak, skip_end, k, streak_thr)) {
			score += popc32(m.hits) + (MODE == SCORE_SIMPLE ? popc32(m.again) : 0);
			streak = m.streak;
			skip_end = m.skip_end;
			prev += m.n;
			return;
		}
#pragma unroll
		for (int j = 0; j < N; ++j) {
			if ((V >> j) & 1u) {
				const int32_t p = p0 + j;
				const bool hit = (H >> j) & 1u;
				if (MODE == SCORE_LENGTH) {
					const int32_t m = p == prev + 1 ? score : 0;
					score = hit ? (m == 0 ? k : m + 1) : 0;
				} else if (p >= skip_end) {
					if (p != prev + 1)
						streak = 0;
					if (hit) {
						if (MODE == SCORE_HARMONIC)
							hscore = lane_harmonic(hscore, (uint32_t)streak, terms);
						else
							score += MODE == SCORE_BINOMIAL ? 1 : (streak ? 2 : 1);
						++streak;
					} else {
						if (streak >= streak_thr)
							skip_end = p + k;
						streak = 0;
					}
				}
				prev = p;
			}
		}
	}

	/* The walk's state as score_value (score_value.cuh) takes it. */
	BBT_HD void result(ScoreState &s) const
	{
		score_init(s);
		s.run = (uint32_t)score;
		s.score = MODE == SCORE_HARMONIC ? hscore
		        : MODE == SCORE_SIMPLE ? 0.5 * (double)score : (double)score;
	}
};

} // namespace bbt

#endif
