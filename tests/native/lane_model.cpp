/*
 * lane_model.cpp -- host build of the lane kernel's walks
 * (biobloom_b200/csrc/lane_walk.cuh): a read eight bases at a time, its frames
 * in steps of N, fed with the oracle's per-frame hit bits.  Frames below a
 * skip window that opens inside a step carry their true hit bit, as the kernel
 * probes them, and must not count.
 */
#include "lane_walk.cuh"
#include "bbt_oracle.h"
#include <vector>

using namespace bbt;

struct Frames {
	std::vector<uint8_t> valid, hit;
	std::vector<uint32_t> cost;
	Frames(const char *seq, uint64_t len, const oracle_bf *bf)
	    : valid(len + 8), hit(len + 8), cost(len + 8)
	{
		oracle_ntitr it;
		for (oracle_ntitr_init(&it, seq, len, bf->h, bf->k); !oracle_ntitr_end(&it);
				oracle_ntitr_next(&it)) {
			uint64_t c = 0;
			valid[it.pos] = 1;
			hit[it.pos] = (uint8_t)oracle_bf_contains(bf, it.hv, &c);
			cost[it.pos] = (uint32_t)c;
		}
	}
};

static uint32_t bad_bases(const char *seq, uint64_t len, uint64_t pos)
{
	uint32_t bad = 0;
	for (int j = 0; j < 8; ++j) {
		/* bytes past the read are somebody else's */
		const char c = pos + j < len ? (char)(seq[pos + j] & 0xDF) : 'N';
		if (c != 'A' && c != 'C' && c != 'G' && c != 'T')
			bad |= 1u << j;
	}
	return bad;
}

/* Decision (1 accept) and probes of the sequential algorithm; -1 when the
 * validity of a frame differs from the oracle's. */
template <int MODE, int N>
static int eval_as(const char *seq, uint64_t len, const oracle_bf *bf, double threshold,
		unsigned streak_thr, uint32_t bthres, uint64_t *alg, bool count)
{
	const int k = (int)bf->k;
	if (len < (uint64_t)k)
		return 0;
	const Frames fr(seq, len, bf);
	double terms[kHarmTerms];
	for (int i = 0; i < kHarmTerms; ++i)
		terms[i] = harmonic_term(i);
	LaneEval<MODE> ev;
	ev.start();
	lane_thresholds<MODE>(ev.thres, ev.anti_thres, ev.hthres, threshold, 1.0 - threshold,
			(uint32_t)(threshold + 0.5), bthres, (uint32_t)(len - k + 1), (uint32_t)len);
	uint32_t run = 0;
	for (uint64_t pos = 0; pos < len; pos += 8) {
		const uint32_t V = lane_valid(bad_bases(seq, len, pos),
				(uint32_t)(len - pos < 8 ? len - pos : 8), run, k);
		for (int s = 0; s < 8; s += N) {
			const int32_t p0 = (int32_t)pos + s - k + 1;
			uint32_t Vs = (V >> s) & ((1u << N) - 1u), H = 0;
			for (int j = 0; j < N; ++j) {
				const int32_t p = p0 + j;
				if (((Vs >> j) & 1u) != (uint32_t)(p >= 0 && fr.valid[p]))
					return -1;
				if (((Vs >> j) & 1u) && p >= ev.skip_end && fr.hit[p])
					H |= 1u << j;
			}
			if (!Vs)
				continue;
			uint32_t vis = 0;
			const int d = ev.template step<N>(Vs, H, p0, k, (int32_t)streak_thr, terms,
					count ? &vis : nullptr);
			for (int j = 0; j < N; ++j)
				if ((vis >> j) & 1u)
					*alg += fr.cost[p0 + j];
			if (d)
				return d == EVAL_ACCEPT;
		}
	}
	return 0;
}

/* Frame by frame with the probes counted, and by masks where the step allows:
 * the same decision (-2 when not). */
template <int MODE, int N>
static int eval(const char *seq, uint64_t len, const oracle_bf *bf, double threshold,
		unsigned streak_thr, uint32_t bthres, uint64_t *alg)
{
	const int d = eval_as<MODE, N>(seq, len, bf, threshold, streak_thr, bthres, alg, true);
	return eval_as<MODE, N>(seq, len, bf, threshold, streak_thr, bthres, alg, false) == d ? d : -2;
}

template <int N>
static int eval_mode(const char *seq, uint64_t len, const oracle_bf *bf, double threshold,
		unsigned streak_thr, int scoring, uint64_t *alg)
{
	switch (scoring) {
	case ORACLE_LENGTH: return eval<SCORE_LENGTH, N>(seq, len, bf, threshold, streak_thr, 0, alg);
	case ORACLE_HARMONIC:
		return eval<SCORE_HARMONIC, N>(seq, len, bf, threshold, streak_thr, 0, alg);
	case ORACLE_BINOMIAL:
		return eval<SCORE_BINOMIAL, N>(seq, len, bf, threshold, streak_thr, len < bf->k ? 0u :
				oracle_calc_min_count((unsigned)(len - bf->k + 1), oracle_bf_fpr(bf), threshold),
				alg);
	default: return eval<SCORE_SIMPLE, N>(seq, len, bf, threshold, streak_thr, 0, alg);
	}
}

extern "C" int lane_eval(const char *seq, uint64_t len, const oracle_bf *bf, double threshold,
		unsigned streak_thr, int scoring, int n, uint64_t *alg)
{
	return n == 8 ? eval_mode<8>(seq, len, bf, threshold, streak_thr, scoring, alg)
	     : n == 4 ? eval_mode<4>(seq, len, bf, threshold, streak_thr, scoring, alg)
	              : eval_mode<2>(seq, len, bf, threshold, streak_thr, scoring, alg);
}

template <int MODE, int N>
static double score(const char *seq, uint64_t len, const oracle_bf *bf, unsigned streak_thr,
		double fpr)
{
	const int k = (int)bf->k;
	LaneScore<MODE> sc;
	sc.start();
	if (len >= (uint64_t)k) {
		const Frames fr(seq, len, bf);
		double terms[kHarmTerms];
		for (int i = 0; i < kHarmTerms; ++i)
			terms[i] = harmonic_term(i);
		uint32_t run = 0;
		for (uint64_t pos = 0; pos < len; pos += 8) {
			const uint32_t V = lane_valid(bad_bases(seq, len, pos),
					(uint32_t)(len - pos < 8 ? len - pos : 8), run, k);
			for (int s = 0; s < 8; s += N) {
				const int32_t p0 = (int32_t)pos + s - k + 1;
				const uint32_t Vs = (V >> s) & ((1u << N) - 1u);
				uint32_t H = 0;
				for (int j = 0; j < N; ++j)
					if (((Vs >> j) & 1u) && fr.hit[p0 + j] &&
							(MODE == SCORE_LENGTH || p0 + j >= sc.skip_end))
						H |= 1u << j;
				sc.template step<N>(Vs, H, p0, k, (int32_t)streak_thr, terms);
			}
		}
	}
	ScoreState st;
	sc.result(st);
	if (MODE == SCORE_LENGTH)
		return (double)st.run;
	if (MODE == SCORE_BINOMIAL)
		return len < (uint64_t)k ? log10(1.0) * -10
		                         : log10(oracle_binom_sf((unsigned)(len - k + 1), fpr,
				(unsigned)st.score)) * -10;
	return score_normalize(st.score, len, (unsigned)k);
}

extern "C" double lane_score(const char *seq, uint64_t len, const oracle_bf *bf, int scoring,
		unsigned streak_thr, double fpr)
{
	switch (scoring) {
	case ORACLE_LENGTH: return score<SCORE_LENGTH, 4>(seq, len, bf, streak_thr, fpr);
	case ORACLE_HARMONIC: return score<SCORE_HARMONIC, 4>(seq, len, bf, streak_thr, fpr);
	case ORACLE_BINOMIAL: return score<SCORE_BINOMIAL, 4>(seq, len, bf, streak_thr, fpr);
	default: return score<SCORE_SIMPLE, 4>(seq, len, bf, streak_thr, fpr);
	}
}

/* Hash values v for which lane_word disagrees with v mod 32 m5. */
extern "C" uint64_t lane_word_errors(const uint64_t *v, uint64_t n, uint32_t m5)
{
	const uint64_t inv = ~0ull / m5, m = 32ull * m5;
	uint64_t bad = 0;
	for (uint64_t i = 0; i < n; ++i) {
		const uint64_t b = v[i] % m;
		const uint32_t w = lane_word(v[i], m5, (uint32_t)(inv >> 32), (uint32_t)inv);
		bad += w != b >> 5 || (v[i] & 31u) != (b & 31u);
	}
	return bad;
}
