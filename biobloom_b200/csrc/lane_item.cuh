/*
 * lane_item.cuh -- the lane kernel's building blocks (lane.cu): rolling hash
 * tables, bases, probes level by level, and a long read by a whole warp, which
 * the warp kernel (classify.cu) uses too.
 */
#ifndef BBT_LANE_ITEM_CUH
#define BBT_LANE_ITEM_CUH

#include "bbt.h"
#include "classify.cuh"
#include "lane.cuh"
#include "lane_walk.cuh"
#include "score_value.cuh"
#include "window.cuh"

namespace bbt {

constexpr uint64_t kLaneKeepBytes = 126ull << 20; /* L2 */

/* A filter as the lane kernel probes it (m = 32 m5 bits). */
struct LaneFilter {
	const uint32_t *words;
	uint64_t kmul;
	uint32_t m5, inv_hi, inv_lo, h, k;
	uint32_t keep;              /* the filter fits L2 */
};

__host__ __device__ inline LaneFilter lane_filter(const FilterDev &F)
{
	LaneFilter f;
	f.words = F.words;
	f.kmul = F.kmul;
	f.m5 = (uint32_t)(F.m >> 5);
	const uint64_t inv = ~0ull / f.m5;
	f.inv_hi = (uint32_t)(inv >> 32);
	f.inv_lo = (uint32_t)inv;
	f.h = F.h;
	f.k = F.k;
	f.keep = F.m / 8 <= kLaneKeepBytes;
	return f;
}

#if defined(__CUDACC__)

/* What a walk is for: decisions, scores, or both (the frames that a decision
 * visits are the first of those that a score does, with the same skip windows). */
enum { kLaneHits = 0, kLaneScores = 1, kLaneBoth = 2 };

/* Rolling tables of the filter's k, by outgoing code << 2 | incoming code, and
 * the hashes of k bases of code 0. */
struct LaneTables {
	uint64_t fw[16], rc[16];
	uint64_t f0, r0;
};

/* Seeds by base code: ASCII codes are (byte >> 1) & 3 (A, C, T, G), packed
 * ones A, C, G, T. */
template <bool PACKED>
__device__ __forceinline__ uint64_t lane_seed(int c, bool complement)
{
	const int x = PACKED ? c : c ^ (c >> 1); /* to A, C, G, T */
	return complement ? seed_rc_of_code(x) : seed_fw_of_code(x);
}

/* The tables, by the first warp of a block. */
template <bool PACKED>
__device__ void lane_tables(LaneTables &t, unsigned k, int lane)
{
	if (lane < 16) {
		const int out = lane >> 2, in = lane & 3;
		t.fw[lane] = rolk(lane_seed<PACKED>(out, false), k) ^ lane_seed<PACKED>(in, false);
		t.rc[lane] = ror1(lane_seed<PACKED>(out, true)) ^
				rolk(lane_seed<PACKED>(in, true), k - 1);
	}
	uint64_t f = lane < (int)k ? rolk(lane_seed<PACKED>(0, false), lane) : 0ull;
	uint64_t r = lane < (int)k ? rolk(lane_seed<PACKED>(0, true), lane) : 0ull;
	for (int o = 16; o; o >>= 1) {
		f ^= __shfl_xor_sync(kFull, f, o);
		r ^= __shfl_xor_sync(kFull, r, o);
	}
	if (lane == 0) {
		t.f0 = f;
		t.r0 = r;
	}
}

/* A filter word, not kept in L1 (an SM seldom probes a line twice, and the lines
 * would push out the reads' bases), with the L2 policy of lane_policy. */
__device__ __forceinline__ uint32_t lane_probe(const uint32_t *p, uint64_t pol)
{
	uint32_t v;
	asm("ld.global.nc.L1::no_allocate.L2::cache_hint.b32 %0, [%1], %2;"
			: "=r"(v) : "l"(p), "l"(pol));
	return v;
}

/* L2 policy of a filter's words: kept against everything else when the filter
 * fits L2 (no_allocate alone also makes L2 drop the line early: the ten filters
 * of 68 MB then took 17.7 ms per 400k pairs instead of 8.7), the first to go
 * when it does not (the reads' bases stay: 9.7 -> 9.3 ms per 2M reads over a
 * 2.1 GB filter). */
__device__ __forceinline__ uint64_t lane_policy(bool keep)
{
	uint64_t last, first;
	asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(last));
	asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(first));
	return keep ? last : first;
}

__device__ __forceinline__ uint32_t lane_ld(const uint32_t *p, uint64_t pol)
{
	uint32_t v;
	asm("ld.global.nc.L2::cache_hint.b32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol));
	return v;
}

/* Eight bases of a read from base g of its mate array, nb of them before its
 * end: nibbles (code of base j at bits 4j) and a mask of bases that are not
 * ACGT.  Loads are aligned 4-byte words, none of which lies wholly past the
 * read; the lines are in L1 from one call to the next. */
template <bool PACKED>
__device__ __forceinline__ void lane_bases(const ClassifyArgs &a, uint32_t mate, uint64_t g,
		uint32_t nb, uint32_t &nib, uint32_t &bad)
{
	const uint64_t pol = evict_first_policy(); /* the next filter reads them again, much later */
	if (PACKED) {
		const uint32_t *p = reinterpret_cast<const uint32_t *>(a.seq[mate]) + (g >> 4);
		const uint32_t at = (uint32_t)(g & 15u);
		const uint32_t c0 = lane_ld(p, pol), c1 = at + nb > 16u ? lane_ld(p + 1, pol) : 0u;
		uint32_t x = __funnelshift_r(c0, c1, 2u * at) & 0xFFFFu;
		x = (x | (x << 8)) & 0x00FF00FFu;
		x = (x | (x << 4)) & 0x0F0F0F0Fu;
		nib = (x | (x << 2)) & 0x33333333u;
		bad = 0;
		if (a.valid[mate]) {
			const uint32_t *v = a.valid[mate] + (g >> 5);
			const uint32_t vat = (uint32_t)(g & 31u);
			const uint32_t v0 = lane_ld(v, pol), v1 = vat + nb > 32u ? lane_ld(v + 1, pol) : 0u;
			bad = ~__funnelshift_r(v0, v1, vat) & 0xFFu;
		}
		return;
	}
	const uintptr_t q = (uintptr_t)(a.seq[mate] + g);
	const uint32_t *p = (const uint32_t *)(q & ~(uintptr_t)3);
	const uint32_t at = (uint32_t)(q & 3u), end = at + nb;
	const uint32_t w0 = lane_ld(p, pol), w1 = end > 4u ? lane_ld(p + 1, pol) : 0u;
	const uint32_t w2 = end > 8u ? lane_ld(p + 2, pol) : 0u;
	const uint32_t x = __funnelshift_r(w0, w1, 8u * at), y = __funnelshift_r(w1, w2, 8u * at);
	const uint32_t cx = (x >> 1) & 0x03030303u, cy = (y >> 1) & 0x03030303u;
	nib = __byte_perm(cx | (cx >> 4), cy | (cy >> 4), 0x6420);
	/* the bytes those codes stand for ("ACTG"), against the bytes read */
	const uint32_t dx = (x & 0xDFDFDFDFu) ^ __byte_perm(0x47544341u, 0, nib & 0xFFFFu);
	const uint32_t dy = (y & 0xDFDFDFDFu) ^ __byte_perm(0x47544341u, 0, nib >> 16);
	bad = 0;
	if (dx | dy) {
#pragma unroll
		for (int j = 0; j < 4; ++j) {
			bad |= ((dx >> (8 * j)) & 0xFFu) ? 1u << j : 0u;
			bad |= ((dy >> (8 * j)) & 0xFFu) ? 16u << j : 0u;
		}
	}
}

/* BloomFilter::contains of a lane's frames (bit j of live: canon[j] is probed):
 * the frames all of whose bits are set.  cost (COUNT): words read per frame. */
template <bool COUNT, int N>
__device__ __forceinline__ uint32_t lane_levels(const LaneFilter &f, const uint64_t (&canon)[N],
		uint32_t live, uint64_t pol, uint32_t *cost)
{
	if (COUNT)
		for (int j = 0; j < N; ++j)
			cost[j] = 0;
	for (uint32_t i = 0; i < f.h; ++i) {
		if (!__any_sync(kFull, live != 0u))
			break;
		const uint64_t mul = (uint64_t)i ^ f.kmul;
		uint32_t word[N], bit[N];
#pragma unroll
		for (int j = 0; j < N; ++j) {
			uint64_t v = canon[j];
			if (i) { /* extra_hash(canon, k, i) */
				v *= mul;
				v ^= v >> kMultiShift;
			}
			const uint32_t x = lane_word(v, f.m5, f.inv_hi, f.inv_lo);
			bit[j] = (uint32_t)v;
			word[j] = 0;
			if ((live >> j) & 1u)
				word[j] = lane_probe(f.words + x, pol);
			if (COUNT)
				cost[j] += (live >> j) & 1u;
		}
		live = 0; /* a frame that was not probed has no word */
#pragma unroll
		for (int j = 0; j < N; ++j)
			live += (__funnelshift_r(word[j], word[j], bit[j]) & 1u) * (1u << j);
	}
	return live;
}

/* Frames [p, p + 8) of a read of len bases from base `start` on, hashed by one
 * lane: canonical hashes and validity (frames past the read's end are not
 * valid).  The hash rolls through the bases before the one that ends frame p,
 * from a multiple of eight bases back; a base before the read counts as one
 * that is not ACGT. */
template <bool PACKED>
__device__ __forceinline__ uint32_t lane_hash8(const ClassifyArgs &a, unsigned k, const LaneTables &tab,
		uint32_t mate, uint64_t start, int64_t len, int64_t p, uint64_t (&canon)[8])
{
	const int warm = (int)(k + 6u) >> 3; /* blocks before the frames' last bases */
	int64_t s = p + k - 1 - 8 * warm;
	const uint32_t q8 = (k + 7u) >> 3, sh = 4u * (8u * q8 - k);
	uint32_t P1 = 0, P2 = 0, P3 = 0, P4 = 0, run = 0, V = 0;
	uint64_t F = tab.f0, R = tab.r0;
	for (int b = 0; b <= warm; ++b, s += 8) {
		uint32_t nib = 0, bad = 0xFFu, nb = 0;
		if (s < len) {
			const int64_t from = s < 0 ? 0 : s;
			nb = (uint32_t)min((int64_t)8, len - from);
			lane_bases<PACKED>(a, mate, start + (uint64_t)from, nb, nib, bad);
			if (s < 0) {
				nib <<= 4 * (int)-s;
				bad = (bad << (int)-s) | ((1u << (int)-s) - 1u);
				nb = min(8u, nb + (uint32_t)-s);
			}
		}
		V = lane_valid(bad, nb, run, k);
		const uint32_t lo = q8 == 4u ? P4 : q8 == 3u ? P3 : q8 == 2u ? P2 : P1;
		const uint32_t hi = q8 == 4u ? P3 : q8 == 3u ? P2 : q8 == 2u ? P1 : nib;
		const uint32_t pairs = nib | (__funnelshift_r(lo, hi, sh) << 2);
		P4 = P3;
		P3 = P2;
		P2 = P1;
		P1 = nib;
#pragma unroll
		for (int j = 0; j < 8; ++j) {
			const uint32_t e = (pairs >> (4 * j)) & 15u;
			F = rol1(F) ^ tab.fw[e];
			R = ror1(R) ^ tab.rc[e];
			canon[j] = F < R ? F : R; /* the last block's remain */
		}
	}
	return V;
}

/* Frames that a long read probes next: none of them can decide it before
 * `least` more frames, whose hits (or misses) alone would. */
__device__ __forceinline__ int lane_long_step(int64_t least)
{
	return least < 32 ? 32 : least > 256 ? 256 : (int)least;
}

/* A window of wn frames (each lane's eight: V, H) that the walk passes without a
 * gap, a skip window or a decision, as most windows of a read that is not in
 * the filter do: the totals at once, in ~60 instructions of the warp against
 * ~150 dependent ones per 32 frames.  False when it is not such a window. */
__device__ __forceinline__ bool lane_long_plain(SimpleState &st, uint32_t V, uint32_t H, int wn,
		int streak_thr, int lane)
{
	if (st.in_window || streak_thr > 8)
		return false;
	const uint32_t full = low_mask(wn - 8 * lane) & 0xFFu;
	/* bits 8-15: this lane's frames; 0-7: the eight before them */
	uint32_t before = __shfl_up_sync(kFull, H, 1);
	if (lane == 0)
		before = 0xFFu & ~(0xFFu >> min(st.streak, 8));
	const uint32_t x = (H << 8) | before, miss = full & ~H;
	uint32_t run = 0xFFu;
	for (int q = 1; q <= streak_thr; ++q)
		run &= x >> (8 - q);
	if (__any_sync(kFull, V != full || (miss & run)))
		return false;
	const int hits = __popc(H), again = st.flat ? hits : __popc(H & (x >> 7));
	const int dS = (int)__reduce_add_sync(kFull, (unsigned)(hits + again));
	const int dA = (int)__reduce_add_sync(kFull, (unsigned)__popc(miss));
	if (st.score2 + dS >= st.thres2 || st.anti + dA >= st.anti_thres)
		return false;
	st.score2 += dS;
	st.anti += dA;
	st.started = 1;
	const unsigned m = __ballot_sync(kFull, miss != 0u);
	if (m) {
		const int l = 31 - __clz((int)m);
		const int top = 31 - __clz((int)__shfl_sync(kFull, miss, l)); /* the last miss: 8 l + top */
		st.streak = min(64, wn - 1 - (8 * l + top));
	} else {
		st.streak = min(64, st.streak + wn);
	}
	return true;
}

/* A long read against filter fi (f) by the whole warp: its decision, or its score
 * (into sa).  Windows of up to
 * 256 frames, eight consecutive ones per lane, so that a window costs the
 * latency of h dependent probes; their hit bits then go through the warp's
 * chunk machine 32 at a time.  A window is no longer than the frames that the
 * earliest decision needs.  wmem: 16 words. */
template <int MODE, int WHAT, bool COUNT, bool PACKED>
__device__ __noinline__ int lane_long_item(const ClassifyArgs &a, const ScoreArgs *sa,
		const LaneFilter f, uint32_t fi, const LaneTables &tab, uint64_t r, uint32_t *wmem,
		int lane, unsigned long long *acc)
{
	constexpr bool SCORE = WHAT != kLaneHits, HITS = WHAT != kLaneScores;
	const int k = (int)f.k;
	const uint64_t pol = lane_policy(f.keep != 0);
	const uint32_t mate = r >= a.n ? 1u : 0u;
	const uint64_t i = r - (mate ? a.n : 0);
	const uint64_t start = a.off[mate][i] - a.off_base[mate];
	const uint64_t len = a.off[mate][i + 1] - a.off[mate][i];
	const uint64_t frames = len < f.k ? 0 : len - f.k + 1;
	uint32_t *vw = wmem, *hw = wmem + 8;
	SimpleState st;
	LengthState ls;
	SeqState qs;
	ScoreState sc;
	if (SCORE)
		score_init(sc);
	if (!HITS)
		;
	else if (MODE == SCORE_HARMONIC)
		harmonic_init(qs, a.score, a.one_minus, frames);
	else if (MODE == SCORE_BINOMIAL)
		binomial_simple_init(st, frames ? a.bthres[fi * a.bthres_rows + frames] : 0u, frames);
	else if (MODE == SCORE_LENGTH)
		length_init(ls, a.min_len, len, k);
	else
		simple_init(st, a.score, a.one_minus, frames);
	int decided = EVAL_OPEN;
	int wn;
	for (uint64_t w0 = 0; w0 < frames && (SCORE || !decided); w0 += wn) {
		wn = 256;
		if (!SCORE) {
			if (MODE == SCORE_LENGTH)
				wn = 64;
			else if (MODE == SCORE_HARMONIC)
				wn = lane_long_step((int64_t)fmin(qs.thres - qs.score,
						qs.anti_thres - (double)qs.anti));
			else
				wn = lane_long_step(min((st.thres2 - st.score2) / 2, st.anti_thres - st.anti));
		}
		wn = (int)min((uint64_t)wn, frames - w0);
		const int64_t p = (int64_t)w0 + 8 * lane;
		uint64_t canon[8];
		uint32_t V = lane_hash8<PACKED>(a, f.k, tab, mate, start,
				8 * lane < wn ? (int64_t)len : 0, p, canon);
		V &= low_mask(wn - 8 * lane);
		const int64_t from = MODE == SCORE_LENGTH ? 0 : SCORE ? sc.skip_end
				: MODE == SCORE_HARMONIC ? seq_probe_from(qs) : (int64_t)st.skip_until;
		const int64_t sk = from - p;
		uint32_t live = sk <= 0 ? V : sk >= 8 ? 0u : V & (0xFFu << sk);
		if (a.dust[0])
			for (int j = 0; j < 8; ++j)
				if (((live >> j) & 1u) && dust_low(a.dust[mate], start + (uint64_t)(p + j)))
					live &= ~(1u << j);
		uint32_t cost[COUNT ? 8 : 1];
		live = lane_levels<COUNT, 8>(f, canon, live, pol, cost);
		reinterpret_cast<unsigned char *>(vw)[lane] = (unsigned char)V;
		reinterpret_cast<unsigned char *>(hw)[lane] = (unsigned char)live;
		__syncwarp();
		if (!SCORE && !COUNT && (MODE == SCORE_SIMPLE || MODE == SCORE_BINOMIAL) &&
				lane_long_plain(st, V, live, wn, (int)a.streak_thr, lane))
			continue;
		uint32_t seen = 0; /* COUNT: this lane's frames that the algorithm probes */
		for (int c = 0; c < wn && (SCORE || !decided); c += 32) {
			const uint32_t Vc = vw[c >> 5], Hc = hw[c >> 5];
			const int nf = min(32, wn - c);
			const int64_t b = (int64_t)w0 + c;
			uint32_t alg = 0;
			if (SCORE)
				score_chunk(sc, Vc, Hc, b, nf, k, a.streak_thr, MODE);
			if (!HITS || decided)
				continue;
			if (MODE == SCORE_LENGTH)
				decided = length_chunk(ls, Vc, Hc, b, nf, COUNT ? &alg : nullptr);
			else if (MODE == SCORE_HARMONIC)
				decided = seq_chunk(qs, Vc, Hc, b, nf, k, a.streak_thr, COUNT ? &alg : nullptr);
			else
				decided = simple_chunk(st, Vc, Hc, (int32_t)b, nf, k, (int)a.streak_thr,
						COUNT ? &alg : nullptr);
			if (COUNT && (lane >> 2) == (c >> 5))
				seen = (alg >> (8 * (lane & 3))) & 0xFFu;
		}
		__syncwarp();
		if (COUNT) {
			acc[1] += __popc(V);
			for (int j = 0; j < 8; ++j) {
				acc[0] += cost[j];
				acc[2] += ((seen >> j) & 1u) ? cost[j] : 0u;
			}
		}
	}
	if (SCORE) {
		const double v = score_value<MODE>(sc, len, f.k, MODE == SCORE_BINOMIAL ? sa->fpr[fi] : 0.0,
				lane);
		if (lane == 0)
			sa->scores[mate][i * a.nf + fi] = v;
	}
	return decided;
}

#endif /* __CUDACC__ */

} // namespace bbt

#endif
