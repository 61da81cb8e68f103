/*
 * classify_read.cuh -- one read evaluated against filters by one warp: the
 * body of the warp kernels (classify.cu) and of the lane kernel's long reads
 * (lane.cu).
 */
#ifndef BBT_CLASSIFY_READ_CUH
#define BBT_CLASSIFY_READ_CUH

#include "bbt.h"
#include "classify.cuh"
#include "seqeval_chunk.cuh"
#include "window.cuh"

namespace bbt {

/* Valid-frame bits of frames [c, c + n) of the window (n <= 32). */
template <int SEG>
__device__ __forceinline__ uint32_t step_bits(const Window<SEG> &win, int c, int n)
{
	const int vi = c >> 5, vs = c & 31;
	uint32_t V = win.vmask[vi] >> vs;
	if (vs && vi + 1 < SEG)
		V |= win.vmask[vi + 1] << (32 - vs);
	if (n < 32)
		V &= (1u << n) - 1u;
	return V;
}

/* Build setting: a read whose frames mostly hit reads all h bits of a frame
 * at once (1) instead of the first, then the others together (0). */
#ifndef BBT_HIT_READS_ALL
#define BBT_HIT_READS_ALL 0
#endif

/* Evaluate read r against filters [f0, f1).  Returns the hit bits of those
 * filters that fall in word f0 / 64 (bit f % 64); read-major launches call it
 * with the whole filter range and write every word themselves.  WIDE: every
 * lane probes two frames per step (steps of up to 64 frames), twice the word
 * reads in flight per warp. */
template <int SEG, bool COUNT, int MODE, bool WIDE>
__device__ void classify_read(const ClassifyArgs &a, uint64_t r, uint32_t f0, uint32_t f1,
		const Window<SEG> &win, int lane, uint64_t &myword, unsigned long long &probe_acc,
		unsigned long long &frame_acc, unsigned long long &alg_acc)
{
	constexpr int W = Window<SEG>::W;
	const uint32_t mate = r >= a.n ? 1u : 0u;
	const uint64_t i = r - (mate ? a.n : 0);
	const uint64_t *off = a.off[mate];
	const uint64_t start = off[i] - a.off_base[mate];
	const uint64_t len = off[i + 1] - off[i];
	const Bases s = read_bases(a, mate, start);
	unsigned cached_k = 0;
	int64_t cached_w0 = -1;
	unsigned reads = 0;
	for (uint32_t f = f0; f < f1; ++f) {
		const FilterDev F = a.filters[f];
		const unsigned k = F.k;
		if (len < k)
			continue;
		const uint64_t frames = len - k + 1;
		SimpleState st;
		LengthState ls;
		SeqState qs;
		constexpr bool length_mode = MODE == BBT_SCORE_LENGTH;
		/* HARMONIC walks frame by frame (seq_chunk); BINOMIAL is SIMPLE's
		 * machine with integer hits (binomial_simple_init) */
		constexpr bool seq_mode = MODE == BBT_SCORE_HARMONIC;
		if (MODE == BBT_SCORE_HARMONIC)
			harmonic_init(qs, a.score, a.one_minus, frames);
		else if (MODE == BBT_SCORE_BINOMIAL)
			binomial_simple_init(st, a.bthres[f * a.bthres_rows + frames], frames);
		else if (length_mode)
			length_init(ls, a.min_len, len, (int)k);
		else
			simple_init(st, a.score, a.one_minus, frames);
		int decided = EVAL_OPEN;
		/* decision-sized steps read a frame's bits after the first together
		 * while at least half of the read's frames probed in its last step
		 * were hits (a read from the filter's reference: every bit gets read
		 * anyway, in fewer round trips), one after another otherwise (a read
		 * that is not in the filter: most frames stop at the first or second
		 * clear bit, so fewer filter reads); warp-uniform, from the step's
		 * ballots */
		bool hitting = true;
		for (uint64_t w0 = 0; w0 < frames && !decided; w0 += W) {
			const int wn = (int)min((uint64_t)W, frames - w0);
			if (cached_k != k || cached_w0 != (int64_t)w0) {
				if (cached_k != k)
					set_tables<SEG>(win, k, lane);
				hash_window<SEG>(s, w0, wn, k, win, lane);
				cached_k = k;
				cached_w0 = (int64_t)w0;
				if (COUNT)
					frame_acc += (lane == 0) ? (unsigned long long)wn : 0ull;
			}
			for (int c = 0; c < wn;) {
				/* frames [c, c + nfc) of the window this step: lane l probes
				 * frame c + l, and with WIDE also frame c + 32 + l; the
				 * machine then takes them 32 at a time, in frame order */
				constexpr int cap = WIDE ? 64 : 32;
				const int nfc = min((length_mode || seq_mode || !a.tight_steps) ? cap
						: simple_step_frames(st, cap), wn - c);
				const int n0 = min(nfc, 32);
				/* frames below this were in a skip window when the step began */
				const int32_t pf = length_mode ? INT32_MIN
						: seq_mode ? (int32_t)seq_probe_from(qs) : st.skip_until;
				auto probe_at = [&](uint32_t V, int q) {
					const int32_t p = (int32_t)w0 + q;
					return ((V >> lane) & 1u) && p >= pf &&
							!dust_low(a.dust[mate], start + (uint64_t)p);
				};
				auto advance = [&](uint32_t V, uint32_t H, int b, int n, uint32_t *alg) {
					return length_mode ? length_chunk(ls, V, H, (int64_t)w0 + b, n, alg)
							: seq_mode ? seq_chunk(qs, V, H, (int64_t)w0 + b, n, (int)k,
									a.streak_thr, alg)
							: simple_chunk(st, V, H, (int32_t)w0 + b, n, (int)k,
									(int)a.streak_thr, alg);
				};
				const uint32_t V0 = step_bits<SEG>(win, c, n0);
				const bool probe0 = probe_at(V0, c + lane);
				uint32_t alg = 0;
				if (WIDE) {
					const int n1 = nfc - n0;
					const uint32_t V1 = n1 > 0 ? step_bits<SEG>(win, c + 32, n1) : 0u;
					const bool probe1 = probe_at(V1, c + 32 + lane);
					bool hit0, hit1;
					unsigned ra = 0, rb = 0;
					contains2(F, probe0 ? win.h0[c + lane] : 0ull, probe0,
							probe1 ? win.h0[c + 32 + lane] : 0ull, probe1, hit0, hit1, ra, rb);
					reads += ra + rb;
					const uint32_t H0 = __ballot_sync(kFull, hit0);
					const uint32_t H1 = __ballot_sync(kFull, hit1);
					decided = advance(V0, H0, c, n0, COUNT ? &alg : nullptr);
					if (COUNT && ((alg >> lane) & 1u))
						alg_acc += ra;
					if (!decided && n1 > 0) {
						alg = 0;
						decided = advance(V1, H1, c + 32, n1, COUNT ? &alg : nullptr);
						if (COUNT && ((alg >> lane) & 1u))
							alg_acc += rb;
					}
				} else {
					const unsigned r0 = reads;
					unsigned sq = 0;
					const bool split = a.tight_steps && hitting;
					const bool hit = probe0 && (split
							? (BBT_HIT_READS_ALL
								? contains_all(F, win.h0[c + lane], reads, sq)
								: contains_split(F, win.h0[c + lane], reads, sq))
							: contains(F, win.h0[c + lane], reads));
					const uint32_t H = __ballot_sync(kFull, hit);
					if (a.tight_steps) {
						const uint32_t P = __ballot_sync(kFull, probe0);
						if (P)
							hitting = 2 * __popc(H) >= __popc(P);
					}
					decided = advance(V0, H, c, n0, COUNT ? &alg : nullptr);
					if (COUNT && ((alg >> lane) & 1u))
						alg_acc += split ? sq : reads - r0;
				}
				if (decided)
					break;
				c += nfc;
			}
		}
		if (decided == EVAL_ACCEPT && lane == (int)(f >> 6))
			myword |= 1ull << (f & 63);
	}
	if (COUNT)
		probe_acc += reads;
}

} // namespace bbt

#endif
