/*
 * mibf_scan.cuh -- the miBF query of reads whose counters fit 16 bits, over the
 * dense ID map (included by mibf.cu, which holds the general kernel for the
 * rank layout, more than kMibfSmemIds IDs and longer reads).
 *
 * One warp per read (pair), a frame per lane per step, as the general kernel.
 * What bounds a query is the random 128-byte line fill of each probe; the
 * general kernel reached half of that rate, because it ran 16 warps per SM
 * (100 registers, 24-byte tally slots) and ~1465 instructions per 32 frames:
 *
 *   hashing  a spaced seed's value is an XOR over its care positions of the
 *            bases' rotated seeds.  With running XORs P(t) of the bases before
 *            t, each base rotated by its own position, a run of care positions
 *            is P(end) ^ P(begin), and the value one rotation of the sum by the
 *            frame's position.  So a value takes two reads for the whole span
 *            and one (or two) per run of positions left out, at consecutive
 *            addresses over the lanes (no bank conflicts), instead of a table
 *            read per pair of bases: 8 for a seed of weight 19 and span 25,
 *            against 13 that conflict.  The running XORs cost one warp scan
 *            per 32 bases, shared by all seeds.
 *   tally    six 16-bit counters in three 32-bit words per ID (native
 *            shared-memory additions, half the memory); and the counters of
 *            the ID that most frames of the read agree on stay in registers,
 *            from two warp sums per step, where all lanes would add to one
 *            address.
 *
 *   overlap  a step's entries are tallied while the next step's are on the way.
 *
 * What is left is the probes: 500k reads of 150 bp against 500 targets (1.7 GB
 * map, 189 M probes) 7.2 -> 4.1 ms, 46 G probes/s of the 50 G/s that random
 * line fills reach (0.9 ms with the probes left out); 50k pairs of 75 to 300 bp
 * against 100 targets (350 MB map) 1.6 -> 0.8 ms.
 */
#ifndef BBT_MIBF_SCAN_CUH
#define BBT_MIBF_SCAN_CUH

/* For each value of a frame, the 16-byte entries of the warp's ring to XOR, as
 * byte offsets from the lane's frame: running XORs at 16 t, single bases at
 * kScanSingles + 16 t. */
constexpr int kScanSingles = 64 * 16;
constexpr int kScanEntries = 32;
struct ScanLists {
	uint16_t n[kMibfMaxSeeds];
	uint16_t off[kMibfMaxSeeds][kScanEntries];
};

/* The shorter of: first and last care position and each run left out between
 * them (one position as a single base, more by its ends), or the care positions
 * one by one. */
static ScanLists scan_lists(const std::vector<std::string> &seeds, unsigned k)
{
	ScanLists l;
	memset(&l, 0, sizeof l);
	const size_t ns = seeds.empty() ? 1 : seeds.size();
	for (size_t s = 0; s < ns && s < kMibfMaxSeeds; ++s) {
		const std::string seed = seeds.empty() ? std::string(k, '1') : seeds[s];
		std::vector<uint16_t> runs, ones;
		size_t a = seed.find('1');
		if (a != std::string::npos) {
			const size_t b = seed.rfind('1') + 1;
			runs = {(uint16_t)(16 * a), (uint16_t)(16 * b)};
			for (size_t i = a; i < b; ++i) {
				if (seed[i] == '1') {
					ones.push_back((uint16_t)(kScanSingles + 16 * i));
					continue;
				}
				size_t e = i;
				while (seed[e] != '1')
					++e;
				if (e == i + 1) {
					runs.push_back((uint16_t)(kScanSingles + 16 * i));
				} else {
					runs.push_back((uint16_t)(16 * i));
					runs.push_back((uint16_t)(16 * e));
				}
				i = e - 1;
			}
		}
		const std::vector<uint16_t> &v = runs.size() <= ones.size() ? runs : ones;
		l.n[s] = (uint16_t)v.size();
		for (size_t i = 0; i < v.size() && i < (size_t)kScanEntries; ++i)
			l.off[s][i] = v[i];
	}
	return l;
}

constexpr int kScanThreads = 256;
constexpr int kScanBlocks = 3;  /* per SM: 24 warps at 80 registers */
constexpr size_t kScanSmemPerSm = 140 << 10;

__host__ __device__ inline uint32_t scan_slots(uint32_t nids)
{
	return (nids + 127u) & ~127u;
}

__host__ inline size_t scan_smem(uint32_t nids)
{
	return 2048 + (size_t)(kScanThreads / 32) * (2048 + (size_t)scan_slots(nids) * 12);
}

/* Counters of one ID: A = count | nonSatCount << 16, B = solidCount |
 * totalCount << 16, C = totalNonSatCount | nonSatFrameCount << 16. */
struct ScanIds {
	uint32_t *A, *B, *C;
	uint32_t id, a, b, c;   /* the ID whose counters are in registers (0: none) */
};

/* A step's entries e (0: no hit): each lane's frame into its IDs' counters. */
template <int H>
__device__ __forceinline__ void scan_tally(const MibfArgs &g, const uint32_t (&e)[H], ScanIds &t,
		uint32_t &satc, LaneCounts &lc, int lane)
{
	const uint32_t h = g.f.h, nids = g.f.nids, need = g.need;
	uint32_t any = 0, id[H];
	bool agree = true;
#pragma unroll
	for (int v = 0; v < H; ++v) {
		any |= e[v];
		lc.hits += e[v] ? 1u : 0u;
		id[v] = e[v] & 0x7FFFu;
		agree = agree && (v >= (int)h || id[v] == id[0]);
	}
	const bool anysat = any & kMibfSat;
	satc += __popc(__ballot_sync(kFull, anysat));
	agree = agree && id[0] >= 1 && id[0] < nids;
	const unsigned m = __ballot_sync(kFull, agree);
	if (m && !__ballot_sync(kFull, agree && id[0] == t.id)) {
		/* another ID's frames: its counters come into registers */
		__syncwarp();
		if (lane == 0 && t.id) {
			t.A[t.id] += t.a;
			t.B[t.id] += t.b;
			t.C[t.id] += t.c;
		}
		__syncwarp();
		t.id = __shfl_sync(kFull, id[0], __ffs(m) - 1);
		t.a = t.b = t.c = 0;
	}
	if (t.id) {
		uint32_t hits = 0, ns = 0;
#pragma unroll
		for (int v = 0; v < H; ++v)
			if (id[v] == t.id) {
				++hits;
				ns += (e[v] & kMibfSat) ? 0u : 1u;
			}
		uint32_t p = 0;
		if (hits)
			p = (hits >= need ? 1u : 0u) | (ns >= need ? 1u << 8 : 0u) | (hits == h ? 1u << 16 : 0u) |
					(hits >= need && !anysat ? 1u << 24 : 0u);
		const uint32_t s = __reduce_add_sync(kFull, p);
		const uint32_t u = __reduce_add_sync(kFull, hits | (ns << 16));
		t.a += (s & 0xFFu) | ((s << 8) & 0xFF0000u);
		t.b += ((s >> 16) & 0xFFu) | (u << 16);
		t.c += (u >> 16) | ((s >> 8) & 0xFF0000u);
	}
#pragma unroll
	for (int r = 0; r < H; ++r) {
		bool first = id[r] >= 1 && id[r] < nids && id[r] != t.id;
#pragma unroll
		for (int v = 0; v < r; ++v)
			first = first && id[v] != id[r];
		if (first) {
			uint32_t hits = 0, ns = 0;
#pragma unroll
			for (int v = 0; v < H; ++v)
				if (id[v] == id[r]) {
					++hits;
					ns += (e[v] & kMibfSat) ? 0u : 1u;
				}
			const uint32_t a = (hits >= need ? 1u : 0u) | (ns >= need ? 1u << 16 : 0u);
			const uint32_t b = (hits == h ? 1u : 0u) | (hits << 16);
			const uint32_t c = ns | (hits >= need && !anysat ? 1u << 16 : 0u);
			if (a)
				atomicAdd(t.A + id[r], a);
			atomicAdd(t.B + id[r], b);
			if (c)
				atomicAdd(t.C + id[r], c);
		}
	}
}

/* All frames of one mate. */
template <int H>
__device__ __forceinline__ void scan_mate(const MibfArgs &g, const ScanLists &l, uint64_t pol,
		uint32_t m5, uint32_t inv_hi, uint32_t inv_lo, const ulonglong2 *rot, unsigned char *ring,
		const Bases &src, uint64_t len, ScanIds &t, uint32_t &satc, LaneCounts &lc, int lane)
{
	const uint32_t k = g.f.k, h = g.f.h;
	if (len < k)
		return;
	const uint32_t n = (uint32_t)len, frames = n - k + 1;
	const uint32_t kmask = k >= 32 ? ~0u : (1u << k) - 1u;
	ulonglong2 *P = reinterpret_cast<ulonglong2 *>(ring), *S = P + 64;
	const unsigned char *mine = ring + 16 * lane;
	ulonglong2 carry = {0ull, 0ull}, oldP, oldS = {0ull, 0ull};
	uint32_t inv0 = 0;
	uint8_t next = lane < n ? base_code_at(src, lane) : (uint8_t)4;
	oldP = carry;
	uint32_t e[H]; /* entries read for the step before, tallied while this one's are on the way */
#pragma unroll
	for (int v = 0; v < H; ++v)
		e[v] = 0;
	for (uint32_t c0 = 0;; c0 += 32) {
		/* bases [c0, c0 + 32): lane's base rotated by its position, and the
		 * running XORs */
		const uint8_t code = next;
		next = c0 + 32 + lane < n ? base_code_at(src, (uint64_t)c0 + 32 + lane) : (uint8_t)4;
		const uint32_t inv1 = __ballot_sync(kFull, code & 4u);
		ulonglong2 b = rot[4 * lane + (code & 3)];
		if (c0 & 32u) {
			b.x = (b.x << 32) | (b.x >> 32);
			b.y = (b.y << 32) | (b.y >> 32);
		}
		ulonglong2 s = b;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const unsigned long long x = __shfl_up_sync(kFull, s.x, o);
			const unsigned long long y = __shfl_up_sync(kFull, s.y, o);
			if (lane >= o) {
				s.x ^= x;
				s.y ^= y;
			}
		}
		const ulonglong2 p = {carry.x ^ s.x ^ b.x, carry.y ^ s.y ^ b.y};
		carry.x ^= __shfl_sync(kFull, s.x, 31);
		carry.y ^= __shfl_sync(kFull, s.y, 31);
		__syncwarp();
		P[lane] = oldP;
		S[lane] = oldS;
		P[32 + lane] = p;
		S[32 + lane] = b;
		__syncwarp();
		oldP = p;
		oldS = b;
		if (c0 > 0) {
			/* frames [q0, q0 + 32), whose bases are the two chunks held */
			const uint32_t q0 = c0 - 32;
			const bool ok = q0 + lane < frames &&
					!(__funnelshift_r(inv0, inv1, lane) & kmask);
			const uint32_t turn = (uint32_t)lane ^ (q0 & 32u); /* (q0 + lane) mod 64 */
			uint32_t en[H];
			uint64_t vals[H];
#pragma unroll
			for (int v = 0; v < H; ++v) {
				vals[v] = 0;
				if (v < (int)h && (v == 0 || !g.f.kmer_mode)) {
					unsigned long long F = 0, R = 0;
					const int ne = l.n[v];
#pragma unroll 4
					for (int i = 0; i < ne; ++i) {
						const ulonglong2 x =
								*reinterpret_cast<const ulonglong2 *>(mine + l.off[v][i]);
						F ^= x.x;
						R ^= x.y;
					}
					F = rotl64(F, (turn + k - 1u) & 63u);
					R = rotl64(R, (64u - turn) & 63u);
					vals[v] = F < R ? F : R;
				} else if (v < (int)h) {
					vals[v] = extra_hash(vals[0], k, v);
				}
			}
#pragma unroll
			for (int v = 0; v < H; ++v) {
				en[v] = 0;
				if (ok && v < (int)h) {
					const uint16_t *at = g.f.dense +
							((uint64_t)lane_word(vals[v], m5, inv_hi, inv_lo) * 32u +
							 ((uint32_t)vals[v] & 31u));
					uint16_t x;
					asm("ld.global.nc.L1::no_allocate.L2::cache_hint.u16 %0, [%1], %2;"
							: "=h"(x) : "l"(at), "l"(pol));
					en[v] = x;
				}
			}
			lc.frames += ok ? 1u : 0u;
			lc.probes += ok ? h : 0u;
			if (q0)
				scan_tally<H>(g, e, t, satc, lc, lane);
#pragma unroll
			for (int v = 0; v < H; ++v)
				e[v] = en[v];
			if (c0 >= frames) /* the last frame is below c0 */
				break;
		}
		inv0 = inv1;
	}
	scan_tally<H>(g, e, t, satc, lc, lane);
}

__device__ __forceinline__ void scan_prefetch(const Bases &b)
{
	const void *p = b.ascii ? (const void *)(b.ascii + b.g0) : (const void *)(b.words + (b.g0 >> 4));
	asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

template <int H>
__global__ void __launch_bounds__(kScanThreads, kScanBlocks) mibf_scan_kernel(
		const __grid_constant__ MibfArgs g, const __grid_constant__ ScanLists l)
{
	extern __shared__ __align__(16) unsigned char smem[];
	const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
	const uint32_t nids = g.f.nids, T = scan_slots(nids), k = g.f.k;
	ulonglong2 *rot = reinterpret_cast<ulonglong2 *>(smem);
	if (threadIdx.x < 128) { /* base code c at position p mod 32: both strands' seeds */
		const int p = threadIdx.x >> 2, c = threadIdx.x & 3;
		rot[threadIdx.x] = {rolk(seed_fw_of_code(c), 64 - p), rolk(seed_rc_of_code(c), p)};
	}
	unsigned char *ring = smem + 2048 + (size_t)wib * (2048 + (size_t)T * 12);
	ScanIds t;
	t.A = reinterpret_cast<uint32_t *>(ring + 2048);
	t.B = t.A + T;
	t.C = t.B + T;
	uint4 *T4 = reinterpret_cast<uint4 *>(t.A);
	for (uint32_t i = lane; i < 3 * T / 4; i += 32)
		T4[i] = make_uint4(0, 0, 0, 0);
	__syncthreads();
	const uint32_t m5 = (uint32_t)(g.f.m >> 5);
	const uint64_t inv = ~0ull / m5;
	const uint32_t inv_hi = (uint32_t)(inv >> 32), inv_lo = (uint32_t)inv;
	const uint64_t pol = lane_policy(2 * g.f.m <= kLaneKeepBytes);
	unsigned long long *above = g.counts, *unique = g.counts + (nids + 2);
	LaneCounts lc;
	for (;;) {
		unsigned long long r0 = 0;
		if (lane == 0)
			r0 = atomicAdd(g.work, (unsigned long long)kReadsPerGrab);
		r0 = __shfl_sync(kFull, r0, 0);
		if (r0 >= g.n_reads)
			break;
		const uint64_t r1 = r0 + kReadsPerGrab < g.n_reads ? r0 + kReadsPerGrab : g.n_reads;
		/* the reads' offsets, one per lane, and their first bases into L1 */
		uint64_t o1 = 0, o2 = 0;
		if (r0 + lane <= r1) {
			o1 = g.off[r0 + lane];
			o2 = g.seq2 ? g.off2[r0 + lane] : 0;
		}
		const bool has1 = __shfl_down_sync(kFull, o1, 1) > o1;
		const bool has2 = __shfl_down_sync(kFull, o2, 1) > o2;
		if (r0 + lane < r1 && has1)
			scan_prefetch(mate_bases(g, 0, o1));
		if (r0 + lane < r1 && has2)
			scan_prefetch(mate_bases(g, 1, o2));
		for (uint64_t r = r0; r < r1; ++r) {
			const int j = (int)(r - r0);
			const uint64_t b1 = __shfl_sync(kFull, o1, j), b2 = __shfl_sync(kFull, o2, j);
			const uint64_t len1 = __shfl_sync(kFull, o1, j + 1) - b1;
			const uint64_t len2 = __shfl_sync(kFull, o2, j + 1) - b2;
			/* frameCount (MIBFClassifier.hpp:774, 802-803) */
			const uint32_t fc = len1 >= k ? (uint32_t)(len1 - k + 1)
					: (len2 >= k ? (uint32_t)(len2 - k + 1) : 0u);
			uint32_t satc = 0, cmask = 0, maxns = 0;
			Cand best = {0ull, 0ull};
			/* entry 0 of a minCount row is the smallest of the others */
			const uint32_t *mrow = g.minc + (size_t)fc * nids;
			const uint32_t least = fc ? max(__ldg(mrow), 1u) : 0u;
			if (fc) {
				t.id = t.a = t.b = t.c = 0;
				scan_mate<H>(g, l, pol, m5, inv_hi, inv_lo, rot, ring, mate_bases(g, 0, b1), len1, t,
						satc, lc, lane);
				if (g.seq2)
					scan_mate<H>(g, l, pol, m5, inv_hi, inv_lo, rot, ring, mate_bases(g, 1, b2),
							len2, t, satc, lc, lane);
				__syncwarp();
				if (lane == 0 && t.id) {
					t.A[t.id] += t.a;
					t.B[t.id] += t.b;
					t.C[t.id] += t.c;
				}
				__syncwarp();
				/* significant IDs: bit 4 i + j of cmask is slot 128 i + 4 lane + j */
				for (uint32_t i = 0; i < T / 128; ++i) {
					const uint4 q = T4[32 * i + lane];
					const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
					for (int j = 0; j < 4; ++j) {
						const uint32_t cnt = w[j] & 0xFFFFu, ns = w[j] >> 16;
						const uint32_t s = 128 * i + 4 * lane + j;
						if (cnt >= least && s >= 1 && s < nids && cnt >= __ldg(mrow + s) &&
								(g.min_nonsat == 0 || ns >= g.min_nonsat)) {
							cmask |= 1u << (4 * i + j);
							const Cand c = {((unsigned long long)cnt << 32) | ns,
									((unsigned long long)(t.B[s] >> 16) << 32) | (0xFFFFFFFFull - s)};
							if (cand_less(best, c))
								best = c;
							maxns = ns > maxns ? ns : maxns;
						}
					}
				}
			}
			uint32_t n_out = 0;
			if (__any_sync(kFull, cmask)) {
				best = warp_best(best);
				maxns = __reduce_max_sync(kFull, maxns);
				if (!(g.best_agree && maxns > (uint32_t)best.k1)) {
					const double thr = (double)(uint32_t)(best.k1 >> 32) - g.multi;
					Cand cur = best;
					for (;;) {
						const uint32_t id = 0xFFFFFFFFu - (uint32_t)cur.k2;
						if (lane == 0) {
							if (n_out < g.max_hits) {
								const uint32_t A = t.A[id], B = t.B[id], C = t.C[id];
								bbt_mibf_hit o;
								o.id = id;
								o.nonSatFrameCount = C >> 16;
								o.solidCount = B & 0xFFFFu;
								o.count = A & 0xFFFFu;
								o.nonSatCount = A >> 16;
								o.totalNonSatCount = C & 0xFFFFu;
								o.totalCount = B >> 16;
								g.hits[r * g.max_hits + n_out] = o;
							}
							atomicAdd(above + id, 1ull);
						}
						++n_out;
						/* next: the best candidate below cur that passes the threshold */
						Cand nx = {0ull, 0ull};
						for (uint32_t b = cmask; b; b &= b - 1u) {
							const uint32_t i = __ffs(b) - 1;
							const uint32_t s = 128 * (i >> 2) + 4 * lane + (i & 3u);
							const uint32_t A = t.A[s];
							const Cand c = {((unsigned long long)(A & 0xFFFFu) << 32) | (A >> 16),
									((unsigned long long)(t.B[s] >> 16) << 32) | (0xFFFFFFFFull - s)};
							if (cand_less(c, cur) && (double)(A & 0xFFFFu) > thr && cand_less(nx, c))
								nx = c;
						}
						if (!__any_sync(kFull, nx.k1 != 0ull))
							break;
						cur = warp_best(nx);
					}
				}
			}
			if (lane == 0) {
				g.n_hits[r] = n_out;
				g.sat[r] = satc;
				if (n_out > g.max_hits)
					atomicOr(g.flags, 1u);
				if (n_out == 0) {
					if (!g.skip_empty_summary)
						atomicAdd(g.counts + 2 * (nids + 2) + 1, 1ull);
				} else if (n_out == 1) {
					atomicAdd(unique + (0xFFFFFFFFu - (uint32_t)best.k2), 1ull);
				} else {
					atomicAdd(g.counts + 2 * (nids + 2), 1ull);
				}
			}
			__syncwarp();
			if (fc)
				for (uint32_t i = lane; i < 3 * T / 4; i += 32)
					T4[i] = make_uint4(0, 0, 0, 0);
			__syncwarp();
		}
	}
#pragma unroll
	for (int o = 16; o; o >>= 1) {
		lc.frames += __shfl_xor_sync(kFull, lc.frames, o);
		lc.probes += __shfl_xor_sync(kFull, lc.probes, o);
		lc.hits += __shfl_xor_sync(kFull, lc.hits, o);
	}
	if (lane == 0 && (lc.frames || lc.probes)) {
		atomicAdd(g.stat, lc.frames);
		atomicAdd(g.stat + 1, lc.probes);
		atomicAdd(g.stat + 2, lc.hits);
	}
}

#endif
