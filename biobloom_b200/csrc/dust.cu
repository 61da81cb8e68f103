/*
 * dust.cu -- SDUST low-complexity masking on the GPU (-D, -T, -W).
 *
 * With opt::dust the reference builds an SDust object per evaluated read
 * (Common/SDust.hpp), which runs sdust (Common/sdust.c: the symmetric DUST
 * algorithm of Morgulis et al., J Comput Biol 2006, as minimap2 implements
 * it) over the read, and SeqEval then treats every frame whose start lies in
 * a masked interval as a miss without probing the filter
 * (Common/SeqEval.h:53,78,132,...).
 *
 * Here one thread runs the same sequential algorithm per read (the algorithm
 * is a scan with a sliding window and a list of pending "perfect intervals";
 * reads are independent, so the batch is the parallel dimension) and sets,
 * for every masked base position, a bit in a per-mate bit array indexed like
 * the batch's bases.  The classification kernels read that bit for each
 * frame they evaluate.
 *
 * Most reads hold no perfect interval, and the window's counters alone show it
 * (the search starts when 10 rw > L T).  Pass 0, a thread per read, keeps just
 * those, in shared memory, and lists the reads for which the search would
 * start; pass 1 runs the full scan on these, a warp per read.  A thread per read
 * for the full scan of all took 977 us per 100k reads of 101 to 151 bases: its
 * counters and list lie in local memory, and its lanes search at different
 * places.  Where most reads are listed it is no slower: 100k random reads of 150 bases
 * 1460 -> 566 us, with T = 5, which lists nearly all of them, 48.4 -> 16.4 ms; all
 * ending in 40 As 385 -> 298 ms and all of six-base repeats 1714 -> 1726 ms, most of it
 * pass 2.
 *
 * The list of pending perfect intervals is short for ordinary sequence but
 * grows with the square of the window on long homopolymers and short tandem
 * repeats (thousands of entries for W = 64).  Pass 1 keeps it in a small
 * array per warp; a read that outgrows it is queued and recomputed from
 * the start by pass 2, whose threads each own a slice of global memory large
 * enough for any read (W^2 + 2W + 64 entries: the list, plus the entries one
 * window step adds before they are merged in).  A read outgrowing even that is
 * reported through an error counter and fails the call.
 *
 * The algorithm, in the reference's terms: words are the triplets of
 * consecutive A/C/G/T bases (either case); the window holds the last W - 2
 * triplets; a set of triplets scores sum over kinds of c(c-1)/2.  cw / rw
 * count the whole window; cv / rv count its longest suffix (L triplets) in
 * which no kind occurs more than 2T/10 times.  When 10 rw > L T the window
 * may hold perfect intervals (suffixes with 10 r > T l whose score is at
 * least that of every perfect interval starting inside them); they are kept
 * by descending start.  One whose start falls out of the window is saved as
 * masked, merged with the previous masked interval when they touch.  A base
 * that is not A/C/G/T, and the end of the read, flush the pending intervals
 * but leave the window as it is.
 */
#include "dust.cuh"

#include <algorithm>

#include "dust_core.cuh"

namespace bbt {

namespace {

constexpr int kLocalPerfect = 160;  /* pass-1 capacity of the perfect list (and of the
                                       entries a window step adds before they merge) */

/* Set bits [a, b) of the read's mask (positions clamped to the read). */
__device__ void mask_range(uint32_t *mask, uint64_t base, int64_t a, int64_t b, uint64_t len)
{
	if (a < 0)
		a = 0;
	if (b > (int64_t)len)
		b = (int64_t)len;
	for (int64_t p = a; p < b;) {
		const uint64_t g = base + (uint64_t)p;
		const uint32_t bit = (uint32_t)(g & 31u);
		const int64_t n = min((int64_t)(32u - bit), b - p);
		const uint32_t bits = (n == 32 ? 0xffffffffu : ((1u << n) - 1u)) << bit;
		atomicOr(mask + (g >> 5), bits);
		p += n;
	}
}

/* Bases in order, eight at a time: one aligned 8-byte load per 8 bases
 * (each thread scans its own read, so byte loads would not coalesce). */
struct BaseStream {
	const uint8_t *p;
	uint64_t word = 0;
	int64_t word_at = -1; /* address / 8 of the word held */
	__device__ __forceinline__ uint8_t operator()(int i)
	{
		const uintptr_t a = (uintptr_t)(p + i);
		const int64_t w = (int64_t)(a >> 3);
		if (w != word_at) {
			word = __ldg(reinterpret_cast<const unsigned long long *>(a & ~(uintptr_t)7));
			word_at = w;
		}
		return (uint8_t)(word >> ((a & 7u) * 8u));
	}
};

__device__ bool dust_read(const uint8_t *__restrict__ seq, uint64_t len, int T, int W,
		DustPerfect *perf, int pcap, uint8_t *ring, uint32_t *mask, uint64_t mask_base)
{
	BaseStream bs{seq};
	return dust_scan(bs, len, T, W, perf, pcap, ring, [&](int a, int b) {
		mask_range(mask, mask_base, a, b, len);
	});
}

__device__ __forceinline__ void read_at(const DustArgs &a, uint64_t r, const uint8_t *&s,
		uint64_t &len, uint32_t *&mask, uint64_t &base)
{
	const uint32_t mate = r >= a.n ? 1u : 0u;
	const uint64_t i = r - (mate ? a.n : 0);
	const uint64_t *off = a.off[mate];
	base = off[i] - a.off_base[mate];
	len = off[i + 1] - off[i];
	s = a.seq[mate] + base;
	mask = a.mask[mate];
}

/* Words [64 kinds][thread], 32 bits (a bank per lane), then rings
 * [W - 2][thread], 16 bits. */
__global__ void __launch_bounds__(128) dust_pass0_kernel(DustArgs a)
{
	extern __shared__ uint32_t smem[];
	const int nt = blockDim.x;
	uint32_t *kinds = smem + threadIdx.x;
	uint16_t *rings = reinterpret_cast<uint16_t *>(smem + 64 * nt) + threadIdx.x;
	const uint64_t total = a.n * a.mates;
	for (uint64_t r = (uint64_t)blockIdx.x * nt + threadIdx.x; r < total;
			r += (uint64_t)gridDim.x * nt) {
		const uint8_t *s;
		uint64_t len, base;
		uint32_t *mask;
		read_at(a, r, s, len, mask, base);
		for (int t = 0; t < 64; ++t)
			kinds[t * nt] = 0;
		BaseStream bs{s};
		if (dust_may_mask(bs, len, a.T, a.W,
				[&](unsigned t) -> uint32_t & { return kinds[t * nt]; },
				[&](int i) -> uint16_t & { return rings[i * nt]; }))
			a.todo[atomicAdd(a.todo_count, 1ull)] = r;
	}
}

/* dust_scan (dust_core.cuh) of one read by a warp: every lane holds the same
 * scalars, lane 0 writes the shared state, and find_perfect's scores of all
 * window suffixes are computed together (a suffix adds, for its first triplet,
 * the number of that kind after it: the shared counters plus the lanes before
 * with the same kind), which leaves the sequential part to the few suffixes
 * that pass the threshold.  False when the interval list outgrows
 * kLocalPerfect. */
struct DustWarp {
	DustPerfect perf[kLocalPerfect];
	uint16_t cw[64], cv[64], c[64];
	uint8_t ring[kDustMaxWindow];
};

__device__ bool dust_read_warp(const uint8_t *__restrict__ seq, uint64_t len, int T, int W,
		DustWarp &w, uint32_t *mask, uint64_t mask_base, int lane)
{
	constexpr unsigned kAll = 0xffffffffu;
	BaseStream bs{seq};
	__syncwarp();
	for (int i = lane; i < 64; i += 32)
		w.cw[i] = w.cv[i] = 0;
	__syncwarp();
	int rw = 0, rv = 0, L = 0, head = 0, size = 0, np = 0, res_f = 0, l = 0;
	bool have_res = false;
	unsigned t = 0;
	const int n = (int)len;
	auto slot = [&](int i) -> int { return head + i >= W ? head + i - W : head + i; };
	/* one element of shared state, by lane 0 */
	auto put = [&](uint16_t &x, int v) {
		__syncwarp();
		if (lane == 0)
			x = (uint16_t)v;
		__syncwarp();
	};
	auto save = [&](int start) {
		if (np == 0 || w.perf[np - 1].start >= start)
			return;
		const int ps = w.perf[np - 1].start, pf = w.perf[np - 1].finish;
		int from = ps, to = pf;
		if (have_res && ps <= res_f) {
			from = res_f;
			to = res_f > pf ? res_f : pf;
		}
		if (lane == 0 && to > from)
			mask_range(mask, mask_base, from, to, len);
		have_res = true;
		res_f = to;
		while (np > 0 && w.perf[np - 1].start < start)
			--np;
	};
	for (int i = 0; i <= n; ++i) {
		const int b = i < n ? dust_code(bs(i)) : 4;
		if (b >= 4) {
			int start = (l - W + 1 > 0 ? l - W + 1 : 0) + (i + 1 - l);
			while (np)
				save(start++);
			l = 0;
			t = 0;
			continue;
		}
		++l;
		t = (t << 2 | (unsigned)b) & 63u;
		if (l < 3)
			continue;
		const int start = (l - W > 0 ? l - W : 0) + (i + 1 - l);
		save(start);
		/* shift_window */
		if (size >= W - 2) {
			const int s = w.ring[head];
			head = head + 1 == W ? 0 : head + 1;
			--size;
			const int x = w.cw[s] - 1;
			rw -= x;
			put(w.cw[s], x);
			if (L > size) {
				--L;
				const int y = w.cv[s] - 1;
				rv -= y;
				put(w.cv[s], y);
			}
		}
		const int x = w.cw[t], y = w.cv[t];
		__syncwarp();
		if (lane == 0) {
			w.ring[slot(size)] = (uint8_t)t;
			w.cw[t] = (uint16_t)(x + 1);
			w.cv[t] = (uint16_t)(y + 1);
		}
		__syncwarp();
		++size;
		++L;
		rw += x;
		rv += y;
		if ((y + 1) * 10 > T * 2) {
			int s;
			do {
				s = w.ring[slot(size - L)];
				const int v = w.cv[s] - 1;
				rv -= v;
				put(w.cv[s], v);
				--L;
			} while (s != (int)t);
		}
		if (rw * 10 <= L * T)
			continue;
		/* find_perfect: suffixes k = size - L - 1 down to 0, 32 at a time */
		for (int q = lane; q < 64; q += 32)
			w.c[q] = w.cv[q];
		__syncwarp();
		int r = rv, max_r = 0, max_l = 0, jp = 0, nn = 0;
		for (int k0 = size - L - 1; k0 >= 0; k0 -= 32) {
			const int k = k0 - lane;
			const int tk = k >= 0 ? w.ring[slot(k)] : 64 + lane;
			const unsigned same = __match_any_sync(kAll, tk);
			int v = k >= 0 ? w.c[tk] + __popc(same & ((1u << lane) - 1u)) : 0;
			__syncwarp();
			if (k >= 0 && lane == __ffs(same) - 1)
				w.c[tk] = (uint16_t)(w.c[tk] + __popc(same));
			for (int o = 1; o < 32; o <<= 1) {
				const int u = __shfl_up_sync(kAll, v, o);
				if (lane >= o)
					v += u;
			}
			v += r;
			r = __shfl_sync(kAll, v, 31);
			__syncwarp();
			for (unsigned m = __ballot_sync(kAll, k >= 0 && v * 10 > T * (size - k - 1)); m;
					m &= m - 1u) {
				const int j = __ffs(m) - 1;
				const int new_r = __shfl_sync(kAll, v, j), kk = k0 - j, new_l = size - kk - 1;
				for (; jp < np && w.perf[jp].start >= kk + start; ++jp) {
					const int pr = w.perf[jp].r, pl = w.perf[jp].l;
					if (max_r == 0 || pr * max_l > max_r * pl) {
						max_r = pr;
						max_l = pl;
					}
				}
				if (max_r == 0 || new_r * max_l >= max_r * new_l) {
					max_r = new_r;
					max_l = new_l;
					if (np + 2 * nn + 2 > kLocalPerfect)
						return false;
					if (lane == 0)
						w.perf[kLocalPerfect - 1 - nn] = {kk + start, size + 2 + start, new_r,
								(int)((unsigned)jp << 11 | (unsigned)new_l)};
					++nn;
				}
			}
			__syncwarp();
		}
		if (nn) {
			if (lane == 0) {
				/* backward merge into [0, np + nn), as dust_scan */
				int wr = np + nn - 1, io = np - 1;
				for (int ei = nn - 1; ei >= 0; --ei) {
					DustPerfect e = w.perf[kLocalPerfect - 1 - ei];
					const int pos = (int)((unsigned)e.l >> 11);
					e.l = (int)((unsigned)e.l & 2047u);
					while (io >= pos)
						w.perf[wr--] = w.perf[io--];
					w.perf[wr--] = e;
				}
			}
			np += nn;
			__syncwarp();
		}
	}
	return true;
}

__global__ void __launch_bounds__(128) dust_pass1_kernel(DustArgs a)
{
	__shared__ DustWarp warps[4];
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const uint64_t total = *(volatile unsigned long long *)a.todo_count;
	for (uint64_t q = (uint64_t)blockIdx.x * 4 + warp; q < total; q += (uint64_t)gridDim.x * 4) {
		const uint64_t r = a.todo[q];
		const uint8_t *s;
		uint64_t len, base;
		uint32_t *mask;
		read_at(a, r, s, len, mask, base);
		if (!dust_read_warp(s, len, a.T, a.W, warps[warp], mask, base, lane) && lane == 0)
			a.redo[atomicAdd(a.redo_count, 1ull)] = r;
	}
}

__global__ void __launch_bounds__(128) dust_pass2_kernel(DustArgs a)
{
	uint8_t ring[kDustMaxWindow];
	const uint64_t redo_n = *(volatile unsigned long long *)a.redo_count;
	const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
	DustPerfect *perf = reinterpret_cast<DustPerfect *>(a.scratch) + tid * a.scratch_per_thread;
	for (uint64_t q = tid; q < redo_n; q += (uint64_t)gridDim.x * blockDim.x) {
		const uint8_t *s;
		uint64_t len, base;
		uint32_t *mask;
		read_at(a, a.redo[q], s, len, mask, base);
		if (!dust_read(s, len, a.T, a.W, perf, (int)a.scratch_per_thread, ring, mask, base))
			atomicAdd(a.failed, 1ull);
	}
}

} // namespace

size_t dust_perfect_bytes()
{
	return sizeof(DustPerfect);
}

/* Shared memory of a block of nt threads of pass 0; above kDustPass0Block a block
 * has fewer threads. */
static size_t dust_pass0_bytes(unsigned nt, int W)
{
	return (size_t)nt * (64 * 4 + (size_t)(W - 2) * 2);
}
constexpr size_t kDustPass0Block = 56u << 10;

cudaError_t launch_dust_pass1(const DustArgs &a, int num_sms, cudaStream_t s)
{
	const uint64_t total = a.n * a.mates;
	if (total == 0)
		return cudaSuccess;
	/* threads per block: as many as keep four blocks on an SM, from 128 (W = 64:
	 * 47.5 KB) down to 32, of which three fit from W = 770 on (W = 1024: 72 KB).  The
	 * limit is the most that any W takes, not this one's: it belongs to the process,
	 * where another thread's context may have a larger W. */
	unsigned nt = 128;
	while (nt > 32 && dust_pass0_bytes(nt, a.W) > kDustPass0Block)
		nt /= 2;
	const size_t bytes = dust_pass0_bytes(nt, a.W);
	cudaError_t e = cudaFuncSetAttribute(dust_pass0_kernel,
			cudaFuncAttributeMaxDynamicSharedMemorySize,
			(int)std::max(kDustPass0Block, dust_pass0_bytes(32, kDustMaxWindow)));
	if (e != cudaSuccess)
		return e;
	const uint64_t need = (total + nt - 1) / nt;
	const uint64_t cap = (uint64_t)num_sms * 64;
	dust_pass0_kernel<<<(unsigned)(need < cap ? need : cap), nt, bytes, s>>>(a);
	if ((e = cudaGetLastError()) != cudaSuccess)
		return e;
	/* a full grid: how many reads are listed is known on the device */
	dust_pass1_kernel<<<(unsigned)(num_sms * 8), 128, 0, s>>>(a);
	return cudaGetLastError();
}

cudaError_t launch_dust_pass2(const DustArgs &a, uint32_t threads, cudaStream_t s)
{
	if (a.n * a.mates == 0)
		return cudaSuccess;
	const uint32_t blocks = (threads + 31) / 32;
	dust_pass2_kernel<<<blocks, 32, 0, s>>>(a);
	return cudaGetLastError();
}

} // namespace bbt
