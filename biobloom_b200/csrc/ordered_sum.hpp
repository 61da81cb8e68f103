/*
 * ordered_sum.hpp -- a sum whose terms are computed on several threads.
 */
#ifndef BBT_ORDERED_SUM_HPP
#define BBT_ORDERED_SUM_HPP

#include <stdint.h>

#include <algorithm>
#include <exception>
#include <thread>
#include <vector>

namespace bbt {

/* sum + fn(lo) + ... + fn(hi - 1), added in this order: the same value on any
 * number of threads.  Up to `most` compute the terms, each at least 1024; parts
 * whose thread does not start, and all of them without memory for the terms, are
 * computed by the caller's thread, so that nothing is thrown.  fn must not
 * throw.  Thread: std::thread, or what a test puts in its place. */
template <class Thread = std::thread, class Fn>
double ordered_sum(uint64_t lo, uint64_t hi, double sum, unsigned most, Fn fn)
{
	const uint64_t n = hi > lo ? hi - lo : 0;
	const uint64_t parts = std::max<uint64_t>(1, std::min<uint64_t>(most, n / 1024));
	std::vector<double> terms;
	std::vector<Thread> threads;
	auto part = [&](uint64_t p) {
		for (uint64_t i = n * p / parts; i < n * (p + 1) / parts; ++i)
			terms[(size_t)i] = fn(lo + i);
	};
	if (parts > 1) {
		try {
			terms.resize((size_t)n);
			threads.reserve((size_t)parts);
		} catch (const std::exception &) {
			terms.clear();
		}
	}
	if (terms.empty()) {
		for (uint64_t i = lo; i < lo + n; ++i)
			sum += fn(i);
		return sum;
	}
	uint64_t p = 1;
	try {
		for (; p < parts; ++p)
			threads.emplace_back(part, p);
	} catch (const std::exception &) { /* parts p and up have no thread */
	}
	part(0);
	for (; p < parts; ++p)
		part(p);
	for (Thread &t : threads)
		t.join();
	for (double v : terms)
		sum += v;
	return sum;
}

} // namespace bbt

#endif
