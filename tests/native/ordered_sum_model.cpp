/*
 * ordered_sum_model.cpp -- ordered_sum (biobloom_b200/csrc/ordered_sum.hpp) with
 * threads that stop starting.  TEST INFRASTRUCTURE ONLY.
 */
#include "ordered_sum.hpp"

#include <cmath>
#include <system_error>

namespace {

int g_left; /* threads that still start */

struct FewThreads {
	std::thread t;
	template <class Fn>
	FewThreads(Fn fn, uint64_t p)
	{
		if (g_left-- <= 0)
			throw std::system_error(std::make_error_code(std::errc::resource_unavailable_try_again));
		t = std::thread(fn, p);
	}
	FewThreads(FewThreads &&) = default;
	void join() { t.join(); }
};

} // namespace

extern "C" double model_ordered_sum(uint64_t lo, uint64_t hi, double sum, unsigned most, int start)
{
	g_left = start;
	return bbt::ordered_sum<FewThreads>(lo, hi, sum, most,
			[](uint64_t i) { return std::pow(1.0 - std::exp(-1e-7 * (double)i), 3.0); });
}
