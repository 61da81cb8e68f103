/*
 * dust_may_model.cpp -- the masking kernel's pass 0 (dust_may_mask,
 * dust_core.cuh) compiled for the host.  TEST INFRASTRUCTURE ONLY.
 */
#include <stdint.h>

#include <vector>

#include "dust_core.cuh"

extern "C" int model_may_mask(const char *seq, uint64_t len, int T, int W)
{
	std::vector<uint32_t> kinds(64, 0u);
	std::vector<uint16_t> ring((size_t)W - 2);
	const uint8_t *bases = (const uint8_t *)seq;
	return bbt::dust_may_mask([&](int i) { return bases[i]; }, len, T, W,
			[&](unsigned t) -> uint32_t & { return kinds.at(t); },
			[&](int i) -> uint16_t & { return ring.at((size_t)i); });
}
