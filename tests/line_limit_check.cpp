// The line kernels' particle indices at the largest particle counts they are given: for every number of splits, the end of the
// last split and the start of the chunk after its last one (cc_lines.cuh line_rho_body: j0 + per_split, cj + chunk) stay below
// 2^31. Exit 1 on a failure.
#include <algorithm>
#include <climits>
#include <cstdio>

#include "../modules_b200/csrc/cc_plan.h"

int main()
{
	const int64_t counts[] = {cc::kLineMaxParticles, cc::kLineMaxParticles - 1, cc::kLineMaxParticles - 4095};
	int fails = 0;
	for (int64_t N : counts)
		for (int64_t ns = 1; ns <= cc::kLineMaxSplits; ns++) {
			const int64_t per = std::max<int64_t>(8, ((N + ns - 1) / ns + 7) / 8 * 8), real = (N + per - 1) / per;
			const int64_t j0 = (real - 1) * per, j1 = std::min(N, j0 + per);
			for (int64_t chunk = 8; chunk <= cc::kLineMaxChunk; chunk *= 2)
				fails += j0 + per > INT_MAX || j0 + (j1 - j0 + chunk - 1) / chunk * chunk > INT_MAX;
		}
	std::printf("%d\n", fails);
	return fails ? 1 : 0;
}
