// The choice between the line and the segment kernels (cc_plan.cpp lines_preferred): reads k-sets from stdin as "d M K" with K
// particle counts, then the counts, then M lines of d integers; prints for each count "<lines with forces><lines for rho alone>"
// (1 or 0; - without a line plan) at 148 SMs.
#include <cstdio>
#include <vector>

#include "../modules_b200/csrc/cc_plan.h"

int main()
{
	int d, K;
	long M;
	while (std::scanf("%d %ld %d", &d, &M, &K) == 3) {
		std::vector<long> N((size_t)K);
		for (long &n : N)
			if (std::scanf("%ld", &n) != 1)
				return 2;
		std::vector<int32_t> modes((size_t)M * d);
		for (int32_t &m : modes)
			if (std::scanf("%d", &m) != 1)
				return 2;
		const std::vector<double> V((size_t)M, 1.0);
		const cc::Plan p = cc::build_plan(d, M, modes.data(), V.data(), 8);
		const cc::LinePlan L = cc::build_line_plan(p);
		for (long n : N) {
			if (!L.ok) {
				std::printf("- ");
				continue;
			}
			const cc::LineLaunch g = cc::line_launch(L, d, n, 148);
			std::printf("%d%d ", (int)cc::lines_preferred(p, L, g, n, true), (int)cc::lines_preferred(p, L, g, n, false));
		}
		std::printf("\n");
	}
	return 0;
}
