// Plans k-sets read from stdin ("d M", then M lines of d integers and a weight) and prints for each the segments, the distinct
// modes and the sum of the slots' weights.
#include <cstdio>
#include <vector>

#include "../modules_b200/csrc/cc_plan.h"

int main()
{
	int d;
	long M;
	while (std::scanf("%d %ld", &d, &M) == 2) {
		std::vector<int32_t> modes((size_t)M * d);
		std::vector<double> V((size_t)M);
		for (long m = 0; m < M; m++) {
			for (int e = 0; e < d; e++)
				if (std::scanf("%d", &modes[(size_t)m * d + e]) != 1)
					return 2;
			if (std::scanf("%lf", &V[(size_t)m]) != 1)
				return 2;
		}
		const cc::Plan p = cc::build_plan(d, M, modes.data(), V.data(), 8);
		double sum = 0.0;
		for (double v : p.slotV)
			sum += v;
		std::printf("%ld %ld %.17g\n", (long)p.real_segs, (long)p.unique_modes, sum);
	}
	return 0;
}
