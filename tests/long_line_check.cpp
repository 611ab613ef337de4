// The line plan of sets with very long lines: reads "half lines" pairs from stdin, plans the 2D set of prefixes 1 .. lines
// with last indices -half .. half (weights 1), and checks that every grouping gives each row's column tiles to its tasks
// once, in shares of 1 to kLineTiles. Prints "ok=<0|1> nj=<tiles of the first row>" per set; exit 1 on a failure.
#include <cstdio>
#include <vector>

#include "../modules_b200/csrc/cc_plan.h"

using namespace cc;

int main()
{
	long half, lines;
	int fails = 0;
	while (std::scanf("%ld %ld", &half, &lines) == 2) {
		std::vector<int32_t> modes;
		for (long p = 1; p <= lines; p++)
			for (long c = -half; c <= half; c++) {
				modes.push_back((int32_t)p);
				modes.push_back((int32_t)c);
			}
		const int64_t M = (int64_t)modes.size() / 2;
		const std::vector<double> V((size_t)M, 1.0);
		const LinePlan L = build_line_plan(build_plan(2, M, modes.data(), V.data(), 8));
		for (const LineGroups &G : L.groupings) {
			std::vector<int> seen((size_t)L.nunit, 0);
			for (const LineTask &k : G.tasks) {
				if (k.n < 0 || k.n > kLineTiles || k.u0 < 0 || k.u0 + k.n > L.nunit) {
					fails++;
					continue;
				}
				for (int j = 0; j < k.n; j++)
					seen[(size_t)(k.u0 + j)]++;
			}
			for (int s : seen)
				fails += s != 1;
		}
		std::printf("ok=%d nj=%d\n", L.ok ? 1 : 0, L.rows.empty() ? 0 : L.rows[0].nj);
	}
	return fails ? 1 : 0;
}
