// CPU run of the line kernels' index arithmetic (modules_b200/csrc/cc_lines.cuh on the plan of cc_plan.cpp): reads k-sets
// from stdin as  d M  then M lines of d integers and a weight, and for each that has a line plan walks the rho groups, the
// split reduction, the weights and the force phases lane by lane with the kernels' own offsets, every index checked
// against its buffer, every output written exactly once. The rho per slot and the integer-index gradients are compared
// with direct sums (long double phases) to 1e-11 of their scales. Prints one line per k-set; exit 1 on a failure.
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../modules_b200/csrc/cc_plan.h"

using namespace cc;
typedef std::complex<double> Z;

static int fails = 0;
#define CHECK(c)                                                                                       \
	do {                                                                                               \
		if (!(c)) {                                                                                    \
			if (fails++ < 20)                                                                          \
				std::printf("FAIL line %d: %s\n", __LINE__, #c);                                       \
		}                                                                                              \
	} while (0)

static Z phase(long double t)
{
	t -= std::rint(t);
	return Z((double)std::cos(2 * M_PIl * t), (double)std::sin(2 * M_PIl * t));
}

// build_line_tables for one particle (entries outside every run stay NaN)
static std::vector<Z> tables(int d, const LineTabs &tb, const double *s)
{
	std::vector<Z> row((size_t)tb.row, Z(NAN, NAN));
	const int axis[4] = {0, d == 3 ? 1 : d - 1, d - 1, d - 1};
	int items = 0, items16 = 0;
	CHECK(d == 3 || tb.n[1] == 0);
	for (int r = 0; r < 4; r++) {
		const int n = r < 3 ? tb.n[r] : tb.nh, lo = r < 3 ? tb.lo[r] : tb.hlo, off = r < 3 ? tb.off[r] : tb.offh;
		CHECK(off >= 0 && off + n <= tb.row);
		items += (n + 7) / 8;
		items16 += (n + 15) / 16;
		for (int k = 0; k < n; k++)
			row[(size_t)off + k] = phase((long double)(lo + k) * s[axis[r]]);
	}
	CHECK(items == tb.items && items16 == tb.items16 && tb.row <= kLineMaxRow);
	return row;
}

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
		const Plan p = build_plan(d, M, modes.data(), V.data(), 8);
		const LinePlan L = build_line_plan(p);
		std::printf("d=%d M=%ld ok=%d rows=%zu units=%d groups=%zu phases=%zu\n", d, M, (int)L.ok, L.rows.size(), L.nunit,
		            L.ok ? L.groupings[0].groups.size() : 0, L.phases.size());
		if (!L.ok)
			continue;
		const int N = 11;   // particles, padded to 12 (rho) and 16 (forces) as the kernels pad theirs
		std::vector<double> s((size_t)N * d);
		unsigned long long x = 88172645463325252ull;
		for (double &v : s) {
			x ^= x << 13;
			x ^= x >> 7;
			x ^= x << 17;
			v = (double)(x >> 11) / 9007199254740992.0;
		}
		// rho groups, in every grouping
		std::vector<Z> part;
		for (const LineGroups &G : L.groupings) {
			CHECK(G.ntask >= 8 && G.ntask <= 16 && G.ntask % 4 == 0 && L.groupings[0].ntask == 8);
			CHECK(G.tasks.size() == G.groups.size() * G.ntask && G.tlines.size() == G.tasks.size() * kLineRow);
			part.assign((size_t)L.nunit * 128, Z(NAN, NAN));
			std::vector<int> wrote(part.size(), 0);
			for (size_t grp = 0; grp < G.groups.size(); grp++) {
				const LineTabs &tb = G.groups[grp];
				CHECK(tb.row % 4 == 2);
				std::vector<std::vector<Z> > tab;
				for (int j = 0; j < N; j++)
					tab.push_back(tables(d, tb, &s[(size_t)j * d]));
				int active = 0;
				for (int w = 0; w < G.ntask; w++) {
					const LineTask task = G.tasks[grp * G.ntask + w];
					CHECK(task.n >= 0 && task.n <= kLineTiles);
					active += task.n > 0;
					if (!task.n)
						continue;
					for (int half = 0; half < 2; half++)
						for (int lane = 0; lane < 32; lane++) {
							const int g = lane >> 2, t = lane & 3;
							const LineIdx l = G.tlines[(grp * G.ntask + w) * kLineRow + half * 8 + g];
							for (int j = 0; j < task.n; j++) {
								Z A = 0, B = 0;
								for (int i = 0; i < N; i++) {
									const std::vector<Z> &row = tab[i];
									CHECK(l.p0 >= 0 && l.p0 < tb.row);
									Z X = row[l.p0];
									if (d == 3) {
										CHECK(l.p1 >= 0 && l.p1 < tb.row);
										X *= row[l.p1];
									}
									if (tb.n[2] > 0) {
										CHECK(l.c >= 0 && l.c < tb.row);
										X *= row[l.c];
									}
									const int c = task.hoff + 4 * j + t;   // columns 2t, 2t + 1 of tile j
									CHECK(2 * task.hoff + 8 * j + 7 < 2 * tb.row && c >= tb.offh && c < tb.offh + tb.nh);
									A += X * row[c].real();
									B += X * row[c].imag();
								}
								const size_t o = (size_t)task.u0 * 128 + j * 128 + half * 64 + lane;
								CHECK(o + 32 < part.size());
								part[o] = Z(A.real(), B.real());
								part[o + 32] = Z(A.imag(), B.imag());
								wrote[o]++;
								wrote[o + 32]++;
							}
						}
				}
				CHECK(active == tb.ntask);
			}
			for (int w : wrote)
				CHECK(w == 1);
		}
		// reduction: every slot with a mode once, equal to the direct sum; weights in place
		std::vector<Z> u((size_t)p.nslot), wts((size_t)L.nunit * 256, Z(NAN, NAN));
		std::vector<int> slots((size_t)p.nslot, 0), wset(wts.size(), 0);
		std::vector<Z> rho((size_t)p.nslot);
		CHECK(L.cells.size() == (size_t)L.nunit * 64 && L.cellV.size() == 2 * L.cells.size());
		for (int cell = 0; cell < L.nunit * 64; cell++) {
			const int cell0 = cell / 8 * 8, ci = cell % 8;
			const size_t at = (size_t)(cell0 >> 6) * 128 + ((cell0 >> 5) & 1) * 64 + (cell0 & 31) + ci;
			const double ar = part[at].real(), br = part[at].imag(), ai = part[at + 32].real(), bi = part[at + 32].imag();
			const LineCell &c = L.cells[cell];
			Z up = 0, um = 0;
			if (c.sp >= 0) {
				slots[c.sp]++;
				rho[c.sp] = Z(ar - bi, ai + br);
				up = u[c.sp] = L.cellV[2 * cell] * std::conj(rho[c.sp]);
			}
			if (c.sm >= 0) {
				slots[c.sm]++;
				rho[c.sm] = Z(ar + bi, ai - br);
				um = u[c.sm] = L.cellV[2 * cell + 1] * std::conj(rho[c.sm]);
			}
			for (int q = 0; q < 4; q++) {
				const int unit = cell >> 6, line = (cell & 63) >> 2, t = cell & 3;
				const size_t o = ((size_t)unit * 8 + (line >> 1)) * 32 + (4 * (line & 1) + q) * 4 + t;
				const Z a = up + um, b = up - um;
				CHECK(o < wts.size());
				wts[o] = q == 0 ? Z(a.real(), -b.imag()) : q == 1 ? Z(a.imag(), b.real())
				       : (double)c.h * (q == 2 ? Z(b.real(), -a.imag()) : Z(b.imag(), a.real()));
				wset[o]++;
			}
		}
		for (int w : wset)
			CHECK(w == 1);
		std::vector<int> has((size_t)p.nslot, 0);
		double umax = 0, nmax = 1;
		std::vector<double> ref((size_t)N * d, 0.0);
		for (long m = 0; m < M; m++) {
			const int q = p.mode_slot[(size_t)m];
			if (has[q]++)
				continue;
			CHECK(slots[q] == 1);
			Z r = 0;
			for (int i = 0; i < N; i++) {
				long double t = 0;
				for (int e = 0; e < d; e++)
					t += (long double)modes[(size_t)m * d + e] * s[(size_t)i * d + e];
				const Z z = phase(t);
				r += z;
				for (int e = 0; e < d; e++)
					ref[(size_t)i * d + e] += modes[(size_t)m * d + e] * (u[q] * z).imag();
			}
			CHECK(std::abs(r - rho[q]) < 1e-11 * N);
			umax += std::abs(u[q]);
			for (int e = 0; e < d; e++)
				nmax = std::max(nmax, (double)std::abs(modes[(size_t)m * d + e]));
		}
		for (int q = 0; q < p.nslot; q++)
			CHECK(has[q] ? slots[q] == 1 : slots[q] == 0);
		// force phases: every unit once
		std::vector<int> used((size_t)L.nunit, 0);
		std::vector<double> grad((size_t)N * d, 0.0);
		CHECK(L.lines.size() == L.rows.size() * kLineRow);
		for (const LineTabs &tb : L.phases) {
			CHECK(tb.row % 8 == 4 && tb.hlo % 4 == 0 && tb.nh % 4 == 0);
			std::vector<std::vector<Z> > tab;
			for (int j = 0; j < N; j++)
				tab.push_back(tables(d, tb, &s[(size_t)j * d]));
			for (int r = tb.r0; r < tb.r0 + tb.ntask; r++) {
				CHECK(r >= 0 && r < (int)L.rows.size());
				const int jb = tb.hlo >> 2, je = (tb.hlo + tb.nh) >> 2, nj = std::min(je, L.rows[r].nj) - jb;
				for (int j = 0; j < nj; j++)
					used[(size_t)L.rows[r].ubase + jb + j]++;
				for (int line = 0; line < kLineRow; line++) {
					const LineIdx li = L.lines[(size_t)r * kLineRow + line];
					const int o0 = tb.off[0] + li.p0 - tb.lo[0], o1 = tb.off[1] + li.p1 - tb.lo[1],
					          oc = tb.off[2] + li.c - tb.lo[2];
					CHECK(o0 >= 0 && o0 < tb.row && (d < 3 || (o1 >= 0 && o1 < tb.row)) &&
					      (tb.n[2] == 0 || (oc >= 0 && oc < tb.row)));
					for (int i = 0; i < N; i++) {
						Z T = 0, D = 0;
						for (int j = 0; j < nj; j++)
							for (int t = 0; t < 4; t++) {
								const Z c = tab[i][(size_t)tb.offh + 4 * j + t];
								CHECK(4 * j + t < tb.nh);
								double v[4];
								for (int q = 0; q < 4; q++) {   // fragment lane 4 g + t, g = 4 (line & 1) + q
									const size_t w = ((size_t)(L.rows[r].ubase + jb + j) * 8 + line / 2) * 32 + (4 * (line & 1) + q) * 4 + t;
									CHECK(w < wts.size());
									v[q] = wts[w].real() * c.real() + wts[w].imag() * c.imag();
								}
								T += Z(v[0], v[1]);
								D += Z(v[2], v[3]);
							}
						Z X = tab[i][(size_t)o0];
						if (d == 3)
							X *= tab[i][(size_t)o1];
						if (tb.n[2] > 0)
							X *= tab[i][(size_t)oc];
						const double S = (X * T).imag();
						grad[(size_t)i * d] += li.p0 * S;
						if (d == 3)
							grad[(size_t)i * d + 1] += li.p1 * S;
						grad[(size_t)i * d + d - 1] += li.c * S + (X * D).imag();
					}
				}
			}
		}
		for (int w : used)
			CHECK(w == 1);
		for (size_t i = 0; i < grad.size(); i++)
			CHECK(std::fabs(grad[i] - ref[i]) <= 1e-11 * (umax * nmax + 1e-300));
	}
	if (fails)
		std::printf("%d checks failed\n", fails);
	return fails ? 1 : 0;
}
