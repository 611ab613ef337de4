// cc_plan.cpp — host-side planning (see cc_plan.h).
#include "cc_plan.h"

#include <algorithm>
#include <array>
#include <cmath>
#include <numeric>
#include <random>
#include <set>

namespace cc {

namespace {

const double kTwoPi = 6.283185307179586476925286766559;

// Lexicographic order on (prefix..., last).
struct ModeLess {
	const int32_t *m;
	int d;
	bool operator()(int64_t a, int64_t b) const
	{
		for (int e = 0; e < d; e++)
			if (m[a * d + e] != m[b * d + e])
				return m[a * d + e] < m[b * d + e];
		return false;
	}
};

// The modes' lexicographic order, equal ones in input order: the indices, less each axis' least, packed into one key and
// sorted by digits of 11 bits where the key fits 64 (40002 modes of a circle in any order 0.3 ms, a comparison sort through
// the index 5), else by comparisons.
std::vector<int64_t> mode_order(int d, int64_t M, const int32_t *modes)
{
	std::vector<int64_t> idx((size_t)M);
	std::iota(idx.begin(), idx.end(), 0);
	int64_t lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};
	for (int64_t m = 0; m < M; m++)
		for (int e = 0; e < d; e++) {
			const int64_t v = modes[m * d + e];
			lo[e] = m == 0 ? v : std::min(lo[e], v);
			hi[e] = m == 0 ? v : std::max(hi[e], v);
		}
	int shift[3] = {0, 0, 0}, bits = 0;
	for (int e = d - 1; e >= 0; e--) {
		shift[e] = bits;
		while (((hi[e] - lo[e]) >> (bits - shift[e])) != 0)
			bits++;
	}
	if (M < 128 || bits > 64) {
		std::stable_sort(idx.begin(), idx.end(), ModeLess{modes, d});
		return idx;
	}
	std::vector<uint64_t> key((size_t)M);
	bool sorted = true;
	for (int64_t m = 0; m < M; m++) {
		uint64_t k = 0;
		for (int e = 0; e < d; e++)
			if (hi[e] > lo[e])
				k |= (uint64_t)(modes[m * d + e] - lo[e]) << shift[e];
		key[(size_t)m] = k;
		sorted &= m == 0 || key[(size_t)m - 1] <= k;
	}
	if (sorted)
		return idx;
	constexpr int kDigit = 11;
	std::vector<int64_t> to((size_t)M);
	std::vector<int64_t> at((size_t)1 << kDigit);
	for (int b = 0; b < bits; b += kDigit) {
		const uint64_t mask = (1u << kDigit) - 1;
		std::fill(at.begin(), at.end(), 0);
		for (int64_t m = 0; m < M; m++)
			at[(key[(size_t)m] >> b) & mask]++;
		int64_t sum = 0;
		for (int64_t &n : at) {
			const int64_t c = n;
			n = sum;
			sum += c;
		}
		for (int64_t m : idx)
			to[(size_t)at[(key[(size_t)m] >> b) & mask]++] = m;
		idx.swap(to);
	}
	return idx;
}

// Index ranges of a set of segments, per axis (prefix axes: p0, p1; last axis: segment starts).
struct Ranges {
	int lo[3], hi[3];
	bool empty = true;
	void add(int d, const Seg &s)
	{
		int v[3] = {s.p0, s.p1, 0};
		v[d - 1] = s.start;
		for (int e = 0; e < d; e++) {
			if (empty || v[e] < lo[e])
				lo[e] = v[e];
			if (empty || v[e] > hi[e])
				hi[e] = v[e];
		}
		empty = false;
	}
};

TabSpec make_spec(int d, const Ranges &r)
{
	TabSpec t = {};
	int off = 0;
	for (int e = 0; e < d; e++) {
		// (indices of either sign span up to 2^32; what does not fit a table is cut off by the caller, by its row)
		const int range = (int)std::min<int64_t>((int64_t)r.hi[e] - r.lo[e] + 1, 1 << 28);
		t.lo[e] = r.lo[e];
		if (e < d - 1 && range <= kFullMax) {
			t.full[e] = 1;
			t.offc[e] = off;
			t.run[t.nrun++] = TabRun{e, 1, r.lo[e], range, off};
			off += range;
		} else {
			const int nc = (range + 7) / 8;
			t.full[e] = 0;
			t.offc[e] = off;
			t.run[t.nrun++] = TabRun{e, 8, r.lo[e], nc, off};
			off += nc;
			t.offf[e] = off;
			t.run[t.nrun++] = TabRun{e, 1, 0, 8, off};
			off += 8;
		}
	}
	t.row = off;
	t.items = 0;
	for (int i = 0; i < t.nrun; i++)
		t.items += (t.run[i].count + 7) / 8;
	return t;
}

int spec_row(int d, const Ranges &r) { return make_spec(d, r).row; }

}  // namespace

Plan build_plan(int d, int64_t M, const int32_t *modes, const double *V, int L)
{
	Plan p;
	p.d = d;
	const std::vector<int64_t> idx = mode_order(d, M, modes);
	// unique modes in sorted order, with summed weights
	std::vector<std::array<int32_t, 3> > u;
	std::vector<double> uV;
	std::vector<int64_t> mode_u((size_t)M);
	for (size_t i = 0; i < idx.size(); i++) {
		const int64_t m = idx[i];
		std::array<int32_t, 3> key = {0, 0, 0};
		for (int e = 0; e < d; e++)
			key[e] = modes[m * d + e];
		if (u.empty() || key != u.back()) {
			u.push_back(key);
			uV.push_back(0.0);
		}
		uV.back() += V[m];
		mode_u[m] = (int64_t)u.size() - 1;
	}
	p.unique_modes = (int64_t)u.size();
	if (L <= 0)
		L = 8;
	p.L = L;
	std::vector<int64_t> u_slot(u.size());
	int len = 0;
	for (size_t i = 0; i < u.size(); i++) {
		bool cont = i > 0 && len < L && u[i][d - 1] == u[i - 1][d - 1] + 1;
		for (int e = 0; e + 1 < d && cont; e++)
			cont = u[i][e] == u[i - 1][e];
		if (cont) {
			len++;
			p.segs.back().len = len;
		} else {
			Seg s;
			s.p0 = d >= 2 ? u[i][0] : 0;
			s.p1 = d >= 3 ? u[i][1] : 0;
			s.start = u[i][d - 1];
			s.len = 1;
			p.segs.push_back(s);
			len = 1;
		}
		u_slot[i] = (int64_t)(p.segs.size() - 1) * L + (len - 1);
	}
	// rho groups: up to 32 consecutive segments whose tables fit kMaxRow entries, padded to 32
	std::vector<Seg> raw;
	raw.swap(p.segs);
	p.real_segs = (int64_t)raw.size();
	std::vector<int64_t> where(raw.size());
	size_t i0 = 0;
	while (i0 < raw.size()) {
		Ranges r;
		size_t j = i0;
		while (j < raw.size() && (int)(j - i0) < kGroupSegs) {
			Ranges t = r;
			t.add(d, raw[j]);
			if (j > i0 && spec_row(d, t) > kMaxRow)
				break;
			r = t;
			j++;
		}
		for (size_t k = i0; k < j; k++) {
			where[k] = (int64_t)p.segs.size();
			p.segs.push_back(raw[k]);
		}
		while (p.segs.size() % kGroupSegs)
			p.segs.push_back(Seg{0, 0, 0, 0});
		p.rspec.push_back(make_spec(d, r));
		p.rho_max_row = std::max(p.rho_max_row, p.rspec.back().row);
		i0 = j;
	}
	// slot of (segment q, step r) = r * nseg + q: a warp's 32 segments are contiguous for every r
	const int64_t nseg = (int64_t)p.segs.size();
	for (size_t i = 0; i < u.size(); i++) {
		const int64_t seg = u_slot[i] / L, r = u_slot[i] % L;
		u_slot[i] = r * nseg + where[(size_t)seg];
	}
	// block groups: up to kBlockGroups consecutive rho groups whose joint tables fit kMaxRow entries
	{
		const int ng = p.ngroups();
		int g = 0;
		while (g < ng) {
			Ranges r;
			int h = g;
			while (h < ng && h - g < kBlockGroups) {
				Ranges t = r;
				for (int q = h * kGroupSegs; q < (h + 1) * kGroupSegs; q++)
					if (p.segs[q].len > 0)
						t.add(d, p.segs[q]);
				if (h > g && spec_row(d, t) > kMaxRow)
					break;
				r = t;
				h++;
			}
			p.bstart.push_back(g);
			p.bspec.push_back(make_spec(d, r));
			p.block_max_row = std::max(p.block_max_row, p.bspec.back().row);
			g = h;
		}
		p.bstart.push_back(ng);
	}
	p.nslot = (int)p.segs.size() * L;
	p.slotV.assign((size_t)p.nslot, 0.0);
	for (size_t i = 0; i < u.size(); i++)
		p.slotV[(size_t)u_slot[i]] = uV[i];
	p.mode_slot.resize((size_t)M);
	p.modeV.assign(V, V + M);
	for (int64_t m = 0; m < M; m++)
		p.mode_slot[(size_t)m] = (int)u_slot[(size_t)mode_u[(size_t)m]];
	return p;
}

ForceSplits force_splits(const Plan &p, int want)
{
	ForceSplits f;
	const int nseg = (int)p.segs.size();
	want = std::max(1, std::min(want, std::max(1, (int)p.real_segs)));
	const int64_t target = (p.real_segs + want - 1) / want;   // real segments per split
	int i = 0;
	while (i < nseg) {
		Ranges r;
		int j = i, real = 0;
		while (j < nseg) {
			if (p.segs[j].len == 0) {   // padding: no table entries
				j++;
				continue;
			}
			if (real >= target)
				break;
			Ranges t = r;
			t.add(p.d, p.segs[j]);
			if (real > 0 && spec_row(p.d, t) > kMaxRow)
				break;
			r = t;
			real++;
			j++;
		}
		if (real == 0)   // trailing padding only: attach to the previous split
		{
			if (!f.start.empty()) {
				i = nseg;
				break;
			}
			Seg z = {0, 0, 0, 1};
			r.add(p.d, z);
		}
		f.start.push_back(i);
		f.spec.push_back(make_spec(p.d, r));
		f.max_row = std::max(f.max_row, f.spec.back().row);
		i = j;
	}
	f.start.push_back(nseg);
	return f;
}

namespace {

struct Line {
	LineIdx ix;
	int hmax;        // cells 0 .. hmax
	int a, b;        // first and last last index
	int s0, s1;      // segments [s0, s1) of the plan (padding segments among them)
};

struct Span {
	int lo = 0, hi = -1;
	void add(int v)
	{
		if (hi < lo) {
			lo = hi = v;
		} else {
			lo = std::min(lo, v);
			hi = std::max(hi, v);
		}
	}
	int n() const { return hi - lo + 1; }
};

// Table layout for prefix spans a (axis 0), b (axis 1), centres c and cells [hlo, hlo + nh). The entries per particle are
// padded to `mod` modulo 8, the row stride with which the kernels' fragment loads meet no bank twice.
LineTabs line_tabs(int d, bool centres, const Span &a, const Span &b, const Span &c, int hlo, int nh, int mod)
{
	LineTabs t = {};
	const Span *s[3] = {&a, &b, &c};
	const bool use[3] = {true, d == 3, centres};
	int off = 0;
	for (int e = 0; e < 3; e++) {
		t.lo[e] = use[e] ? s[e]->lo : 0;
		t.n[e] = use[e] ? s[e]->n() : 0;
		t.off[e] = off;
		off += t.n[e];
		t.items += (t.n[e] + 7) / 8;
		t.items16 += (t.n[e] + 15) / 16;
	}
	t.hlo = hlo;
	t.nh = nh;
	t.offh = off;
	off += nh;
	t.items += (nh + 7) / 8;
	t.items16 += (nh + 15) / 16;
	t.row = off + ((mod - off) % 8 + 8) % 8;
	return t;
}

constexpr int kRhoRowMod = 2, kForceRowMod = 4;
constexpr int kLineForceCells = 64;      // cells per force phase when the whole set's tables do not fit

// Groups of up to `most` tasks for blocks of `ntask` warps; false when a task's tables do not fit.
bool line_groups(const LinePlan &L, int d, bool centres, int ntask, int most, LineGroups *out)
{
	LineGroups &G = *out;
	G = LineGroups();
	G.ntask = ntask;
	const int nrow = (int)L.rows.size();
	// rho tasks: a row's tiles in even shares of up to 4; a few rows at a time, so that a group of consecutive tasks shares
	// few table entries (16 tasks on 4 rows x 4 shares need 128, on 2 x 8 160)
	struct T {
		int r, j0, n;
	};
	auto shares = [&](int r) { return (L.rows[r].nj + kLineTiles - 1) / kLineTiles; };
	std::vector<T> tasks;
	const int rstep = ntask > kLineTasks && shares(0) >= 4 && nrow > 4 ? 4 : 2;
	for (int r2 = 0; r2 < nrow; r2 += rstep)
		for (int i = 0, top = shares(r2); i < top; i++) {
			const int k = (r2 / rstep) % 2 ? top - 1 - i : i;   // back and forth, so that a group across two bands spans few cells
			for (int r = r2; r < std::min(nrow, r2 + rstep); r++) {
				const int64_t nj = L.rows[r].nj, nt = shares(r);   // (nj * k passes 2^31 on lines of 4e5 cells)
				if (k < nt)
					tasks.push_back(T{r, (int)(nj * k / nt), (int)(nj * (k + 1) / nt - nj * k / nt)});
			}
		}
	const size_t ngroup = (tasks.size() + most - 1) / most;
	for (size_t t0 = 0, g = 0; t0 < tasks.size(); g++) {
		size_t want = (tasks.size() * (g + 1) + ngroup - 1) / ngroup;   // even groups
		want = std::max(want, t0 + 1);
		Span a, b, c, h;
		LineTabs tabs = {};
		size_t t1 = t0;
		while (t1 < tasks.size() && t1 < want && t1 - t0 < (size_t)most) {
			Span na = a, nb = b, nc = c, nh = h;
			for (int i = 0; i < kLineRow; i++) {
				const LineIdx &x = L.lines[(size_t)tasks[t1].r * kLineRow + i];
				na.add(x.p0);
				nb.add(x.p1);
				nc.add(x.c);
			}
			nh.add(4 * tasks[t1].j0);
			nh.add(4 * (tasks[t1].j0 + tasks[t1].n) - 1);
			if ((int64_t)na.hi - na.lo > kLineMaxRow || (int64_t)nb.hi - nb.lo > kLineMaxRow ||
			    (int64_t)nc.hi - nc.lo > kLineMaxRow)
				break;
			const LineTabs n = line_tabs(d, centres, na, nb, nc, nh.lo, nh.n(), kRhoRowMod);
			if (n.row > kLineMaxRow)
				break;
			a = na, b = nb, c = nc, h = nh;
			tabs = n;
			t1++;
		}
		if (t1 == t0)
			return false;
		tabs.ntask = (int)(t1 - t0);
		G.row = std::max(G.row, tabs.row);
		G.groups.push_back(tabs);
		// warp w runs on the SM's sub-partition w mod 4, each with its own FP64 unit: the tasks, largest first, go to the
		// sub-partition with the least work
		std::vector<T> mine(tasks.begin() + t0, tasks.begin() + t1), at((size_t)ntask, T{0, 0, 0});
		std::stable_sort(mine.begin(), mine.end(), [](const T &x, const T &y) { return x.n > y.n; });
		int load[4] = {0, 0, 0, 0}, used[4] = {0, 0, 0, 0};
		for (const T &x : mine) {
			int s = -1;
			for (int q = 0; q < 4; q++)
				if (used[q] < ntask / 4 && (s < 0 || load[q] < load[s]))
					s = q;
			at[(size_t)(4 * used[s] + s)] = x;
			used[s]++;
			load[s] += x.n;
		}
		// a unit is 4 DMMAs of 16 cycles per 4 particles; an entry about 21 cycles per 32
		G.cycles += 16.0 * *std::max_element(load, load + 4) + 0.165 * tabs.row;
		for (const T &x : at) {
			const LineTask k = x.n ? LineTask{L.rows[x.r].ubase + x.j0, x.n, tabs.offh + 4 * x.j0 - tabs.hlo, x.r}
			                       : LineTask{0, 0, 0, 0};
			G.tasks.push_back(k);
			for (int i = 0; i < kLineRow; i++) {
				const LineIdx &l = L.lines[(size_t)k.row * kLineRow + i];
				G.tlines.push_back(k.n ? LineIdx{tabs.off[0] + l.p0 - tabs.lo[0],
				                                 d == 3 ? tabs.off[1] + l.p1 - tabs.lo[1] : 0,
				                                 centres ? tabs.off[2] + l.c - tabs.lo[2] : 0, 0}
				                       : LineIdx{0, 0, 0, 0});
			}
		}
		t0 = t1;
	}
	G.cycles /= (double)G.groups.size();
	return true;
}

}  // namespace

LinePlan build_line_plan(const Plan &p)
{
	LinePlan L;
	const int d = p.d, nseg = (int)p.segs.size();
	if (d < 2 || p.real_segs < 1)
		return L;
	// lines: the (sorted) segments of one prefix without a gap of more than 8 last indices
	std::vector<Line> lines;
	for (int q = 0; q < nseg; q++) {
		const Seg &s = p.segs[q];
		if (s.len == 0)
			continue;
		if (std::abs((int64_t)s.start) > (1 << 28))
			return L;
		const int last = s.start + s.len - 1;
		if (!lines.empty() && lines.back().ix.p0 == s.p0 && lines.back().ix.p1 == s.p1 && s.start - lines.back().b <= 8) {
			lines.back().b = last;
			lines.back().s1 = q + 1;
		} else {
			lines.push_back(Line{LineIdx{s.p0, s.p1, 0, 0}, 0, s.start, last, q, q + 1});
		}
	}
	// centres: all 0 (no centre factor in the kernels) unless centring each line saves more than a seventh of the cells
	int64_t at0 = 0, centred = 0;
	for (const Line &l : lines) {
		at0 += std::max(std::abs(l.a), std::abs(l.b)) / 4 + 1;
		centred += ((l.b - l.a + 1) / 2) / 4 + 1;
	}
	const bool centres = 7 * at0 > 8 * centred + 56;
	for (Line &l : lines) {
		l.ix.c = centres ? l.a + (l.b - l.a) / 2 : 0;
		l.hmax = std::max(std::abs(l.a - l.ix.c), std::abs(l.b - l.ix.c));
	}
	std::stable_sort(lines.begin(), lines.end(), [](const Line &x, const Line &y) { return x.hmax / 4 > y.hmax / 4; });
	// rows and units
	const int nrow = (int)((lines.size() + kLineRow - 1) / kLineRow);
	int64_t nunit = 0;
	for (int r = 0; r < nrow; r++) {
		const int nj = lines[(size_t)r * kLineRow].hmax / 4 + 1;
		L.rows.push_back(LineRow{(int)nunit, nj});
		nunit += nj;
		if (nunit > (1 << 20))
			return L;
	}
	// A unit costs what 128 slots cost at the matrix unit's rate whether it is full or not; a slot of the segment kernels
	// costs about 3.5 times as much (12 FP64 operations at 60 % of the pipe against 6 at 90 %).
	if ((double)nunit * 128.0 > 3.5 * 8.0 * (double)std::max<int64_t>(p.real_segs, kGroupSegs))
		return L;
	L.nunit = (int)nunit;
	L.lines.resize((size_t)nrow * kLineRow);
	L.cells.assign((size_t)nunit * 64, LineCell{-1, -1, 0, 0});
	L.cellV.assign((size_t)nunit * 128, 0.0);
	for (size_t q = 0; q < L.lines.size(); q++) {
		const Line &l = lines[std::min(q, lines.size() - 1)];
		L.lines[q] = l.ix;
		const LineRow &R = L.rows[q / kLineRow];
		const int i = (int)(q % kLineRow);
		auto cell = [&](int h) { return ((size_t)(R.ubase + h / 4) * 2 + i / 8) * 32 + 4 * (i % 8) + h % 4; };
		for (int h = 0; h < 4 * R.nj; h++)
			L.cells[cell(h)].h = h;
		if (q >= lines.size())
			continue;
		for (int k = l.s0; k < l.s1; k++)
			for (int m = 0; m < p.segs[k].len; m++) {
				const int h = p.segs[k].start + m - l.ix.c, slot = m * nseg + k;
				const size_t c = cell(std::abs(h));
				(h >= 0 ? L.cells[c].sp : L.cells[c].sm) = slot;
				L.cellV[2 * c + (h >= 0 ? 0 : 1)] = p.slotV[(size_t)slot];
			}
	}
	int ntotal = 0;
	for (int r = 0; r < nrow; r++)
		ntotal += (L.rows[r].nj + kLineTiles - 1) / kLineTiles;
	struct {
		int warps, tasks;
	} want[3] = {{kLineTasks, kLineTasks}, {0, 0}, {0, 0}};
	if (ntotal > kLineTasks / 2 && ntotal <= 4 * kLineMaxTasks)
		want[1] = {kLineTasks, kLineTasks / 2};
	if (ntotal > kLineTasks)
		want[2].warps = want[2].tasks = std::min(kLineMaxTasks, (ntotal + 3) / 4 * 4);
	for (const auto &w : want)
		if (w.warps) {
			L.groupings.emplace_back();
			if (!line_groups(L, d, centres, w.warps, w.tasks, &L.groupings.back()))
				return LinePlan();   // one task's tables do not fit
		}
	// force phases: the whole set when its tables fit, else chunks of kLineForceCells cells and of rows
	const int hall = 4 * (nrow ? L.rows[0].nj : 0);
	for (int whole = 1; whole >= 0 && L.phases.empty(); whole--) {
		const int hstep = whole ? hall : kLineForceCells;
		for (int h0 = 0; h0 < hall; h0 += hstep) {
			int rmax = 0;   // rows with cells in this chunk (rows are sorted by decreasing extent)
			while (rmax < nrow && 4 * L.rows[rmax].nj > h0)
				rmax++;
			const int nh = std::min(hstep, hall - h0);
			for (int r0 = 0; r0 < rmax;) {
				Span a, b, c;
				LineTabs tabs = {};
				int r1 = r0;
				while (r1 < rmax) {
					Span na = a, nb = b, nc = c;
					for (int i = 0; i < kLineRow; i++) {
						const LineIdx &x = L.lines[(size_t)r1 * kLineRow + i];
						na.add(x.p0);
						nb.add(x.p1);
						nc.add(x.c);
					}
					if ((int64_t)na.hi - na.lo > kLineMaxRow || (int64_t)nb.hi - nb.lo > kLineMaxRow ||
					    (int64_t)nc.hi - nc.lo > kLineMaxRow)
						break;
					const LineTabs n = line_tabs(d, centres, na, nb, nc, h0, nh, kForceRowMod);
					if (n.row > kLineMaxRow)
						break;
					a = na, b = nb, c = nc;
					tabs = n;
					r1++;
				}
				if (r1 == r0 || (whole && r1 < rmax)) {
					if (!whole)
						return LinePlan();
					L.phases.clear();
					h0 = hall;
					break;
				}
				tabs.r0 = r0;
				tabs.ntask = r1 - r0;
				L.phase_row = std::max(L.phase_row, tabs.row);
				L.phases.push_back(tabs);
				r0 = r1;
			}
		}
	}
	L.ok = true;
	return L;
}

// The line kernels' grids.
// rho: the grouping and the particle splits (multiples of 8 particles) with the least estimated time: whole waves of blocks,
// each with a fixed cost and its FP64 cycles at a rate, plus a cost per partial row (the reduction). The constants are a fit
// to 490 timings of evaluations on B200 (2D and 3D, N = 300 to 100000, every grouping, 8 to 1024 particles per split);
// what it picks is within 8 % of the best of them, mostly the best. Two blocks of 8 warps share an SM at 1846 cycles per us
// (of 1965), one alone reaches 1124, a block of 12 or 16 warps 1726: 3D N=2000 chi=0.45 takes 13.3 us with 3 groups of 4
// tasks and 24 particles a split, 13.7 with 2 of 8, 14.0 with one of 12; 2D N=1e5 1.95 ms with groups of 8, 2.03 of 16; 2D
// N=7001 26.7 with one wave of wide blocks, 28.4 with groups of 8.
// force: tiles of 8 particles per block and warps per block, by whole waves of what one wave measured (3D, 67 units: 9.4,
// 15.2, 20.6 and 28.7 us for 1 to 4 tiles with 8 warps, two blocks to an SM; 9.0, 11.8 and 16.8 for 2 to 4 tiles with 16).
constexpr double kLineFixedUs = 1.5, kLineRowUs = 0.012;

LineLaunch line_launch(const LinePlan &p, int d, int64_t N, int sms)
{
	LineLaunch l;
	l.nsplit = 1;
	l.per_split = 8;
	double best = 1e300;
	for (size_t gi = 0; gi < p.groupings.size(); gi++) {
		const LineGroups &g = p.groupings[gi];
		const int64_t G = std::max<int64_t>(1, (int64_t)g.count());
		const bool two = g.ntask <= kLineTasks;
		const int64_t wave = (two ? 2 : 1) * (int64_t)sms, maxns = std::max<int64_t>(1, std::min<int64_t>((N + 7) / 8, kLineMaxSplits));
		for (int64_t ns = 1; ns <= maxns; ns++) {
			const int64_t per = std::max<int64_t>(8, ((N + ns - 1) / ns + 7) / 8 * 8),
			              real = std::max<int64_t>(1, (N + per - 1) / per);
			const int64_t full = G * real / wave, rest = G * real - full * wave;
			const double cyc = (double)per * g.cycles;
			const double full_us = two ? 0.55 + 2.0 * cyc / 1846.0 : 0.28 + cyc / 1726.0;
			const double last_us = rest == 0 ? 0.0 : two && rest <= sms ? 0.72 + cyc / 1124.0 : full_us;
			const double c = (double)full * full_us + last_us + (double)real * kLineRowUs;
			if (c < best) {
				best = c;
				l.grouping = (int)gi;
				l.nsplit = (int)real;
				l.per_split = (int)per;
			}
			if (G * real > 8LL * sms)
				break;
		}
	}
	l.rho_us = best;
	// chunks: a power of two that holds a split, or as many particles as fit (and have a thread per coordinate)
	const LineGroups &g = p.groupings[l.grouping];
	const size_t row = (size_t)g.row * 2 * sizeof(double);
	const size_t room = (g.ntask <= kLineTasks ? 100 : 204) * 1024;
	const int most = std::min(kLineMaxChunk, g.ntask * 32 / d);
	l.chunk = 8;
	while (l.chunk < l.per_split && 2 * l.chunk <= most && 2 * l.chunk * row <= room)
		l.chunk *= 2;
	// force
	best = 1e300;
	static const struct {
		int mt, warps;
		double unit_us;   // per unit and wave
	} opt[] = {{1, 8, 0.117}, {2, 8, 0.205}, {3, 8, 0.285}, {4, 8, 0.406}, {2, 16, 0.112}, {3, 16, 0.154}, {4, 16, 0.228}};
	l.mt = 1;
	l.fwarps = 8;
	for (const auto &o : opt) {
		const double waves = (double)((N + 8 * o.mt - 1) / (8 * o.mt)) / ((o.warps == 8 ? 2.0 : 1.0) * sms);
		// few waves: whole ones; many: the blocks of a new wave start as those of the last one end
		const double whole = waves < 4.0 ? std::ceil(waves) : waves + 0.5;
		const double c = whole * (kLineFixedUs + o.unit_us * p.nunit);
		if (c < best) {
			best = c;
			l.waves = whole;
			l.mt = o.mt;
			l.fwarps = o.warps;
		}
	}
	l.force_us = best;
	return l;
}

// Segment or line kernels for N particles. The line kernels do fewer operations per particle and mode, but a block takes all of
// a set's units (forces) or a share of them (rho) one after another, however few particles there are; the segment kernels
// split the modes over the SMs too. Both estimates, in us, are fits to 1500 evaluations of sets with a line plan on B200 (lines of
// 41 to 2001 modes, discs and balls of radius 8 to 250, shells, triangles, boxes of density 0.1 to 1, 2D and 3D, N = 1 to
// 40000); the choice is within 5 % of the faster one in 96 % of them, and at most a third off. Measured, segments against lines: 2D
// disc of radius 250 (98000 modes) N=100 41 / 108 us, N=1000 147 / 125; 3D ball of radius 30 (57000) N=100 32 / 67, N=1000
// 105 / 79; 16 lines of 2001 N=100 28 / 62, N=1000 120 / 68; 2D disc of radius 60 N=100 19 / 12; stealthy sets of chi < 0.5 take
// lines at every N. Without forces: disc of 250, N=100, 26 / 40.
bool lines_preferred(const Plan &p, const LinePlan &L, const LineLaunch &g, int64_t N, bool forces)
{
	const double n = (double)N, segs = (double)std::min<int64_t>(p.real_segs, 2000);
	const double pairs = n * p.nslot, tables = n * p.nbgroups() * p.block_max_row;
	if (!forces) {
		const double seg = 7.76 + 0.58e-6 * pairs + 4.69e-6 * tables + 2.47e-3 * segs + 0.21e-3 * n;
		return 4.64 + 1.1 * g.rho_us + 0.0476 * L.nunit <= seg;
	}
	const double seg = 12.2 + 1.147e-6 * pairs + 8.12e-6 * tables + 7.27e-3 * segs + (N < 64 ? 3.6 : 0.0) + 0.097e-3 * n;
	const double rows = (p.d == 3 ? 0.19 : 0.026) * (double)L.rows.size();
	const double line = 4.32 + 1.108 * g.rho_us + 0.879 * g.force_us + g.waves * (2.12 * ((double)L.phases.size() - 1.0) + rows) +
	                    0.116e-3 * n;
	return line <= 1.05 * seg;
}

bool cell_geometry(int d, const double *a, double *volume, double *recip)
{
	double inv[9] = {0};
	double det;
	if (d == 1) {
		det = a[0];
		if (det == 0)
			return false;
		inv[0] = 1.0 / det;
	} else if (d == 2) {
		det = a[0] * a[3] - a[1] * a[2];
		if (det == 0)
			return false;
		inv[0] = a[3] / det;
		inv[1] = -a[1] / det;
		inv[2] = -a[2] / det;
		inv[3] = a[0] / det;
	} else {
		const double c00 = a[4] * a[8] - a[5] * a[7], c01 = a[5] * a[6] - a[3] * a[8], c02 = a[3] * a[7] - a[4] * a[6];
		det = a[0] * c00 + a[1] * c01 + a[2] * c02;
		if (det == 0)
			return false;
		// inverse = adjugate / det
		inv[0] = c00 / det;
		inv[3] = c01 / det;
		inv[6] = c02 / det;
		inv[1] = (a[2] * a[7] - a[1] * a[8]) / det;
		inv[4] = (a[0] * a[8] - a[2] * a[6]) / det;
		inv[7] = (a[1] * a[6] - a[0] * a[7]) / det;
		inv[2] = (a[1] * a[5] - a[2] * a[4]) / det;
		inv[5] = (a[2] * a[3] - a[0] * a[5]) / det;
		inv[8] = (a[0] * a[4] - a[1] * a[3]) / det;
	}
	if (!std::isfinite(det))
		return false;
	*volume = std::fabs(det);
	// b_e = 2 pi (row e of inv^T) = 2 pi (column e of inv)
	for (int e = 0; e < d; e++)
		for (int c = 0; c < d; c++)
			recip[e * d + c] = kTwoPi * inv[c * d + e];
	return true;
}

bool cartesian_to_modes(int d, const double *basis, int64_t M, const double *k, int32_t *modes)
{
	for (int64_t m = 0; m < M; m++)
		for (int e = 0; e < d; e++) {
			double x = 0;
			for (int c = 0; c < d; c++)
				x += k[m * d + c] * basis[e * d + c];
			x /= kTwoPi;
			const double r = std::nearbyint(x);
			if (!std::isfinite(x) || std::fabs(x - r) > 1e-9 * std::max(1.0, std::fabs(x)) || std::fabs(r) > 1e9)
				return false;
			modes[m * d + e] = (int32_t)r;
		}
	return true;
}

bool stealthy_kset(int d, const double *basis, int64_t N, double chi, int type, std::vector<int32_t> &modes,
                   std::vector<double> &V)
{
	double vol, recip[9];
	if (!cell_geometry(d, basis, &vol, recip))
		return false;
	const double want_d = std::ceil(chi * (double)N * d);
	if (!(want_d < 5e7))
		return false;
	const size_t want = (size_t)want_d;
	// the CLI's radius: half the diagonal of a cube of 2 d want reciprocal cells
	const double maxk = (std::sqrt((double)d) / 2) * std::pow(2 * (double)d * (double)want, 1.0 / d) *
	                    (kTwoPi / std::pow(vol, 1.0 / d));
	int64_t bound[3] = {0, 0, 0};
	double box = 1;
	for (int e = 0; e < d; e++) {
		double alen = 0;
		for (int c = 0; c < d; c++)
			alen += basis[e * d + c] * basis[e * d + c];
		bound[e] = (int64_t)std::floor(maxk * std::sqrt(alen) / kTwoPi) + 1;
		box *= 2.0 * bound[e] + 1;
	}
	if (box > 4e8)
		return false;
	struct Cand {
		double k2;
		int32_t n[3];
	};
	std::vector<Cand> c;
	int64_t n[3] = {0, 0, 0};
	const int64_t lo0 = 0;   // half space: the first index is >= 0
	for (n[0] = lo0; n[0] <= bound[0]; n[0]++)
		for (n[1] = (d >= 2 ? -bound[1] : 0); n[1] <= (d >= 2 ? bound[1] : 0); n[1]++)
			for (n[2] = (d >= 3 ? -bound[2] : 0); n[2] <= (d >= 3 ? bound[2] : 0); n[2]++) {
				int sign = 0;
				for (int e = 0; e < d && sign == 0; e++)
					sign = n[e] > 0 ? 1 : (n[e] < 0 ? -1 : 0);
				if (sign <= 0)
					continue;
				double k[3] = {0, 0, 0};
				for (int e = 0; e < d; e++)
					for (int cc = 0; cc < d; cc++)
						k[cc] += (double)n[e] * recip[e * d + cc];
				double k2 = 0;
				for (int cc = 0; cc < d; cc++)
					k2 += k[cc] * k[cc];
				if (!(k2 < maxk * maxk))   // the enumeration radius is exclusive
					continue;
				Cand x;
				x.k2 = k2;
				for (int e = 0; e < 3; e++)
					x.n[e] = (int32_t)n[e];
				c.push_back(x);
			}
	std::sort(c.begin(), c.end(), [](const Cand &a, const Cand &b) {
		if (a.k2 != b.k2)
			return a.k2 < b.k2;
		for (int e = 0; e < 3; e++)
			if (a.n[e] != b.n[e])
				return a.n[e] < b.n[e];
		return false;
	});
	size_t count = 0;
	double last = 0;
	while (count < c.size()) {
		if (!(count < want || std::fabs((last - c[count].k2) / last) < 1e-10))
			break;
		last = c[count].k2;
		count++;
	}
	const double K2 = count < c.size() ? c[count].k2 : 0.0;
	modes.resize(count * d);
	V.resize(count);
	for (size_t m = 0; m < count; m++) {
		for (int e = 0; e < d; e++)
			modes[m * d + e] = c[m].n[e];
		double w = 1.0;
		if (type >= 1 && type <= 3 && K2 > 0) {
			const double x = std::sqrt(c[m].k2 / K2);
			if (type == 1)
				w = std::acos(x) - x * std::sqrt(1 - c[m].k2 / K2);
			else if (type == 2)
				w = std::pow(1.0 - x, 6.0);
			else
				w = std::pow(1.0 - x, 2.0);
		}
		V[m] = w;
	}
	return true;
}

namespace {

int64_t gcd64(int64_t a, int64_t b)
{
	a = a < 0 ? -a : a;
	b = b < 0 ? -b : b;
	while (b) {
		const int64_t t = a % b;
		a = b;
		b = t;
	}
	return a;
}

// Cartesian k = sum_e n_e b_e, accumulated axis by axis from zero (as GeometryVector sums), and k.k.
void lattice_k(int d, const double *recip, const int64_t *n, double *k)
{
	for (int x = 0; x < d; x++)
		k[x] = 0.0;
	for (int e = 0; e < d; e++)
		for (int x = 0; x < d; x++)
			k[x] = k[x] + (double)n[e] * recip[e * d + x];
}

double mod2(int d, const double *k)
{
	double s = 0.0;
	for (int x = 0; x < d; x++)
		s += k[x] * k[x];
	return s;
}

double dot(int d, const double *u, const double *v)
{
	double s = 0.0;
	for (int x = 0; x < d; x++)
		s += u[x] * v[x];
	return s;
}

// Reciprocal basis formed as the reference's cell forms it (core/PeriodicCellList.h:999-1030): b_i = a_i minus its
// projections on the Gram-Schmidt orthogonalised other basis vectors, scaled by 2 pi / (b_i . a_i). Same algebra as
// cell_geometry's inverse, but the same rounding as the reference, so lattice vectors of equal length compare equal
// (and order) exactly as there.
void reciprocal_by_projection_impl(int d, const double *a, double *recip)
{
	for (int i = 0; i < d; i++) {
		double r[3], ortho[2][3];
		int no = 0;
		for (int x = 0; x < d; x++)
			r[x] = a[i * d + x];
		for (int j = 0; j < d; j++) {
			if (j == i)
				continue;
			double t[3];
			for (int x = 0; x < d; x++)
				t[x] = a[j * d + x];
			for (int o = 0; o < no; o++) {
				const double c = dot(d, t, ortho[o]) / mod2(d, ortho[o]);
				for (int x = 0; x < d; x++)
					t[x] -= ortho[o][x] * c;
			}
			for (int x = 0; x < d; x++)
				ortho[no][x] = t[x];
			no++;
		}
		for (int o = 0; o < no; o++) {
			const double c = dot(d, ortho[o], r) / mod2(d, ortho[o]);
			for (int x = 0; x < d; x++)
				r[x] -= ortho[o][x] * c;
		}
		const double sc = 2.0 * M_PI / dot(d, r, a + i * d);
		for (int x = 0; x < d; x++)
			recip[i * d + x] = r[x] * sc;
	}
}

}  // namespace

void reciprocal_by_projection(int d, const double *basis, double *recip)
{
	reciprocal_by_projection_impl(d, basis, recip);
}

bool isotropic_ks(int d, const double *basis, double circ_kmax, double lin_kmax, double sample_prob, double circ_kmin,
                  std::vector<int32_t> &modes, std::vector<double> &kamp, size_t max_ks)
{
	modes.clear();
	kamp.clear();
	double vol = 0.0, recip[9];
	if (d < 1 || d > 3 || !cell_geometry(d, basis, &vol, recip))
		return false;
	if (!(circ_kmax > 0.0) || !(lin_kmax > 0.0))
		return true;
	reciprocal_by_projection_impl(d, basis, recip);
	std::mt19937 rng(98765u);
	auto keep = [&]() { return sample_prob >= 1.0 || (double)rng() / 4294967296.0 < sample_prob; };
	auto push = [&](int64_t n0, int64_t n1, int64_t n2, double amp) {
		const int64_t n[3] = {n0, n1, n2};
		for (int e = 0; e < d; e++) {
			if (n[e] > INT32_MAX || n[e] < INT32_MIN)
				return false;
			modes.push_back((int32_t)n[e]);
		}
		kamp.push_back(amp);
		return kamp.size() <= max_ks;
	};
	if (d == 1) {
		const double b = recip[0];
		if (!(b > 0.0))
			return false;
		if (circ_kmin <= 0.0) {
			for (int64_t i = 1;; i++) {
				const double kx = (double)i * b;
				if (kx > lin_kmax)
					break;
				if (keep() && !push(i, 0, 0, std::sqrt(kx * kx)))
					return false;
			}
			return true;
		}
		std::vector<int64_t> seed;
		std::vector<double> seedk;
		for (int64_t i = 1;; i++) {
			const double kx = (double)i * b;
			if (kx > circ_kmax)
				break;
			if (kx > circ_kmin && keep()) {
				if (!push(i, 0, 0, std::sqrt(kx * kx)))
					return false;
				seed.push_back(i);
				seedk.push_back(kx);
			}
		}
		if (seed.empty())
			return true;
		for (int64_t i = 2;; i++) {
			for (size_t j = 0; j < seed.size(); j++) {
				const double kx = (double)i * seedk[j];
				if (kx > lin_kmax)
					return true;
				if (keep() && !push(i * seed[j], 0, 0, std::sqrt(kx * kx)))
					return false;
			}
		}
	}
	// d >= 2: half-space points of the circle, by (|k|^2, k_x)
	int64_t lim[3] = {0, 0, 0};
	for (int e = 0; e < d; e++) {
		double a2 = 0.0;
		for (int x = 0; x < d; x++)
			a2 += basis[e * d + x] * basis[e * d + x];
		lim[e] = (int64_t)std::ceil(circ_kmax * std::sqrt(a2) / (2.0 * M_PI));
		if (lim[e] > 100000)
			return false;
	}
	struct P {
		int64_t n[3];
		double k2, kx;
	};
	std::vector<P> circle;
	const double K2 = circ_kmax * circ_kmax, Kmin2 = circ_kmin * circ_kmin;
	// the reference's odometer order (axis 0 fastest): std::sort below then orders ties as the reference's does
	int64_t n[3] = {0, 0, 0};
	for (n[2] = (d == 3 ? -lim[2] : 0); n[2] <= (d == 3 ? lim[2] : 0); n[2]++)
		for (n[1] = -lim[1]; n[1] <= lim[1]; n[1]++)
			for (n[0] = -lim[0]; n[0] <= lim[0]; n[0]++) {
				int first = 0;
				for (int e = 0; e < d && first == 0; e++)
					first = n[e] > 0 ? 1 : n[e] < 0 ? -1 : 0;
				if (first < 0)
					continue;   // the inverted half (k = 0 fails the k^2 > kmin^2 test below)
				double k[3];
				lattice_k(d, recip, n, k);
				const double k2 = mod2(d, k);
				if (k2 < K2 && k2 > Kmin2) {
					circle.push_back({{n[0], n[1], n[2]}, k2, k[0]});
					if (circle.size() > max_ks)
						return false;
				}
			}
	std::sort(circle.begin(), circle.end(), [](const P &a, const P &b) {
		if (a.k2 != b.k2)
			return a.k2 < b.k2;
		return a.kx < b.kx;
	});
	if (lin_kmax == circ_kmax) {
		for (const P &q : circle)
			if (!push(q.n[0], q.n[1], q.n[2], std::sqrt(q.k2)))
				return false;
		return true;
	}
	// the first point of each lattice direction (directions compared as primitive integer vectors)
	std::set<std::array<int64_t, 3> > seen;
	std::vector<P> first;
	for (const P &q : circle) {
		int64_t g = 0;
		for (int e = 0; e < d; e++)
			g = gcd64(g, q.n[e]);
		std::array<int64_t, 3> key = {q.n[0] / g, q.n[1] / g, d == 3 ? q.n[2] / g : 0};
		if (!seen.insert(key).second)
			continue;
		first.push_back(q);
	}
	const double L2 = lin_kmax * lin_kmax;
	for (const P &q : first) {
		double k[3];
		lattice_k(d, recip, q.n, k);
		for (int64_t i = 1;; i++) {
			double t[3];
			for (int x = 0; x < d; x++)
				t[x] = (double)i * k[x];
			const double t2 = mod2(d, t);
			if (t2 > L2)
				break;
			if (keep() && !push(i * q.n[0], i * q.n[1], i * q.n[2], std::sqrt(t2)))
				return false;
		}
	}
	return true;
}

}  // namespace cc
