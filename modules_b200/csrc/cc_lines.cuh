// cc_lines.cuh — the FP64 direct sums as contractions on the FP64 matrix unit (DMMA, mma.sync.m8n8k4.f64).
//
// The phase of a mode factors over the axes: with the prefix (p0[, p1]) and the last index c + h of a mode,
//     exp(2 pi i n.s) = X(p, c) w^h,  X = T0(p0) [T1(p1)] [Tc(c)],  w = exp(2 pi i s_last),  w^h = C_h + i S_h,
// so over the particles j, for the two modes +h and -h of a line (cc_plan.h LinePlan)
//     rho(c + h) = A_h + i B_h,  rho(c - h) = A_h - i B_h,  A_h = sum_j X_j C_jh,  B_h = sum_j X_j S_jh:
// a matrix product [lines x particles] . [particles x cells] with real right-hand factors, 2 multiply-adds per mode and
// particle (the recurrences of cc_kernels.cuh spend 4 operations and the seeds). The forces need, per particle and line,
//     T = sum_m u_m w^(m - c) = sum_h a_h C_h + i b_h S_h,         a = u_+ + u_-, b = u_+ - u_-,
//     D = sum_m (m - c) u_m w^(m - c) = sum_h h (b_h C_h + i a_h S_h),
// [particles x cells] . [cells x lines], 4 multiply-adds per mode and particle; then g_p += p Im(X T),
// g_last += c Im(X T) + Im(X D).
//
// What bounds it: the FP64 pipe, which DMMA and DFMA share (measured on B200: 37.0 TFLOP/s of DMMA from four warps per
// SM on, 34.0 of register-only DFMA, 25 of DFMA whose second factor comes from shared memory: a DMMA takes each operand
// from one lane instead of broadcasting it to 32). Tables hold every phase that is used, from exactly reduced arguments
// (8 entries from each sincospi), so no recurrence error grows along a line.
//
// Fragments of mma.m8n8k4 (lane = 4 g + t): A[g][t], B[t][g], C[g][2t], C[g][2t + 1]. The order within the contraction
// index and within the columns is free as long as both factors agree on it; the layouts below are chosen so that a lane
// holds all of a cell (rho) and so that the weights of the forces are read in fragment order.
#pragma once
#include <type_traits>
#include "cc_kernels.cuh"

namespace cc {

constexpr int kLineThreads = 256;

__device__ __forceinline__ void dmma(double2 &c, double a, double b)
{
	asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
	    : "+d"(c.x), "+d"(c.y)
	    : "d"(a), "d"(b));
}

// The same with 16 rows and contraction length 8: rows g (c0) and g + 8 (c1); a[i][k]: row g + 8 i, index t + 4 k; b[k].
__device__ __forceinline__ void dmma16(double2 &c0, double2 &c1, double a00, double a10, double a01, double a11, double b0,
                                       double b1)
{
	asm("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
	    : "+d"(c0.x), "+d"(c0.y), "+d"(c1.x), "+d"(c1.y)
	    : "d"(a00), "d"(a10), "d"(a01), "d"(a11), "d"(b0), "d"(b1));
}

// Tables. An item is E = 8 or 16 consecutive entries of one run of one particle (row: its table, s: its coordinates): the
// first entry and the step from exactly reduced sincospi, the rest by products; with E = 16 the second half starts from
// z_8 = z_0 ((w^2)^2)^2, so that two chains run side by side and no entry is more than 11 products away from sincospi. An
// item longer than 8 halves the sincospi per entry, a shorter one the latency. A particle that does not exist gets zeros,
// so it adds nothing.
template <int E> __device__ __forceinline__ int line_items(const LineTabs &tb)
{
	return E == 8 ? tb.items : tb.items16;
}
template <int D, int E>
__device__ __forceinline__ void build_line_item(const LineTabs &tb, int k, const double *s, bool exists, double2 *row)
{
	const int b0 = (tb.n[0] + E - 1) / E, b1 = b0 + (tb.n[1] + E - 1) / E, b2 = b1 + (tb.n[2] + E - 1) / E;
	int axis, lo, n, off, k0;
	if (k < b0) {
		axis = 0;
		lo = tb.lo[0];
		n = tb.n[0];
		off = tb.off[0];
		k0 = E * k;
	} else if (k < b1) {
		axis = D == 3 ? 1 : D - 1;
		lo = tb.lo[1];
		n = tb.n[1];
		off = tb.off[1];
		k0 = E * (k - b0);
	} else if (k < b2) {
		axis = D - 1;
		lo = tb.lo[2];
		n = tb.n[2];
		off = tb.off[2];
		k0 = E * (k - b1);
	} else {
		axis = D - 1;
		lo = tb.hlo;
		n = tb.nh;
		off = tb.offh;
		k0 = E * (k - b2);
	}
	const int cn = min(E, n - k0);
	double2 *dst = row + off + k0;
	if (!exists) {
		for (int e = 0; e < cn; e++)
			dst[e] = make_double2(0.0, 0.0);
		return;
	}
	const double x = s[axis];
	double2 z = expi2pi(phase1(lo + k0, x));
	const double2 w = expi2pi(phase1(1, x));
	if (E == 16 && cn > 8) {
		double2 w8 = cmul(w, w);
		w8 = cmul(w8, w8);
		w8 = cmul(w8, w8);
		double2 y = cmul(z, w8);
		for (int e = 0; e < 8; e++) {
			dst[e] = z;
			if (8 + e < cn)
				dst[8 + e] = y;
			z = cmul(z, w);
			y = cmul(y, w);
		}
	} else {
		for (int e = 0; e < cn; e++) {
			dst[e] = z;
			z = cmul(z, w);
		}
	}
}

// The tables of `cnt` particles at pos (cnt x D fractional coordinates in shared memory), rows of tabs.row entries, of
// which the first `nvalid` exist, by the whole block. Thread tid builds items of particle tid mod PP (PP = 2^log2pp >=
// cnt): the lanes of a warp write rows that start in different banks (a warp along one row would write all its items to
// the same bank: 8-way conflicts, 28 % of the shared-memory pipe at 2D N=1e5), and the run tests are uniform.
template <int D, int E>
__device__ __forceinline__ void build_line_tables(const LineTabs &tb, const double *pos, int log2pp, int cnt,
                                                  int nvalid, double2 *tab)
{
	const int i = threadIdx.x & ((1 << log2pp) - 1);
	if (i >= cnt)
		return;
	for (int k = threadIdx.x >> log2pp; k < line_items<E>(tb); k += (int)blockDim.x >> log2pp)
		build_line_item<D, E>(tb, k, pos + i * D, i < nvalid, tab + (size_t)i * tb.row);
}

// A 16-byte aligned record copied field by field through the read-only path (one round trip, uniform over the block).
template <typename T> __device__ __forceinline__ T load_rec(const T *p)
{
	static_assert(sizeof(T) % 16 == 0, "records are read as 16-byte words");
	union {
		T v;
		int4 w[sizeof(T) / 16];
	} u;
#pragma unroll
	for (int i = 0; i < (int)(sizeof(T) / 16); i++)
		u.w[i] = __ldg(reinterpret_cast<const int4 *>(p) + i);
	return u.v;
}

// ---------------------------------------------------------------------------------------------------------------
// rho pass
// ---------------------------------------------------------------------------------------------------------------
struct LineRhoArgs {
	const double *frac;       // N x D fractional coordinates
	int N;
	int per_split;            // particles per block (a multiple of 8)
	int chunk, log2chunk;     // particles whose tables are staged at once (a power of two, 8 to 64)
	int ngroup, nunit;
	int ntask;                // warps of a block (8 to 16)
	const LineTabs *groups;
	const LineTask *tasks;    // ngroup x ntask
	const LineIdx *tlines;    // ngroup x ntask x 16
	double2 *partial;         // [nsplit][nunit][2 halves][Re X, Im X][32 lanes]: (A_h, B_h) components
	const int *skip;
	const int *stage;
	int want_stage;
	double *frac_copy;        // as RhoArgs
	int early;                // as RhoArgs
};

// staged coordinates in front of the tables
__host__ __device__ constexpr size_t line_pos_bytes(int particles, int d)
{
	return ((size_t)particles * d * sizeof(double) + 15) / 16 * 16;
}

// Block (group, split): warp w owns task w of the group, 16 lines x up to 16 cells held in registers over all the
// block's particles, eight particles a step. The tables are staged chunk by chunk: every warp builds, then every warp
// contracts (a dependent chain of FP64 operations advances one operation per matrix instruction of its neighbours while
// these run, so the two do not mix well on one SM). The sums of a split are one partial row.
template <int D>
__device__ __forceinline__ void line_rho_body(const LineRhoArgs &a, const int grp, const int split, const ItemCtl ctl)
{
	constexpr int E = 16;
	extern __shared__ __align__(16) unsigned char smem[];
	double *pos = reinterpret_cast<double *>(smem);   // chunk x D
	double2 *tab = reinterpret_cast<double2 *>(smem + line_pos_bytes(a.chunk, D));
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int t = lane & 3, g = lane >> 2;
	// one round trip for everything that does not depend on the positions
	const LineTabs tb = load_rec(a.groups + grp);
	const LineTask task = load_rec(a.tasks + grp * a.ntask + warp);
	const LineIdx l0 = load_rec(a.tlines + (grp * a.ntask + warp) * kLineRow + g);
	const LineIdx l1 = load_rec(a.tlines + (grp * a.ntask + warp) * kLineRow + 8 + g);
	const int j0 = min(a.N, split * a.per_split);
	const int j1 = min(a.N, j0 + a.per_split);
	if (!a.early)
		cudaGridDependencySynchronize();
	if (eval_skipped(a.skip, ctl.stage, ctl.want_stage))
		return;
	const bool centres = tb.n[2] > 0;
	double2 re[2][kLineTiles], im[2][kLineTiles];
#pragma unroll
	for (int r = 0; r < 2; r++)
#pragma unroll
		for (int j = 0; j < kLineTiles; j++)
			re[r][j] = im[r][j] = make_double2(0.0, 0.0);

	// coordinate threadIdx.x of the chunk at c0 (chunk x D <= blockDim.x), loaded a chunk ahead
	auto load = [&](int c0) {
		double v = 0.0;
		if ((int)threadIdx.x < a.chunk * D && c0 + (int)threadIdx.x / D < j1) {
			v = a.frac[(size_t)c0 * D + threadIdx.x];
			if (a.frac_copy && grp == 0)
				a.frac_copy[(size_t)c0 * D + threadIdx.x] = v;
		}
		return v;
	};
	double next = load(j0);
	for (int cj = j0; cj < j1; cj += a.chunk) {
		const int nv = min(a.chunk, j1 - cj), cnt = (nv + 7) & ~7;
		if ((int)threadIdx.x < a.chunk * D)
			pos[threadIdx.x] = next;
		__syncthreads();   // positions in place; the previous chunk's tables are no longer read
		build_line_tables<D, E>(tb, pos, a.log2chunk, a.chunk, nv, tab);
		if (cj + a.chunk < j1)
			next = load(cj + a.chunk);
		__syncthreads();
		const double2 *row = tab + t * tb.row;
		const int up = 4 * tb.row;
		for (int k = 0; k < (task.n ? cnt : 0); k += 8, row += 2 * up) {
			double2 x00 = row[l0.p0], x10 = row[l1.p0], x01 = row[l0.p0 + up], x11 = row[l1.p0 + up];
			if (D == 3) {
				x00 = cmul(x00, row[l0.p1]);
				x10 = cmul(x10, row[l1.p1]);
				x01 = cmul(x01, row[l0.p1 + up]);
				x11 = cmul(x11, row[l1.p1 + up]);
			}
			if (centres) {
				x00 = cmul(x00, row[l0.c]);
				x10 = cmul(x10, row[l1.c]);
				x01 = cmul(x01, row[l0.c + up]);
				x11 = cmul(x11, row[l1.c + up]);
			}
			const double *b = reinterpret_cast<const double *>(row + task.hoff) + g;
#pragma unroll
			for (int j = 0; j < kLineTiles; j++)
				if (j < task.n) {
					const double b0 = b[8 * j], b1 = b[8 * j + 2 * up];   // C_h (g even) or S_h (g odd), h = 4 j + g / 2
					dmma16(re[0][j], re[1][j], x00.x, x10.x, x01.x, x11.x, b0, b1);
					dmma16(im[0][j], im[1][j], x00.y, x10.y, x01.y, x11.y, b0, b1);
				}
		}
	}
	if (a.early)   // as rho_body: only the partial rows wait for the previous evaluation
		cudaGridDependencySynchronize();
	cudaTriggerProgrammaticLaunchCompletion();
	// lane 4 g + t holds cell h = 4 j + t of line g
	double2 *out = a.partial + ((size_t)split * a.nunit + task.u0) * 128 + lane;
#pragma unroll
	for (int j = 0; j < kLineTiles; j++)
		if (j < task.n) {
			out[j * 128] = re[0][j];
			out[j * 128 + 32] = im[0][j];
			out[j * 128 + 64] = re[1][j];
			out[j * 128 + 96] = im[1][j];
		}
}

// (up to 16 warps: 128 registers; blocks of 8 warps run two to an SM)
template <int D> __global__ void __launch_bounds__(512, 1) cc_line_rho_kernel(LineRhoArgs a)
{
	line_rho_body<D>(a, blockIdx.x, blockIdx.y, ItemCtl{a.stage, a.want_stage});
}

// ---------------------------------------------------------------------------------------------------------------
// split reduction, energy, force weights
// ---------------------------------------------------------------------------------------------------------------
struct LineReduceArgs {
	const double2 *partial;   // [nsplit][nunit][128]
	int nsplit, nunit;
	const LineCell *cells;
	const double2 *cellV;     // (plus, minus)
	const double2 *cellS0;    // S2 targets, or null
	double npart;
	double rho_offset;
	double2 *rho_slot;        // rho per slot
	double2 *weights;         // force weights in fragment order (may be null)
	double *eblock;           // [blocks]
	unsigned *ticket;
	double inv_vol, shift;
	double *E_out;
	int finalize;
	const int *skip;
	const int *stage;
	int want_stage;
};

constexpr int kLineRedCells = 8;     // cells per block
constexpr int kLineRedThreads = 256; // 8 cells x 2 components x 16 row chunks

// The force weights of a cell: for comp = 0..3 (T_re, T_im, D_re, D_im) the factors of (C_h, S_h).
__device__ __forceinline__ double2 line_weight(int comp, int h, double2 up, double2 um)
{
	const double2 a = make_double2(up.x + um.x, up.y + um.y), b = make_double2(up.x - um.x, up.y - um.y);
	const double hd = (double)h;
	switch (comp) {
	case 0: return make_double2(a.x, -b.y);
	case 1: return make_double2(a.y, b.x);
	case 2: return make_double2(hd * b.x, -hd * a.y);
	default: return make_double2(hd * b.y, hd * a.x);
	}
}
__device__ __forceinline__ size_t line_weight_at(int cell, int comp)
{
	const int unit = cell >> 6, line = (cell & 63) >> 2, t = cell & 3;   // line of the row, h & 3
	return ((size_t)unit * 8 + (line >> 1)) * 32 + (4 * (line & 1) + comp) * 4 + t;
}

// Sum of the n energy terms of the reduce blocks by 256 threads in a fixed order (valid in thread 0), the same whoever
// sums: the last reduce block of an evaluation without forces, or the force kernel's energy block.
__device__ __forceinline__ double line_energy_sum(const double *eblock, int n)
{
	double *sh = reinterpret_cast<double *>(body_shared().red);
	double e = 0.0;
	for (int b = threadIdx.x; threadIdx.x < kLineThreads && b < n; b += kLineThreads)
		e += __ldcg(eblock + b);
#pragma unroll
	for (int o = 16; o > 0; o >>= 1)
		e += __shfl_down_sync(0xffffffffu, e, o);
	if ((threadIdx.x & 31) == 0 && threadIdx.x < kLineThreads)
		sh[threadIdx.x >> 5] = e;
	__syncthreads();
	e = sh[0];
#pragma unroll
	for (int w = 1; w < 8; w++)
		e += sh[w];
	return e;
}

// Block `item` (8 cells). Every component is summed over the rows in 16 chunks of consecutive rows, each in row order, the
// chunks in order; all loads of a thread are independent, so a block costs about one trip to L2.
__device__ __forceinline__ void line_reduce_body(const LineReduceArgs &a, const int item, const int nitems,
                                                 const ItemCtl ctl)
{
	double2 (&sh)[8][32] = body_shared().red;
	int &sh_last = body_shared().last;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int ci = lane & 7, comp = (lane >> 3) & 1, chunk = 2 * warp + (lane >> 4);
	const int cell0 = item * kLineRedCells;
	// components of cell c: unit * 128 + half * 64 + {0, 32} + lane
	const size_t at = (size_t)(cell0 >> 6) * 128 + ((cell0 >> 5) & 1) * 64 + comp * 32 + (cell0 & 31) + ci;
	const LineCell cl = load_rec(a.cells + cell0 + ci);
	const double2 V = __ldg(a.cellV + cell0 + ci);
	cudaGridDependencySynchronize();
	cudaTriggerProgrammaticLaunchCompletion();
	if (ctl.ready)
		wait_ready(ctl.ready, ctl.ready_need, ctl.err, ctl.ready_spins);
	if (eval_skipped(a.skip, ctl.stage, ctl.want_stage))
		return;
	const int per = (a.nsplit + 15) >> 4;
	const int s0 = min(a.nsplit, chunk * per), s1 = min(a.nsplit, s0 + per);
	const size_t stride = (size_t)a.nunit * 128;
	double2 v = make_double2(0.0, 0.0);
	int s = s0;
	for (; s + 8 <= s1; s += 8) {
		double2 x[8];
#pragma unroll
		for (int i = 0; i < 8; i++)
			x[i] = __ldcg(a.partial + (size_t)(s + i) * stride + at);
#pragma unroll
		for (int i = 0; i < 8; i++) {
			v.x += x[i].x;
			v.y += x[i].y;
		}
	}
	{
		double2 x[8];
#pragma unroll
		for (int i = 0; i < 8; i++)
			if (s + i < s1)
				x[i] = __ldcg(a.partial + (size_t)(s + i) * stride + at);
#pragma unroll
		for (int i = 0; i < 8; i++)
			if (s + i < s1) {
				v.x += x[i].x;
				v.y += x[i].y;
			}
	}
	// the two chunks of a warp, then the warps in order
	v.x += __shfl_down_sync(0xffffffffu, v.x, 16);
	v.y += __shfl_down_sync(0xffffffffu, v.y, 16);
	if (lane < 16)
		sh[warp][lane] = v;
	__syncthreads();
	if (warp == 0) {
		v = sh[0][lane & 15];
#pragma unroll
		for (int w = 1; w < 8; w++) {
			v.x += sh[w][lane & 15].x;
			v.y += sh[w][lane & 15].y;
		}
		// every lane of the cell (4 of them) gets A and B: lane ci holds (Re A, Re B), lane ci + 8 (Im A, Im B)
		const double ar = __shfl_sync(0xffffffffu, v.x, ci), br = __shfl_sync(0xffffffffu, v.y, ci);
		const double ai = __shfl_sync(0xffffffffu, v.x, ci + 8), bi = __shfl_sync(0xffffffffu, v.y, ci + 8);
		const int q = lane >> 3;   // the weight component the lane stores
		double e = 0.0;
		double2 up = make_double2(0.0, 0.0), um = up;
		if (cl.sp >= 0) {
			const double2 r = make_double2(ar - bi + a.rho_offset, ai + br);
			const double r2 = r.x * r.x + r.y * r.y;
			double w = V.x;
			if (a.cellS0) {
				const double ds = r2 / a.npart - __ldg(a.cellS0 + cell0 + ci).x;
				w *= ds;
				e = w * ds;
			} else {
				e = w * r2;
			}
			up = make_double2(w * r.x, -w * r.y);
			if (q == 0)
				a.rho_slot[cl.sp] = r;
		}
		if (cl.sm >= 0) {
			const double2 r = make_double2(ar + bi + a.rho_offset, ai - br);
			const double r2 = r.x * r.x + r.y * r.y;
			double w = V.y;
			if (a.cellS0) {
				const double ds = r2 / a.npart - __ldg(a.cellS0 + cell0 + ci).y;
				w *= ds;
				e += w * ds;
			} else {
				e += w * r2;
			}
			um = make_double2(w * r.x, -w * r.y);
			if (q == 0)
				a.rho_slot[cl.sm] = r;
		}
		if (a.weights)
			a.weights[line_weight_at(cell0 + ci, q)] = line_weight(q, cl.h, up, um);
		// the block's energy: its 8 cells by a fixed tree
		e = q == 0 ? e : 0.0;
#pragma unroll
		for (int o = 4; o > 0; o >>= 1)
			e += __shfl_down_sync(0xffffffffu, e, o);
		if (lane == 0)
			a.eblock[item] = e;
	}
	if (!a.finalize)
		return;
	__threadfence();
	__syncthreads();
	if (threadIdx.x == 0)
		sh_last = (atomicAdd(a.ticket, 1u) == (unsigned)nitems - 1);
	__syncthreads();
	if (!sh_last)
		return;
	__threadfence();
	const double e = line_energy_sum(a.eblock, nitems);
	if (threadIdx.x == 0) {
		*a.E_out = e * a.inv_vol + a.shift;
		*a.ticket = 0u;
	}
}

// Item `item` of the reduction in the batch launch: two units (128 cells, a thread per component), every component summed
// over the rows in row order. Wide items, as reduce_body_wide: a batch's many small reductions cost few of them.
constexpr int kLineWideUnits = 2;
__device__ __forceinline__ void line_reduce_wide_body(const LineReduceArgs &a, const int item, const ItemCtl ctl)
{
	double2 *sh = &body_shared().red[0][0];   // 256 entries
	double *she = body_shared().pos;          // one energy per warp
	const int unit = item * kLineWideUnits + ((int)threadIdx.x >> 7), part = threadIdx.x & 127;
	const int half = part >> 6, comp = (part >> 5) & 1, lane = part & 31;
	const bool on = unit < a.nunit;
	const int cell = unit * 64 + half * 32 + lane;
	LineCell cl = {-1, -1, 0, 0};
	double2 V = make_double2(0.0, 0.0);
	if (on) {
		cl = load_rec(a.cells + cell);
		V = __ldg(a.cellV + cell);
	}
	if (ctl.ready)
		wait_ready(ctl.ready, ctl.ready_need, ctl.err, ctl.ready_spins);
	if (eval_skipped(a.skip, ctl.stage, ctl.want_stage))
		return;
	double2 v = make_double2(0.0, 0.0);
	if (on) {
		const double2 *p = a.partial + (size_t)unit * 128 + part;
		const size_t stride = (size_t)a.nunit * 128;
		int s = 0;
		for (; s + 8 <= a.nsplit; s += 8) {
			double2 x[8];
#pragma unroll
			for (int i = 0; i < 8; i++)
				x[i] = __ldcg(p + (size_t)(s + i) * stride);
#pragma unroll
			for (int i = 0; i < 8; i++) {
				v.x += x[i].x;
				v.y += x[i].y;
			}
		}
		for (; s < a.nsplit; s++) {
			const double2 x = __ldcg(p + (size_t)s * stride);
			v.x += x.x;
			v.y += x.y;
		}
	}
	sh[threadIdx.x] = v;
	__syncthreads();
	const double2 ra = sh[threadIdx.x & ~32], ia = sh[threadIdx.x | 32];   // (Re A, Re B), (Im A, Im B)
	double e = 0.0;
	double2 up = make_double2(0.0, 0.0), um = up;
	if (cl.sp >= 0) {
		const double2 r = make_double2(ra.x - ia.y + a.rho_offset, ia.x + ra.y);
		e = V.x * (r.x * r.x + r.y * r.y);
		up = make_double2(V.x * r.x, -V.x * r.y);
	}
	if (cl.sm >= 0) {
		const double2 r = make_double2(ra.x + ia.y + a.rho_offset, ia.x - ra.y);
		e += V.y * (r.x * r.x + r.y * r.y);
		um = make_double2(V.y * r.x, -V.y * r.y);
	}
	if (on) {
		a.weights[line_weight_at(cell, 2 * comp)] = line_weight(2 * comp, cl.h, up, um);
		a.weights[line_weight_at(cell, 2 * comp + 1)] = line_weight(2 * comp + 1, cl.h, up, um);
	}
	e = comp == 0 ? e : 0.0;
#pragma unroll
	for (int o = 16; o > 0; o >>= 1)
		e += __shfl_down_sync(0xffffffffu, e, o);
	if ((threadIdx.x & 31) == 0)
		she[threadIdx.x >> 5] = e;
	__syncthreads();
	if (threadIdx.x == 0) {
		double t = 0.0;
#pragma unroll
		for (int w = 0; w < 8; w++)
			t += she[w];
		a.eblock[item] = t;
	}
}

static __global__ void __launch_bounds__(kLineRedThreads) cc_line_reduce_kernel(LineReduceArgs a)
{
	line_reduce_body(a, blockIdx.x, gridDim.x, ItemCtl{a.stage, a.want_stage});
}

// The force weights from u per slot (the sub-configurations of the S2 form combine their rho first).
static __global__ void cc_line_weights_kernel(const LineCell *__restrict__ cells, const double2 *__restrict__ u_slot,
                                              int ncell, double2 *__restrict__ weights)
{
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	const int cell = i >> 2, q = i & 3;
	if (cell >= ncell)
		return;
	const LineCell cl = load_rec(cells + cell);
	const double2 zero = make_double2(0.0, 0.0);
	weights[line_weight_at(cell, q)] = line_weight(q, cl.h, cl.sp >= 0 ? u_slot[cl.sp] : zero, cl.sm >= 0 ? u_slot[cl.sm] : zero);
}

// ---------------------------------------------------------------------------------------------------------------
// force pass
// ---------------------------------------------------------------------------------------------------------------
struct LineForceArgs {
	const double *frac;       // N x D
	int N;
	int nphase;
	int tiles, teams;         // in a batch: tiles per item, teams of a block's warps (8 MT particles each)
	const LineTabs *phases;
	const LineRow *rows;
	const LineIdx *lines;     // rows x 16
	const double2 *weights;   // [nunit][8 line pairs][32 lanes]
	double recip[9];
	double fscale;
	double *F_out;
	double *gfrac_out;
	const double *eblock;
	int neblock;
	double inv_vol, shift;
	double *E_out;
	const int *skip;
	const int *stage;
	int want_stage;
};

// The energy, by a block of its own.
__device__ __forceinline__ void line_energy_body(const LineForceArgs &a, const ItemCtl ctl)
{
	cudaGridDependencySynchronize();
	cudaTriggerProgrammaticLaunchCompletion();
	if (ctl.ready)
		wait_ready(ctl.ready, ctl.ready_need, ctl.err, ctl.ready_spins);
	if (eval_skipped(a.skip, ctl.stage, ctl.want_stage))
		return;
	const double e = line_energy_sum(a.eblock, a.neblock);
	if (threadIdx.x == 0)
		*a.E_out = e * a.inv_vol + a.shift;
}

// Line pairs per warp task: with one tile of particles a table fragment is used for four pairs, else for two (3D N=2000,
// MT = 1: 13.7 us per evaluation with four pairs, 15.9 with two; MT = 2 with 16 warps: 13.6 and 13.3).
__host__ __device__ constexpr int line_nt(int mt) { return mt == 1 ? 4 : 2; }

// Tiles [tile0, tile1), W warps. Per tile (8 MT particles) and phase the particles' tables are built, then the warps take the
// phase's rows in turn (8 / NT warps a row, NT line pairs each) and contract the row's cells: per 4 cells NT weight fragments of 512 B
// from L2 (read once per block, in fragment order) against MT table fragments from shared memory, 2 MT NT DMMAs. What is
// left beside the DMMAs is instructions per step and the product with X per task, so weights with T's and D's factors
// written out (64 B a cell) beat 32 B ones expanded here (2D N=1e5: 2.05 against 2.17 ms per evaluation; 3D N=20000: 178
// against 187 us), and a ring of asynchronous copies for the weights gains nothing over loads one step ahead.
// With two teams (one phase only) a tile is 16 MT particles and each half of the warps contracts half of them with every row:
// more work between barriers, and rows of few tasks no longer leave warps idle. A warp of a team stands for the two warps of a
// block of one team one after the other, so that the sums are the same in every bit.
template <int D, int MT, int W>
__device__ __forceinline__ void line_force_body(const LineForceArgs &a, const int tile0, const int tile1, const ItemCtl ctl,
                                                const int teams = 1)
{
	constexpr int E = MT <= 2 ? 8 : 16, NT = line_nt(MT), SUB = 8 / NT;
	const int P = 8 * MT * teams, LOG2P = (MT == 1 ? 3 : MT == 2 ? 4 : 5) + teams - 1, WT = W / teams;
	extern __shared__ __align__(16) unsigned char smem[];
	double *pos = reinterpret_cast<double *>(smem);    // P x D
	double2 *tab = reinterpret_cast<double2 *>(smem + line_pos_bytes(P, D));
	LineTabs tb = load_rec(a.phases);
	// the sums of W warps x P x D: of one team over the tables, after the loops; else behind them
	double *sh_g = reinterpret_cast<double *>(teams == 1 ? tab : tab + (size_t)P * tb.row);
	const int lane = threadIdx.x & 31, team = teams == 1 ? 0 : (int)(threadIdx.x >> 5) / WT;
	const int warp = (int)(threadIdx.x >> 5) - team * WT;
	const int t = lane & 3, g = lane >> 2, g0 = team * 8 * MT + g;   // the lane's first particle of the tile
	// (as force_body: a finished instance builds no tables, but waits for its reduce items where there are any)
	if (eval_skipped(a.skip, ctl.stage, ctl.want_stage)) {
		if (ctl.ready)
			wait_ready(ctl.ready, ctl.ready_need, ctl.err, ctl.ready_spins);
		return;
	}
	// coordinate threadIdx.x of a tile, loaded a tile ahead
	auto load = [&](int tile) {
		return (int)threadIdx.x < min(P, a.N - tile * P) * D ? a.frac[(size_t)tile * P * D + threadIdx.x] : 0.0;
	};
	double next = load(tile0);
	for (int tile = tile0; tile < tile1; tile++) {
		const int pbase = tile * P;
		const int nvalid = min(P, a.N - pbase);
		if (tile > tile0) {
			tb = load_rec(a.phases);
			__syncthreads();   // the previous tile's sums are read
		}
		if ((int)threadIdx.x < P * D)
			pos[threadIdx.x] = next;
		__syncthreads();
		// The tables need only the positions, which the rho pass of this evaluation has already read: they are built while
		// the reduce kernel still runs (programmatic dependent launch).
		build_line_tables<D, E>(tb, pos, LOG2P, P, nvalid, tab);
		if (tile == tile0) {
			cudaGridDependencySynchronize();
			if (ctl.ready)
				wait_ready(ctl.ready, ctl.ready_need, ctl.err, ctl.ready_spins);
			if (eval_skipped(a.skip, ctl.stage, ctl.want_stage))
				return;
		}
		if (tile + 1 < tile1)
			next = load(tile + 1);
		double gs[MT][D];
		auto clear_sums = [&] {
#pragma unroll
			for (int m = 0; m < MT; m++)
#pragma unroll
				for (int e = 0; e < D; e++)
					gs[m][e] = 0.0;
		};
		// the four lanes of a particle; then the sums of "warp" w of W
		auto add_lanes = [&] {
#pragma unroll
			for (int m = 0; m < MT; m++)
#pragma unroll
				for (int e = 0; e < D; e++) {
					gs[m][e] += __shfl_xor_sync(0xffffffffu, gs[m][e], 1);
					gs[m][e] += __shfl_xor_sync(0xffffffffu, gs[m][e], 2);
				}
		};
		auto store_sums = [&](int w) {
			if (t == 0) {
#pragma unroll
				for (int m = 0; m < MT; m++)
#pragma unroll
					for (int e = 0; e < D; e++)
						sh_g[(w * P + g0 + m * 8) * D + e] = gs[m][e];
			}
		};
		clear_sums();
		int wsum = warp;   // the warp of a team of one whose tasks this warp is at

		for (int ph = 0; ph < a.nphase; ph++) {
			if (ph > 0) {
				tb = load_rec(a.phases + ph);
				__syncthreads();
				build_line_tables<D, E>(tb, pos, LOG2P, P, nvalid, tab);
			}
			__syncthreads();
			const bool centres = tb.n[2] > 0;
			const int jb = tb.hlo >> 2, je = (tb.hlo + tb.nh) >> 2;
			const double2 *trow = tab + (size_t)g0 * tb.row;
			// the weights are read one step ahead, across tasks; a task's row record one task ahead
			const int ntask = tb.ntask * SUB;
			int2 ri = make_int2(0, 0), rn = ri;
			double2 bq[NT];
			auto row_rec = [&](int q) { return __ldg(reinterpret_cast<const int2 *>(a.rows) + tb.r0 + q / SUB); };
			auto first_w = [&](int q, int2 x) { return a.weights + ((size_t)(x.x + jb) * 8 + (q % SUB) * NT) * 32 + lane; };
			if (warp < ntask) {
				ri = row_rec(warp);
				const double2 *w = first_w(warp, ri);
#pragma unroll
				for (int n = 0; n < NT; n++)
					bq[n] = __ldcg(w + n * 32);
			}
			for (int s = warp, sn; s < ntask; s = sn) {
				const int r = tb.r0 + s / SUB, pair = (s % SUB) * NT;
				sn = s + W;
				const bool last = sn >= ntask;   // of the tasks of warp wsum
				if (teams > 1 && last && wsum + WT < W)
					sn = wsum + WT;
				const bool more = sn < ntask;
				if (more)
					rn = row_rec(sn);
				const int nj = min(je, ri.y) - jb;   // > 0: the phase's rows all reach its first cells
				const double2 *w = first_w(s, ri);
				const double2 *wn = more ? first_w(sn, rn) : w;
				ri = rn;
				double2 acc[MT][NT];
				LineIdx li[NT];
#pragma unroll
				for (int n = 0; n < NT; n++)
					li[n] = load_rec(a.lines + (size_t)r * kLineRow + (pair + n) * 2 + (t >> 1));
#pragma unroll
				for (int m = 0; m < MT; m++)
#pragma unroll
					for (int n = 0; n < NT; n++)
						acc[m][n] = make_double2(0.0, 0.0);
				const double2 *th = trow + tb.offh + t;
				for (int j = 0; j < nj; j++, th += 4) {
					double2 f[NT];
#pragma unroll
					for (int n = 0; n < NT; n++)
						f[n] = bq[n];   // lane (t, g): cell 4 j + t, line g / 4 of the pair, component g % 4
					w = j + 1 < nj ? w + 8 * 32 : wn;
#pragma unroll
					for (int n = 0; n < NT; n++)
						bq[n] = __ldcg(w + n * 32);
					// (C_h, S_h) of particle 8 m + g, h = 4 j + t
					double2 c[MT];
#pragma unroll
					for (int m = 0; m < MT; m++)
						c[m] = th[m * 8 * tb.row];
#pragma unroll
					for (int m = 0; m + 1 < MT; m += 2)
#pragma unroll
						for (int n = 0; n < NT; n++)
							dmma16(acc[m][n], acc[m + 1][n], c[m].x, c[m + 1].x, c[m].y, c[m + 1].y, f[n].x, f[n].y);
					if (MT & 1) {
#pragma unroll
						for (int n = 0; n < NT; n++)
							dmma(acc[MT - 1][n], c[MT - 1].x, f[n].x);
#pragma unroll
						for (int n = 0; n < NT; n++)
							dmma(acc[MT - 1][n], c[MT - 1].y, f[n].y);
					}
				}
				// lane (g, t): particle 8 m + g, line t / 2 of pair n: T for even t, D for odd t. Stage by stage over the MT x NT
				// tiles: each FP64 operation may wait behind another warp's matrix instructions, so the chains run side by side.
				double2 x[MT][NT];
#pragma unroll
				for (int n = 0; n < NT; n++) {
					const int o0 = tb.off[0] + li[n].p0 - tb.lo[0], o1 = tb.off[1] + li[n].p1 - tb.lo[1];
#pragma unroll
					for (int m = 0; m < MT; m++) {
						x[m][n] = trow[m * 8 * tb.row + o0];
						if (D == 3)
							x[m][n] = cmul(x[m][n], trow[m * 8 * tb.row + o1]);
					}
				}
				if (centres) {
#pragma unroll
					for (int n = 0; n < NT; n++)
#pragma unroll
						for (int m = 0; m < MT; m++)
							x[m][n] = cmul(x[m][n], trow[m * 8 * tb.row + tb.off[2] + li[n].c - tb.lo[2]]);
				}
				double S[MT][NT];
#pragma unroll
				for (int m = 0; m < MT; m++)
#pragma unroll
					for (int n = 0; n < NT; n++)
						S[m][n] = x[m][n].y * acc[m][n].x;
#pragma unroll
				for (int m = 0; m < MT; m++)
#pragma unroll
					for (int n = 0; n < NT; n++)
						S[m][n] = fma(x[m][n].x, acc[m][n].y, S[m][n]);
#pragma unroll
				for (int n = 0; n < NT; n++) {
					const double k0 = (t & 1) ? 0.0 : (double)li[n].p0;
					const double k1 = (t & 1) ? 0.0 : (double)li[n].p1;
					const double kl = (t & 1) ? 1.0 : (double)li[n].c;
#pragma unroll
					for (int m = 0; m < MT; m++) {
						gs[m][0] = fma(k0, S[m][n], gs[m][0]);
						if (D == 3)
							gs[m][1] = fma(k1, S[m][n], gs[m][1]);
						gs[m][D - 1] = fma(kl, S[m][n], gs[m][D - 1]);
					}
				}
				if (teams > 1 && last && more) {
					add_lanes();
					store_sums(wsum);
					clear_sums();
					wsum += WT;
				}
			}
		}
		if (tile + 1 == tile1)
			cudaTriggerProgrammaticLaunchCompletion();
		add_lanes();
		if (teams == 1)
			__syncthreads();   // the tables are read
		store_sums(wsum);
		if (teams > 1 && wsum + WT < W) {   // no tasks of that warp
			clear_sums();
			store_sums(wsum + WT);
		}
		__syncthreads();
		// the warps in order
		if ((int)threadIdx.x < nvalid) {
			double v[D];
#pragma unroll
			for (int e = 0; e < D; e++) {
				v[e] = sh_g[threadIdx.x * D + e];
#pragma unroll
				for (int w2 = 1; w2 < W; w2++)
					v[e] += sh_g[(w2 * P + threadIdx.x) * D + e];
			}
			write_force_out<D>(a.F_out, a.gfrac_out, a.recip, a.fscale, pbase + threadIdx.x, v);
		}
	}
}

// dynamic shared memory of the two kernels
__host__ __device__ constexpr size_t line_rho_smem(int row, int chunk, int d)
{
	return line_pos_bytes(chunk, d) + (size_t)row * chunk * sizeof(double2);
}
__host__ __device__ constexpr size_t line_force_smem(int row, int mt, int warps, int d, int teams = 1)
{
	const size_t tables = (size_t)row * 8 * mt * teams * sizeof(double2);
	const size_t sums = (size_t)warps * 8 * mt * teams * d * sizeof(double);
	return line_pos_bytes(8 * mt * teams, d) + (teams > 1 ? tables + sums : tables > sums ? tables : sums);
}

// 8 warps: two blocks to an SM; 16 warps: one, for grids of one wave (8 warps alone on an SM leave its matrix units idle
// half the time).
template <int D, int MT, int W>
__global__ void __launch_bounds__(32 * W, W == 8 ? 2 : 1) cc_line_force_kernel(LineForceArgs a)
{
	// with an energy to write, block 0 sums it
	const int tile = (int)blockIdx.x - (a.E_out ? 1 : 0);
	if (tile < 0)
		line_energy_body(a, ItemCtl{a.stage, a.want_stage});
	else
		line_force_body<D, MT, W>(a, tile, tile + 1, ItemCtl{a.stage, a.want_stage});
}

// ---------------------------------------------------------------------------------------------------------------
// fused batch evaluation with line plans
// ---------------------------------------------------------------------------------------------------------------
// The launch of cc_mbatch_kernel (one work queue, phases ordered by completion counts) for batches in which some instance
// takes the line kernels: such an instance's FP64 items are line items, its mixed items (and every item of the other instances)
// segment items. An instance's phase holds the larger of its two item counts, so that the queue does not depend on the
// stages; the surplus items do nothing and are counted.
struct LBatchArgs {
	MBatchArgs m;
	const LineRhoArgs *lrho;
	const LineReduceArgs *lred;
	const LineForceArgs *lforce;
	const int *own;       // 6 x B: segment items of the three phases, line items (0: on the segment kernels)
};

union LineItemDesc {
	RhoArgs rho;
	ReduceArgs red;
	ForceArgs force;
	LineRhoArgs lrho;
	LineReduceArgs lred;
	LineForceArgs lforce;
};
// An item taken from the queue: its place there (it.x), phase, instance and item within the phase, and everything uniform that
// its body starts from.
struct LineItem {
	int4 it;
	int dim, count;          // items that do work; those beyond them are empty
	int line, mixed, shape;  // line items; the segment items' precision and groups
	unsigned need;           // the count its phase waits for
	const int *stage;
	LineItemDesc desc;
};

// The bodies as calls: inlined together into one kernel they spill (1.4 KB a thread at 128 registers).
template <int D> __device__ __noinline__ void line_rho_call(const LineRhoArgs &r, int local, const ItemCtl &ctl)
{
	line_rho_body<D>(r, local % r.ngroup, local / r.ngroup, ctl);
}
constexpr int kLineBatchMT = 3;      // tiles of 8 particles in a batch's force tile
template <int D> __device__ __noinline__ void line_force_call(const LineForceArgs &f, int local, const ItemCtl &ctl)
{
	const int P = 8 * kLineBatchMT * f.teams;
	const int ntile = (f.N + P - 1) / P, t0 = local * f.tiles;
	line_force_body<D, kLineBatchMT, 8>(f, t0, min(ntile, t0 + f.tiles), ctl, f.teams);
}
template <int D, bool MIXED> __device__ __noinline__ void seg_rho_call(const RhoArgs &r, int ng, int local, const ItemCtl &ctl)
{
	rho_body<D, 8, MIXED, false>(r, local % ng, local / ng, ctl);
}
template <int D, bool MIXED> __device__ __noinline__ void seg_force_call(const ForceArgs &f, int pg, int local, const ItemCtl &ctl)
{
	force_body<D, 8, MIXED>(f, local % pg, local / pg, ctl);
}

// MODE as mbatch_item: 0 FP64, 1 mixed, 2 each instance at the precision of its stage word
template <int D, int MODE>
__device__ __forceinline__ void lbatch_item(const MBatchArgs &A, const LineItem &s)
{
	const int phase = s.it.y, b = s.it.z, local = s.it.w;
	ItemCtl ctl;
	ctl.err = A.count + 3 * A.B;
	ctl.ready_spins = A.spins;
	ctl.want_stage = A.want_stage;
	ctl.stage = MODE == 2 ? nullptr : s.stage;
	if (phase > 0) {
		ctl.ready = A.count + (phase - 1) * A.B + b;
		ctl.ready_need = s.need;
	}
	if (local >= s.count)
		return;
	if constexpr (MODE != 1 && D >= 2) {
		if (s.line) {
			if (phase == 0) {
				line_rho_call<D>(s.desc.lrho, local, ctl);
			} else if (phase == 1) {
				line_reduce_wide_body(s.desc.lred, local, ctl);
			} else {
				const LineForceArgs &f = s.desc.lforce;
				line_force_call<D>(f, local, ctl);
				// the instance's first force item also sums the energy (its reduce items are complete)
				if (local == 0 && f.E_out && !eval_skipped(f.skip, ctl.stage, ctl.want_stage)) {
					const double e = line_energy_sum(f.eblock, f.neblock);
					if (threadIdx.x == 0)
						*f.E_out = e * f.inv_vol + f.shift;
				}
			}
			return;
		}
	}
	if (phase == 0) {
		if constexpr (MODE != 0) {
			if (s.mixed) {
				seg_rho_call<D, true>(s.desc.rho, s.shape, local, ctl);
				return;
			}
		}
		if constexpr (MODE != 1)
			seg_rho_call<D, false>(s.desc.rho, s.shape, local, ctl);
	} else if (phase == 1) {
		reduce_body_wide(s.desc.red, local, ctl);
	} else {
		if constexpr (MODE != 0) {
			if (s.mixed) {
				seg_force_call<D, true>(s.desc.force, s.shape, local, ctl);
				return;
			}
		}
		if constexpr (MODE != 1)
			seg_force_call<D, false>(s.desc.force, s.shape, local, ctl);
	}
}

// Queue position -> (phase, instance, item within the phase), phase by phase: by the time an instance's force items come up,
// its reduce items are long done. (Its force items straight behind its reduce items, as cc_mbatch_kernel has them, waited 5
// us for them in every block, instance after instance: 48 uneven instances 210 us, with this order 177.)
__device__ __forceinline__ int4 lbatch_decode(const MBatchArgs &A, int item)
{
	int phase = 0, at = item;
	while (phase < 2 && at >= A.total[phase])
		at -= A.total[phase++];
	const int *pre = A.pre + phase * (A.B + 1);
	const int b = find_instance(pre, A.B, at);
	return make_int4(item, phase, b, at - __ldg(pre + b));
}

// The record of queue position `item` (lane 0's), by one warp.
template <int MODE> __device__ __forceinline__ void lbatch_fetch(const LBatchArgs &L, int item, LineItem &s)
{
	const MBatchArgs &A = L.m;
	const int lane = threadIdx.x & 31;
	item = __shfl_sync(0xffffffffu, item, 0);
	if (item >= A.total[0] + A.total[1] + A.total[2]) {
		if (lane == 0)
			s.it = make_int4(item, 0, 0, 0);
		return;
	}
	const int4 it = lbatch_decode(A, item);
	const int phase = it.y, b = it.z;
	const int *stage = A.rho[b].stage;
	const int dim = __ldg(A.dim + b), nseg = __ldg(L.own + phase * A.B + b), nline = __ldg(L.own + (3 + phase) * A.B + b);
	const bool mixed = MODE == 1 || (MODE == 2 && stage && *(volatile const int *)stage == 0);
	const bool line = !mixed && dim >= 2 && nline > 0;
	auto copy = [&](const auto *src, auto &dst) {
		using T = std::remove_reference_t<decltype(dst)>;
		static_assert(sizeof(T) % 8 == 0 && alignof(T) >= 8, "descriptors are copied as 8-byte words");
		const unsigned long long *from = reinterpret_cast<const unsigned long long *>(src);
		unsigned long long *to = reinterpret_cast<unsigned long long *>(&dst);
#pragma unroll
		for (int w = 0; w < (int)(sizeof(T) / 8); w += 32)
			if (w + lane < (int)(sizeof(T) / 8))
				to[w + lane] = __ldg(from + w + lane);
	};
	if (phase == 0) {
		if (line)
			copy(L.lrho + b, s.desc.lrho);
		else
			copy(A.rho + b, s.desc.rho);
	} else if (phase == 1) {
		if (line)
			copy(L.lred + b, s.desc.lred);
		else
			copy(A.red + b, s.desc.red);
	} else {
		if (line)
			copy(L.lforce + b, s.desc.lforce);
		else
			copy(A.force + b, s.desc.force);
	}
	if (lane == 0) {
		s.it = it;
		s.dim = dim;
		s.count = line ? nline : nseg;
		s.line = line;
		s.mixed = mixed;
		s.shape = __ldg(A.shape + phase * A.B + b);
		const int *pre = A.pre + (phase - 1) * (A.B + 1) + b;
		s.need = phase == 0 ? 0u : (unsigned)(__ldg(pre + 1) - __ldg(pre)) + (phase == 1 && b == 0 ? A.phantom : 0u);
		s.stage = stage;
	}
}

// Between an item and the next one, warp 1 takes the next (position, record and descriptor: three dependent round trips) while
// warp 0 counts the one that ended: 3 us between items before, when one thread did both in turn and the block then fetched
// the descriptor. The count does not wait for the fetch (warp 1 only arrives at the barrier before it), and the position is not
// taken earlier: taken at the start of an item, it kept items that others waited for behind long ones (60 instances 187 -> 204
// us).
template <int MODE>
__global__ void __launch_bounds__(kMBatchThreads, MODE == 1 ? 3 : 2) cc_lbatch_kernel(LBatchArgs L)
{
	const MBatchArgs &A = L.m;
	__shared__ LineItem items[2];
	const int T = A.total[0] + A.total[1] + A.total[2];
	const bool fetches = (threadIdx.x >> 5) == 1;
	cudaGridDependencySynchronize();
	auto take = [&] { return threadIdx.x == 32 ? (int)atomicAdd(A.queue, 1u) : 0; };
	if (fetches)
		lbatch_fetch<MODE>(L, take(), items[0]);
	__syncthreads();
	for (int at = 0;; at ^= 1) {
		const LineItem &s = items[at];
		if (s.it.x >= T)
			break;
		if (s.dim == 3)
			lbatch_item<3, MODE>(A, s);
		else if (s.dim == 2)
			lbatch_item<2, MODE>(A, s);
		else
			lbatch_item<1, MODE>(A, s);
		const int next = take();
		__threadfence();   // the item's results are visible before its count rises
		if (fetches) {
			asm volatile("barrier.cta.arrive 1, %0;" ::"n"(kMBatchThreads) : "memory");
			lbatch_fetch<MODE>(L, next, items[at ^ 1]);
		} else {
			asm volatile("barrier.cta.sync 1, %0;" ::"n"(kMBatchThreads) : "memory");
			if (threadIdx.x == 0)
				mbatch_count(A, s.it);
		}
		__syncthreads();
	}
	queue_leave(A.queue);
}

}  // namespace cc
