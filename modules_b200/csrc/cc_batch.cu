// cc_batch.cu — batches of independent configurations (cc_batch_* in include/cc_gpu.h).
//
// A batch evaluates many configurations of uneven size and dimension together: ONE launch of the fused batch kernel
// (cc_lbatch_kernel, cc_lines.cuh; cc_mbatch_kernel, cc_kernels.cuh, where no instance takes the line kernels) per energy + gradient step, whose work queue holds the rho blocks, split-reduction
// chunks and force blocks of every instance; per-instance completion counts order the three phases of an instance.
// Its batched L-BFGS (cc_batch_minimize) keeps every instance's positions, gradient and history on the device and
// enqueues blocks of iterations (one fused evaluation and the L-BFGS kernels each). The reference
// evaluates one configuration per Objective call (potential/StructureOptimization.cpp:447-578).
#include "cc_internal.h"
#include "cc_multi_launch.h"

#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

using namespace cci;

namespace {

// carve 256-byte aligned pieces out of one device allocation
struct Arena {
	unsigned char *base = nullptr;
	size_t used = 0, cap = 0;
	size_t take(size_t bytes)
	{
		const size_t off = used;
		used += (bytes + 255) / 256 * 256;
		return off;
	}
	template <class T> T *at(size_t off) { return reinterpret_cast<T *>(base + off); }
};

using cc::kBatchChunk;
using cc::kBatchPerSplit;
using cc::kBatchSegsPerSplit;

// an instance's evaluation buffers in the batch arena
struct BatchBufs {
	size_t o_part, o_rho, o_u, o_eb, o_tk, o_pg, o_fc, o_w;
};

// Particles whose tables a line rho block stages at once (two blocks share an SM).
int batch_line_chunk(const cc::LineGroups &g, int per_split)
{
	int c = 8;
	while (c < per_split && c < 64 && (size_t)2 * c * g.row * sizeof(double2) <= 96 * 1024)
		c *= 2;
	return c;
}

// tile shapes the autotuner times: particles per rho block, segments per force block
constexpr int kTuneSplits[] = {32, 64, 128, 256, 512, 1024};
constexpr int kTuneSegs[] = {32, 64, 128, 256, 512, 1024};

constexpr int kApartWaves = 8;   // cc_batch_minimize: launches of their own for the instances of either stage
constexpr size_t kBatchLineSmem = 104 * 1024;   // line items: two blocks to an SM

// dynamic shared memory the fused kernel is allowed (its largest table rows in FP64, any dimension)
size_t mbatch_smem_cap()
{
	return std::max(kBatchLineSmem, std::max(rho_smem<double2>(cc::kMaxRow, kBatchChunk, 8), force_smem<double2>(cc::kMaxRow, 3)));
}

template <auto KERNEL, class ARGS> int mbatch_launch_t(const ARGS &a, const int *totals, size_t smem, cudaStream_t st)
{
	static const cudaError_t attr =
	    cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mbatch_smem_cap());
	if (attr != cudaSuccess)
		return fail(CC_ERR_CUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(attr));
	// resident blocks per SM for this shared memory size (looked up once per size)
	static std::mutex mu;
	static std::map<size_t, int> per_sm;
	int resident = 0;
	{
		std::lock_guard<std::mutex> lk(mu);
		auto it = per_sm.find(smem);
		if (it == per_sm.end()) {
			int n = 0;
			CC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, KERNEL, cc::kMBatchThreads, smem));
			it = per_sm.emplace(smem, std::max(1, n)).first;
		}
		resident = it->second * sm_count();
	}
	const int total = totals[0] + totals[1] + totals[2];
	if (total <= 0)
		return CC_OK;
	CC_CUDA(launch_pdl_n(KERNEL, dim3(std::min(total, resident)), dim3(cc::kMBatchThreads), smem,
	                     st, a));
	return CC_OK;
}

}  // namespace

int cc::launch_mbatch(int mode, const MBatchArgs &a, int rho_row, int force_row, int maxd, cudaStream_t st)
{
	if (a.B < 1)
		return CC_OK;
	const size_t smem = std::max(rho_smem<double2>(rho_row, kBatchChunk, 8), force_smem<double2>(force_row, maxd));
	switch (mode) {
	case 0: return mbatch_launch_t<cc::cc_mbatch_kernel<0> >(a, a.total, smem, st);
	case 1: return mbatch_launch_t<cc::cc_mbatch_kernel<1> >(a, a.total, smem, st);
	default: return mbatch_launch_t<cc::cc_mbatch_kernel<2> >(a, a.total, smem, st);
	}
}

struct cc_batch {
	std::vector<cc_handle *> h;
	std::vector<int64_t> N;
	std::vector<int> order;                  // instances by decreasing work: their order in the fused launch
	Arena arena;
	std::vector<size_t> off_frac, off_F, off_E;
	std::vector<BatchBufs> bufs;
	int per_split = 0, segs_per_split = 0;   // the tile shape in use
	cudaStream_t stream = nullptr;
	unsigned char *meta = nullptr;           // one allocation for the arrays down to d_count
	// the fused launch's descriptors in `order`: set 0 evaluates the batch positions into the batch outputs, set 1 a
	// minimisation's trial points into its L-BFGS buffers
	cc::RhoArgs *d_rho[2] = {nullptr, nullptr};
	cc::ReduceArgs *d_red[2] = {nullptr, nullptr};
	cc::ForceArgs *d_force[2] = {nullptr, nullptr};
	int *d_dim = nullptr;                    // B
	int *d_pre = nullptr;                    // 3 queues (one per mode) of 4 x (B + 1): rho, reduce, force, reduce +
	                                         // force items per instance
	int *d_shape = nullptr;                  // 3 x B
	// instances on the line kernels (uses_lines): their FP64 descriptors (set 0 / 1), and the two item counts of every instance
	bool any_line = false, all_line = false;
	std::vector<char> line;                  // by instance: FP64 on the line kernels
	cc::LineRhoArgs *d_lrho[2] = {nullptr, nullptr};
	cc::LineReduceArgs *d_lred[2] = {nullptr, nullptr};
	cc::LineForceArgs *d_lforce[2] = {nullptr, nullptr};
	int *d_own = nullptr;                    // 6 x B
	size_t line_smem = 0;
	std::vector<int> seg_force;              // segment force items of every instance (launch order)
	std::vector<cc::LineRhoArgs> lrho;       // host copies of set 0
	std::vector<cc::LineReduceArgs> lred;
	std::vector<cc::LineForceArgs> lforce;
	unsigned *d_queue = nullptr;             // 2 words
	unsigned *d_count = nullptr;             // 3 x B completion counts + 1 error word
	int total[3][3] = {};                    // items per mode and phase
	int rho_row = 1, force_row = 1, maxd = 1;
	unsigned wait_spins = 0, wait_phantom = 0;   // cc_batch_set_wait_test
	std::vector<cc::RhoArgs> rho;            // host copies of set 0 (in `order`)
	std::vector<cc::ReduceArgs> red;
	std::vector<cc::ForceArgs> force;
	// L-BFGS state of cc_batch_minimize, kept between calls (grow-only): a minimisation makes no allocation call
	// into the CUDA driver once the batch has run one
	unsigned char *lb_base = nullptr;
	size_t lb_cap = 0;
	cc::LbInst *d_lb = nullptr;              // the instances in `order`, their start values and final positions
	cc::LbStart *d_start = nullptr;
	double **d_final = nullptr;
	cc::LbBrief *d_brief = nullptr;
	int d_lb_cap = 0;
	// Host transfers go through one pinned buffer and one copy each way: positions, forces and energies of all instances
	// are contiguous in the arena (a copy per instance costs 8 to 15 us of driver time).
	size_t pos_bytes = 0, F_off = 0, F_bytes = 0, E_off = 0;
	unsigned char *h_pin = nullptr;          // positions, or forces + energies + error word, or status + error word
};

namespace {

cc::MBatchArgs batch_args(const cc_batch *b, int set, int mode)
{
	cc::MBatchArgs a;
	a.rho = b->d_rho[set];
	a.red = b->d_red[set];
	a.force = b->d_force[set];
	a.dim = b->d_dim;
	a.pre = b->d_pre + (size_t)mode * 4 * (b->order.size() + 1);
	a.shape = b->d_shape;
	a.B = (int)b->order.size();
	for (int k = 0; k < 3; k++)
		a.total[k] = b->total[mode][k];
	a.want_stage = mode == 1 ? 0 : 1;
	a.queue = b->d_queue;
	a.count = b->d_count;
	a.spins = b->wait_spins;
	a.phantom = b->wait_phantom;
	return a;
}

// (Re)build the evaluation descriptors (set 0) for a tile shape: per_split particles per rho block and force splits
// of about segs_per_split segments; the arena holds the buffers of every candidate shape.
int batch_build(cc_batch *b, int per_split, int segs_per_split)
{
	const int B = (int)b->order.size();
	std::vector<int> pre(3 * 4 * (B + 1), 0), shape(3 * B, 0), dim(B, 0), own(6 * B, 0);
	b->rho.clear();
	b->red.clear();
	b->force.clear();
	b->lrho.clear();
	b->lred.clear();
	b->lforce.clear();
	b->line_smem = 0;
	b->rho_row = b->force_row = 1;
	b->maxd = 1;
	for (int k = 0; k < B; k++) {
		const int i = b->order[k];
		cc_handle *h = b->h[i];
		const cc::Plan &p = h->main.plan;
		const BatchBufs &q = b->bufs[i];
		const int64_t n = b->N[i];
		const int nsplit = (int)((n + per_split - 1) / per_split);
		// reduce items of kWideSlots slots each (their energy terms are the force items' eblock entries)
		const int nchunks = (p.nslot + cc::kWideSlots - 1) / cc::kWideSlots, pgroups = (int)((n + 31) / 32);
		const DevSplits *f = nullptr;
		const int want = (int)std::max<int64_t>(1, (p.real_segs + segs_per_split - 1) / segs_per_split);
		if (int rc = get_splits(h->main, want, &f))
			return rc;
		cc::RhoArgs ra = {};
		ra.frac = b->arena.at<double>(b->off_frac[i]);
		ra.N = (int)n;
		ra.per_split = per_split;
		ra.chunk = kBatchChunk;
		ra.segs = h->main.segs;
		ra.bstart = h->main.bstart;
		ra.bspec = h->main.bspec;
		ra.nseg = (int)p.segs.size();
		ra.nslot = p.nslot;
		ra.partial = b->arena.at<double2>(q.o_part);
		cc::ReduceArgs rr = {};
		rr.partial = ra.partial;
		rr.nsplit = nsplit;
		rr.nslot = p.nslot;
		rr.slotV = h->main.slotV;
		rr.rho_offset = h->rho_offset;
		rr.rho_slot = b->arena.at<double2>(q.o_rho);
		rr.u_slot = b->arena.at<double2>(q.o_u);
		rr.eblock = b->arena.at<double>(q.o_eb);
		rr.ticket = b->arena.at<unsigned>(q.o_tk);
		rr.inv_vol = 1.0 / h->volume;
		rr.shift = h->shift;
		rr.E_out = b->arena.at<double>(b->off_E[i]);
		rr.finalize = 0;   // the force items sum the energy terms
		cc::ForceArgs fa = {};
		fa.frac = ra.frac;
		fa.N = ra.N;
		fa.segs = h->main.segs;
		fa.kstart = f->kstart;
		fa.kspec = f->kspec;
		fa.nksplit = f->host.count();
		fa.u_slot = rr.u_slot;
		fa.nseg = ra.nseg;
		fa.partialG = b->arena.at<double>(q.o_pg);
		fa.counters = b->arena.at<unsigned>(q.o_fc);
		for (int c = 0; c < 9; c++)
			fa.recip[c] = h->recip[c];
		fa.fscale = 2.0 / h->volume;
		fa.F_out = b->arena.at<double>(b->off_F[i]);
		fa.gfrac_out = nullptr;
		fa.eblock = rr.eblock;
		fa.neblock = nchunks;
		fa.inv_vol = rr.inv_vol;
		fa.shift = rr.shift;
		fa.E_out = rr.E_out;
		b->rho.push_back(ra);
		b->red.push_back(rr);
		b->force.push_back(fa);
		const int c[3] = {p.nbgroups() * nsplit, nchunks, pgroups * fa.nksplit};
		cc::LineRhoArgs lr = {};
		cc::LineReduceArgs ld = {};
		cc::LineForceArgs lf = {};
		for (int ph = 0; ph < 3; ph++)
			own[ph * B + k] = c[ph];
		if (b->line[i]) {
			const cc::LinePlan &L = h->main.lplan;
			const DevLines &dl = h->main.line;
			lr.frac = ra.frac;
			lr.N = ra.N;
			// Twice the particles per rho item from 20 items of the instance on: an item's fixed cost (queue, descriptor, table
			// latencies, partial rows: about 4 us) stays small beside its 4 to 8 us of matrix work. 512 uneven instances
			// 1.98 -> 1.82 ms, 60 of the benchmark's kind 214 -> 198 us, 128 x 3D N=2000 0.85 -> 0.79 ms. A rule on the instance
			// alone: its results do not depend on the rest of the batch.
			lr.ngroup = L.groupings[0].count();
			lr.per_split = (long)n * lr.ngroup >= 20L * per_split ? 2 * per_split : per_split;
			const int lsplit = (int)((n + lr.per_split - 1) / lr.per_split);
			lr.chunk = batch_line_chunk(L.groupings[0], lr.per_split);
			lr.log2chunk = __builtin_ctz((unsigned)lr.chunk);
			lr.nunit = L.nunit;
			lr.ntask = cc::kLineTasks;
			lr.groups = dl.groups[0].groups;
			lr.tasks = dl.groups[0].tasks;
			lr.tlines = dl.groups[0].tlines;
			lr.partial = ra.partial;
			ld.partial = lr.partial;
			ld.nsplit = lsplit;
			ld.nunit = L.nunit;
			ld.cells = dl.cells;
			ld.cellV = dl.cellV;
			ld.rho_offset = h->rho_offset;
			ld.weights = b->arena.at<double2>(q.o_w);
			ld.eblock = rr.eblock;
			lf.frac = ra.frac;
			lf.N = ra.N;
			lf.nphase = (int)L.phases.size();
			lf.phases = dl.phases;
			lf.rows = dl.rows;
			lf.lines = dl.lines;
			lf.weights = ld.weights;
			for (int e = 0; e < 9; e++)
				lf.recip[e] = h->recip[e];
			lf.fscale = fa.fscale;
			lf.F_out = fa.F_out;
			lf.eblock = rr.eblock;
			lf.neblock = (L.nunit + cc::kLineWideUnits - 1) / cc::kLineWideUnits;
			lf.inv_vol = fa.inv_vol;
			lf.shift = fa.shift;
			lf.E_out = fa.E_out;
			lf.tiles = lf.teams = 1;   // set below
			const int lc[3] = {lr.ngroup * lsplit, lf.neblock, (int)((n + 8 * cc::kLineBatchMT - 1) / (8 * cc::kLineBatchMT))};
			for (int ph = 0; ph < 3; ph++)
				own[(3 + ph) * B + k] = lc[ph];
			b->line_smem = std::max(b->line_smem, std::max(cc::line_rho_smem(L.groupings[0].row, lr.chunk, h->d),
			                                               cc::line_force_smem(L.phase_row, cc::kLineBatchMT, 8, h->d)));
		}
		b->lrho.push_back(lr);
		b->lred.push_back(ld);
		b->lforce.push_back(lf);
		const int sh[3] = {p.nbgroups(), nchunks, pgroups};
		for (int ph = 0; ph < 3; ph++)
			shape[ph * B + k] = sh[ph];
		dim[k] = h->d;
		b->rho_row = std::max(b->rho_row, p.block_max_row);
		b->force_row = std::max(b->force_row, f->host.max_row);
		b->maxd = std::max(b->maxd, h->d);
	}
	// Line force items. From 1.5 tiles of 24 particles per resident block on, a block's warps work as two teams on 48 particles
	// (line_force_body: the results are the same) where their tables leave two blocks to an SM: the fixed cost of a tile (table
	// and reduction latencies: 4 us) is paid half as often, 48 uneven instances 181 -> 151 us, 512 2.11 -> 1.96 ms; with fewer
	// tiles the longer ones cost more (12 instances 25 against 28 us). Then several tiles per item where the batch has many, so
	// that an item's fixed cost (queue, descriptor, completion) stays small: two from 4.6 per block on (833 tiles, 2.8 a block:
	// 250 us with one, 289 with two; 1478, 5.0 a block: 151 and 145).
	int64_t tiles = 0;
	for (int k = 0; k < B; k++)
		tiles += own[5 * B + k];
	const bool teams = 2 * tiles >= 3 * 2 * sm_count();
	tiles = 0;
	for (int k = 0; k < B; k++) {
		const cc_handle *h = b->h[b->order[k]];
		const cc::LinePlan &L = h->main.lplan;
		if (!b->line[b->order[k]])
			continue;
		const size_t two = cc::line_force_smem(L.phase_row, cc::kLineBatchMT, 8, h->d, 2);
		if (teams && L.phases.size() == 1 && two <= kBatchLineSmem) {
			b->lforce[k].teams = 2;
			own[5 * B + k] = (own[5 * B + k] + 1) / 2;
			b->line_smem = std::max(b->line_smem, two);
		}
		tiles += own[5 * B + k];
	}
	const int per_item = (int)std::max<int64_t>(1, std::min<int64_t>(8, tiles * 10 / (46 * sm_count())));
	for (int k = 0; k < B; k++) {
		b->lforce[k].tiles = per_item;
		own[5 * B + k] = (own[5 * B + k] + per_item - 1) / per_item;
	}
	// the queue of each mode: 0 line items for instances on the line kernels, 1 segment items, 2 (an instance's stage decides) the
	// larger of the two counts
	for (int mode = 0; mode < 3; mode++) {
		int *q = pre.data() + (size_t)mode * 4 * (B + 1);
		for (int k = 0; k < B; k++) {
			int c[3];
			for (int ph = 0; ph < 3; ph++) {
				const int seg = own[ph * B + k], line = own[(3 + ph) * B + k];
				c[ph] = mode == 1 || line == 0 ? seg : mode == 0 ? line : std::max(seg, line);
				q[ph * (B + 1) + k + 1] = q[ph * (B + 1) + k] + c[ph];
			}
			q[3 * (B + 1) + k + 1] = q[3 * (B + 1) + k] + c[1] + c[2];   // its reduce and force items, consecutive
		}
		for (int ph = 0; ph < 3; ph++)
			b->total[mode][ph] = q[ph * (B + 1) + B];
	}
	int rc;
	cudaStream_t st = b->stream;
	if ((rc = upload_into(b->d_rho[0], b->rho, st)) || (rc = upload_into(b->d_red[0], b->red, st)) ||
	    (rc = upload_into(b->d_force[0], b->force, st)) || (rc = upload_into(b->d_pre, pre, st)) ||
	    (rc = upload_into(b->d_shape, shape, st)) || (rc = upload_into(b->d_dim, dim, st)) ||
	    (rc = upload_into(b->d_lrho[0], b->lrho, st)) || (rc = upload_into(b->d_lred[0], b->lred, st)) ||
	    (rc = upload_into(b->d_lforce[0], b->lforce, st)) || (rc = upload_into(b->d_own, own, st)))
		return rc;
	CC_CUDA(cudaStreamSynchronize(st));   // evaluations may run on a caller's stream
	b->seg_force.assign(own.begin() + 2 * B, own.begin() + 3 * B);
	b->per_split = per_split;
	b->segs_per_split = segs_per_split;
	return CC_OK;
}

// One fused launch evaluating every instance (descriptor set `set`). Precision CC_PREC_SCHEDULE evaluates each
// instance at the precision of its stage word; CC_PREC_FP64 / CC_PREC_MIXED skip instances whose stage word (set 1
// only) differs from 1 / 0.
int batch_eval(cc_batch *b, int set, int precision, cudaStream_t st)
{
	const int mode = precision == CC_PREC_SCHEDULE ? 2 : precision == CC_PREC_MIXED ? 1 : 0;
	if (b->any_line) {
		cc::LBatchArgs a;
		a.m = batch_args(b, set, mode);
		a.lrho = b->d_lrho[set];
		a.lred = b->d_lred[set];
		a.lforce = b->d_lforce[set];
		a.own = b->d_own;
		// segment items need their own shared memory: mixed ones, and those of the other instances
		size_t smem = mode == 1 ? 0 : b->line_smem;
		if (mode != 0 || !b->all_line)
			smem = std::max(smem, std::max(rho_smem<double2>(b->rho_row, kBatchChunk, 8),
			                               force_smem<double2>(b->force_row, b->maxd)));
		switch (mode) {
		case 0: return mbatch_launch_t<cc::cc_lbatch_kernel<0> >(a, a.m.total, smem, st);
		case 1: return mbatch_launch_t<cc::cc_lbatch_kernel<1> >(a, a.m.total, smem, st);
		default: return mbatch_launch_t<cc::cc_lbatch_kernel<2> >(a, a.m.total, smem, st);
		}
	}
	return cc::launch_mbatch(mode, batch_args(b, set, mode), b->rho_row, b->force_row, b->maxd, st);
}

// A bounded wait of the fused kernel that ran out leaves the error word set: `err` is its copy (read after a
// synchronisation of the batch's stream); report and clear it.
int batch_check_wait(cc_batch *b, unsigned err)
{
	if (err) {
		// in place before a launch on any stream: a later clear would erase that launch's error
		CC_CUDA(cudaMemsetAsync(b->d_count + 3 * b->order.size(), 0, sizeof(unsigned), b->stream));
		CC_CUDA(cudaStreamSynchronize(b->stream));
		return fail(CC_ERR_TIMEOUT, "a bounded wait of the fused batch kernel ran out");
	}
	return CC_OK;
}

int batch_check_wait(cc_batch *b)
{
	unsigned err = 0;
	CC_CUDA(cudaMemcpy(&err, b->d_count + 3 * b->order.size(), sizeof(unsigned), cudaMemcpyDeviceToHost));
	return batch_check_wait(b, err);
}

// The pinned buffer, made once with room for every transfer of the batch (pinning 2 MB takes over a millisecond).
int batch_pin(cc_batch *b)
{
	if (b->h_pin)
		return CC_OK;
	const size_t count = b->h.size();
	const size_t bytes = std::max(b->pos_bytes, std::max(b->F_bytes + count * sizeof(double), count * sizeof(cc::LbBrief)) +
	                                                sizeof(unsigned));
	const cudaError_t e = cudaHostAlloc(reinterpret_cast<void **>(&b->h_pin), bytes, cudaHostAllocDefault);
	if (e != cudaSuccess) {
		cudaGetLastError();
		b->h_pin = nullptr;
		return fail(CC_ERR_OOM, std::string("cudaHostAlloc: ") + cudaGetErrorString(e));
	}
	return CC_OK;
}

// Every instance's coordinates, wrapped into [0, 1) (floor twice), into the pinned buffer at its place among the
// positions. Coordinates already in [0, 1) are checked and copied in one pass.
int batch_stage(cc_batch *b, const double *const *frac)
{
	if (int rc = batch_pin(b))
		return rc;
	for (size_t i = 0; i < b->h.size(); i++) {
		const size_t n = (size_t)b->N[i] * b->h[i]->d;
		const double *x = frac[i];
		double *w = reinterpret_cast<double *>(b->h_pin + (b->off_frac[i] - b->off_frac[0]));
		long bad = 0;
		for (size_t k = 0; k < n; k++) {
			const double v = x[k];
			w[k] = v;
			bad |= (long)!(v >= 0.0) | (long)!(v < 1.0);
		}
		if (!bad)
			continue;
		for (size_t k = 0; k < n; k++) {
			if (!std::isfinite(x[k]))
				return fail(CC_ERR_ARG, "non-finite fractional coordinate");
			const double v = x[k] - std::floor(x[k]);
			w[k] = v - std::floor(v);
		}
	}
	return CC_OK;
}

// Energies, the error word and, if F is not null, forces of the evaluation just enqueued on the batch's stream.
int batch_results(cc_batch *b, double *E, double *const *F)
{
	const size_t count = b->h.size(), e_bytes = count * sizeof(double), fb = F ? b->F_bytes : 0;
	if (int rc = batch_pin(b))
		return rc;
	cudaStream_t st = b->stream;
	if (fb)
		CC_CUDA(cudaMemcpyAsync(b->h_pin, b->arena.base + b->F_off, fb, cudaMemcpyDeviceToHost, st));
	CC_CUDA(cudaMemcpyAsync(b->h_pin + fb, b->arena.base + b->E_off, e_bytes, cudaMemcpyDeviceToHost, st));
	CC_CUDA(cudaMemcpyAsync(b->h_pin + fb + e_bytes, b->d_count + 3 * count, sizeof(unsigned), cudaMemcpyDeviceToHost, st));
	CC_CUDA(cudaStreamSynchronize(st));
	unsigned err;
	std::memcpy(&err, b->h_pin + fb + e_bytes, sizeof(err));
	if (int rc = batch_check_wait(b, err))
		return rc;
	std::memcpy(E, b->h_pin + fb, e_bytes);
	if (F)
		for (size_t i = 0; i < count; i++)
			if (F[i])
				std::memcpy(F[i], b->h_pin + (b->off_F[i] - b->F_off), sizeof(double) * b->N[i] * b->h[i]->d);
	return CC_OK;
}

}  // namespace

extern "C" {

int cc_batch_create(int count, cc_handle *const *handles, const int64_t *N, cc_batch **out)
{
	if (!out || count < 1 || !handles || !N)
		return fail(CC_ERR_ARG, "invalid batch arguments");
	*out = nullptr;
	for (int i = 0; i < count; i++) {
		if (!handles[i] || N[i] < 1 || N[i] > (1 << 26) || handles[i]->main.plan.nslot == 0)
			return fail(CC_ERR_ARG, "every instance needs a handle with constraints and 1 <= N <= 2^26");
		if (handles[i]->d_slotS0)
			return fail(CC_ERR_ARG, "batches hold the plain collective-coordinate form only");
	}
	cc_batch *b = new cc_batch();
	b->h.assign(handles, handles + count);
	b->N.assign(N, N + count);
	// per instance: buffers sized for every tile shape the autotuner may choose (the most particle splits and force
	// splits among the candidates), carved out of one arena
	b->off_frac.resize(count);
	b->off_F.resize(count);
	b->off_E.resize(count);
	b->bufs.resize(count);
	b->line.assign(count, 0);
	for (int i = 0; i < count; i++)
		b->off_frac[i] = b->arena.take(sizeof(double) * N[i] * handles[i]->d);
	b->pos_bytes = b->arena.used - b->off_frac[0];
	for (int i = 0; i < count; i++)
		b->off_F[i] = b->arena.take(sizeof(double) * N[i] * handles[i]->d);
	b->F_off = b->off_F[0];
	b->F_bytes = b->arena.used - b->F_off;
	b->E_off = b->arena.take(sizeof(double) * count);
	for (int i = 0; i < count; i++)
		b->off_E[i] = b->E_off + sizeof(double) * i;
	for (int i = 0; i < count; i++) {
		cc_handle *h = handles[i];
		const cc::Plan &p = h->main.plan;
		const int64_t n = N[i];
		BatchBufs &q = b->bufs[i];
		int max_nks = 1;
		for (int segs : kTuneSegs) {
			const DevSplits *f = nullptr;
			const int want = (int)std::max<int64_t>(1, (p.real_segs + segs - 1) / segs);
			if (int rc = get_splits(h->main, want, &f)) {
				delete b;
				return rc;
			}
			max_nks = std::max(max_nks, f->host.count());
		}
		const int max_nsplit = (int)((n + kTuneSplits[0] - 1) / kTuneSplits[0]);
		const int nchunks = (p.nslot + 31) / 32, pgroups = (int)((n + 31) / 32);
		const cc::LinePlan &L = h->main.lplan;
		b->line[i] = uses_lines(h->main, n);   // (a rule on the instance alone)
		if (b->line[i])
			if (int rc = ensure_lines(h->main)) {
				delete b;
				return rc;
			}
		const size_t row = std::max((size_t)p.nslot, b->line[i] ? (size_t)L.nunit * 128 : 0);   // entries of a partial row
		b->any_line |= b->line[i] != 0;
		q.o_part = b->arena.take(sizeof(double2) * (size_t)max_nsplit * row);
		q.o_rho = b->arena.take(sizeof(double2) * p.nslot);
		q.o_u = b->arena.take(sizeof(double2) * p.nslot);
		q.o_eb = b->arena.take(sizeof(double) * std::max(nchunks, L.nunit));
		q.o_w = b->arena.take(sizeof(double2) * (size_t)L.nunit * 256);
		q.o_tk = b->arena.take(sizeof(unsigned));
		q.o_pg = b->arena.take(sizeof(double) * (size_t)max_nks * n * h->d);
		q.o_fc = b->arena.take(sizeof(unsigned) * pgroups);
	}
	b->all_line = true;
	for (int i = 0; i < count; i++)
		b->all_line &= b->line[i] != 0;
	int rc;
	if ((rc = dev_alloc(&b->arena.base, b->arena.used))) {
		cc_batch_destroy(b);
		return rc;
	}
	b->arena.cap = b->arena.used;
	if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess ||
	    cudaMemsetAsync(b->arena.base, 0, b->arena.used, b->stream) != cudaSuccess) {
		cc_batch_destroy(b);
		return fail(CC_ERR_CUDA, "batch initialisation failed");
	}
	// instances by decreasing work: the work queue hands out the longest items first
	b->order.resize(count);
	for (int i = 0; i < count; i++)
		b->order[i] = i;
	std::stable_sort(b->order.begin(), b->order.end(), [&](int x, int y) {
		return (double)N[x] * handles[x]->main.plan.real_segs > (double)N[y] * handles[y]->main.plan.real_segs;
	});
	// descriptors, queues and counts: pieces of one allocation, zeroed
	const size_t B = (size_t)count;
	size_t used = 0;
	std::vector<std::pair<void **, size_t> > pieces;
	auto take = [&](auto **p, size_t n) {
		pieces.push_back(std::make_pair(reinterpret_cast<void **>(p), used));
		used += (n * sizeof(**p) + 255) / 256 * 256;
	};
	for (int w = 0; w < 2; w++) {
		take(&b->d_rho[w], B);
		take(&b->d_red[w], B);
		take(&b->d_force[w], B);
		take(&b->d_lrho[w], B);
		take(&b->d_lred[w], B);
		take(&b->d_lforce[w], B);
	}
	take(&b->d_pre, 3 * 4 * (B + 1));
	take(&b->d_shape, 3 * B);
	take(&b->d_own, 6 * B);
	take(&b->d_dim, B);
	take(&b->d_queue, 2);
	take(&b->d_count, 3 * B + 1);
	if ((rc = dev_alloc(&b->meta, used))) {
		cc_batch_destroy(b);
		return rc;
	}
	for (const auto &p : pieces)
		*p.first = b->meta + p.second;
	if (cudaMemsetAsync(b->meta, 0, used, b->stream) != cudaSuccess) {
		cc_batch_destroy(b);
		return fail(CC_ERR_CUDA, "batch initialisation failed");
	}
	if ((rc = batch_build(b, kBatchPerSplit, kBatchSegsPerSplit))) {
		cc_batch_destroy(b);
		return rc;
	}
	*out = b;
	return CC_OK;
}

int cc_batch_autotune(cc_batch *b, int reps, int *per_split, int *segs_per_split)
{
	if (!b || reps < 1)
		return fail(CC_ERR_ARG, "invalid autotune arguments");
	cudaEvent_t e0, e1;
	CC_CUDA(cudaEventCreate(&e0));
	CC_CUDA(cudaEventCreate(&e1));
	float best = 1e30f;
	int bp = b->per_split, bs = b->segs_per_split, rc = CC_OK;
	// `reps` evaluations at a precision, after one that is not timed
	auto timed = [&](int precision, float *ms) -> int {
		if (int r2 = batch_eval(b, 0, precision, b->stream))
			return r2;
		if (cudaEventRecord(e0, b->stream) != cudaSuccess)
			return fail(CC_ERR_CUDA, "cudaEventRecord failed");
		for (int r = 0; r < reps; r++)
			if (int r2 = batch_eval(b, 0, precision, b->stream))
				return r2;
		if (cudaEventRecord(e1, b->stream) != cudaSuccess || cudaEventSynchronize(e1) != cudaSuccess ||
		    cudaEventElapsedTime(ms, e0, e1) != cudaSuccess)
			return fail(CC_ERR_CUDA, "autotune timing failed");
		return CC_OK;
	};
	float ms = 0.0f, mixed_ms = 0.0f;
	if (!b->any_line) {
		for (int ps : kTuneSplits)
			for (int sg : kTuneSegs) {
				if (rc || (rc = batch_build(b, ps, sg)) || (rc = timed(CC_PREC_FP64, &ms)))
					continue;
				if (ms < best) {
					best = ms;
					bp = ps;
					bs = sg;
				}
			}
	} else {
		// FP64 evaluations of instances on the line kernels do not read the segment tile: the particles per rho block are chosen
		// by FP64, the segments then by FP64 (the other instances) and mixed evaluations (every instance) together
		for (int ps : kTuneSplits) {
			if (rc || (rc = batch_build(b, ps, bs)) || (rc = timed(CC_PREC_FP64, &ms)))
				continue;
			if (ms < best) {
				best = ms;
				bp = ps;
			}
		}
		best = 1e30f;
		for (int sg : kTuneSegs) {
			if (rc || (rc = batch_build(b, bp, sg)) || (!b->all_line && (rc = timed(CC_PREC_FP64, &ms))) ||
			    (rc = timed(CC_PREC_MIXED, &mixed_ms)))
				continue;
			const float both = mixed_ms + (b->all_line ? 0.0f : ms);
			if (both < best) {
				best = both;
				bs = sg;
			}
		}
	}
	cudaEventDestroy(e0);
	cudaEventDestroy(e1);
	if (rc)
		return rc;
	if ((rc = batch_check_wait(b)))
		return rc;
	if ((rc = batch_build(b, bp, bs)))
		return rc;
	if (per_split)
		*per_split = bp;
	if (segs_per_split)
		*segs_per_split = bs;
	return CC_OK;
}

int cc_batch_destroy(cc_batch *b)
{
	if (!b)
		return CC_OK;
	if (b->stream)
		cudaStreamSynchronize(b->stream);
	cudaFree(b->meta);
	cudaFree(b->arena.base);
	cudaFree(b->lb_base);
	cudaFree(b->d_lb);
	cudaFree(b->d_brief);
	cudaFree(b->d_start);
	cudaFree(b->d_final);
	cudaFreeHost(b->h_pin);
	if (b->stream)
		cudaStreamDestroy(b->stream);
	delete b;
	return CC_OK;
}

int cc_batch_set_positions(cc_batch *b, const double *const *frac)
{
	if (!b || !frac)
		return fail(CC_ERR_ARG, "invalid batch arguments");
	if (int rc = batch_stage(b, frac))
		return rc;
	CC_CUDA(cudaMemcpyAsync(b->arena.base + b->off_frac[0], b->h_pin, b->pos_bytes, cudaMemcpyHostToDevice, b->stream));
	CC_CUDA(cudaStreamSynchronize(b->stream));
	return CC_OK;
}

int cc_batch_set_wait_test(cc_batch *b, unsigned polls, int phantom)
{
	if (!b || phantom < 0)
		return fail(CC_ERR_ARG, "invalid wait test arguments");
	b->wait_spins = polls;
	b->wait_phantom = (unsigned)phantom;
	return CC_OK;
}

int cc_batch_eval_device(cc_batch *b, int precision, void *stream)
{
	if (!b)
		return fail(CC_ERR_ARG, "null batch");
	if (int rc = check_prec(precision))
		return rc;
	return batch_eval(b, 0, precision, stream ? static_cast<cudaStream_t>(stream) : b->stream);
}

int cc_batch_energy_grad(cc_batch *b, double *E, double *const *F, int precision)
{
	if (!b || !E)
		return fail(CC_ERR_ARG, "invalid batch arguments");
	if (int rc = cc_batch_eval_device(b, precision, b->stream))
		return rc;
	return batch_results(b, E, F);
}

int cc_batch_minimize(cc_batch *b, double *const *frac, const cc_lbfgs_opts *opts, cc_lbfgs_result *results)
{
	if (!b || !frac)
		return fail(CC_ERR_ARG, "invalid batch arguments");
	cc_lbfgs_opts o;
	cc_lbfgs_defaults(&o);
	if (opts)
		o = *opts;
	if (o.history < 1 || o.history > cc::kLbMaxHist || o.iters_per_check < 1 ||
	    (o.precision != CC_PREC_FP64 && o.precision != CC_PREC_MIXED && o.precision != CC_PREC_SCHEDULE))
		return fail(CC_ERR_ARG, "invalid minimisation options");
	const int count = (int)b->h.size(), m = o.history;
	int maxn = 0;
	for (int i = 0; i < count; i++)
		maxn = std::max(maxn, (int)(b->N[i] * b->h[i]->d));
	const int nblk = cc::lb_blocks(maxn, cc::kLbMaxBlocks);
	// L-BFGS buffers of every instance in one allocation
	Arena ar;
	std::vector<size_t> ox(count), og(count), od(count), oxt(count), ogt(count), oS(count), oY(count), op(count),
	    ost(count);
	for (int i = 0; i < count; i++)   // laid out as the batch's positions: one copy brings every start
		ox[i] = ar.take(8 * (size_t)b->N[i] * b->h[i]->d);
	for (int i = 0; i < count; i++)
		ost[i] = ar.take(sizeof(cc::LbState));
	const size_t st_bytes = ar.used - ost[0];
	for (int i = 0; i < count; i++) {
		const size_t n = (size_t)b->N[i] * b->h[i]->d;
		og[i] = ar.take(8 * n);
		od[i] = ar.take(8 * n);
		oxt[i] = ar.take(8 * n);
		ogt[i] = ar.take(8 * n);
		oS[i] = ar.take(8 * n * m);
		oY[i] = ar.take(8 * n * m);
		op[i] = ar.take(8 * (size_t)nblk * cc::lb_ndots(m));
	}
	int rc;
	if ((rc = batch_stage(b, frac)))   // (a non-finite start changes nothing)
		return rc;
	if (b->lb_cap < ar.used) {
		cudaFree(b->lb_base);
		b->lb_base = nullptr;
		b->lb_cap = 0;
		if ((rc = dev_alloc(&b->lb_base, ar.used)))
			return rc;
		b->lb_cap = ar.used;
	}
	if (b->d_lb_cap < count) {
		cudaFree(b->d_lb);
		cudaFree(b->d_brief);
		cudaFree(b->d_start);
		cudaFree(b->d_final);
		b->d_lb = nullptr;
		b->d_brief = nullptr;
		b->d_start = nullptr;
		b->d_final = nullptr;
		b->d_lb_cap = 0;
		if ((rc = dev_alloc(&b->d_lb, (size_t)count)) || (rc = dev_alloc(&b->d_brief, count)) ||
		    (rc = dev_alloc(&b->d_start, count)) || (rc = dev_alloc(&b->d_final, count)))
			return rc;
		b->d_lb_cap = count;
	}
	ar.base = b->lb_base;
	std::vector<cc::LbInst> lbi(count);   // by instance index
	for (int i = 0; i < count; i++) {
		cc::LbInst &l = lbi[i];
		l.n = (int)(b->N[i] * b->h[i]->d);
		l.m = m;
		l.x = ar.at<double>(ox[i]);
		l.g = ar.at<double>(og[i]);
		l.d = ar.at<double>(od[i]);
		l.xt = ar.at<double>(oxt[i]);
		l.gt = ar.at<double>(ogt[i]);
		l.S = ar.at<double>(oS[i]);
		l.Y = ar.at<double>(oY[i]);
		l.part = ar.at<double>(op[i]);
		l.st = ar.at<cc::LbState>(ost[i]);
	}
	// the L-BFGS instances in the launch order, and the minimisation descriptors (set 1): evaluate at x_trial into
	// the L-BFGS buffers, skip finished instances
	std::vector<cc::LbInst> lbo(count);
	std::vector<cc::LbStart> start(count);
	std::vector<double *> final_pos(count);
	std::vector<cc::RhoArgs> ra = b->rho;
	std::vector<cc::ReduceArgs> rr = b->red;
	std::vector<cc::ForceArgs> fa = b->force;
	std::vector<cc::LineRhoArgs> lra = b->lrho;
	std::vector<cc::LineReduceArgs> lrr = b->lred;
	std::vector<cc::LineForceArgs> lfa = b->lforce;
	for (int k = 0; k < count; k++) {
		const int i = b->order[k];
		lbo[k] = lbi[i];
		start[k].stopval = o.stopval == CC_STOPVAL_GROUND_STATE ? 1e-20 * (double)b->N[i] : o.stopval;
		start[k].switch_E = o.switch_energy_per_particle * (double)b->N[i];
		final_pos[k] = b->arena.at<double>(b->off_frac[i]);
		const int *status = &lbi[i].st->status, *stage = &lbi[i].st->stage;
		ra[k].frac = lbi[i].xt;
		ra[k].skip = status;
		ra[k].stage = stage;
		rr[k].E_out = &lbi[i].st->Et;
		rr[k].skip = status;
		rr[k].stage = stage;
		fa[k].frac = lbi[i].xt;
		fa[k].E_out = &lbi[i].st->Et;
		fa[k].gfrac_out = lbi[i].gt;
		fa[k].F_out = nullptr;
		fa[k].skip = status;
		fa[k].stage = stage;
		lra[k].frac = ra[k].frac;
		lra[k].skip = lrr[k].skip = lfa[k].skip = status;
		lra[k].stage = lrr[k].stage = lfa[k].stage = stage;
		lfa[k].frac = fa[k].frac;
		lfa[k].E_out = fa[k].E_out;
		lfa[k].gfrac_out = fa[k].gfrac_out;
		lfa[k].F_out = nullptr;
	}
	cudaStream_t st = b->stream;
	if ((rc = upload_into(b->d_lb, lbo, st)) || (rc = upload_into(b->d_rho[1], ra, st)) ||
	    (rc = upload_into(b->d_red[1], rr, st)) || (rc = upload_into(b->d_force[1], fa, st)) ||
	    (rc = upload_into(b->d_lrho[1], lra, st)) || (rc = upload_into(b->d_lred[1], lrr, st)) ||
	    (rc = upload_into(b->d_lforce[1], lfa, st)) || (rc = upload_into(b->d_start, start, st)) ||
	    (rc = upload_into(b->d_final, final_pos, st)))
		return rc;
	const bool sched = o.precision == CC_PREC_SCHEDULE;
	CC_CUDA(cudaMemcpyAsync(b->lb_base + ox[0], b->h_pin, b->pos_bytes, cudaMemcpyHostToDevice, st));
	CC_CUDA(cudaMemsetAsync(b->lb_base + ost[0], 0, st_bytes, st));
	const dim3 all((maxn + 255) / 256, count);
	cc::lb_start_kernel<<<all, 256, 0, st>>>(b->d_lb, b->d_start, o.gtol, o.ftol, o.max_evals,
	                                         o.precision == CC_PREC_FP64 ? 1 : 0, sched ? 1 : 0);
	CC_CUDA(cudaGetLastError());
	// A block of iterations is enqueued kernel by kernel: an iteration keeps the GPU busy for far longer (40 us and more)
	// than its four launches take, and capturing a graph of them on every call cost 2 ms. Schedule: each instance at its
	// stage's precision while some instance is in the mixed stage; then FP64 only. The launch that holds both precisions has
	// the registers of the line items, two blocks to an SM, and mixed items run at two thirds of the speed of the mixed
	// launch's three: while the running instances' mixed force items fill more than kApartWaves times that, the instances of
	// either stage have a launch of their own (the other ones' items are skipped, which costs some 25 us; the same items, so the
	// results are the same). 64 uneven instances, 100 steps in the mixed stage 66 -> 54 ms; with 2 instead of 8, 32 of N <= 1000
	// to their ground states 93 -> 97.
	bool apart = false;
	auto choose_apart = [&](const std::vector<cc::LbBrief> *hs) {
		int64_t mixed = 0;
		for (int k = 0; k < count; k++)
			if (!hs || ((*hs)[k].status == cc::kLbRunning && (*hs)[k].stage == 0))
				mixed += b->seg_force[k];
		apart = sched && b->any_line && mixed > (int64_t)kApartWaves * 2 * sm_count();
	};
	choose_apart(nullptr);
	auto iterations = [&](int prec, int count_it) -> int {
		for (int it = 0; it < count_it; it++) {
			if (prec == CC_PREC_SCHEDULE && apart) {
				if (int r2 = batch_eval(b, 1, CC_PREC_MIXED, st))
					return r2;
				if (int r2 = batch_eval(b, 1, CC_PREC_FP64, st))
					return r2;
			} else if (int r2 = batch_eval(b, 1, prec, st))
				return r2;
			CC_CUDA(cc::lb_step(b->d_lb, count, nblk, maxn, st, count == 1 ? &lbo[0] : nullptr));
		}
		return CC_OK;
	};
	std::vector<cc::LbBrief> hs(count);   // in launch order
	const size_t hs_bytes = sizeof(cc::LbBrief) * count;
	CC_CUDA(cudaStreamSynchronize(st));   // the staged starts are out of the pinned buffer
	int stage = 0;
	int64_t left = o.max_evals;   // an instance still running has made one evaluation per iteration
	const int64_t max_rounds = o.max_evals / o.iters_per_check + 2;
	for (int64_t round = 0; round < max_rounds; round++) {
		const int its = (int)std::max<int64_t>(1, std::min<int64_t>(o.iters_per_check, left));
		left -= its;
		rc = iterations(stage ? CC_PREC_FP64 : o.precision, its);
		bool running = false, any_mixed = false;
		cudaError_t e = cudaSuccess;
		if (!rc) {
			cc::lb_brief_kernel<<<(count + 127) / 128, 128, 0, st>>>(b->d_lb, count, b->d_brief);
			e = cudaGetLastError();
			if (e == cudaSuccess)
				e = cudaMemcpyAsync(b->h_pin, b->d_brief, hs_bytes, cudaMemcpyDeviceToHost, st);
			if (e == cudaSuccess)
				e = cudaMemcpyAsync(b->h_pin + hs_bytes, b->d_count + 3 * count, sizeof(unsigned), cudaMemcpyDeviceToHost,
				                    st);
		}
		const cudaError_t es = cudaStreamSynchronize(st);
		if (rc)
			return rc;
		if (e == cudaSuccess)
			e = es;
		if (e != cudaSuccess)
			return fail(CC_ERR_CUDA, std::string("batch minimisation: ") + cudaGetErrorString(e));
		unsigned err;
		std::memcpy(&err, b->h_pin + hs_bytes, sizeof(err));
		if ((rc = batch_check_wait(b, err)))
			return rc;
		std::memcpy(hs.data(), b->h_pin, hs_bytes);
		for (int k = 0; k < count; k++) {
			running |= hs[k].status == cc::kLbRunning;
			any_mixed |= hs[k].status == cc::kLbRunning && hs[k].stage == 0;
		}
		if (!running)
			break;
		if (sched && stage == 0 && !any_mixed)
			stage = 1;
		choose_apart(&hs);
	}
	// results: positions wrapped into [0,1) become the bound ones, FP64 energies of the results (one batched evaluation)
	cc::lb_finish_kernel<<<all, 256, 0, st>>>(b->d_lb, b->d_final);
	CC_CUDA(cudaGetLastError());
	std::vector<double> E(count);
	if ((rc = batch_eval(b, 0, CC_PREC_FP64, st)) || (rc = batch_results(b, E.data(), nullptr)))
		return rc;
	CC_CUDA(cudaMemcpyAsync(b->h_pin, b->arena.base + b->off_frac[0], b->pos_bytes, cudaMemcpyDeviceToHost, st));
	CC_CUDA(cudaStreamSynchronize(st));
	for (int i = 0; i < count; i++)
		std::memcpy(frac[i], b->h_pin + (b->off_frac[i] - b->off_frac[0]), sizeof(double) * b->N[i] * b->h[i]->d);
	if (results)
		for (int k = 0; k < count; k++) {
			const int i = b->order[k];
			results[i].E = E[i];
			results[i].evals = hs[k].evals;
			results[i].iters = hs[k].iters;
			results[i].status = hs[k].status == cc::kLbRunning ? cc::kLbMaxEval : hs[k].status;
		}
	return CC_OK;
}

}  // extern "C"
