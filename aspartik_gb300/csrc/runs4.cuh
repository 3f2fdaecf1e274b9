// runs4.cuh -- run-synchronous FP32 pruning walks, single calculator and
// batched.  Included by kernels4.cu inside its anonymous namespace (uses
// v4_apply, v4_mul, rescale_pow2, transition4 and the Neumaier helpers).
//
// The one-thread-per-column walk leaves the GPU with only patterns x
// categories threads, about 14 warps per SM on the largest workload, and it
// is latency-bound.  Here a block owns a tile of patterns and walks the
// schedule run by run (a run is a sequence of mutually independent entries,
// e.g. one level of the tree).  Inside a run its (entry, category, pattern)
// items are spread over all threads of the block, so a wide level keeps
// every thread busy; a __syncthreads() separates runs.
//
// Thread layout: column col = c * tile + pl (fixed per thread, patterns
// fastest, so a warp touches 32 consecutive patterns of one category) and
// group g; group g handles entries g, g + groups, ... of every run.

// Everything one tile walk needs; the single-calculator kernel fills it from
// PruneParams, the batched kernel from the member's descriptor.
struct TileArgs {
	const uint8_t *tips;
	float4 *part;
	int32_t *scales;
	const float4 *ptab;
	const double *pi;
	const uint32_t *weights;
	double *site_lnl;
	double *cat_lnl;
	uint32_t ldp, C, L, tile, n, n_runs, tips_smem;
	double log_inv_c;
	// inline tables (RunSmem::tabs set): their sources
	const ModelDev *model;
	const double *lengths;
	const double *matrices;
};

// Shared-memory extras of the run walk (all null: none).  sp/ss: slot
// partials and counts (the entries' slot codes travel in NodeOp::pad of the
// schedule's shared-memory copy); tabs: two buffers of
// tab_stride float4 for the per-run tables; eig (V, V^-1, lambda in FP32),
// rate (clock rate x category rate) and len (edge lengths, or null: read
// from global memory) feed the table builder.
struct RunSmem {
	float4 *sp;
	int32_t *ss;
	float4 *tabs;
	uint32_t tab_stride;
	const float *eig;
	const double *rate;
	const double *len;
};

// Transition tables of entries [lo, hi) into buf, entry lo first, in
// ptab4_kernel's layout and with its arithmetic (the same FP32 eigensystem,
// the same product of the length and the rates in FP64), one matrix per
// thread.
__device__ __forceinline__ void build_run_tables(const TileArgs &a,
						 const RunSmem &rs,
						 uint32_t lo, uint32_t hi,
						 float4 *buf)
{
	const uint32_t C = a.C;
	const uint32_t count = (hi - lo) * 2 * C;
	// highest threads first: the last group walks the fewest entries
	for (uint32_t k = blockDim.x - 1u - threadIdx.x; k < count; k += blockDim.x) {
		const uint32_t id = lo * 2 * C + k;
		const uint32_t c = id % C, es = id / C;
		float P[16];
		if (a.matrices) {
			const double *src = a.matrices + (size_t)id * 16;
			for (int q = 0; q < 16; q++)
				P[q] = (float)src[q];
		} else {
			const double len = rs.len ? rs.len[es] : a.lengths[es];
			transition4f_eig(a.model, rs.eig, len * rs.rate[c], P);
		}
		float4 *out = buf + k * 5;
#pragma unroll
		for (int q = 0; q < 4; q++)
			out[q] = make_float4(P[q], P[4 + q], P[8 + q], P[12 + q]);
		out[4] = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
	}
}

// Root: frequency-weighted sum of the partial vector, in FP32 (the FP64
// pipe runs at 1/64 of the FP32 rate on this part, and the root mixing of
// every pattern sits on the critical path of a short dirty list).
__device__ __forceinline__ float root_dot4(const float *pi, const float4 &y)
{
	return fmaf(pi[3], y.w, fmaf(pi[2], y.z, fmaf(pi[1], y.y, pi[0] * y.x)));
}

// Per-thread constants of a tile walk.  Tip codes come from the block's
// shared-memory tile (tip_row = tile) or from global memory (tips_p = tips
// + p, tip_row = ldp); the schedule and the slot codes from shared memory.
// A listed child whose output sits in a shared-memory slot (sp/ss: slot k
// of column col at k * cols + col) is read from there: the children of a
// whole-tree list are then never read back from L2 or DRAM.
template <typename Idx>
struct WalkCtx {
	const NodeOp *ops; // pad: the entry's slot codes
	float4 *sp;
	int32_t *ss;
	const uint8_t *tips_p;
	const float *pi;
	const float4 *tab; // tables of entry tab_i0 first
	uint32_t tab_i0;
	uint32_t tip_row, c, col, cols;
	uint32_t half; // the thread's second column: col + half (pattern + half)
	Idx stride, col_off;
};

// sum_k x_k * row_k for two vectors with the same four table rows (loaded
// once), in v4_apply's order.
__device__ __forceinline__ void v4_apply_pair(const float4 *pt, float4 &x0,
					      float4 &x1)
{
	const float4 r[4] = {pt[0], pt[1], pt[2], pt[3]};
	x0 = v4_apply(r, x0);
	x1 = v4_apply(r, x1);
}

// One child of entry i for the thread's two columns: a tip gives its
// table rows (the products themselves), a partial its vectors and
// cumulative counts (transformed by the caller).
template <typename Idx>
__device__ __forceinline__ void load_child2(const TileArgs &a,
					    const WalkCtx<Idx> &w, uint32_t id,
					    uint32_t slot, const float4 *tb,
					    float4 &x0, float4 &x1, int32_t &s0,
					    int32_t &s1)
{
	if (id & kTipBit) {
		const uint8_t *tp = w.tips_p + (Idx)(id & ~kTipBit) * w.tip_row;
		x0 = tb[tp[0]];
		x1 = tb[tp[w.half]];
		s0 = 0;
		s1 = 0;
	} else if (slot != kNoSlot) {
		const uint32_t k = slot * w.cols + w.col;
		x0 = w.sp[k];
		x1 = w.sp[k + w.half];
		s0 = w.ss[k];
		s1 = w.ss[k + w.half];
	} else {
		const Idx ix = (Idx)id * w.stride + w.col_off;
		x0 = a.part[ix];
		x1 = a.part[ix + w.half];
		s0 = a.scales[ix];
		s1 = a.scales[ix + w.half];
	}
}

// Entry i of the current run for the thread's two columns: both children
// (a tip's table row, a slot, or global memory), the products, the
// rescalings, the stores to global memory (read by later evaluations) and,
// when the entry has one, to its slot; the list's last entry (the root)
// leaves its frequency-weighted sums and counts in s_dot / s_cnt.  The
// entry's schedule word, slot codes and table rows are read once for both
// columns.  The host gives an entry one of its own children's slots or a
// slot released in an earlier run, so no other entry of the run reads the
// slot it writes.
template <typename Idx>
__device__ __forceinline__ void run_item2(const TileArgs &a,
					  const WalkCtx<Idx> &w, uint32_t i,
					  float *s_dot, int32_t *s_cnt)
{
	const NodeOp op = w.ops[i];
	const uint32_t sw = op.pad;
	const float4 *tl = w.tab + ((2 * (i - w.tab_i0)) * a.C + w.c) * 5;
	const float4 *tr = tl + 5 * a.C;
	float4 a0, a1, b0, b1;
	int32_t sa0, sa1, sb0, sb1;
	load_child2<Idx>(a, w, op.left, (sw >> 8) & 0xFFu, tl, a0, a1, sa0, sa1);
	load_child2<Idx>(a, w, op.right, (sw >> 16) & 0xFFu, tr, b0, b1, sb0,
			 sb1);
	if (!(op.left & kTipBit))
		v4_apply_pair(tl, a0, a1);
	if (!(op.right & kTipBit))
		v4_apply_pair(tr, b0, b1);
	float4 y0 = v4_mul(a0, b0), y1 = v4_mul(a1, b1);
	const int32_t n0 = sa0 + sb0 + rescale_pow2(y0);
	const int32_t n1 = sa1 + sb1 + rescale_pow2(y1);
	const Idx ox = (Idx)op.out * w.stride + w.col_off;
	a.part[ox] = y0;
	a.part[ox + w.half] = y1;
	a.scales[ox] = n0;
	a.scales[ox + w.half] = n1;
	const uint32_t os = sw & 0xFFu;
	if (os != kNoSlot) {
		const uint32_t k = os * w.cols + w.col;
		w.sp[k] = y0;
		w.sp[k + w.half] = y1;
		w.ss[k] = n0;
		w.ss[k + w.half] = n1;
	}
	if (i == a.n - 1) {
		s_dot[w.col] = root_dot4(w.pi, y0);
		s_dot[w.col + w.half] = root_dot4(w.pi, y1);
		s_cnt[w.col] = n0;
		s_cnt[w.col + w.half] = n1;
	}
}

__device__ double tile_root(const TileArgs &a, uint32_t t, const float *s_dot,
			    const int32_t *s_cnt, double *s_red);

// One pattern tile t: every run of the schedule, then the category mixing
// of the root.  Returns the tile's weighted site sum in thread 0.  Ends with
// the block synchronised.  s_dot/s_cnt hold tile * C entries, s_red 32;
// rs the run walk's shared-memory extras.  The run walk reads each entry's
// slot codes from NodeOp::pad of s_ops (0xFFFFFF: no slots).
template <typename Idx, bool kPrefetch = false>
__device__ double tile_walk(const TileArgs &a, uint32_t t, float *s_dot,
			    int32_t *s_cnt, double *s_red,
			    const NodeOp *s_ops, const uint32_t *s_runs,
			    uint8_t *s_tips, const RunSmem &rs = RunSmem{})
{
	const uint32_t tile = a.tile, C = a.C;
	const uint32_t cols = tile * C;
	const uint32_t groups = blockDim.x / cols;
	const uint32_t tid = threadIdx.x;
	const uint32_t col = tid % cols;
	const uint32_t c = col / tile, pl = col - c * tile;
	const Idx stride = (Idx)C * a.ldp;
	const uint32_t p = t * tile + pl;
	const Idx col_off = (Idx)c * a.ldp + p;

	__shared__ float s_pi[4];
	if (tid < 4)
		s_pi[tid] = (float)a.pi[tid];
	const bool serial = groups == 1;
	const uint8_t *tips_p, *tips_base;
	uint32_t tip_row;
	if (a.tips_smem) {
		// 4-byte loads: rows start at multiples of 32 patterns
		const uint32_t wpr = tile >> 2;
		const uint32_t total = a.L * wpr;
		uint32_t *s_t32 = (uint32_t *)s_tips;
		for (uint32_t k = tid; k < total; k += blockDim.x) {
			const uint32_t leaf = k / wpr, w4 = k - leaf * wpr;
			s_t32[k] = *(const uint32_t *)(a.tips + (size_t)leaf * a.ldp +
						       t * tile + w4 * 4);
		}
		tips_base = s_tips;
		tip_row = tile;
	} else {
		tips_base = a.tips + t * tile;
		tip_row = a.ldp;
	}
	tips_p = tips_base + pl;
	const bool inl = !serial && rs.tabs != nullptr && a.n_runs != 0;
	if (inl)
		build_run_tables(a, rs, s_runs[0], s_runs[1], rs.tabs);
	__syncthreads();
	if (serial) {
		// One thread per column (tile * C == blockDim.x) walks the whole
		// list in order, with no barrier: a child that is the output of
		// one of the two previous entries comes from registers, any other
		// listed child from memory (written earlier by this thread).  The
		// walk is issue-bound (about 700 cycles an entry at 16 warps per
		// SM), so clean inputs are loaded plainly: staging them ahead in
		// shared memory was measured to gain nothing.
		float4 y0 = make_float4(0.f, 0.f, 0.f, 0.f), y1 = y0;
		int32_t c0 = 0, c1 = 0;
		uint32_t o0 = 0xFFFFFFFFu, o1 = 0xFFFFFFFFu;
		// A child that is neither a tip nor one of the two previous
		// outputs is read from global memory (a clean subtree, usually
		// not in L2).  With kPrefetch (the fused short-list kernel, whose
		// registers allow it) its load for entry i + 1 is issued before
		// entry i's product, so the latency overlaps the arithmetic: it is
		// never entry i's or i-1's output, and any earlier output it may
		// be was stored by this thread before the load.
		float4 pf[2];
		int32_t pfs[2];
		auto fetch = [&](const NodeOp &op, uint32_t f0, uint32_t f1) {
			const uint32_t ids[2] = {op.left, op.right};
#pragma unroll
			for (int j = 0; j < 2; ++j)
				if (!(ids[j] & kTipBit) && ids[j] != f0 && ids[j] != f1) {
					const Idx ix = (Idx)ids[j] * stride + col_off;
					pf[j] = a.part[ix];
					pfs[j] = a.scales[ix];
				}
		};
		auto input = [&](uint32_t id, const float4 *tb, int j, float4 &v,
				 int32_t &sc) {
			if (id & kTipBit) {
				v = tb[tips_p[(Idx)(id & ~kTipBit) * tip_row]];
				sc = 0;
			} else if (id == o0) {
				v = v4_apply(tb, y0);
				sc = c0;
			} else if (id == o1) {
				v = v4_apply(tb, y1);
				sc = c1;
			} else if (kPrefetch) {
				v = v4_apply(tb, pf[j]);
				sc = pfs[j];
			} else {
				const Idx ix = (Idx)id * stride + col_off;
				sc = a.scales[ix];
				v = v4_apply(tb, a.part[ix]);
			}
		};
		if (kPrefetch && a.n)
			fetch(s_ops[0], o0, o1);
		for (uint32_t i = 0; i < a.n; ++i) {
			const NodeOp op = s_ops[i];
			const float4 *tl = a.ptab + ((size_t)(2 * i) * C + c) * 5;
			const float4 *tr = tl + 5 * C;
			float4 ca, cb;
			int32_t sa, sb;
			input(op.left, tl, 0, ca, sa);
			input(op.right, tr, 1, cb, sb);
			if (kPrefetch && i + 1 < a.n) // forwards after this entry: op.out, o0
				fetch(s_ops[i + 1], op.out, o0);
			float4 y = v4_mul(ca, cb);
			const int32_t cnt = sa + sb + rescale_pow2(y);
			const Idx ox = (Idx)op.out * stride + col_off;
			a.part[ox] = y;
			a.scales[ox] = cnt;
			y1 = y0;
			c1 = c0;
			o1 = o0;
			y0 = y;
			c0 = cnt;
			o0 = op.out;
		}
		s_dot[col] = root_dot4(s_pi, y0);
		s_cnt[col] = c0;
		__syncthreads();
	}
	if (!serial) {
		// two columns per thread: patterns ph and ph + tile / 2 of one
		// category, so a warp still reads 32 consecutive patterns
		const uint32_t half = tile >> 1, tcols = cols >> 1;
		const uint32_t rgroups = blockDim.x / tcols;
		const uint32_t ct = tid % tcols, rg = tid / tcols;
		const uint32_t rc = ct / half, ph = ct - rc * half;
		WalkCtx<Idx> w;
		w.ops = s_ops;
		w.sp = rs.sp;
		w.ss = rs.ss;
		w.tab = a.ptab;
		w.tab_i0 = 0;
		w.tips_p = tips_base + ph;
		w.pi = s_pi;
		w.tip_row = tip_row;
		w.c = rc;
		w.col = rc * tile + ph;
		w.cols = cols;
		w.half = half;
		w.stride = stride;
		w.col_off = (Idx)rc * a.ldp + t * tile + ph;
		for (uint32_t r = 0; r < a.n_runs; ++r) {
			const uint32_t start = s_runs[r], end = s_runs[r + 1];
			if (inl) {
				// the next run's tables into the other buffer (last
				// read before the previous barrier)
				if (r + 1 < a.n_runs)
					build_run_tables(a, rs, end, s_runs[r + 2],
							 rs.tabs + ((r + 1) & 1u) * rs.tab_stride);
				w.tab = rs.tabs + (r & 1u) * rs.tab_stride;
				w.tab_i0 = start;
			}
			for (uint32_t i = start + rg; i < end; i += rgroups)
				run_item2<Idx>(a, w, i, s_dot, s_cnt);
			__syncthreads();
		}
	}
	return tile_root(a, t, s_dot, s_cnt, s_red);
}

// x 2^e.  A category's count lies above the largest of the positive ones only
// where its own value is zero or below: an invariant class keeps the count 0
// of its all-zero vectors while the others' fall with the tree, and by two
// factors 2^128 would be an infinity, its product with zero NaN.  For e <= 0
// (zero below 2^-252, which no sum with a term of at least 2^-126 beside it
// notices) two exact powers of two instead of ldexpf's cases.
__device__ __forceinline__ float scale_to(float x, int32_t e)
{
	if (e > 0)
		return ldexpf(x, e);
	const int32_t lo = max(e, -126), hi = max(e - lo, -126);
	x *= __uint_as_float((uint32_t)(127 + lo) << 23);
	return x * __uint_as_float((uint32_t)(127 + hi) << 23);
}

// Root of the pattern at column k of a tile (p of the whole) after the walk
// left pi . x and the exponent of every column in s_dot / s_cnt: category
// mixing and site values.  Returns the weighted site value.
__device__ __forceinline__ double
pattern_root(const float *s_dot, const int32_t *s_cnt, uint32_t tile, uint32_t C, uint32_t k,
	     uint32_t ldp, uint32_t p, double log_inv_c, double *site_lnl, double *cat_lnl,
	     const uint32_t *weights)
{
	const uint32_t wgt = weights[p];
	int32_t emax = INT32_MIN;
	for (uint32_t c = 0; c < C; c++)
		if (s_dot[c * tile + k] > 0.f)
			emax = max(emax, s_cnt[c * tile + k]);
	double site;
	if (emax == INT32_MIN) {
		site = -INFINITY;
	} else {
		// categories mixed in FP32 at the largest exponent; only the
		// exact exponent term and the constant join in FP64
		float acc = 0.f;
		for (uint32_t c = 0; c < C; c++)
			acc += scale_to(s_dot[c * tile + k], s_cnt[c * tile + k] - emax);
		site = (double)logf(acc) +
		       fma((double)emax, 0.69314718055994530942, log_inv_c);
	}
	site_lnl[p] = site;
	if (cat_lnl)
		for (uint32_t c = 0; c < C; c++)
			cat_lnl[(size_t)c * ldp + p] =
				log((double)s_dot[c * tile + k]) +
				(double)s_cnt[c * tile + k] * 0.69314718055994530942;
	return wgt ? site * (double)wgt : 0.0;
}

// Root of tile t: threads 0 .. tile-1 a pattern each, and the tile's weighted
// sum in a fixed order, returned in thread 0.  Ends with the block
// synchronised.
__device__ double tile_root(const TileArgs &a, uint32_t t, const float *s_dot,
			    const int32_t *s_cnt, double *s_red)
{
	const uint32_t tile = a.tile;
	const uint32_t tid = threadIdx.x;
	double contrib = 0.0;
	if (tid < tile)
		contrib = pattern_root(s_dot, s_cnt, tile, a.C, tid, a.ldp, t * tile + tid,
				       a.log_inv_c, a.site_lnl, a.cat_lnl, a.weights);
	// tile sum in a fixed order (warp shuffles, then warps in order)
	for (int off = 16; off > 0; off >>= 1)
		contrib += __shfl_down_sync(0xffffffffu, contrib, off);
	if ((tid & 31u) == 0 && tid < tile)
		s_red[tid >> 5] = contrib;
	__syncthreads();
	double tsum = 0.0;
	if (tid == 0)
		for (uint32_t w2 = 0; w2 < (tile + 31u) / 32u; w2++)
			tsum += s_red[w2];
	__syncthreads();
	return tsum;
}

// Sum `count` doubles at `sums` in a fixed order: lane l of warp 0 adds
// entries l, l + 32, ... in order, then a warp-shuffle tree.  The result is
// returned in thread 0; no barrier, so only warp 0 needs to call it (s_red
// is unused).  Pairwise FP64 over a few hundred block sums loses nothing at
// the FP32 form's accuracy, and keeps the serial tail of the launch to a
// few dependent FP64 adds (the pipe runs at 1/64 of the FP32 rate here).
// With `parts` > 1 every sum is given as that many parts, added in order first.
__device__ double block_fold(const double *sums, uint32_t count, double *s_red,
			     uint32_t parts = 1)
{
	(void)s_red;
	const uint32_t tid = threadIdx.x;
	if (tid >= 32)
		return 0.0;
	double sum = 0.0;
	for (uint32_t k = tid; k < count; k += 32) {
		double one = 0.0;
		for (uint32_t u = 0; u < parts; ++u)
			one += __ldcg(sums + k * parts + u);
		sum += one;
	}
	for (int off = 16; off > 0; off >>= 1)
		sum += __shfl_down_sync(0xffffffffu, sum, off);
	return sum;
}

// shared memory (byte offsets as prune4_runs_smem computes them):
// [dot: cols][cnt: cols/2][red: 32][ops][runs][tips], 16-byte aligned
// [list tables], [run table buffers: 2 * max_run * 2C * 5 float4][rates: C
// doubles, rounded up to even][eigensystem: 40 floats][lengths: 2n
// doubles], 16-byte aligned [slot partials: n_slots * cols][slot counts:
// n_slots * cols]
template <typename Idx, int kThreads>
__global__ void __launch_bounds__(kThreads, 1024 / kThreads)
	prune4_runs_kernel(PruneParams prm)
{
	const uint32_t cols = prm.tile * prm.C;
	const uint32_t tid = threadIdx.x;
	extern __shared__ __align__(16) double smem[];
	double *s_dot = smem;
	int32_t *s_cnt = (int32_t *)(smem + cols);
	double *s_red = smem + cols + (cols + 1) / 2; // one per warp
	NodeOp *s_ops = (NodeOp *)(s_red + 32);
	uint32_t *s_runs = (uint32_t *)(s_ops + prm.n);
	uint8_t *s_tips = (uint8_t *)(s_runs + ((prm.n_runs + 4) & ~3u));
	float4 *s_ptab = (float4 *)(((uintptr_t)s_tips +
				     (prm.tips_smem ? prm.num_leaves * prm.tile : 0u) + 15) &
				    ~(uintptr_t)15);
	float4 *s_tabs = s_ptab + (prm.ptab_smem ? prm.n * 2 * prm.C * 5 : 0u);
	const uint32_t tab_stride = prm.max_run * 2 * prm.C * 5;
	double *s_rate = (double *)(s_tabs + (prm.tables_inline ? 2 * tab_stride : 0u));
	float *s_eig = (float *)(s_rate + (prm.tables_inline ? (prm.C + 1) & ~1u : 0u));
	double *s_len = (double *)(s_eig + (prm.tables_inline ? 40 : 0));
	float4 *s_sp = (float4 *)(((uintptr_t)(s_len + (prm.lengths_smem ? 2 * prm.n : 0u)) +
				   15) &
				  ~(uintptr_t)15);
	int32_t *s_ss = (int32_t *)(s_sp + (size_t)prm.n_slots * cols);
	__shared__ unsigned s_last;

	if (prm.tables_inline) {
		const ModelDev *m = prm.model;
		if (tid < 16)
			s_eig[tid] = (float)m->V[tid];
		else if (tid < 32)
			s_eig[tid] = (float)m->Vinv[tid - 16];
		else if (tid < 36)
			s_eig[tid] = (float)m->lambda[tid - 32];
		else if (tid == 36)
			s_eig[36] = m->shortcuts ? 1.0f : 0.0f;
		else if (tid < 40 + prm.C && tid >= 40)
			s_rate[tid - 40] = prm.clock_rate * m->cat_rates[tid - 40];
		if (prm.lengths_smem)
			for (uint32_t k = tid; k < 2 * prm.n; k += blockDim.x)
				s_len[k] = prm.lengths[k];
	}

	const bool slots = prm.n_slots != 0;
	for (uint32_t k = tid; k < prm.n; k += blockDim.x) {
		NodeOp op = prm.ops[k];
		op.pad = slots ? prm.slots[k] : 0xFFFFFFu;
		s_ops[k] = op;
	}
	for (uint32_t k = tid; k <= prm.n_runs; k += blockDim.x)
		s_runs[k] = prm.runs[k];

	TileArgs a;
	a.tips = prm.tips;
	a.part = (float4 *)prm.partials;
	a.scales = prm.scales;
	a.ptab = (const float4 *)prm.ptab;
	a.pi = prm.pi;
	a.weights = prm.weights;
	a.site_lnl = prm.site_lnl;
	a.cat_lnl = prm.cat_lnl;
	a.ldp = prm.ldp;
	a.C = prm.C;
	a.L = prm.num_leaves;
	a.tile = prm.tile;
	a.n = prm.n;
	a.n_runs = prm.n_runs;
	a.tips_smem = prm.tips_smem;
	a.log_inv_c = prm.log_inv_c;
	a.model = prm.model;
	a.lengths = prm.lengths;
	a.matrices = prm.matrices;
	RunSmem rs{};
	if (slots) {
		rs.sp = s_sp;
		rs.ss = s_ss;
	}
	if (prm.tables_inline) {
		rs.tabs = s_tabs;
		rs.tab_stride = tab_stride;
		rs.eig = s_eig;
		rs.rate = s_rate;
		rs.len = prm.lengths_smem ? s_len : nullptr;
	}
	if (prm.ptab_smem) {
		// every table row of the list, once per block (one load latency)
		const uint32_t rows = prm.n * 2 * prm.C * 5;
		for (uint32_t k = tid; k < rows; k += blockDim.x)
			s_ptab[k] = a.ptab[k];
		a.ptab = s_ptab;
	}

	__syncthreads(); // the schedule and the table sources are staged
	double cta_sum = 0.0, cta_comp = 0.0; // thread 0: this block's tiles
	const uint32_t ntiles = prm.ldp / prm.tile;
	for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
		const double tsum = tile_walk<Idx>(a, t, (float *)s_dot, s_cnt,
						   s_red, s_ops, s_runs, s_tips, rs);
		if (tid == 0)
			neumaier_add(cta_sum, cta_comp, tsum);
	}
	if (prm.sums_host) { // the host folds the blocks' sums
		if (tid == 0)
			prm.sums_host[blockIdx.x] =
				isfinite(cta_sum) ? cta_sum + cta_comp : cta_sum;
		return;
	}
	if (tid == 0) {
		prm.block_sums[blockIdx.x] =
			isfinite(cta_sum) ? cta_sum + cta_comp : cta_sum;
		__threadfence();
		const unsigned tk = atomicAdd(prm.ticket, 1u);
		s_last = (tk == gridDim.x - 1u);
	}
	__syncthreads();
	if (!s_last)
		return;
	// without a host fold the last block folds the block sums in a
	// fixed-shape tree
	__threadfence();
	const double total = block_fold(prm.block_sums, gridDim.x, s_red);
	if (tid == 0) {
		*prm.lnl_out = total;
		if (prm.lnl_host)
			*prm.lnl_host = total;
		*prm.ticket = 0u;
	}
}

// ---------------------------------------------------------------------------
// Fused evaluation of a short list in one launch (FP32, four states, kC =
// 1, 2 or 4 categories, 128-pattern tiles: one thread per column, serial
// walk).  Every block converts the device eigensystem to FP32, builds the
// list's transition tables in shared memory with the same arithmetic as the
// transition kernels (so results match a two-kernel evaluation bit for
// bit), walks its tiles, and writes its sum to host-mapped memory, which
// the host folds (with sums_host null: the last block folds the sums and
// writes the root lnL to the device and to the host-mapped word).
//
// The walk is a chain: each entry needs the previous one's output, and its
// other child is a clean partial written long ago (mostly in DRAM) or a tip
// code.  Every clean input and tip code is known before the walk starts
// (the host marks each child's source in NodeOp::pad), so they are copied to
// shared memory kDirectAhead entries ahead of their use by cp.async, each
// thread for its own column (no barrier), the first ones before the tables
// are built.  The two previous outputs stay in registers; an older output is
// read back when needed (written by the same thread earlier).
//
// Every word the walk reads is staged in shared memory first: a kernel
// parameter read through the constant bank costs a cache miss of about 30 ns
// for each 64-byte line, one after another along the chain (reading the
// parameters through their generic address costs one load latency in all).
// (Four entries ahead cover a DRAM round trip at the walk's 500 cycles an
// entry; the batched kernel, whose blocks hold the largest list's tables,
// takes two so that two blocks share an SM.)
constexpr uint32_t kDirectAhead = 4, kBatchAhead = 2;

// Dynamic shared memory of the short-list kernels: tables of n entries, the
// list, the columns' root values and counts, and the input ring.
template <uint32_t kC, uint32_t kA> struct DirectSmem {
	static constexpr uint32_t kCols = 128 * kC;
	float4 *tab;
	NodeOp *ops;
	float4 *ring_x; // [kA][2][kCols]
	int32_t *ring_s;
	float *dot;
	int32_t *cnt;
	__device__ DirectSmem(unsigned char *base, uint32_t n)
	{
		tab = reinterpret_cast<float4 *>(base);
		ring_x = tab + n * 2 * kC * 5;
		ops = reinterpret_cast<NodeOp *>(ring_x + kA * 2 * kCols);
		ring_s = reinterpret_cast<int32_t *>(ops + n);
		dot = reinterpret_cast<float *>(ring_s + kA * 2 * kCols);
		cnt = reinterpret_cast<int32_t *>(dot + kCols);
	}
	static constexpr size_t bytes(uint32_t n)
	{
		return (size_t)n * (2 * kC * 5 * sizeof(float4) + sizeof(NodeOp)) +
		       kA * 2 * kCols * (sizeof(float4) + 4) + 8 * kCols;
	}
};

__device__ __forceinline__ void cp_async4(void *dst, const void *src)
{
	asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
			     (uint32_t)__cvta_generic_to_shared(dst)),
		     "l"(src)
		     : "memory");
}

// Columns a thread walks: two (patterns pl and pl + 64 of one category) where
// a tile has 512.  The walk's shared-memory reads are then shared (eight
// 16-byte table rows an entry and thread took 830 cycles of an SM's load path
// for 512 threads); with fewer columns the chain's latency, not the load
// path, sets the time.
template <uint32_t kC> constexpr uint32_t kDirectCols = kC == 4 ? 2 : 1;
template <uint32_t kC> constexpr uint32_t kDirectThreads = 128 * kC / kDirectCols<kC>;

// Per-thread constants of one tile's walk.
template <typename Idx, uint32_t kC> struct DirectCtx {
	static constexpr uint32_t kR = kDirectCols<kC>, kHalf = 128 / kR;
	const uint8_t *tips; // tips + the first pattern of this thread's 4-byte word
	float4 *part;        // the first column's element of slot 0
	int32_t *scales;
	uint32_t ldp, tip_shift; // bit position of the pattern's code in its word
	uint32_t col;            // first column inside the tile
	__device__ DirectCtx(const uint8_t *all_tips, float4 *p, int32_t *s, uint32_t ldp_,
			     uint32_t t)
	    : ldp(ldp_)
	{
		const uint32_t c = threadIdx.x / kHalf, pl = threadIdx.x % kHalf;
		const uint32_t pat = t * 128u + pl;
		tips = all_tips + (pat & ~3u);
		tip_shift = 8u * (pat & 3u); // the same 64 patterns further
		part = p + ((Idx)c * ldp_ + pat);
		scales = s + ((Idx)c * ldp_ + pat);
		col = c * 128u + pl;
	}
	__device__ Idx slot(uint32_t id) const { return (Idx)id * ((Idx)kC * ldp); }
};

// Copies entry i's clean inputs (and tip words) of this thread's columns into
// the ring; one cp.async group in any case.
template <typename Idx, uint32_t kC, uint32_t kA>
__device__ __forceinline__ void direct_issue(const DirectCtx<Idx, kC> &w, const NodeOp &op,
					     uint32_t i, const DirectSmem<kC, kA> &sm)
{
	typedef DirectCtx<Idx, kC> W;
	const uint32_t ids[2] = {op.left, op.right};
#pragma unroll
	for (uint32_t j = 0; j < 2; ++j) {
		const uint32_t sr = (op.pad >> (8 * j)) & 0xFFu;
		const uint32_t at = ((i & (kA - 1)) * 2 + j) * (128 * kC) + w.col;
		if (sr == kSrcTip) {
			const uint8_t *tips = w.tips + (size_t)(ids[j] & ~kTipBit) * w.ldp;
#pragma unroll
			for (uint32_t r = 0; r < W::kR; ++r)
				cp_async4(sm.ring_s + at + W::kHalf * r, tips + W::kHalf * r);
		} else if (sr == kSrcClean) {
			const Idx ix = w.slot(ids[j]);
#pragma unroll
			for (uint32_t r = 0; r < W::kR; ++r) {
				cp_async16(sm.ring_x + at + W::kHalf * r,
					   w.part + ix + W::kHalf * r);
				cp_async4(sm.ring_s + at + W::kHalf * r,
					  w.scales + ix + W::kHalf * r);
			}
		}
	}
}

// The first kA entries' inputs of a tile.
template <typename Idx, uint32_t kC, uint32_t kA>
__device__ __forceinline__ void direct_prefetch(const DirectCtx<Idx, kC> &w, const NodeOp *ops,
						uint32_t n, const DirectSmem<kC, kA> &sm)
{
#pragma unroll
	for (uint32_t i = 0; i < kA; ++i) {
		if (i < n)
			direct_issue<Idx, kC, kA>(w, ops[i], i, sm);
		cp_async_commit();
	}
}

// The serial walk of a tile after direct_prefetch: leaves pi . x and the
// exponent of the root in sm.dot / sm.cnt (not synchronised).
template <typename Idx, uint32_t kC, uint32_t kA>
__device__ __forceinline__ void direct_walk(const DirectCtx<Idx, kC> &w, uint32_t n,
					    const DirectSmem<kC, kA> &sm, const float *s_pi)
{
	typedef DirectCtx<Idx, kC> W;
	constexpr uint32_t kR = W::kR, kHalf = W::kHalf;
	const uint32_t c = w.col >> 7;
	float4 y0[kR], y1[kR];
	int32_t c0[kR], c1[kR];
#pragma unroll
	for (uint32_t r = 0; r < kR; ++r) {
		y0[r] = y1[r] = make_float4(0.f, 0.f, 0.f, 0.f);
		c0[r] = c1[r] = 0;
	}
	for (uint32_t i = 0; i < n; ++i) {
		const NodeOp op = sm.ops[i];
		const float4 *tl = sm.tab + ((size_t)(2 * i) * kC + c) * 5;
		float4 in[2][kR];
		int32_t cnt[kR];
#pragma unroll
		for (uint32_t r = 0; r < kR; ++r)
			cnt[r] = 0;
		const uint32_t ids[2] = {op.left, op.right};
		cp_async_wait<kA - 1>(); // this entry's inputs
#pragma unroll
		for (uint32_t j = 0; j < 2; ++j) {
			const float4 *tb = tl + 5 * kC * j;
			const uint32_t sr = (op.pad >> (8 * j)) & 0xFFu;
			const uint32_t at = ((i & (kA - 1)) * 2 + j) * (128 * kC) + w.col;
			if (sr == kSrcTip) {
#pragma unroll
				for (uint32_t r = 0; r < kR; ++r)
					in[j][r] = tb[((uint32_t)sm.ring_s[at + kHalf * r] >>
						       w.tip_shift) &
						      0xFFu];
			} else {
				// the internal child's vectors, then one product (one
				// copy of the code for every source)
				float4 x[kR];
				int32_t sc[kR];
				if (sr == kSrcClean) {
#pragma unroll
					for (uint32_t r = 0; r < kR; ++r) {
						x[r] = sm.ring_x[at + kHalf * r];
						sc[r] = sm.ring_s[at + kHalf * r];
					}
				} else if (sr == kSrcPrev) {
#pragma unroll
					for (uint32_t r = 0; r < kR; ++r) {
						x[r] = y0[r];
						sc[r] = c0[r];
					}
				} else if (sr == kSrcPrev2) {
#pragma unroll
					for (uint32_t r = 0; r < kR; ++r) {
						x[r] = y1[r];
						sc[r] = c1[r];
					}
				} else {
					const Idx ix = w.slot(ids[j]);
#pragma unroll
					for (uint32_t r = 0; r < kR; ++r) {
						x[r] = w.part[ix + kHalf * r];
						sc[r] = w.scales[ix + kHalf * r];
					}
				}
				const float4 rows[4] = {tb[0], tb[1], tb[2], tb[3]};
#pragma unroll
				for (uint32_t r = 0; r < kR; ++r) {
					in[j][r] = v4_apply(rows, x[r]);
					cnt[r] += sc[r];
				}
			}
		}
		// the ring slot just consumed takes entry i + kA
		if (i + kA < n)
			direct_issue<Idx, kC, kA>(w, sm.ops[i + kA], i, sm);
		cp_async_commit();
		const Idx ox = w.slot(op.out);
#pragma unroll
		for (uint32_t r = 0; r < kR; ++r) {
			float4 y = v4_mul(in[0][r], in[1][r]);
			cnt[r] += rescale_pow2(y);
			w.part[ox + kHalf * r] = y;
			w.scales[ox + kHalf * r] = cnt[r];
			y1[r] = y0[r];
			c1[r] = c0[r];
			y0[r] = y;
			c0[r] = cnt[r];
		}
	}
#pragma unroll
	for (uint32_t r = 0; r < kR; ++r) {
		sm.dot[w.col + kHalf * r] = root_dot4(s_pi, y0[r]);
		sm.cnt[w.col + kHalf * r] = c0[r];
	}
}

// Root of a tile, thread = pattern (tid < 128) with its weight: tile_root's
// arithmetic with everything it needs at hand.  Returns the tile's sum in
// thread 0; ends with the block synchronised.
template <uint32_t kC>
__device__ __forceinline__ double direct_root(const float *s_dot, const int32_t *s_cnt,
					      double *site_lnl, uint32_t p, uint32_t weight,
					      double log_inv_c, double *s_red)
{
	const uint32_t tid = threadIdx.x;
	if (tid < 128) {
		float dot[kC];
		int32_t cnt[kC], emax = INT32_MIN;
#pragma unroll
		for (uint32_t k = 0; k < kC; k++) {
			dot[k] = s_dot[k * 128 + tid];
			cnt[k] = s_cnt[k * 128 + tid];
			if (dot[k] > 0.f)
				emax = max(emax, cnt[k]);
		}
		double site = -INFINITY;
		if (emax != INT32_MIN) {
			float acc = 0.f;
#pragma unroll
			for (uint32_t k = 0; k < kC; k++)
				acc += scale_to(dot[k], cnt[k] - emax);
			site = (double)logf(acc) +
			       fma((double)emax, 0.69314718055994530942, log_inv_c);
		}
		site_lnl[p] = site;
		double contrib = weight ? site * (double)weight : 0.0;
		for (int off = 16; off > 0; off >>= 1)
			contrib += __shfl_down_sync(0xffffffffu, contrib, off);
		if ((tid & 31u) == 0)
			s_red[tid >> 5] = contrib;
	}
	__syncthreads();
	double tsum = 0.0;
	if (tid == 0)
		for (uint32_t q = 0; q < 4; q++)
			tsum += s_red[q];
	__syncthreads();
	return tsum;
}

// The list's transition tables (entry, side, category) in shared memory,
// laid out as ptab4_kernel's, from the FP32 eigensystem in s_eig and the
// scaled category rates in s_rate (same arithmetic as the transition
// kernels).
template <uint32_t kC>
__device__ __forceinline__ void direct_tables(const ModelDev *m, const float *s_eig,
					      const double *s_rate,
					      const double (&length)[kDirectCols<kC>], uint32_t n,
					      float4 *s_tab)
{
	// a table a thread and round; `length`: of the table's entry and side
#pragma unroll
	for (uint32_t r = 0; r < kDirectCols<kC>; ++r) {
		const uint32_t at = threadIdx.x + r * kDirectThreads<kC>;
		if (at >= n * 2 * kC)
			break;
		float P[16];
		transition4f_eig(m, s_eig, length[r] * s_rate[at % kC], P);
		float4 *out = s_tab + at * 5;
#pragma unroll
		for (int k = 0; k < 4; k++)
			out[k] = make_float4(P[k], P[4 + k], P[8 + k], P[12 + k]);
		out[4] = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
	}
}
template <uint32_t kC>
__device__ __forceinline__ void direct_lengths(const double *lengths, uint32_t n,
					       double (&length)[kDirectCols<kC>])
{
#pragma unroll
	for (uint32_t r = 0; r < kDirectCols<kC>; ++r) {
		const uint32_t at = threadIdx.x + r * kDirectThreads<kC>;
		length[r] = at < n * 2 * kC ? lengths[at / kC] : 0.0;
	}
}

template <typename Idx, uint32_t kC>
__global__ void __launch_bounds__(kDirectThreads<kC>, 8 / kC)
prune4_direct_kernel(const __grid_constant__ DirectParams prm)
{
	constexpr uint32_t kTile = 128;
	extern __shared__ __align__(16) unsigned char direct_smem[];
	__shared__ float s_eig[37];
	__shared__ double s_rate[kC];
	__shared__ float s_pi[4];
	__shared__ double s_red[32];
	__shared__ unsigned s_last;
	const uint32_t tid = threadIdx.x;
	const uint32_t n = prm.n;
	const uint32_t ntiles = prm.ldp / kTile;
	const DirectSmem<kC, kDirectAhead> sm(direct_smem, n);
	float4 *part = (float4 *)prm.partials;
	// the parameters through their generic address (the constant bank would
	// serve a warp's different words one after another)
	const DirectParams *gp = &prm;
	asm volatile("" : "+l"(gp));
	double length[kDirectCols<kC>];
	direct_lengths<kC>(gp->lengths, n, length);
	if (tid < n)
		sm.ops[tid] = gp->ops[tid];
	else if (tid >= 64 && tid < 64 + 37)
		s_eig[tid - 64] = gp->eig[tid - 64];
	else if (tid >= 104 && tid < 104 + kC)
		s_rate[tid - 104] = gp->rate[tid - 104];
	else if (tid >= 112 && tid < 116)
		s_pi[tid - 112] = (float)gp->pi[tid - 112];
	// the first pattern tile's addresses and weights, and the constants the
	// root needs, under the same wait
	DirectCtx<Idx, kC> w(prm.tips, part, prm.scales, prm.ldp, blockIdx.x);
	uint32_t weight = 0;
	if (tid < kTile && blockIdx.x < ntiles)
		weight = prm.weights[blockIdx.x * kTile + tid];
	const double log_inv_c = prm.log_inv_c;
	double *site_lnl = prm.site_lnl, *sums_host = prm.sums_host;
	asm volatile("" ::"l"(w.tips), "l"(w.part), "l"(w.scales), "r"(w.ldp), "d"(log_inv_c),
		     "l"(site_lnl), "l"(sums_host));
	__syncthreads();
	// clean inputs of the first entries of the first tile, in flight while
	// the tables are built
	if (blockIdx.x < ntiles)
		direct_prefetch<Idx, kC, kDirectAhead>(w, sm.ops, n, sm);
	direct_tables<kC>(prm.model, s_eig, s_rate, length, n, sm.tab);
	__syncthreads();

	double cta_sum = 0.0, cta_comp = 0.0; // thread 0: this block's tiles
	for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
		if (t != blockIdx.x) {
			w = DirectCtx<Idx, kC>(prm.tips, part, prm.scales, prm.ldp, t);
			if (tid < kTile)
				weight = prm.weights[t * kTile + tid];
			direct_prefetch<Idx, kC, kDirectAhead>(w, sm.ops, n, sm);
		}
		direct_walk<Idx, kC, kDirectAhead>(w, n, sm, s_pi);
		__syncthreads();
		const double tsum = direct_root<kC>(sm.dot, sm.cnt, site_lnl, t * kTile + tid,
						    weight, log_inv_c, s_red);
		if (gridDim.x >= ntiles) { // this block's only tile
			cta_sum = tsum;
			break;
		}
		if (tid == 0)
			neumaier_add(cta_sum, cta_comp, tsum);
	}
	if (sums_host) { // the host folds the blocks' sums
		if (tid == 0)
			sums_host[blockIdx.x] =
				isfinite(cta_sum) ? cta_sum + cta_comp : cta_sum;
		return;
	}
	if (tid == 0) {
		prm.block_sums[blockIdx.x] =
			isfinite(cta_sum) ? cta_sum + cta_comp : cta_sum;
		__threadfence();
		const unsigned tk = atomicAdd(prm.ticket, 1u);
		s_last = (tk == gridDim.x - 1u);
	}
	__syncthreads();
	if (!s_last)
		return;
	__threadfence();
	const double total = block_fold(prm.block_sums, gridDim.x, s_red);
	if (tid == 0) {
		*prm.lnl_out = total;
		*prm.lnl_host = total;
		*prm.ticket = 0u;
	}
}

constexpr uint32_t kBatchMembers = 256;

// prefix[m] = items of the members before m, for m up to M, by warp 0; ends
// with the block synchronised.  (One thread adding them up waited for a load a
// member: the short-list kernel of 32 members took 45 us, now 33.)
template <typename F>
__device__ __forceinline__ void member_prefix(uint32_t M, uint32_t *prefix, F items)
{
	if (threadIdx.x < 32) {
		uint32_t before = 0;
		for (uint32_t m0 = 0; m0 < M; m0 += 32) {
			const uint32_t m = m0 + threadIdx.x;
			const uint32_t mine = m < M ? items(m) : 0u;
			uint32_t sum = mine;
			for (uint32_t off = 1; off < 32; off *= 2) {
				const uint32_t v = __shfl_up_sync(0xffffffffu, sum, off);
				sum += threadIdx.x >= off ? v : 0u;
			}
			if (m < M)
				prefix[m] = before + sum - mine;
			before += __shfl_sync(0xffffffffu, sum, 31);
		}
		if (threadIdx.x == 0)
			prefix[M] = before;
	}
	__syncthreads();
}

// The member whose items hold w.
__device__ __forceinline__ uint32_t member_of(const uint32_t *prefix, uint32_t M, uint32_t w)
{
	uint32_t lo = 0, hi = M;
	while (hi - lo > 1) {
		const uint32_t mid = (lo + hi) >> 1;
		if (prefix[mid] <= w)
			lo = mid;
		else
			hi = mid;
	}
	while (lo + 1 < M && prefix[lo + 1] <= w)
		++lo;
	return lo;
}

// Batched short lists: persistent blocks take (member, 128-pattern tile)
// items of the members whose step is direct and has kC categories from
// their own counter (work_next[1], [2], [3] for 4, 2, 1 categories;
// costliest member first); a block that moves to another
// member copies its list, marks every child's source, converts the
// member's eigensystem to FP32 and builds the list's tables (as the
// single-calculator kernel does, so values match it), then walks the tile
// serially with clean inputs copied two entries ahead.  Each tile's
// weighted sum goes to the member's tile slot; the block finishing a
// member's last tile folds its sums (fixed order).
template <typename Idx, uint32_t kC>
__global__ void __launch_bounds__(kDirectThreads<kC>, 8 / kC)
prune4_direct_batch_kernel(BatchParams bp)
{
	constexpr uint32_t kTile = 128;
	extern __shared__ __align__(16) unsigned char direct_smem[];
	const DirectSmem<kC, kBatchAhead> sm(direct_smem, kDirectMax);
	NodeOp *const s_ops = sm.ops;
	__shared__ float s_eig[37];
	__shared__ double s_rate[kC];
	__shared__ float s_pi[4];
	__shared__ double s_red[32];
	__shared__ uint32_t s_prefix[kBatchMembers + 1];
	__shared__ uint32_t s_work;
	__shared__ unsigned s_last;
	const uint32_t tid = threadIdx.x;
	const uint32_t M = bp.num_members;
	member_prefix(M, s_prefix, [&](uint32_t m) {
		const MemberStep &st = bp.steps[m];
		return st.n && st.kind == kListShort && bp.members[m].C == kC
			       ? bp.members[m].ldp / kTile
			       : 0u;
	});
	const uint32_t total = s_prefix[M];
	uint32_t cur = 0xFFFFFFFFu, n = 0;
	const MemberDesc *md = nullptr;
	double log_inv_c = 0.0;
	// items come in chunks of consecutive tiles (mostly of one member), so
	// that a block rebuilds a member's tables less often: as many as a block
	// gets, at most four (30 members of 13 tiles on 304 blocks, this kernel
	// alone: 65 us with always four, 45 with two)
	const uint32_t chunk = min(4u, max(1u, (total + gridDim.x - 1u) / gridDim.x));
	for (;;) {
		if (tid == 0)
			s_work = atomicAdd(bp.work_next + (kC == 4 ? 1 : kC == 2 ? 2 : 3), chunk);
		__syncthreads();
		const uint32_t w0 = s_work;
		__syncthreads();
		if (w0 >= total)
			break;
	for (uint32_t w = w0; w < min(w0 + chunk, total); ++w) {
		const uint32_t m = member_of(s_prefix, M, w), t = w - s_prefix[m];
		md = &bp.members[m];
		if (m != cur) {
			const MemberStep st = bp.steps[m];
			n = st.n;
			const NodeOp *g_ops = (const NodeOp *)md->stage;
			for (uint32_t k = tid; k < n; k += blockDim.x)
				s_ops[k] = g_ops[k];
			const ModelDev *mod = md->model;
			if (tid < 16) {
				s_eig[tid] = (float)mod->V[tid];
				s_eig[16 + tid] = (float)mod->Vinv[tid];
			} else if (tid < 20) {
				s_eig[32 + tid - 16] = (float)mod->lambda[tid - 16];
			} else if (tid == 20) {
				s_eig[36] = mod->shortcuts ? 1.0f : 0.0f;
			} else if (tid >= 32 && tid < 32 + kC) {
				s_rate[tid - 32] = st.clock_rate * mod->cat_rates[tid - 32];
			} else if (tid >= 64 && tid < 68) {
				s_pi[tid - 64] =
					(float)((const double *)(md->stage + md->off_pi))[tid - 64];
			}
			__syncthreads();
			// where each child comes from (as the host classifies it for
			// the single-calculator kernel)
			uint32_t marks = 0;
			if (tid < n) {
				const NodeOp op = s_ops[tid];
				const uint32_t ids[2] = {op.left, op.right};
				for (int j = 0; j < 2; ++j) {
					const uint32_t id = ids[j];
					uint32_t sr = kSrcClean;
					if (id & kTipBit) {
						sr = kSrcTip;
					} else if (tid >= 1 && id == s_ops[tid - 1].out) {
						sr = kSrcPrev;
					} else if (tid >= 2 && id == s_ops[tid - 2].out) {
						sr = kSrcPrev2;
					} else {
						for (uint32_t k = 0; k + 2 < tid; ++k)
							if (s_ops[k].out == id) {
								sr = kSrcEarlier;
								break;
							}
					}
					marks |= sr << (8 * j);
				}
			}
			__syncthreads();
			if (tid < n)
				s_ops[tid].pad = marks;
			__syncthreads();
			log_inv_c = md->log_inv_c;
			double length[kDirectCols<kC>];
			direct_lengths<kC>((const double *)(md->stage + md->off_in), n, length);
			direct_prefetch<Idx, kC, kBatchAhead>(
				DirectCtx<Idx, kC>(md->tips, (float4 *)md->partials, md->scales,
						   md->ldp, t),
				s_ops, n, sm);
			direct_tables<kC>(mod, s_eig, s_rate, length, n, sm.tab);
			cur = m;
			__syncthreads();
		} else {
			direct_prefetch<Idx, kC, kBatchAhead>(
				DirectCtx<Idx, kC>(md->tips, (float4 *)md->partials, md->scales,
						   md->ldp, t),
				s_ops, n, sm);
		}
		const uint32_t weight = tid < kTile ? md->weights[t * kTile + tid] : 0u;
		direct_walk<Idx, kC, kBatchAhead>(
			DirectCtx<Idx, kC>(md->tips, (float4 *)md->partials, md->scales, md->ldp, t),
			n, sm, s_pi);
		__syncthreads();
		const double tsum = direct_root<kC>(sm.dot, sm.cnt, md->site_lnl, t * kTile + tid,
						    weight, log_inv_c, s_red);
		const uint32_t tiles = md->ldp / kTile;
		if (tid == 0) {
			md->tile_sums[t] = tsum;
			__threadfence();
			const unsigned tk = atomicAdd(md->ticket, 1u);
			s_last = (tk == tiles - 1u);
		}
		__syncthreads();
		if (s_last) {
			__threadfence();
			const double lnl = block_fold(md->tile_sums, tiles, s_red);
			if (tid == 0) {
				bp.lnl_out[m] = lnl;
				*md->ticket = 0u;
			}
		}
		__syncthreads();
	}
	}
}

// ---------------------------------------------------------------------------
// Batched evaluation: many calculators (chains) in one launch.

__global__ void __launch_bounds__(32) ptab4_batch_kernel(BatchParams bp)
{
	const uint32_t m = blockIdx.y;
	const MemberStep st = bp.steps[m];
	if (st.n == 0 || st.kind == kListShort)
		return;
	const MemberDesc &md = bp.members[m];
	const uint32_t C = md.C;
	const uint32_t id = blockIdx.x * blockDim.x + threadIdx.x;
	if (id >= st.n * 2u * C)
		return;
	const uint32_t c = id % C, es = id / C;
	const double *lengths = (const double *)(md.stage + md.off_in);
	const double d = lengths[es] * (st.clock_rate * md.model->cat_rates[c]);
	float P[16];
	transition4f(md.model, d, P);
	float *out = md.ptab + (size_t)id * 20;
	for (int k = 0; k < 4; k++)
		for (int j = 0; j < 4; j++)
			out[k * 4 + j] = P[j * 4 + k];
	for (int j = 0; j < 4; j++)
		out[16 + j] = 1.0f;
}

// Persistent blocks take (member, tile) work items from a counter; members
// are visited in the order of the descriptor array (the host puts the
// costliest first).  Each tile's weighted sum goes to the member's tile
// slots; the block that finishes a member's last tile folds that member's
// sums (in the order of its own tiles, MemberStep::fold, so that the result
// depends neither on scheduling nor on the other members).
template <typename Idx>
__global__ void __launch_bounds__(512, 2) prune4_batch_kernel(BatchParams bp)
{
	__shared__ uint32_t s_prefix[kBatchMembers + 1];
	__shared__ uint32_t s_work;
	__shared__ unsigned s_last;
	extern __shared__ double smem[];
	const uint32_t tid = threadIdx.x;
	const uint32_t M = bp.num_members;
	double *s_dot = smem;
	int32_t *s_cnt = (int32_t *)(smem + bp.max_cols);
	double *s_red = smem + bp.max_cols + (bp.max_cols + 1) / 2;
	NodeOp *s_ops = (NodeOp *)(s_red + 2 * blockDim.x);
	uint8_t *s_tips = (uint8_t *)s_ops + bp.smem_ops_bytes;
	float4 *s_ptab = (float4 *)(((uintptr_t)s_tips + bp.smem_tips_bytes + 15) &
				    ~(uintptr_t)15);

	member_prefix(M, s_prefix, [&](uint32_t m) {
		const MemberStep &st = bp.steps[m];
		return st.n && st.kind == kListRuns ? bp.members[m].ldp / st.tile : 0u;
	});
	const uint32_t total = s_prefix[M];
	uint32_t cur = 0xFFFFFFFFu;
	TileArgs a;
	uint32_t fold = 0;
	uint32_t *s_runs = nullptr;
	for (;;) {
		if (tid == 0)
			s_work = atomicAdd(bp.work_next, 1u);
		__syncthreads();
		const uint32_t w = s_work;
		__syncthreads();
		if (w >= total)
			break;
		const uint32_t m = member_of(s_prefix, M, w), t = w - s_prefix[m];
		const MemberDesc &md = bp.members[m];
		if (m != cur) {
			const MemberStep st = bp.steps[m];
			a.tips = md.tips;
			a.part = (float4 *)md.partials;
			a.scales = md.scales;
			a.ptab = (const float4 *)md.ptab;
			a.pi = (const double *)(md.stage + md.off_pi);
			a.weights = md.weights;
			a.site_lnl = md.site_lnl;
			a.cat_lnl = nullptr;
			a.ldp = md.ldp;
			a.C = md.C;
			a.L = md.L;
			a.tile = st.tile;
			fold = st.fold;
			a.n = st.n;
			a.n_runs = st.n_runs;
			a.tips_smem = st.tips_smem;
			a.log_inv_c = md.log_inv_c;
			const NodeOp *g_ops = (const NodeOp *)md.stage;
			const uint32_t *g_runs = (const uint32_t *)(md.stage + md.off_runs);
			s_runs = (uint32_t *)(s_ops + st.n);
			for (uint32_t k = tid; k < st.n; k += blockDim.x) {
				NodeOp op = g_ops[k];
				op.pad = 0xFFFFFFu; // no slots
				s_ops[k] = op;
			}
			for (uint32_t k = tid; k <= st.n_runs; k += blockDim.x)
				s_runs[k] = g_runs[k];
			// a small list's tables in shared memory (see the single-
			// calculator kernel)
			const uint32_t rows = st.n * 2 * md.C * 5;
			if (rows * sizeof(float4) <= bp.smem_ptab_bytes) {
				for (uint32_t k = tid; k < rows; k += blockDim.x)
					s_ptab[k] = ((const float4 *)md.ptab)[k];
				a.ptab = s_ptab;
			}
			cur = m;
			__syncthreads();
		}
		tile_walk<Idx>(a, t, (float *)s_dot, s_cnt, s_red, s_ops, s_runs, s_tips);
		// the sums of every 32 patterns, or of a tile of 16
		const uint32_t tiles = md.ldp / a.tile, units = (a.tile + 31u) / 32u;
		if (tid < 32) {
			if (tid < units)
				md.tile_sums[t * units + tid] = s_red[tid];
			__threadfence();
			__syncwarp();
			if (tid == 0)
				s_last = atomicAdd(md.ticket, 1u) == tiles - 1u;
		}
		__syncthreads();
		if (s_last) {
			__threadfence();
			if (a.tile < min(fold, 32u)) {
				// halves of a warp's patterns: its sum over again, from
				// the site values, in tile_root's order
				for (uint32_t p = tid; p < md.ldp; p += blockDim.x) {
					const uint32_t wgt = md.weights[p];
					double sum = wgt ? __ldcg(md.site_lnl + p) * (double)wgt : 0.0;
					for (int off = 16; off > 0; off >>= 1)
						sum += __shfl_down_sync(0xffffffffu, sum, off);
					if ((tid & 31u) == 0)
						md.tile_sums[p / 32u] = sum;
				}
				__syncthreads();
			}
			const double lnl = block_fold(md.tile_sums, md.ldp / fold, s_red,
						      (fold + 31u) / 32u);
			if (tid == 0) {
				bp.lnl_out[m] = lnl;
				*md.ticket = 0u;
			}
		}
		__syncthreads();
	}
}
