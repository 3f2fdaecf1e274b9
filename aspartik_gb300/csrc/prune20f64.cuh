// prune20f64.cuh -- 20-state pruning, plain FP64 form, products on the
// integer pipes (soft64.cuh).  Included by kernels4.cu inside its anonymous
// namespace after prune20.cuh (uses cp_async16 and the transposed FP64
// tables of ptab20_kernel).
//
// An internal child takes 400 FP64 multiply-adds a column, 64 cycles each of
// a scheduler partition's FP64 pipe; as integers a term takes about 11
// issue slots.  A group of four warps owns 64 patterns of one category:
// thread (w, lane) computes states 5 w .. 5 w + 4 of patterns lane and
// lane + 32, so that a table word (the same for the whole warp) serves two
// columns and a significand five states: shared-memory reads (26 cycles of
// the SM's load path for a state k) then stay below the arithmetic (110
// issue slots of one scheduler).  Per entry a group
//   1. splits both internal children's 64 x 20 doubles into significands and
//      exponents in shared memory (the tables of the entry arrived by
//      cp.async while the previous entry was computed);
//   2. finds every sum's largest exponent, then adds the aligned products;
//   3. multiplies the children, votes on the rescaling across its warps
//      (cpu4.rs:403-433's rule with 20 entries) and writes the rows through
//      shared memory as coalesced 16-byte stores.
// The list is walked run by run (prm.runs) by 1 to 4 groups a block, group g
// taking entries g, g + G, ... of a run, so that a small alignment still
// fills the SMs.  A column with a value that is not a positive normal number
// (or any, where the table holds one) takes the FP64 instructions.
//
// Whole tree, 61 taxa x 2,003 patterns, four categories: 1,055 us with FP64
// instructions (one thread a column, 64 blocks), 240 us here with four groups
// (375 with one, 290 with two); a product term takes 16 cycles of a scheduler
// at four warps each, 37 at one.
//
// Category c of a tile is a block of its own: the last of a tile's C blocks
// to finish mixes the categories (one logarithm a pattern, as finish_root)
// and writes the tile's weighted sum to mapped host memory.

constexpr uint32_t kP20Tile = 64;
constexpr uint32_t kTab20Chunks = sizeof(SoftTab20) / 16; // 336
constexpr uint32_t kXStride = kP20Tile + 1;
// significands of a child: 2^62 <= X < 2^63; of a table entry 2^59 <= M <
// 2^60, value M 2^(E - 1082), so that twenty products fit 64 bits
constexpr int32_t kSoftBias20 = 1082;
constexpr int32_t kSoftDotBias20 = 2103;
// a sum loses a unit or so of its terms' last place in each of 20
// truncations; half a unit of each shift and three quarters of each product
// are given back at once
constexpr uint64_t kSoftLoss20 = 25;

struct __align__(16) P20Group {
	SoftTab20 tab[2][2]; // [buffer][side]
	uint2 x[2][kS20][kXStride];     // [side][k][pattern] (hi, lo)
	uint32_t xe[2][kS20][kXStride]; // exponent in both halves; bit 15: special
	uint8_t below[4][kP20Tile];
	uint8_t code[2][kP20Tile];
	double dot[kP20Tile]; // root
};
constexpr uint32_t kYStride = 22; // doubles a staged row, 16-byte aligned
static_assert(sizeof(uint2) * 2 * kS20 * kXStride >= sizeof(double) * kP20Tile * kYStride,
	      "the rows are staged over the significands");

__device__ __forceinline__ void bar_group(uint32_t g)
{
	asm volatile("bar.sync %0, 128;" ::"r"(g + 1) : "memory");
}

// Sums of five states for one child and two columns.  Returns a mask of the
// columns (bit 0, 1) with a special value; the caller's sums of those are
// meaningless.
struct P20Vec {
	uint64_t m[2][5];
	int32_t e[2][5];
};

__device__ __forceinline__ uint32_t soft_dot20(const SoftTab20 &t, const uint2 (*x)[kXStride],
					       const uint32_t (*xe)[kXStride], uint32_t w,
					       uint32_t lane, P20Vec &v)
{
	uint32_t mx[2][3] = {{0, 0, 0}, {0, 0, 0}};
#pragma unroll 5
	for (int k = 0; k < kS20; ++k) {
		const uint4 pe = *reinterpret_cast<const uint4 *>(t.rec[k][w]);
#pragma unroll
		for (int c = 0; c < 2; ++c) {
			const uint32_t e = xe[k][lane + 32 * c];
			mx[c][0] = soft_max2(mx[c][0], pe.x + e);
			mx[c][1] = soft_max2(mx[c][1], pe.y + e);
			mx[c][2] = soft_max2(mx[c][2], pe.z + e);
		}
	}
	const uint32_t special = ((mx[0][0] >> 15) & 1u) | (((mx[1][0] >> 15) & 1u) << 1);
#pragma unroll
	for (int c = 0; c < 2; ++c)
#pragma unroll
		for (int i = 0; i < 5; ++i)
			v.m[c][i] = kSoftLoss20;
#pragma unroll 2
	for (int k = 0; k < kS20; ++k) {
		const uint4 *r = reinterpret_cast<const uint4 *>(t.rec[k][w]);
		const uint4 pe = r[0], r1 = r[1], r2 = r[2];
		const uint2 r3 = *reinterpret_cast<const uint2 *>(r + 3);
		const uint32_t hi[5] = {r1.x, r1.y, r1.z, r1.w, r2.x};
		const uint32_t lo[5] = {r2.y, r2.z, r2.w, r3.x, r3.y};
#pragma unroll
		for (int c = 0; c < 2; ++c) {
			const uint32_t e = xe[k][lane + 32 * c];
			const uint2 xx = x[k][lane + 32 * c];
			const uint32_t d01 = mx[c][0] - (pe.x + e), d23 = mx[c][1] - (pe.y + e),
				       d4 = mx[c][2] - (pe.z + e);
			const uint32_t d[5] = {d01 & 0xFFFFu, d01 >> 16, d23 & 0xFFFFu, d23 >> 16,
					       d4 & 0xFFFFu};
#pragma unroll
			for (int i = 0; i < 5; ++i)
				v.m[c][i] += soft_shr(soft_prod(xx.x, xx.y, hi[i], lo[i]), d[i]);
		}
	}
#pragma unroll
	for (int c = 0; c < 2; ++c) {
		const uint32_t e[5] = {mx[c][0] & 0xFFFFu, mx[c][0] >> 16, mx[c][1] & 0xFFFFu,
				       mx[c][1] >> 16, mx[c][2] & 0xFFFFu};
#pragma unroll
		for (int i = 0; i < 5; ++i) {
			const int lz = soft_clz((uint32_t)(v.m[c][i] >> 32));
			v.m[c][i] <<= lz;
			v.e[c][i] = (int32_t)e[i] - kSoftDotBias20 - lz;
		}
	}
	return special;
}

__device__ __forceinline__ void soft_tip20(const SoftTab20 &t, const uint8_t *code, uint32_t w,
					   uint32_t lane, P20Vec &v)
{
#pragma unroll
	for (int c = 0; c < 2; ++c) {
		const uint32_t *r = t.rec[code[lane + 32 * c]][w];
#pragma unroll
		for (int i = 0; i < 5; ++i) {
			v.m[c][i] = (((uint64_t)r[4 + i] << 32) | r[9 + i]) << 4;
			v.e[c][i] = (int32_t)reinterpret_cast<const uint16_t *>(r)[i] -
				    kSoftBias20 - 4;
		}
	}
}

// State i of an entry in FP64 instructions (prune20_kernel's arithmetic).
__device__ __noinline__ double p20_plain(const PruneParams &prm, uint32_t left, uint32_t right,
					 uint32_t e, uint32_t c, uint32_t p, uint32_t i)
{
	double out[2];
	const uint32_t ids[2] = {left, right};
	for (int j = 0; j < 2; ++j) {
		const double *tab = (const double *)prm.ptab +
				    ((size_t)(2 * e + j) * prm.C + c) * (kP20Rows * kS20);
		if (ids[j] & kTipBit) {
			const uint32_t code =
				prm.tips[(size_t)(ids[j] & ~kTipBit) * prm.ldp + p];
			out[j] = tab[min(code, (uint32_t)kS20) * kS20 + i];
		} else {
			const double *x = (const double *)prm.partials +
					  (((size_t)ids[j] * prm.C + c) * prm.ldp + p) * kS20;
			double s = x[0] * tab[i];
			for (int k = 1; k < kS20; ++k)
				s = fma(x[k], tab[k * kS20 + i], s);
			out[j] = s;
		}
	}
	return out[0] * out[1];
}

__global__ void __launch_bounds__(512) prune20_f64_kernel(PruneParams prm)
{
	extern __shared__ __align__(16) unsigned char p20_smem[];
	const uint32_t G = blockDim.x / 128u, g = threadIdx.x / 128u, t = threadIdx.x & 127u;
	const uint32_t w = t >> 5, lane = t & 31u;
	P20Group &sm = reinterpret_cast<P20Group *>(p20_smem)[g];
	uint32_t *s_runs = reinterpret_cast<uint32_t *>(
		reinterpret_cast<P20Group *>(p20_smem) + G);
	__shared__ uint32_t s_last;
	__shared__ double s_red[2];
	const uint32_t tile = blockIdx.x, c = blockIdx.y, C = prm.C, ldp = prm.ldp;
	const uint32_t p0 = tile * kP20Tile;
	double *partials = (double *)prm.partials;
	const SoftTab20 *soft = (const SoftTab20 *)prm.soft20;
	// the runs' first entries in shared memory unless they are too many
	const uint32_t *runs = prm.n_runs <= kP20RunsSmem ? s_runs : prm.runs;
	if (runs == s_runs)
		for (uint32_t k = threadIdx.x; k <= prm.n_runs; k += blockDim.x)
			s_runs[k] = prm.runs[k];
	__syncthreads();
	auto fill = [&](uint32_t e, uint32_t buf) { // tables of entry e
		if (e < prm.n) {
			const uint4 *src[2] = {(const uint4 *)(soft + (size_t)(2 * e) * C + c),
					       (const uint4 *)(soft + (size_t)(2 * e + 1) * C + c)};
			uint4 *dst = (uint4 *)&sm.tab[buf][0];
			for (uint32_t k = t; k < 2 * kTab20Chunks; k += 128)
				cp_async16(dst + k, k < kTab20Chunks ? src[0] + k
								     : src[1] + (k - kTab20Chunks));
		}
		cp_async_commit();
	};
	// this group's entry after e of run r (prm.n: none)
	auto next_of = [&](uint32_t r, uint32_t e) {
		e += G;
		while (e >= runs[r + 1]) {
			if (++r >= prm.n_runs)
				return prm.n;
			e = runs[r] + g;
		}
		return e;
	};
	const SoftNum mult = soft_split((uint32_t)__double2hiint(prm.scale_mult),
					(uint32_t)__double2loint(prm.scale_mult));
	const uint64_t thr = (uint64_t)__double_as_longlong(prm.scale_threshold);
	uint32_t buf = 0;
	{
		uint32_t r = 0, e = g;
		while (e >= runs[r + 1]) {
			if (++r >= prm.n_runs) {
				e = prm.n;
				break;
			}
			e = runs[r] + g;
		}
		fill(e, 0);
	}
	int32_t cnt[2] = {0, 0};
	for (uint32_t run = 0; run < prm.n_runs; ++run) {
		const uint32_t hi_e = runs[run + 1];
		for (uint32_t e = runs[run] + g; e < hi_e; e += G) {
			const NodeOp op = prm.ops[e];
			const uint32_t ids[2] = {op.left, op.right};
			cnt[0] = cnt[1] = 0;
#pragma unroll
			for (int j = 0; j < 2; ++j) {
				if (ids[j] & kTipBit) {
					if (t < kP20Tile)
						sm.code[j][t] = (uint8_t)min(
							(uint32_t)prm.tips[(size_t)(ids[j] & ~kTipBit) *
										   ldp +
									   p0 + t],
							(uint32_t)kS20);
					continue;
				}
				const size_t row0 = ((size_t)ids[j] * C + c) * ldp + p0;
				const double2 *src = (const double2 *)(partials + row0 * kS20);
				double2 v[5];
#pragma unroll
				for (int q = 0; q < 5; ++q)
					v[q] = src[t + 128 * q];
				cnt[0] += prm.scales[row0 + lane];
				cnt[1] += prm.scales[row0 + lane + 32];
#pragma unroll
				for (int q = 0; q < 5; ++q) {
					const uint32_t at = 2 * (t + 128 * q);
					const uint32_t p = at / kS20, k = at - p * kS20;
					const double d[2] = {v[q].x, v[q].y};
#pragma unroll
					for (int u = 0; u < 2; ++u) {
						const uint32_t dh = (uint32_t)__double2hiint(d[u]);
						const SoftNum n =
							soft_split(dh, (uint32_t)__double2loint(d[u]));
						sm.x[j][k + u][p] = make_uint2(n.hi, n.lo);
						sm.xe[j][k + u][p] =
							soft_normal(dh) ? n.e * 0x10001u : 0x8000u;
					}
				}
			}
			cp_async_wait<0>(); // this entry's tables
			bar_group(g);
			fill(next_of(run, e), buf ^ 1u);
			const SoftTab20 &tl = sm.tab[buf][0], &tr = sm.tab[buf][1];
			buf ^= 1u;
			P20Vec a, b;
			uint32_t special = (tl.rec[0][0][3] | tr.rec[0][0][3]) ? 3u : 0u;
			if (op.left & kTipBit)
				soft_tip20(tl, sm.code[0], w, lane, a);
			else
				special |= soft_dot20(tl, sm.x[0], sm.xe[0], w, lane, a);
			if (op.right & kTipBit)
				soft_tip20(tr, sm.code[1], w, lane, b);
			else
				special |= soft_dot20(tr, sm.x[1], sm.xe[1], w, lane, b);
			// tip-tip nodes are never rescaled (cpu4.rs:288-318)
			const bool cherry = ((op.left & op.right) & kTipBit) != 0;
			uint64_t bits[2][5];
#pragma unroll
			for (int cc = 0; cc < 2; ++cc) {
				bool ok = ((special >> cc) & 1u) == 0u, below = true;
#pragma unroll
				for (int i = 0; i < 5; ++i) {
					bool in;
					bits[cc][i] = soft_mul_round(a.m[cc][i], a.e[cc][i],
								     b.m[cc][i], b.e[cc][i], in);
					ok = ok && in;
					below = below && bits[cc][i] < thr;
				}
				if (!ok) {
					special |= 1u << cc;
					below = true;
					for (int i = 0; i < 5; ++i) {
						const double v = p20_plain(prm, op.left, op.right, e, c,
									   p0 + lane + 32 * cc,
									   5 * w + i);
						bits[cc][i] = (uint64_t)__double_as_longlong(v);
						below = below && v < prm.scale_threshold;
					}
				}
				sm.below[w][lane + 32 * cc] = below && !cherry;
			}
			bar_group(g); // votes in, significands read
			double *sy = reinterpret_cast<double *>(&sm.x[0][0][0]);
#pragma unroll
			for (int cc = 0; cc < 2; ++cc) {
				const uint32_t p = lane + 32 * cc;
				if (sm.below[0][p] & sm.below[1][p] & sm.below[2][p] &
				    sm.below[3][p]) {
					++cnt[cc];
#pragma unroll
					for (int i = 0; i < 5; ++i)
						bits[cc][i] =
							((special >> cc) & 1u)
								? (uint64_t)__double_as_longlong(
									  __longlong_as_double(
										  (long long)bits[cc][i]) *
									  prm.scale_mult)
								: soft_scale(bits[cc][i], mult);
				}
#pragma unroll
				for (int i = 0; i < 5; ++i)
					sy[p * kYStride + 5 * w + i] =
						__longlong_as_double((long long)bits[cc][i]);
			}
			bar_group(g); // rows staged
			const size_t orow = ((size_t)op.out * C + c) * ldp + p0;
			double2 *dst = (double2 *)(partials + orow * kS20);
#pragma unroll
			for (int q = 0; q < 5; ++q) {
				const uint32_t at = 2 * (t + 128 * q);
				const uint32_t p = at / kS20, k = at - p * kS20;
				dst[t + 128 * q] =
					*reinterpret_cast<const double2 *>(sy + p * kYStride + k);
			}
			if (w == 0) {
				prm.scales[orow + lane] = cnt[0];
				prm.scales[orow + lane + 32] = cnt[1];
			}
			if (e + 1 == prm.n && t < kP20Tile) {
				double dot = 0.0;
				for (int i = 0; i < kS20; ++i)
					dot = fma(prm.pi[i], sy[t * kYStride + i], dot);
				sm.dot[t] = dot;
			}
			bar_group(g); // rows copied out, before the next split
		}
		__syncthreads(); // the run's outputs are visible to every group
	}
	// the group that walked the last entry, the root (group 0 unless the list
	// is not one tree and unrelated entries share the root's run)
	if (g == (prm.n - 1 - runs[prm.n_runs - 1]) % G && t < kP20Tile) {
		// w is 0 or 1 here: patterns t = lane + 32 w
		const int32_t n = w ? cnt[1] : cnt[0];
		const double dot = sm.dot[t];
		prm.root_val[(size_t)c * ldp + p0 + t] = dot;
		prm.root_exp[(size_t)c * ldp + p0 + t] = n;
		if (prm.cat_lnl) // cpu4.rs:277-284, unsigned product as there
			prm.cat_lnl[(size_t)c * ldp + p0 + t] =
				log(dot) - (double)((uint32_t)n * prm.scale_ln);
		__threadfence();
	}
	__syncthreads();
	if (threadIdx.x == 0) {
		const unsigned tk = atomicAdd(prm.ticket + tile, 1u);
		s_last = tk == C - 1u;
		if (s_last)
			prm.ticket[tile] = 0u;
	}
	__syncthreads();
	if (!s_last)
		return;
	__threadfence();
	double contrib = 0.0;
	if (threadIdx.x < kP20Tile) {
		const uint32_t p = p0 + threadIdx.x;
		const RootColumns root(prm, p, (double *)p20_smem + threadIdx.x, kP20Tile);
		double site = mix_categories_f64(
			C, [&](uint32_t k) { return root.val(k); },
			[&](uint32_t k) { return root.exp(k); }, prm.scale_ln, prm.log_inv_c,
			prm.scale_pow);
		prm.site_lnl[p] = site;
		const uint32_t wgt = prm.weights[p];
		contrib = wgt ? site * (double)wgt : 0.0;
		for (int off = 16; off > 0; off >>= 1)
			contrib += __shfl_down_sync(0xffffffffu, contrib, off);
		if ((threadIdx.x & 31u) == 0)
			s_red[threadIdx.x >> 5] = contrib;
	}
	__syncthreads();
	if (threadIdx.x == 0)
		prm.sums_host[tile] = s_red[0] + s_red[1];
}
