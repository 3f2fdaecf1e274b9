// prune4f64.cuh -- walk of the plain FP64 form with its products on the
// integer pipes (soft64.cuh).  Included by kernels4.cu inside its anonymous
// namespace (uses v4_apply, v4_mul, rescale_threshold, finish_root).
//
// One thread owns one (pattern, category) column and walks the list depth
// first; a warp's columns share one category, so its transition tables are
// the same for every lane.  Where the columns leave the schedulers short of
// warps, several groups of a block walk disjoint subtrees first.
//   - Tables: each warp keeps a ring of kF64Ring entries (schedule word and
//     the two soft tables of its category, 432 bytes) in shared memory,
//     filled by one 16-byte cp.async a lane and entry, so no table load
//     waits on global memory and no block barrier exists in the walk.
//   - Children: the partials of entry i + 1 are loaded before entry i is
//     computed; a child that is entry i's output is taken from registers (no
//     other output can be missing: this thread stored it earlier).
//   - Arithmetic: soft_dot4, soft_mul_round and soft_scale.  A lane whose inputs or
//     result are not positive normal numbers, and a warp whose table is
//     not, take the FP64 instructions of the plain walk for that entry.
//
// Whole tree, 256 taxa x 17,764 patterns, four categories: 1,290 us as the
// plain walk (bound by the FP64 pipe), 400 us here (about 430 instructions a
// column and entry at 3.65 warps a scheduler: issue and dependent latency).
// Tried and slower: four lanes a column, one state each (1,027 against 480
// us, and 50 against 34 us on a 64-taxon path: the inputs are split and the
// table words read four times over).

constexpr uint32_t kF64Ring = 4;
struct __align__(16) F64Entry {
	NodeOp op;
	SoftTab4 tab[2];
};
static_assert(sizeof(F64Entry) == 27 * 16, "27 copies of 16 bytes");

__device__ __forceinline__ void cp_async16(void *dst, const void *src)
{
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
			     (uint32_t)__cvta_generic_to_shared(dst)),
		     "l"(src)
		     : "memory");
}
__device__ __forceinline__ void cp_async_commit()
{
	asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int kPending> __device__ __forceinline__ void cp_async_wait()
{
	asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory");
}

// A child's contribution: state 0 as a double, states 1..3 as significands
// with their exponents (value = m 2^e).
struct SoftVec {
	double d0;
	uint64_t m[3];
	int32_t e[3];
};

__device__ __forceinline__ uint64_t soft_pair(uint32_t hi, uint32_t lo)
{
	return ((uint64_t)hi << 32) | lo;
}

__device__ __forceinline__ SoftRow4 soft_row(const SoftRow4 &r)
{
	const uint4 a = *reinterpret_cast<const uint4 *>(&r);
	const uint4 b = *(reinterpret_cast<const uint4 *>(&r) + 1);
	SoftRow4 v;
	v.hi[0] = a.x;
	v.hi[1] = a.y;
	v.hi[2] = a.z;
	v.lo1 = a.w;
	v.lo2 = b.x;
	v.lo3 = b.y;
	v.d0 = __hiloint2double((int)b.w, (int)b.z);
	return v;
}

__device__ __forceinline__ void soft_tip(const SoftTab4 &t, uint32_t code, SoftVec &v)
{
	const SoftRow4 r = soft_row(t.row[code]);
	const uint2 e = *reinterpret_cast<const uint2 *>(t.e[code]);
	v.d0 = r.d0;
	v.m[0] = soft_pair(r.hi[0], r.lo1);
	v.m[1] = soft_pair(r.hi[1], r.lo2);
	v.m[2] = soft_pair(r.hi[2], r.lo3);
	v.e[0] = (int32_t)(e.x & 0xFFFFu) - kSoftBias;
	v.e[1] = (int32_t)(e.x >> 16) - kSoftBias;
	v.e[2] = (int32_t)e.y - kSoftBias;
}

// Sums sum_k P[i][k] x[k]; false: some x[k] is not a positive normal number
// (the integer sums are then meaningless).
__device__ __forceinline__ bool soft_dot4(const SoftTab4 &t, const double4_32a &x, SoftVec &v)
{
	const double xs[4] = {x.x, x.y, x.z, x.w};
	SoftNum n[4];
	bool ok = true;
	uint32_t s12[4], s3[4];
#pragma unroll
	for (int k = 0; k < 4; ++k) {
		const uint32_t dh = (uint32_t)__double2hiint(xs[k]);
		ok = ok && soft_normal(dh);
		n[k] = soft_split(dh, (uint32_t)__double2loint(xs[k]));
		const uint2 te = *reinterpret_cast<const uint2 *>(t.e[k]);
		s12[k] = te.x + __byte_perm(n[k].e, 0, 0x1010); // halves below 4096
		s3[k] = te.y + n[k].e;
	}
	const uint32_t m12 =
		soft_max2(soft_max2(s12[0], s12[1]), soft_max2(s12[2], s12[3]));
	const uint32_t m3 = max(max(s3[0], s3[1]), max(s3[2], s3[3]));
	v.m[0] = v.m[1] = v.m[2] = 0;
#pragma unroll
	for (int k = 0; k < 4; ++k) {
		const SoftRow4 r = soft_row(t.row[k]);
		v.d0 = k == 0 ? r.d0 * xs[0] : fma(r.d0, xs[k], v.d0);
		const uint32_t d12 = m12 - s12[k], d3 = m3 - s3[k]; // no borrow
		v.m[0] += soft_shr(soft_prod(n[k].hi, n[k].lo, r.hi[0], r.lo1), d12 & 0xFFFFu);
		v.m[1] += soft_shr(soft_prod(n[k].hi, n[k].lo, r.hi[1], r.lo2), d12 >> 16);
		v.m[2] += soft_shr(soft_prod(n[k].hi, n[k].lo, r.hi[2], r.lo3), d3);
	}
	v.e[0] = (int32_t)(m12 & 0xFFFFu) - kSoftDotBias;
	v.e[1] = (int32_t)(m12 >> 16) - kSoftDotBias;
	v.e[2] = (int32_t)m3 - kSoftDotBias;
	return ok;
}

struct F64Child {
	double4_32a x;
	int32_t s;
	uint32_t code;
};

// Four doubles of a partial, 32-byte aligned.  Volatile, so that the load
// stays where it is written, ahead of the previous entry's arithmetic (left
// to the compiler it sinks below it, and every entry then waits a memory
// round trip: 400 of 3,080 cycles an entry).
__device__ __forceinline__ double4_32a ld_partial(const double4_32a *p)
{
	double4_32a v;
	asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
		     : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w)
		     : "l"(p)
		     : "memory");
	return v;
}

template <typename Idx>
__device__ __forceinline__ void f64_load(const PruneParams &prm, uint32_t id,
					 uint32_t forward, uint32_t p, Idx stride, Idx col,
					 F64Child &in)
{
	if (id & kTipBit) {
		in.code = prm.tips[(size_t)(id & ~kTipBit) * prm.ldp + p];
		in.s = 0;
	} else if (id != forward) {
		const Idx ix = (Idx)id * stride + col;
		in.x = ld_partial((const double4_32a *)prm.partials + ix);
		in.s = prm.scales[ix];
	}
}

// Entry i in FP64 instructions (plain_batch's arithmetic), from the double
// tables and the inputs in global memory (a forwarded one was stored by
// this thread), so that nothing of it stays in registers while the integer
// form runs.
__device__ __forceinline__ double4_32a f64_apply_plain(const PruneParams &prm,
							const double4_32a *tab, uint32_t id,
							uint32_t p, uint32_t c)
{
	if (id & kTipBit)
		return tab[prm.tips[(size_t)(id & ~kTipBit) * prm.ldp + p]];
	const double4_32a *partials = (const double4_32a *)prm.partials;
	return v4_apply(tab, partials[((size_t)id * prm.C + c) * prm.ldp + p]);
}
__device__ __noinline__ double4_32a f64_plain_entry(const PruneParams &prm, uint32_t left,
						    uint32_t right, uint32_t i, uint32_t p,
						    uint32_t c)
{
	const double4_32a *tl =
		(const double4_32a *)prm.ptab + ((size_t)(2 * i) * prm.C + c) * 5;
	return v4_mul(f64_apply_plain(prm, tl, left, p, c),
		      f64_apply_plain(prm, tl + (size_t)prm.C * 5, right, p, c));
}

// One entry for one column.  Returns the number of rescalings (0 or 1) by
// cpu4.rs:403-433's rule: all four entries below the threshold, and none at
// tip-tip nodes (cpu4.rs:288-318).  The threshold is positive, so comparing
// the bits of non-negative numbers as integers decides as comparing the
// doubles does.
__device__ __forceinline__ int32_t f64_entry(const PruneParams &prm, const F64Entry &en,
					     const NodeOp &op, uint32_t i, uint32_t p,
					     uint32_t c, const F64Child &l, const F64Child &r,
					     const SoftNum &mult, double4_32a &y)
{
	const bool cherry = ((op.left & op.right) & kTipBit) != 0;
	const uint64_t thr = (uint64_t)__double_as_longlong(prm.scale_threshold);
	bool ok = (en.tab[0].plain | en.tab[1].plain) == 0u;
	SoftVec a, b;
	if (op.left & kTipBit)
		soft_tip(en.tab[0], l.code, a);
	else
		ok = soft_dot4(en.tab[0], l.x, a) && ok;
	if (op.right & kTipBit)
		soft_tip(en.tab[1], r.code, b);
	else
		ok = soft_dot4(en.tab[1], r.x, b) && ok;
	y.x = a.d0 * b.d0;
	uint64_t bits[3];
#pragma unroll
	for (int k = 0; k < 3; ++k) {
		bool in;
		bits[k] = soft_mul_round(a.m[k], a.e[k], b.m[k], b.e[k], in);
		ok = ok && in;
	}
	if (!ok) {
		y = f64_plain_entry(prm, op.left, op.right, i, p, c);
		return cherry ? 0
			      : rescale_threshold(y, prm.scale_threshold, prm.scale_mult);
	}
	int32_t own = 0;
	if (!cherry && bits[0] < thr && bits[1] < thr && bits[2] < thr &&
	    (uint64_t)__double_as_longlong(y.x) < thr) {
		own = 1;
		y.x *= prm.scale_mult;
#pragma unroll
		for (int k = 0; k < 3; ++k)
			bits[k] = soft_scale(bits[k], mult);
	}
	y.y = __longlong_as_double((long long)bits[0]);
	y.z = __longlong_as_double((long long)bits[1]);
	y.w = __longlong_as_double((long long)bits[2]);
	return own;
}

// The warp's copy of entry e (schedule word and the two tables of category
// c) into `dst`, a 16-byte piece a lane; commits a group in any case.
__device__ __forceinline__ void f64_fill(const PruneParams &prm, F64Entry *dst, uint32_t e,
					 uint32_t c, uint32_t lane)
{
	if (e < prm.n && lane < 27) {
		const uint32_t side = lane < 14 ? 0u : 1u, k = lane - 1 - 13 * side;
		const void *src =
			lane == 0 ? (const void *)(prm.ops + e)
				  : (const void *)((const uint4 *)(prm.soft +
								   ((size_t)(2 * e + side) * prm.C + c)) +
						   k);
		cp_async16((uint4 *)dst + lane, src);
	}
	cp_async_commit();
}

__device__ __forceinline__ double f64_root_dot(const PruneParams &prm, const double4_32a &y)
{
	return prm.pi[0] * y.x + prm.pi[1] * y.y + prm.pi[2] * y.z + prm.pi[3] * y.w;
}

// A block of (tp patterns, C categories, G groups).  Several groups share the
// list in phases (prm.segs, the host's depth-first order): in phase ph group
// g walks entries [segs[ph G + g], segs[ph G + g + 1]) of its columns, whole
// subtrees first, then the entries above them run by run; a barrier ends a
// phase.  Group 0 walks the last entry, the root.
template <typename Idx, bool kGroups>
__global__ void __launch_bounds__(512) prune4_f64_kernel(PruneParams prm)
{
	const uint32_t tp = blockDim.x, c = threadIdx.y, C = prm.C;
	const uint32_t g = kGroups ? threadIdx.z : 0u, G = kGroups ? blockDim.z : 1u;
	const uint32_t p = blockIdx.x * tp + threadIdx.x;
	const Idx stride = (Idx)C * prm.ldp, col = (Idx)c * prm.ldp + p;
	extern __shared__ __align__(16) double smem[];
	const uint32_t tid = (g * C + c) * tp + threadIdx.x, lane = tid & 31u;
	F64Entry *rings = reinterpret_cast<F64Entry *>(smem + 2 * tp * C * G + 32);
	F64Entry *ring = rings + (tid >> 5) * kF64Ring;
	uint32_t *s_segs = reinterpret_cast<uint32_t *>(rings + tp / 32u * C * G * kF64Ring);
	if constexpr (kGroups) {
		for (uint32_t k = tid; k <= prm.phases * G; k += tp * C * G)
			s_segs[k] = prm.segs[k];
		__syncthreads();
	}
	// this group's next entry to copy: fe of phase fp, until fend
	uint32_t fp = 0, fe = kGroups ? s_segs[g] : 0, fend = kGroups ? s_segs[g + 1] : prm.n;
	uint32_t slot = 0;
	auto fill = [&] {
		while (kGroups && fe >= fend && fp + 1 < prm.phases) {
			++fp;
			fe = s_segs[fp * G + g];
			fend = s_segs[fp * G + g + 1];
		}
		f64_fill(prm, ring + slot, fe < fend ? fe : prm.n, c, lane);
		++fe;
		slot = (slot + 1) & (kF64Ring - 1);
	};
	wait_for_tables();
#pragma unroll
	for (uint32_t e = 0; e < kF64Ring; ++e)
		fill();
	const NodeOp none{kTipBit, kTipBit, kTipBit, 0};
	const SoftNum mult = soft_split((uint32_t)__double2hiint(prm.scale_mult),
					(uint32_t)__double2loint(prm.scale_mult));
	double4_32a y = v4_make<double4_32a, double>(0, 0, 0, 0);
	int32_t cnt = 0;
	uint32_t cur = 0; // ring slot of the current entry
	auto walk = [&](uint32_t lo, uint32_t hi) {
		if (lo >= hi)
			return;
		cp_async_wait<kF64Ring - 2>(); // the first two entries have landed
		__syncwarp();
		NodeOp op = ring[cur].op;
		NodeOp nop = lo + 1 < hi ? ring[(cur + 1) & (kF64Ring - 1)].op : none;
		F64Child l, r;
		f64_load<Idx>(prm, op.left, kTipBit, p, stride, col, l);
		f64_load<Idx>(prm, op.right, kTipBit, p, stride, col, r);
		for (uint32_t i = lo; i < hi; ++i) {
			F64Child nl, nr;
			if (i + 1 < hi) {
				f64_load<Idx>(prm, nop.left, op.out, p, stride, col, nl);
				f64_load<Idx>(prm, nop.right, op.out, p, stride, col, nr);
			}
			cp_async_wait<kF64Ring - 3>(); // entry i + 2 has landed
			__syncwarp();
			const NodeOp nnop =
				i + 2 < hi ? ring[(cur + 2) & (kF64Ring - 1)].op : none;
			const int32_t own =
				f64_entry(prm, ring[cur], op, i, p, c, l, r, mult, y);
			cnt = l.s + r.s + own;
			const Idx ox = (Idx)op.out * stride + col;
			((double4_32a *)prm.partials)[ox] = y;
			prm.scales[ox] = cnt;
			__syncwarp(); // every lane has read the slot that is filled next
			fill();
			cur = (cur + 1) & (kF64Ring - 1);
			l = nl;
			r = nr;
			if (nop.left == op.out) {
				l.x = y;
				l.s = cnt;
			}
			if (nop.right == op.out) {
				r.x = y;
				r.s = cnt;
			}
			op = nop;
			nop = nnop;
		}
	};
	if constexpr (kGroups) {
		for (uint32_t ph = 0; ph < prm.phases; ++ph) {
			walk(s_segs[ph * G + g], s_segs[ph * G + g + 1]);
			__syncthreads(); // the phase's outputs are visible to every group
		}
	} else {
		walk(0, prm.n);
	}
	finish_root<false>(prm, smem, tp, threadIdx.x, blockIdx.x * tp, c, g == 0,
			   f64_root_dot(prm, y), cnt);
}
