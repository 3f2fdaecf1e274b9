// prune4f64.cuh -- walk of the plain FP64 form with its products on the
// integer pipes (soft64.cuh).  Included by kernels4.cu inside its anonymous
// namespace (uses v4_apply, v4_mul, rescale_threshold, finish_root).
//
// One thread owns one (pattern, category) column and walks the whole
// children-first list, as the plain walk does; a warp's columns share one
// category, so its transition tables are the same for every lane.
//   - Tables: each warp keeps a ring of kF64Ring entries (schedule word and
//     the two soft tables of its category, 432 bytes) in shared memory,
//     filled by one 16-byte cp.async a lane and entry, so no table load
//     waits on global memory and no block barrier exists in the walk.
//   - Children: the partials of entry i + 1 are loaded before entry i is
//     computed; a child that is entry i's output is taken from registers (no
//     other output can be missing: this thread stored it earlier).
//   - Arithmetic: soft_dot4 and soft_mul_round.  A lane whose inputs or
//     result are not positive normal numbers, and a warp whose table is
//     not, take the FP64 instructions of the plain walk for that entry.

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

// A child's contribution: four significands, their exponents and whether
// the soft arithmetic holds for it.
struct SoftVec {
	uint64_t m[4];
	int32_t e[4]; // value = m 2^e
};

__device__ __forceinline__ void soft_tip(const SoftTab4 &t, uint32_t code, SoftVec &v)
{
	const uint4 hi = *reinterpret_cast<const uint4 *>(t.hi[code]);
	const uint4 lo = *reinterpret_cast<const uint4 *>(t.lo[code]);
	const uint2 e = *reinterpret_cast<const uint2 *>(t.e[code]);
	v.m[0] = ((uint64_t)hi.x << 32) | lo.x;
	v.m[1] = ((uint64_t)hi.y << 32) | lo.y;
	v.m[2] = ((uint64_t)hi.z << 32) | lo.z;
	v.m[3] = ((uint64_t)hi.w << 32) | lo.w;
	v.e[0] = (int32_t)(e.x & 0xFFFFu) - kSoftBias;
	v.e[1] = (int32_t)(e.x >> 16) - kSoftBias;
	v.e[2] = (int32_t)(e.y & 0xFFFFu) - kSoftBias;
	v.e[3] = (int32_t)(e.y >> 16) - kSoftBias;
}

// Sums sum_k P[i][k] x[k], i = 0..3; false: some x[k] is not a positive
// normal number (the sums are then meaningless).
__device__ __forceinline__ bool soft_dot4(const SoftTab4 &t, const double4_32a &x, SoftVec &v)
{
	const double xs[4] = {x.x, x.y, x.z, x.w};
	SoftNum n[4];
	bool ok = true;
	uint32_t s01[4], s23[4];
#pragma unroll
	for (int k = 0; k < 4; ++k) {
		const uint32_t dh = (uint32_t)__double2hiint(xs[k]);
		ok = ok && soft_normal(dh);
		n[k] = soft_split(dh, (uint32_t)__double2loint(xs[k]));
		const uint32_t e2 = __byte_perm(n[k].e, 0, 0x1010);
		const uint2 te = *reinterpret_cast<const uint2 *>(t.e[k]);
		s01[k] = te.x + e2; // both halves stay below 4096
		s23[k] = te.y + e2;
	}
	const uint32_t m01 = soft_max2(soft_max2(s01[0], s01[1]), soft_max2(s01[2], s01[3]));
	const uint32_t m23 = soft_max2(soft_max2(s23[0], s23[1]), soft_max2(s23[2], s23[3]));
#pragma unroll
	for (int i = 0; i < 4; ++i)
		v.m[i] = 0;
#pragma unroll
	for (int k = 0; k < 4; ++k) {
		const uint4 hi = *reinterpret_cast<const uint4 *>(t.hi[k]);
		const uint4 lo = *reinterpret_cast<const uint4 *>(t.lo[k]);
		const uint32_t d01 = m01 - s01[k], d23 = m23 - s23[k]; // no borrow
		v.m[0] += soft_shr(soft_prod(n[k].hi, n[k].lo, hi.x, lo.x), d01 & 0xFFFFu);
		v.m[1] += soft_shr(soft_prod(n[k].hi, n[k].lo, hi.y, lo.y), d01 >> 16);
		v.m[2] += soft_shr(soft_prod(n[k].hi, n[k].lo, hi.z, lo.z), d23 & 0xFFFFu);
		v.m[3] += soft_shr(soft_prod(n[k].hi, n[k].lo, hi.w, lo.w), d23 >> 16);
	}
	v.e[0] = (int32_t)(m01 & 0xFFFFu) - kSoftDotBias;
	v.e[1] = (int32_t)(m01 >> 16) - kSoftDotBias;
	v.e[2] = (int32_t)(m23 & 0xFFFFu) - kSoftDotBias;
	v.e[3] = (int32_t)(m23 >> 16) - kSoftDotBias;
	return ok;
}

struct F64Child {
	double4_32a x;
	int32_t s;
	uint32_t code;
};

// The same entry in FP64 instructions (plain_batch's arithmetic), from the
// double tables in global memory.
__device__ __noinline__ double4_32a f64_plain_entry(const double4_32a *tl,
						    const double4_32a *tr, uint32_t left,
						    uint32_t right, F64Child l, F64Child r)
{
	const double4_32a a = (left & kTipBit) ? tl[l.code] : v4_apply(tl, l.x);
	const double4_32a b = (right & kTipBit) ? tr[r.code] : v4_apply(tr, r.x);
	return v4_mul(a, b);
}

// One entry for one column: its value before rescaling.
__device__ __forceinline__ double4_32a f64_entry(const F64Entry &en, const double4_32a *ptab,
						 uint32_t i, uint32_t C, uint32_t c,
						 const F64Child &l, const F64Child &r)
{
	const NodeOp op = en.op;
	SoftVec a, b;
	bool ok = (en.tab[0].plain | en.tab[1].plain) == 0u;
	if (op.left & kTipBit)
		soft_tip(en.tab[0], l.code, a);
	else
		ok = soft_dot4(en.tab[0], l.x, a) && ok;
	if (op.right & kTipBit)
		soft_tip(en.tab[1], r.code, b);
	else
		ok = soft_dot4(en.tab[1], r.x, b) && ok;
	uint64_t bits[4];
#pragma unroll
	for (int q = 0; q < 4; ++q) {
		bool in;
		bits[q] = soft_mul_round(a.m[q], a.e[q], b.m[q], b.e[q], in);
		ok = ok && in;
	}
	double4_32a y;
	y.x = __longlong_as_double((long long)bits[0]);
	y.y = __longlong_as_double((long long)bits[1]);
	y.z = __longlong_as_double((long long)bits[2]);
	y.w = __longlong_as_double((long long)bits[3]);
	if (!ok) {
		const double4_32a *tl = ptab + ((size_t)(2 * i) * C + c) * 5;
		y = f64_plain_entry(tl, tl + (size_t)C * 5, op.left, op.right, l, r);
	}
	return y;
}

// rescale_threshold with the comparisons on the bit patterns: thr > 0, so a
// double is below it exactly when its bits, as a signed integer, are (all
// negative numbers included; a NaN made here is positive and is not).
__device__ __forceinline__ int32_t f64_rescale(double4_32a &y, double thr, double mult)
{
	const long long t = __double_as_longlong(thr);
	if (__double_as_longlong(y.x) < t && __double_as_longlong(y.y) < t &&
	    __double_as_longlong(y.z) < t && __double_as_longlong(y.w) < t) {
		y.x *= mult;
		y.y *= mult;
		y.z *= mult;
		y.w *= mult;
		return 1;
	}
	return 0;
}

__device__ __forceinline__ void f64_load(const PruneParams &prm,
					 const double4_32a *__restrict__ partials, uint32_t id,
					 uint32_t forward, uint32_t p, uint32_t c, F64Child &in)
{
	if (id & kTipBit) {
		in.code = prm.tips[(size_t)(id & ~kTipBit) * prm.ldp + p];
		in.s = 0;
	} else if (id != forward) {
		const size_t ix = ((size_t)id * prm.C + c) * prm.ldp + p;
		in.x = partials[ix];
		in.s = prm.scales[ix];
	}
}

__global__ void __launch_bounds__(512) prune4_f64_kernel(PruneParams prm)
{
	const uint32_t tp = blockDim.x, c = threadIdx.y, C = prm.C;
	const uint32_t p = blockIdx.x * tp + threadIdx.x;
	double4_32a *partials = (double4_32a *)prm.partials;
	extern __shared__ __align__(16) double smem[];
	const uint32_t tid = threadIdx.y * tp + threadIdx.x, lane = tid & 31u;
	F64Entry *ring = reinterpret_cast<F64Entry *>(smem + 2 * tp * C + 32) +
			 (tid >> 5) * kF64Ring;
	auto fill = [&](uint32_t e) {
		if (e < prm.n && lane < 27) {
			F64Entry *dst = ring + (e & (kF64Ring - 1));
			const uint32_t side = lane < 14 ? 0u : 1u, q = lane - 1 - 13 * side;
			const void *src =
				lane == 0 ? (const void *)(prm.ops + e)
					  : (const void *)((const uint4 *)(prm.soft +
									   ((size_t)(2 * e + side) * C + c)) +
							   q);
			cp_async16((uint4 *)dst + lane, src);
		}
		cp_async_commit();
	};
#pragma unroll
	for (uint32_t e = 0; e < kF64Ring; ++e)
		fill(e);
	cp_async_wait<kF64Ring - 1>();
	__syncwarp();
	F64Child l, r;
	uint32_t prev = kTipBit; // the previous entry's output: none yet
	f64_load(prm, partials, ring[0].op.left, prev, p, c, l);
	f64_load(prm, partials, ring[0].op.right, prev, p, c, r);
	double4_32a y = v4_make<double4_32a, double>(0, 0, 0, 0);
	int32_t cnt = 0;
	for (uint32_t i = 0; i < prm.n; ++i) {
		// entries i and i + 1 have landed
		cp_async_wait<kF64Ring - 2>();
		__syncwarp();
		const F64Entry &en = ring[i & (kF64Ring - 1)];
		const uint32_t left = en.op.left, right = en.op.right, out = en.op.out;
		F64Child nl, nr;
		uint32_t next_l = kTipBit, next_r = kTipBit;
		if (i + 1 < prm.n) {
			const F64Entry &nx = ring[(i + 1) & (kF64Ring - 1)];
			next_l = nx.op.left;
			next_r = nx.op.right;
			f64_load(prm, partials, next_l, out, p, c, nl);
			f64_load(prm, partials, next_r, out, p, c, nr);
		}
		y = f64_entry(en, (const double4_32a *)prm.ptab, i, C, c, l, r);
		// tip-tip nodes are never rescaled (cpu4.rs:288-318)
		const int32_t own =
			((left & right) & kTipBit)
				? 0
				: f64_rescale(y, prm.scale_threshold, prm.scale_mult);
		cnt = l.s + r.s + own;
		const size_t ox = ((size_t)out * C + c) * prm.ldp + p;
		partials[ox] = y;
		prm.scales[ox] = cnt;
		__syncwarp(); // every lane has read the slot that is filled next
		fill(i + kF64Ring);
		l = nl;
		r = nr;
		if (next_l == out) {
			l.x = y;
			l.s = cnt;
		}
		if (next_r == out) {
			r.x = y;
			r.s = cnt;
		}
	}
	const double root_dot = prm.pi[0] * y.x + prm.pi[1] * y.y + prm.pi[2] * y.z +
				prm.pi[3] * y.w;
	finish_root<false>(prm, smem, tp, threadIdx.x, p, c, true, root_dot, cnt);
}
