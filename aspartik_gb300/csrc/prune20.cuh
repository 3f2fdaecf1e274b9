// prune20.cuh -- 20-state (protein) pruning: the transition tables of both
// forms and the FP32 form's walk on the CUDA cores.  Included by kernels4.cu
// inside its anonymous namespace (uses finish_root and the launch plumbing
// there).
//
// The arithmetic generalises the reference's CPU pruner (crates/b3/src/
// calculator/cpu4.rs:170-433) from 4 to S = 20 states: a tip child
// contributes the column P[.][code] (all ones for an unknown code), an
// internal child the matrix-vector product P x, and the node is the
// element-wise product of its two children.  Tables are the transposed
// P(t) = V diag(exp(lambda t)) V^-1 of every (entry, side, category) with a
// 21st row of ones, so both child kinds read whole 20-element rows.
//
// Layouts (S = 20, R = float or double):
//   partials  R  [2I][C][ldp][20]  80 B (FP32), 160 B (FP64)
//   scales    i32 [2I][C][ldp]
//   ptab      R  [n][2][C][21][20]

constexpr int kS20 = 20;
constexpr uint32_t kP20Rows = kS20 + 1;
// Integer form of an FP64 table (prune20f64.cuh): row k (state or unknown) of
// the transposed table, states 5 w .. 5 w + 4 together:
// [w] {e0|e1<<16, e2|e3<<16, e4, plain, hi[5], lo[5], -, -}
struct __align__(16) SoftTab20 {
	uint32_t rec[kP20Rows][4][16];
};

// Entry P[i][k] = v of the integer form (its `plain` word is the caller's).
__device__ __forceinline__ void soft20_store(SoftTab20 *dst, uint32_t k, uint32_t i, double v)
{
	const uint32_t dh = (uint32_t)__double2hiint(v), dl = (uint32_t)__double2loint(v);
	const uint32_t w = i / 5, q = i - 5 * w;
	uint32_t *r = dst->rec[k][w];
	reinterpret_cast<uint16_t *>(r)[q] = (uint16_t)(dh >> 20);
	r[4 + q] = (((dh & 0xFFFFFu) | 0x100000u) << 7) | (dl >> 25);
	r[9 + q] = dl << 7;
}


// Element (i, j) = (t / 20, t % 20) of the P(t) of table `id` = (entry * 2 +
// side) * C + category, by thread t < 400 of a block of at least 400 (every
// thread calls: the block synchronises).  V diag(e) is formed once per table
// in shared memory, so an element costs 20 FP64 multiply-adds instead of 20
// products more (the FP64 pipe, 64 cycles an instruction and scheduler
// partition, bounds this kernel).
struct Ptab20Smem {
	double e[kS20];
	double Ve[kS20 * kS20];
};
__device__ __forceinline__ double ptab20_element(const PtabParams &prm, uint32_t id, uint32_t t,
						 Ptab20Smem &sm)
{
	constexpr uint32_t S = kS20;
	const uint32_t c = id % prm.C, es = id / prm.C;
	const ModelDev *m = prm.model;
	const uint32_t i = t / S, j = t - i * S;
	if (prm.matrices)
		return t < S * S ? prm.matrices[(size_t)id * S * S + t] : 0.0;
	const double d = prm.lengths[es] * (prm.clock_rate * m->cat_rates[c]);
	if (m->shortcuts && d > 20.0) // transition_freqs (substitution.rs:245-252)
		return t < S * S ? m->pi[j] : 0.0;
	if (m->shortcuts && d < 1e-10) // transition_q (substitution.rs:258-268)
		return t >= S * S ? 0.0 : i == j ? 1.0 : m->Q[i * S + j] * d;
	if (t < S)
		sm.e[t] = exp(m->lambda[t] * d);
	__syncthreads();
	if (t < S * S)
		sm.Ve[t] = m->V[t] * sm.e[j];
	__syncthreads();
	if (t >= S * S)
		return 0.0;
	double s = 0.0;
#pragma unroll
	for (uint32_t k = 0; k < S; k++)
		s = fma(sm.Ve[i * S + k], m->Vinv[k * S + j], s);
	return s;
}

// One block per table, one thread per element, computed in FP64 (the same
// for both forms: the FP32 form only stores it in single precision) and
// written transposed with a 21st row of ones; the FP64 form's integer table
// beside it.
template <typename R>
__global__ void __launch_bounds__(kS20 *kS20) ptab20_kernel(PtabParams prm)
{
	constexpr uint32_t S = kS20;
	__shared__ Ptab20Smem sm;
	const uint32_t id = blockIdx.x, t = threadIdx.x, i = t / S, j = t - i * S;
	const double P = ptab20_element(prm, id, t, sm);
	R *out = (R *)prm.ptab + (size_t)id * (S + 1) * S;
	out[j * S + i] = (R)P;
	if (t < S)
		out[S * S + t] = (R)1.0;
	if constexpr (sizeof(R) == 8) {
		SoftTab20 *st = (SoftTab20 *)prm.soft20 + id;
		soft20_store(st, j, i, P);
		if (t < S)
			soft20_store(st, S, t, 1.0);
		const int plain = __syncthreads_or(
			!soft_normal((uint32_t)__double2hiint(P)));
		if (t == 0)
			st->rec[0][0][3] = plain ? 1u : 0u;
	}
}

// 20 consecutive elements (16-byte aligned) into registers.  kRO: data
// that no thread writes during the launch (tables, tips) may take the
// read-only path; partials written earlier in the walk may not.
template <bool kRO>
__device__ __forceinline__ void load20(const float *src, float v[20])
{
	const float4 *s4 = reinterpret_cast<const float4 *>(src);
#pragma unroll
	for (int q = 0; q < 5; q++) {
		const float4 a = kRO ? __ldg(s4 + q) : s4[q];
		v[4 * q] = a.x;
		v[4 * q + 1] = a.y;
		v[4 * q + 2] = a.z;
		v[4 * q + 3] = a.w;
	}
}
__device__ __forceinline__ void store20(float *dst, const float v[20])
{
	float4 *d4 = reinterpret_cast<float4 *>(dst);
#pragma unroll
	for (int q = 0; q < 5; q++)
		d4[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
}
// One child: tip row lookup or table-times-partial (k-outer, so every
// table row is one contiguous read shared by the warp's columns).
template <typename Idx>
__device__ __forceinline__ void child20(const PruneParams &prm, uint32_t id,
					const float *__restrict__ tab, Idx stride,
					Idx col, uint32_t p, float out[20],
					int32_t &sc)
{
	constexpr int S = kS20;
	if (id & kTipBit) {
		const uint8_t code = prm.tips[(size_t)(id & ~kTipBit) * prm.ldp + p];
		load20<true>(tab + (size_t)code * S, out);
		sc = 0;
		return;
	}
	const Idx ix = (Idx)id * stride + col;
	float x[S];
	load20<false>((const float *)prm.partials + (size_t)ix * S, x);
	sc = prm.scales[ix];
	float row[S];
	load20<true>(tab, row);
#pragma unroll
	for (int i = 0; i < S; i++)
		out[i] = x[0] * row[i];
#pragma unroll
	for (int k = 1; k < S; k++) {
		load20<true>(tab + k * S, row);
#pragma unroll
		for (int i = 0; i < S; i++)
			out[i] = fma(x[k], row[i], out[i]);
	}
}

// FP32 form: exact power-of-two normalisation of the largest entry into
// [1, 2); returns the exponent (see rescale_pow2).
__device__ __forceinline__ int32_t rescale_pow2_20(float y[20])
{
	float m = y[0];
#pragma unroll
	for (int i = 1; i < 20; i++)
		m = fmaxf(m, y[i]);
	if (!(m > 0.0f))
		return 0; // all zero: the pattern is impossible
	int32_t shift = 0;
	uint32_t ex = (__float_as_uint(m) >> 23) & 0xffu;
	if (ex == 0u) { // subnormal maximum: lift by 2^64 first (exact)
		const float lift = 18446744073709551616.0f;
#pragma unroll
		for (int i = 0; i < 20; i++)
			y[i] *= lift;
		shift = -64;
		m *= lift;
		ex = (__float_as_uint(m) >> 23) & 0xffu;
	}
	const int32_t e = (int32_t)ex - 127;
	const float f = __uint_as_float((uint32_t)(127 - e) << 23); // 2^-e
#pragma unroll
	for (int i = 0; i < 20; i++)
		y[i] *= f;
	return e + shift;
}

// One thread per (pattern, category) column walks the whole children-first
// list.  Block (32, C): 32 patterns of every category, so the root's
// category mixing stays in the block (finish_root).
template <typename Idx>
__global__ void __launch_bounds__(256) prune20_kernel(PruneParams prm)
{
	constexpr int S = kS20;
	const uint32_t tp = blockDim.x, c = threadIdx.y;
	const uint32_t p = blockIdx.x * tp + threadIdx.x;
	extern __shared__ double smem[];
	const Idx stride = (Idx)prm.C * prm.ldp;
	const Idx col = (Idx)c * prm.ldp + p;
	const size_t tab_stride = (size_t)(S + 1) * S;
	float y[S];
#pragma unroll
	for (int i = 0; i < S; i++)
		y[i] = 0.0f;
	int32_t cnt = 0;
	for (uint32_t e = 0; e < prm.n; ++e) {
		const NodeOp op = prm.ops[e];
		const float *tl = (const float *)prm.ptab + ((size_t)(2 * e) * prm.C + c) * tab_stride;
		const float *tr = tl + (size_t)prm.C * tab_stride;
		float a[S], b[S];
		int32_t sa, sb;
		child20<Idx>(prm, op.left, tl, stride, col, p, a, sa);
		child20<Idx>(prm, op.right, tr, stride, col, p, b, sb);
#pragma unroll
		for (int i = 0; i < S; i++)
			y[i] = a[i] * b[i];
		const int32_t own = rescale_pow2_20(y);
		cnt = sa + sb + own;
		const Idx ox = (Idx)op.out * stride + col;
		store20((float *)prm.partials + (size_t)ox * S, y);
		prm.scales[ox] = cnt;
	}
	double root_dot = 0.0;
#pragma unroll
	for (int i = 0; i < S; i++)
		root_dot = fma(prm.pi[i], (double)y[i], root_dot);
	finish_root<true>(prm, smem, tp, threadIdx.x, blockIdx.x * tp, c, true, root_dot,
			   cnt);
}
