// prune20.cuh -- 20-state (protein) pruning: the transition tables of both
// forms and the FP32 form's walk with register matrix instructions.  Included by kernels4.cu
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
//   partials  FP64 [2I][C][ldp][20]; FP32 [2I][C][ldp/128][10][128][2]
//             (state pairs inside 128-pattern tiles, both FP32 engines)
//   scales    i32 [2I][C][ldp]
//   ptab      R  [n][2][C][21][20]

constexpr int kS20 = 20;
constexpr uint32_t kP20RunsSmem = 2048; // runs staged in shared memory
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


// Element base + t = (i, j) of the P(t) of table `id` = (entry * 2 + side) * C
// + category, row by row, by thread t < count (whole rows) of a block of at
// least 20 threads (every thread calls: the block synchronises).  V diag(e) is
// formed once per table in shared memory, so an element costs 20 FP64
// multiply-adds instead of 20 products more (the FP64 pipe, 64 cycles an
// instruction and scheduler partition, bounds this kernel).
struct Ptab20Smem {
	double e[kS20];
	double Ve[kS20 * kS20];
};
__device__ __forceinline__ double ptab20_element(const PtabParams &prm, uint32_t id, uint32_t t,
						 Ptab20Smem &sm, uint32_t base = 0,
						 uint32_t count = kS20 * kS20)
{
	constexpr uint32_t S = kS20;
	const uint32_t c = id % prm.C, es = id / prm.C;
	const ModelDev *m = prm.model;
	const uint32_t i = (base + t) / S, j = (base + t) - i * S;
	if (prm.matrices)
		return t < count ? prm.matrices[(size_t)id * S * S + base + t] : 0.0;
	const double d = prm.lengths[es] * (prm.clock_rate * m->cat_rates[c]);
	if (m->shortcuts && d > 20.0) // transition_freqs (substitution.rs:245-252)
		return t < count ? m->pi[j] : 0.0;
	if (m->shortcuts && d < 1e-10) // transition_q (substitution.rs:258-268)
		return t >= count ? 0.0 : i == j ? 1.0 : m->Q[i * S + j] * d;
	if (t < S)
		sm.e[t] = exp(m->lambda[t] * d);
	__syncthreads();
	if (t < count)
		sm.Ve[t] = m->V[base + t] * sm.e[j];
	__syncthreads();
	if (t >= count)
		return 0.0;
	const double *Ve = sm.Ve + (t - j);
	double s = 0.0;
#pragma unroll
	for (uint32_t k = 0; k < S; k++)
		s = fma(Ve[k], m->Vinv[k * S + j], s);
	return s;
}

// NaN with a payload that split_tf32_int keeps.
__device__ __forceinline__ float quiet_nan(float x)
{
	return x != x ? __uint_as_float(0x7FC00000u) : x;
}

// One thread per element, computed in FP64 (the same for both forms: the FP32
// form only stores it in single precision) and written transposed with a 21st
// row of ones; the FP64 form's integer table beside it.  A table is one block,
// or in the FP32 form kParts blocks of 20 / kParts rows each where the list's
// tables would leave SMs idle (64 tables of a path of 8 entries: 7.5 -> 6.7 us
// beside 2.2 of an empty event pair; an evaluation 39.2 -> 37.5 us).
template <typename R, uint32_t kParts>
__global__ void __launch_bounds__(kS20 *kS20 / kParts) ptab20_kernel(PtabParams prm)
{
	constexpr uint32_t S = kS20, kCount = S * S / kParts;
	static_assert(kParts == 1 || sizeof(R) == 4, "the integer table's flag is one block's");
	__shared__ Ptab20Smem sm;
	const uint32_t id = blockIdx.x / kParts, base = (blockIdx.x % kParts) * kCount;
	const uint32_t t = threadIdx.x, i = (base + t) / S, j = (base + t) - i * S;
	const double P = ptab20_element(prm, id, t, sm, base, kCount);
	R *out = (R *)prm.ptab + (size_t)id * (S + 1) * S;
	if constexpr (sizeof(R) == 4)
		out[j * S + i] = quiet_nan((float)P);
	else
		out[j * S + i] = P;
	if (t < S && base == 0)
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

// The C <= 8 categories' root values and counts of pattern p, read together
// (they are used three times over) into this thread's shared-memory words: at
// [k * pitch] of `words`, the counts behind 8 * pitch doubles.
struct RootColumns {
	double *v;
	uint32_t pitch;
	__device__ RootColumns(const PruneParams &prm, uint32_t p, double *words, uint32_t pitch_)
	    : v(words), pitch(pitch_)
	{
#pragma unroll 4
		for (uint32_t k = 0; k < prm.C; ++k) {
			const size_t at = (size_t)k * prm.ldp + p;
			const double x = __ldcg(prm.root_val + at);
			const int32_t n = __ldcg(prm.root_exp + at);
			v[k * pitch] = x;
			((int32_t *)(v + (8 + k) * pitch))[0] = n;
		}
	}
	__device__ double val(uint32_t k) const { return v[k * pitch]; }
	__device__ int32_t exp(uint32_t k) const
	{
		return ((const int32_t *)(v + (8 + k) * pitch))[0];
	}
};

// ---------------------------------------------------------------------------
// FP32 walk with register matrix instructions.
//
// A warp owns 32 patterns of one category and computes an internal child as
// out[p][i] = sum_k x[p][k] P[i][k], two m16n8k8 row tiles by three column
// and three K tiles (20 states padded to 24), in the 3xTF32 split form (x =
// x_hi + x_lo, P = P_hi + P_lo; x_lo P_hi, x_hi P_lo and x_hi P_hi, FP32
// accumulation).  State 8 s + 2 q + j is K index 4 j + q of K tile s, so that
// a product's fragment (row lane / 4, columns 2 (lane % 4) + {0, 1}) is the
// fragment the next product reads: values never change lanes, and a chain of
// entries passes through registers.
//
// Whole tree, 128 taxa x 4,989 patterns, four categories: 124 us (about 2,100
// cycles an entry and warp alone, 2,650 with two warps a scheduler), dirty
// path of eight entries 10 us of walk; 44,000 patterns: 767 us.
// Why not the other two engines: scalar FMAs need a broadcast shared-memory
// word per multiply-add and warp (the load path 70 % busy), and on the
// fifth-generation tensor cores (prune20tc.cuh) an entry is a chain of a bulk
// copy, a split through shared memory, an MMA round trip and a tensor-memory
// read of about 5,000 cycles for at most 0.1 of them of tensor work (168 us
// with its root kernel; 853 us at 44,000 patterns).  Here an internal
// child of 32 patterns takes 54 instructions of 8 cycles each (measured) of
// its scheduler's matrix pipe and about as many issue slots beside them.
//
// Partials are stored as [10][128][2] inside 128-pattern tiles (state pairs):
// every 8-byte access of a fragment covers whole 32-byte sectors.
//   - Tables and schedule words reach each warp by cp.async into a ring of
//     its own, two entries ahead; TF32 halves are made from the FP32 table.
//   - The list comes depth first (heavier subtree first), so an entry has at
//     most one child from memory unless it has two clean ones: the other is
//     a tip or the previous entry's output, still in registers.  The host
//     marks each entry (NodeOp::pad): which side to multiply first, and each
//     side's source.  The first side is never the previous output, so its
//     rows (or codes) are loaded an entry ahead.
//   - Where the tiles leave the schedulers short of warps, G warps of a block
//     share a list in phases (prm.segs): disjoint subtrees first, then the
//     entries above them, run by run.
// A block covers one category of a tile; the last of a tile's C blocks to
// finish mixes the categories and writes the tile's weighted sum to mapped
// host memory.
constexpr uint32_t kS20Ring = 3;
struct __align__(16) S20Entry {
	NodeOp op;
	float tab[2][kP20Rows * kS20];
};
constexpr uint32_t kS20TabChunks = kP20Rows * kS20 / 4; // 105
static_assert(sizeof(S20Entry) == 16 + 2 * 16 * kS20TabChunks, "16-byte copies");

// Offset of (pattern p, state pair 0) of a 20-state FP32 partial from its
// (slot, category) block; pair k is 256 k further.
__host__ __device__ __forceinline__ uint32_t off20(uint32_t p)
{
	return (p >> 7) * (kS20 * 128u) + 2u * (p & 127u);
}

// A fragment of 32 patterns: rows 16 m + 8 h + lane / 4, state pairs 4 s +
// lane % 4 (pairs 10 and 11 do not exist: zero).
struct S20Frag {
	float2 v[2][2][3];
};

__device__ __forceinline__ float2 ld_f2(const float *p)
{
	float2 v; // volatile: stays ahead of the arithmetic it overlaps
	asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p) : "memory");
	return v;
}

__device__ __forceinline__ void mma_tf32_k8(float c[4], const uint32_t a[4], uint32_t b0,
					    uint32_t b1)
{
	asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, "
		     "{%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
		     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
		     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// TF32 head and tail of x as tc::split_tf32 makes them (round to nearest,
// halves away from zero), in integer arithmetic: a conversion instruction
// issues at an eighth of its rate.  A NaN must be quiet_nan's: arithmetic's own
// (0x7FFFFFFF) would wrap to -0, so the tables and s20_rescale replace it.
__device__ __forceinline__ void split_tf32_int(float x, uint32_t &hi, uint32_t &lo)
{
	hi = (__float_as_uint(x) + 0x1000u) & 0xFFFFE000u;
	lo = (__float_as_uint(x - __uint_as_float(hi)) + 0x1000u) & 0xFFFFE000u;
}

// One child: `x` holds an internal child's rows, `code` a tip's four codes
// (rows [m][h]).
__device__ __forceinline__ void s20_apply(const float *__restrict__ tab, uint32_t id,
					  const int32_t code[2][2], const S20Frag &x,
					  uint32_t lane, S20Frag &out)
{
	const uint32_t q = lane & 3u, r = lane >> 2;
	if (id & kTipBit) {
#pragma unroll
		for (int m = 0; m < 2; m++)
#pragma unroll
			for (int h = 0; h < 2; h++)
#pragma unroll
				for (int s = 0; s < 3; s++)
					out.v[m][h][s] =
						s == 2 && q >= 2
							? make_float2(0.f, 0.f)
							: *reinterpret_cast<const float2 *>(
								  tab + code[m][h] * kS20 + 8 * s + 2 * q);
		return;
	}
	float acc[2][3][4];
#pragma unroll
	for (int m = 0; m < 2; m++)
#pragma unroll
		for (int n = 0; n < 3; n++)
#pragma unroll
			for (int j = 0; j < 4; j++)
				acc[m][n][j] = 0.0f;
#pragma unroll
	for (int s = 0; s < 3; s++) {
		// P halves of K tile s: states 8 s + 2 q (+ 1), columns 8 n + r
		uint32_t bh[3][2], bl[3][2];
#pragma unroll
		for (int n = 0; n < 3; n++)
#pragma unroll
			for (int j = 0; j < 2; j++) {
				const bool pad = (s == 2 && q >= 2) || (n == 2 && r >= 4);
				const float v =
					pad ? 0.0f : tab[(8 * s + 2 * q + j) * kS20 + 8 * n + r];
				split_tf32_int(v, bh[n][j], bl[n][j]);
			}
		uint32_t ah[2][4], al[2][4];
#pragma unroll
		for (int m = 0; m < 2; m++) {
			const float v[4] = {x.v[m][0][s].x, x.v[m][1][s].x, x.v[m][0][s].y,
					    x.v[m][1][s].y};
#pragma unroll
			for (int j = 0; j < 4; j++)
				split_tf32_int(v[j], ah[m][j], al[m][j]);
		}
		// six independent accumulators between two uses of one
#pragma unroll
		for (int m = 0; m < 2; m++)
#pragma unroll
			for (int n = 0; n < 3; n++)
				mma_tf32_k8(acc[m][n], al[m], bh[n][0], bh[n][1]);
#pragma unroll
		for (int m = 0; m < 2; m++)
#pragma unroll
			for (int n = 0; n < 3; n++)
				mma_tf32_k8(acc[m][n], ah[m], bl[n][0], bl[n][1]);
#pragma unroll
		for (int m = 0; m < 2; m++)
#pragma unroll
			for (int n = 0; n < 3; n++)
				mma_tf32_k8(acc[m][n], ah[m], bh[n][0], bh[n][1]);
	}
#pragma unroll
	for (int m = 0; m < 2; m++)
#pragma unroll
		for (int n = 0; n < 3; n++) {
			out.v[m][0][n] = make_float2(acc[m][n][0], acc[m][n][1]);
			out.v[m][1][n] = make_float2(acc[m][n][2], acc[m][n][3]);
		}
}

// Largest of three, NaN if one of them is.
__device__ __forceinline__ float max3_nan(float a, float b, float c)
{
	float r;
	asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
	return r;
}
__device__ __forceinline__ float max_nan(float a, float b)
{
	float r;
	asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
	return r;
}

// Exact power-of-two normalisation of each row's largest entry (20 states
// over four lanes) into [1, 2), adding the exponent to the row's count (see
// rescale_pow2).  The four rows' exchanges overlap.  Of a row with an overflow
// or NaN every entry that is not finite leaves as quiet_nan's NaN (an infinity
// has no tail to split: what is multiplied with one is NaN).
__device__ __forceinline__ void s20_rescale(S20Frag &y, int32_t cnt[2][2])
{
	float m[4];
#pragma unroll
	for (int k = 0; k < 4; k++) {
		const float2 *v = y.v[k >> 1][k & 1];
		m[k] = max3_nan(max3_nan(v[0].x, v[0].y, v[1].x), max_nan(v[1].y, v[2].x), v[2].y);
	}
#pragma unroll
	for (int k = 0; k < 4; k++)
		m[k] = max_nan(m[k], __shfl_xor_sync(0xffffffffu, m[k], 1));
#pragma unroll
	for (int k = 0; k < 4; k++)
		m[k] = max_nan(m[k], __shfl_xor_sync(0xffffffffu, m[k], 2));
	uint32_t rare = 0; // a maximum that is not a positive normal number
#pragma unroll
	for (int k = 0; k < 4; k++)
		rare = max(rare, __float_as_uint(m[k]) - 0x00800000u);
	if (!__any_sync(0xffffffffu, rare >= 0x7F000000u)) {
#pragma unroll
		for (int k = 0; k < 4; k++) {
			const uint32_t e = __float_as_uint(m[k]) & 0x7F800000u;
			const float f = __uint_as_float(0x7F000000u - e); // 2^-exponent
			cnt[k >> 1][k & 1] += (int32_t)(e >> 23) - 127;
#pragma unroll
			for (int s = 0; s < 3; s++) {
				y.v[k >> 1][k & 1][s].x *= f;
				y.v[k >> 1][k & 1][s].y *= f;
			}
		}
		return;
	}
	constexpr float kTiny = 1.17549435e-38f; // smallest normal number
#pragma unroll
	for (int k = 0; k < 4; k++) {
		if (m[k] < kTiny && m[k] > 0.0f) {
			// subnormal maximum: lift by 2^64 first (exact)
			const float lift = 18446744073709551616.0f;
#pragma unroll
			for (int s = 0; s < 3; s++) {
				y.v[k >> 1][k & 1][s].x *= lift;
				y.v[k >> 1][k & 1][s].y *= lift;
			}
			m[k] *= lift;
			cnt[k >> 1][k & 1] -= 64;
		}
		// all zero (the pattern is impossible): no scaling
		const int32_t e =
			m[k] > 0.0f ? (int32_t)((__float_as_uint(m[k]) >> 23) & 0xffu) - 127 : 0;
		const float f = __uint_as_float((uint32_t)(127 - e) << 23);
		cnt[k >> 1][k & 1] += e;
#pragma unroll
		for (int s = 0; s < 3; s++) {
			float2 &v = y.v[k >> 1][k & 1][s];
			v.x *= f;
			v.y *= f;
			v.x = fabsf(v.x) <= 3.402823466e+38f ? v.x : quiet_nan(NAN);
			v.y = fabsf(v.y) <= 3.402823466e+38f ? v.y : quiet_nan(NAN);
		}
	}
}

template <typename Idx, bool kGroups>
__global__ void __launch_bounds__(128, 3) prune20_kernel(PruneParams prm)
{
	extern __shared__ __align__(16) unsigned char s20_smem[];
	const uint32_t lane = threadIdx.x & 31u;
	const uint32_t g = kGroups ? threadIdx.x >> 5 : 0u, G = kGroups ? blockDim.x >> 5 : 1u;
	const uint32_t q = lane & 3u, r = lane >> 2;
	S20Entry *ring = reinterpret_cast<S20Entry *>(s20_smem) + g * kS20Ring;
	__shared__ uint32_t s_last;
	const uint32_t tile = blockIdx.x, c = blockIdx.y, C = prm.C, ldp = prm.ldp;
	const uint32_t p0 = tile * 32u;
	const Idx stride = (Idx)C * ldp, col = (Idx)c * ldp;
	// this lane's first row and state pair; the others: 32 floats a row of
	// 16 patterns, 16 a row of 8, 1,024 a K tile
	float *part = (float *)prm.partials + off20(p0 + r) + 256 * q;
	// a child's rows and counts, or its tip codes, for this lane
	auto load = [&](uint32_t id, S20Frag &x, int32_t sc[2][2]) {
		if (id & kTipBit) {
			const uint8_t *tips = prm.tips + (size_t)(id & ~kTipBit) * ldp + p0 + r;
#pragma unroll
			for (int k = 0; k < 4; k++)
				sc[k >> 1][k & 1] = tips[8 * k]; // 0..20
		} else {
			const Idx ix = (Idx)id * stride + col;
			const float *src = part + (size_t)ix * kS20;
#pragma unroll
			for (int m = 0; m < 2; m++)
#pragma unroll
				for (int h = 0; h < 2; h++)
#pragma unroll
					for (int s = 0; s < 3; s++)
						x.v[m][h][s] = s == 2 && q >= 2
								       ? make_float2(0.f, 0.f)
								       : ld_f2(src + 32 * m + 16 * h +
									       1024 * s);
			const int32_t *cs = prm.scales + ix + p0 + r;
#pragma unroll
			for (int k = 0; k < 4; k++)
				sc[k >> 1][k & 1] = cs[8 * k];
		}
	};
	S20Frag y;
	int32_t cnt[2][2] = {{0, 0}, {0, 0}};
	// prm.segs in shared memory; this warp's next entry to copy: fe of phase
	// fp, until fend
	uint32_t *s_segs =
		reinterpret_cast<uint32_t *>(reinterpret_cast<S20Entry *>(s20_smem) + G * kS20Ring);
	if constexpr (kGroups) {
		for (uint32_t k = threadIdx.x; k <= prm.phases * G; k += blockDim.x)
			s_segs[k] = prm.segs[k];
		__syncthreads();
	}
	uint32_t fp = 0, fe = kGroups ? s_segs[g] : 0, fend = kGroups ? s_segs[g + 1] : prm.n;
	uint32_t slot = 0;
	auto fill = [&] { // the next entry into the next slot
		while (kGroups && fe >= fend && fp + 1 < prm.phases) {
			++fp;
			fe = s_segs[fp * G + g];
			fend = s_segs[fp * G + g + 1];
		}
		if (fe < fend) {
			const float *tab = (const float *)prm.ptab +
					   ((size_t)(2 * fe) * C + c) * (kP20Rows * kS20);
			uint4 *dst = (uint4 *)(ring + slot);
			const uint4 *s0 = (const uint4 *)tab;
			const uint4 *s1 = (const uint4 *)(tab + (size_t)C * (kP20Rows * kS20)) -
					  kS20TabChunks;
#pragma unroll
			for (uint32_t k = 0; k < 7; ++k) {
				const uint32_t at = lane + 32 * k;
				if (at < 2 * kS20TabChunks)
					cp_async16(dst + 1 + at,
						   (at < kS20TabChunks ? s0 : s1) + at);
			}
			if (lane == 0)
				cp_async16(dst, prm.ops + fe);
			++fe;
		}
		cp_async_commit();
		slot = slot + 1 == kS20Ring ? 0 : slot + 1;
	};
#pragma unroll
	for (uint32_t e = 0; e < kS20Ring - 1; ++e)
		fill();
	uint32_t cur = 0; // ring slot of the current entry
	// entries [lo, hi) of one phase
	auto walk = [&](uint32_t lo, uint32_t hi) {
		if (lo >= hi)
			return;
		cp_async_wait<kS20Ring - 2>(); // the first entry has landed
		__syncwarp();
		NodeOp op = ring[cur].op;
		S20Frag x1;
		int32_t s1[2][2];
		load((op.pad & kS20Swap) ? op.right : op.left, x1, s1);
		for (uint32_t e = lo; e < hi; ++e) {
			const S20Entry &en = ring[cur];
			const uint32_t f = (op.pad & kS20Swap) ? 1u : 0u;
			const uint32_t first = f ? op.right : op.left;
			const uint32_t second = f ? op.left : op.right;
			// the second side: the previous output, a tip's codes, or
			// (two clean children) rows from memory
			int32_t s2[2][2];
			if (op.pad & kS20Prev) {
#pragma unroll
				for (int k = 0; k < 4; k++)
					s2[k >> 1][k & 1] = cnt[k >> 1][k & 1];
			} else {
				load(second, y, s2);
			}
			S20Frag a;
			s20_apply(en.tab[f], first, s1, x1, lane, a);
#pragma unroll
			for (int k = 0; k < 4; k++)
				cnt[k >> 1][k & 1] = ((first & kTipBit) ? 0 : s1[k >> 1][k & 1]) +
						     ((second & kTipBit) ? 0 : s2[k >> 1][k & 1]);
			fill(); // the slot of the entry before this one
			cp_async_wait<kS20Ring - 2>(); // the next entry has landed
			__syncwarp();
			const uint32_t nxt = cur + 1 == kS20Ring ? 0 : cur + 1;
			NodeOp nop = op;
			if (e + 1 < hi) {
				nop = ring[nxt].op;
				load((nop.pad & kS20Swap) ? nop.right : nop.left, x1, s1);
			}
			S20Frag b;
			s20_apply(en.tab[f ^ 1u], second, s2, y, lane, b);
#pragma unroll
			for (int m = 0; m < 2; m++)
#pragma unroll
				for (int h = 0; h < 2; h++)
#pragma unroll
					for (int s = 0; s < 3; s++) {
						y.v[m][h][s].x = a.v[m][h][s].x * b.v[m][h][s].x;
						y.v[m][h][s].y = a.v[m][h][s].y * b.v[m][h][s].y;
					}
			s20_rescale(y, cnt);
			const Idx ox = (Idx)op.out * stride + col;
			float *dst = part + (size_t)ox * kS20;
#pragma unroll
			for (int m = 0; m < 2; m++)
#pragma unroll
				for (int h = 0; h < 2; h++) {
#pragma unroll
					for (int s = 0; s < 3; s++)
						if (s < 2 || q < 2)
							*reinterpret_cast<float2 *>(
								dst + 32 * m + 16 * h + 1024 * s) =
								y.v[m][h][s];
					if (q == 0)
						prm.scales[ox + p0 + r + 16 * m + 8 * h] = cnt[m][h];
				}
			op = nop;
			cur = nxt;
		}
	};
	if constexpr (kGroups) {
		for (uint32_t ph = 0; ph < prm.phases; ++ph) {
			walk(s_segs[ph * G + g], s_segs[ph * G + g + 1]);
			__syncthreads(); // the phase's outputs are visible to every warp
		}
		if (g != 0) // warp 0 walked the last entry, the root
			return;
	} else {
		walk(0, prm.n);
	}
	double *root_val = prm.root_val + (size_t)c * ldp + p0;
	int32_t *root_exp = prm.root_exp + (size_t)c * ldp + p0;
	double pi[3][2]; // read together
#pragma unroll
	for (int s = 0; s < 3; s++) {
		const bool pad = s == 2 && q >= 2;
		pi[s][0] = pad ? 0.0 : prm.pi[8 * s + 2 * q];
		pi[s][1] = pad ? 0.0 : prm.pi[8 * s + 2 * q + 1];
	}
#pragma unroll
	for (int m = 0; m < 2; m++)
#pragma unroll
		for (int h = 0; h < 2; h++) {
			double dot = 0.0;
#pragma unroll
			for (int s = 0; s < 3; s++)
				if (s < 2 || q < 2) {
					dot = fma(pi[s][0], (double)y.v[m][h][s].x, dot);
					dot = fma(pi[s][1], (double)y.v[m][h][s].y, dot);
				}
			dot += __shfl_xor_sync(0xffffffffu, dot, 1);
			dot += __shfl_xor_sync(0xffffffffu, dot, 2);
			if (q == 0) {
				root_val[16 * m + 8 * h + r] = dot;
				root_exp[16 * m + 8 * h + r] = cnt[m][h];
			}
		}
	__threadfence();
	__syncwarp();
	const uint32_t p = p0 + lane;
	if (prm.cat_lnl)
		prm.cat_lnl[(size_t)c * ldp + p] =
			log(__ldcg(root_val + lane)) +
			(double)__ldcg(root_exp + lane) * 0.69314718055994530942;
	if (lane == 0) {
		const unsigned tk = atomicAdd(prm.ticket + tile, 1u);
		s_last = tk == C - 1u;
		if (tk == C - 1u)
			prm.ticket[tile] = 0u;
		__threadfence();
	}
	__syncwarp();
	if (!s_last)
		return;
	const RootColumns root(prm, p, (double *)s20_smem + lane, 32);
	const double site = mix_categories_pow2(
		C, [&](uint32_t k) { return root.val(k); },
		[&](uint32_t k) { return root.exp(k); }, prm.log_inv_c);
	prm.site_lnl[p] = site;
	const uint32_t w = prm.weights[p];
	double contrib = w ? site * (double)w : 0.0;
	for (int off = 16; off > 0; off >>= 1)
		contrib += __shfl_down_sync(0xffffffffu, contrib, off);
	if (lane == 0)
		prm.sums_host[tile] = contrib;
}
