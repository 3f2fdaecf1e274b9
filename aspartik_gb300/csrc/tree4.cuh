// tree4.cuh -- depth-first FP32 pruning walk of whole-tree (and other
// single-tree) lists.  Included by kernels4.cu inside its anonymous namespace
// after runs4.cuh (uses v4_apply_pair, v4_mul, rescale_pow2, root_dot4,
// pattern_root and the cp.async helpers).
//
// Every output is stored for later evaluations, so no walk beats the time of
// those stores (20 bytes a column and entry).  What kept the run-synchronous
// walk away from it were its instructions (163 a column's warp-entry: the
// schedule, sources and addresses decoded by every group, every child through
// shared memory) and a barrier a run.  Here a warp owns 64 patterns of one
// category and walks a list depth first (heavier subtree first), so that two
// thirds of the internal children of a random tree are the previous entry's
// output and stay in registers; the others wait in a shared-memory slot that
// the host assigned (Calculator::stage_tree), and so do the clean
// children of a list that is not the whole tree, copied there early.
//
// Lane l holds patterns 2l and 2l + 1: the table rows are read once for both
// columns, a tip child's two codes are one 16-bit read, the outputs of a
// column pair one 32-byte store.  Tables and schedule words arrive by
// cp.async in chunks of four entries, 16-byte pieces whose addresses advance
// by a constant.
//
// One such warp a column set leaves the GPU with too few warps (two a
// scheduler at the largest workload), so a block holds several groups of C
// warps on the same patterns: the host splits the list into phases, disjoint
// subtrees a group first, then the entries above them, with a barrier after
// each phase.
//
// Kernel time of a whole tree, the run walk -> this: 256 taxa x 17,764 patterns
// x 4 categories 106 -> 69 us (362 MB stored, 5.2 TB/s; 42 us is what the SMs'
// store ports need, 50 us DRAM); 64 x 7,855 x 4 30 -> 20 us, of which the
// tables, the prologue and the root are half.  No unit is full (of the active
// cycles at 8 warps an SM: busiest L1 unit 67 %, issue slots 43 %); its warps
// wait on fixed latencies and shared-memory reads.  16 warps an SM (four
// groups) were no faster (91 against 88 us a call), more at fewer registers
// spill and were slower (96 -> 113 us).
struct __align__(16) TreeEntry {
	float4 tab[10]; // first child's four rows and ones, second's
	TreeOp op;
};
constexpr uint32_t kTreePieces = kTreeChunk * (sizeof(TreeEntry) / 16);
static_assert(kTreePieces > 32 && kTreePieces <= 64, "two pieces a lane");

// Shared memory of a slot for one category's 64 columns, and of a warp's ring.
constexpr uint32_t kTreeColBytes = sizeof(float4) + sizeof(int32_t);
constexpr uint32_t kTreeRingBytes = kTreeRing * sizeof(TreeEntry);

// Two neighbouring columns' vectors in one 32-byte store.
__device__ __forceinline__ void store_pair(float4 *dst, const float4 &a, const float4 &b)
{
	asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst),
		     "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z),
		     "f"(b.w)
		     : "memory");
}

// rescale_pow2 of two vectors, with one test for the rare subnormal or zero
// maximum.
__device__ __forceinline__ void rescale_pair(float4 &a, float4 &b, int2 &cnt)
{
	const float ma = fmaxf(fmaxf(a.x, a.y), fmaxf(a.z, a.w));
	const float mb = fmaxf(fmaxf(b.x, b.y), fmaxf(b.z, b.w));
	const uint32_t ea = __float_as_uint(ma) & 0x7F800000u;
	const uint32_t eb = __float_as_uint(mb) & 0x7F800000u;
	if (min(ea, eb) == 0u) {
		cnt.x += rescale_pow2(a);
		cnt.y += rescale_pow2(b);
		return;
	}
	const float fa = __uint_as_float(0x7F000000u - ea), fb = __uint_as_float(0x7F000000u - eb);
	a = make_float4(a.x * fa, a.y * fa, a.z * fa, a.w * fa);
	b = make_float4(b.x * fb, b.y * fb, b.z * fb, b.w * fb);
	cnt.x += (int32_t)(ea >> 23) - 127;
	cnt.y += (int32_t)(eb >> 23) - 127;
}

// Two products of neighbouring values in one instruction each.
__device__ __forceinline__ float4 mul_pairs(const float4 &a, const float4 &b)
{
	float4 r;
	asm("{\n\t.reg .b64 p, q;\n\t"
	    "mov.b64 p, {%4, %5};\n\tmov.b64 q, {%8, %9};\n\t"
	    "mul.rn.f32x2 p, p, q;\n\tmov.b64 {%0, %1}, p;\n\t"
	    "mov.b64 p, {%6, %7};\n\tmov.b64 q, {%10, %11};\n\t"
	    "mul.rn.f32x2 p, p, q;\n\tmov.b64 {%2, %3}, p;\n\t}"
	    : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w)
	    : "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w));
	return r;
}

// sum_k x_k * row_k for a lane's vectors with the same four table rows.
template <uint32_t kV>
__device__ __forceinline__ void apply_rows(const float4 *tab, float4 (&x)[kV])
{
	const float4 r[4] = {tab[0], tab[1], tab[2], tab[3]};
#pragma unroll
	for (uint32_t v = 0; v < kV; ++v)
		x[v] = v4_apply(r, x[v]);
}

// One tile of a list: returns its weighted site sum in thread 0, the block
// synchronised.  Block = `groups` x C warps (further ones only keep the
// barriers), 64 kR patterns (lane l: 2l and 2l + 1 of every
// 64).  Dynamic shared memory: [dot: C x tile floats][cnt: C x tile][a part a
// category: its groups' rings, its slots' vectors (for every 64 columns the
// even ones, then the odd ones), their counts][tips: num_leaves + 1 rows,
// kTips].  kTips: the tile's tip codes are in
// shared memory.  kClean: the list has children outside it.
//
// The schedule is linear for a group; an entry's word also has what is read
// ahead for the two entries after it, so that nothing but the word and the
// values read is carried from one entry to the next.  A second child's
// vectors, table rows or slot, are read by one formula: base + 16 x code for
// each column, the codes of a slot child being the lane's place in it (the
// row behind the last leaf's).
template <uint32_t kR, bool kTips, bool kClean>
__device__ __forceinline__ double tree_tile(const PruneParams &prm, uint32_t t, double *smem)
{
	const uint32_t C = prm.C, G = prm.groups;
	const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
	const uint32_t g = wid / C, c = wid - g * C;
	constexpr uint32_t kTreeTile = 64 * kR;
	const uint32_t p0 = t * kTreeTile;
	float *s_dot = (float *)smem;
	int32_t *s_cnt = (int32_t *)(s_dot + C * kTreeTile);
	const uint32_t part_bytes = G * kTreeRingBytes + prm.n_slots * (kTreeTile * kTreeColBytes);
	char *base = (char *)(s_cnt + C * kTreeTile) + c * part_bytes;
	uint8_t *s_tips = (uint8_t *)(s_cnt + C * kTreeTile) + C * part_bytes;
	TreeEntry *ring = (TreeEntry *)(base + g * kTreeRingBytes);
	float4 *sx = (float4 *)(base + G * kTreeRingBytes) + lane;
	int2 *sc = (int2 *)(base + G * kTreeRingBytes + prm.n_slots * (kTreeTile * 16u)) + lane;

	// segs: first entry of every group, n, then the groups' heads
	const bool walks = g < G;
	const uint32_t first = walks ? prm.segs[g] : 0u;
	const uint32_t count = walks ? prm.segs[g + 1] - first : 0u;
	TreeHead head{};
	if (walks)
		head = ((const TreeHead *)(prm.segs + G + 1))[g];
	else
		head.barriers = prm.phases - 1;
	const size_t col = (size_t)c * prm.ldp + p0 + 2 * lane;
	const uint32_t stride = C * prm.ldp;
	float4 *part = (float4 *)prm.partials + col;
	int32_t *scales = prm.scales + col;
	const TreeOp *tree_ops = (const TreeOp *)prm.ops;
	const uint32_t stride16 = stride * 16u, stride4 = stride * 4u;
	// this lane's two pieces of a chunk
	const char *src[2];
	uint32_t step[2], dst[2], of[2];
#pragma unroll
	for (uint32_t j = 0; j < 2; ++j) {
		const uint32_t k = lane + 32 * j, e = k / 12u, pc = k - e * 12u;
		of[j] = k < kTreePieces ? e : 0x80000000u;
		dst[j] = (uint32_t)__cvta_generic_to_shared(ring) + e * sizeof(TreeEntry) +
			 pc * 16u;
		if (pc < 10) {
			const uint32_t side = pc / 5u;
			src[j] = (const char *)prm.ptab +
				 ((size_t)(2 * (first + e) + side) * C + c) * 80u +
				 (pc - side * 5u) * 16u;
			step[j] = kTreeChunk * C * 160u;
		} else {
			src[j] = (const char *)(tree_ops + first + e) + (pc - 10u) * 16u;
			step[j] = kTreeChunk * sizeof(TreeOp);
		}
	}
	// chunk q, and the clean children of chunk q - 1 (whose words are here)
	auto fill = [&](uint32_t q) {
		const uint32_t at = (q & 3u) * (kTreeChunk * sizeof(TreeEntry));
#pragma unroll
		for (uint32_t j = 0; j < 2; ++j) {
			if (q * kTreeChunk + of[j] < count)
				asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
						     dst[j] + at),
					     "l"(src[j])
					     : "memory");
			src[j] += step[j];
		}
		if constexpr (kClean) {
			for (uint32_t e = (q - 1) * kTreeChunk;
			     q > 0 && e < q * kTreeChunk && e < count; ++e) {
				const TreeOp &op = ring[e & (kTreeRing - 1)].op;
#pragma unroll
				for (uint32_t j = 0; j < 2; ++j) {
					if (!(op.more & (j ? kTreeCleanB : kTreeCleanA)))
						continue;
					const uint32_t s = op.more >> (j ? 16 : 8) & 0xFFu;
					const size_t ix = (size_t)op.id[j] * stride;
#pragma unroll
					for (uint32_t r = 0; r < kR; ++r) {
						const size_t x = ix + 64 * r;
						int32_t *n = (int32_t *)(sc + (s * kR + r) * 32);
						cp_async16(sx + (s * kR + r) * 64, part + x);
						cp_async16(sx + (s * kR + r) * 64 + 32,
							   part + x + 1);
						cp_async4(n, scales + x);
						cp_async4(n + 1, scales + x + 1);
					}
				}
			}
		}
		cp_async_commit();
	};
	if constexpr (kTips) {
		constexpr uint32_t kRow = kTreeTile / 16; // pieces of a row
		for (uint32_t k = threadIdx.x; k < prm.num_leaves * kRow; k += blockDim.x)
			cp_async16((uint4 *)s_tips + k, prm.tips + (size_t)(k / kRow) * prm.ldp +
								p0 + (k % kRow) * 16u);
		cp_async_commit();
		for (uint32_t h = wid; h < kR; h += C * G)
			((uint16_t *)(s_tips + prm.num_leaves * kTreeTile))[h * 32 + lane] =
				(uint16_t)((h * 64 + lane) | (h * 64 + lane + 32u) << 8);
	}
	wait_for_tables();
	fill(0);
	if (kClean) { // chunk 0's words
		cp_async_wait<0>();
		__syncwarp();
	}
	fill(1);
	cp_async_wait<0>();
	__syncthreads(); // the tips and two chunks are here
	fill(2);
	const uint8_t *tips = kTips ? s_tips + 2 * lane : prm.tips + p0 + 2 * lane;
	struct Codes {
		uint32_t v[kR]; // columns 2l, 2l + 1 of every 64
	};
	auto codes = [&](uint32_t tip) { // kTips: a byte offset
		Codes c;
#pragma unroll
		for (uint32_t r = 0; r < kR; ++r) {
			const uint32_t at = r * 64 + lane;
			if constexpr (kTips)
				c.v[r] = *(const uint16_t *)(tips + tip + r * 64);
			else if (tip == kTreeNoTip)
				c.v[r] = at | (at + 32u) << 8;
			else
				c.v[r] = *(const uint16_t *)(tips + (size_t)tip * prm.ldp +
							     r * 64);
		}
		return c;
	};
	struct Vecs {
		float4 v[2 * kR];
	};
	auto rows = [&](const char *b, const Codes &code, Vecs &x) {
#pragma unroll
		for (uint32_t r = 0; r < kR; ++r) {
			x.v[2 * r] = *(const float4 *)(b + (code.v[r] & 0xFFu) * 16u);
			x.v[2 * r + 1] = *(const float4 *)(b + (code.v[r] >> 8) * 16u);
		}
	};
	auto slot_counts = [&](uint32_t s, int2 (&n)[kR]) {
#pragma unroll
		for (uint32_t r = 0; r < kR; ++r)
			n[r] = sc[(s * kR + r) * 32];
	};
	auto memory = [&](uint32_t id, Vecs &x, int2 (&n)[kR]) {
#pragma unroll
		for (uint32_t r = 0; r < kR; ++r) {
			const size_t ix = (size_t)id * stride + 64 * r;
			x.v[2 * r] = part[ix];
			x.v[2 * r + 1] = part[ix + 1];
			n[r] = *(const int2 *)(scales + ix);
		}
	};
	auto barriers = [&](uint32_t count) {
		for (; count; --count)
			__syncthreads(); // a phase's outputs are visible to every group
	};

	Vecs y{};
	int2 cnt[kR] = {};
	// one entry: its word, tables, first child's codes and second child, and
	// the same for the next
	auto entry = [&](const TreeEntry &en, const uint4 &op, const Codes &ca, Vecs &b,
			 const TreeEntry &next, uint4 &op1, Codes &ca1, Vecs &b1, Codes &cb) {
		const float4 *tab = en.tab;
		const Codes cb1 = cb;
		rows(base + (op.y >> 16) * 16u, cb1, b1);
		op1 = *(const uint4 *)&next.op;
		ca1 = codes(op.z);
		cb = codes(op.w);
		// two kinds of entry of a whole tree in straight code of their own
		// (previous x tip, cherry), anything else through slots or memory
		const uint32_t kind = op.y & kTreeKind;
		if (kind == kTreePrevTip) {
			apply_rows(tab, y.v);
		} else if (kind == kTreeTipTip) {
			rows((const char *)tab, ca, y);
#pragma unroll
			for (uint32_t r = 0; r < kR; ++r)
				cnt[r] = make_int2(0, 0);
		} else {
			int2 cs[kR] = {};
			if (op.y & kTreeInB) {
				if (op.y & kTreeMemB)
					memory(en.op.id[1], b, cs);
				else
					slot_counts(en.op.more >> 16 & 0xFFu, cs);
				apply_rows(tab + 5, b.v);
			}
			if (op.y & kTreeInA) {
				if (op.y & kTreeMemA) {
					memory(en.op.id[0], y, cnt);
				} else if (!(op.y & kTreePrev)) {
					const uint32_t s = en.op.more >> 8 & 0xFFu;
#pragma unroll
					for (uint32_t v = 0; v < 2 * kR; ++v)
						y.v[v] = sx[s * kTreeTile + v * 32];
					slot_counts(s, cnt);
				}
				apply_rows(tab, y.v);
			} else {
				rows((const char *)tab, ca, y);
#pragma unroll
				for (uint32_t r = 0; r < kR; ++r)
					cnt[r] = make_int2(0, 0);
			}
#pragma unroll
			for (uint32_t r = 0; r < kR; ++r) {
				cnt[r].x += cs[r].x;
				cnt[r].y += cs[r].y;
			}
		}
#pragma unroll
		for (uint32_t r = 0; r < kR; ++r) {
			y.v[2 * r] = mul_pairs(y.v[2 * r], b.v[2 * r]);
			y.v[2 * r + 1] = mul_pairs(y.v[2 * r + 1], b.v[2 * r + 1]);
			rescale_pair(y.v[2 * r], y.v[2 * r + 1], cnt[r]);
		}
		char *po = (char *)part + (size_t)op.x * stride16;
		char *so = (char *)scales + (size_t)op.x * stride4;
#pragma unroll
		for (uint32_t r = 0; r < kR; ++r) {
			store_pair((float4 *)po + 64 * r, y.v[2 * r], y.v[2 * r + 1]);
			*((int2 *)so + 32 * r) = cnt[r];
		}
		if (op.y & (kTreeKeep | kTreeBarrier)) {
			if (op.y & kTreeKeep) {
				const uint32_t s = op.y >> 8 & 0xFFu;
#pragma unroll
				for (uint32_t v = 0; v < 2 * kR; ++v)
					sx[s * kTreeTile + v * 32] = y.v[v];
#pragma unroll
				for (uint32_t r = 0; r < kR; ++r)
					sc[(s * kR + r) * 32] = cnt[r];
			}
			if (op.y & kTreeBarrier) { // and the next entry's slot is filled
				barriers(en.op.barriers);
				rows(base + (op.y >> 16) * 16u, cb1, b1);
			}
		}
	};
	barriers(head.barriers);
	if (count) {
		Codes caa = codes(head.tip[0]), cab = caa, cb = codes(head.tip[1]);
		Vecs ba, bb;
		uint4 opa = *(const uint4 *)&ring[0].op, opb = opa;
		rows(base + head.base * 16u, cb, ba);
		cb = codes(head.tip[2]);
#pragma unroll 1
		for (uint32_t k = 0;; k += 2) {
			if ((k & (kTreeChunk - 1)) == 0) {
				// the chunks of entries k .. k + 7 have landed, the one
				// before k is free (and with clean children, whose words
				// the fill reads, the chunk after those has landed too)
				cp_async_wait<kClean ? 0 : 1>();
				__syncwarp();
				fill(k / kTreeChunk + 3);
			}
			const TreeEntry *at = ring + (k & (kTreeRing - 1));
			entry(at[0], opa, caa, ba, at[1], opb, cab, bb, cb);
			if (k + 1 >= count)
				break;
			entry(at[1], opb, cab, bb, ring[(k + 2) & (kTreeRing - 1)], opa, caa, ba,
			      cb);
			if (k + 2 >= count)
				break;
		}
	}
	if (g == 0) {
		const float pi[4] = {(float)prm.pi[0], (float)prm.pi[1], (float)prm.pi[2],
				     (float)prm.pi[3]};
#pragma unroll
		for (uint32_t v = 0; v < 2 * kR; ++v) {
			const uint32_t at = c * kTreeTile + (v >> 1) * 64 + 2 * lane + (v & 1u);
			s_dot[at] = root_dot4(pi, y.v[v]);
			s_cnt[at] = v & 1u ? cnt[v >> 1].y : cnt[v >> 1].x;
		}
	}
	__syncthreads();
	// tile_root's arithmetic; one warp takes 32 patterns at a time
	__shared__ double s_red[2 * kR];
	for (uint32_t h = wid; h < 2 * kR; h += C * G) {
		const uint32_t k = h * 32 + lane;
		double sum = pattern_root(s_dot, s_cnt, kTreeTile, C, k, prm.ldp, p0 + k,
					  prm.log_inv_c, prm.site_lnl, prm.cat_lnl,
					  prm.weights);
		for (int off = 16; off > 0; off >>= 1)
			sum += __shfl_down_sync(0xffffffffu, sum, off);
		if (lane == 0)
			s_red[h] = sum;
	}
	__syncthreads();
	double sum = 0.0;
	for (uint32_t h = 0; h < 2 * kR; ++h)
		sum += s_red[h];
	return sum;
}

template <uint32_t kR, bool kTips, bool kClean>
__global__ void __launch_bounds__(512) prune4_tree_kernel(PruneParams prm)
{
	extern __shared__ __align__(16) double smem[];
	const double sum = tree_tile<kR, kTips, kClean>(prm, blockIdx.x, smem);
	if (threadIdx.x == 0)
		prm.sums_host[blockIdx.x] = sum;
}

// The long single-tree lists of a batch, 64 patterns and as many groups as a
// block of 16 warps has: two lists of 183 entries x 1,664 patterns x 4
// categories 37 us on 52 SMs, where the run walk's tiles took 62 us on all of
// them; the short lists' blocks run on the others meanwhile (a step of 32
// chains, two whole trees and 30 paths, 105 -> 69 us on the device).
__global__ void __launch_bounds__(512) prune4_tree_batch_kernel(BatchParams bp)
{
	extern __shared__ __align__(16) double smem[];
	__shared__ uint32_t s_prefix[kBatchMembers + 1];
	__shared__ unsigned s_last;
	const uint32_t M = bp.num_members;
	member_prefix(M, s_prefix, [&](uint32_t m) {
		const MemberStep &st = bp.steps[m];
		return st.n && st.kind == kListTree ? bp.members[m].ldp / 64u : 0u;
	});
	const uint32_t total = s_prefix[M];
	for (uint32_t w = blockIdx.x; w < total; w += gridDim.x) {
		const uint32_t m = member_of(s_prefix, M, w), t = w - s_prefix[m];
		const MemberDesc &md = bp.members[m];
		const MemberStep &st = bp.steps[m];
		PruneParams prm{};
		prm.tips = md.tips;
		prm.partials = md.partials;
		prm.scales = md.scales;
		prm.ops = (const NodeOp *)(md.stage + md.off_tree);
		prm.ptab = md.ptab;
		prm.segs = (const uint32_t *)(md.stage + md.off_runs);
		prm.groups = st.groups;
		prm.phases = st.phases;
		prm.pi = (const double *)(md.stage + md.off_pi);
		prm.weights = md.weights;
		prm.site_lnl = md.site_lnl;
		prm.n = st.n;
		prm.ldp = md.ldp;
		prm.C = md.C;
		prm.num_leaves = md.L;
		prm.n_slots = st.n_slots;
		prm.log_inv_c = md.log_inv_c;
		const double sum = !st.tips_smem ? tree_tile<1, false, true>(prm, t, smem)
				   : st.clean    ? tree_tile<1, true, true>(prm, t, smem)
						 : tree_tile<1, true, false>(prm, t, smem);
		const uint32_t tiles = md.ldp / 64u;
		if (threadIdx.x == 0) {
			md.tile_sums[t] = sum;
			__threadfence();
			s_last = atomicAdd(md.ticket, 1u) == tiles - 1u;
		}
		__syncthreads();
		if (s_last) {
			__threadfence();
			const double lnl = block_fold(md.tile_sums, tiles, nullptr);
			if (threadIdx.x == 0) {
				bp.lnl_out[m] = lnl;
				*md.ticket = 0u;
			}
		}
		__syncthreads();
	}
}
